"""Performance cases of the MR-fingerprinting path: dictionary generation,
matching, refinement, derivatives and compression, called as a user's program
calls them (snapmrf_b200), over the sizes of this repository's configurations
and the ranges around them.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call, on the GPU
  run(state)          one pass through the public entry points
  work(case)          bytes and operations that pass cannot do without
  exact(case, seed)   what run returns, in plain 64-bit torch

The inputs (schedules, dictionaries to match against, voxels) are made here
with torch, not by the library.  Schedules are the repository's: flip angles
lo + amp |sin(pi t / period)|, TR uniform in a 4 ms window, TE = TR / 2.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import snapmrf_b200 as snap

PI = math.pi


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # the smallest whole map: 837 atoms, a 64 x 64 slice, FP32 as the
        # mrf command runs it by default (no B1 map, no flags)
        dict(name="map_small", kind="map", nt1=30, nt2=29, grid="linear", nx=64, T=1000, w=20),
        # the B1-mapped dictionary of the headline map: 6,938 (T1, T2) pairs x
        # 41 B1 values, imaginary rows, norms and the BF16 matching operand
        dict(name="dict_fisp_b1", kind="dict_fisp", step=0.05, nb1=41, T=1000, w=50, form="operand"),
        # bSSFP with off-resonance (the reference's default echo type)
        dict(name="dict_ssfp_b0", kind="dict_ssfp", step=0.05, nb0=8, nb1=2, T=500, w=50),
        # ROA Bloch simulation, 100 isochromats per atom
        dict(name="dict_roa_iso", kind="dict_roa", step=0.05, nb0=8, n_iso=100, T=500),
        # a 240 x 240 slice matched in FP32 within each voxel's B1 block
        dict(name="match_fp32_b1", kind="match_b1", step=0.05, nb1=41, nx=240, T=1000, w=50, precision="fp32"),
        # the headline match: BF16 scores, top-16 rescored in FP32
        dict(name="match_bf16_b1", kind="match_b1", step=0.05, nb1=41, nx=240, T=1000, w=50, precision="bf16"),
        # bSSFP atoms (complex), no B1 map: every voxel against every atom
        dict(name="match_fp16_ssfp", kind="match_all", step=0.05, nb0=8, nb1=2, nx=128, T=500, w=50,
             precision="fp16"),
        # sub-grid start and Gauss-Newton refinement of a matched 240 x 240 slice
        dict(name="refine_fisp", kind="refine_fisp", step=0.05, nb1=41, nx=240, T=1000, w=50),
        # bSSFP refinement of T1, T2, B0 and B1 of one 128 x 128 slice
        dict(name="refine_ssfp", kind="refine_ssfp", nx=128, T=500, w=50, b1map=False),
        # backward pass of the signal for 4,096 atoms: dL/d(T1, T2, B1) and the schedule
        dict(name="adjoint_fisp", kind="adjoint", echo="epg_fisp", n=4096, T=1000, w=50),
        # one step of a schedule design loop: Cramer-Rao bounds of three tissues
        # and their flip-angle gradient (a small call, all latency)
        dict(name="crb_design", kind="crb", n=3, T=1000, w=50),
        # low-rank compression of five B1 blocks
        dict(name="svd_compress", kind="svd", step=0.05, nb1=5, T=1000, w=50),
    ]


KINDS = ("map", "dict_fisp", "dict_ssfp", "dict_roa", "match_b1", "match_all", "refine_fisp", "refine_ssfp",
         "adjoint", "crb", "svd")


def draw(rng) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(KINDS)
    T = rng.choice([rng.randint(200, 1000), 1000, 500, 2 * rng.randint(100, 500)])
    w = rng.choice([20, 50, rng.randint(12, 64)])
    step = rng.choice([0.05, round(rng.uniform(0.05, 0.2), 3)])
    if kind == "map":
        return dict(kind=kind, nt1=rng.randint(10, 40), nt2=rng.randint(10, 40), grid="linear", nx=log(8, 96), T=T, w=w)
    if kind == "dict_fisp":
        return dict(kind=kind, step=step, nb1=log(1, 41), T=T, w=w, form=rng.choice(["operand", "complex", "unit"]))
    if kind == "dict_ssfp":
        return dict(kind=kind, step=step, nb0=log(1, 8), nb1=rng.randint(1, 2), T=min(T, 500), w=w)
    if kind == "dict_roa":
        return dict(kind=kind, step=step, nb0=log(1, 8), n_iso=rng.choice([1, 1, 100, rng.randint(2, 128)]),
                    T=min(T, 500))
    if kind == "match_b1":
        return dict(kind=kind, step=step, nb1=log(2, 41), nx=log(16, 240), T=T, w=50,
                    precision=rng.choice(["fp32", "bf16", "fp16"]))
    if kind == "match_all":
        return dict(kind=kind, step=max(step, 0.06), nb0=log(1, 8), nb1=rng.randint(1, 2), nx=log(8, 96),
                    T=min(T, 500), w=w, precision=rng.choice(["fp32", "fp16"]))
    if kind == "refine_fisp":
        return dict(kind=kind, step=0.05, nb1=log(3, 41), nx=log(16, 240), T=T, w=w)
    if kind == "refine_ssfp":
        return dict(kind=kind, nx=log(16, 128), T=min(T, 500), w=w, b1map=rng.random() < 0.5)
    if kind == "adjoint":
        echo = rng.choice(["epg_fisp", "epg_ssfp"])
        return dict(kind=kind, echo=echo, n=log(16, 4096) if echo == "epg_fisp" else log(16, 1024),
                    T=T if echo == "epg_fisp" else min(T, 500), w=w)
    if kind == "crb":
        return dict(kind=kind, n=log(1, 64), T=T, w=w)
    return dict(kind=kind, step=max(step, 0.06), nb1=rng.randint(1, 5), T=T, w=50)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float32)


def _fisp_schedule(T, seed, inversion=True):
    """h_mrf [4][T]: flip (rad), phase, TR, TE (ms), as epg_fisp takes them."""
    r = np.random.default_rng(seed)
    a = 10.0 + 50.0 * np.abs(np.sin(PI * np.arange(T) / 250.0))
    if inversion:
        a[0] = 180.0
    tr = r.uniform(11.0, 15.0, T)
    return np.array([np.deg2rad(a), np.zeros(T), tr, tr / 2], np.float32)


def _ssfp_schedule(T, seed):
    """h_mrf [4][T] in the CSV convention of epg_ssfp / roa_ssfp: flip as a
    fraction of 60 deg, phase in degrees, TR - 16 ms, TE - 3.5 ms."""
    r = np.random.default_rng(seed)
    t = np.arange(T)
    a = 5.0 + 55.0 * np.abs(np.sin(PI * t / 200.0))
    tr = r.uniform(10.0, 14.0, T)
    return np.array([a / 60.0, 180.0 * (t % 2), tr - 16.0, tr / 2 - 3.5], np.float32)


def _geometric(lo, hi, step):
    n = int(math.floor(math.log(hi / lo) / math.log1p(step) + 1e-9)) + 1
    return (lo * (1.0 + step) ** np.arange(n)).astype(np.float32)


def _grid(case):
    """(params [NATOMS][4], atoms per B1 block, B1 values)."""
    if case.get("grid") == "linear":
        t1 = np.arange(1, case["nt1"] + 1, dtype=np.float32) * 100
        t2 = 20 + np.arange(case["nt2"], dtype=np.float32) * 10
    else:
        t1, t2 = _geometric(100.0, 5000.0, case["step"]), _geometric(10.0, 2000.0, case["step"])
    nb1, nb0 = case.get("nb1", 1), case.get("nb0", 1)
    if case["kind"] in ("dict_ssfp", "match_all"):
        b1 = (0.9 + 0.1 * np.arange(nb1)).astype(np.float32)
    else:
        b1 = (1.0 + 0.02 * (np.arange(nb1) - nb1 // 2)).astype(np.float32)
    b0 = ((np.arange(nb0) - nb0 // 2) * 12.0).astype(np.float32)
    p = snap.trans_params(t1, t2, b0, b1)
    return p, p.shape[0] // nb1, b1


def _tissue(g, n, seed, t1=(300.0, 3000.0), t2=(30.0, 400.0)):
    """(T1, T2) of n voxels: five tissues, +-5 % per voxel."""
    r = np.random.default_rng(seed)
    c1 = r.uniform(*t1, 5)
    c2 = np.array([r.uniform(t2[0], min(t2[1], v / 3)) for v in c1])
    k = torch.randint(0, 5, (n,), generator=g, device="cuda")
    a = torch.tensor(c1, device="cuda", dtype=torch.float32)[k] * _uniform(g, n, 0.95, 1.05)
    b = torch.tensor(c2, device="cuda", dtype=torch.float32)[k] * _uniform(g, n, 0.95, 1.05)
    return a, b


def _b1_field(nx, lo, hi):
    """The smooth field 1 + 0.3 (x^2 + y^2 - 0.5), clipped to the B1 values."""
    v = torch.linspace(-1, 1, nx, device="cuda", dtype=torch.float32)
    f = 1 + 0.3 * (v[None, :] ** 2 + v[:, None] ** 2 - 0.5)
    return f.reshape(-1).clamp(float(lo), float(hi)).contiguous()


def _measured(sig, g, snr=40.0):
    """Complex voxels [n][T][2] of the complex signals: M0, a random phase, noise."""
    n, T = sig.shape
    sig = sig * torch.polar(_uniform(g, n, 0.6, 1.0), _uniform(g, n, 0.0, 2 * PI))[:, None].to(sig.dtype)
    sigma = torch.linalg.vector_norm(sig, dim=1, keepdim=True) / math.sqrt(T) / snr / math.sqrt(2.0)
    noise = torch.randn((n, T, 2), generator=g, device="cuda", dtype=torch.float32)
    return (torch.view_as_real(sig).float() + sigma.float()[:, :, None] * noise).contiguous()


# ---------------------------------------------------------------------------
# the signal models in torch (float32 for inputs, float64 for exact values)
# ---------------------------------------------------------------------------

def _f64(x):
    return (x if isinstance(x, torch.Tensor) else torch.tensor(np.asarray(x), device="cuda")).double()


def _cis(angle):
    return torch.complex(torch.cos(angle), torch.sin(angle))


class _Fisp:
    """Zero-phase FISP: F+ and F- purely imaginary, Z real, states [3][w][n];
    the flip angle is alpha_t * B1."""

    def __init__(self, T1, T2, B1, w):
        self.T1, self.T2, self.B1, self.w = T1, T2, B1, w

    def start(self):
        x = self.T1.new_zeros((3, self.w, self.T1.numel()))
        x[2, 0] = 1
        return x

    def step(self, x, alpha, phi, TR, TE):
        """(state after the step, Im of the readout)."""
        a = alpha * self.B1
        C, S = torch.cos(a), torch.sin(a)
        p, m, z = x[0], x[1], x[2]
        u, v = (p + m) / 2, (p - m) / 2
        q = v * C - S * z
        np_, nm, nz = u + q, u - q, S * v + C * z
        f = torch.exp(-TE / self.T2) * np_[0]
        E1, E2 = torch.exp(-TR / self.T1), torch.exp(-TR / self.T2)
        nz = torch.cat([(nz[0] * E1 + (1 - E1))[None], nz[1:] * E1])
        return torch.stack([torch.cat([-nm[1:2], np_[:-1]]) * E2,
                            torch.cat([nm[1:], torch.zeros_like(nm[:1])]) * E2, nz]), f


class _Ssfp:
    """bSSFP with off-resonance: complex states [3][w][n], 180 deg inversion
    with TI = 40 ms; readout F+[0] after the decay and precession over TE."""

    def __init__(self, T1, T2, B0, B1, w):
        self.T1, self.T2, self.B0, self.B1, self.w = T1, T2, B0, B1, w

    def start(self):
        dt = torch.complex128 if self.T1.dtype == torch.float64 else torch.complex64
        x = torch.zeros((3, self.w, self.T1.numel()), dtype=dt, device=self.T1.device)
        z0 = (1 - 2 * torch.exp(-40.0 / self.T1)).to(dt)
        return torch.cat([x[:2], torch.cat([z0[None], x[2, 1:]])[None]])

    def step(self, x, alpha, phi, TR, TE):
        a = alpha * self.B1
        C, S = torch.cos(a), torch.sin(a)
        z = complex(math.cos(phi), math.sin(phi))
        zc = z.conjugate()
        p, m, l = zc * x[0], z * x[1], x[2]          # the pulse along x in the frame of its phase
        u, v = (p + m) / 2, (p - m) / 2
        q = v * C - 1j * S * l
        np_, nm, nz = z * (u + q), zc * (u - q), -1j * S * v + C * l
        s = torch.exp(-TE / self.T2) * _cis(2 * PI * self.B0 * (TE / 1000.0)) * np_[0]
        rot = torch.exp(-TR / self.T2) * _cis(2 * PI * self.B0 * (TR / 1000.0))
        E1 = torch.exp(-TR / self.T1)
        np_, nm = np_ * rot, nm * rot.conj()
        nz = torch.cat([(nz[0] * E1 + (1 - E1))[None], nz[1:] * E1])
        return torch.stack([torch.cat([nm[1:2].conj(), np_[:-1]]),
                            torch.cat([nm[1:], torch.zeros_like(nm[:1])]), nz]), s


def _schedule_steps(echo, h):
    """(alpha, phi, TR, TE) per step in rad and ms."""
    h = h.astype(np.float64)
    if echo == "epg_fisp":
        return list(zip(*h.tolist()))
    return list(zip((h[0] * PI / 3).tolist(), (h[1] * PI / 180).tolist(), (h[2] + 16.0).tolist(),
                    (h[3] + 3.5).tolist()))


def _signal(model, steps):
    """[n][T] of the model."""
    x, out = model.start(), []
    for s in steps:
        x, f = model.step(x, *s)
        out.append(f)
    return torch.stack(out, 1)


def _fisp_atoms(p, h, w, dtype=torch.float32):
    p = p.to(dtype)
    return _signal(_Fisp(p[:, 0], p[:, 1], p[:, 3], w), _schedule_steps("epg_fisp", h))


def _ssfp_atoms(p, h, w, dtype=torch.float32):
    """Unit-norm atoms."""
    p = p.to(dtype)
    s = _signal(_Ssfp(p[:, 0], p[:, 1], p[:, 2], p[:, 3], w), _schedule_steps("epg_ssfp", h))
    return s / torch.linalg.vector_norm(s, dim=1, keepdim=True)


def _roa_atoms(p, h, n_iso):
    """Unit-norm mean of n_iso isochromats, 64 bits: the pulse, relaxation
    over TR, precession by half the angle, readout, the other half."""
    p = p.double()
    T1, T2, B0 = p[:, 0], p[:, 1], p[:, 2]
    d = (torch.arange(n_iso, device=p.device, dtype=torch.float64) * (PI / n_iso))[:, None]
    xy = torch.zeros((n_iso, p.shape[0]), dtype=torch.complex128, device=p.device)
    z = torch.full((n_iso, p.shape[0]), -1.0, dtype=torch.float64, device=p.device)
    out = []
    for a, phi, TR, _ in _schedule_steps("roa_ssfp", h):
        ca, sa = math.cos(a), math.sin(a)
        x, y = xy.real, ca * xy.imag + sa * z
        E1, E2 = torch.exp(-TR / T1), torch.exp(-TR / T2)
        z = E1 * (ca * z - sa * xy.imag) + (1 - E1)
        rot = _cis(-(PI * B0 * (TR / 1000.0) + d))
        xy = torch.complex(x, y) * (complex(math.cos(2 * phi), -math.sin(2 * phi)) * E2) * rot
        out.append(xy.mean(0))
        xy = xy * rot
    s = torch.stack(out, 1)
    return s / torch.linalg.vector_norm(s, dim=1, keepdim=True)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def _real(s):
    """Complex rows [n][T][2] of purely imaginary signals."""
    return torch.stack([torch.zeros_like(s), s], -1).contiguous()


def _precision(case):
    return {"fp32": snap.PREC_FP32, "bf16": snap.PREC_BF16, "fp16": snap.PREC_FP16}[case["precision"]]


def _voxels(case, g, seed, h, b1, w):
    """FISP voxels with a B1 field: (image, B1 map, T1, T2)."""
    nx = case["nx"]
    b1map = _b1_field(nx, b1[0], b1[-1])
    T1, T2 = _tissue(g, nx * nx, seed)
    sig = _signal(_Fisp(T1, T2, b1map, w), _schedule_steps("epg_fisp", h))
    return _measured(torch.complex(torch.zeros_like(sig), sig), g), b1map, T1, T2


def prepare(case, seed):
    k, g, T = case["kind"], _generator(seed), case["T"]
    s = dict(case=case, T=T, w=case.get("w", 0))
    new = lambda *shape, dt=torch.float32: torch.empty(shape, device="cuda", dtype=dt)  # noqa: E731
    if k in ("map", "dict_fisp", "match_b1", "refine_fisp", "svd"):
        s["h"] = _fisp_schedule(T, seed)
    elif k == "adjoint" and case["echo"] == "epg_fisp" or k == "crb":
        s["h"] = _fisp_schedule(T, seed, inversion=k == "adjoint")
    else:
        s["h"] = _ssfp_schedule(T, seed)
    if "nb1" in case or "nb0" in case or "grid" in case:
        p, s["natoms"], b1 = _grid(case)
        s["p"], s["N"] = torch.from_numpy(p).cuda(), p.shape[0]
    h, N = s["h"], s.get("N")
    if k == "map":
        n = case["nx"] ** 2
        T1 = _uniform(g, n, 150.0, 100.0 * case["nt1"])
        T2 = torch.minimum(_uniform(g, n, 20.0, 20.0 + 10.0 * case["nt2"]), 0.8 * T1)
        sig = _signal(_Fisp(T1, T2, torch.ones_like(T1), s["w"]), _schedule_steps("epg_fisp", h))
        s.update(img=_measured(torch.complex(torch.zeros_like(sig), sig), g, snr=30.0), nvox=n)
        s.update(atoms=new(N, T, 2), maps=new(n, 5), index=new(n, dt=torch.int64))
    elif k == "dict_fisp":
        if case["form"] == "operand":
            s.update(atoms=new(N, T), norms=new(N), packed=new(N, snap.api.packed_pitch(T), dt=torch.bfloat16))
        else:
            s.update(atoms=new(N, T, 2), norms=new(N))
    elif k in ("dict_ssfp", "dict_roa"):
        s.update(atoms=new(N, T, 2))
    elif k == "match_b1":
        s["img"], s["b1map"], _, _ = _voxels(case, g, seed, h, b1, s["w"])
        n = s["nvox"] = case["nx"] ** 2
        rows = _fisp_atoms(s["p"], h, s["w"])
        norms = torch.linalg.vector_norm(rows, dim=1)
        if case["precision"] == "fp32":
            s["atoms"] = _real(rows / norms[:, None])
        else:
            dt = torch.bfloat16 if case["precision"] == "bf16" else torch.float16
            s.update(atoms=rows.contiguous(), norms=norms)
            s["packed"] = torch.zeros((N, snap.api.packed_pitch(T)), device="cuda", dtype=dt)
            s["packed"][:, :T] = (rows / norms[:, None]).to(dt)
        s.update(maps=new(n, 5), index=new(n, dt=torch.int64))
    elif k == "match_all":
        n = s["nvox"] = case["nx"] ** 2
        s["atoms"] = torch.view_as_real(_ssfp_atoms(s["p"], h, s["w"])).contiguous()
        T1, T2 = _tissue(g, n, seed)
        span = 12.0 * case["nb0"] / 2
        sig = _signal(_Ssfp(T1, T2, _uniform(g, n, -span, span), _uniform(g, n, 0.88, 0.92 + 0.1 * (case["nb1"] - 1)),
                            s["w"]), _schedule_steps("epg_ssfp", h))
        s.update(img=_measured(sig, g), maps=new(n, 5), index=new(n, dt=torch.int64))
    elif k == "refine_fisp":
        s["img"], s["b1map"], T1, T2 = _voxels(case, g, seed, h, b1, s["w"])
        n = s["nvox"] = case["nx"] ** 2
        s["atoms"] = _fisp_atoms(s["p"], h, s["w"]).contiguous()
        # the matched atom: the nearest (T1, T2) of the grid in the nearest B1 block
        block = s["p"][: s["natoms"]]
        ref = torch.log(block[:, :2])
        near = torch.cat([torch.cdist(torch.log(torch.stack([a, b], 1)), ref).argmin(1)
                          for a, b in zip(T1.split(8192), T2.split(8192))])
        bins = (s["b1map"][:, None] - torch.from_numpy(b1).cuda()[None, :]).abs().argmin(1)
        s["index"] = (near + bins * s["natoms"]).contiguous()
        s["matched"] = torch.cat([s["p"][s["index"]], torch.ones((n, 1), device="cuda")], 1).contiguous()
        s.update(maps=s["matched"].clone(), m0=new(n))
    elif k == "refine_ssfp":
        n = s["nvox"] = case["nx"] ** 2
        T1, T2 = _tissue(g, n, seed)
        B0, B1 = _uniform(g, n, -80.0, 80.0), _uniform(g, n, 0.82, 1.18)
        sig = _signal(_Ssfp(T1, T2, B0, B1, s["w"]), _schedule_steps("epg_ssfp", h))
        s["img"] = _measured(sig, g)
        s["b1map"] = B1 if case["b1map"] else None
        off = [v * _uniform(g, n, 0.98, 1.02) for v in (T1, T2)] + [B0 + _uniform(g, n, -1.5, 1.5),
                                                                  B1 * _uniform(g, n, 0.98, 1.02)]
        s["matched"] = torch.stack(off + [torch.ones_like(T1)], 1).contiguous()
        s.update(maps=s["matched"].clone(), m0=new(n))
    elif k in ("adjoint", "crb"):
        n, ssfp = case["n"], case.get("echo") == "epg_ssfp"
        T1 = torch.exp(_uniform(g, n, math.log(400.0), math.log(4000.0)))
        T2 = torch.exp(_uniform(g, n, math.log(30.0), math.log(300.0)))
        B0 = _uniform(g, n, -80.0, 80.0) if ssfp else torch.zeros_like(T1)
        s["p"] = torch.stack([T1, T2, B0, _uniform(g, n, 0.8, 1.2)], 1).contiguous()
        if k == "crb":
            s.update(loss=new(n), ga=new(T), signals=new(n, 3, T))
        else:
            s["g"] = 0.1 * torch.randn((n, T, 2), generator=g, device="cuda", dtype=torch.float32)
            s.update(sig=new(n, T, 2), gp=new(n, 4 if ssfp else 3), ga=new(T))
    elif k == "svd":
        s["atoms"] = _fisp_atoms(s["p"], h, s["w"])
        s["atoms"] = _real(s["atoms"] / torch.linalg.vector_norm(s["atoms"], dim=1, keepdim=True))
    return s


def run(s):
    c, k, T, h, w = s["case"], s["case"]["kind"], s["T"], s["h"], s["w"]
    if k == "map":
        snap.MRF_dict(s["atoms"], s["p"], h, T, T, s["N"], s["natoms"], 4, w, "epg_fisp")
        snap.normalize(s["atoms"], T, s["N"])
        snap.MRF_match(s["maps"], s["img"], s["atoms"], s["p"], T, T, s["N"], s["natoms"], s["nvox"],
                       d_index=s["index"])
        return {"atoms": s["atoms"], "maps": s["maps"], "index": s["index"]}
    if k == "dict_fisp":
        if c["form"] == "operand":
            snap.MRF_dict(s["atoms"], s["p"], h, T, T, s["N"], s["natoms"], 4, w, "epg_fisp",
                          flags=snap.DICT_ALL_B1_BLOCKS | snap.DICT_NORMALIZE_OPERAND | snap.DICT_IMAG_ROWS,
                          d_norms=s["norms"], d_packed=s["packed"], packed_precision=snap.PREC_BF16)
            return {"rows": s["atoms"], "norms": s["norms"], "operand": s["packed"]}
        snap.MRF_dict(s["atoms"], s["p"], h, T, T, s["N"], s["natoms"], 4, w, "epg_fisp",
                      flags=snap.DICT_ALL_B1_BLOCKS | (snap.DICT_NORMALIZE if c["form"] == "unit" else 0),
                      d_norms=s["norms"])
        return {"atoms": s["atoms"], "norms": s["norms"]}
    if k == "dict_ssfp":
        snap.MRF_dict(s["atoms"], s["p"], h, T, T, s["N"], s["natoms"], 4, w, "epg_ssfp")
        return s["atoms"]
    if k == "dict_roa":
        snap.MRF_dict(s["atoms"], s["p"], h, T, T, s["N"], s["natoms"], 4, 101, "roa_ssfp", n_iso=c["n_iso"],
                      flags=snap.DICT_ALL_B1_BLOCKS)
        return s["atoms"]
    if k == "match_b1":
        flags = snap.MATCH_ASSUME_UNIFORM_B1 | snap.MATCH_IMAG_ATOMS
        more = {}
        if c["precision"] != "fp32":
            flags |= snap.MATCH_IMAG_ROWS
            more = dict(packed_atoms=s["packed"], atom_norms=s["norms"])
        snap.MRF_match(s["maps"], s["img"], s["atoms"], s["p"], T, T, s["N"], s["natoms"], s["nvox"],
                       in_b1map=s["b1map"], precision=_precision(c), flags=flags, d_index=s["index"], **more)
        return {"maps": s["maps"], "index": s["index"]}
    if k == "match_all":
        snap.MRF_match(s["maps"], s["img"], s["atoms"], s["p"], T, T, s["N"], s["natoms"], s["nvox"],
                       precision=_precision(c), d_index=s["index"])
        return {"maps": s["maps"], "index": s["index"]}
    if k == "refine_fisp":
        s["maps"].copy_(s["matched"])
        snap.refine_start(s["maps"], s["img"], s["atoms"], s["p"], s["index"], T, s["N"], s["natoms"], s["nvox"],
                          d_b1map=s["b1map"], imag_atoms=True, imag_rows=True)
        snap.refine_gn(s["maps"], s["img"], h, T, T, s["nvox"], w, "epg_fisp", iterations=3, tol=1e-3,
                       d_b1map=s["b1map"], d_m0=s["m0"])
        return {"maps": s["maps"], "m0": s["m0"]}
    if k == "refine_ssfp":
        s["maps"].copy_(s["matched"])
        snap.refine_gn(s["maps"], s["img"], h, T, T, s["nvox"], w, "epg_ssfp", iterations=3, tol=1e-3,
                       d_b1map=s["b1map"], d_m0=s["m0"])
        return {"maps": s["maps"], "m0": s["m0"]}
    if k == "adjoint":
        snap.epg_adjoint(s["p"], h, T, T, c["n"], s["g"], s["gp"], 4, w, c["echo"], d_signal=s["sig"],
                         d_grad_alpha=s["ga"])
        return {"signal": s["sig"], "grad_params": s["gp"], "grad_alpha": s["ga"]}
    if k == "crb":
        snap.crb_gradient(s["p"], h, T, T, c["n"], s["loss"], s["ga"], 4, w, "epg_fisp", d_signals=s["signals"])
        return {"loss": s["loss"], "grad_alpha": s["ga"], "signals": s["signals"]}
    r = snap.svd_compress(s["atoms"], T, s["N"], s["natoms"], sfrac=0.99999, imag_atoms=True)
    return {"basis": r.basis, "coeffs": r.coeffs, "rank": r.rank, "sv": r.sv}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; operations of the real
    recursion (16 per state and step: eight multiply-adds), the complex one
    (48: sixteen multiply-adds of the pulse, eight of the precession), an
    isochromat (32), and the products of the scores."""
    k, T, w = case["kind"], case["T"], case.get("w", 0)
    N = natoms = nb1 = 0
    if "nb1" in case or "nb0" in case or "grid" in case:
        p, natoms, b1 = _grid(case)
        N, nb1 = p.shape[0], len(b1)
    nvox = case.get("nx", 0) ** 2
    if k == "map":
        return {"bytes": 8 * T * (N + nvox) + 28 * nvox, "flops": 16.0 * N * T * w + 8.0 * N * nvox * T}
    if k == "dict_fisp":
        row = 4 * T + 2 * T if case["form"] == "operand" else 8 * T
        return {"bytes": N * (row + 20.0), "flops": 16.0 * N * T * w}
    if k == "dict_ssfp":
        return {"bytes": N * (8.0 * T + 16), "flops": 48.0 * N * T * w}
    if k == "dict_roa":
        return {"bytes": N * (8.0 * T + 16), "flops": 32.0 * N * T * case["n_iso"]}
    if k == "match_b1":
        atom = 4 * T if case["precision"] == "fp32" else 2 * T
        return {"bytes": N * float(atom) + nvox * (8.0 * T + 32), "flops": 4.0 * natoms * nvox * T}
    if k == "match_all":
        return {"bytes": 8.0 * T * (N + nvox) + 28 * nvox, "flops": 8.0 * N * nvox * T}
    if k == "refine_fisp":
        return {"bytes": nvox * (8.0 * T + 60), "flops": 60.0 * nvox * T * w}
    if k == "refine_ssfp":
        nt = 3 if case["b1map"] else 4
        return {"bytes": nvox * (8.0 * T + 60), "flops": 48.0 * (1 + nt) * nvox * T * w}
    if k == "adjoint":
        ops = (16.0 if case["echo"] == "epg_fisp" else 48.0) * 4  # forward, recomputation, transpose, products
        return {"bytes": case["n"] * (16.0 * T + 40), "flops": ops * case["n"] * T * w}
    if k == "crb":
        return {"bytes": case["n"] * 12.0 * T + 20 * T, "flops": 48.0 * 4 * case["n"] * T * w}
    return {"bytes": 8.0 * N * T, "flops": 2.0 * 72 * 8 * N * T}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------

def _exact_match(x, d, p, bins, nbins, natoms, norms=None):
    """First argmax of |<d, x>| within each voxel's block; d complex or, for
    imaginary rows, real."""
    n = x.shape[0]
    maps, index = torch.zeros((n, 5), dtype=torch.float64, device=x.device), torch.zeros(n, dtype=torch.int64,
                                                                                     device=x.device)
    for b in range(nbins):
        who = (bins == b).nonzero()[:, 0] if bins is not None else torch.arange(n, device=x.device)
        D = d[b * natoms:(b + 1) * natoms]
        D = D.conj().resolve_conj().to(torch.complex128) if D.is_complex() else D.double()
        for v in who.split(2048):
            if not D.is_complex():
                sc = torch.hypot(x[v].real @ D.T, x[v].imag @ D.T)
            else:
                sc = (x[v] @ D.T).abs()
            if norms is not None:
                sc = sc / norms[b * natoms:(b + 1) * natoms]
            best, at = sc.max(1)
            index[v] = at + b * natoms
            maps[v, :4], maps[v, 4] = p[index[v]].double(), best
    return {"maps": maps, "index": index}


def _jacobian(kind, th, h, w, nt):
    """Signal [n][T] and its tangents by the first nt columns of th, 64 bits,
    by forward-mode differentiation of one step at a time."""
    jvp = torch.func.jvp
    cols = th.unbind(1)
    make = (lambda c: _Fisp(c[0], c[1], c[2], w)) if kind == "epg_fisp" else (
        lambda c: _Ssfp(c[0], c[1], c[2], c[3], w))
    m = make(cols)
    one, nil = torch.ones_like(cols[0]), torch.zeros_like(cols[0])
    unit = [tuple(one if i == j else nil for i in range(len(cols))) for j in range(nt)]
    x = m.start()
    tx = [jvp(lambda *c: make(c).start() + 0 * c[0], cols, u)[1] for u in unit]
    f, J = [], [[] for _ in unit]
    for st in _schedule_steps(kind, h):
        for j, u in enumerate(unit):
            (x1, f1), (tx[j], df) = jvp(lambda x_, *c: make(c).step(x_, *st), (x,) + tuple(cols), (tx[j],) + u)
            J[j].append(df)
        x = x1
        f.append(f1)
    return torch.stack(f, 1), [torch.stack(q, 1) for q in J]


def _exact_refine(kind, maps, img, h, w, nt, b1, its=3, tol=1e-3):
    """Gauss-Newton with the complex scale eliminated (variable projection),
    steps within 20 %, at most `its` of them, until a step is within tol."""
    maps = maps.double().clone()
    x = torch.view_as_complex(img.double().contiguous())
    n = maps.shape[0]
    m0 = torch.zeros(n, dtype=torch.float64, device=maps.device)
    if b1 is not None:
        maps[:, 3] = b1.double()
    cols = [0, 1, 3] if kind == "epg_fisp" else [0, 1, 2, 3]
    left = torch.arange(n, device=maps.device)
    for it in range(its):
        moving = []
        for v in left.split(32768):
            th = maps[v][:, cols]
            s, J = _jacobian(kind, th, h, w, nt)
            J = torch.stack(J, 2)
            if kind == "epg_fisp":
                s, J = 1j * s, 1j * J
            xv = x[v]
            ss = s.abs().square().sum(1)
            P = (s.conj() * xv).sum(1)
            G = (s.conj()[:, :, None] * J).sum(1)
            H = torch.einsum("ntj,ntk->njk", J.conj(), J).real
            Q = torch.einsum("ntj,nt->nj", J.conj(), xv)
            rho = P / ss
            A = rho.abs().square()[:, None, None] * (H - (G.conj()[:, :, None] * G[:, None, :]).real / ss[:, None, None])
            b = (rho.conj()[:, None] * (Q - G.conj() * rho[:, None])).real
            dl = torch.linalg.solve(A, b)
            lim = 0.2 * torch.stack([th[:, 0], th[:, 1], torch.full_like(th[:, 0], 50.0), th[:, -1]], 1)[:, :nt]
            dl = torch.maximum(torch.minimum(dl, lim), -lim)
            new = th[:, :nt] + dl
            new[:, 1] = new[:, 1].clamp_min(1e-3)
            new[:, 0] = torch.maximum(new[:, 0], new[:, 1] * (1 + 1e-4))
            dl = new - th[:, :nt]
            maps[v[:, None], torch.tensor(cols[:nt], device=v.device)] = new
            big = (dl[:, :2].abs() > tol * th[:, :2]).any(1)
            if nt > 2:
                big |= dl[:, 2].abs() > tol * 100
            if nt > 3:
                big |= dl[:, 3].abs() > tol * th[:, 3]
            Pn = P + (Q * dl).sum(1)
            sn = ss + 2 * (G.real * dl).sum(1) + torch.einsum("nj,njk,nk->n", dl, H, dl)
            maps[v, 4] = Pn.abs() / sn.sqrt()
            m0[v] = Pn.abs() / sn
            moving.append(v[big])
        left = torch.cat(moving)
        if not left.numel():
            break
    return {"maps": maps, "m0": m0}


def _exact_adjoint(s, case):
    """Reverse mode, one step at a time over the stored states."""
    ssfp = case["echo"] == "epg_ssfp"
    p = s["p"].double()
    par = [p[:, j].clone().requires_grad_() for j in ((0, 1, 2, 3) if ssfp else (0, 1, 3))]
    model = _Ssfp(*par, s["w"]) if ssfp else _Fisp(*par, s["w"])
    steps = _schedule_steps(case["echo"], s["h"])
    g = torch.view_as_complex(s["g"].double().contiguous())
    dot = lambda a, b: (a.conj() * b).real.sum() if a.is_complex() else (a * b).sum()  # noqa: E731
    states, sig = [], []
    with torch.no_grad():
        x = model.start()
        for st in steps:
            states.append(x)
            x, f = model.step(x, *st)
            sig.append(f)
    lam = torch.zeros_like(x)
    gp, ga = [torch.zeros_like(v) for v in par], torch.zeros(len(steps), dtype=torch.float64, device=p.device)
    scale = PI / 3 if ssfp else 1.0
    for t in reversed(range(len(steps))):
        x0 = states.pop().detach().requires_grad_()
        a = torch.tensor(steps[t][0], dtype=torch.float64, device=p.device, requires_grad=True)
        x1, f = model.step(x0, a, *steps[t][1:])
        L = dot(lam, x1) + (dot(g[:, t], f) if ssfp else (g[:, t].imag * f).sum())
        got = torch.autograd.grad(L, [x0, a] + par, allow_unused=True)
        lam, ga[t] = got[0], got[1] * scale
        gp = [u if v is None else u + v for u, v in zip(gp, got[2:])]
    x0 = model.start()
    if x0.requires_grad:
        got = torch.autograd.grad(dot(lam, x0), par, allow_unused=True)
        gp = [u if v is None else u + v for u, v in zip(gp, got)]
    sig = torch.stack(sig, 1).detach()
    sig = torch.view_as_real(sig) if ssfp else _real(sig)
    return {"signal": sig, "grad_params": torch.stack(gp, 1).detach(), "grad_alpha": ga}


def _exact_crb(s):
    """Forward mode for f, df/dT1, df/dT2 and reverse mode for the flip
    angles.  The chain over all steps is kept: a few tissues only."""
    p, h = s["p"].double(), s["h"]
    T1, T2, B1 = p[:, 0], p[:, 1], p[:, 3]
    al = torch.tensor(h[0].astype(np.float64), device=p.device, requires_grad=True)
    st = _schedule_steps("epg_fisp", h)
    n, w = p.shape[0], s["w"]
    x = torch.zeros((3, 3, w, n), dtype=torch.float64, device=p.device)  # [signal, dT1, dT2][p, m, z]
    x[0, 2, 0] = 1
    out = []
    e0 = torch.zeros((w, 1), dtype=torch.float64, device=p.device)
    e0[0] = 1
    zero = torch.zeros((3, 1, n), dtype=torch.float64, device=p.device)
    for t, (_, _, TR, TE) in enumerate(st):
        a = al[t] * B1
        C, S = torch.cos(a), torch.sin(a)
        u, v = (x[:, 0] + x[:, 1]) / 2, (x[:, 0] - x[:, 1]) / 2
        q = v * C - S * x[:, 2]
        pp, m, z = u + q, u - q, S * v + C * x[:, 2]
        Ea = torch.exp(-TE / T2)
        out.append(torch.stack([Ea * pp[0, 0], Ea * pp[1, 0], Ea * pp[2, 0] + Ea * TE / T2 ** 2 * pp[0, 0]]))
        pp, m = torch.cat([-m[:, 1:2], pp[:, :-1]], 1), torch.cat([m[:, 1:], zero], 1)
        E1, E2 = torch.exp(-TR / T1), torch.exp(-TR / T2)
        d1, d2 = E1 * TR / T1 ** 2, E2 * TR / T2 ** 2
        one = lambda c0, c1, c2: torch.stack([c0, c1, c2])  # noqa: E731
        x = torch.stack([one(E2 * pp[0], E2 * pp[1], E2 * pp[2] + d2 * pp[0]),
                         one(E2 * m[0], E2 * m[1], E2 * m[2] + d2 * m[0]),
                         one(E1 * z[0] + (1 - E1) * e0, E1 * z[1] + d1 * z[0] - d1 * e0, E1 * z[2])], 1)
    f = torch.stack(out, 2).permute(1, 0, 2)  # [n][3][T]: f, f1, f2
    V = torch.stack([f[:, 1], f[:, 2], f[:, 0]], 2)
    Mi = torch.linalg.inv(V.transpose(1, 2) @ V)
    loss = Mi[:, 0, 0] / T1 ** 2 + Mi[:, 1, 1] / T2 ** 2
    return {"loss": loss.detach(), "grad_alpha": torch.autograd.grad(loss.sum(), al)[0], "signals": f.detach()}


def exact(case, seed):
    s, k = prepare(case, seed), case["kind"]
    if k == "map":
        a = _fisp_atoms(s["p"], s["h"], s["w"], torch.float64)
        a = a / torch.linalg.vector_norm(a, dim=1, keepdim=True)
        x = torch.view_as_complex(s["img"].double())
        return {"atoms": _real(a), **_exact_match(x, a, s["p"], None, 1, s["N"])}
    if k == "dict_fisp":
        a = torch.cat([_fisp_atoms(q, s["h"], s["w"], torch.float64) for q in s["p"].split(65536)])
        n = torch.linalg.vector_norm(a, dim=1)
        if case["form"] == "operand":
            op = torch.zeros(s["packed"].shape, dtype=torch.float64, device="cuda")
            op[:, : s["T"]] = a / n[:, None]
            return {"rows": a, "norms": n, "operand": op}
        return {"atoms": _real(a / n[:, None] if case["form"] == "unit" else a), "norms": n}
    if k == "dict_ssfp":
        return torch.cat([torch.view_as_real(_ssfp_atoms(q, s["h"], s["w"], torch.float64))
                          for q in s["p"].split(32768)])
    if k == "dict_roa":
        return torch.cat([torch.view_as_real(_roa_atoms(q, s["h"], case["n_iso"])) for q in s["p"].split(16384)])
    if k in ("match_b1", "match_all"):
        x = torch.view_as_complex(s["img"].double())
        if k == "match_all":
            return _exact_match(x, torch.view_as_complex(s["atoms"]), s["p"], None, 1, s["N"])
        d = s["atoms"][..., 1] if case["precision"] == "fp32" else s["atoms"]
        norms = None if case["precision"] == "fp32" else torch.linalg.vector_norm(d.double(), dim=1)
        b1 = s["p"][:: s["natoms"], 3]
        bins = (s["b1map"][:, None] - b1[None, :]).abs().argmin(1)
        return _exact_match(x, d, s["p"], bins, len(b1), s["natoms"], norms)
    if k == "refine_fisp":
        # (the same fit, from the match itself)
        return _exact_refine("epg_fisp", s["matched"], s["img"], s["h"], s["w"], 2, s["b1map"])
    if k == "refine_ssfp":
        return _exact_refine("epg_ssfp", s["matched"], s["img"], s["h"], s["w"], 3 if case["b1map"] else 4,
                             s["b1map"])
    if k == "adjoint":
        return _exact_adjoint(s, case)
    if k == "crb":
        return _exact_crb(s)
    d = s["atoms"][..., 1].double().reshape(-1, s["natoms"], s["T"])
    sv = torch.linalg.eigvalsh(d.transpose(1, 2) @ d).flip(1).clamp_min(0).sqrt()[:, :64]
    return {"basis": None, "coeffs": None, "rank": None, "sv": sv}
