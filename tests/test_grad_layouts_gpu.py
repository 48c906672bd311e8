"""The adjoint's and the CRB sweeps' layouts: one atom per warp for few atoms,
several for many, state counts at the edges of each (2P states per lane, 8 /
16 / 32 lanes), segments of any length.

Adjoint: dL/dT1 and dL/dT2 against the forward-mode tangents (epg_jvp, another
kernel) contracted with the same dL/ds, the signal against the dictionary, the
schedule gradient of one layout against the other's.  Both sides are FP32
recursions of T = 150 steps, about 1e-6 of the terms' sum off each: 1e-4 of it
is allowed (signal: 1e-5 of the peak).
CRB: signals and losses do not depend on the layout or the segments (bit for
bit), the gradients' sums over lanes and tissues only by their order (1e-5 of
the largest)."""
import numpy as np
import pytest

from cases import mrf_schedule
from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu
T = 150


def _params(n, seed):
    rng = np.random.default_rng(seed)
    t1 = np.exp(rng.uniform(np.log(300), np.log(3000), n))
    t2 = np.minimum(np.exp(rng.uniform(np.log(20), np.log(300), n)), 0.8 * t1)
    return np.stack([t1, t2, np.zeros(n), rng.uniform(0.8, 1.2, n)], 1).astype(np.float32)


def _adjoint(snap, torch, p, g, h, w, echo):
    n = p.shape[0]
    gp, ga = torch.empty((n, 3), device="cuda"), torch.empty(T, device="cuda")
    per, sig = torch.empty((n, T), device="cuda"), torch.empty((n, T, 2), device="cuda")
    snap.epg_adjoint(p, h, T, T, n, g, gp, 4, w, echo, d_signal=sig, d_grad_alpha=ga, d_grad_alpha_atoms=per)
    return gp.double(), ga.double(), per.double(), sig


@pytest.mark.parametrize("echo", ["epg_fisp", "epg_sr"])
@pytest.mark.parametrize("w", [1, 2, 15, 16, 17, 31, 32, 33, 50, 63, 64, 65, 130, 193, 256])
def test_adjoint_layouts(snap, w, echo):
    torch = torch_cuda()
    h = mrf_schedule(T, seed=w)
    few, many = 5, 2500
    p = torch.from_numpy(np.tile(_params(few, w), (many // few, 1))).cuda()
    g = torch.from_numpy(np.random.default_rng(w).standard_normal((few, T, 2)).astype(np.float32)).cuda()
    g = g.repeat(many // few, 1, 1).contiguous()
    a = _adjoint(snap, torch, p[:few].contiguous(), g[:few].contiguous(), h, w, echo)
    b = _adjoint(snap, torch, p, g, h, w, echo)
    J = torch.empty((few, 3, T), device="cuda")
    snap.epg_jvp(p[:few].contiguous(), h, T, T, few, J, 4, w, echo)
    d = torch.empty((few, T, 2), device="cuda")
    snap.MRF_dict(d, p[:few].contiguous(), h, T, T, few, 1, 4, w, echo, flags=snap.DICT_ALL_B1_BLOCKS)
    J, gs = J.double(), g[:few, :, 1].double()
    for gp, _, per, sig in (a, (b[0][:few], b[1], b[2][:few], b[3][:few])):
        assert (sig - d).abs().max() <= 1e-5 * d.abs().max()
        for k in (0, 1):
            terms = gs * J[:, 1 + k]
            assert ((gp[:, k] - terms.sum(1)).abs() <= 1e-4 * terms.abs().sum(1)).all(), (w, k)
        assert (per - a[2]).abs().max() <= 1e-4 * a[2].abs().max()
        assert (gp[:, 2] - a[0][:, 2]).abs().max() <= 1e-4 * a[0][:, 2].abs().max()
    # the last atoms of a partly filled warp
    assert torch.equal(b[0][:few], b[0][-few:])
    assert (b[1] - b[2].sum(0)).abs().max() <= 1e-5 * b[2].abs().sum(0).max()


@pytest.mark.parametrize("w", [1, 2, 32, 33, 50, 100, 256])
def test_crb_layouts_and_segments(snap, w):
    torch = torch_cuda()
    h = mrf_schedule(T, seed=w + 7, inversion=False)

    def crb(p, every):
        n = p.shape[0]
        loss, ga, sig = (torch.empty(s, device="cuda") for s in ((n,), (T,), (n, 3, T)))
        snap.crb_gradient(p, h, T, T, n, loss, ga, 4, w, "epg_fisp", d_signals=sig, checkpoint_every=every)
        return loss, ga.double(), sig

    p = torch.from_numpy(_params(3, w)).cuda()
    ref = crb(p, 0)
    assert torch.isfinite(ref[2]).all()
    for every in (1, 7, T, 3 * T):
        loss, ga, sig = crb(p, every)
        assert torch.equal(sig, ref[2])
        np.testing.assert_array_equal(loss.cpu().numpy(), ref[0].cpu().numpy())
        np.testing.assert_array_equal(ga.cpu().numpy(), ref[1].cpu().numpy())
    loss, ga, sig = crb(p.repeat(300, 1).contiguous(), 0)
    assert torch.equal(sig[:3], ref[2]) and torch.equal(sig[-3:], ref[2])
    np.testing.assert_array_equal(loss[:3].cpu().numpy(), ref[0].cpu().numpy())
    if torch.isfinite(ref[1]).all():
        assert (ga / 300 - ref[1]).abs().max() <= 1e-5 * ref[1].abs().max()


@pytest.mark.parametrize("n", [3, 2500])
@pytest.mark.parametrize("w", [7, 20, 50])
def test_adjoint_does_not_depend_on_the_segments(snap, n, w):
    """A schedule long enough that the checkpoint interval changes the sweep's
    segments (16 steps, or more where that would keep too many checkpoints):
    the same bits from each."""
    torch = torch_cuda()
    long = 4000 if n == 3 else 1600
    h = mrf_schedule(long, seed=w)
    p = torch.from_numpy(_params(n, w)).cuda()
    g = torch.randn((n, long, 2), device="cuda", generator=torch.Generator("cuda").manual_seed(w))
    out = []
    for every in (0, 1, 40, long):
        gp, ga = torch.empty((n, 3), device="cuda"), torch.empty(long, device="cuda")
        sig, per = torch.empty((n, long, 2), device="cuda"), torch.empty((n, long), device="cuda")
        snap.epg_adjoint(p, h, long, long, n, g, gp, 4, w, "epg_fisp", d_signal=sig, d_grad_alpha=ga,
                         d_grad_alpha_atoms=per, checkpoint_every=every)
        out.append((gp, ga, sig, per))
    assert torch.isfinite(out[0][0]).all()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert torch.equal(x, y)


@pytest.mark.parametrize("n", [2, 2500])
def test_adjoint_of_a_vanished_t2(snap, n):
    """T2 so short that 1 / T2^2 leaves FP32's range: the gradients of a T2 of
    1e-10 ms, whose decay is as complete."""
    torch = torch_cuda()
    h = mrf_schedule(T, seed=1)
    p = torch.from_numpy(_params(n, 1)).cuda()
    g = torch.randn((1, T, 2), device="cuda", generator=torch.Generator("cuda").manual_seed(1)).repeat(n, 1, 1)
    out = []
    for t2 in (1e-10, 1e-20):
        p[:, 1] = t2
        out.append(_adjoint(snap, torch, p, g.contiguous(), h, 20, "epg_fisp"))
    for x, y in zip(*out):
        assert torch.isfinite(x).all() and torch.equal(x, y)


@pytest.mark.parametrize("w,n", [(50, 450), (100, 390), (200, 160), (256, 200)])
def test_crb_of_more_tissues_than_shared_memory_holds(snap, w, n):
    """One tissue per warp, the segments' states in global memory: losses and
    signals bit for bit those of a few tissues, whose states are on chip."""
    torch = torch_cuda()
    h = mrf_schedule(T, seed=w + 7, inversion=False)
    out = []
    p = torch.from_numpy(_params(2, w)).cuda()
    for q in (p, p.repeat(n // 2, 1).contiguous()):
        loss, ga, sig = (torch.empty(s, device="cuda") for s in ((len(q),), (T,), (len(q), 3, T)))
        snap.crb_gradient(q, h, T, T, len(q), loss, ga, 4, w, "epg_fisp", d_signals=sig, checkpoint_every=T // 2)
        out.append((loss, ga.double(), sig))
    (loss, ga, sig), (loss_n, ga_n, sig_n) = out
    assert torch.equal(sig_n[-2:], sig) and torch.equal(loss_n[:2], loss)
    assert torch.isfinite(ga).all()
    assert (ga_n / (n // 2) - ga).abs().max() <= 1e-5 * ga.abs().max()
