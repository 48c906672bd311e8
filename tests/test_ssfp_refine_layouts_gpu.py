"""bSSFP refinement: the layouts (two states per lane for few voxels; 2 to 5
states in groups of any width for many, the warp's last lanes idle) at state
counts around their edges give the same refined voxels.  The layouts differ by
the order of the inner products' sums only, about 1e-6 of the normal
equations' entries, which one step of a well-posed voxel passes on to its
parameters at most some tens of times: 1e-4 of a parameter (0.01 Hz for B0) is
allowed.  Both must also move towards the voxels' own parameters."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


def _schedule(T, seed):
    r = np.random.default_rng(seed)
    t = np.arange(T)
    tr = r.uniform(10, 14, T)
    return np.array([(5 + 55 * np.abs(np.sin(np.pi * t / 70))) / 60, 180.0 * (t % 2), tr - 16, tr / 2 - 3.5], np.float32)


@pytest.mark.parametrize("use_map", [True, False])
@pytest.mark.parametrize("w", [10, 15, 16, 20, 33, 50, 51, 64, 65, 100, 128])
def test_layouts_refine_alike(snap, w, use_map):
    torch = torch_cuda()
    T, few, rep = 203, 7, 400
    r = np.random.default_rng(w)
    t1 = r.uniform(600, 1800, few)
    p = np.stack([t1, t1 * r.uniform(0.05, 0.15, few), r.uniform(-30, 30, few), r.uniform(0.9, 1.1, few)], 1)
    p = p.astype(np.float32)
    h = _schedule(T, w)
    d_p = torch.from_numpy(p).cuda()
    atoms = torch.empty((few, T, 2), device="cuda")
    for i in range(few):  # one B1 block per voxel: its own flip angles
        snap.MRF_dict(atoms[i], d_p[i:i + 1].contiguous(), h, T, T, 1, 1, 4, w, "epg_ssfp")
    start = p * np.float32([1.02, 0.98, 1.0, 1.0]) + np.float32([0, 0, 0.7, 0])
    if not use_map:
        start[:, 3] *= 1.01
    start = np.concatenate([start, np.ones((few, 1), np.float32)], 1)
    out = []
    for n in (1, rep):
        maps = torch.from_numpy(np.tile(start, (n, 1))).cuda()
        img = atoms.repeat(n, 1, 1).contiguous()
        b1 = d_p[:, 3].repeat(n).contiguous() if use_map else None
        snap.refine_gn(maps, img, h, T, T, few * n, w, "epg_ssfp", iterations=1, tol=0.0, d_b1map=b1)
        out.append(maps.cpu().numpy())
    a, b = out[0], out[1][:few]
    np.testing.assert_array_equal(out[1][-few:], b)
    np.testing.assert_allclose(a[:, [0, 1, 3, 4]], b[:, [0, 1, 3, 4]], rtol=1e-4)
    np.testing.assert_allclose(a[:, 2], b[:, 2], atol=0.01)
    truth = np.concatenate([p, np.ones((few, 1), np.float32)], 1)
    assert np.median(np.abs(a[:, :2] / truth[:, :2] - 1)) < 5e-3
    assert np.median(np.abs(a[:, 2] - truth[:, 2])) < 0.2


@pytest.mark.parametrize("echo", ["epg_fisp", "epg_ssfp"])
def test_vanished_t2(snap, echo):
    """T2 so short that 1 / T2^2 leaves FP32's range, sampled at TE = 0 (there
    is a signal): its derivative is as 0 as at a T2 of 1e-10 ms."""
    torch = torch_cuda()
    T, w = 60, 10
    r = np.random.default_rng(2)
    h = np.stack([r.uniform(0.2, 0.9, T), np.zeros(T), np.full(T, 12.0), np.zeros(T)]).astype(np.float32)
    if echo == "epg_ssfp":
        h[2:] -= np.float32([[16.0], [3.5]])
    img = torch.randn((2, T, 2), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    img[1] = img[0]
    maps = torch.tensor([[800, 1e-10, 0, 1, 1], [800, 1e-20, 0, 1, 1]], device="cuda")
    snap.refine_gn(maps, img, h, T, T, 2, w, echo, iterations=1, tol=0.0)
    maps = maps.cpu().numpy()
    assert np.isfinite(maps).all()
    np.testing.assert_array_equal(maps[0], maps[1])
