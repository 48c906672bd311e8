"""The FP32 form screened on the tensor cores chooses the atoms that the FP32
kernel alone chooses.  snapmrf_mrf_match_noalloc always runs that kernel over
every atom, so maps and indices of the two are compared bit for bit: at the
edges of the screen's tiles (64 / 128 voxels, 256 / 128 atoms, 32 elements of
K), with purely imaginary and complex atoms, odd strides, a B1 map with empty
and one-voxel blocks, atoms of very different norms, exact duplicates, and
voxels and atoms that the screen must leave to the FP32 kernel (zero, tiny,
huge, infinite, NaN; a grid so fine that more atoms than a list holds lie
within the screen's bound)."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def take_the_screen(monkeypatch):
    """Whatever a call's size (the rule keeps small calls with the FP32 kernel)."""
    monkeypatch.setenv("SNAPMRF_SCREEN", "1")


def _both(snap, img, atoms, params, nreps, natoms, b1map=None, imag=False):
    torch = torch_cuda()
    N, stride = atoms.shape
    nvox = img.shape[0]
    d_atoms = torch.from_numpy(np.ascontiguousarray(atoms).view(np.float32)).cuda()
    d_img = torch.from_numpy(np.ascontiguousarray(img).view(np.float32)).cuda()
    d_p = torch.from_numpy(params).cuda()
    d_b1 = None if b1map is None else torch.from_numpy(b1map).cuda()
    out = []
    for call in ("screened", "plain"):
        maps = torch.full((nvox, 5), -3.0, device="cuda")
        idx = torch.full((nvox,), -9, dtype=torch.int64, device="cuda")
        if call == "screened":
            snap.MRF_match(maps, d_img, d_atoms, d_p, stride, nreps, N, natoms, nvox, in_b1map=d_b1, d_index=idx,
                           img_stride=img.shape[1], flags=snap.MATCH_IMAG_ATOMS if imag else 0)
        else:
            snap.MRF_match_noalloc(maps, d_img, d_atoms, d_p, stride, nreps, N, natoms, nvox, d_b1map=d_b1,
                                   img_stride=img.shape[1], d_index=idx)
        torch.cuda.synchronize()
        out.append((maps.cpu().numpy(), idx.cpu().numpy()))
    assert snap.device_error(reset=True) == 0
    return out


def _inputs(nvox, natoms, T, nb, imag, seed, smooth=40.0):
    """Atoms along a smooth two-parameter family (neighbours correlate as a
    dictionary's do) and voxels near them."""
    rng = np.random.default_rng(seed)
    t = np.arange(T)[None, :] / T
    u = np.arange(natoms)[:, None] / smooth
    atoms = []
    for b in range(nb):
        f = 0.1 * np.sin(6 * t * (1 + u) + 0.2 * b) * np.exp(-t * u) + 0.05 * np.cos(25 * t + u)
        atoms.append(1j * f if imag else f * np.exp(1j * (3 * t * u + 0.1 * b)))
    atoms = np.concatenate(atoms)
    atoms /= np.linalg.norm(atoms, axis=1, keepdims=True)
    s = atoms[rng.integers(0, len(atoms), nvox)] + 0.2 * atoms[rng.integers(0, len(atoms), nvox)]
    s = s * (rng.uniform(0.5, 1, nvox) * np.exp(6.28j * rng.uniform(size=nvox)))[:, None]
    s = s + 0.02 / np.sqrt(T) * (rng.standard_normal(s.shape) + 1j * rng.standard_normal(s.shape))
    params = rng.uniform(1, 100, (len(atoms), 4)).astype(np.float32)
    params[:, 3] = np.repeat(0.8 + 0.1 * np.arange(nb), natoms)
    return atoms.astype(np.complex64), s.astype(np.complex64), params


@pytest.mark.parametrize("nvox,natoms,T,nb,use_map,imag,pad", [
    (4096, 837, 100, 1, False, False, 0), (1025, 129, 257, 1, False, True, 0), (63, 4097, 128, 1, False, True, 1),
    (129, 1283, 333, 1, False, False, 3), (1, 30000, 1000, 1, False, True, 0), (30011, 7, 97, 1, False, False, 0),
    (2500, 300, 200, 5, True, True, 0), (1500, 257, 161, 6, True, False, 1), (20000, 1999, 64, 3, True, True, 2)])
def test_screened_match_equals_the_fp32_kernel(snap, nvox, natoms, T, nb, use_map, imag, pad):
    atoms, img, params = _inputs(nvox, natoms, T, nb, imag, seed=nvox + T)
    nreps = T - pad
    b1map = None
    if use_map:
        b1map = np.random.default_rng(1).uniform(0.78, 0.82 + 0.1 * (nb - 1), nvox).astype(np.float32)
        b1map[np.abs(b1map - 0.9) < 0.05] = 0.8      # block 1: one voxel
        b1map[5] = 0.9
    a, b = _both(snap, img, atoms, params, nreps, natoms, b1map, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("imag", [True, False])
def test_inputs_left_to_the_fp32_kernel(snap, imag):
    atoms, img, params = _inputs(700, 1500, 150, 1, imag, seed=3)
    atoms[700] = atoms[11]                        # duplicates: the lower index wins
    atoms[1499] = atoms[1498]
    atoms *= np.float32(10.0) ** np.random.default_rng(4).integers(-3, 4, (1500, 1))
    img[0] = 0
    img[1, 7] = np.nan
    img[2, 9] = np.inf
    img[3] = 1e-20
    img[4] *= np.float32(1e-25)
    img[5] *= np.float32(1e17)
    img[6] = atoms[11]
    img[7, 1:] = 0
    # (an infinite voxel: the complex form's products of the zero real parts
    # are NaN, the imaginary form has no such products and scores inf; the
    # comparison call is the complex form)
    same = np.arange(700) != 2 if imag else slice(None)
    a, b = _both(snap, img, atoms, params, 150, 1500, None, imag)
    np.testing.assert_array_equal(a[1][same], b[1][same])
    np.testing.assert_array_equal(a[0][same], b[0][same])
    for value in (np.inf, np.nan, 1e25, 1e-22):   # an atom out of the screen's range
        bad = atoms.copy()
        bad[77, 5] = complex(0.0, value)
        a, b = _both(snap, img, bad, params, 150, 1500, None, imag)
        np.testing.assert_array_equal(a[1][same], b[1][same])
        np.testing.assert_array_equal(a[0][same], b[0][same])
    a, b = _both(snap, img, atoms * np.float32(1e-19), params, 150, 1500, None, imag)
    np.testing.assert_array_equal(a[1][same], b[1][same])
    np.testing.assert_array_equal(a[0][same], b[0][same])


@pytest.mark.parametrize("imag", [True, False])
def test_more_near_ties_than_a_list_holds(snap, imag):
    """20,000 atoms along one slow curve: hundreds lie within the bound."""
    atoms, img, params = _inputs(300, 20000, 120, 1, imag, seed=8, smooth=20000.0)
    a, b = _both(snap, img, atoms, params, 120, 20000, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("T", [8, 9, 16, 17, 31, 33, 48])
def test_short_rows(snap, imag, T):
    """Few samples: the split of the operands, not the sums' rounding, decides
    the screen's bound."""
    atoms, img, params = _inputs(2100, 1300, T, 1, imag, seed=T)
    a, b = _both(snap, img, atoms, params, T, 1300, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("imag", [True, False])
def test_parts_left_out_by_the_split(snap, imag):
    """Rows made for the split's largest error: 15 of 16 samples just below
    and just above 1 + 2^-8 round to neighbouring BF16 values, the products of
    the low parts that the screen leaves out have opposite signs, and the atom
    that scores higher in FP32 (by 2k ulp) looks worse to the screen by 2^-15."""
    T, n = 16, 1100
    f = np.float32
    x = np.zeros((1100, T), f)
    # (scaled to unit norm by a factor a few ulp off 1: m keeps them above the tie)
    x[:, :15] = f(1 + 2.0 ** -8) / 4 + (1 + np.arange(1100) % 64)[:, None].astype(f) * f(2.0 ** -25)
    x[:, 15] = np.sqrt(1 - 15 * x[:, 0].astype(np.float64) ** 2)
    img = np.where((np.arange(1100) % 2 == 0)[:, None], x * 1j, x + 0j).astype(np.complex64)
    params = np.random.default_rng(2).uniform(1, 100, (n, 4)).astype(f)
    for k in (1, 2, 3, 8):
        d = np.zeros((n, T), f)     # (the other atoms score 0: nothing else is listed)
        d[20, :15] = f(1 + 2.0 ** -8) - f(k * 2.0 ** -23)
        d[320, :15] = f(1 + 2.0 ** -8) + f(k * 2.0 ** -23)
        a, b = _both(snap, img, (1j * d if imag else d + 0j).astype(np.complex64), params, T, n, None, imag)
        np.testing.assert_array_equal(a[1], b[1])
        np.testing.assert_array_equal(a[0], b[0])
        assert (b[1] == 320).all()


@pytest.mark.parametrize("imag", [True, False])
def test_sums_that_the_tensor_core_cuts(snap, imag):
    """A large first product, then small ones that an FP32 sum and the tensor
    core's round differently (1.25 2^-24 beside 1: up to 2^-23 and down to
    2^-24), against the same products in the other order."""
    T, n = 1000, 300
    rng = np.random.default_rng(11)
    d = np.full((n, T), np.sqrt(1.25 * 2.0 ** -24))
    d[:, 0] = 1.0
    d[n // 2:] = d[n // 2:, ::-1]
    d *= 1 + 4e-5 * rng.uniform(-1, 1, (n, 1))
    x = np.full((120, T), np.sqrt(1.25 * 2.0 ** -24)) * (1 + 1e-3 * rng.standard_normal((120, T)))
    x[:, 0] = x[:, -1] = 1.0
    x = (x * np.exp(1j * np.pi / 2 * rng.integers(0, 4, (120, 1)))).astype(np.complex64)
    params = rng.uniform(1, 100, (n, 4)).astype(np.float32)
    a, b = _both(snap, x, (1j * d if imag else d + 0j).astype(np.complex64), params, T, n, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("imag", [True, False])
def test_blocks_without_voxels_are_not_looked_at(snap, imag):
    """A B1 block that no voxel falls into: whatever its atoms hold (a real
    part, NaN, another scale) changes nothing."""
    nb, natoms = 4, 700
    atoms, img, params = _inputs(600, natoms, 90, nb, imag, seed=21)
    b1map = np.random.default_rng(1).choice(np.float32([0.8, 1.0]), 600)      # blocks 0 and 2
    want = _both(snap, img, atoms, params, 90, natoms, b1map, imag)
    other = atoms.copy()
    other[natoms:2 * natoms] *= 1e12
    other[natoms + 3, 5] = 0.25 + 1j
    other[3 * natoms + 1, 2] = np.nan
    other[3 * natoms + 2, 2] = 1e30
    a, b = _both(snap, img, other, params, 90, natoms, b1map, imag)
    for got in (a, b, want[0]):
        np.testing.assert_array_equal(got[1], want[1][1])
        np.testing.assert_array_equal(got[0], want[1][0])


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("nvox,natoms,smooth", [(300, 40000, 4000.0), (70, 70000, 20000.0), (2000, 17000, 600.0),
                                                (100, 17000, 0.0)])
def test_long_lists(snap, imag, nvox, natoms, smooth):
    """Lists that grow with the dictionary, are compacted or overflow, and are
    rescored by several warps per voxel (0: all atoms the same, the first wins)."""
    if smooth:
        atoms, img, params = _inputs(nvox, natoms, 110, 1, imag, seed=natoms, smooth=smooth)
    else:
        atoms, img, params = _inputs(nvox, 50, 110, 1, imag, seed=9)
        atoms = np.repeat(atoms[7:8], natoms, 0)
        params = np.random.default_rng(1).uniform(1, 100, (natoms, 4)).astype(np.float32)
    a, b = _both(snap, img, atoms, params, 110, natoms, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


def _row_bytes(T, imag):
    """Operand bytes of an atom and of a voxel: 32 elements in 128 bytes."""
    chunks = ((1 if imag else 2) * T + 31) // 32
    return (1 if imag else 2) * chunks * 128, (2 if imag else 1) * chunks * 128


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("nb,natoms,per_atoms,per_voxels,lists", [
    (5, 700, 1500, 1 << 20, 1 << 30),     # two blocks per pass, the last alone
    (3, 700, 300, 1 << 20, 1 << 30),      # a block in chunks of 256, the last short
    (1, 3000, 600, 500, 1 << 30),         # chunks, and five ranges of voxels
    (4, 700, 100000, 500, 1 << 30),       # ranges of voxels alone
    (1, 3000, 600, 100000, 1 << 23),      # ranges from the lists' room
    (5, 700, 1500, 50, 1 << 16)])         # more padded slots than room: the FP32 kernel
def test_passes(snap, monkeypatch, imag, nb, natoms, per_atoms, per_voxels, lists):
    """Dictionaries, images and lists larger than one pass: atom norms that
    rise and fall from chunk to chunk, blocks with and without voxels."""
    T, nvox = 130, 2100
    atoms, img, params = _inputs(nvox, natoms, T, nb, imag, seed=natoms + nb)
    atoms = (atoms * np.float32(10.0) ** np.linspace(-1, 1, len(atoms), dtype=np.float32)[:, None]).astype(np.complex64)
    atoms[len(atoms) // 2:] = atoms[:len(atoms) // 2 - 1:-1].copy()
    b1map = None
    if nb > 1:
        b1map = np.random.default_rng(3).choice(np.float32(0.8 + 0.1 * np.arange(1, nb)), nvox)
    rb = _row_bytes(T, imag)
    monkeypatch.setenv("SNAPMRF_SCREEN_PASS", f"{per_atoms * rb[0]},{per_voxels * rb[1]},{lists}")
    a, b = _both(snap, img, atoms, params, T, natoms, b1map, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("smooth", [20000.0, 2000.0])
def test_lists_across_chunks(snap, monkeypatch, imag, smooth):
    """Near ties in every chunk of a block: lists that go on from launch to
    launch, fill up and overflow."""
    T = 120
    atoms, img, params = _inputs(300, 20000, T, 1, imag, seed=8, smooth=smooth)
    monkeypatch.setenv("SNAPMRF_SCREEN_PASS", f"{3000 * _row_bytes(T, imag)[0]},{1 << 30},{1 << 30}")
    a, b = _both(snap, img, atoms, params, T, 20000, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


def test_a_real_part_in_any_range_fails_the_whole_call(snap, monkeypatch):
    """One error for the call, wherever the voxels of the offending block lie."""
    torch = torch_cuda()
    T, natoms, nvox = 100, 700, 1500
    atoms, img, params = _inputs(nvox, natoms, T, 2, True, seed=4)
    atoms[natoms + 9, 3] += 0.5
    b1map = np.where(np.arange(nvox) < 1490, 0.8, 0.9).astype(np.float32)
    monkeypatch.setenv("SNAPMRF_SCREEN_PASS", f"{1 << 30},{400 * _row_bytes(T, True)[1]},{1 << 30}")
    maps = torch.full((nvox, 5), -3.0, device="cuda")
    idx = torch.full((nvox,), -9, dtype=torch.int64, device="cuda")
    snap.MRF_match(maps, torch.from_numpy(img.view(np.float32)).cuda(), torch.from_numpy(atoms.view(np.float32)).cuda(),
                   torch.from_numpy(params).cuda(), T, T, 2 * natoms, natoms, nvox,
                   in_b1map=torch.from_numpy(b1map).cuda(), d_index=idx, img_stride=T, flags=snap.MATCH_IMAG_ATOMS)
    torch.cuda.synchronize()
    assert snap.device_error(reset=True) == 7
    assert torch.isnan(maps).all() and (idx == -1).all()


@pytest.mark.parametrize("imag", [True, False])
def test_a_wait_that_runs_out_leaves_the_call_to_the_fp32_kernel(snap, monkeypatch, imag):
    atoms, img, params = _inputs(700, 1500, 150, 1, imag, seed=3)
    monkeypatch.setenv("SNAPMRF_SCREEN_WAIT_ERROR", "1")
    a, b = _both(snap, img, atoms, params, 150, 1500, None, imag)
    np.testing.assert_array_equal(a[1], b[1])
    np.testing.assert_array_equal(a[0], b[0])


@pytest.mark.parametrize("use_map", [True, False])
def test_host_image_in_two_ranges(snap, use_map):
    """A host image of five copies: all but the last two chunks' voxels are
    matched first, as the same image on the device is in one range."""
    from gpu_util import run_match
    T, nb, natoms, nvox = 1000, 2, 300, 10500
    atoms, img, params = _inputs(nvox, natoms, T, nb, True, seed=6)
    b1map = np.random.default_rng(3).choice(np.float32([0.8, 0.9]), nvox) if use_map else None
    out = [run_match(snap, img, atoms, params, natoms=natoms, b1map=b1map, device_img=dev, flags=snap.MATCH_IMAG_ATOMS)
           for dev in (False, True)]
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("nvox,natoms,T,imag,screened", [
    (300, 400, 64, True, False), (300, 400, 64, False, False), (1024, 2800, 200, True, True),
    (4096, 837, 1000, False, True), (40, 6900, 1000, True, False), (5000, 20, 100, True, False)])
def test_rule(snap, monkeypatch, nvox, natoms, T, imag, screened):
    """Small calls stay with the FP32 kernel, which takes half the launches."""
    atoms, img, params = _inputs(nvox, natoms, T, 1, imag, seed=5)
    count = []
    for force in ("0", "1", None):
        if force is None:
            monkeypatch.delenv("SNAPMRF_SCREEN")
        else:
            monkeypatch.setenv("SNAPMRF_SCREEN", force)
        before = snap.kernel_launches()
        a, b = _both(snap, img, atoms, params, T, natoms, None, imag)
        count.append(snap.kernel_launches() - before)
        np.testing.assert_array_equal(a[1], b[1])
        np.testing.assert_array_equal(a[0], b[0])
    assert count[0] < count[1]
    assert count[2] == count[int(screened)]
