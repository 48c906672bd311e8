"""roa_ssfp (src/functions.cu:1021-1222) over the isochromat layouts (an odd
and an even number per lane, idle slots, groups of 8 to 32 lanes), step counts
off the staging chunk and atom counts off the block, against the FP64 oracle."""
import numpy as np
import pytest

from gpu_util import run_dict

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_iso", [1, 2, 9, 31, 57, 105, 113, 209, 225])
@pytest.mark.parametrize("T", [1, 17, 50])
def test_layouts_vs_oracle(snap, oracle, n_iso, T):
    rng = np.random.default_rng(n_iso)
    h = np.zeros((4, T), np.float32)
    h[0] = rng.uniform(0.1, 1.0, T)       # fraction of 60 degrees
    h[1] = rng.uniform(0.0, 360.0, T)     # RF phase, degrees
    h[2] = rng.uniform(0.0, 4.0, T)       # TR extension
    n = 133 if n_iso == 1 else 19
    p = np.zeros((n, 4), np.float32)
    p[:, 0] = rng.uniform(200, 3000, n)
    p[:, 1] = rng.uniform(20, 200, n)
    p[:, 2] = rng.uniform(-100, 100, n)
    p[:, 3] = 1.0
    got, norms = run_dict(snap, "roa_ssfp", p, h, T, natoms=n, n_iso=n_iso, want_norms=True)
    ref = oracle.dict_atoms("roa_ssfp", p, h, T, natoms=n, n_iso=n_iso)
    # (unit-norm atoms; the bound of the other comparisons with the oracle:
    # the sines of the fast path, 2^-21 per rotation, over T steps)
    assert np.abs(got - ref).max() < 1e-4 * np.abs(ref).max()
    assert np.isfinite(norms).all() and (norms > 0).all()
    np.testing.assert_allclose(np.linalg.norm(got.astype(np.complex128), axis=1), 1.0, rtol=1e-5)
