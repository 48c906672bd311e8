"""epg_ssfp in the frame of the RF phase against the reference's order of
operations (SNAPMRF_DICT_REFERENCE_ORDER): the same recursion with the same
constants, so the atoms agree to rounding, far inside the parity bar of 1e-5
of an atom's peak (1e-5 is what is asked here), at the edges of its layouts
(state counts around multiples of the lanes, few and many atoms, one state),
partial chunks of steps, and any RF phase; norms too."""
import numpy as np
import pytest

from gpu_util import run_dict

pytestmark = pytest.mark.gpu


def _schedule(T, phases, seed):
    r = np.random.default_rng(seed)
    t = np.arange(T)
    ph = {"alternating": 180.0 * (t % 2), "zero": 0.0 * t, "quadratic": (58.5 * t * t) % 360.0}[phases]
    tr = r.uniform(-6, -2, T)
    return np.array([0.1 + 0.9 * np.abs(np.sin(t / 40)), ph, tr, (tr + 16) / 2 - 3.5], np.float32)


@pytest.mark.parametrize("phases", ["alternating", "zero", "quadratic"])
@pytest.mark.parametrize("T,w,n", [(1, 50, 3), (17, 1, 40), (40, 2, 5), (33, 3, 9000), (150, 20, 33), (160, 50, 7001),
                                   (100, 51, 300), (64, 52, 9001), (90, 101, 4000), (50, 128, 50), (45, 250, 20),
                                   (30, 256, 700)])
def test_frame_recursion_equals_reference_order(snap, T, w, n, phases):
    r = np.random.default_rng(w + n)
    t1 = r.uniform(200, 3000, n)
    p = np.stack([t1, t1 * r.uniform(0.03, 0.6, n), r.uniform(-100, 100, n), np.ones(n)], 1).astype(np.float32)
    p = np.concatenate([p, p * np.float32([1, 1, 1, 0.9])])  # a second B1 block
    h = _schedule(T, phases, w)
    a, na = run_dict(snap, "epg_ssfp", p, h, T, natoms=n, nstates=w, want_norms=True)
    b, nb = run_dict(snap, "epg_ssfp", p, h, T, natoms=n, nstates=w, want_norms=True, flags=snap.DICT_REFERENCE_ORDER)
    assert np.isfinite(a).all()
    d = np.abs(a - b).max(axis=1) / np.abs(b).max(axis=1)
    assert d.max() <= 1e-5, d.max()
    np.testing.assert_allclose(na, nb, rtol=1e-5)
