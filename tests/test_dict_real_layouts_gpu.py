"""The real-valued FISP / SR dictionary over the layouts of its pairs of
states (src/functions.cu:1077-1131): the shift at the ends of a lane, widths
that pad 0, 1, 2 and more states, row ends and steps off the unrolling and
the chunk, and every form of the output from the same recursion."""
import numpy as np
import pytest

from cases import mrf_schedule
from gpu_util import run_dict

pytestmark = pytest.mark.gpu


def _params(n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros((n, 4), np.float32)
    p[:, 0] = rng.uniform(200, 3000, n)
    p[:, 1] = rng.uniform(20, 300, n)
    p[:, 3] = 1.0
    return p


@pytest.mark.parametrize("echo", ["epg_fisp", "epg_sr"])
@pytest.mark.parametrize("w", [1, 2, 3, 25, 26, 49, 50, 51, 52, 64, 65, 130])
@pytest.mark.parametrize("T", [1, 33, 70])
def test_layouts_match_reference_order(snap, echo, w, T):
    """With the relaxations apart the operations are the reference order's,
    bit for bit; folded, an RF step and its relaxation round a few times
    differently: 8 roundings per step of a contraction, so 8 T eps / 2 of the
    peak bounds them (and 4 eps the shortest)."""
    h, p = mrf_schedule(T, seed=3), _params(37, 5)
    ref = run_dict(snap, echo, p, h, T, natoms=37, nstates=w, flags=snap.DICT_REFERENCE_ORDER)
    apart = run_dict(snap, echo, p, h, T, natoms=37, nstates=w, flags=snap.DICT_SEPARATE_RELAX)
    np.testing.assert_array_equal(apart, ref)
    got = run_dict(snap, echo, p, h, T, natoms=37, nstates=w)
    tol = max(4, 4 * T) * np.finfo(np.float32).eps
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    assert not got.real.any()
    unit = run_dict(snap, echo, p, h, T, natoms=37, nstates=w, flags=snap.DICT_NORMALIZE)
    n = np.linalg.norm(got.astype(np.complex128), axis=1, keepdims=True)
    n[n == 0] = 1.0  # (a schedule that starts with a zero flip angle: zero atoms stay zero)
    np.testing.assert_allclose(unit.imag, (got / n).imag, rtol=0, atol=(T + 4) * np.finfo(np.float32).eps)


@pytest.mark.parametrize("echo", ["epg_fisp", "epg_sr"])
@pytest.mark.parametrize("w", [257, 400, 512, 513, 800, 1024])
def test_wide_layouts(snap, oracle, echo, w):
    """More than 256 states: two atoms and one atom per warp.  A state k is
    reached after k steps, so in 120 steps the atoms are those of 256 states,
    the most that the reference order takes: bit for bit with the relaxations
    apart, to the roundings of 120 folded steps (see above) otherwise.  Steps
    enough to reach the last states: against the CPU oracle, whose sines and
    exponentials are the host's (2e-5 of the peak is the bar at 120 steps
    elsewhere; the roundings add up with the steps)."""
    T, n = 120, 37
    h, p = mrf_schedule(T, seed=3), _params(n, 5)
    ref = run_dict(snap, echo, p, h, T, natoms=n, nstates=256, flags=snap.DICT_REFERENCE_ORDER)
    apart = run_dict(snap, echo, p, h, T, natoms=n, nstates=w, flags=snap.DICT_SEPARATE_RELAX)
    np.testing.assert_array_equal(apart, ref)
    got = run_dict(snap, echo, p, h, T, natoms=n, nstates=w)
    assert np.abs(got - ref).max() <= 4 * T * np.finfo(np.float32).eps * np.abs(ref).max()
    T, n = w + 30, 5
    h, p = mrf_schedule(T, seed=4), _params(n, 6)
    ref = oracle.dict_atoms(echo, p, h, T, natoms=n, nstates=w)
    for flags in (0, snap.DICT_SEPARATE_RELAX):
        got = run_dict(snap, echo, p, h, T, natoms=n, nstates=w, flags=flags)
        assert (np.abs(got - ref).max(1) <= 2e-5 * T / 120 * np.abs(ref).max(1)).all()
