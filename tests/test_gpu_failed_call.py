"""A stepping call that fails on the device leaves a simulation that says so and can be read.

The step loop of small beds bounds every wait of its blocks for one another.
Here it waits for a block that was never launched: the wait runs out (about a
second), the call raises, and what the failed call had done by then (here the
first half of a step, in which some spheres left the box) is what is read.
"""
import numpy as np
import pytest

from tests import parity_util as pu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rp():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import rusty_particles_gb300 as m
    return m


@pytest.mark.parametrize("n", [900, 9000])
def test_wait_that_runs_out(rp, n):
    lo, hi = (-0.25, -0.25, -0.25), (0.25, 0.25, 0.25)
    st = pu.random_bed(7, n, lo, hi, 0.008, 0.012, ascale=0.0, tscale=0.0)
    n = len(st["radius"])
    out = np.arange(5, n, 97)
    st["position"][out, 0] = 1.25 + 1e-6  # beyond the bound: dropped in the first half
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0)
    g.set_debug(False)
    L = g._L
    rp._lib.check(L.rp_debug_absent_blocks(g._h, 1))
    stay = np.ones(n, bool)
    stay[out] = False
    for call in (1, 2):  # the second one from the state as it was read
        with pytest.raises(RuntimeError, match="did not meet"):
            g.steps(40)
        s = g.stats()
        assert s["status_bits"] & 16 and s["steps"] == 0 and s["removed"] == len(out)
        assert g.get_particle_count() == n - len(out)
        got = g.get_state()
        np.testing.assert_array_equal(got["radius"], st["radius"][stay])
        # the first half of the step that could not go on is a drift (a = 0)
        assert np.abs(got["position"] - (st["position"][stay] + st["velocity"][stay] * 1e-5 * call)).max() < 1e-12
    with pytest.raises(ValueError):
        rp._lib.check(L.rp_debug_absent_blocks(g._h, -1))
    rp._lib.check(L.rp_debug_absent_blocks(g._h, 0))
    g.steps(3)  # the setting has it uploaded afresh
    assert g.stats()["steps"] == 3 and np.isfinite(g.get_state()["acceleration"]).all()
