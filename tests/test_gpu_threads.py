"""Simulations stepped from several threads at once give what each gives alone.

Every simulation has its own streams, graph and buffers. The step loop of small
beds is one launch of blocks that wait for one another: launches of several
simulations share the device, one after the other or side by side.
"""
import threading

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


# (spheres, normal, precision): below and above four lanes a sphere, below and above 262,144, and one with a side stream
BEDS = [(700, 1, 0), (20011, 1, 0), (9000, 4, 1), (1500, 3, 0), (270000, 1, 1)]


def _bed(rp, n, normal, precision):
    half = 0.5 * int(np.ceil(n ** (1 / 3))) * 0.0165
    lo, hi = (-half,) * 3, (half,) * 3
    st = pu.random_bed(n, n, lo, hi, 0.007, 0.009, vscale=0.5)
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, normal, 0, (True, False, True), material=(1e7, 0.3, 2500.0, 0.5, 0.5,
                                                                                0.05 if normal >= 3 else 0.0),
                   precision=precision)
    g.set_debug(False)
    if normal == 3:
        g.set_jkr_solver("certified")
    return g


def _drive(g, out, key, start=None):
    if start is not None:
        start.wait()
    try:
        states = []
        for n in (1, 40, 3, 40):
            g.steps(n)
            states.append(g.get_state())
        out[key] = states
    except Exception as e:  # the thread's error is the test's
        out[key] = e


def test_simulations_in_threads(rp):
    alone, together = {}, {}
    for key, bed in enumerate(BEDS + BEDS[:2]):
        _drive(_bed(rp, *bed), alone, key)
    sims = [_bed(rp, *bed) for bed in BEDS + BEDS[:2]]
    start = threading.Barrier(len(sims))
    ts = [threading.Thread(target=_drive, args=(g, together, key, start)) for key, g in enumerate(sims)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for key in alone:
        assert isinstance(alone[key], list), alone[key]
        assert isinstance(together[key], list), (BEDS + BEDS[:2])[key] + (together[key],)
        for a, b in zip(alone[key], together[key]):
            for k in a:
                np.testing.assert_array_equal(a[k], b[k], err_msg=k)
