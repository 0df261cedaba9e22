"""Buffers that a stepping call outgrows: the call halts, grows them and goes on.

Where the lists, the wall candidates or the pair list turn out too short, the
step that found it is finished on larger ones and the rest of the call runs on;
room never changes a result, so every run here is compared bit for bit with one
that had room from the start (or with the host-issued loop).
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


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("tangential", [2, 1], ids=["mindlin", "linear_spring"])
@pytest.mark.parametrize("loop", [1, 0], ids=["device_loop", "host_loop"])
def test_springs_survive_list_growth_inside_a_call(rp, loop, tangential):
    # a bed that is squeezed towards its middle: its rows grow from rebuild to
    # rebuild and outgrow their capacity in the middle of a call, after an even
    # and after an odd number of rebuilds since the call began
    lo, hi = (-0.15, -0.15, -0.15), (0.15, 0.15, 0.15)
    rng = np.random.default_rng(41)
    n = 2000
    x = rng.uniform(-0.1, 0.1, (n, 3))
    r = rng.uniform(0.008, 0.01, n)
    st = {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3,
          "velocity": rng.normal(0, 0.5, (n, 3)) - 40.0 * x, "angular_velocity": rng.normal(0, 1.0, (n, 3)),
          "acceleration": np.zeros((n, 3)), "torque": np.zeros((n, 3)), "fixed": np.zeros(n, np.uint8)}

    def run(cap, calls):
        g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, tangential, mode=1, material=(1e3, 0.3, 2500.0, 0.5, 0.5, 0.0))
        g.set_debug(False)
        g.set_neighbor_capacity(cap)
        g.set_skin(4e-4)
        g._L.rp_set_device_loop(g._h, loop)
        grown = []
        for steps in calls:
            g.steps(steps)
            s = g.stats()
            grown.append((s["neighbor_rebuilds"], s["max_neighbors"], s["status_bits"] & 4))
        return g, grown

    _, track = run(160, [1] * 80)
    rebuilds = [r for r, _, _ in track]
    cap = track[0][1]  # the longest row of the first lists
    full = rebuilds[next(k for k, t in enumerate(track) if t[1] > cap)]  # the rebuild that finds a longer one
    assert full >= 6
    for before in (2, 3):  # rebuilds in the call before: an even or odd number remains
        first = rebuilds.index(before) + 1
        calls = [first, 80 - first]
        ref, _ = run(160, calls)
        g, grown = run(cap, calls)
        assert np.abs(ref.get_state()["torque"]).max() > 0
        assert not grown[0][2] and grown[1][2] and grown[1][0] == rebuilds[-1]
        _same(g.get_state(), ref.get_state())
