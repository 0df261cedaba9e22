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


def _cloud(seed, n, half, rmin, rmax, squeeze=0.0):
    """Spheres at random in a cube of half-width `half` (overlapping freely), drawn together at `squeeze` per second."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-half, half, (n, 3))
    r = rng.uniform(rmin, rmax, n)
    return {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3,
            "velocity": rng.normal(0, 0.5, (n, 3)) - squeeze * x, "angular_velocity": rng.normal(0, 1.0, (n, 3)),
            "acceleration": np.zeros((n, 3)), "torque": rng.normal(0, 1e-6, (n, 3)), "fixed": np.zeros(n, np.uint8)}


# (normal, tangential, mode, precision, solver, surface energy): the last form's pairs all go to the list beside the fold
FORMS = {
    "hertz": (1, 0, 0, 0, "newton", 0.0),
    "hertz-mixed-springs": (1, 2, 1, 1, "newton", 0.0),
    "jkr-newton": (3, 0, 0, 0, "newton", 0.05),
    "jkr-certified": (3, 0, 0, 0, "certified", 0.05),
    "jkr-certified-mixed": (3, 0, 0, 1, "certified", 0.05),
    "jkr-all-beside-the-fold": (3, 0, 0, 0, "certified", 1e-11),
}


def _run(rp, st, form, lo, hi, loop, cap, calls, skin, dt=1e-6, **kw):
    normal, tangential, mode, precision, solver, gamma = FORMS[form]
    g = pu.gpu_sim(rp, st, dt, lo, hi, normal, tangential, mode=mode, precision=precision,
                   material=(1e4, 0.3, 2500.0, 0.5, 0.5, gamma), **kw)
    g.set_debug(False)
    g.set_jkr_solver(solver)
    if cap:
        g.set_neighbor_capacity(cap)
    g.set_skin(skin)
    g._L.rp_set_device_loop(g._h, loop)
    for n in calls:
        g.steps(n)
    return g


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("loop", [1, 0], ids=["device_loop", "host_loop"])
def test_pair_list_outgrown(rp, form, loop):
    # rows as short as the longest one and contacts in most of their places: more
    # evaluated pairs than the list for them starts with
    lo, hi = (-0.3, -0.3, -0.3), (0.3, 0.3, 0.3)
    st = _cloud(11, 20000, 0.1, 0.0085, 0.01)
    probe = _run(rp, st, form, lo, hi, 1, 400, [1], 1e-4)
    longest = probe.stats()["max_neighbors"]
    fold = form == "jkr-all-beside-the-fold"  # that list starts shorter and grows in every run
    ref = _run(rp, st, form, lo, hi, loop, 400, [3, 2], 1e-4)
    g = _run(rp, st, form, lo, hi, loop, int(longest), [3, 2], 1e-4)
    assert (ref.stats()["status_bits"] & (4 | 32) == 0 or fold) and g.stats()["status_bits"] & 32
    _same(g.get_state(), ref.get_state())


@pytest.mark.parametrize("n", [33, 1000, 8193])
@pytest.mark.parametrize("form", ["jkr-newton", "jkr-certified", "jkr-certified-mixed"])
def test_jkr_loops_agree_across_rebuilds_and_growth(rp, form, n):
    # beds with JKR take a kernel for each pass inside the device loop, at any
    # size, and in FP64 the spins are kicked in the contact filter: rebuilds, a
    # list that overflows with a kick still due and spheres that leave
    lo, hi = (-0.3, -0.3, -0.3), (0.3, 0.3, 0.3)
    half = 0.1 * (n / 2000) ** (1 / 3)
    st = _cloud(n, n, half, 0.008, 0.01, squeeze=100.0)
    out = np.arange(7, n, 101)
    st["position"][out, 0] = 1.2995
    st["velocity"][out, 0] = np.linspace(5.0, 20.0, len(out))
    calls = [60, 1, 19]
    one = _run(rp, st, form, lo, hi, 1, 200, [1], 2e-4, dt=1e-5).stats()["max_neighbors"]
    got = [_run(rp, st, form, lo, hi, loop, cap, calls, 2e-4, dt=1e-5)
           for loop, cap in ((1, 200), (0, 200), (1, int(one)), (0, int(one)))]
    s = [g.stats() for g in got]
    assert all(q["steps"] == 80 and q["neighbor_rebuilds"] > 10 and q["removed"] > 0 for q in s)
    if n >= 1000:
        assert s[2]["status_bits"] & s[3]["status_bits"] & 4 and not s[0]["status_bits"] & 4
    for g in got[1:]:
        _same(g.get_state(), got[0].get_state())


def _floor(half, m):
    xs = np.linspace(-half, half, m + 1)
    X0, Z0 = np.meshgrid(xs[:-1], xs[:-1], indexing="ij")
    X1, Z1 = np.meshgrid(xs[1:], xs[1:], indexing="ij")
    a, b, c, d = (np.stack([X, np.zeros_like(X), Z], -1).reshape(-1, 3) for X, Z in ((X0, Z0), (X1, Z0), (X0, Z1), (X1, Z1)))
    v = np.concatenate([np.concatenate([a, c, b], 1), np.concatenate([b, c, d], 1)]).astype(np.float32).astype(float)
    return v, np.tile([0.0, 1.0, 0.0], (len(v), 1))


@pytest.mark.parametrize("form,side,size", [("jkr-newton", 19, 0.001), ("jkr-certified", 19, 0.001), ("hertz", 513, 0.012)],
                         ids=["jkr-newton", "jkr-certified", "hertz-263169"])
def test_wall_candidates_outgrow_their_buffer_in_the_device_loop(rp, form, side, size):
    # a layer of spinning spheres on a floor of small triangles, in the loop of
    # kernels (JKR, or more than 262,144 spheres) whose contact filter kicks the
    # spins: the filter that finds the buffer full has kicked them, and the step
    # that is run again must not kick them twice
    rng = np.random.default_rng(side)
    g2 = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2) - (side - 1) / 2
    n = len(g2)
    r = np.full(n, 0.006)
    x = np.stack([g2[:, 0] * 0.013, (0.002 if size < 0.006 else 0.0055) + rng.uniform(0, 1e-4, n), g2[:, 1] * 0.013], 1)
    st = {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3, "velocity": rng.normal(0, 0.05, (n, 3)),
          "angular_velocity": rng.normal(0, 1.0, (n, 3)), "acceleration": np.zeros((n, 3)),
          "torque": rng.normal(0, 1e-4, (n, 3)), "fixed": np.zeros(n, np.uint8)}
    half = side * 0.0065 + 0.05
    lo, hi = (-half, -0.1, -half), (half, 0.2, half)
    tris = _floor(half, int(2 * half / size))
    got = [_run(rp, st, form, lo, hi, loop, 0, [4], 1e-3, tris=tris, wall=(1e5, 0.25, 7800.0, 0.3, 0.6, 0.0))
           for loop in (1, 0)]
    for g in got:
        assert g.stats()["status_bits"] & 8 and g.stats()["steps"] == 4
    a, b = (g.get_state() for g in got)
    assert np.abs(a["angular_velocity"] - st["angular_velocity"]).max() > 0
    _same(a, b)


def test_memory_of_a_bed(rp):
    # bytes a place of the rows (32 a sphere): 8 for the two rows, 8 for a
    # record, 48 for its result, 4 for the list of evaluated pairs; a sphere's
    # own arrays take under 1,100
    torch = pytest.importorskip("torch")
    n = 524288
    st = pu.random_bed(3, n, (-0.8,) * 3, (0.8,) * 3, 0.0095, 0.0098)
    assert len(st["radius"]) == n
    free = []
    for solver in ("newton", "certified"):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        g = pu.gpu_sim(rp, st, 1e-6, (-0.8,) * 3, (0.8,) * 3, 3, 0, material=(1e7, 0.3, 2500.0, 0.5, 0.5, 0.05))
        g.set_debug(False)
        g.set_jkr_solver(solver)
        g.steps(2)
        free.append((before - torch.cuda.mem_get_info()[0]) / n)
        assert not g.stats()["status_bits"] & (4 | 32)
        del g
    assert free[0] <= 1100 + 68 * 32, free
    assert free[1] <= 1100 + 72 * 32, free
