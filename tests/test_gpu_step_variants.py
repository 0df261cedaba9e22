"""The step's forms against each other and the oracle where they change over.

* Small beds run many steps in one cooperative launch (with four lanes a
  particle up to 8,192 particles), large ones a kernel for each pass: both give
  the same bits, at the sizes where lanes, warps and the rules change.
* The list rows of adhesive beds end where the force does, and pairs without a
  force are left out for the reference's own JKR Newton too: the oracle's forces.
* The pair law's seeded roots and quotients: the oracle's forces over masses
  from 1e-200 to 1e200 kg (the library's range as well as the seeds').
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


def _box_walls(lo, hi):
    from tests.stl_util import box_tris
    tris = box_tris(lo, hi)
    v = np.array([np.concatenate(t) for t in tris], np.float32).astype(np.float64)
    n = np.array([np.cross(t[1] - t[0], t[2] - t[0]) / np.linalg.norm(np.cross(t[1] - t[0], t[2] - t[0])) for t in tris],
                 np.float32).astype(np.float64)
    return v, n


# (normal, tangential, mode, precision, periodic, walls, fixed fraction, particles thrown out)
FORMS = {
    "hertz-coulomb-walls": (1, 0, 0, 0, (False, False, False), True, 0.1, 0),
    "sjkr-mixed-periodic": (4, 0, 0, 1, (True, False, True), False, 0.0, 0),
    "springs-physical": (0, 1, 1, 0, (True, True, True), False, 0.05, 0),
    "hertz-mindlin-removal": (1, 2, 0, 0, (False, False, True), False, 0.0, 7),
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 8191, 8193, 20011])
def test_one_launch_equals_kernel_by_kernel(rp, n, form):
    normal, tangential, mode, precision, periodic, walls, fixed, thrown = FORMS[form]
    m = int(np.ceil(n ** (1 / 3)))
    half = max(0.5 * m * 0.016, 0.05)
    lo, hi = (-half,) * 3, (half,) * 3
    st = pu.random_bed(900 + n, n, lo, hi, 0.007, 0.009, vscale=0.5, fixed_frac=fixed)
    n = len(st["radius"])
    rng = np.random.default_rng(n)
    idx = rng.choice(n, size=min(thrown, n), replace=False)
    st["position"][idx, 0] = half + 0.99995  # leave through an open face within the run
    st["velocity"][idx, 0] = 3.0
    out = []
    for loop in (1, 0):
        g = pu.gpu_sim(rp, st, 2e-5, lo, hi, normal, tangential, periodic, mode,
                       (1e7, 0.3, 2500.0, 0.5, 0.5, 0.05 if normal == 4 else 0.0), precision=precision,
                       tris=_box_walls(lo, hi) if walls else None, cell=0.11)
        g.set_debug(False)
        g.set_skin(1e-3)  # the lists are rebuilt inside the run
        g._L.rp_set_device_loop(g._h, loop)
        g.steps(30)
        g.steps(3)
        out.append((g.get_state(), g.stats()))
    (a, sa), (b, sb) = out
    assert sa["steps"] == sb["steps"] == 33 and sa["removed"] == sb["removed"] == len(idx)
    assert sa["neighbor_rebuilds"] == sb["neighbor_rebuilds"]
    if n > 100:
        assert sa["neighbor_rebuilds"] > 2
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_one_launch_above_its_largest_bed(rp):
    # the first size that takes a kernel for each pass inside the device loop
    lo, hi = (-0.6, -0.6, -0.6), (0.6, 0.6, 0.6)
    st = pu.random_bed(5, 262145, lo, hi, 0.0088, 0.0094, vscale=0.5)
    assert len(st["radius"]) == 262145
    out = []
    for loop in (1, 0):
        g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0)
        g.set_debug(False)
        g._L.rp_set_device_loop(g._h, loop)
        g.steps(3)
        out.append(g.get_state())
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)


@pytest.mark.parametrize("normal,gamma,periodic", [(3, 0.05, (True, True, True)), (3, 0.0, (False, False, False)),
                                                   (3, 0.5, (True, False, False)), (4, 0.5, (True, True, True))])
def test_adhesive_rows_end_where_the_force_does(rp, oracle_mod, normal, gamma, periodic):
    # radii 5-20 um: gaps on both sides of the end of the force (0.02-0.2 um)
    rng = np.random.default_rng(31)
    n, L = 3000, 4.4e-4
    lo, hi = (0.0, 0.0, 0.0), (L, L, L)
    m = 15
    g3 = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    r = rng.uniform(5e-6, 20e-6, n)
    st = {"position": (g3 + 0.5) * (L / m) + rng.uniform(-3e-6, 3e-6, (n, 3)), "radius": r,
          "mass": 2000.0 * 4.0 / 3.0 * np.pi * r ** 3, "velocity": rng.normal(0, 0.05, (n, 3)),
          "angular_velocity": rng.normal(0, 100.0, (n, 3)), "acceleration": np.zeros((n, 3)),
          "torque": np.zeros((n, 3)), "fixed": np.zeros(n, np.uint8)}
    mat = (5e8, 0.25, 2000.0, 0.5, 0.5, gamma)
    o = pu.oracle_sim(oracle_mod, st, 1e-9, lo, hi, normal, 0, periodic=periodic, material=mat)
    g = pu.gpu_sim(rp, st, 1e-9, lo, hi, normal, 0, periodic=periodic, material=mat)
    g.set_debug(False)
    o.step()
    g.step()
    so, sg = o.state(), g.get_state()
    FS, TS = o.last_force_scale()
    assert (FS > 0).sum() > n // 4
    np.testing.assert_array_equal(sg["position"], so["x"])
    # accelerations and torques carry the forces: 1e-9 of the particle's force scale
    assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= 1e-9 * FS / st["mass"] + 1e-9)
    assert np.all(np.abs(sg["torque"] - so["tau"]).max(1) <= 1e-9 * TS + 1e-25)


@pytest.mark.parametrize("normal,tangential,mode", [(1, 0, 0), (0, 0, 0), (1, 2, 1), (0, 1, 1)])
def test_roots_and_quotients_over_the_range(rp, oracle_mod, normal, tangential, mode):
    # pairs of spheres with masses from 1e-200 to 1e200 kg (products and
    # quotients from the seeds' range into the library's) and overlaps down to
    # rounding; one step from the same state
    rng = np.random.default_rng(77)
    pairs = 400
    k = np.arange(pairs)
    base = np.stack([k % 8, k // 8 % 8, k // 64], 1) * 0.1 - 0.35
    r = rng.uniform(0.005, 0.02, (pairs, 2))
    gap = r.sum(1) * (1.0 - 10.0 ** rng.uniform(-15, -2, pairs))
    u = rng.normal(size=(pairs, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    x = np.concatenate([base, base + u * gap[:, None]])
    mass = 10.0 ** rng.uniform(-200, 200, 2 * pairs)
    n = 2 * pairs
    st = {"position": x, "radius": np.concatenate([r[:, 0], r[:, 1]]), "mass": mass,
          "velocity": rng.normal(0, 0.5, (n, 3)), "angular_velocity": rng.normal(0, 1.0, (n, 3)),
          "acceleration": np.zeros((n, 3)), "torque": np.zeros((n, 3)), "fixed": np.ones(n, np.uint8)}
    lo, hi = (-0.6,) * 3, (0.6,) * 3
    o = pu.oracle_sim(oracle_mod, st, 1e-9, lo, hi, normal, tangential, mode=mode)
    g = pu.gpu_sim(rp, st, 1e-9, lo, hi, normal, tangential, mode=mode)
    o.step()
    g.step()
    Fo, To = o.last_forces()
    Fg, Tg = g.debug_forces()
    FS, TS = o.last_force_scale()
    assert (FS > 0).sum() > n // 2
    np.testing.assert_array_equal(np.isfinite(Fg), np.isfinite(Fo))
    fin = np.isfinite(Fo).all(1) & np.isfinite(FS)
    assert np.all(np.linalg.norm(Fg - Fo, axis=1)[fin] <= 1e-9 * FS[fin])
    assert np.all(np.linalg.norm(Tg - To, axis=1)[fin] <= 1e-9 * TS[fin])
