"""Spheres that leave (or join) while others hold them in their lists.

A sphere that crosses an open face is dropped at once (src/simulation.rs:199-219),
while the rows of the spheres next to it name it until the lists are rebuilt:
nothing of it may reach them, whichever of the two has the higher slot. Between
stepping calls the slots are compacted or appended to, and every remaining
contact keeps its tangential spring (src/contact.rs:4-17).

Positions to 1e-12 m; forces and torques to 1e-9 of a particle's sum of
contact-force magnitudes (FP64), 1e-5 (mixed, whose pair law is in FP32).
"""
import numpy as np
import pytest

from tests import parity_util as pu
from tests.test_gpu_history import sheared_bed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rp():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import rusty_particles_gb300 as m
    return m


def _state(x, r, v, w):
    n = len(x)
    return {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3, "velocity": v,
            "angular_velocity": w, "acceleration": np.zeros((n, 3)), "torque": np.zeros((n, 3)),
            "fixed": np.zeros(n, np.uint8)}


def _clusters(seed, lo, hi):
    """Triples of overlapping spheres straddling the removal bounds of the open faces, moving outward, each triple
    turned another way, so that a leaving sphere is found before and after its neighbours in the slots."""
    rng = np.random.default_rng(seed)
    x, v = [], []
    for axis, side in [(0, 0), (0, 1), (1, 0), (2, 0), (2, 1)]:
        bound = lo[axis] - 1.0 if side == 0 else hi[axis] + 1.0
        out = -1.0 if side == 0 else 1.0
        for k in range(40):
            c = np.zeros(3)
            c[axis] = bound - out * rng.uniform(0.0002, 0.0008)
            a, b = (axis + 1) % 3, (axis + 2) % 3
            c[a], c[b] = lo[a] + 0.06 * (k % 8) - 0.02, lo[b] + 0.08 * (k // 8)
            u = np.linalg.qr(rng.normal(size=(3, 3)))[0]
            for d in (0.0 * u[0], 0.0185 * u[0], 0.0185 * u[1]):
                x.append(c + d)
                vel = rng.normal(0, 0.05, 3)
                vel[axis] = out * 3.0
                v.append(vel)
    x = np.array(x)
    keep = (x >= lo - 1.0).all(1) & (x[:, [0, 2]] <= hi[[0, 2]] + 1.0).all(1)
    x, v = x[keep], np.array(v)[keep]
    return _state(x, np.full(len(x), 0.01), v, rng.normal(0, 1.0, (len(x), 3)))


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("loop", [1, 0], ids=["device_loop", "host_loop"])
@pytest.mark.parametrize("mode", [0, 1], ids=["parity", "physical"])
def test_touching_spheres_leave_one_by_one(rp, oracle_mod, mode, loop, precision):
    lo, hi = np.full(3, -0.2), np.full(3, 0.2)
    st = _clusters(3, lo, hi)
    o = pu.oracle_sim(oracle_mod, st, 1e-5, lo, hi, 1, 0, mode=mode)
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0, mode=mode, precision=precision)
    g.set_skin(0.01)  # no rebuild after the first within a call
    g._L.rp_set_device_loop(g._h, loop)
    n0, tol = len(st["radius"]), 1e-5 if precision else 1e-9
    # a call's results are those of its last step. Coulomb friction lets two
    # roundings part, so the mixed form takes single steps, each from the same state
    for steps in [1] * 24 if precision else (3, 1, 5, 2, 7, 6):
        o.steps(steps)
        g.steps(steps)
        assert g.get_particle_count() == o.get_particle_count()
        so, sg = o.state(), g.get_state()
        FS, TS = o.last_force_scale()
        assert np.all(np.abs(sg["position"] - so["x"]).max(1) <= (1e-9 if precision else 1e-12))
        assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= tol * (FS / so["m"] + 10.0))
        assert np.all(np.abs(sg["torque"] - so["tau"]).max(1) <= tol * TS + 1e-25)
        if precision:
            o.set_state({"x": sg["position"], "v": sg["velocity"], "a": sg["acceleration"],
                         "w": sg["angular_velocity"], "tau": sg["torque"]})
    assert 20 < o.get_particle_count() < n0 - 100


@pytest.mark.parametrize("loop", [1, 0], ids=["device_loop", "host_loop"])
def test_partner_drops_out_of_the_grid_of_a_thin_bed(rp, oracle_mod, loop):
    # a periodic length below four cutoffs: the FP32 pretest is off and every
    # row entry a candidate. In each pair the lower sphere falls through the
    # open floor, where the reference's grid no longer lists it
    # (src/grid.rs:18-30), while the upper one keeps it in its row; clusters of
    # touching spheres in between leave their forces in the same buffers.
    rng = np.random.default_rng(8)
    lo, hi = np.array([0.0, 0.0, -0.45]), np.array([0.06, 0.5, 0.45])
    r, skin = 0.01, 4e-3
    x, v = [], []
    for k in range(24):
        z = -0.32 + 0.0275 * k
        up = np.array([0.03, 2 * r + skin + rng.uniform(2e-4, 4e-4), z])
        low = np.array([0.03, rng.uniform(2e-4, 6e-4), z + rng.uniform(-2e-3, 2e-3)])
        x += [up, low]
        v += [np.zeros(3), np.array([0.0, -3.0, 0.0])]
    for k in range(24):
        c = np.array([0.03, 0.2, -0.32 + 0.0275 * k])
        for d in ([0, 0, 0], [0.0, 0.0185, 0.0], [0.011, 0.009, 0.0]):
            x.append(c + d)
            v.append(rng.normal(0, 0.05, 3))
    x, v = np.array(x), np.array(v)
    st = _state(x, np.full(len(x), r), v, rng.normal(0, 1.0, (len(x), 3)))
    per = (True, False, False)
    o = pu.oracle_sim(oracle_mod, st, 1e-5, lo, hi, 1, 0, per)
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0, per)
    g.set_skin(skin)
    g._L.rp_set_device_loop(g._h, loop)
    crossed = False  # while the rows of the first step still stand
    for step in range(50):
        o.step()
        g.step()
        so, sg = o.state(), g.get_state()
        FS, _ = o.last_force_scale()
        assert np.all(np.abs(sg["position"] - so["x"]).max(1) <= 1e-12), step
        assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= 1e-9 * (FS / so["m"] + 10.0)), step
        crossed |= bool((so["x"][1:48:2, 1] < 0).any()) and g.stats()["neighbor_rebuilds"] == 1
    assert crossed and (so["x"][1:48:2, 1] < 0).all()


@pytest.mark.parametrize("change", ["removal", "insertion", "both"])
@pytest.mark.parametrize("tangential", [2, 1], ids=["mindlin", "linear_spring"])
def test_springs_survive_a_change_of_the_bed(rp, oracle_mod, tangential, change):
    # a sheared bed with loaded springs; between stepping calls some spheres
    # have left it (the slots are compacted) or join it (appended)
    lo, hi = (-0.25, -0.25, -0.25), (0.25, 0.25, 0.25)
    st = sheared_bed(71 + tangential, 1900, lo, hi)
    if change != "insertion":
        out = np.random.default_rng(2).choice(1900, 9, replace=False)
        st["position"][out] = np.stack([np.full(9, 1.2499), np.linspace(-0.2, 0.2, 9), np.linspace(-0.2, 0.2, 9)], 1)
        st["velocity"][out] = np.stack([np.linspace(0.3, 3.0, 9), np.zeros(9), np.zeros(9)], 1)  # one after the other
    dt = 1e-5
    o = pu.oracle_sim(oracle_mod, st, dt, lo, hi, 1, tangential, mode=1)
    g = pu.gpu_sim(rp, st, dt, lo, hi, 1, tangential, mode=1)
    g.set_skin(3e-5)  # rebuilds every few steps
    inserted = 0
    for call in range(12):
        o.steps(4)
        g.steps(4)
        assert g.get_particle_count() == o.get_particle_count()
        so, sg = o.state(), g.get_state()
        assert float(np.max(np.abs(sg["position"] - so["x"]))) <= 1e-12, call
        FS, TS = o.last_force_scale()
        To = so["tau"]
        assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= 1e-9 * (FS / so["m"] + 10.0)), call
        assert np.all(np.abs(sg["torque"] - To).max(1) <= 1e-9 * TS + 1e-25), call
        assert np.count_nonzero(np.linalg.norm(To, axis=1) > 1e-6 * TS) > 400  # loaded springs
        if change != "removal" and call % 4 == 1:
            p = np.array([[0.5, 0.1 * inserted, 0.0]])  # away from the bed
            g.add_particles(p, np.array([0.009]), np.array([0.008]))
            o.add_particle(p[0, 0], p[0, 1], p[0, 2], 0.009, 0.008)
            inserted += 1
    s = g.stats()
    assert s["state_uploads"] == 1
    if change != "insertion":
        assert s["compactions"] >= 2 and s["removed"] >= 5
    if change != "removal":
        assert s["device_inserts"] == inserted == 3


def test_diagnostics_of_a_call_that_removed_spheres(rp, oracle_mod):
    # forces and contact pairs of the last step in the ids of the spheres that
    # remain (removals are compacted when the call ends, which moves the slots)
    lo, hi = (-0.2, -0.2, -0.2), (0.2, 0.2, 0.2)
    st = pu.random_bed(53, 1500, lo, hi, 0.008, 0.012, ascale=0.0)
    out = np.arange(0, 1500, 50)
    st["position"][out, 0] = 1.19999
    st["velocity"][out, 0] = np.linspace(0.5, 3.0, len(out))
    o = pu.oracle_sim(oracle_mod, st, 1e-5, lo, hi, 1, 0)
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0)
    for steps in (2, 1, 1):
        n0 = o.get_particle_count()
        o.steps(steps)
        g.steps(steps)
        assert g.get_particle_count() == o.get_particle_count()
        Fo, To = o.last_forces()
        Fg, Tg = g.debug_forces()
        FS, TS = o.last_force_scale()
        assert len(Fg) == len(Fo)
        assert np.all(np.linalg.norm(Fg - Fo, axis=1) <= 1e-9 * FS)
        assert np.all(np.linalg.norm(Tg - To, axis=1) <= 1e-9 * TS + 1e-25)
        assert pu.pair_counter_gpu(g) == pu.pair_counter_oracle(o)
        assert o.get_particle_count() < n0 or steps == 1
    assert g.stats()["compactions"] >= 1


def test_spheres_that_have_flown_off_touch(rp, oracle_mod):
    # nothing is removed above the box: pairs from the box's top to 200 m above
    # it, turned every way, touching by 1e-6 to 1e-3 of a radius or just apart
    # (the pretest's margin is its own for pairs outside the box and one for all
    # inside, and both ends of a pair must take the same one)
    rng = np.random.default_rng(17)
    lo, hi = np.array([-0.2, -0.2, -0.2]), np.array([0.2, 0.2, 0.2])
    x, r = [], []
    for k in range(600):
        y = 10.0 ** rng.uniform(-1.2, 2.3) if k % 2 else rng.uniform(0.2, 0.45)
        c = np.array([0.05 * (k % 8) - 0.18, y, 0.05 * (k // 8 % 8) - 0.18])
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        ra = rng.uniform(0.008, 0.012, 2)
        gap = ra.sum() * (1.0 + rng.choice([-1, 1]) * 10.0 ** rng.uniform(-6, -3))
        x += [c, c + gap * u]
        r += list(ra)
    x, r = np.array(x), np.array(r)
    st = _state(x, r, rng.normal(0, 0.1, (len(x), 3)), rng.normal(0, 1.0, (len(x), 3)))
    o = pu.oracle_sim(oracle_mod, st, 1e-6, lo, hi, 1, 0, mode=1)
    g = pu.gpu_sim(rp, st, 1e-6, lo, hi, 1, 0, mode=1)
    for step in range(5):
        o.step()
        g.step()
        so, sg = o.state(), g.get_state()
        FS, TS = o.last_force_scale()
        assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= 1e-9 * (FS / so["m"] + 10.0)), step
        assert np.all(np.abs(sg["torque"] - so["tau"]).max(1) <= 1e-9 * TS + 1e-25), step
    assert pu.pair_counter_gpu(g) == pu.pair_counter_oracle(o)
    assert np.count_nonzero((FS > 0) & (so["x"][:, 1] > 1.0)) > 50


def test_sphere_far_away_slows_nobody(rp):
    lo, hi = (-0.6, -0.6, -0.6), (0.6, 0.6, 0.6)
    st = pu.random_bed(6, 300_000, lo, hi, 0.0085, 0.0088, vscale=0.05, ascale=0.0, tscale=0.0)
    took = []
    for far in (False, True):
        g = pu.gpu_sim(rp, st, 1e-6, lo, hi, 1, 0)
        g.set_debug(False)
        g.set_skin(0.009)  # rows of 18, six of them near
        if far:
            g.add_particle(0.0, 1e7, 0.0, 0.001, 1.0, True)
        g.steps(20)
        t = []
        for _ in range(7):
            a = g.stats()["device_ms"]
            g.steps(20)
            t.append(g.stats()["device_ms"] - a)
        took.append(sorted(t)[3])
    assert took[1] < 1.2 * took[0], took


@pytest.mark.parametrize("skin", [0.0, 0.03])
def test_sphere_written_whole_periods_away(rp, oracle_mod, skin):
    # positions written between calls that lie two box lengths off: the step
    # wraps them by one, so the spheres meet their neighbours as periodic images
    # in the middle of the box, although nothing has moved by the minimum image
    lo, hi = (-0.2, -0.2, -0.2), (0.2, 0.2, 0.2)
    st = pu.random_bed(19, 3000, lo, hi, 0.0125, 0.0135, vscale=0.05, ascale=0.0, tscale=0.0)
    per = (True, False, True)
    o = pu.oracle_sim(oracle_mod, st, 1e-6, lo, hi, 1, 0, per, mode=1)
    g = pu.gpu_sim(rp, st, 1e-6, lo, hi, 1, 0, per, mode=1)
    if skin:
        g.set_skin(skin)
    o.step()
    g.step()
    x = g.get_state()["position"]
    x[::7, 0] += 0.8
    x[3::7, 2] -= 0.8
    o.set_state({"x": x})
    g.set_state({"position": x})
    for step in range(3):
        o.step()
        g.step()
        so, sg = o.state(), g.get_state()
        FS, TS = o.last_force_scale()
        np.testing.assert_allclose(sg["position"], so["x"], rtol=0, atol=1e-12)
        assert np.all(np.abs(sg["acceleration"] - so["a"]).max(1) <= 1e-9 * (FS / so["m"] + 10.0)), step
    assert np.count_nonzero(FS[::7]) > 100
