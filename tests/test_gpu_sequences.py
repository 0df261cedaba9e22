"""Random sequences of calls on one simulation: steps, state written and restored, spheres added and thrown out, settings.

Two simulations go through the same calls, one with the device loop and one with
the host-issued loop: the same bits after every action. In FP64, beds without
springs take one more step from their present state beside the oracle: the same
positions bit for bit, accelerations to 1e-9 of a sphere's sum of contact-force
magnitudes (1e-6 under the certified JKR solver).
"""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from tests import parity_util as pu

pytestmark = pytest.mark.gpu

ACTIONS = ["steps", "steps", "one", "shift", "velocity", "insert", "setting", "throw", "getter", "restore"]


@pytest.fixture(scope="module")
def rp():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import rusty_particles_gb300 as m
    return m


def _pick(rng, k, share):
    return rng.choice(k, max(1, k // share), replace=False)


class Bed:
    """A bed drawn at random and what was drawn."""

    def __init__(self, seed):
        rng = self.rng = np.random.default_rng(seed)
        self.rm = rm = 0.01
        n = int(np.exp(rng.uniform(np.log(5), np.log(4000))))
        self.normal, self.tangential, self.mode = int(rng.integers(0, 5)), int(rng.integers(0, 3)), int(rng.integers(0, 2))
        self.precision = int(rng.integers(0, 4) == 0)
        gamma = float(rng.choice([0.05, 0.5])) if self.normal >= 3 else 0.0
        self.solver = str(rng.choice(["newton", "certified"])) if self.normal == 3 else "newton"
        L = np.full(3, np.ceil(n ** (1 / 3)) * 2.0 * rm) * rng.uniform(0.85, 1.2, 3)
        if rng.integers(0, 5) == 0:  # a thin bed: the FP32 pretest is off where it is periodic
            L[rng.integers(0, 3)] = rm * rng.uniform(3, 7)
        self.L, self.lo, self.hi = L, -L / 2, L / 2
        self.periodic = tuple(bool(b) for b in rng.integers(0, 2, 3))
        x = self.place(n)
        for _ in range(40):
            pairs = cKDTree(x).query_pairs(0.3 * rm)
            for _, b in pairs:
                x[b] = self.place(1)[0]
        r = rng.uniform(0.7, 1.0, n) * rm
        self.state = {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3,
                      "velocity": rng.normal(0, float(rng.choice([0.1, 3.0, 50.0])), (n, 3)),
                      "angular_velocity": rng.normal(0, 1, (n, 3)), "acceleration": np.zeros((n, 3)),
                      "torque": np.zeros((n, 3)), "fixed": (rng.uniform(0, 1, n) < rng.choice([0, 0.2])).astype(np.uint8)}
        self.cell, self.skin = float(rng.choice([1.0, 2.2 * rm, 5 * rm])), float(rm * rng.choice([0.02, 0.2, 1.0]))
        self.capacity, self.material = int(rng.choice([0, 5, 40])), (1e5, 0.3, 2500.0, 0.5, 0.5, gamma)
        self.tris = self.motion = None
        if rng.integers(0, 3):
            T = int(rng.integers(1, 200))
            v = (self.place(T)[:, None] + rng.normal(0, rm * float(rng.choice([0.3, 2.0, 20.0])), (T, 3, 3)))
            v = v.reshape(T, 9).astype(np.float32).astype(float)
            q = v.reshape(-1, 3, 3)
            nrm = np.cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0])
            nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-30)
            self.tris = (v, nrm.astype(np.float32).astype(float))
            self.motion = (np.zeros(3), rng.normal(0, 5, 3), rng.normal(0, 1, 3)) if rng.integers(0, 2) else None

    def place(self, k):
        return self.lo + self.rng.uniform(0, 1, (k, 3)) * self.L

    def gpu(self, rp, loop):
        g = pu.gpu_sim(rp, self.state, 1e-6, self.lo, self.hi, self.normal, self.tangential, self.periodic, self.mode,
                       self.material, cell=self.cell, precision=self.precision)
        g.set_debug(False)
        g.set_skin(self.skin)
        g.set_jkr_solver(self.solver)
        if self.capacity:
            g.set_neighbor_capacity(self.capacity)
        if self.tris is not None:
            g.add_triangles(*self.tris, motion=self.motion)
        g._L.rp_set_device_loop(g._h, loop)
        return g

    def oracle(self, oracle_mod, state):
        o = pu.oracle_sim(oracle_mod, state, 1e-6, self.lo, self.hi, self.normal, self.tangential, self.periodic, self.mode,
                          self.material, cell=self.cell)
        if self.tris is not None:
            o.add_triangles(*self.tris, motion=self.motion)
        o.set_state({"xres": state["position_residual"], "vres": state["velocity_residual"],
                     "wres": state["angular_velocity_residual"]})
        return o

    def act(self, what, sims, a):
        rng, k = self.rng, len(a["mass"])
        if what == "steps":
            q = int(rng.integers(1, 60))
            return [g.steps(q) for g in sims]
        if what == "insert":
            c = int(rng.integers(1, 9))
            x, r = self.place(c), np.minimum(rng.uniform(0.7, 0.99, c) * self.rm, a["radius"].max(initial=0.007))
            return [g.add_particles(x, r, 2500.0 * 4.0 / 3.0 * np.pi * r ** 3) for g in sims]
        if what == "setting":
            s = float(self.rm * rng.choice([0.02, 0.2, 1.0]))
            return [g.set_skin(s) for g in sims]
        if k == 0 or what == "one":
            return None
        if what == "restore":
            return [g.set_state(a) for g in sims]
        if what == "getter":
            i = int(rng.integers(0, k))
            return [(g.get_particle_position(i), g.set_particle_velocity(i, 1.0, 2.0, 3.0)) for g in sims]
        if what == "velocity":
            w = {"velocity": a["velocity"] * float(rng.uniform(-1, 1.5)), "angular_velocity": -a["angular_velocity"]}
            return [g.set_state(w) for g in sims]
        ax, x, v = int(rng.integers(0, 3)), a["position"].copy(), a["velocity"].copy()
        if what == "shift":  # whole periods on a periodic axis
            x[_pick(rng, k, 10), ax] += rng.choice([-2, -1, 1, 2, 0.001]) * (self.L[ax] if self.periodic[ax] else 0.3 * self.rm)
            return [g.set_state({"position": x}) for g in sims]
        idx = _pick(rng, k, 20)  # thrown out: at the removal bound
        x[idx, ax] = self.hi[ax] + 1.0 + rng.uniform(-1e-4, 1e-4, len(idx))
        v[idx, ax] = 20.0
        return [g.set_state({"position": x, "velocity": v}) for g in sims]


@pytest.mark.parametrize("first", range(0, 120, 20))
def test_random_calls(rp, oracle_mod, first):
    compared = 0
    for seed in range(first, first + 20):
        bed = Bed(seed)
        springs = bed.mode == 1 and bed.tangential != 0
        sims = [bed.gpu(rp, loop) for loop in (1, 0)]
        done = []
        for _ in range(10):
            what = str(bed.rng.choice(ACTIONS))
            done.append(what)
            bed.act(what, sims, sims[0].get_state())
            before = sims[0].get_state()
            if len(before["mass"]) == 0:
                break
            for g in sims:
                g.step()
            a, b = (g.get_state() for g in sims)
            for key in a:
                np.testing.assert_array_equal(a[key], b[key], err_msg=f"{key}: seed {seed} after {done}")
            if bed.precision or springs or not np.isfinite(before["velocity"]).all():
                continue
            o = bed.oracle(oracle_mod, before)
            o.step()
            so = o.state()
            assert len(so["m"]) == len(a["mass"]), (seed, done)
            if len(so["m"]) == 0:
                break
            np.testing.assert_array_equal(a["position"], so["x"], err_msg=f"seed {seed} after {done}")
            FS, _ = o.last_force_scale()
            ok = np.isfinite(so["a"]).all(1)
            if cKDTree(so["x"]).query_pairs(1.1e-6):
                continue  # such pairs take +Y as their normal from either end in the reference
            tol = 1e-6 if bed.solver == "certified" else 1e-9
            assert np.all(np.abs(a["acceleration"] - so["a"]).max(1)[ok] <= tol * (FS / so["m"] + 10.0)[ok]), (seed, done)
            compared += 1
    assert compared > 40
