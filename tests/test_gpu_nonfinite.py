"""Infinities and NaN in a bed: they reach what the reference's operations let them reach, and nothing else.

A fixed sphere is not integrated, so whatever velocity and spin it is given
enters its contacts as it is. The spheres that touch it turn out as the oracle's
(finite, infinite or NaN component by component), their neighbours stay as they are.
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


NEG_NAN = np.copysign(np.nan, -1.0)
ODD = [np.inf, -np.inf, np.nan, NEG_NAN]
# finite, but their squares are not. At a wall only: in a pair the reference's
# |F_n| overflows where the magnitude formed here stays finite
HUGE = [1e200, -1e160, 1e308]


def _kind(x):
    return np.where(np.isnan(x), 2, np.where(np.isinf(x), 1, 0))


def _pairs():
    """A fixed sphere with one odd velocity or spin component beside a free one, every kind of value, several
    directions; and pairs without any."""
    rng = np.random.default_rng(12)
    x, v, w, fixed = [], [], [], []
    k = 0
    for val in ODD + [0.0]:
        for comp in range(6):
            for rep in range(3):
                c = np.array([k % 8, k // 8 % 8, k // 64]) * 0.1 - 0.35
                u = rng.normal(size=3)
                u /= np.linalg.norm(u)
                if rep == 0:
                    u = np.eye(3)[comp % 3]
                x += [c, c + 0.0195 * u]
                q = np.zeros(6)
                q[comp] = val
                v += [q[:3], rng.normal(0, 0.3, 3)]
                w += [q[3:], rng.normal(0, 1.0, 3)]
                fixed += [1, 0]
                k += 1
    n = len(x)
    r = np.full(n, 0.01)
    return {"position": np.array(x), "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3,
            "velocity": np.array(v), "angular_velocity": np.array(w), "acceleration": np.zeros((n, 3)),
            "torque": np.zeros((n, 3)), "fixed": np.array(fixed, np.uint8)}


@pytest.mark.parametrize("path", [0, 1], ids=["contacts", "particles"])
@pytest.mark.parametrize("normal", [0, 1, 2, 4])
def test_odd_velocities_of_a_fixed_sphere(rp, oracle_mod, normal, path):
    st = _pairs()
    lo, hi = (-0.6,) * 3, (0.6,) * 3
    mat = (1e7, 0.3, 2500.0, 0.5, 0.5, 0.05 if normal == 4 else 0.0)
    o = pu.oracle_sim(oracle_mod, st, 1e-7, lo, hi, normal, 0, material=mat)
    g = pu.gpu_sim(rp, st, 1e-7, lo, hi, normal, 0, material=mat, force_path=path)
    o.step()
    g.step()
    so, sg = o.state(), g.get_state()
    odd = ~np.isfinite(so["a"]).all(1)
    assert odd[1::2][:18].all() or normal == 2
    assert g.stats()["status_bits"] & 2
    for k, q in (("acceleration", "a"), ("torque", "tau"), ("velocity", "v"), ("angular_velocity", "w")):
        np.testing.assert_array_equal(_kind(sg[k]), _kind(so[q]), err_msg=k)
    assert np.isfinite(sg["acceleration"][-36:]).all()


def test_odd_velocities_at_a_wall(rp, oracle_mod):
    # spheres with odd spins on a floor: the wall law's comparisons
    n = len(ODD + HUGE) * 3
    x = np.stack([-0.3 + 0.025 * np.arange(n), np.full(n, 0.0095), np.zeros(n)], 1)
    w = np.zeros((n, 3))
    w[np.arange(n), np.arange(n) % 3] = np.repeat(ODD + HUGE, 3)
    r = np.full(n, 0.01)
    st = {"position": x, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3, "velocity": np.zeros((n, 3)),
          "angular_velocity": w, "acceleration": np.zeros((n, 3)), "torque": np.zeros((n, 3)),
          "fixed": np.zeros(n, np.uint8)}
    tri = np.array([[-1, 0, -1, -1, 0, 1, 1, 0, -1], [1, 0, -1, -1, 0, 1, 1, 0, 1]], float)
    nrm = np.tile([0.0, 1.0, 0.0], (2, 1))
    lo, hi = (-0.6,) * 3, (0.6,) * 3
    o = pu.oracle_sim(oracle_mod, st, 1e-7, lo, hi, 1, 0, tris=(tri, nrm))
    g = pu.gpu_sim(rp, st, 1e-7, lo, hi, 1, 0, tris=(tri, nrm))
    o.step()
    g.step()
    so, sg = o.state(), g.get_state()
    for k, q in (("acceleration", "a"), ("torque", "tau"), ("velocity", "v")):
        np.testing.assert_array_equal(_kind(sg[k]), _kind(so[q]), err_msg=k)


@pytest.mark.parametrize("steps", [1, 4])
@pytest.mark.parametrize("n,normal", [(40, 1), (9000, 1), (300, 3)], ids=["quads", "scalar", "kernels"])
def test_infinite_spins_in_flight(rp, oracle_mod, n, normal, steps):
    # spheres that touch nothing: kicked by no torque, an infinite spin turns
    # into NaN by its compensated sum; set before the first step and in between
    m = int(np.ceil(n ** (1 / 3)))
    g3 = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    rng = np.random.default_rng(n)
    w = rng.normal(0, 1.0, (n, 3))
    w[::5, 0], w[1::5, 1], w[2::5, 2] = np.inf, -np.inf, np.nan
    r = np.full(n, 0.005)
    st = {"position": g3 * 0.02 - 0.25, "radius": r, "mass": 2500.0 * 4.0 / 3.0 * np.pi * r ** 3,
          "velocity": rng.normal(0, 0.1, (n, 3)), "angular_velocity": w, "acceleration": np.zeros((n, 3)),
          "torque": np.zeros((n, 3)), "fixed": np.zeros(n, np.uint8)}
    lo, hi = (-0.6,) * 3, (0.6,) * 3
    for late in (False, True):
        first = dict(st, angular_velocity=np.zeros((n, 3))) if late else st
        o = pu.oracle_sim(oracle_mod, first, 1e-7, lo, hi, normal, 0)
        g = pu.gpu_sim(rp, first, 1e-7, lo, hi, normal, 0)
        g.set_debug(False)
        if late:
            o.step()
            g.step()
            o.set_state({"w": w})
            g.set_state({"angular_velocity": w})
        o.steps(steps)
        g.steps(steps)
        so, sg = o.state(), g.get_state()
        for k, q in (("angular_velocity", "w"), ("angular_velocity_residual", "wres"), ("velocity", "v")):
            np.testing.assert_array_equal(sg[k], so[q], err_msg=k)
