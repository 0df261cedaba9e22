"""Settings changed between stepping calls keep the state that the device holds."""
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


SETTINGS = {
    "debug": lambda g: g.set_debug(False),
    "gravity": lambda g: g.set_gravity(0.0, -9.81, 0.0),
    "material": lambda g: g.set_particle_material(1e7, 0.3, 2500.0, 0.5, 0.5, 0.0),
    "models": lambda g: g.set_contact_models("hertz", "coulomb"),
    "periodic": lambda g: g.set_periodic_boundary(False, False, False),
    "skin": lambda g: g.set_skin(2e-3),
    "capacity": lambda g: g.set_neighbor_capacity(48),
    "mode": lambda g: g.set_interaction_mode("parity"),
    "precision": lambda g: g.set_precision("fp64"),
    "solver": lambda g: g.set_jkr_solver("certified"),
    "wall_material": lambda g: g.set_wall_material(1e8, 0.3, 7800.0, 0.3, 0.6),
    "group_material": lambda g: g.set_group_material(3, 1e7, 0.3, 2500.0, 0.5, 0.5, 0.0),
    "triangles": lambda g: g.add_triangles(np.array([[5, 5, 5, 6, 5, 5, 5, 6, 5]], np.float32)),
    "launch_shape": lambda g: g.set_launch_shape(128, 128, 128, 0),
}


@pytest.mark.parametrize("what", sorted(SETTINGS))
def test_setting_between_calls_keeps_the_state(rp, oracle_mod, what):
    lo, hi = (-0.1, -0.1, -0.1), (0.1, 0.1, 0.1)
    st = pu.random_bed(5, 300, lo, hi, 0.008, 0.012, vscale=0.5)
    o = pu.oracle_sim(oracle_mod, st, 1e-5, lo, hi, 1, 0)
    g = pu.gpu_sim(rp, st, 1e-5, lo, hi, 1, 0)
    g.set_gravity(0.0, -9.81, 0.0)
    o.steps(7)
    g.steps(7)
    before = g.get_state()
    SETTINGS[what](g)
    after = g.get_state()
    for k in before:
        np.testing.assert_array_equal(after[k], before[k], err_msg=k)
    o.steps(5)
    g.steps(5)
    assert float(np.max(np.abs(g.get_state()["position"] - o.state()["x"]))) <= 1e-12
