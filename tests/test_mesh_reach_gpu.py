"""GPU: the mesh pass's distance test ahead of the collision predicate changes no
hit: events and candidates as the oracle's with slow and fast bodies, one very fast
body, long, zero and backward timesteps."""
import numpy as np
import pytest

import oracle
from conftest import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [1e-3, 0.05, 0.0, -1e-3])
@pytest.mark.parametrize("speed,fast", [(0.0, 0.0), (1e-3, 0.0), (0.5, 0.0), (1e-3, 40.0)])
def test_same_events(lib, dt, speed, fast):
    from ncorpion_b200 import api
    n, cells, gam = 3000, 32, 0.05
    rng = np.random.default_rng(7)
    b = np.zeros((n, 8))
    b[:, :3] = rng.uniform(-0.6, 0.6, (n, 3))
    b[:, 3:6] = rng.normal(0, 1, (n, 3)) * speed
    b[17, 3:6] += fast
    b[:, 6] = 10.0 ** rng.uniform(-9, -7, n)
    b[:, 7] = rng.uniform(2e-3, 2.4e-2, n)
    ex = np.ones(n, np.int32)
    ex[::29] = 0
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    kw = dict(collision_bool=1, collision_type=1, collision_parameter=1.5, brute_force_bool=0, mesh_bool=1,
              collision_cube_cells=cells, collision_cube_min=gam * cells)
    api.init(n, make_params(**kw))
    api.upload(b, ex, cm)
    api.set_timestep(dt)
    n_pairs, n_events, tn = api.mesh(gam, True)
    w = oracle.PortWorld(n, make_params(**kw))
    w.set_state(b, ex, cm, dt=dt, gam=gam)
    w.lib.orc_w_mesh()
    assert np.array_equal(api.events(), w.events())
    assert np.array_equal(api.pairs(), w.pairs())
    bg, exg, _ = api.download(n)
    b_ref, ex_ref, _ = w.get_state()
    assert np.array_equal(exg, ex_ref) and np.array_equal(bg[exg == 1], b_ref[ex_ref == 1])
    api.finalize()


@pytest.mark.parametrize("spread", [0.02, 0.045, 0.09, 0.3])
def test_candidate_lists(lib, spread):
    """From hundreds of candidates a body (walked again, several rounds) over a few
    past a queue's 32 to a few each: pairs[] in order, as the oracle's."""
    from ncorpion_b200 import api
    n, cells, gam = 900, 32, 0.05
    rng = np.random.default_rng(3)
    b = np.zeros((n, 8))
    b[:, :3] = rng.normal(0, spread, (n, 3))
    b[:, 3:6] = rng.normal(0, 1e-2, (n, 3))
    b[:, 6] = 1e-9
    b[:, 7] = 1e-4
    ex = np.ones(n, np.int32)
    ex[::31] = 0
    cm = np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])
    kw = dict(collision_bool=1, collision_type=1, collision_parameter=1.5, brute_force_bool=0, mesh_bool=1,
              collision_cube_cells=cells, collision_cube_min=gam * cells, how_many_neighbours=400.0)
    api.init(n, make_params(**kw))
    api.upload(b, ex, cm)
    api.set_timestep(1e-3)
    api.mesh(gam, True)
    w = oracle.PortWorld(n, make_params(**kw))
    w.set_state(b, ex, cm, dt=1e-3, gam=gam)
    w.lib.orc_w_mesh()
    assert np.array_equal(api.pairs(), w.pairs()) and np.array_equal(api.events(), w.events())
    api.finalize()
