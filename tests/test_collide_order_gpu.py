"""GPU: the brute-force sweep's hits put in order by the event kernel itself (up to
4,096 slots: in shared memory to 2,048 hits, by rows past that) and by the host's
sort (past it), at the sweep's tile edges: events and states as the oracle's, bit
for bit (merged radii within 1 ulp, as in test_collide_gpu.py).  More hits than the
list holds end a step before it drifts."""
import numpy as np
import pytest

import oracle
from conftest import make_params
from test_collide_gpu import assert_state_equal

pytestmark = pytest.mark.gpu


def cluster(n, spread, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros((n, 8))
    b[:, :3] = [1.0, 0.0, 0.0] + rng.normal(0, spread, (n, 3))
    b[:, 3:6] = rng.normal(0, 1e-2, (n, 3))
    b[:, 4] += 1.0
    b[:, 6] = 10.0 ** rng.uniform(-9, -7, n)
    b[:, 7] = rng.uniform(5e-4, 2e-3, n)
    ex = np.ones(n, np.int32)
    ex[::13] = 0
    return b, ex, np.array([0, 0, 0, 0, 0, 0, 1.0, 1.0])


# (slots, spread): no hit; a few; tile edges; past 2,048 hits; past 4,096 slots
# (host's sort, 32 bodies j a CTA); thousands of hits, in every row
@pytest.mark.parametrize("n,spread", [(2, 1.0), (33, 2e-2), (128, 2e-2), (129, 1e-2), (161, 1e-2), (220, 6e-4),
                                      (4096, 6e-2), (4097, 6e-2), (4096, 1e-2)])
@pytest.mark.parametrize("ctype", [1, 2])
def test_sweep(lib, n, spread, ctype):
    from ncorpion_b200 import api
    if ctype == 2 and spread < 1e-3:
        pytest.skip("mergers leave few hits to order")
    if ctype == 1 and (n, spread) == (4096, 1e-2):
        pytest.skip("thousands of rebounds in a row take seconds; the mergers have the same hits to order")
    b, ex, cm = cluster(n, spread, n)
    kw = dict(collision_bool=1, collision_type=ctype, collision_parameter=1.5, one_collision_only_bool=int(spread < 1e-3))
    api.init(max(n, 64), make_params(**kw))
    api.upload(b, ex, cm)
    api.set_timestep(1e-3)
    w = oracle.PortWorld(max(n, 64), make_params(**kw))
    w.set_state(b, ex, cm, dt=1e-3)
    ev = []
    for _ in range(2):  # the second sweep meets the first one's marks cleared
        api.collide_brute()
        w.lib.orc_w_brute_force()
        ev.append(api.events())
        assert np.array_equal(np.concatenate(ev), w.events())  # (the oracle's log goes on)
    bg, exg, _ = api.download(max(n, 64))
    b_ref, ex_ref, _ = w.get_state()
    assert_state_equal(bg, exg, b_ref, ex_ref)
    api.finalize()


def test_step_ends_before_the_drift_when_the_hits_do_not_fit(lib):
    """1,800 bodies inside one another, half of the pairs approaching: 0.8 million hits, more than the 2^19
    that the list holds.  As with an error of a sweep by itself, nothing is resolved and nothing moves."""
    from ncorpion_b200 import api
    b, ex, cm = cluster(1800, 1e-5, 3)
    ex[:] = 1
    b[:, 6], b[:, 7] = 1e-20, 2e-3
    api.init(2048, make_params(collision_bool=1, collision_type=1, collision_parameter=1.5, reduce_to_COM_bool=0))
    api.upload(b, ex, cm)
    api.set_timestep(1e-3)
    with pytest.raises(api.NcgpuError) as e:
        api.step_brute_force()
    assert e.value.status == api.E_CAPACITY
    b1, ex1, _ = api.download(2048)
    assert np.array_equal(ex1, ex) and np.array_equal(b1[:, :3], b[:, :3])
    assert not np.array_equal(b1[:, 3:6], b[:, 3:6])
    api.finalize()
