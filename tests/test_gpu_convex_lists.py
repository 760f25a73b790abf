"""Pairs in worlds of few and many: how a warp takes its pairs in GJK, in the convex contact
pass and in the one-box routines depends on their number in the world, the result of a scene
does not.  One scene alone equals the oracle (lockstep); every copy of it in a larger world
equals it."""
import numpy as np
import pytest

from tests.parity import gpu_keys

pytestmark = pytest.mark.gpu

FRAMES = 30


@pytest.fixture(scope="module")
def alone(gpu_lib, oracle_lib):
    from oracle.port_api import OracleScene
    from physecs_gb300 import scenes
    from physecs_gb300.api import World
    s = scenes.batch_scene(31, n_bodies=70, chain_prob=0.0)
    w, o = World([s]), OracleScene(s)
    for f in range(FRAMES):
        w.step()
        ids, _, meta = w.contacts()
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0, f
    st, so = w.read_bodies(), o.state()
    for k in so:
        assert np.array_equal(st[k].view(np.uint32), so[k].view(np.uint32)), k
    assert len(ids) > 20 and w.counts()["error"] == 0
    return s, st


@pytest.mark.parametrize("copies", [2, 40, 400, 3000, 8000])
def test_copies_equal_the_scene_alone(alone, copies):
    from physecs_gb300.api import World
    s, want = alone
    w = World([s] * copies)
    for _ in range(FRAMES):
        w.step()
    got = w.read_bodies()
    for k in want:
        a = got[k].reshape((copies,) + want[k].shape)
        assert (a.view(np.uint32) == want[k].view(np.uint32)[None]).all(), k
    assert w.counts()["error"] == 0
    w.close()
