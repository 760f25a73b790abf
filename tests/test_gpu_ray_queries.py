"""Ray queries: coincident colliders, the first query of a world, and a world in error.

Of colliders in one place the lowest is hit: a box that a ray enters behind the best hit so far is passed over, and the entry distance of
a collider's bounds can round above its own hit, so which of two coincident boxes is found
depends on which is met first.  The walk meets them in collider order, as the oracle does.
The table that names the hits is uploaded by a world's first query.  A query that ends in an
error leaves the caller's records as they were."""
import numpy as np
import pytest

from physecs_gb300 import scenes

pytestmark = pytest.mark.gpu


def _twins(n, seed):
    """n static boxes in n / 3 places, three to a place or so, of three sizes."""
    rng = np.random.default_rng(seed)
    he, pos = rng.uniform(0.3, 1.5, (n, 3)), rng.uniform(-4, 4, (n, 3))
    pos, he = pos[rng.integers(0, n // 3, n)], he[rng.integers(0, 3, n)]
    s = scenes.SceneData("twins")
    s.add_bodies(pos=pos, quat=[scenes.IDENTITY_Q] * n, flags=0, inv_mass=0.0, com=np.zeros(3), inv_inertia=np.zeros(9),
                 col_type=scenes.BOX, col_params=np.concatenate([he, np.zeros((n, 1))], 1))
    return s.finalize()


@pytest.mark.parametrize("n,seed", [(6, 0), (60, 1), (300, 2), (300, 3), (1500, 4)])
def test_coincident_boxes(n, seed, gpu_lib, oracle_lib):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World
    s = _twins(n, seed)
    rng = np.random.default_rng(seed + 100)
    rays = np.zeros((20000, 8), np.float32)
    o = rng.uniform(-4, 30, (len(rays), 3))
    o[:, 0] = rng.uniform(6, 30, len(rays))
    d = rng.uniform(-3, 3, o.shape) - o
    rays[:, 1:4], rays[:, 4:7], rays[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), 200.0
    w = World([s])
    g, want = w.raycast(rays), OracleScene(s).raycast(rays)
    hit = want["body"] >= 0
    assert hit.sum() > 1000
    assert np.array_equal(g["body"], want["body"])
    assert np.array_equal(g["distance"][hit].view(np.uint32), want["distance"][hit].view(np.uint32))
    w.close()


def _down(n, scene=0):
    rays = np.zeros((n, 8), np.float32)
    rays[:, 1] = 3.0 * np.arange(n)
    rays[:, 2], rays[:, 5], rays[:, 7] = 50.0, -1.0, 200.0
    rays.view(np.int32)[:, 0] = scene
    return rays


def test_first_query_of_a_world(gpu_lib):
    from physecs_gb300.api import World
    n = 20000
    s = scenes.SceneData("row")
    s.add_bodies(pos=np.stack([3.0 * np.arange(n), 0 * np.arange(n), 0 * np.arange(n)], 1), quat=[scenes.IDENTITY_Q] * n,
                 flags=0, inv_mass=0.0, com=np.zeros(3), inv_inertia=np.zeros(9), col_type=scenes.SPHERE,
                 col_params=[1.0, 0, 0, 0])
    s.finalize()
    s.arrays["entity"][:] = 7 * np.arange(n)[::-1]
    rays = _down(n)
    rays[:, 0] = 0
    for _ in range(5):
        w = World([s])
        h = w.raycast(rays)
        assert np.array_equal(h["body"], np.arange(n)) and (h["collider"] == 0).all()
        assert np.array_equal(h["entity"], s.arrays["entity"])
        w.close()


def test_error_leaves_the_records(gpu_lib):
    import ctypes as C
    from physecs_gb300.api import PsxError, World
    n = 60
    m, com, inertia = scenes.mass_sphere(0.5)
    s = scenes.SceneData("heap")
    s.add_bodies(pos=np.random.default_rng(0).uniform(-0.1, 0.1, (n, 3)), quat=[scenes.IDENTITY_Q] * n,
                 flags=scenes.BODY_DYNAMIC, inv_mass=1.0 / m, com=com, inv_inertia=np.linalg.inv(inertia).T.ravel(),
                 col_type=scenes.SPHERE, col_params=[0.5, 0, 0, 0])
    w = World([s.finalize()], pairs_per_collider=1)      # room for 1024 pairs, 1770 met
    w.step()
    with pytest.raises(PsxError, match="CAPACITY"):
        w.synchronize()
    rays, hits = _down(4), np.full((4, 7), 123.0, np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert gpu_lib.load().psx_world_raycast(w.h, 4, p(rays), None, p(hits)) == 3   # PSX_ERR_CAPACITY
    assert (hits == 123.0).all()
    w.close()
