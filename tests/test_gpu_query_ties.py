"""Rays against colliders that lie in one place: the lowest collider of equal hits.

A box that a ray enters behind the best hit so far is passed over, and the entry distance of
a collider's bounds can round above its own hit, so which of two coincident boxes is found
depends on which is met first.  The walk meets them in collider order, as the oracle does."""
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
