"""The broadphase walk at the sizes where its forms change (few leaves are tested without
the tree, large leaves walk alone, scattered lanes walk alone): the same contacts as the
oracle's, and the same order of contacts wherever the scene lies in its world."""
import os
import sys

import numpy as np
import pytest

from tests.parity import gpu_keys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from scene_variants import character_scene  # noqa: E402

pytestmark = pytest.mark.gpu


def _scene(kind, n):
    from physecs_gb300 import scenes
    if kind == "tower":        # balls between walls, a ramp and a ground, each much larger than a ball
        return character_scene(n_chars=1, n_balls=n - 5)[0]
    s = scenes.batch_scene(21, n_bodies=n - 1)
    if kind == "scattered":    # a few neighbours here and there in a wide volume
        rng = np.random.default_rng(5)
        at = rng.uniform(-200, 200, ((n - 1 + 3) // 4, 3)) + [0, 300, 0]
        s.arrays["pos"][1:n] = (at.repeat(4, 0)[: n - 1] + rng.uniform(-0.4, 0.4, (n - 1, 3))).astype(np.float32)
    return s


@pytest.mark.parametrize("n", [2, 33, 513, 514, 640, 1500])
@pytest.mark.parametrize("kind", ["mixed", "tower", "scattered"])
def test_pairs_of_the_walk(gpu_lib, oracle_lib, kind, n):
    from oracle.port_api import OracleScene
    from physecs_gb300 import scenes
    from physecs_gb300.api import World
    if kind == "tower" and n < 8:
        pytest.skip("the walls alone are more")
    s = _scene(kind, n)
    alone, second = World([s]), World([scenes.batch_scene(3, n_bodies=20), s])
    o = OracleScene(s)
    met = 0
    for f in range(25 if kind == "mixed" and n == 33 else 3):
        alone.step()
        second.step()
        ids, _, meta = alone.contacts()
        ids2, _, meta2 = second.contacts()
        sel = ids2[:, 0] == 1
        assert np.array_equal(gpu_keys(ids, meta), gpu_keys(ids2[sel], meta2[sel])), f
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0, f
        st, so = alone.read_bodies(), o.state()
        for k in so:
            assert np.array_equal(st[k].view(np.uint32), so[k].view(np.uint32)), (f, k)
        met += len(ids)
    assert met or n == 2
    assert alone.counts()["error"] == 0 and second.counts()["error"] == 0
