"""MTD queries and character controllers by warps (up to 4096 a call) and by threads
(above): the same call in one piece and in pieces gives the same bytes."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from scene_variants import character_moves, character_scene  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reach", [0.5, 8.0])   # a few colliders a query; more than a warp holds at a time
def test_mtd_queries_in_one_call_and_in_pieces(gpu_lib, reach):
    from physecs_gb300 import scenes
    from physecs_gb300.api import World
    rng = np.random.default_rng(7)
    few = [scenes.large_mixed(n_bodies=64, cells=16)] if reach < 1 else []   # a mesh: a wide shape meets too many triangles
    w = World([scenes.batch_scene(11, n_bodies=120), character_scene(n_balls=80)[0]] + few)
    n = 4500
    qs = []
    for i in range(n):
        q = rng.normal(size=4)
        qs.append({"scene": i % (2 + len(few)), "pos": rng.uniform(-4, 4, 3) + [0, 2, 0], "quat": (q / np.linalg.norm(q)).astype(np.float32),
                   "type": (scenes.SPHERE, scenes.CAPSULE, scenes.BOX)[i // 3 % 3], "params": reach * rng.uniform(0.3, 1, 3)})
    counts, hits = w.overlap_mtd(qs, cap=48)
    lo = 0
    for m in (1, 2, 31, 370, 4096):
        c, h = w.overlap_mtd(qs[lo:lo + m], cap=48)
        assert np.array_equal(c, counts[lo:lo + m])
        for k in range(m):
            a, b = h[k], hits[lo + k]
            assert [x[:3] for x in a] == [x[:3] for x in b]
            assert np.array_equal(np.array([[*x[3], x[4]] for x in a], np.float32).view(np.uint32),
                                  np.array([[*x[3], x[4]] for x in b], np.float32).view(np.uint32))
        lo += m
    assert lo == n and counts.max() > (32 if reach > 1 else 1)


def test_controllers_in_one_call_and_in_pieces(gpu_lib):
    from physecs_gb300.api import World
    per, count = 60, 70
    s, chars = character_scene(n_chars=per)
    specs = [{"scene": i, "body": b, "height": 1.0, "radius": 0.3} for i in range(count) for b in chars]
    moves = character_moves(len(specs), 3)
    runs = []
    for pieces in ([count], [1, 2, 40, 27]):   # whole scenes: the controllers of one scene see each other
        w = World([s] * count)
        out = []
        for f in range(3):
            lo = 0
            for m in pieces:
                out.append(w.move_characters(specs[lo:lo + m * per], moves[f][lo:lo + m * per]))
                lo += m * per
            assert lo == per * count
            w.step()
        runs.append((np.concatenate(out), w.read_bodies()))
        assert w.counts()["error"] == 0
        w.close()
    assert np.array_equal(runs[0][0], runs[1][0]) and runs[0][0].any()
    for k in runs[0][1]:
        assert np.array_equal(runs[0][1][k].view(np.uint32), runs[1][1][k].view(np.uint32)), k
