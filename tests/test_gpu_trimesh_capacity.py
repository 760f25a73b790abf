"""Body-mesh pairs at the lists' ends, against the oracle.

A body whose bounds cover more than 48 triangles (what a lane keeps) while it touches a few
is walked again by its warp; on a flat mesh, a flat box over sixteen triangles has as many
manifolds as a pair has room for and a wider one more.  The first must give the oracle's frames without an error, in every frame, alone and among bodies that
meet few triangles; the last must report the triangle capacity and nothing else.
Tolerance: 1e-5, the parity bar of a frame from identical state."""
import numpy as np
import pytest

from physecs_gb300 import scenes
from tests.parity import gpu_keys, rel_state_diff

pytestmark = pytest.mark.gpu

KEPT, MANIFOLDS, TRI_CAPACITY = 48, 16, 8


def _turn(axis, degrees):
    a = np.asarray(axis, float) / np.linalg.norm(axis)
    h = np.radians(degrees) / 2
    return list(a * np.sin(h)) + [np.cos(h)]


# kind: (shape, parameters, orientation, height above the mesh)
WIDE = {"sphere": (scenes.SPHERE, [1.5, 0, 0, 0], _turn([0.3, 0, 1], 25), 1.49),
        "capsule": (scenes.CAPSULE, [1.5, 0.2, 0, 0], _turn([0.2, 0, 1], 65), 0.82),
        "box": (scenes.BOX, [1.0, 0.2, 1.0, 0], _turn([1, 0.2, 0.7], 35), 0.94),
        "hull": (scenes.CONVEX_MESH, [1.0, 1.0, 1.0, 0], _turn([1, 0.2, 1], 30), 0.95)}
SMALL = (scenes.SPHERE, [0.2, 0, 0, 0], scenes.IDENTITY_Q, 0.185)


def _scene(bodies, cells, cell, rough=0.0):
    """Bodies (shape, parameters, orientation, position) above a mesh of cells x cells, flat or
    a little rough (on a flat one every contact ties in distance, and the order of ties is
    free; so is it among more than sixteen contacts, hence the box on its corner)."""
    s = scenes.SceneData("flat")
    g = np.arange(cells + 1) * cell - cells * cell / 2
    y = np.random.default_rng(2).uniform(-rough, 0, (cells + 1) ** 2)
    verts = np.stack([np.repeat(g, cells + 1), y, np.tile(g, cells + 1)], 1)
    i = np.arange(cells)[:, None] * (cells + 1) + np.arange(cells)[None]
    tri = np.stack([np.stack([i, i + 1, i + cells + 2], -1), np.stack([i, i + cells + 2, i + cells + 1], -1)], 2)
    s.trimesh.append((verts, tri.reshape(-1).astype(np.uint32)))
    s.add_bodies(pos=[[0.0, 0.0, 0.0]], quat=[scenes.IDENTITY_Q], flags=0, inv_mass=0.0, com=np.zeros(3),
                 inv_inertia=np.zeros(9), col_type=scenes.TRIANGLE_MESH, col_params=[0.0] * 4, col_mesh=0)
    s.convex.extend(scenes._hull_pool(scenes.SplitMix64(5), count=1))
    for shape, params, quat, pos in bodies:
        s.add_bodies(pos=[pos], quat=[quat], flags=scenes.BODY_DYNAMIC, inv_mass=1.0, com=np.zeros(3),
                     inv_inertia=np.eye(3).ravel() / 0.3, col_type=shape, col_params=params,
                     col_mesh=0 if shape == scenes.CONVEX_MESH else -1, vel=[[0.3, -1.0, 0.2]])
    s.finalize()
    corners = verts[tri.reshape(-1, 3)]
    return s, corners.min(1), corners.max(1)


def _met(o, lo, hi, body, margin=0.011):
    """Triangles whose bounds meet a body's, both without the body's margin."""
    ids, b = o.bounds()
    mn, mx = b[ids[:, 0] == body][0, :3] + margin, b[ids[:, 0] == body][0, 3:] - margin
    return int(((lo <= mx) & (hi >= mn)).all(1).sum())


def _lockstep(s, lo, hi, wide, frames=5):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World
    g, o = World([s]), OracleScene(s)
    touched, most = set(), dict.fromkeys(wide, 0)
    for frame in range(frames):
        most = {b: max(most[b], _met(o, lo, hi, b)) for b in wide}
        g.step()
        assert g.counts()["error"] == 0
        ids, _, meta = g.contacts()
        assert (meta[:, 1] >= 0).all()
        touched |= set(ids[:, 6].tolist()) | set(ids[:, 4].tolist())
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0
        assert rel_state_diff(g.read_bodies(), o.state()) <= 1e-5, frame
    assert all(n > KEPT for n in most.values())
    assert touched == set(range(len(s.arrays["pos"])))
    g.close()


@pytest.mark.parametrize("kind", list(WIDE))
def test_a_body_above_many_triangles(kind, gpu_lib, oracle_lib):
    shape, params, quat, y = WIDE[kind]
    _lockstep(*_scene([(shape, params, quat, [0.07, y, 0.03])], 48, 0.25, 0.01), wide=[1])


def test_wide_and_small_bodies_in_one_group(gpu_lib, oracle_lib):
    bodies, wide = [], []
    for i in range(25):
        shape, params, quat, y = (list(WIDE.values()) + [SMALL])[i % 5]
        bodies.append((shape, params, quat, [4.3 * (i % 5 - 2) + 0.07, y, 4.3 * (i // 5 - 2) + 0.03]))
        if shape is not SMALL[0] or params is not SMALL[1]:
            wide.append(i + 1)
    _lockstep(*_scene(bodies, 96, 0.25, 0.01), wide=wide)


def _flat_box(hx, hz, cells, cell):
    return _scene([(scenes.BOX, [hx, 0.2, hz, 0], scenes.IDENTITY_Q, [0.0, 0.19, 0.0])], cells, cell)


def test_as_many_manifolds_as_a_pair_has_room_for(gpu_lib, oracle_lib):
    from physecs_gb300.api import World
    s, lo, hi = _flat_box(0.95, 1.95, 8, 1.0)
    w = World([s])
    w.step()
    assert len(w.contacts()[0]) == MANIFOLDS
    w.close()
    _lockstep(s, lo, hi, wide=[])


@pytest.mark.parametrize("hx,hz,cells,cell", [(1.05, 1.95, 8, 1.0), (0.5, 0.5, 48, 0.11)])   # 30 manifolds; > 64 triangles
def test_more_than_a_pair_has_room_for(hx, hz, cells, cell, gpu_lib):
    from physecs_gb300.api import PsxError, World
    s, _, _ = _flat_box(hx, hz, cells, cell)
    w = World([s])
    w.step()
    assert w.counts()["error"] == TRI_CAPACITY
    with pytest.raises(PsxError, match="CAPACITY"):
        w.synchronize()
    w.close()
