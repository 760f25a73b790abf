"""Bodies with many joints in a scene that the whole grid solves.

A body's joint rows that have an error are counted, and its position integration divides
its pseudo velocities by their number; in the whole grid's solver the count and the body's
finished joints share a word (csrc/solver_words.cuh).  Hubs of one joint kind put the count
just below and above 255, at even and odd numbers of hundreds, and the joints at and past
the number above which the scene is solved with barriers.  One block, whose solver counts
rows in a float, gives the same scene the same bytes; with one kind of row (spherical
joints) so does the oracle, within 1e-5, the parity bar of a frame from identical state.
Toggling bodies between kinematic and simulated moves which joints wait for which."""
import numpy as np
import pytest

from physecs_gb300 import scenes
from tests.parity import gpu_keys, rel_state_diff
from tests.scene_variants import delta_schedule

pytestmark = pytest.mark.gpu

GRID = dict(block_scene_max_dyn=1, launch={"large_scene_solver": 2})
ROWS = {scenes.JOINT_FIXED: 6, scenes.JOINT_REVOLUTE: 5, scenes.JOINT_SPHERICAL: 3}


def _hub(n, kind, pitch=0.5, seed=3):
    """A free hub with n joints of one kind to small balls on a ring around it, every row of
    each off by a little; below a pitch of 0.3 neighbouring balls touch."""
    rng = np.random.default_rng(seed)
    s = scenes.SceneData("hub%d" % n)
    at = 2 * np.pi * np.arange(n) / n
    radius = max(1.0, n * pitch / (2 * np.pi))
    ring = radius * np.stack([np.cos(at), 0 * at, np.sin(at)], 1)
    q = rng.normal(0, 0.03, (n + 1, 4)) + [0, 0, 0, 1]
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    m, com, inertia = scenes.mass_sphere(0.6)
    s.add_bodies(pos=[[0.0, 5.0, 0.0]], quat=q[:1], flags=scenes.BODY_DYNAMIC, inv_mass=1.0 / m, com=com,
                 inv_inertia=np.linalg.inv(inertia).T.ravel(), col_type=scenes.SPHERE, col_params=[0.6, 0, 0, 0])
    m, com, inertia = scenes.mass_sphere(0.15)
    s.add_bodies(pos=ring + [0, 5, 0], quat=q[1:], flags=scenes.BODY_DYNAMIC, inv_mass=1.0 / m, com=com,
                 inv_inertia=np.linalg.inv(inertia).T.ravel(), col_type=scenes.SPHERE, col_params=[0.15, 0, 0, 0],
                 vel=rng.normal(0, 0.2, (n, 3)))
    fr = np.zeros((n, 14))
    fr[:, 0:3] = ring + rng.normal(0, 0.01, (n, 3))
    fr[:, 6] = fr[:, 13] = 1.0
    s.add_joints(kind, np.zeros(n, np.int32), np.arange(1, n + 1, dtype=np.int32), fr)
    return s.finalize()


def _same_as_one_block(s, frames):
    """Steps s by the grid and by a block; returns its joint rows and the contacts met."""
    from physecs_gb300.api import World
    g, b = World([s], **GRID), World([s], block_scene_max_dyn=1 << 20)
    met = 0
    for frame in range(frames):
        g.step()
        b.step()
        g.synchronize()
        met += len(g.contacts()[0])
        x, y = g.read_bodies(), b.read_bodies()
        for k in x:
            assert np.isfinite(x[k]).all()
            assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), (frame, k)
    assert g.counts()["error"] == 0 and b.counts()["error"] == 0
    rows = g.counts()["rows"]
    g.close()
    b.close()
    return rows, met


def _lockstep(s, frames, deltas=None):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World, pack_deltas
    g, o = World([s], **GRID), OracleScene(s)
    for frame in range(frames):
        if deltas and frame in deltas:
            d = pack_deltas(deltas[frame])
            o.apply_deltas(d)
            g.apply_deltas(d)
        g.step()
        g.synchronize()
        ids, _, meta = g.contacts()
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0
        assert rel_state_diff(g.read_bodies(), o.state()) <= 1e-5, frame
    assert g.counts()["error"] == 0
    g.close()


@pytest.mark.parametrize("pitch", [0.5, 0.28])
@pytest.mark.parametrize("kind,n", [
    (scenes.JOINT_FIXED, 42), (scenes.JOINT_FIXED, 43), (scenes.JOINT_FIXED, 60), (scenes.JOINT_FIXED, 101),
    (scenes.JOINT_REVOLUTE, 51), (scenes.JOINT_REVOLUTE, 52), (scenes.JOINT_REVOLUTE, 103),
    (scenes.JOINT_SPHERICAL, 85), (scenes.JOINT_SPHERICAL, 86), (scenes.JOINT_SPHERICAL, 171)])
def test_hub_of_many_joints(kind, n, pitch, gpu_lib):
    rows, met = _same_as_one_block(_hub(n, kind, pitch), 3)
    assert rows == n * ROWS[kind]
    assert (met > 0) == (pitch < 0.3)


@pytest.mark.parametrize("n", [85, 86, 100, 171])
def test_hub_matches_the_oracle(n, gpu_lib, oracle_lib):
    _lockstep(_hub(n, scenes.JOINT_SPHERICAL), 3)


@pytest.mark.parametrize("n", [8191, 8192])   # kFlowJoints, and one more: solved with barriers
def test_hub_at_the_limit_of_the_counts(n, gpu_lib):
    s = _hub(n, scenes.JOINT_FIXED)
    s.num_substeps, s.num_iterations = 1, 1
    rows, _ = _same_as_one_block(s, 2)
    assert rows == 6 * n


def test_kinematic_toggles_of_jointed_bodies(gpu_lib, oracle_lib):
    s = scenes.joint_chains(n_chains=6, links=9, substeps=3, iterations=3)
    _lockstep(s, 24, deltas=delta_schedule(s, 24, seed=11, every=2))


def test_a_wait_through_many_sweeps_is_not_a_timeout(gpu_lib):
    """The position of a body whose joints other lanes solve waits for every iteration of the
    substep; a limit that each barrier keeps does not end it."""
    from physecs_gb300.api import World
    s = _hub(40, scenes.JOINT_SPHERICAL)
    s.num_substeps, s.num_iterations = 1, 400
    g, b = World([s], **GRID), World([s], block_scene_max_dyn=1 << 20)
    g.set_wait_limit(4096)
    g.step()
    g.synchronize()
    b.step()
    x, y = g.read_bodies(), b.read_bodies()
    for k in x:
        assert np.array_equal(x[k].view(np.uint32), y[k].view(np.uint32)), k
    g.close()
    b.close()
