"""The solver's contact forms and record placements against the oracle.

A colour's contacts are solved in the order of their point count, by a form made for one,
two or four points or for soft contacts, with records in shared memory, in the world's
buffers, or split between the two.  Scenes with every point count, with and without soft
materials, step in lockstep with the oracle fed the GPU's contact order, at body counts
around a warp and a block.  Tolerance: 1e-5 relative, the parity bar of a frame from
identical state.
"""
import numpy as np
import pytest

from physecs_gb300 import scenes
from tests.parity import gpu_keys, rel_state_diff

pytestmark = pytest.mark.gpu


def _scene(n, soft):
    """n mixed bodies falling on each other, with flat boxes for contacts of four points."""
    s = scenes.batch_scene(500 + n, n_bodies=n, chain_prob=1.0 if n == 33 else 0.0)
    a = s.arrays
    box = np.nonzero(a["col_type"][1:n + 1] == scenes.BOX)[0] + 1
    a["quat"][box[::2]] = scenes.IDENTITY_Q
    a["pos"][1:n + 1, 1] -= 0.4
    a["vel"][1:n + 1, 1] = -3.0
    if soft:
        a["col_material"][1::3] = (0.5, 8.0, 0.7)
    return s


@pytest.mark.parametrize("soft", [False, True])
@pytest.mark.parametrize("n,opts", [
    (1, {}), (31, {}), (33, {}), (300, {}), (1030, {}),
    (300, {"launch": {"solver_smem_kb": 16}}),                                       # records split
    (1000, {"launch": {"solver_smem_kb": 16}}),                                      # velocities do not fit either
    (300, {"launch": {"large_scene_solver": 2}, "block_scene_max_dyn": 64}),         # the whole grid
    (300, {"launch": {"large_scene_solver": 1}, "block_scene_max_dyn": 64}),         # a cluster
])
def test_contact_forms_match_the_oracle(n, opts, soft, gpu_lib, oracle_lib):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World
    s = _scene(n, soft)
    g, o = World([s], **opts), OracleScene(s)
    seen = set()
    for frame in range(12):
        g.step()
        g.synchronize()
        ids, _, meta = g.contacts()
        seen |= set((ids[:, 3] & 0xff).tolist())
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0
        assert rel_state_diff(g.read_bodies(), o.state()) <= 1e-5, frame
    assert g.counts()["error"] == 0
    if n >= 300:
        assert {1, 2, 4} <= seen
    g.close()


def _lockstep(s, frames, **opts):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World
    g, o = World([s], **opts), OracleScene(s)
    for frame in range(frames):
        g.step()
        g.synchronize()
        ids, _, meta = g.contacts()
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0
        assert rel_state_diff(g.read_bodies(), o.state()) <= 1e-5, frame
    assert g.counts()["error"] == 0
    g.close()


@pytest.mark.parametrize("substeps,iterations", [(1, 0), (1, 1), (3, 5)])
@pytest.mark.parametrize("name", ["chains", "mechanisms", "free"])
def test_whole_grid_without_barriers_between_colours(name, substeps, iterations, gpu_lib, oracle_lib):
    """Joints of every kind, contacts alone and no contacts at all, solved by the whole grid
    as each body's earlier solves finish; sweeps with no iteration, one and several."""
    from tests.scene_variants import apart_scene, mechanism_scene
    if name == "chains":
        s = scenes.joint_chains(n_chains=9, links=11)
    elif name == "mechanisms":
        s = mechanism_scene()
        s = s[0] if isinstance(s, tuple) else s
    else:
        s = apart_scene()
    s.num_substeps, s.num_iterations = substeps, iterations
    _lockstep(s, 8, block_scene_max_dyn=1, launch={"large_scene_solver": 2})


def test_whole_grid_beyond_the_colour_limit(gpu_lib, oracle_lib):
    """A serial last colour keeps its contact order on the grid as well."""
    from tests.test_gpu_parity import _plate_with_spheres
    _lockstep(_plate_with_spheres(), 3, block_scene_max_dyn=1, launch={"large_scene_solver": 2})
