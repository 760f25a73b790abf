"""Contact rows that are not live leave a -0 as it is.

A row past a contact's points, or the friction row of a contact without tangential velocity,
is skipped by the reference; the solver evaluates it with an impulse of zero.  Bodies that
have not turned yet hold velocity components of -0, which adding zero would turn into +0.
With no iteration the relaxation is the only sweep, and such components reach the state.
The oracle's frame, bit for bit."""
import numpy as np
import pytest

from physecs_gb300 import scenes
from tests.parity import gpu_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [{}, {"block_scene_max_dyn": 1, "launch": {"large_scene_solver": 2}}])
@pytest.mark.parametrize("knobs", [(1, 0), (2, 0), (1, 1)])
@pytest.mark.parametrize("index,n", [(3, 40), (4, 200), (5, 700)])
def test_frames_keep_the_sign_of_zero(index, n, knobs, opts, gpu_lib, oracle_lib):
    from oracle.port_api import OracleScene
    from physecs_gb300.api import World
    s = scenes.batch_scene(index, n_bodies=n, chain_prob=0.0)
    s.num_substeps, s.num_iterations = knobs
    s.arrays["pos"][(s.arrays["flags"] & scenes.BODY_DYNAMIC) != 0, 1] -= 0.5
    g, o = World([s], **opts), OracleScene(s)
    for f in range(4):
        g.step()
        g.synchronize()
        ids, _, meta = g.contacts()
        assert len(ids)
        o.set_contact_order(gpu_keys(ids, meta))
        o.step()
        assert o.order_error() == 0
        st, so = g.read_bodies(), o.state()
        for k in so:
            assert np.array_equal(st[k].view(np.uint32), so[k].view(np.uint32)), (f, k)
    g.close()
