"""Grass slab tasks sorted by lod and cell before their marches: frames at the
edges of tiles, warps and record limits against the oracle, and a batch whose
task records run out against the plain mode (inline marches).  Tolerance 0:
the sort changes the order of the marches only."""
import numpy as np
import pytest

from parity import run_parity
from vxe import _abi as A
from vxe import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,slabs", [((1, 1), 0), ((8, 8), 0), ((9, 33), 0), ((129, 65), 0), ((160, 90), 31),
                                        ((160, 90), 33), ((160, 90), 4097)])
def test_sorted_slab_marches_bit_exact(size, slabs):
    sc = scenes.config2(present=size, render_scale=1.0)
    res = run_parity(sc, frames=2, setup=lambda r: r.set_record_limits(0, slabs))
    assert all(r == {} for r in res), res


@pytest.mark.parametrize("limits", [(0, 0), (0, 1000), (500, 0)])
def test_batch_marches_left_open_match_inline_marches(limits):
    import torch

    from vxe.batch import make_batch
    from vxe.renderer import Renderer
    from vxe.scenes import FrameDriver

    sc = scenes.config2(present=(64, 36))
    drv = FrameDriver(sc)
    ups = drv.initial_uploads()
    w = drv.world
    r = Renderer(64, 36, 1.0, node_capacity=w.node_capacity, chunk_capacity=w.chunk_capacity,
                 grid_capacity=w.grid_capacity, clip_levels=sc.clip_levels, clip_res=sc.clip_res)
    try:
        r.upload_world(w, ups)
        _, _, clip, cam = drv.step()
        r.write_clipmap_updates(*clip)
        r.write_camera(cam)
        b = make_batch(w, torch, seed=9, n_viewports=5, n_queries=1, vp_range=((1, 330), (1, 190)), q_range=(100, 1000))
        r.submit_batch(b.requests, (8, 4), 1, A.BATCH_PLAIN)
        want = [t.cpu().numpy().copy() for t in b.outputs]
        for t in b.outputs:
            t.zero_()
        torch.cuda.synchronize()
        r.set_record_limits(*limits)
        r.submit_batch(b.requests, (8, 4), 1, A.BATCH_PERSISTENT)
        for i, (t, x) in enumerate(zip(b.outputs, want)):
            assert np.array_equal(t.cpu().numpy(), x), i
    finally:
        r.close()

