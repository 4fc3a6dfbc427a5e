"""Batches of more viewport rays than the deferred passes have room for are
refused before anything is launched."""
import pytest

from vxe import _abi as A
from vxe.renderer import Renderer
from vxe.world import build_camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [A.BATCH_PERSISTENT, A.BATCH_GRAPH])
@pytest.mark.parametrize("side", [16384, 25000])  # 16384^2: one ray more than 30-bit probe indices have room for
def test_batch_beyond_its_ray_buffers_is_refused(side, mode):
    r = Renderer(8, 8, 1.0, node_capacity=64, chunk_capacity=1, grid_capacity=1, clip_levels=1, clip_res=16)
    try:
        q = A.Request()
        q.kind, q.width, q.height = A.REQ_VIEWPORT, side, side
        q.camera = build_camera((0, 0, 0), 0.0, 0.0, (side, side), (side, side), frame_index=1, time_s=0.0, jitter=False)
        q.d_out = 256  # never written: the batch is refused
        with pytest.raises(A.VxeError) as e:
            r.submit_batch([q], (8, 4), 1, mode)
        assert A.STATUS_NAMES[e.value.status] == "VXE_ERR_CAPACITY"
    finally:
        r.close()
