"""Slab marches of frames with enough tasks for 64 a warp, at the edges of where
those chunks begin, against the one-kernel schedule (marches inline).
Tolerance 0."""
import numpy as np
import pytest

from parity import make_renderer, read_gpu_frame
from vxe import _abi as A
from vxe.scenes import FrameDriver, config2

pytestmark = pytest.mark.gpu


def _frames(sc, extra, limit, frames=2):
    drv = FrameDriver(sc)
    ups = drv.initial_uploads()
    r = make_renderer(sc, drv.world, A.FLAG_GODRAY_MACRO_ALIAS | A.FLAG_HIT_RECORDS | extra)
    try:
        r.upload_world(drv.world, ups)
        r.set_record_limits(0, limit)
        out = []
        for _ in range(frames):
            _, _, clip, cam = drv.step()
            r.write_clipmap_updates(*clip)
            r.write_camera(cam)
            r.encode_compute()
            out.append(read_gpu_frame(r))
        return out, r.frame_stats()["slab_tasks"]
    finally:
        r.close()


def test_wide_chunks_match_inline_marches():
    import torch

    wide = torch.cuda.get_device_properties(0).multi_processor_count * 64 * 32  # tasks from which a warp takes 64
    sc = config2(present=(640, 360), render_scale=1.0)
    want, _ = _frames(sc, A.FLAG_PRIMARY_MEGAKERNEL, 0)
    for limit in (0, wide - 1, wide, wide + 1, wide + 33, wide + 63):
        got, tasks = _frames(sc, 0, limit)
        assert tasks > wide + 64, tasks
        for f, (g, w) in enumerate(zip(got, want)):
            for k in w:
                assert np.array_equal(g[k].view(np.uint8), w[k].view(np.uint8)), (limit, f, k)
