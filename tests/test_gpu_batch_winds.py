"""Batches whose viewports have different winds: the grass cell table holds the
first one's, the others derive their cells, and tasks of both meet in one
warp's chunk of slab marches.  Enough tasks for the 64-wide chunks, at the
edges of where they begin, and too few; against the plain mode (inline
marches).  Tolerance 0."""
import numpy as np
import pytest

from vxe import _abi as A
from vxe.renderer import Renderer
from vxe.scenes import FrameDriver, config2
from vxe.world import build_camera

pytestmark = pytest.mark.gpu


def _wide_tasks():
    """Slab tasks from which on a warp takes 64 at a time: 32 for each of its 64 warps per SM."""
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count * 64 * 32


@pytest.fixture(scope="module")
def scene():
    import torch

    sc = config2(present=(64, 36))
    drv = FrameDriver(sc)
    ups = drv.initial_uploads()
    w = drv.world
    r = Renderer(64, 36, 1.0, node_capacity=w.node_capacity, chunk_capacity=w.chunk_capacity,
                 grid_capacity=w.grid_capacity, clip_levels=sc.clip_levels, clip_res=sc.clip_res)
    r.upload_world(w, ups)
    _, _, clip, cam = drv.step()
    r.write_clipmap_updates(*clip)
    r.write_camera(cam)
    yield torch, sc, w, r
    r.close()


def _requests(torch, sc, w, views):
    """views: (path frame, width, height, wind time, wind strength scale)."""
    reqs, outs = [], []
    for f, vw, vh, t, k in views:
        pos, yaw, pitch = sc.path(f)
        cam = build_camera(pos, yaw, pitch, (vw, vh), (vw, vh), frame_index=1, time_s=t, world=w, jitter=False)
        cam.voxel_params[2] *= k
        out = torch.zeros(vw * vh * 32, dtype=torch.uint8, device="cuda")
        q = A.Request()
        q.kind, q.width, q.height, q.camera, q.d_out = A.REQ_VIEWPORT, vw, vh, cam, out.data_ptr()
        reqs.append(q)
        outs.append(out)
    return reqs, outs


WIDE = [(0, 480, 270, 0.0, 1.0), (24, 480, 270, 1.7, 1.0), (0, 480, 270, 1.7, 1.0), (24, 480, 270, 0.0, 0.5)]
NARROW = [(0, 33, 17, 0.3, 1.0), (24, 160, 90, 1.7, 1.0), (0, 1, 1, 1.7, 1.0)]


def _plain(torch, r, reqs, outs):
    r.set_record_limits(0, 0)
    r.submit_batch(reqs, (8, 4), 1, A.BATCH_PLAIN)
    return [o.cpu().numpy().copy() for o in outs]


@pytest.mark.parametrize("mode", [A.BATCH_PERSISTENT, A.BATCH_GRAPH])
@pytest.mark.parametrize("views,edge", [(NARROW, None), (WIDE, None), (WIDE, -1), (WIDE, 0), (WIDE, 1), (WIDE, 33),
                                        (WIDE[::-1], 63)])
def test_two_winds_in_one_batch_match_inline_marches(scene, views, edge, mode):
    torch, sc, w, r = scene
    reqs, outs = _requests(torch, sc, w, views)
    want = _plain(torch, r, reqs, outs)
    r.set_record_limits(0, 0 if edge is None else _wide_tasks() + edge)
    try:
        for _ in range(2):  # (graph mode: captured, then replayed)
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            r.submit_batch(reqs, (8, 4), 1, mode)
            for i, (o, x) in enumerate(zip(outs, want)):
                assert np.array_equal(o.cpu().numpy(), x), i
    finally:
        r.set_record_limits(0, 0)


def test_wide_batch_reaches_the_wide_chunks(scene):
    """The same cameras' cold frames meet more slab tasks than a 64-wide chunk asks for."""
    torch, sc, w, r = scene
    tasks = 0
    for f, vw, vh, t, _ in WIDE:
        r.resize_output(vw, vh)
        pos, yaw, pitch = sc.path(f)
        r.write_camera(build_camera(pos, yaw, pitch, (vw, vh), (vw, vh), frame_index=1, time_s=t, world=w, jitter=False))
        r.encode_compute()
        tasks += r.frame_stats()["slab_tasks"]
    r.resize_output(64, 36)
    assert tasks > _wide_tasks() + 64, tasks


@pytest.mark.parametrize("first,other", [(0.1, 0.05), (0.12, 0.1)])
def test_voxel_sizes_in_one_batch_match_cold_frames(scene, first, other):
    # the table holds cells of the first viewport's voxel size only
    torch, sc, w, r = scene
    reqs, outs = _requests(torch, sc, w, [(0, 160, 90, 0.0, 1.0), (0, 160, 90, 0.0, 1.0), (24, 97, 61, 0.0, 1.0)])
    for q, vs in zip(reqs, (first, other, other)):
        q.camera.voxel_params[0] = vs
    r.set_flags(r.flags | A.FLAG_HIT_RECORDS)
    want = []
    for q in reqs:
        r.resize_output(q.width, q.height)
        r.write_camera(q.camera)
        r.encode_compute()
        want.append(r.read_image(A.IMG_HITS).tobytes())
    r.resize_output(64, 36)
    r.set_flags(r.flags & ~A.FLAG_HIT_RECORDS)
    for mode in (A.BATCH_PLAIN, A.BATCH_PERSISTENT, A.BATCH_GRAPH, A.BATCH_GRAPH):
        r.submit_batch(reqs, (8, 4), 1, mode)
        for i, (o, x) in enumerate(zip(outs, want)):
            assert o.cpu().numpy().tobytes() == x, (mode, i)
            o.zero_()
        torch.cuda.synchronize()
