"""Batched ray queries (rays refilled lane by lane, phases voted by the warp)
against vxe_trace_rays, which the oracle pins, at counts around a warp, a
share and more rays than the GPU holds; rays that start outside the grid, on
its faces, inside solid voxels and along the axes; several requests and
tmax values in one batch.  Records equal bit for bit."""
import numpy as np
import pytest

from vxe import _abi as A
from vxe.renderer import Renderer
from vxe.scenes import FrameDriver, config2, features

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[config2, features])
def world(request):
    import torch

    sc = request.param(present=(64, 36))
    drv = FrameDriver(sc)
    ups = drv.initial_uploads()
    w = drv.world
    r = Renderer(64, 36, 1.0, node_capacity=w.node_capacity, chunk_capacity=w.chunk_capacity,
                 grid_capacity=w.grid_capacity, clip_levels=sc.clip_levels, clip_res=sc.clip_res)
    r.upload_world(w, ups)
    r.write_camera(drv.step()[3])
    yield torch, w, r
    r.close()


def rays(world, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = world.world_aabb_m()
    span = hi - lo
    o = rng.uniform(lo - 0.1 * span, hi + 0.1 * span, size=(n, 3))
    o[::7, 1] = lo[1]                                # on the grid's floor
    o[3::11] = np.round(o[3::11] / 6.4) * 6.4        # on chunk corners
    d = rng.normal(size=(n, 3))
    d[::5] = np.eye(3)[rng.integers(0, 3, len(d[::5]))] * rng.choice([-1.0, 1.0], (len(d[::5]), 1))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


@pytest.mark.parametrize("sizes", [[1], [31], [33], [1, 32, 2, 127], [5000, 1, 700], [100_003]])
def test_batched_queries_match_single_queries(world, sizes):
    torch, w, r = world
    reqs, outs, want = [], [], []
    for k, n in enumerate(sizes):
        o, d = rays(w, n, 31 * n + k)
        tmax = 120.0 if k % 2 == 0 else 9.0
        to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
        out = torch.full((n, 32), 0xCD, dtype=torch.uint8, device="cuda")
        q = A.Request()
        q.kind, q.ray_count, q.tmax = A.REQ_QUERY, n, tmax
        q.d_origins, q.d_dirs, q.d_out = to.data_ptr(), td.data_ptr(), out.data_ptr()
        reqs.append(q)
        outs.append((out, to, td))
        want.append(r.trace_rays(o, d, tmax))
    torch.cuda.synchronize()
    for mode in (A.BATCH_PERSISTENT, A.BATCH_GRAPH):
        r.submit_batch(reqs, (8, 4), 1, mode)
        for (out, _, _), x in zip(outs, want):
            assert out.cpu().numpy().tobytes() == x.tobytes()
            out.fill_(0xCD)
        torch.cuda.synchronize()
