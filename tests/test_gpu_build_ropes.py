"""The voxels' ropes, written by a kernel of their own with eight lanes per
level-5 node: chunks whose level-5 lists end anywhere in a block, alone and in
batches with air and collapsed chunks, into buffers with exactly the nodes the
largest chunk needs (the rows behind a smaller chunk's nodes stay as they were)
and with one node fewer (that chunk writes no ropes at all), on rope buffers
that allow vector stores and on one that does not.  Byte for byte against the
host builder."""
import ctypes as C

import numpy as np
import pytest

from vxe import _abi as A
from vxe.renderer import Renderer
from vxe.world import WorldSpec, build_chunk

pytestmark = pytest.mark.gpu

SPEC = WorldSpec(seed=31, height_min=6, height_max=50, dirt_depth=3, cave_threshold=0.6, features=1)
AIR = (0, 4, 0)


def _build(r, coords, cap, nodes, ropes):
    """vxe_build_chunks_device into the caller's buffers; the counts."""
    import torch

    n, dev = coords.shape[0], coords.device
    macro = torch.empty((n, A.MACRO_WORDS_PER_CHUNK), dtype=torch.int32, device=dev)
    colinfo = torch.empty((n, A.COLINFO_WORDS_PER_CHUNK), dtype=torch.int32, device=dev)
    counts = torch.empty((n, 2), dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    params = SPEC.params()
    r._check(r._lib.vxe_build_chunks_device(r._ctx, C.byref(params), coords.data_ptr(), n, cap, nodes.data_ptr(),
                                            ropes.data_ptr(), macro.data_ptr(), colinfo.data_ptr(),
                                            counts.data_ptr()), "vxe_build_chunks_device")
    r.synchronize()
    return counts.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("keys", [[(0, 0, 0)], [AIR], [(3, 0, -2), AIR, (0, -1, 0)],
                                [(x, y, 5) for y in (0, 1) for x in range(-3, 4)]],
                         ids=["one", "air", "mixed", "fourteen"])
@pytest.mark.parametrize("short,offset", [(0, 0), (1, 0), (0, 1)], ids=["exact", "short", "unaligned"])
def test_voxel_ropes_equal_host_builder(keys, short, offset):
    import torch

    refs = [build_chunk(SPEC, *k) for k in keys]
    cap = max(len(c.nodes) for c in refs) - short
    n, dev = len(keys), "cuda:0"
    r = Renderer(64, 36, 1.0, node_capacity=1 << 16, chunk_capacity=16, grid_capacity=16, clip_levels=1, clip_res=16)
    try:
        coords = torch.tensor(keys, dtype=torch.int32, device=dev)
        nodes = torch.full((n, max(cap, 1), 4), -7, dtype=torch.int32, device=dev)
        flat = torch.full((n * max(cap, 1) * 8 + 4,), -7, dtype=torch.int32, device=dev)
        ropes = flat[offset:offset + n * max(cap, 1) * 8].view(n, max(cap, 1), 8)
        out = _build(r, coords, cap, nodes, ropes)
        got_n, got_r = (t.cpu().numpy().view(np.uint32) for t in (nodes, ropes))
        keep = np.uint32(2 ** 32 - 7)
        for j, ref in enumerate(refs):
            m = len(ref.nodes)
            assert out[j, 0] == m
            if m > cap:
                assert (got_r[j] == keep).all()
                continue
            assert np.array_equal(got_n[j, :m].reshape(-1), ref.nodes.view(np.uint32).reshape(-1)), keys[j]
            assert np.array_equal(got_r[j, :m].reshape(-1), ref.ropes.view(np.uint32).reshape(-1)), keys[j]
            assert (got_r[j, m:] == keep).all()
        assert (flat[offset + n * max(cap, 1) * 8:] == -7).all()
        assert r.read_error_word() == 0
    finally:
        r.close()
