"""Local-light rays that skip cells of an air cube already found, where that
cube must not stand for its cells: voxels so small that a far world's centres
are rounded by whole voxels, and slots whose meta stands elsewhere than the
grid cell they serve.  Against the oracle's cell by cell queries.  Tolerance 0."""
import ctypes as C

import numpy as np
import pytest

import parity
from parity import run_parity
from vxe import _abi as A
from vxe.scenes import FrameDriver, Scene
from vxe.world import WorldSpec, ground_height

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vs,ox,oz,k", [(1e-4, -129997, 0, 3), (1e-4, 150004, 0, 4), (1e-5, 130003, 130003, 3),
                                        (1e-5, 130007, 130007, 7), (0.003, 155, -3, 1), (3.0, -157, 155, 2)])
def test_light_rays_of_any_voxel_size_bit_exact(vs, ox, oz, k):
    spec = WorldSpec(seed=100 + k, height_min=5, height_max=60, dirt_depth=3, carve_mod=(0, 50)[k % 2],
                     cave_threshold=(0.6, 0.5, 2.0)[k % 3], height_scale_vox=(4.0, 8.0, 16.0, 48.0)[k % 4], features=3)
    at = np.array([ox * 64 + 20.0 + k * 3, 0.0, oz * 64 + 20.0])
    at[1] = ground_height(spec, int(at[0]), int(at[2])) + (10, 20, 40, 5)[k % 4]
    sc = Scene("lights", spec, (ox, 0, oz), (3, 1, 3), (65, 41), 1.0, 3, 128, 2, node_capacity=1 << 20,
               path=lambda f: (vs * (at + 5 * f), 0.7 + k, -0.25 - 0.1 * (k % 3)))

    def voxel_size(cam):
        cam.voxel_params[0] = vs

    res = run_parity(sc, frames=2, cam_hook=voxel_size)
    assert all(r == {} for r in res), res


@pytest.mark.parametrize("macro", [True, False])
@pytest.mark.parametrize("seed,light,shift", [(825, (62, 22, 58), -38), (825, (62, 22, 58), -33), (825, (61, 27, 3), -33),
                                              (823, (62, 21, 41), -37), (777, (62, 20, 30), -64), (777, (62, 20, 30), 5)])
def test_light_rays_past_a_slot_that_stands_elsewhere(monkeypatch, seed, light, shift, macro):
    # lights just outside a grid cell whose slot's chunk reaches over its border
    worlds = []

    class Kept(FrameDriver):
        def initial_uploads(self):
            worlds.append(self.world)
            return super().initial_uploads()

    def move(r):
        w = worlds[-1]
        m, slot = w.metas[:w.chunk_count], w.key_to_slot[(1, 0, 0)]
        m[slot, 0] = 64 + shift
        if not macro:
            m[slot, 6] = A.INVALID_U32
        r._check(r._lib.vxe_write_meta(r._ctx, 0, m.ctypes.data_as(C.POINTER(A.ChunkMeta)), len(m)), "vxe_write_meta")

    monkeypatch.setattr(parity, "FrameDriver", Kept)
    spec = WorldSpec(seed=seed, height_min=10, height_max=30, dirt_depth=3, carve_mod=50, cave_threshold=0.62,
                     height_scale_vox=48.0, features=3)
    at = np.array([8.6, 0.1 * light[1] + 1.5, 0.1 * light[2] + 0.2])
    sc = Scene("lights", spec, (0, 0, 0), (2, 1, 1), (97, 61), 1.0, 3, 128, 2, node_capacity=1 << 20,
               path=lambda f: (at, -1.5708, -0.6))
    res = run_parity(sc, frames=2, setup=move)
    assert all(r == {} for r in res), res
