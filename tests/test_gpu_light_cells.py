"""Local-light rays that skip cells of an air cube already found, where that
cube must not stand for its cells: voxels so small that a far world's centres
are rounded by whole voxels.  Against the oracle's cell by cell queries.
Tolerance 0."""
import numpy as np
import pytest

from parity import run_parity
from vxe.scenes import Scene
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
