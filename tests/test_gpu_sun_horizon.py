"""Sun rays cleared by the grid's horizon map against the oracle's full shadow
marches: grids of different shapes, cameras inside, at the rim and outside of
the grid, trees and caves.  Tolerance 0: a cleared ray's transmittance is
exactly the march's 1."""
import numpy as np
import pytest

from parity import run_parity
from vxe.scenes import Scene
from vxe.world import WorldSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,pos,look", [
    ((1, 1, 1), (3.2, 6.0, -2.0), (0.0, -0.4)),       # outside, before the grid
    ((2, 1, 5), (6.39, 4.6, 12.8), (0.8, -0.3)),      # on a chunk border
    ((5, 2, 1), (33.0, 9.0, 3.0), (-1.57, -0.35)),    # outside, behind the grid on the sun's way
    ((3, 2, 3), (9.6, 14.0, 9.6), (0.8, -0.9)),       # above every top
    ((4, 1, 3), (12.8, 2.0, 9.6), (2.4, 0.15)),       # under the surface or in a cave
])
def test_cleared_sun_rays_bit_exact(dims, pos, look):
    spec = WorldSpec(seed=4242, height_min=10, height_max=40, dirt_depth=3, carve_mod=50, cave_threshold=0.6,
                     height_scale_vox=48.0, features=3)
    at = lambda f: (np.array(pos) + 0.07 * f, look[0] + 0.02 * f, look[1])  # noqa: E731
    sc = Scene("sun", spec, (0, 0, 0), dims, (97, 61), 1.0, 3, 128, 2, node_capacity=1 << 20, path=at)
    for alias in (True, False):
        res = run_parity(sc, frames=2, godray_alias=alias)
        assert all(r == {} for r in res), res
