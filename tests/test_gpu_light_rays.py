"""Local-light rays that skip cells of an air cube already found, against the
oracle's cell by cell queries: worlds at the origin, across the 1000 m line
beyond which every cell is looked up, and far out, on both sides of zero.
Tolerance 0."""
import numpy as np
import pytest

from parity import run_parity
from vxe.scenes import Scene
from vxe.world import WorldSpec, ground_height

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("origin", [(0, 0, 0), (155, 0, -3), (-157, 0, 155), (400, 0, -400)])
def test_light_rays_bit_exact(origin):
    spec = WorldSpec(seed=777, height_min=10, height_max=30, dirt_depth=3, carve_mod=50, cave_threshold=0.62,
                     height_scale_vox=48.0, features=3)
    at = np.array([origin[0] * 6.4 + 7.0, 0.0, origin[2] * 6.4 + 7.0])
    at[1] = 0.1 * ground_height(spec, int(at[0] * 10), int(at[2] * 10)) + 1.2
    sc = Scene("lights", spec, origin, (2, 1, 2), (97, 61), 1.0, 3, 128, 2, node_capacity=1 << 20,
               path=lambda f: (at + 0.05 * f, 0.7 + 0.3 * f, -0.5))
    res = run_parity(sc, frames=2)
    assert all(r == {} for r in res), res
