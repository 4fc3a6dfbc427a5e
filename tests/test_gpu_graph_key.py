"""Frames replayed as a CUDA graph while what its launches depend on changes:
the schedule flag, on grids whose width has the flag's bits and others, and
the grid's width under either schedule.  Against the oracle.  Tolerance 0."""
import numpy as np
import pytest

from parity import run_parity
from vxe import _abi as A
from vxe.scenes import Scene
from vxe.world import WorldSpec

pytestmark = pytest.mark.gpu


def _scene(dims):
    spec = WorldSpec(seed=99, height_min=10, height_max=40, dirt_depth=3, carve_mod=50, cave_threshold=0.6,
                     height_scale_vox=48.0, features=1)
    at = lambda f: (np.array([3.2 * dims[0], 5.5, 1.0]) + 0.07 * f, 0.6 + 0.02 * f, -0.3)  # noqa: E731
    return Scene("graph", spec, (0, 0, 0), dims, (97, 61), 1.0, 3, 128, 6, node_capacity=1 << 21, path=at)


@pytest.mark.parametrize("first", [0, A.FLAG_PRIMARY_MEGAKERNEL])
@pytest.mark.parametrize("width", [1, 8, 12, 16])
def test_schedule_flag_between_graph_frames(width, first):
    def toggle(g, o, bad, r, ora):
        r.set_flags(r.flags ^ A.FLAG_PRIMARY_MEGAKERNEL)

    res = run_parity(_scene((width, 1, 2)), frames=4, graph=True, extra_flags=first, on_frame=toggle)
    assert all(r == {} for r in res), res


@pytest.mark.parametrize("flags", [0, A.FLAG_PRIMARY_MEGAKERNEL])
def test_grid_width_between_graph_frames(flags):
    frame = iter(range(4))

    def narrow(cam):  # 4 columns wide, 12 wide, ...: the wider grid's slots are read at other cells of the narrower
        if next(frame) % 2 == 0:
            cam.grid_dims[0] = 4

    res = run_parity(_scene((12, 1, 2)), frames=4, graph=True, extra_flags=flags, cam_hook=narrow)
    assert all(r == {} for r in res), res
