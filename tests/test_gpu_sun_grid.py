"""Sun horizons of large grids: a context of any grid capacity can be made, and
frames of grids around the largest that has a horizon equal the oracle's.  A
few chunks stand in a wide, otherwise empty grid.  Tolerance 0."""
import numpy as np
import pytest

from oracle import oracle as O
from parity import compare_frame, make_renderer, read_gpu_frame, run_parity
from vxe import _abi as A
from vxe.renderer import Renderer
from vxe.scenes import FrameDriver, Scene
from vxe.world import WorldSpec, ground_height

pytestmark = pytest.mark.gpu


def test_grid_capacity_beyond_any_horizon():
    # 2^27 cells (0.5 GB); a horizon for as many columns would take 275 GB
    r = Renderer(8, 8, 1.0, node_capacity=64, chunk_capacity=1, grid_capacity=1 << 27, clip_levels=1, clip_res=16)
    r.close()


def test_lane_bytes_count_the_horizon():
    sizes = []
    for cells in (1, 1000, 128 * 128, 128 * 128 + 1):
        r = Renderer(8, 8, 1.0, node_capacity=64, chunk_capacity=1, grid_capacity=cells, clip_levels=1, clip_res=16)
        sizes.append(r.view_lane_bytes(64, 36, 1.0))
        r.close()
    column = 2 * 16 * 16 * 4 + 4  # horizon and tops of 16 x 16 cells, their maximum
    assert [s - sizes[0] for s in sizes[1:]] == [999 * column, 16383 * column, 16383 * column]


@pytest.mark.parametrize("dims,at", [((128, 1, 128), (126, 0, 126)), ((129, 1, 128), (60, 0, 60)),
                                     ((16384, 1, 1), (9000, 0, 0)), ((1, 1, 16385), (0, 0, 9000)),
                                     ((3, 300, 3), (0, 2, 0)), ((2, 700, 2), (0, 620, 0)), ((100, 3, 70), (0, 1, 33))])
def test_frames_of_wide_grids_bit_exact(dims, at):
    spec = WorldSpec(seed=4242, height_min=10, height_max=40, dirt_depth=3, carve_mod=50, cave_threshold=0.6,
                     height_scale_vox=48.0, features=1)
    inner = tuple(min(2, d) for d in (dims[0], 1, dims[2]))
    path = lambda f: (np.array([3.2 * inner[0], 5.2, 1.5]) + 0.07 * f, 0.5, -0.25)  # noqa: E731
    sc = Scene("wide", spec, (0, 0, 0), inner, (97, 61), 1.0, 3, 128, 2, node_capacity=1 << 20, path=path)
    drv = FrameDriver(sc)
    ups = drv.initial_uploads()
    w = drv.world
    grid = np.full(dims[::-1], A.INVALID_U32, dtype=np.uint32)
    grid[at[2]:at[2] + inner[2], at[1]:at[1] + 1, at[0]:at[0] + inner[0]] = w.grid.reshape(inner[::-1])
    w.grid, w.grid_dims, w.grid_capacity = grid.reshape(-1), dims, grid.size
    w.grid_origin = tuple(-a for a in at)
    r = make_renderer(sc, w)
    try:
        r.upload_world(w, ups)
        ora = O.OracleFrameRunner(w, sc.internal, sc.present, drv.clip.tex, sc.clip_res, godray_alias=True)
        for _ in range(2):
            _, _, (params, patches), cam = drv.step()
            r.write_clipmap_updates(params, patches)
            r.write_camera(cam)
            r.encode_compute()
            ora.render(cam, params)
            bad = compare_frame(read_gpu_frame(r), ora.outputs())
            assert bad == {}, bad
        assert r.read_error_word() == 0
    finally:
        r.close()


@pytest.mark.parametrize("ox,oz,k", [(33000, 0, 2), (70000, 0, 0), (130000, 0, 6), (-130000, -130000, 3),
                                     (250000, 0, 6), (-250000, -250000, 3)])
def test_far_from_the_origin_bit_exact(ox, oz, k):
    # where binary32 positions are cells apart, a point's own cell is among those read or the ray marches
    spec = WorldSpec(seed=100 + k, height_min=5, height_max=60, dirt_depth=3, carve_mod=(0, 50)[k % 2],
                     cave_threshold=(0.6, 0.5, 2.0)[k % 3], height_scale_vox=(4.0, 8.0, 16.0, 48.0)[k % 4], features=1 + k % 3)
    ox, oz = ox + k, oz + (k if oz else 0)
    at = np.array([ox * 6.4 + 2.0 + k * 0.3, 0.0, oz * 6.4 + 2.0])
    at[1] = 0.1 * ground_height(spec, int(at[0] * 10), int(at[2] * 10)) + (1.0, 2.0, 4.0, 0.5)[k % 4]
    sc = Scene("far", spec, (ox, 0, oz), (3, 1, 3), (97, 61), 1.0, 3, 128, 2, node_capacity=1 << 20,
               path=lambda f: (at + 0.5 * f, 0.7 + k, -0.25 - 0.1 * (k % 3)))
    res = run_parity(sc, frames=2)
    assert all(r == {} for r in res), res
