"""The fine-level vector kernels' tall and short tiles (vec_cells): grids on both sides of the rule
project alike alone and together in one batch, and against the FP64 restatement."""
import numpy as np
import pytest

from fluidsim_b200 import FluidGrid, ProjectionBatch, scenes

pytestmark = pytest.mark.gpu

# Short tiles (one row group, a ragged one, a tile's remainder in both axes) and, with more than 148
# tiles of 64 x 64, tall ones.
SIZES = [(64, 16), (65, 15), (130, 49), (832, 769)]


def _grid(scene, precision):
    g = FluidGrid(scene.width, scene.height, scene.cell_size, precision)
    scenes.upload_scene(g, scene)
    return g


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batch_of_short_and_tall_tiles_equals_single(precision):
    members = [scenes.random_pool(w, h, seed=40 + i, fill=0.55, obstacles=2) for i, (w, h) in enumerate(SIZES)]
    grids = [_grid(s, precision) for s in members]
    batch = ProjectionBatch(grids)
    together = batch.project([s.dt for s in members], 300, 1e-6, relative_tolerance=1e-6)
    for s, g, r in zip(members, grids, together):
        alone = _grid(s, precision)
        a = alone.project(s.dt, 300, 1e-6, relative_tolerance=1e-6)
        assert a.iterations == r.iterations and a.solve_status == "converged"
        x, y = g.download(), alone.download()
        assert np.array_equal(x.u, y.u) and np.array_equal(x.v, y.v) and np.array_equal(x.pressure, y.pressure)
    batch.destroy()


@pytest.mark.parametrize("size", SIZES[:3], ids=lambda s: f"{s[0]}x{s[1]}")
def test_short_tiles_match_restatement(oracle, size):
    """FP64 within 1e-8 of scale and three iterations, the projection tests' bounds."""
    s = scenes.random_pool(*size, seed=7, fill=0.6)
    g = _grid(s, "fp64")
    r = g.project(s.dt, 300, 1e-6)
    o = oracle.OracleGrid(s.width, s.height, s.cell_size)
    o.upload(s.density(), s.u, s.v)
    e = o.project(s.dt, 300, 1e-6)
    u, v, _ = o.download()
    d = g.download()
    assert r.converged and abs(r.iterations - e.iterations) <= 3
    scale = max(np.abs(u).max(), np.abs(v).max())
    assert np.abs(d.u - u).max() <= 1e-8 * scale and np.abs(d.v - v).max() <= 1e-8 * scale
