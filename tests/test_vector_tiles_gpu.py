"""The fine-level vector kernels' tall, short and grouped tiles (vec_cells, kGroupLimit): grids on both
sides of the rules project alike alone and together in one batch, and against the FP64 restatement."""
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


# Grids of short tiles whose groups end after one to four of them, in one column of tiles or several.
GROUPED = [(64, 64), (65, 65), (130, 49), (1, 300), (90, 17), (33, 128), (200, 97), (70, 145)]


@pytest.mark.parametrize("precision,air,preconditioner",
                         [("fp32", "gas", "multigrid"), ("fp64", "gas", "multigrid"), ("mixed", "dirichlet", "multigrid"),
                          ("fp32", "gas", "diagonal")])
def test_crowded_batch_equals_single(precision, air, preconditioner):
    """More than 296 groups of short tiles, and a grid of tall ones: every sum of a grid is formed as
    when it is alone, so the batch equals the grids bit for bit."""
    members = [scenes.random_pool(w, h, seed=i, fill=0.55, obstacles=i % 3) for i, (w, h) in enumerate(GROUPED * 12)]
    members.append(scenes.random_pool(832, 769, seed=1, fill=0.55))
    assert sum(-(-s.width // 64) * -(-s.height // 64) for s in members[:-1]) > 296
    for s in members:
        s.air_model = air
    cap = 300 if preconditioner == "multigrid" else 20
    batch_grids = [_grid(s, precision) for s in members]
    for g in batch_grids:
        g.setPreconditioner(preconditioner)
    batch = ProjectionBatch(batch_grids)
    together = batch.project([s.dt for s in members], cap, 1e-6, relative_tolerance=1e-6)
    for s, g, r in zip(members, batch_grids, together):
        alone = _grid(s, precision)
        alone.setPreconditioner(preconditioner)
        a = alone.project(s.dt, cap, 1e-6, relative_tolerance=1e-6)
        assert a.iterations == r.iterations and a.solve_status == r.solve_status
        assert a.residual_l2 == r.residual_l2 and a.max_divergence == r.max_divergence and a.rhs_l2 == r.rhs_l2
        x, y = g.download(), alone.download()
        assert np.array_equal(x.u, y.u) and np.array_equal(x.v, y.v) and np.array_equal(x.pressure, y.pressure)
        alone.destroy()
    batch.destroy()
