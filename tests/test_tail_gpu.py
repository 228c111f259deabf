"""The multigrid tail (the coarse levels one CTA cycles as register strips) against the oracle's
PressureMultigrid restatement, V-cycle by V-cycle (PressureMultigrid.cpp:386-434).

Every tail threshold moves levels between the strip kernels and the tail. The FP64 V-cycle must
match the restatement to rounding at every threshold. This holds for shapes that stress the
tail's strip layout: the widest and tallest levels it takes (64 columns or rows), odd sides
whose coarse cells keep a shorter last cell, and strips one or two cells thin."""
import numpy as np
import pytest

from fluidsim_b200 import FluidGrid, scenes

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64), (63, 64), (64, 45), (127, 2), (2, 130), (190, 130), (257, 129), (1000, 3)]


def _case(w, h):
    y, x = np.mgrid[0:h, 0:w]
    density = np.where(((x // 3 + y // 5) % 2) == 0, 0.1, 100.0) * (1.0 + 0.25 * np.sin(0.37 * x + 0.11 * y))
    i = np.arange(w * h, dtype=float)
    residual = (np.sin(i * 0.29) + np.cos(i * 0.061)).reshape(h, w)
    return density, residual - residual.mean()


@pytest.mark.parametrize("cells", [64, 256, 1024, 4096])
@pytest.mark.parametrize("size", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_vcycle_matches_restatement_at_every_tail_threshold(oracle, size, cells):
    w, h = size
    density, residual = _case(w, h)
    inv_u, inv_v, _ = oracle.coefficients(density)
    mg = oracle.Multigrid(w, h)
    assert mg.rebuild(inv_u, inv_v)
    expected = mg.apply(residual)

    s = scenes.Scene(w, h, 1.0, 1.0, 1.0, 1.0, np.ones((h, w)), np.zeros((h, w + 1)), np.zeros((h + 1, w)),
                     liquid_mass=[density], gas_mass=[np.zeros((h, w))])
    g = FluidGrid(w, h, 1.0, "fp64")
    scenes.upload_scene(g, s)
    g.setTailCells(cells)
    z = g.applyPreconditioner(residual)
    scale = max(1.0, np.abs(expected).max())
    assert np.abs(z - expected).max() <= 1e-10 * scale


# Around the widths at which a level's row groups take 8, 16 and 32 lanes, heights that fill the last
# group of a warp or leave it short, and grids whose tail is the coarsest level alone.
GROUPS = [(16, 64), (17, 16), (32, 32), (33, 31), (31, 33), (34, 5), (64, 17), (15, 66), (8, 8), (9, 7), (1, 1), (66, 50)]


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-10), ("fp32", 5e-4)])
@pytest.mark.parametrize("size", GROUPS, ids=lambda s: f"{s[0]}x{s[1]}")
def test_vcycle_matches_restatement_at_row_group_edges(oracle, size, precision, bound):
    """The bounds are those of the tests beside this one."""
    w, h = size
    density, residual = _case(w, h)
    inv_u, inv_v, _ = oracle.coefficients(density)
    mg = oracle.Multigrid(w, h)
    assert mg.rebuild(inv_u, inv_v)
    expected = mg.apply(residual)
    s = scenes.Scene(w, h, 1.0, 1.0, 1.0, 1.0, np.ones((h, w)), np.zeros((h, w + 1)), np.zeros((h + 1, w)),
                     liquid_mass=[density], gas_mass=[np.zeros((h, w))])
    g = FluidGrid(w, h, 1.0, precision)
    scenes.upload_scene(g, s)
    g.setTailCells(4096)
    z = g.applyPreconditioner(residual)
    assert np.abs(z - expected).max() <= bound * max(1.0, np.abs(expected).max())


@pytest.mark.parametrize("size", [(64, 64), (190, 130), (1000, 3)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_fp32_tail_stays_close_to_fp64(size):
    """The FP32 tail differs from the FP64 one only by rounding."""
    w, h = size
    density, residual = _case(w, h)
    s = scenes.Scene(w, h, 1.0, 1.0, 1.0, 1.0, np.ones((h, w)), np.zeros((h, w + 1)), np.zeros((h + 1, w)),
                     liquid_mass=[density], gas_mass=[np.zeros((h, w))])
    out = {}
    for precision in ("fp64", "fp32"):
        g = FluidGrid(w, h, 1.0, precision)
        scenes.upload_scene(g, s)
        g.setTailCells(4096)
        out[precision] = g.applyPreconditioner(residual)
    scale = max(1.0, np.abs(out["fp64"]).max())
    assert np.abs(out["fp32"] - out["fp64"]).max() <= 5e-4 * scale


# Grids whose fine level and at least one more smoothed level are in the tail: at the default
# threshold, and at the largest one.
WHOLE = [(20, 20, 1024), (32, 32, 1024), (64, 16, 1024), (33, 31, 1024), (50, 41, 4096), (64, 64, 4096)]


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-10), ("fp32", 5e-4), ("mixed", 5e-4)])
@pytest.mark.parametrize("w,h,cells", WHOLE)
def test_residual_mean_is_taken_off_the_fine_level_alone(oracle, w, h, cells, precision, bound):
    """The preconditioner acts on residual - residual_mean (FluidGridCPU.cpp:1712-1726): a constant
    residual gives exact zeros, and a shifted one what the unshifted one gives. The residual is a
    multiple of 2^-16, so the shifted one is exact in FP32 too and the bounds are those above."""
    density, residual = _case(w, h)
    residual = np.round(residual * 65536.0) / 65536.0
    inv_u, inv_v, _ = oracle.coefficients(density)
    mg = oracle.Multigrid(w, h)
    assert mg.rebuild(inv_u, inv_v)
    expected = mg.apply(residual)
    s = scenes.Scene(w, h, 1.0, 1.0, 1.0, 1.0, np.ones((h, w)), np.zeros((h, w + 1)), np.zeros((h + 1, w)),
                     liquid_mass=[density], gas_mass=[np.zeros((h, w))])
    g = FluidGrid(w, h, 1.0, precision)
    scenes.upload_scene(g, s)
    g.setTailCells(cells)
    assert np.all(g.applyPreconditioner(np.full((h, w), 7.0), 7.0) == 0.0)
    z = g.applyPreconditioner(residual + 3.5, 3.5)
    assert np.abs(z - expected).max() <= bound * max(1.0, np.abs(expected).max())
