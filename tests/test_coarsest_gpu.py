"""The coarsest level's factor where obstacles seal off a part of it (PressureMultigrid.cpp:300-384).

The operator with one cell pinned is then singular: the last pivot of the sealed part is a rounding
error, and its sign decides between a breakdown and a solve. The engine forms the factor with the
operations of the reference's column loop, each product fused into its subtraction; the emulation
here does the same in exact rationals rounded once, so the two decide alike."""
import math
from fractions import Fraction

import numpy as np
import pytest

from fluidsim_b200 import FluidGrid, scenes
from fluidsim_b200._native import FluidCudaError

pytestmark = pytest.mark.gpu


def _sealed(w, h, seed):
    """A wall across the grid, or a 2 x 2 pocket in a ring of obstacles; uneven or equal densities."""
    rng = np.random.default_rng(seed)
    solid = np.zeros((h, w), np.uint8)
    if seed % 2:
        solid[:, int(rng.integers(1, w - 1))] = 1
    else:
        x, y = int(rng.integers(0, w - 4)), int(rng.integers(0, h - 4))
        solid[y:y + 4, x:x + 4] = 1
        solid[y + 1:y + 3, x + 1:x + 3] = 0
    density = rng.uniform(0.5, 100.0, (h, w)) if seed % 3 else np.where(rng.random((h, w)) < 0.5, 10.0, 1.0)
    return scenes.Scene(w, h, 1.0, 1.0, 1.0, 1.0, np.ones((h, w)), np.zeros((h, w + 1)), np.zeros((h + 1, w)),
                        solid=solid, liquid_mass=[density], gas_mass=[np.zeros((h, w))])


def _operator(s):
    """Open cells, and the operator's rows over them as dicts of coefficients."""
    rho, solid, w, h = s.liquid_mass[0], s.solid, s.width, s.height
    right, down = np.zeros((h, w + 1)), np.zeros((h + 1, w))
    right[:, 1:-1] = np.where(solid[:, 1:] | solid[:, :-1], 0.0, 2.0 / (rho[:, :-1] + rho[:, 1:]))
    down[1:-1] = np.where(solid[1:] | solid[:-1], 0.0, 2.0 / (rho[:-1] + rho[1:]))
    diagonal = ((right[:, :-1] + right[:, 1:]) + down[:-1]) + down[1:]
    cells = [(y, x) for y in range(h) for x in range(w) if diagonal[y, x] > 0.0]
    index = {c: i for i, c in enumerate(cells)}
    rows = []
    for y, x in cells:
        row = {index[y, x]: float(diagonal[y, x])}
        for cell, weight in (((y, x - 1), right[y, x]), ((y - 1, x), down[y, x]), ((y, x + 1), right[y, x + 1]),
                             ((y + 1, x), down[y + 1, x])):
            if weight > 0.0:
                row[index[cell]] = -float(weight)
        rows.append(row)
    return cells, rows


def _breaks_down(rows):
    """Cholesky factor of the operator without its first cell, column by column."""
    n = len(rows) - 1
    a = [[rows[r + 1].get(c + 1, 0.0) for c in range(n)] for r in range(n)]
    for k in range(n):
        if not a[k][k] > 0.0:
            return True
        pivot = math.sqrt(a[k][k])
        for r in range(k + 1, n):
            a[r][k] /= pivot
        for r in range(k + 1, n):
            for c in range(k + 1, r + 1):
                if a[r][k] != 0.0 and a[c][k] != 0.0:
                    a[r][c] = float(Fraction(a[r][c]) - Fraction(a[r][k]) * Fraction(a[c][k]))
    return False


@pytest.mark.parametrize("w,h", [(8, 8), (7, 9), (12, 5)])
def test_sealed_parts_decide_as_the_column_loop(w, h):
    decisions = []
    for seed in range(40):
        s = _sealed(w, h, seed)
        cells, rows = _operator(s)
        g = FluidGrid(w, h, 1.0, "fp64")
        scenes.upload_scene(g, s)
        # A residual within the part of the first cell, without a mean there.
        part, todo = {0}, [0]
        while todo:
            for c in rows[todo.pop()]:
                if c not in part:
                    part.add(c)
                    todo.append(c)
        part = sorted(part)
        values = np.random.default_rng(seed).uniform(-1.0, 1.0, len(part))
        residual = np.zeros((h, w))
        for c, value in zip(part, values - values.mean()):
            residual[cells[c]] = value
        decisions.append(_breaks_down(rows))
        if decisions[-1]:
            with pytest.raises(FluidCudaError, match="factorisation failed"):
                g.applyPreconditioner(residual)
            continue
        # The sealed part's pivot of rounding size must not reach this part: the level is solved
        # directly, so its equations hold to rounding (condition below 1e5).
        z = g.applyPreconditioner(residual)
        for c in part:
            value = sum(weight * z[cells[n]] for n, weight in rows[c].items())
            assert abs(value - residual[cells[c]]) <= 1e-10 * max(1.0, np.abs(z).max())
    assert 0 < sum(decisions) < len(decisions)
