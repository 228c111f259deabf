"""The viscosity V-cycle's kernels at the sizes where their tiles, rings and one-CTA levels end, against
the FP64 restatement: variable viscosity and density, so that every coefficient differs."""
import numpy as np
import pytest

from fluidsim_b200 import FluidGrid, FluidGridState
from fluidsim_b200._native import FluidCudaError

pytestmark = pytest.mark.gpu

# A single level, thin lattices, the restriction's and prolongation's 32 x 8 tiles and their
# remainders, levels of at most and of more than one node per thread of the one-CTA cycle, the largest
# squares that are all in it and the next ones (55 and 56 in FP32, 38 and 39 in FP64), and two and
# three levels above it.
SIZES = [(8, 8), (3, 90), (90, 3), (31, 31), (32, 33), (63, 16), (55, 55), (56, 56), (38, 38),
         (39, 39), (66, 65), (97, 130), (257, 66), (300, 211)]


@pytest.mark.parametrize("precision,bound", [("fp64", 1e-10), ("fp32", 1e-3)])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_solve_matches_restatement(oracle, size, precision, bound):
    """FP64 to rounding and the same iteration count. FP32 within 1e-3 of scale: it stops at the same
    1e-4 rule, where a change of rounding moves the iterate by about its own tolerance."""
    w, h = size
    dx, dt = 1.0 / max(w, h), 1.0 / 120.0
    y, x = np.mgrid[0:h, 0:w]
    share = 0.5 + 0.5 * np.sin(0.31 * x + 0.17 * y)
    lm, gm = 900.0 * share * dx * dx, 40.0 * (1.0 - share) * dx * dx
    rng = np.random.default_rng(w * 1000 + h)
    u, v = rng.uniform(-1, 1, (h, w + 1)), rng.uniform(-1, 1, (h + 1, w))
    u, v = u.astype(np.float32).astype(float), v.astype(np.float32).astype(float)
    u[:, 0] = u[:, -1] = 0.0
    v[0] = v[-1] = 0.0
    g = FluidGrid(w, h, dx, precision)
    g.configureMaterials([900.0], [40.0], [2.0], [0.01])
    g.upload(FluidGridState(share, u, v, None, [lm], [gm]))
    it, _ = g.applyViscosity(dt, 1e-4)
    material = oracle.viscosity_material([lm, gm], [900.0, 40.0], [2.0, 0.01], dx)
    expected_it, eu, ev, _ = oracle.Viscosity(w, h).solve(u, v, material, dt, dx, 1e-4)
    s = g.download()
    scale = max(np.abs(eu).max(), np.abs(ev).max())
    if precision == "fp64":
        assert it == expected_it
    assert np.abs(s.u - eu).max() <= bound * scale and np.abs(s.v - ev).max() <= bound * scale


def test_tall_thin_lattice_equals_its_transpose():
    """More rows of tiles than a launch's second dimension holds (65,535): the solve runs, and equals
    the transposed one to the stop rule's tolerance."""
    w, h, dt = 2, 530000, 1.0 / 120.0
    dx = 1.0 / 512.0
    y = np.arange(h)
    rng = np.random.default_rng(5)
    share = np.repeat((0.5 + 0.5 * np.sin(0.003 * y))[:, None], w, axis=1)
    u, v = np.zeros((h, w + 1)), np.zeros((h + 1, w))
    u[:, 1] = rng.uniform(-1, 1, h)
    v[1:-1] = rng.uniform(-1, 1, (h - 1, w))
    out = []
    for transpose in (False, True):
        f = share.T if transpose else share
        g = FluidGrid(*((h, w) if transpose else (w, h)), dx, "fp64")
        g.configureMaterials([900.0], [40.0], [2.0], [0.01])
        g.upload(FluidGridState(f, v.T if transpose else u, u.T if transpose else v, None, [900.0 * f * dx * dx],
                                [40.0 * (1.0 - f) * dx * dx]))
        it, residual = g.applyViscosity(dt, 1e-4)
        assert it > 0 and residual <= 1.1e-4
        s = g.download()
        out.append((s.v.T, s.u.T) if transpose else (s.u, s.v))
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-8 * max(np.abs(b).max(), 1e-30)


@pytest.mark.parametrize("precision,viscosity,mass", [("fp32", 1e39, 1.0), ("fp32", 1e38, 1.0), ("fp64", 2.0, np.inf),
                                                      ("fp32", 2.0, 1e39)])
def test_a_diagonal_beyond_the_precision_is_an_error(precision, viscosity, mass):
    """A cell viscosity, a sum of them, or a face mass that overflows: the solve reports it and leaves
    the velocities (an open face whose inverse diagonal is zero must not count as a closed one)."""
    w, h = 24, 17
    rng = np.random.default_rng(1)
    u, v = rng.uniform(-1, 1, (h, w + 1)), rng.uniform(-1, 1, (h + 1, w))
    masses = np.ones((h, w))
    masses[5:9, 3:8] = mass
    g = FluidGrid(w, h, 1.0, precision)
    g.configureMaterials([1.0], [1.0], [viscosity], [0.0])
    g.upload(FluidGridState(np.ones((h, w)), u, v, None, [masses], [np.zeros((h, w))]))
    before = g.download()
    with pytest.raises(FluidCudaError):
        g.applyViscosity(1.0, 1e-4)
    after = g.download()
    assert np.array_equal(before.u, after.u) and np.array_equal(before.v, after.v)
