"""The step's banded z-solve (csrc/k_zsolve.cu) through the pressure solve, against the
oracle, at the edges of its tiles: the smallest column, halves that are and are not whole
batches of rows, grids whose last tile of mode pairs is partial, every tile width, columns
too long for their factors to be staged, the streaming form of large FP64 VV4 planes, and
low-mode sets that split a tile.

Tolerances: relative to the largest pressure.  FP64: the banded systems' condition numbers
stay below 1e5 on these meshes, so 1e-10 leaves a factor 10 over 1e5 x 1e-16 x 10 operations
per row.  Mixed: float transforms and sweeps, the 6e-6 of the plane kernels' test."""
import numpy as np
import pytest

from cases import COLLOC, HW2, VV4, make_case, rel_err, seeded_field, within

pytestmark = pytest.mark.gpu

# (scheme, NX, NY, NZ, low_modes)
GRIDS = [(s, 8, 8, nz, 0) for s in (HW2, VV4, COLLOC) for nz in (6, 7, 18, 19, 20, 35, 36)]
GRIDS += [
    (VV4, 16, 24, 33, 1), (HW2, 16, 24, 33, 2), (COLLOC, 24, 16, 34, 7),  # low-mode sets
    (VV4, 64, 54, 17, 0), (HW2, 128, 162, 9, 0), (COLLOC, 128, 64, 49, 0),  # partial tiles, wide tiles
    (VV4, 16, 16, 400, 0), (HW2, 16, 16, 700, 0),  # long columns: narrow tiles
    (VV4, 384, 288, 7, 0),  # FP64: one thread per mode
]


# the mixed tolerance is the plane kernels' and holds for their column lengths
CASES = [g + (p,) for g in GRIDS for p in (0, 1) if p == 0 or g[3] <= 64]


@pytest.mark.parametrize("scheme,NX,NY,NZ,low,precision", CASES)
def test_pressure_solve_tiles(scheme, NX, NY, NZ, low, precision):
    import oracle_py as op
    import turbchannel_b200 as tb

    prod, orc, zz = make_case(scheme, NX, NY, NZ, precision=precision, low_modes=low, gamma=1.2)
    S = tb.Solver(prod, zz)
    O = op.Oracle(orc, zz, "f64")
    coll = scheme == COLLOC
    v = seeded_field(S.N, NX * NY, seed=11, wall_w_zero=not coll)
    if coll:
        v[:NX * NY] = 0.0
        v[-NX * NY:] = 0.0
    rhs = O.apply_divergence(v)
    want = O.pressure_solve(rhs)
    err = rel_err(S.LinearSystemSolveFFT(rhs), want)
    S.close()
    assert within(f"zsolve/{scheme}/{NX}x{NY}x{NZ}/p{precision}", err, 1e-10 if precision == 0 else 6e-6), err


@pytest.mark.parametrize("scheme,NZ", [(VV4, 3700), (HW2, 5000)])
def test_long_columns_solve_their_matrix(scheme, NZ):
    """Columns whose factors stay in global memory: the solution's divergence of its gradient
    is the right-hand side (FP64; the residual of a backward-stable band solve, relative to
    the largest matrix entry times the solution)."""
    import turbchannel_b200 as tb

    prod, _, zz = make_case(scheme, 8, 8, NZ, gamma=1.0)
    S = tb.Solver(prod, zz)
    v = seeded_field(S.N, 64, seed=5)
    rhs = S.ApplyDivergence(v)
    p = S.LinearSystemSolveFFT(rhs)
    back = S.ApplyDivergence(S.ApplyGradient(p))
    dz = np.diff(zz)
    scale = 8.0 / dz.min() * np.max(np.abs(p))
    S.close()
    assert np.max(np.abs(back - rhs)) < 1e-13 * scale + 1e-12 * np.max(np.abs(rhs))
