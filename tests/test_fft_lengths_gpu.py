"""Every compiled register-transform length (csrc/k_fft.cuh) along x and along y, and tiles of
rows for y-counts that no power of two divides, through the pressure solve against the
oracle; the divergence of the vector right-hand side where NX is not a multiple of 4.

Tolerances.  FP64: 1e-10 relative to the largest pressure, as the other solve tests.  Mixed:
in the 2-norm against the FP64 solve of the same 32-bit right-hand side of white noise (whose
solution does not amplify the transforms' white errors over its own spectrum, as that of a
divergence does), about 10 butterfly stages in each of four float transforms at 6e-8 per
stage, 2.4e-6."""
import numpy as np
import pytest

from cases import HW2, VV4, make_case, rel_err, seeded_field, within

pytestmark = pytest.mark.gpu

LENGTHS = sorted(2 ** a * 3 ** b for a in range(1, 11) for b in range(7) if 8 <= 2 ** a * 3 ** b <= 1024)
GRIDS = [(n, m) for n in LENGTHS for m in (8, 18)] + [(m, n) for n in LENGTHS for m in (16, 18)]
GRIDS += [(108, 108), (72, 36), (54, 12), (36, 162)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("NX,NY", sorted(set(GRIDS)))
def test_pressure_solve_length(NX, NY, precision):
    import oracle_py as op
    import turbchannel_b200 as tb

    scheme = VV4 if NX % 4 else HW2
    prod, orc, zz = make_case(scheme, NX, NY, 7, precision=precision)
    S = tb.Solver(prod, zz)
    O = op.Oracle(orc, zz, "f64")
    v = seeded_field(S.N, NX * NY, seed=17)
    want = O.pressure_solve(O.apply_divergence(v))
    rhs = O.apply_divergence(v)
    if precision == 0:
        # from the vector: divergence, transforms, solve
        err = rel_err(S.UnapplyGradient(v), want)
        err_s = rel_err(S.LinearSystemSolveFFT(rhs), want)
        S.close()
        assert within(f"fft/{NX}x{NY}/p0/vec", err, 1e-10), err
        assert within(f"fft/{NX}x{NY}/p0/scalar", err_s, 1e-10), err_s
        return
    r32 = v[:, 0] - v[:, 0].mean()
    r32 = r32.astype(np.float32).astype(np.float64)
    want = O.pressure_solve(r32)
    got = S.LinearSystemSolveFFT(r32)
    S.close()
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert within(f"fft/{NX}x{NY}/p1", err, 2.4e-6), err


@pytest.mark.parametrize("NX", [384, 512, 768, 972, 1024])
def test_inverse_x_tiles(NX):
    """The float inverse x-transform with several tiles per CTA: the first pass over its own
    tile (two CTAs per SM at 512, one at 1024), in a buffer of its own (768), and with more
    line segments than threads (972).  The bound is the one above."""
    import oracle_py as op
    import turbchannel_b200 as tb

    prod, orc, zz = make_case(HW2, NX, 1024, 7, precision=1)
    S = tb.Solver(prod, zz)
    r32 = np.random.default_rng(23).standard_normal(S.N)
    r32 = (r32 - r32.mean()).astype(np.float32).astype(np.float64)
    want = op.Oracle(orc, zz, "f64").pressure_solve(r32)
    got = S.LinearSystemSolveFFT(r32)
    S.close()
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert within(f"fft/{NX}x1024/p1/tiles", err, 2.4e-6), err
