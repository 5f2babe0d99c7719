"""The mixed form's z-solve on long columns: tiles of one and two pairs of modes next to the double
tiles of the low modes, with their factors in shared memory and, beyond what a CTA holds, in
global memory.

Tolerance: in the 2-norm against the FP64 solve of the same 32-bit white noise, derived in
test_smem_limit_gpu.py."""
import numpy as np
import pytest

from cases import COLLOC, HW2, VV4, make_case, within

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,NX,NY,NZ,low", [
    (VV4, 16, 16, 400, 0), (HW2, 24, 16, 400, 7), (HW2, 16, 24, 700, 0), (COLLOC, 16, 16, 700, 0),
    (COLLOC, 16, 18, 2000, 0), (VV4, 16, 16, 2000, 0), (VV4, 16, 16, 3700, 0), (HW2, 16, 16, 5000, 0),
])
def test_long_columns(scheme, NX, NY, NZ, low):
    import oracle_py as op
    import turbchannel_b200 as tb

    prod, orc, zz = make_case(scheme, NX, NY, NZ, precision=1, gamma=1.0, low_modes=low)
    rhs = np.random.default_rng(13).standard_normal(NX * NY * NZ)
    rhs = (rhs - rhs.mean()).astype(np.float32).astype(np.float64)
    want = op.Oracle(orc, zz, "f64").pressure_solve(rhs)
    S = tb.Solver(prod, zz)
    got = S.LinearSystemSolveFFT(rhs)
    S.close()
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert within(f"zsolve-mixed/{scheme}/{NX}x{NY}x{NZ}/{low}", err, 2.4e-6 + 8 * 6e-8 * (NZ / 8) ** 1.5), err


@pytest.mark.parametrize("scheme,NX,NY,NZ", [(HW2, 128, 128, 2300), (VV4, 128, 128, 2300), (COLLOC, 192, 128, 1530)])
def test_streamed_columns(scheme, NX, NY, NZ):
    """Grids whose columns are too long for tiles to fill the chip: both precisions stream, and
    differ by the mixed bound; the FP64 solution, on the staggered grids, satisfies its system
    (the divergence of its gradient, with the bound of test_zsolve_gpu's long columns)."""
    import torch

    import turbchannel_b200 as tb

    N = NX * NY * NZ
    r = torch.randn(N, device="cuda", dtype=torch.float64, generator=torch.Generator("cuda").manual_seed(3))
    r = (r - r.mean()).float()
    p = {}
    for precision in (0, 1):
        prod, _, zz = make_case(scheme, NX, NY, NZ, precision=precision, gamma=1.0)
        S = tb.Solver(prod, zz)
        rhs = r.double() if precision == 0 else r
        p[precision] = torch.empty_like(rhs)
        torch.cuda.synchronize()
        S.pressure_solve_device(rhs.data_ptr(), p[precision].data_ptr())
        S.sync()
        if precision == 0 and scheme != COLLOC:
            q = p[0].cpu().numpy()
            back = np.asarray(S.ApplyDivergence(S.ApplyGradient(q)))
            # less the plane means: the mean mode is singular, its pinned row keeps the sum of rhs
            want = r.double().cpu().numpy()
            diff = (back - want).reshape(NZ, -1)
            diff -= diff.mean(axis=1, keepdims=True)
            scale = 8.0 / np.diff(zz).min() * np.max(np.abs(q))
            assert np.max(np.abs(diff)) < 1e-13 * scale + 1e-12 * np.max(np.abs(want))
        S.close()
    err = float(torch.linalg.norm(p[1].double() - p[0]) / torch.linalg.norm(p[0]))
    assert within(f"zsolve-stream/{scheme}/{NX}x{NY}x{NZ}", err, 2.4e-6 + 8 * 6e-8 * (NZ / 8) ** 1.5), err
