"""Shared memory of the z-solve's tiles around the 48 KB that a kernel may use without asking
(csrc/k_zsolve.cu): sizes whose dynamic part stays below the line and crosses it together with
the static part, each as the first solver of a process of its own, since the limit of a kernel
outlives the solver that raised it.

Tolerances.  FP64: 1e-10 relative to the largest pressure, as the other solve tests.  Mixed: in
the 2-norm against the FP64 solve of the same 32-bit white noise.  The transforms give 2.4e-6.
The float sweeps perturb every row's 2/dz by its rounding e = 6e-8; the modes outside the double
set (k >= 4) answer with exp(-k |z - z'|) / (2k), and the independent errors of the rows within
1/k add up to e k^-3/2 dz^-3/2 of the solution, e (NZ / 8)^3/2 at dz = 2 / NZ.  Eight times that
covers the smaller spacing at the walls (2.4 times) and the roundings of the sweeps themselves."""
import os
import subprocess
import sys

import numpy as np
import pytest

from cases import COLLOC, HW2, VV4, make_case, rel_err, seeded_field, within

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
from cases import make_case
import turbchannel_b200 as tb
scheme, NX, NY, NZ, precision = (int(a) for a in sys.argv[1:6])
prod, _, zz = make_case(scheme, NX, NY, NZ, precision=precision, gamma=1.0)
S = tb.Solver(prod, zz)
np.save(sys.argv[7], S.LinearSystemSolveFFT(np.load(sys.argv[6])))
S.close()
"""


def _solve_in_child(tmp_path, scheme, NX, NY, NZ, precision, rhs):
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.environ.get("PYTHONPATH", "")]))
    a, b = str(tmp_path / "rhs.npy"), str(tmp_path / "p.npy")
    np.save(a, rhs)
    r = subprocess.run([sys.executable, "-c", CHILD, *map(str, (scheme, NX, NY, NZ, precision)), a, b], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(b)


@pytest.mark.parametrize("scheme,NX,NY,NZ,precision", [
    (HW2, 16, 16, 490, 0), (COLLOC, 32, 32, 482, 0),  # two pairs per tile
    (HW2, 64, 64, 490, 1),  # four
    (HW2, 32, 32, 1000, 1), (COLLOC, 16, 16, 990, 1), (VV4, 16, 16, 750, 1),  # two
])
def test_first_solver_of_a_process(tmp_path, scheme, NX, NY, NZ, precision):
    import oracle_py as op

    _, orc, zz = make_case(scheme, NX, NY, NZ, precision=precision, gamma=1.0)
    O = op.Oracle(orc, zz, "f64")
    if precision == 0:
        coll = scheme == COLLOC
        v = seeded_field(NX * NY * NZ, NX * NY, seed=3, wall_w_zero=not coll)
        if coll:
            v[:NX * NY] = 0.0
            v[-NX * NY:] = 0.0
        rhs = O.apply_divergence(v)
        err = rel_err(_solve_in_child(tmp_path, scheme, NX, NY, NZ, precision, rhs), O.pressure_solve(rhs))
        tol = 1e-10
    else:
        rhs = np.random.default_rng(3).standard_normal(NX * NY * NZ)
        rhs = (rhs - rhs.mean()).astype(np.float32).astype(np.float64)
        want = O.pressure_solve(rhs)
        err = np.linalg.norm(_solve_in_child(tmp_path, scheme, NX, NY, NZ, precision, rhs) - want) / np.linalg.norm(want)
        tol = 2.4e-6 + 8 * 6e-8 * (NZ / 8) ** 1.5
    assert within(f"smem/{scheme}/{NX}x{NY}x{NZ}/p{precision}", err, tol), err


def test_refused_launch_is_reported(tmp_path):
    """A column that no tile holds: the z-solve's launch is refused, and the call says so although
    it is the process's first and other kernels are set up after it."""
    with pytest.raises(AssertionError, match="pressure_solve"):
        _solve_in_child(tmp_path, VV4, 16, 16, 8000, 1, np.zeros(16 * 16 * 8000))


def test_solvers_of_two_threads():
    """Two threads, each with its own solver, both of them using the same tile kernel with columns
    of different length: neither takes back the shared memory that the other has asked for."""
    import threading

    import torch

    import turbchannel_b200 as tb

    failed = []

    def work(NZ):
        try:
            prod, _, zz = make_case(HW2, 16, 16, NZ, gamma=1.0)
            S = tb.Solver(prod, zz)
            r = torch.zeros(256 * NZ, device="cuda", dtype=torch.float64)
            p = torch.empty_like(r)
            torch.cuda.synchronize()
            for k in range(3000):
                S.pressure_solve_device(r.data_ptr(), p.data_ptr())
                if k % 100 == 99:
                    S.sync()
            S.close()
        except Exception as e:  # noqa: BLE001
            failed.append((NZ, str(e)))

    ts = [threading.Thread(target=work, args=(nz,)) for nz in (600, 1000)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed
