"""The factorisation's bounded waits: with the nodes handed out backwards on one
CTA and a short limit the first wait runs out.  The kernel ends, the solve
returns -1 and keeps no factors, also for a mode that reuses them, and the same
context then factorises and solves as before, bit for bit."""
import numpy as np
import pytest

from goma_gb300 import _lib
from goma_gb300 import problem as pb
from goma_gb300.newton import GomaNewton
from tests.test_gpu_line_sweeps import cavity, cube, system

pytestmark = pytest.mark.gpu

CASES = {"cube": lambda: cube(3, 2, 2), "cavity": lambda: cavity(8, 8),
         "reacting": lambda: pb.reacting_channel_3d(2, 2, 2)}


@pytest.mark.parametrize("ordering", [0, 1], ids=["natural", "multicoloured"])
@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("name", list(CASES))
def test_factorisation_wait_gives_up_and_the_context_recovers(name, fp32, ordering):
    prob = CASES[name]()
    ija, N, a, b = system(prob, 5)
    gn = GomaNewton(prob)
    gn.set_ilu_ordering(ordering)
    opts = dict(linear_tol=1e-10, max_linear_its=100, krylov_dim=30, fp32_preconditioner=fp32)
    want = gn.linear_solve(a, b, **opts)
    assert want[2] <= 1e-10
    gn.set_factor_fault(spin_limit=10000, reverse=True)
    with pytest.raises(_lib.GbError, match="dependency wait gave up"):
        gn.linear_solve(a, b, **dict(opts, max_linear_its=2))
    if ordering == 0:
        with pytest.raises(_lib.GbError, match="dependency wait gave up"):
            gn.ilu0_factors(a, fp32=fp32)
    gn.set_factor_fault()
    got = gn.linear_solve(a, b, **opts)
    assert got[1] == want[1] and np.array_equal(got[0], want[0])
    gn.close()


def test_no_factors_are_reused_after_it():
    prob = pb.lid_cavity_2d(6, 100.0)
    opts = dict(residual_tol=1e-10, linear_tol=1e-10, max_linear_its=500)
    gn = GomaNewton(prob)
    want, conv, _ = gn.solve_nonlinear_problem(None, **opts)
    assert conv
    gn.set_factor_fault(spin_limit=10000, reverse=True)
    with pytest.raises(_lib.GbError, match="dependency wait gave up"):
        gn.solve_nonlinear_problem(None, **dict(opts, max_linear_its=2))
    gn.set_factor_fault()
    x, conv, st = gn.solve_nonlinear_problem(None, factorization_reuse=2, **opts)
    assert conv and st["factorizations"] >= 1
    assert np.abs(x - want).max() <= 1e-8 * np.abs(want).max()
    gn.close()
