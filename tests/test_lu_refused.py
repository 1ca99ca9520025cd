"""Refused cooperative launches: per-panel launches take over from the persistent
factorisation and single-CTA kernels from the cooperative substitutions, for the
factors of one chain and of both ends, from any of a substitution's launches on.
Tolerances of test_lu_two_ends.py."""
import numpy as np
import pytest

from _cases import M, O, params_pair, state
from test_lu_two_ends import backward_error

pytestmark = pytest.mark.gpu

# one chain; from both ends: half bandwidths below and above a panel's width, a last panel of few unknowns
CASES = [(M.LAG, M.F_PULL, 5, 9), (M.STATIC, M.F_CAVI, 1, 31), (M.LAG, M.F_PULL, 8, 8), (M.ALEVB, M.F_PULL, 3, 40),
         (M.ALEVB, M.F_PULL, 17, 17), (M.EUL, M.F_BEND, 11, 16)]


@pytest.mark.parametrize("motion,scenario,n1,n2", CASES)
@pytest.mark.parametrize("factor,solve", [(False, 0), (False, 1), (True, -1), (True, 0)])
def test_solves_match_the_matrix(motion, scenario, n1, n2, factor, solve):
    p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh = M.Mesh(p)
    n, kl = mesh.nmdf, mesh.half_bw
    xms, cps = state(p, mesh, seed=6, amp=1e-2, vel_amp=0.02)
    two = M.two_chain_plan(mesh) is not None
    for precision in (M.PLAIN_FP64, M.FP32_REFINE):
        with M.Solver(mesh, p, precision) as s:
            s.set_refinement(60, 1e-10)
            r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
            K = O.band_to_csr(ab, kl, kl, n)
            s.set_coop_test(factor, solve)
            for b in (r, -2.0 * r):  # the second with the stored factors
                x = s.solve(b)
                if precision == M.PLAIN_FP64:
                    assert backward_error(K, x, b) < n * 2.0 ** -53 * 1e3
                else:
                    assert np.linalg.norm(K @ x + b) <= 1e-10 * np.linalg.norm(b) * (1 + 1e-3)
            assert s.lu_form() == (M.FORM_PANELS if factor else M.FORM_BOTH_ENDS if two else M.FORM_ONE_CHAIN)
            s.set_coop_test()
            s.set_launch_ctas(0)  # all kernels again
            s.calc_r_K(xms, cps, 0.01, 0.01, tangent=False)
            s.solve(r)
            assert s.lu_form() == (M.FORM_BOTH_ENDS if two else M.FORM_ONE_CHAIN)
