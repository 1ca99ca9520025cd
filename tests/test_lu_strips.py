"""The elimination from both ends on strips one and two elements wide, whose bands
are narrower than a panel, and which form of the factorisation a band takes: both
solves in both precisions, with the tolerances of test_lu_two_ends.py."""
import numpy as np
import pytest

from _cases import M, O, params_pair, state
from test_lu_two_ends import backward_error

pytestmark = pytest.mark.gpu

# half bandwidths below 32: the forward chain's panel at the meeting is wider than its
# reach (1 x 31 cavity: panel [64, 96), the backward chain reaches down to 80)
STRIPS = [(M.STATIC, M.F_CAVI, 1, 31), (M.STATIC, M.F_CAVI, 2, 22), (M.STATIC, M.F_COUE, 2, 24),
          (M.STATIC, M.F_POIS, 1, 24), (M.LAG, M.F_BEND, 1, 28), (M.LAG, M.F_PULL, 1, 27), (M.STATIC, M.F_CAVI, 1, 127)]


def _setup(motion, scenario, n1, n2):
    p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh = M.Mesh(p)
    return p, mesh, state(p, mesh, seed=6, amp=1e-2, vel_amp=0.02)


@pytest.mark.parametrize("motion,scenario,n1,n2", STRIPS)
def test_strips_match_the_matrix(motion, scenario, n1, n2):
    p, mesh, (xms, cps) = _setup(motion, scenario, n1, n2)
    n, kl = mesh.nmdf, mesh.half_bw
    assert kl < 32
    with M.Solver(mesh, p) as s:
        r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
        K = O.band_to_csr(ab, kl, kl, n)
        for b in (r, 2.0 * r):  # the first rides along the factorisation, the second uses the stored factors
            assert backward_error(K, s.solve(b), b) < n * 2.0 ** -53 * 1e3
        assert s.lu_form() == M.FORM_BOTH_ENDS and s.fallback_count() == 0
    with M.Solver(mesh, p, M.FP32_REFINE) as s:
        s.set_refinement(60, 1e-10)
        r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
        K = O.band_to_csr(ab, kl, kl, n)
        for b in (r, -2.0 * r):
            assert np.linalg.norm(K @ s.solve(b) + b) <= 1e-10 * np.linalg.norm(b) * (1 + 1e-3)
        assert s.lu_form() == M.FORM_BOTH_ENDS and s.fallback_count() == 0


@pytest.mark.parametrize("motion,n1,n2,form", [
    (M.ALEVB, 6, 5, M.FORM_ONE_CHAIN), (M.LAG, 5, 9, M.FORM_ONE_CHAIN), (M.LAG, 8, 8, M.FORM_BOTH_ENDS),
    (M.ALEVB, 17, 17, M.FORM_BOTH_ENDS), (M.ALEVB, 68, 11, M.FORM_BOTH_ENDS)])
@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_form_of_the_factorisation(motion, n1, n2, form, precision):
    p, mesh, (xms, cps) = _setup(motion, M.F_PULL, n1, n2)
    width = 32 if mesh.half_bw < 600 else 16  # the widest panels of these bands
    assert (M.two_chain_plan(mesh, precision, width) is not None) == (form == M.FORM_BOTH_ENDS)
    with M.Solver(mesh, p, precision) as s:
        assert s.lu_form() == M.FORM_NONE
        for path, want in ((M.LU_AUTO, form), (M.LU_PANELS, M.FORM_PANELS), (M.LU_FULL, M.FORM_FULL)):
            s.set_lu_path(path)
            r, _ = s.calc_r_K(xms, cps, 0.01, 0.01, tangent=False)
            s.solve(r)
            assert s.lu_form() == want
