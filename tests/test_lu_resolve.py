"""Solves with stored FP64 factors on tangents whose diagonal blocks are
ill-conditioned (strips and small patches of the ALE motions, nearly singular): as
accurate as the solve that rides along the factorisation, by the cooperative kernels
and by the single-CTA ones."""
import numpy as np
import pytest

from _cases import M, O, params_pair, state

pytestmark = pytest.mark.gpu

CASES = [(M.ALEV, 1, 16), (M.ALEV, 4, 3), (M.ALEV, 10, 1), (M.ALEV, 1, 40), (M.ALEVB, 1, 30), (M.ALEVB, 18, 2),
         (M.ALEVB, 28, 1), (M.ALEVB, 22, 2), (M.ALEVB, 5, 4), (M.ALEVB, 3, 15), (M.ALEVB, 2, 27)]


@pytest.mark.parametrize("motion,n1,n2", CASES)
def test_second_solve_is_backward_stable(motion, n1, n2):
    """Normwise backward error: a row's sum has at most 2 (kl + 8) + 64 terms, each
    with a rounding of 2^-53 of its size; 16 for the growth of the elimination and
    of the triangles' inverses (first solves measured: 2e-15 at most)."""
    for kb, amp, seed in ((0.5, 1e-5, 1), (2.0, 1e-3, 2), (1.0, 1e-4, 3)):
        p, _ = params_pair(motion, M.F_PULL, n1, n2, kb=kb, pull_speed=0.02)
        mesh = M.Mesh(p)
        n, kl = mesh.nmdf, mesh.half_bw
        xms, cps = state(p, mesh, seed=seed, amp=amp)
        bound = 16 * (2 * (kl + 8) + 64) * 2.0 ** -53
        with M.Solver(mesh, p) as s:
            for path, solve in ((M.LU_AUTO, -1), (M.LU_AUTO, 0), (M.LU_PANELS, -1)):
                s.set_coop_test()
                s.set_launch_ctas(0)
                s.set_lu_path(path)
                r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
                K = O.band_to_csr(ab, kl, kl, n)
                s.solve(r)
                s.set_coop_test(False, solve)
                b = 2.0 * r
                x = s.solve(b)
                assert np.abs(K @ x + b).max() <= bound * ((abs(K) @ np.abs(x)).max() + np.abs(b).max()), (kb, path, solve)
