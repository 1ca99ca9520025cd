"""FP64 node-block LU from both ends (the path of a band at least 10/3 bandwidths
long on enough CTAs): the first solve, whose right-hand side rides along, the
second one with the stored factors, on any number of CTAs, against the matrix.

Tolerance: the normwise backward error |K x + r| / (|K| |x| + |r|) of an LU of n
unknowns is at most about n u g, u = 2^-53, g the growth of the entries; pivoting
inside node blocks has no bound on g of its own, and g <= 10^3 is required here.
"""
import ctypes as C

import numpy as np
import pytest

from _cases import M, O, params_pair, state

pytestmark = pytest.mark.gpu

# (motion, scenario, n1, n2): the shortest bands that qualify (LAG 5 x 9: chains of 5 and 2
# panels), the first ones too short, a long narrow band, every motion and scenario, the
# widest panel count, and a half bandwidth that leaves room for four staged columns only
CASES = [
    (M.LAG, M.F_PULL, 5, 9), (M.LAG, M.F_PULL, 8, 8), (M.ALEVB, M.F_PULL, 8, 8), (M.EUL, M.F_PULL, 5, 9),
    (M.ALEVB, M.F_PULL, 6, 5), (M.LAG, M.F_PULL, 12, 3),
    (M.ALEVB, M.F_PULL, 3, 40), (M.ALEV, M.F_PULL, 9, 21), (M.STATIC, M.F_CAVI, 13, 12),
    (M.STATIC, M.F_COUE, 12, 13), (M.STATIC, M.F_POIS, 12, 12), (M.LAG, M.F_BEND, 9, 17),
    (M.EUL, M.F_BEND, 11, 16), (M.ALEV, M.F_BEND, 10, 13), (M.ALEVB, M.F_PULL, 68, 11),
]


def backward_error(K, x, r):
    res = K @ x + r
    return np.abs(res).max() / (abs(K).sum(axis=1).max() * np.abs(x).max() + np.abs(r).max())


@pytest.mark.parametrize("motion,scenario,n1,n2", CASES)
def test_both_solves_match_the_matrix(motion, scenario, n1, n2):
    p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh = M.Mesh(p)
    n, kl = mesh.nmdf, mesh.half_bw
    xms, cps = state(p, mesh, seed=6, amp=1e-2, vel_amp=0.02)
    tol = n * 2.0 ** -53 * 1e3
    count = M.lib().mafem_fallback_count
    count.restype, count.argtypes = C.c_int64, [C.c_void_p]
    with M.Solver(mesh, p) as s:
        fb = []
        for ctas in (0, 1):  # all CTAs: from both ends; the fewest: from the first unknown
            s.set_launch_ctas(ctas)
            r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
            if ctas == 0:
                ab0 = ab
                K = O.band_to_csr(ab, kl, kl, n)
            assert np.array_equal(ab, ab0)  # the factors leave nothing behind
            f0 = count(s.h)
            assert backward_error(K, s.solve(r), r) < tol
            assert backward_error(K, s.solve(2.0 * r), 2.0 * r) < tol
            s.set_launch_ctas(1)
            assert backward_error(K, s.solve(-r), -r) < tol
            fb.append(count(s.h) - f0)
        assert fb[0] == fb[1]  # neither order needs full pivoting where the other does not
        s.set_launch_ctas(0)
        x = s.solve_band(ab0, r)
        assert backward_error(K, -x, r) < tol
        assert np.array_equal(s.calc_r_K(xms, cps, 0.01, 0.01)[1], ab0)


@pytest.mark.parametrize("motion,scenario,n1,n2", [c for c in CASES if c[2] < 68])
def test_fp32_factors_refine_to_the_stopping_rule(motion, scenario, n1, n2):
    """FP32 factors of both orders: the refinement in FP64 ends by its stopping
    rule |r - K x| <= 1e-10 |r| (2-norm) on the FP32 tangent."""
    p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh = M.Mesh(p)
    n, kl = mesh.nmdf, mesh.half_bw
    xms, cps = state(p, mesh, seed=6, amp=1e-2, vel_amp=0.02)
    with M.Solver(mesh, p, M.FP32_REFINE) as s:
        s.set_refinement(60, 1e-10)
        for ctas in (0, 1):
            s.set_launch_ctas(ctas)
            r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
            K = O.band_to_csr(ab, kl, kl, n)
            for b in (r, -2.0 * r):  # the second with the stored factors
                assert np.linalg.norm(K @ s.solve(b) + b) <= 1e-10 * np.linalg.norm(b) * (1 + 1e-3)
