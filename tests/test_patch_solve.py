"""The batched FP32 solve on one, two and four CTAs per patch, and what the
factorisations leave in the bands for the next one.

First sweep: the factors contract the residual to |r| <= n u g |r0|, u = 2^-24 the
FP32 rounding and g <= 100 the growth of the entries under pivoting inside node
blocks; the refinement then ends with its own criterion.
"""
import numpy as np
import pytest

from _cases import M, O, params_pair, state

pytestmark = pytest.mark.gpu


# half bandwidths below a panel's width, up to one register set of the update warps
# (480), beyond it (543) and an odd mixture; last panels of a few unknowns
@pytest.mark.parametrize("motion,n1,n2", [(M.LAG, 2, 9), (M.LAG, 5, 5), (M.ALEVB, 6, 6), (M.ALEVB, 13, 17),
                                          (M.LAG, 33, 9), (M.ALEVB, 28, 5), (M.ALEVB, 33, 9)])
def test_factors_contract_on_any_cluster(motion, n1, n2):
    p, _ = params_pair(motion, M.F_PULL, n1, n2)
    mesh = M.Mesh(p)
    xms, cps = state(p, mesh, seed=8, amp=1e-3)
    with M.Solver(mesh, p, M.FP32_REFINE) as s:
        s.upload(xms, cps)
        for ctas in (1, 2, 4):
            s.set_patch_ctas(ctas)
            s.trace_patch_solve(0.01, 0.01)
            assert s.last_refine_status[0] == M.OK
            assert s.last_refine_residuals[0] <= mesh.nmdf * 2.0 ** -24 * 100


@pytest.mark.parametrize("motion,n1,n2", [(M.LAG, 8, 8), (M.ALEVB, 5, 9)])
def test_batch_step_after_the_own_solver_is_the_same(motion, n1, n2):
    """The handle's own elimination from both ends fills rows below the band that a
    round's gather has to clear."""
    p, _ = params_pair(motion, M.F_PULL, n1, n2)
    mesh = M.Mesh(p)
    xms, cps = state(p, mesh, seed=8, amp=1e-3)
    out = []
    for own in (False, True):
        with M.Solver(mesh, p, M.FP32_REFINE) as s:
            if own:
                s.solve(s.calc_r_K(xms, cps, 0.01, 0.01)[0])
            s.upload(xms, cps)
            with M.Batch([s]) as b:
                st, _ = b.step(0.01, 0.01)
            assert st == [M.OK]
            if own:  # and the other way round
                r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
                s.set_launch_ctas(0)
                x = s.solve(r)
                K = O.band_to_csr(ab, mesh.half_bw, mesh.half_bw, mesh.nmdf)
                assert np.linalg.norm(K @ x + r) <= 1e-10 * np.linalg.norm(r) * (1 + 1e-3)  # the default criterion
                s.upload(xms, cps)
                with M.Batch([s]) as b:
                    assert b.step(0.01, 0.01)[0] == [M.OK]
            out.append(s.download())
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_bands_are_clean_after_full_pivoting_and_a_callers_band(precision):
    p, _ = params_pair(M.ALEVB, M.F_PULL, 6, 7)
    mesh = M.Mesh(p)
    n, kl = mesh.nmdf, mesh.half_bw
    xms, cps = state(p, mesh, seed=9, amp=1e-2, vel_amp=0.02)
    with M.Solver(mesh, p, precision) as s:
        r, ab = s.calc_r_K(xms, cps, 0.01, 0.01)
        first = s.solve(r)
        s.set_lu_path(M.LU_FULL)
        s.calc_r_K(xms, cps, 0.01, 0.01)
        s.solve(r)
        s.set_lu_path(M.LU_AUTO)
        assert np.array_equal(s.calc_r_K(xms, cps, 0.01, 0.01)[1], ab)
        assert np.array_equal(s.solve(r), first)
        full = np.random.default_rng(1).standard_normal(ab.shape)
        i = np.arange(n)[:, None] + np.arange(ab.shape[1])[None, :] - 2 * kl  # row of entry (j, q)
        full[(i < 0) | (i >= n) | (np.arange(ab.shape[1])[None, :] < kl)] = 0.0
        full[:, 2 * kl] += 100.0 * kl  # dominant diagonal
        s.solve_band(full, r)
        assert np.array_equal(s.calc_r_K(xms, cps, 0.01, 0.01)[1], ab)
        assert np.array_equal(s.solve(r), first)
