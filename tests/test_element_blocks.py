"""Element blocks at the edges of the element kernel's work split: strips one
element wide (two opposite sides, so up to four Neumann entries, on one
element), the smallest patches, and element counts that leave a partial CTA of
the batched tangent kernel, in every motion.  Against the oracle with the
parity tests' tolerances: FP64 rounding of r and K (1e-12, 1e-11 of the largest
entry), FP32 rounding of the FP32 form's K (2e-5)."""
import pytest

from _cases import M, O, params_pair, rel, state

pytestmark = pytest.mark.gpu

CASES = [(m, M.F_PULL, n1, n2) for m in (M.LAG, M.EUL, M.ALEV, M.ALEVB) for n1, n2 in ((1, 1), (1, 4), (3, 1), (5, 3))]
CASES += [(m, M.F_BEND, n1, n2) for m in (M.LAG, M.EUL, M.ALEV) for n1, n2 in ((1, 3), (4, 1))]
CASES += [(M.STATIC, sc, 1, 3) for sc in (M.F_CAVI, M.F_COUE, M.F_POIS)]


@pytest.mark.parametrize("motion,scenario,n1,n2", CASES)
def test_blocks_match_oracle(motion, scenario, n1, n2):
    p, q = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh, om = M.Mesh(p), O.Mesh(q)
    xms, cps = state(p, mesh, seed=11, amp=2e-2, vel_amp=0.05)
    time, dt, kl = 0.37, 0.01, mesh.half_bw
    r0, ab0 = om.calc_r_K(xms, cps, time, dt, nthreads=2)
    for precision, tol in ((M.PLAIN_FP64, 1e-11), (M.FP32_REFINE, 2e-5)):
        with M.Solver(mesh, p, precision) as s:
            r, ab = s.calc_r_K(xms, cps, time, dt)
        assert rel(r, r0) < 1e-12
        assert rel(ab[:, kl:], ab0[:, kl:]) < tol
