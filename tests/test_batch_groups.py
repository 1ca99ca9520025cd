"""A patch of a batched FP32 round gives the same bits whichever patches are beside
it: the round's groups (by CTAs per patch) are refined in different ways -- the
first one's sweeps and residuals in launches of their own, the others' in one
kernel -- and which group a patch is in depends on the others."""
import numpy as np
import pytest

from _cases import M, params_pair, state

pytestmark = pytest.mark.gpu

DT = 0.01


def _run(cases, graphs=True):
    """cases: (motion, n1, n2, CTAs); states after two steps of one batch."""
    solvers = []
    try:
        for k, (motion, n1, n2, ctas) in enumerate(cases):
            p, _ = params_pair(motion, M.F_PULL, n1, n2, pull_speed=0.05, pull_centre=1)
            mesh = M.Mesh(p)
            xms, cps = state(p, mesh, seed=n1, amp=1e-4)
            s = M.Solver(mesh, p, M.FP32_REFINE)
            s.upload(xms, cps)
            s.set_patch_ctas(ctas)
            solvers.append(s)
        with M.Batch(solvers) as b:
            assert b.set_patch_solve(True)
            b.set_rounds(True, graphs)
            t, sweeps = 0.0, []
            for _ in range(2):
                t += DT
                status, st = b.step(t, DT)
                assert status == [M.OK] * len(cases)
                sweeps.append([x["refine_iters"] for x in st])
        return [s.download() for s in solvers], sweeps
    finally:
        for s in solvers:
            s.close()


# the patch looked at (one row block per warp and several; narrow and wide bands)
@pytest.mark.parametrize("case", [(M.ALEVB, 12, 12), (M.LAG, 9, 14), (M.ALEVB, 16, 16), (M.LAG, 33, 9),
                                  (M.ALEVB, 28, 6)])
def test_bits_do_not_depend_on_the_group(case):
    (ref, *_), sw = _run([case + (1,)])
    small, big, wide = (M.LAG, 6, 6), (M.ALEVB, 18, 18), (M.ALEVB, 33, 9)
    for cases in ([case + (1,), small + (1,)], [case + (1,), big + (4,)], [case + (2,), big + (4,), small + (1,)],
                  [case + (4,), wide + (4,)], [case + (1,), big + (2,), wide + (1,)]):
        (got, *_), sw2 = _run(cases)
        assert [s[0] for s in sw2] == [s[0] for s in sw]
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), cases
