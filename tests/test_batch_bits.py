"""What a patch's result may not depend on: the CTAs its factorisation is given and
the patches beside it in a batch.  The same bits are asked for."""
import numpy as np
import pytest

from _cases import M, params_pair, state

pytestmark = pytest.mark.gpu

DT = 0.01


def _patch(motion, n1, n2, seed, **kw):
    p, _ = params_pair(motion, M.F_PULL, n1, n2, pull_speed=0.05, pull_centre=1, **kw)
    mesh = M.Mesh(p)
    return p, mesh, *state(p, mesh, seed=seed, amp=1e-4)


# a short band (one chain), bands eliminated from both ends, one of them many panels long
PATCHES = [(M.LAG, 5, 9), (M.LAG, 8, 8), (M.ALEVB, 9, 9), (M.EUL, 7, 11), (M.ALEVB, 17, 17), (M.LAG, 24, 21)]


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_any_number_of_ctas_gives_the_same_bits(precision):
    for k, (motion, n1, n2) in enumerate(PATCHES):
        p, mesh, xms, cps = _patch(motion, n1, n2, k)
        with M.Solver(mesh, p, precision) as s:
            got = []
            for ctas in (0, 1, 40, 75, 100):
                s.set_launch_ctas(ctas)
                s.upload(xms, cps)
                s.run_analysis([DT] * 2)
                got.append((s.lu_form(), *s.download()))
            for f, x, c in got[1:]:
                assert f == got[0][0]
                assert np.array_equal(x, got[0][1]) and np.array_equal(c, got[0][2]), (motion, n1, n2)


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_patches_of_a_batch_equal_the_patches_alone(precision):
    """Each patch with its own solver (the batched FP32 solve off)."""
    alone, solvers = [], []
    try:
        for k, (motion, n1, n2) in enumerate(PATCHES):
            p, mesh, xms, cps = _patch(motion, n1, n2, k)
            s = M.Solver(mesh, p, precision)
            solvers.append(s)
            s.upload(xms, cps)
            s.run_analysis([DT] * 2)
            alone.append(s.download())
            s.upload(xms, cps)
        with M.Batch(solvers) as b:
            b.set_patch_solve(False)
            t = 0.0
            for _ in range(2):
                t += DT
                status, _ = b.step(t, DT)
                assert status == [M.OK] * len(PATCHES)
        for s, (x0, c0) in zip(solvers, alone):
            x, c = s.download()
            assert np.array_equal(x, x0) and np.array_equal(c, c0)
    finally:
        for s in solvers:
            s.close()
