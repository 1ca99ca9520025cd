"""The batched FP32 solve of a patch whose working vector does not fit one CTA's
shared memory (110 x 110 LAG, 49 k unknowns): it takes the patch, does not hand it
back, and its step is the plain FP64 solver's within the FP32 form's 1e-8; a small
patch refined by the same kernel keeps the bits it has alone."""
import numpy as np
import pytest

from _cases import M, params_pair, rel, state

pytestmark = pytest.mark.gpu

DT = 0.01


def _solver(motion, n, precision, speed, amp):
    p, _ = params_pair(motion, M.F_PULL, n, n, pull_speed=speed, pull_centre=1)
    mesh = M.Mesh(p)
    xms, cps = state(p, mesh, seed=n, amp=amp)
    s = M.Solver(mesh, p, precision)
    s.upload(xms, cps)
    return s


def _step(solvers):
    with M.Batch(solvers) as b:
        assert b.set_patch_solve(True)
        status, _ = b.step(DT, DT)
        assert status == [M.OK] * len(solvers)
    return [s.download() for s in solvers]


def test_110x110_patch_in_the_batched_fp32_solve():
    small = _solver(M.ALEVB, 16, M.FP32_REFINE, 0.05, 1e-4)
    with small:
        small.set_patch_ctas(4)
        (ref,) = _step([small])
    big, small = _solver(M.LAG, 110, M.FP32_REFINE, 5e-4, 0.0), _solver(M.ALEVB, 16, M.FP32_REFINE, 0.05, 1e-4)
    with big, small:
        assert big.nmdf * 4 > 185 * 1024  # beside 40 KB of the sweeps' other buffers
        for s in (big, small):
            s.set_patch_ctas(4)
        (xb, cb), (xs, cs) = _step([big, small])
        assert big.fallback_count() == 0
    assert np.array_equal(xs, ref[0]) and np.array_equal(cs, ref[1])
    with _solver(M.LAG, 110, M.PLAIN_FP64, 5e-4, 0.0) as s:
        s.predict(DT)
        s.time_step_resident(DT, DT)
        x, c = s.download()
    assert rel(xb, x) < 1e-8 and rel(cb, c) < 1e-8
