"""The persistent factorisation's counters: they are kept modulo 2^32 and go on
across factorisations, so a handle that has made many gives the same bits as a new
one (one chain and both ends, both precisions), and one that gave up on a wait
leaves the handle usable.  The wait is made to run out by a count that nothing
raises, with a short limit of polls; every CTA returns."""
import numpy as np
import pytest

from _cases import M, params_pair, state

pytestmark = pytest.mark.gpu

DT = 0.01


def _patch():
    p, _ = params_pair(M.ALEVB, M.F_PULL, 9, 9, pull_speed=0.5)
    mesh = M.Mesh(p)
    return p, mesh, *state(p, mesh, seed=2, amp=1e-3)


def _steps(s, xms, cps, k=2):
    s.upload(xms, cps)
    s.run_analysis([DT] * k)
    return s.download()


# the meeting's count passes 2^31 and 2^32 by itself, epoch x 32 columns at 2^26 and 2^27
@pytest.mark.parametrize("count", [2 ** 31 - 100, 2 ** 31 - 2, 2 ** 32 - 100, 2 ** 32 - 3, 2 ** 26 - 2, 2 ** 27 - 2])
@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_counters_wrap(count, precision):
    p, mesh, xms, cps = _patch()
    for ctas in (0, 1):
        with M.Solver(mesh, p, precision) as s:
            s.set_launch_ctas(ctas)
            x0, c0 = _steps(s, xms, cps)
            s.set_lu_count(count)
            x1, c1 = _steps(s, xms, cps)
            assert np.array_equal(x0, x1) and np.array_equal(c0, c1)


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_a_factorisation_that_gave_up_leaves_the_handle_usable(precision):
    p, mesh, xms, cps = _patch()
    with M.Solver(mesh, p, precision) as s:
        x0, c0 = _steps(s, xms, cps)
        assert s.lu_form() == M.FORM_BOTH_ENDS
        s.set_lu_count(5, missing=1, limit_polls=20000)
        s.upload(xms, cps)
        with pytest.raises(M.MafemError) as e:
            s.time_step_resident(DT, DT)
        assert e.value.code == M.ERR_CUDA and "bounded wait" in str(e.value)
        x1, c1 = s.download()
        assert np.array_equal(x1, xms) and np.array_equal(c1, cps)  # the state is left alone
        x1, c1 = _steps(s, xms, cps)
        assert np.array_equal(x0, x1) and np.array_equal(c0, c1)
