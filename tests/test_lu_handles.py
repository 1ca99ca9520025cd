"""A handle's factorisation does not depend on which other handles exist."""
import pytest

from _cases import M, params_pair, rel, state

pytestmark = pytest.mark.gpu


def _make(motion, n, precision):
    p, _ = params_pair(motion, M.F_PULL, n, n)
    mesh = M.Mesh(p)
    return M.Solver(mesh, p, precision), state(p, mesh, seed=1, amp=1e-3)


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_a_narrow_handle_leaves_a_wide_one_its_persistent_factorisation(precision):
    wide, (xw, cw) = _make(M.ALEVB, 24, precision)
    forms = []
    with wide:
        for other in (None, (M.LAG, 5), (M.LAG, 8)):  # a one-chain band, one that goes from both ends
            if other:
                s, (x, c) = _make(*other, precision)
                with s:
                    s.time_step(x, c, 0.01, 0.01)
            r, _ = wide.calc_r_K(xw, cw, 0.01, 0.01, tangent=False)
            wide.solve(r)
            forms.append(wide.lu_form())
    assert forms == [M.FORM_BOTH_ENDS] * 3


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_a_narrow_handle_leaves_a_wide_one_its_stored_factors(precision):
    """Full partial pivoting: a second solve runs the forward substitution's own kernel."""
    wide, (xw, cw) = _make(M.ALEVB, 12, precision)
    with wide:
        wide.set_lu_path(M.LU_FULL)
        r, _ = wide.calc_r_K(xw, cw, 0.01, 0.01, tangent=False)
        first = wide.solve(r)
        narrow, _ = _make(M.LAG, 4, precision)
        with narrow:
            second = wide.solve(r)
    assert rel(second, first) < 1e-6  # the same factors, so rounding only (times a condition below 1e9)
