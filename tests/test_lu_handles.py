"""A handle's factorisation does not depend on which other handles exist."""
import pytest

from _cases import M, params_pair, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
def test_a_narrow_handle_leaves_a_wide_one_its_persistent_factorisation(precision):
    def make(motion, n):
        p, _ = params_pair(motion, M.F_PULL, n, n)
        mesh = M.Mesh(p)
        return M.Solver(mesh, p, precision), state(p, mesh, seed=1, amp=1e-3)

    wide, (xw, cw) = make(M.ALEVB, 24)
    forms = []
    with wide:
        for other in (None, (M.LAG, 5), (M.LAG, 8)):  # a one-chain band, one that goes from both ends
            if other:
                s, (x, c) = make(*other)
                with s:
                    s.time_step(x, c, 0.01, 0.01)
            r, _ = wide.calc_r_K(xw, cw, 0.01, 0.01, tangent=False)
            wide.solve(r)
            forms.append(wide.lu_form())
    assert forms == [M.FORM_BOTH_ENDS] * 3
