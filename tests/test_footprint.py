"""mafem_footprint_bytes is what mafem_create allocates: admission counts on it."""
import pytest

from _cases import M, params_pair

pytestmark = pytest.mark.gpu

CASES = [(M.LAG, M.F_PULL, 4, 4), (M.ALEVB, M.F_PULL, 5, 7), (M.LAG, M.F_PULL, 1, 27), (M.ALEVB, M.F_PULL, 16, 16),
         (M.STATIC, M.F_CAVI, 13, 12), (M.EUL, M.F_BEND, 11, 16), (M.ALEVB, M.F_PULL, 33, 9), (M.LAG, M.F_PULL, 40, 40),
         (M.ALEVB, M.F_PULL, 68, 11)]


@pytest.mark.parametrize("precision", [M.PLAIN_FP64, M.FP32_REFINE])
@pytest.mark.parametrize("motion,scenario,n1,n2", CASES)
def test_footprint_is_what_a_handle_holds(motion, scenario, n1, n2, precision):
    p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
    mesh = M.Mesh(p)
    with M.Solver(mesh, p, precision) as s:
        held = s.device_bytes
    want = M.footprint_bytes(mesh, precision)
    assert held <= want <= 1.02 * held + 4096
