"""The block form of the batched FP32 factorisation as the numpy model restates it
(oracle/patch_lu_model.py): the explicit inverse of a panel's diagonal block by one
Gauss-Jordan sweep with node-block pivots, and the factors Ai, Y and raw A21."""
import numpy as np
import pytest

from _cases import M, O, params_pair, state
import patch_lu_model as PM

U32 = 2.0 ** -24


def _tangent(motion, n1, n2, kb=0.5):
    p, q = params_pair(motion, M.F_PULL, n1, n2, kb=kb, pull_speed=0.01)
    mesh, om = M.Mesh(p), O.Mesh(q)
    xms, cps = state(p, mesh, seed=3, amp=1e-4)
    om.update_xms(xms, cps, 0.005)
    r, ab = om.calc_r_K(xms, cps, 0.005, 0.005, nthreads=2)
    return om, r, ab.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("w", [1, 2, 7, 8, 9, 31, 32])
def test_gauss_jordan_is_the_inverse(w):
    """Node blocks of four whose last unknown has a zero on the diagonal (a Lagrange
    multiplier), so that rows are exchanged: the row-wise residual bound of a
    Gauss-Jordan inverse, w steps of one product and one sum each on entries of at
    most |A| |A^-1| before them, grown by at most the largest multiplier chain, which
    these blocks keep below 2^6."""
    rng = np.random.default_rng(w)
    D = rng.standard_normal((w, w)).astype(np.float32)
    bend = np.minimum((np.arange(w) // 4 + 1) * 4, w)
    for k in range(3, w, 4):
        D[k, k] = 0.0
    D += np.float32(4.0) * np.kron(np.eye((w + 3) // 4), np.roll(np.eye(4), 1, axis=1))[:w, :w].astype(np.float32)
    if w % 4:  # a last block cut short keeps its own pivots
        q = w - w % 4
        D[q:, q:] += np.float32(4.0) * np.eye(w - q, dtype=np.float32)
    inv = PM.gauss_jordan(D, bend).astype(np.float64)
    A = D.astype(np.float64)
    bound = 2 * w * U32 * 64 * (np.abs(A) @ np.abs(np.linalg.inv(A))).max() * np.linalg.norm(np.linalg.inv(A), np.inf)
    assert np.abs(inv - np.linalg.inv(A)).max() <= bound


def test_no_usable_pivot_is_reported():
    D = np.eye(8, dtype=np.float32)
    D[4:8, 5] = 0.0
    D[0, 5] = 1.0  # outside column 5's node block
    with pytest.raises(ZeroDivisionError):
        PM.gauss_jordan(D, np.repeat([4, 8], 4))


@pytest.mark.parametrize("motion,n1,n2", [(M.LAG, 1, 28), (M.LAG, 8, 8), (M.EUL, 7, 11), (M.ALEVB, 9, 9),
                                          (M.ALEVB, 16, 10)])
def test_block_form_solves_and_contracts(motion, n1, n2):
    """One pass with the factors leaves a residual that the next one contracts tenfold
    or better, down to the solution of an FP64 solve of the same FP32 tangent."""
    om, r, ab0 = _tangent(motion, n1, n2)
    kl, n = om.half_bw, len(r)
    lu = PM.PatchLU(ab0, kl, PM.node_blocks(om.ID_inv))
    assert lu.growth < 1e4
    x, hist = PM.refine(lu, ab0, kl, -r, tol=1e-10)
    assert len(hist) <= 8
    assert all(b <= 0.1 * a for a, b in zip(hist[1:-1], hist[2:])), hist
    K = PM.dense_from_band(ab0, kl, np.float64)
    assert np.linalg.norm(x - np.linalg.solve(K, -r)) <= 1e-8 * np.linalg.norm(x)
