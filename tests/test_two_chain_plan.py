"""The plan of the elimination from both ends (CPU): until the two chains meet, no
entry of the band and no right-hand side entry is touched by both.  Strips one to
six elements wide, whose bands can be narrower than a panel, and square patches, in
every motion and scenario and for every panel width a handle may take."""
import numpy as np
import pytest

from _cases import M, params_pair

KINDS = [(M.STATIC, M.F_CAVI), (M.STATIC, M.F_COUE), (M.STATIC, M.F_POIS), (M.LAG, M.F_BEND), (M.EUL, M.F_BEND),
         (M.ALEV, M.F_BEND)] + [(m, M.F_PULL) for m in (M.LAG, M.EUL, M.ALEV, M.ALEVB)]
SHAPES = [(n1, n2) for n1 in range(1, 7) for n2 in range(4, 90, 3 if n1 > 2 else 1)] + [(60, 1), (31, 2), (12, 12), (24, 21)]


def touched(ps, p, end, kl, kuf, first):
    """Rows and columns (half-open) that panel p writes: its block and the rows below
    (as read by the update), Y and the trailing block; first: its block alone."""
    j0, j1 = int(ps[p]), int(ps[p + 1])
    return (j0, j1, j0, j1) if first else (j0, min(end, j1 + kl), j0, min(end, j1 + kuf))


def check(mesh, width):
    """True if the plan has two chains (then checked), False for one."""
    try:
        plan = M.two_chain_plan(mesh, M.PLAIN_FP64, width)
    except M.MafemError as e:  # a band too wide for panels of this width
        assert e.code == M.ERR_UNSUPPORTED and mesh.half_bw > 600 and width > 8
        return False
    if plan is None:
        return False
    kuf, mid, pm, ps0, ps1 = plan
    n, kl = mesh.nmdf, mesh.half_bw
    assert ps0[0] == 0 and ps0[-1] == mid and ps1[0] == 0 and ps1[-1] == n - mid and kl <= kuf
    assert np.all(np.diff(ps0) > 0) and np.all(np.diff(ps1) > 0)
    assert 0 < pm < len(ps0) - 1
    # before the meeting: panels 0 .. pm - 1 of the forward chain, the factorisation of
    # panel pm's block (whose CTA does not wait), and the whole backward chain
    fwd = [touched(ps0, p, mid, kl, kuf, p == pm) for p in range(pm + 1)]
    bwd = [touched(ps1, p, n, kl, kuf, False) for p in range(len(ps1) - 1)]
    f, b = np.array(fwd), np.array(bwd)
    b = np.stack([n - b[:, 1], n - b[:, 0], n - b[:, 3], n - b[:, 2]], axis=1)  # in the matrix's numbering
    over = ((np.maximum(f[:, None, 0], b[None, :, 0]) < np.minimum(f[:, None, 1], b[None, :, 1])) &
            (np.maximum(f[:, None, 2], b[None, :, 2]) < np.minimum(f[:, None, 3], b[None, :, 3])))
    assert not over.any(), (mesh.num1el, mesh.num2el, n, kuf, mid, pm, ps0, ps1)
    # the right-hand side rides along: rows alone (panel pm carries none before the meeting)
    assert f[:pm, 1].max() <= b[:, 0].min()
    # the substitutions: what is solved between the chains holds every unknown either one needs
    assert ps0[pm] <= mid - kuf
    return True


@pytest.mark.parametrize("motion,scenario", KINDS)
def test_chains_are_apart_until_they_meet(motion, scenario):
    two = narrow = 0
    for n1, n2 in SHAPES:
        p, _ = params_pair(motion, scenario, n1, n2, bend_mf=0.5, bend_tm=2.0)
        mesh = M.Mesh(p)
        for width in (32, 24, 16, 8):
            if check(mesh, width):
                two += 1
                narrow += mesh.half_bw < 32
    assert two > 0
    if motion in (M.STATIC, M.LAG):
        assert narrow > 0  # bands narrower than a panel are among them


def test_one_chain_for_short_bands_and_bad_arguments():
    p, _ = params_pair(M.ALEVB, M.F_PULL, 6, 5)
    mesh = M.Mesh(p)
    assert M.two_chain_plan(mesh) is None
    for width in (0, 33):
        with pytest.raises(M.MafemError):
            M.two_chain_plan(mesh, M.PLAIN_FP64, width)
