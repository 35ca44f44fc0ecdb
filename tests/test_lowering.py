"""The form a plan is lowered to (host work, no device): which plans run as chained
products, which output blocks are cut into K parts, what stage 1 forms."""
import numpy as np
import pytest

from dmrgb200 import _capi as capi
from dmrgb200 import engine as E
from dmrgb200 import models as M
from dmrgb200 import su2u1 as SU


def hpsi_plan(model, bonds, i):
    """The two-site H·psi plan at (i, i + 1)."""
    L, phys = len(model.mpo), model.phys
    handle = lambda p: M.MPOHandle(model.mpo[p], model.symm)
    Lidx, Ridx = E.edge_bindex(model.symm, bonds[0]), E.edge_bindex(model.symm, bonds[L])
    for p in range(i):
        _, Lidx = E.schedule_left_step(phys, bonds[p], bonds[p + 1], handle(p), Lidx, True)
    for p in range(L - 1, i + 1, -1):
        _, Ridx = E.schedule_right_step(phys, bonds[p], bonds[p + 1], handle(p), Ridx, True)
    p12, _ = M.fuse_phys(phys, phys)
    W = M.MPOHandle(M.twosite_for(model, i), model.symm)
    return E.schedule_hpsi(p12, bonds[i], bonds[i + 2], W, Lidx, Ridx).plan


def qc_bonds(model, L, m, i=None, drop=0):
    """Synthetic bonds, the first `drop` sectors of bond i - 1 left out: then the left boundary
    of bond i reaches only some of its sectors."""
    bonds = [list(b) for b in SU.synthetic_bonds(L, model.total_charge, m)]
    if drop:
        bonds[i - 1] = bonds[i - 1][drop:]
    return bonds


def test_null_arguments_are_refused():
    assert capi.lib.dmrgb200_plan_lowering(None, None) == capi.INVALID_ARGUMENT


@pytest.mark.parametrize("L,m,i,drop,cut", [(12, 300, 5, 0, True), (12, 300, 5, 2, True), (12, 300, 5, 4, True),
                                            (10, 150, 4, 3, True), (8, 60, 3, 2, False)])
def test_blocks_without_a_cohort_stay_in_stage3(L, m, i, drop, cut):
    """Output blocks that no cohort writes are set to zero by stage 3, also where its long K
    ranges are cut into parts."""
    model = SU.quantum_chemistry(L, L, 0)
    plan = hpsi_plan(model, qc_bonds(model, L, m, i, drop), i)
    form = E.lowering(plan)
    assert (form.stage3_parts > 1) == cut and not form.chained
    empty = len(plan["out_rows"]) - len(set(plan["c_rb"].tolist()))
    assert (empty > 0) == (drop > 1)
    assert form.stage3_zero_blocks == empty


@pytest.mark.parametrize("L,m,sites", [(12, 300, range(1, 10)), (16, 512, (2, 3, 4, 5, 6, 7, 9))])
def test_quantum_chemistry_stage1_keeps_its_stacked_rows(L, m, sites):
    """Leaving out T blocks that no term reads never costs tile steps: left of the middle each
    task reads a set of its own, and problems by set would undo the row stacking."""
    model = SU.quantum_chemistry(L, L, 0)
    bonds = SU.synthetic_bonds(L, model.total_charge, m)
    for i in sites:
        form = E.lowering(hpsi_plan(model, bonds, i))
        assert 0 < form.stage1_steps <= form.stage1_steps_whole, i


@pytest.mark.parametrize("model,width,m,i,share", [(M.fermi_hubbard(64), 3.5, 1024, 31, 0.70), (M.fermi_hubbard(64), 3.5, 1600, 10, 0.70),
                                                   (M.heisenberg(32), 10.0, 1024, 15, 0.81)])
def test_lattice_stage1_leaves_unread_blocks_out(model, width, m, i, share):
    """On lattice chains a fifth to a third of the T blocks is read by no term."""
    from dmrgb200 import mps as S
    bonds = S.synthetic_bonds(model.phys, len(model.mpo), model.total_charge, m, width)
    form = E.lowering(hpsi_plan(model, bonds, i))
    assert not form.chained and form.stage1_steps <= share * form.stage1_steps_whole
