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


def chain_limits(p):
    """Largest block dimension (rows of the output, K1) and number of eight-column tiles that a
    plan's chained form has, restated from the plan's arrays."""
    kind, dmax, tiles = p["kind"], 0, 0
    left = kind == capi.PLAN_LEFT
    seen = set()
    for c in range(len(p["c_lb"])):
        ls, rs = int(p["c_ls"][c]), int(p["c_rs"][c])
        rb = int(p["c_rb"][c])
        for u in range(p["c_unit"][c], p["c_unit"][c + 1]):
            ms = int(p["u_ms"][u])
            lines = range(p["u_line"][u], p["u_line"][u + 1])
            if ms and any(p["l_term"][x] < p["l_term"][x + 1] for x in lines):
                dmax = max(dmax, ls if kind == capi.PLAN_HPSI else ms)
            if kind == capi.PLAN_HPSI and rb not in seen and ms:
                tiles += (ms + 7) // 8
                dmax = max(dmax, int(p["out_rows"][rb]))
        seen.add(rb)
        if kind != capi.PLAN_HPSI:
            dmax = max(dmax, ls if left else rs)
            tiles += int(p["c_nsrows"][c]) * (((rs if left else ls) + 7) // 8)
    if kind == capi.PLAN_HPSI:
        for ob in set(range(len(p["out_rows"]))) - seen:
            dmax = max(dmax, int(p["out_rows"][ob]))
            tiles += (int(p["out_cols"][ob]) + 7) // 8
    return dmax, tiles


def step_plan(model, bonds, i, left):
    L, phys = len(model.mpo), model.phys
    handle = lambda p: M.MPOHandle(model.mpo[p], model.symm)
    idx = E.edge_bindex(model.symm, bonds[0] if left else bonds[L])
    build = E.schedule_left_step if left else E.schedule_right_step
    for p in (range(i) if left else range(L - 1, i, -1)):
        _, idx = build(phys, bonds[p], bonds[p + 1], handle(p), idx, True)
    return build(phys, bonds[i], bonds[i + 1], handle(i), idx, True)[0].plan


@pytest.mark.parametrize("name,L,width", [("heisenberg", 20, 10.0), ("heisenberg", 20, 3.5), ("hubbard", 16, 3.5),
                                          ("hubbard", 64, 3.5), ("bose", 10, 3.5)])
def test_plans_run_chained_exactly_within_the_limits(name, L, width):
    """Blocks of at most 32 rows (K1 too) in at most 2368 tiles, on both sides of each limit, for
    H·psi and both steps."""
    from dmrgb200 import mps as S
    model = {"heisenberg": M.heisenberg, "hubbard": M.fermi_hubbard, "bose": lambda n: M.bose_hubbard(n, N=n // 2)}[name](L)
    got = set()
    sizes = sorted({int(round(8 * 1.3 ** k)) for k in range(22)} | {40 * k for k in range(1, 30)}) if L < 64 else (400, 560, 600, 900)
    for m in sizes:
        bonds = S.synthetic_bonds(model.phys, L, model.total_charge, m, width)
        i = L // 2 - 1
        for p in (hpsi_plan(model, bonds, i), step_plan(model, bonds, i, True), step_plan(model, bonds, i, False)):
            form = E.lowering(p)
            dmax, tiles = chain_limits(p)
            if not tiles:
                continue
            few = len(p["term_alpha"]) <= 4 * len(p["l_b1"])
            assert bool(form.chained) == (few and dmax <= 32 and tiles <= 2368), (m, p["kind"], dmax, tiles)
            assert not form.chained or form.chain_tiles == tiles
            got.add(bool(form.chained))
    assert got == {True, False} or name == "bose"
