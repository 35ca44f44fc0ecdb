"""Chained products (H·psi and boundary steps of plans with few terms per line, in one
launch) and K-split stage-3 problems on the device, against the oracle and against the
GEMM stages (pinned variants), at sizes around the tiles: blocks of 1 to 33 rows (the chain
takes up to 32; K1 and rows in blocks of 8, columns in tiles of 8, K2 in steps of 4)."""
import numpy as np
import pytest

from dmrgb200 import _capi as capi
from dmrgb200 import engine as E
from dmrgb200 import models as M
from dmrgb200 import mps as S
from dmrgb200 import su2u1 as SU
from helpers import OracleChain, make_chain, random_psi

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# sums of at most a few thousand FP64 products in another order: a few hundred roundings of
# 1.1e-16, taken together in the 2-norm
TOL = 1e-13


def _plan(ctx, ch):
    Lb, Rb = E.to_device(ch.Lval), E.to_device(ch.Rval)
    plan = E.DevicePlan(ctx, ch.sched.plan, left_addr=ch.Lidx.cohort_addresses(Lb.data_ptr()),
                        other_addr=ch.Ridx.cohort_addresses(Rb.data_ptr()))
    return plan, (Lb, Rb)


def one_cohort_plan(ls, rs, ns, n, trans):
    """One T task (x times one block), one cohort of ns MPO rows, every row a multiple of T: y =
    sum over b of L_b (alpha_b T) with K = ns ls."""
    u = lambda *v: np.array(v, dtype=np.uint32)
    rows = np.arange(ns, dtype=np.uint32)
    return {
        "kind": 0, "in_size": ls * n, "out_size": rs * n, "g_t": u(0, 1), "g_c": u(0, 1),
        "in_rows": u(ls), "in_cols": u(n), "in_off": np.array([0], np.uint64),
        "out_rows": u(rs), "out_cols": u(n), "out_off": np.array([0], np.uint64),
        "t_lb": u(0), "t_col": u(0), "t_ci": u(0), "t_trans": np.zeros(1, np.uint8), "t_nb": u(1),
        "t_brows": u(n), "t_bcols": u(n), "t_width": u(),
        "c_lb": u(0), "c_rb": u(0), "c_ls": u(ls), "c_rs": u(rs), "c_ci": u(0), "c_trans": np.array([trans], np.uint8),
        "c_nsrows": u(ns), "c_stripe": u(n), "c_out_ci": u(0), "c_unit": u(0, 1),
        "u_offset": u(0), "u_ms": u(n), "u_line": u(0, ns), "l_b1": rows, "l_term": np.arange(ns + 1, dtype=np.uint32),
        "term_alpha": np.random.default_rng(7).standard_normal(ns), "term_t": 0 * rows, "term_col": 0 * rows}


@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("ls,rs,ns,n,parts", [(63, 40, 200, 33, 16), (64, 33, 12, 64, 1), (63, 70, 13, 40, 2), (33, 34, 250, 17, 11)])
def test_split_up_to_the_most_parts(ls, rs, ns, n, parts, trans):
    """K of 768 (whole) to 12600 (the most parts, 16) in one segment or, transposed, in ns."""
    plan = one_cohort_plan(ls, rs, ns, n, trans)
    form = E.lowering(plan)
    assert not form.chained and (form.stage3_parts == parts or trans)
    rng = np.random.default_rng(ns)
    x, B = rng.standard_normal((ls, n)), rng.standard_normal((n, n))
    L = rng.standard_normal((ns, rs, ls))
    Lb = E.to_device((L.transpose(0, 1, 2) if trans else L.transpose(0, 2, 1)).reshape(-1))  # column-major blocks
    Rb, xd = E.to_device(B.T.reshape(-1)), E.to_device(x.T.reshape(-1))
    p = E.DevicePlan(E.Context(0), plan, left_addr=np.array([Lb.data_ptr()], np.uint64),
                     other_addr=np.array([Rb.data_ptr()], np.uint64))
    ref = np.einsum("b,bij->ij", plan["term_alpha"], L.astype(np.longdouble)) @ (x.astype(np.longdouble) @ B)
    for v in range(capi.lib.dmrgb200_gemm_variant_count()):
        p.set_gemm_variants(0, v)
        yd = torch.full((rs * n,), float("nan"), dtype=torch.float64, device="cuda")
        p.hpsi(xd.data_ptr(), yd.data_ptr())
        torch.cuda.synchronize()
        y = yd.cpu().numpy().reshape(n, rs).T
        # 12600 products whose sum is about a hundredth of the sum of their sizes
        assert float(np.linalg.norm(y - ref) / np.linalg.norm(ref)) <= 1e-13, v


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("name,L,m,i,chained", [
    ("heisenberg", 12, 5, 5, True), ("heisenberg", 16, 64, 3, True), ("heisenberg", 20, 80, 9, True),
    ("heisenberg", 20, 230, 9, False), ("hubbard", 8, 12, 0, False), ("hubbard", 12, 60, 5, True),
    ("hubbard", 14, 333, 4, True), ("hubbard", 14, 600, 6, True), ("hubbard", 14, 660, 6, False), ("bose", 10, 40, 8, True)])
def test_chain_matches_oracle_and_stages(name, L, m, i, chained):
    ctx = E.Context(0)
    model, bonds, tensors, rng = make_chain(name, L, 0, seed=m, synthetic_m=m)
    ch = OracleChain(model, bonds, tensors, i)
    assert bool(E.lowering(ch.sched.plan).chained) == chained
    plan, keep = _plan(ctx, ch)
    x = random_psi(ch.p12, ch.left, ch.right, rng).data
    xd = E.to_device(x)
    yd = torch.full_like(xd, np.nan)
    ref = ch.hpsi(x)
    mask = np.zeros(len(ref), bool)
    p = ch.sched.plan
    for r, c, o in zip(p["out_rows"], p["out_cols"], p["out_off"]):
        mask[int(o):int(o) + int(r) * int(c)] = True
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    torch.cuda.synchronize()
    y = yd.cpu().numpy()
    assert np.all(np.isnan(y[~mask]))  # the padding of y is left untouched
    assert _rel(y[mask], ref[mask]) <= TOL
    # host buffers run the same launch between two copies
    xh = torch.from_numpy(x.copy()).pin_memory()
    yh = torch.zeros_like(xh).pin_memory()
    plan.hpsi_host(xh.data_ptr(), yh.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(yh.numpy()[mask], y[mask])
    # pinned variants run the GEMM stages, with host buffers too
    plan.set_gemm_variants(0, 0)
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    plan.hpsi_host(xh.data_ptr(), yh.data_ptr())
    torch.cuda.synchronize()
    staged = yd.cpu().numpy()
    assert _rel(staged[mask], ref[mask]) <= TOL
    assert np.array_equal(yh.numpy()[mask], staged[mask])


@pytest.mark.parametrize("name,L,m", [("heisenberg", 12, 5), ("heisenberg", 16, 130), ("hubbard", 10, 40), ("hubbard", 12, 333)])
@pytest.mark.parametrize("symmetric", [True, False])
def test_chain_steps_match_oracle(name, L, m, symmetric):
    """Left steps from the left end and right steps from the right end to the middle."""
    ctx = E.Context(0)
    model, bonds, tensors, _ = make_chain(name, L, 0, seed=3, synthetic_m=m)
    for left in (True, False):
        idx = E.edge_bindex(model.symm, bonds[0] if left else bonds[L])
        val = idx.edge_values()
        buf = E.to_device(val)
        for p in (range(L // 2) if left else range(L - 1, L // 2, -1)):
            W, t = M.MPOHandle(model.mpo[p], model.symm), tensors[p]
            if left:
                sch, nidx = E.schedule_left_step(model.phys, bonds[p], bonds[p + 1], W, idx, symmetric)
                val = O.left_step(sch.plan, val, idx, t.data, t.left_paired(), nidx)
                plan = E.DevicePlan(ctx, sch.plan, left_addr=idx.cohort_addresses(buf.data_ptr()))
                ket, bra = E.to_device(t.data), E.to_device(t.left_paired())
            else:
                sch, nidx = E.schedule_right_step(model.phys, bonds[p], bonds[p + 1], W, idx, symmetric)
                val = O.right_step(sch.plan, val, idx, t.data, t.data, nidx)
                plan = E.DevicePlan(ctx, sch.plan, other_addr=idx.cohort_addresses(buf.data_ptr()))
                ket = bra = E.to_device(t.data)
            out = torch.zeros(max(nidx.n_elems, 1), dtype=torch.float64, device="cuda")
            plan.step(ket.data_ptr(), bra.data_ptr(), nidx.cohort_addresses(out.data_ptr()))
            assert _rel(out.cpu().numpy()[:len(val)], val) <= TOL
            idx, buf = nidx, out


def test_chain_non_finite_boundary_stays_local():
    """An infinite boundary element reaches the outputs that read it, as in the oracle, and
    no others."""
    ctx = E.Context(0)
    model, bonds, tensors, rng = make_chain("hubbard", 10, 0, seed=2, synthetic_m=50)
    ch = OracleChain(model, bonds, tensors, 4)
    x = random_psi(ch.p12, ch.left, ch.right, rng).data
    ch.Lval = ch.Lval.copy()
    ch.Lval[int(ch.Lidx.storage_off[0])] = np.inf
    plan, keep = _plan(ctx, ch)
    xd = E.to_device(x)
    yd = torch.zeros_like(xd)
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    torch.cuda.synchronize()
    y, ref = yd.cpu().numpy(), ch.hpsi(x)
    fine = np.isfinite(ref)
    assert not fine.all() and np.all(np.isfinite(y[fine]))
    assert _rel(y[fine], ref[fine]) <= TOL


@pytest.mark.parametrize("L,m,parts", [(8, 100, 1), (10, 150, 3), (12, 200, 6)])
def test_split_stage3_matches_oracle(L, m, parts):
    """Quantum chemistry in SU2U1 form: few output blocks with long K ranges, cut into parts
    (K of up to a few thousand against parts of at least 48 steps of 16)."""
    ctx = E.Context(0)
    model = SU.quantum_chemistry(L, L, 0)
    bonds = SU.synthetic_bonds(L, model.total_charge, m)
    rng = np.random.default_rng(4)
    tensors = S.random_mps(SU.PHYS, bonds, rng)
    ch = OracleChain(model, bonds, tensors, L // 2 - 1)
    assert E.lowering(ch.sched.plan).stage3_parts == parts
    plan, keep = _plan(ctx, ch)
    x = rng.standard_normal(int(ch.sched.plan["in_size"]))
    xd = E.to_device(x)
    yd = torch.zeros_like(xd)
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    torch.cuda.synchronize()
    y, ref = yd.cpu().numpy(), ch.hpsi(x)
    # the lines' sums here have hundreds of terms: a thousand roundings
    assert _rel(y, ref) <= 1e-12
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(yd.cpu().numpy(), y)  # parts are added in order, whichever arrives last


@pytest.mark.parametrize("L,m,drop", [(10, 150, 3), (8, 60, 2)])
def test_blocks_without_a_cohort_are_zero(L, m, drop):
    """Output blocks that no cohort writes come out as zeros, not as what y held, with stage 3
    cut into K parts and not, from device and from host buffers."""
    ctx = E.Context(0)
    model = SU.quantum_chemistry(L, L, 0)
    bonds = [list(b) for b in SU.synthetic_bonds(L, model.total_charge, m)]
    bonds[L // 2 - 2] = bonds[L // 2 - 2][drop:]
    rng = np.random.default_rng(4)
    ch = OracleChain(model, bonds, S.random_mps(SU.PHYS, bonds, rng), L // 2 - 1)
    p = ch.sched.plan
    assert len(set(p["c_rb"].tolist())) < len(p["out_rows"])
    plan, keep = _plan(ctx, ch)
    x = rng.standard_normal(int(p["in_size"]))
    ref = ch.hpsi(x)
    mask = np.zeros(len(ref), bool)
    for r, c, o in zip(p["out_rows"], p["out_cols"], p["out_off"]):
        mask[int(o):int(o) + int(r) * int(c)] = True
    xd = E.to_device(x)
    yd = torch.full((len(ref),), np.nan, dtype=torch.float64, device="cuda")
    xh, yh = torch.from_numpy(x.copy()).pin_memory(), torch.full((len(ref),), np.nan, dtype=torch.float64).pin_memory()
    plan.hpsi(xd.data_ptr(), yd.data_ptr())
    plan.hpsi_host(xh.data_ptr(), yh.data_ptr())
    torch.cuda.synchronize()
    for y in (yd.cpu().numpy(), yh.numpy()):
        assert _rel(y[mask], ref[mask]) <= 1e-12
        assert np.all(y[mask][ref[mask] == 0.0] == 0.0)


@pytest.mark.parametrize("name,L,m,i", [("heisenberg", 16, 64, 7), ("hubbard", 14, 333, 4)])
def test_chained_hpsi_in_place(name, L, m, i):
    """y = x, y overlapping x, and y over the right boundary's blocks: the oracle's H·psi, and
    the bits of the stages (chained products would read what other CTAs have overwritten)."""
    ctx = E.Context(0)
    model, bonds, tensors, rng = make_chain(name, L, 0, seed=m, synthetic_m=m)
    ch = OracleChain(model, bonds, tensors, i)
    assert E.lowering(ch.sched.plan).chained
    x = random_psi(ch.p12, ch.left, ch.right, rng).data
    ref, n = ch.hpsi(x), len(x)
    plan, keep = _plan(ctx, ch)
    pinned, keep2 = _plan(ctx, ch)
    pinned.set_gemm_variants(0, 0)
    buf = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    xd, staged = E.to_device(x), torch.zeros(n, dtype=torch.float64, device="cuda")
    pinned.hpsi(xd.data_ptr(), staged.data_ptr())
    for shift in (0, 0, 0, 0, 8, 128, n // 2):
        buf[:n] = xd
        buf[n:] = 0.0
        plan.hpsi(buf.data_ptr(), buf[shift:].data_ptr())
        torch.cuda.synchronize()
        mask = torch.from_numpy(ref != 0.0).cuda()
        assert _rel(buf[shift:shift + n][mask].cpu().numpy(), ref[ref != 0.0]) <= TOL, shift
        assert torch.equal(buf[shift:shift + n][mask], staged[mask]), shift
    # y at the start of the right boundary's storage (which it overwrites)
    Lb = E.to_device(ch.Lval)
    Rb = torch.zeros(max(len(ch.Rval), n), dtype=torch.float64, device="cuda")
    Rb[:len(ch.Rval)] = E.to_device(ch.Rval)
    over = E.DevicePlan(ctx, ch.sched.plan, left_addr=ch.Lidx.cohort_addresses(Lb.data_ptr()),
                        other_addr=ch.Ridx.cohort_addresses(Rb.data_ptr()))
    over.hpsi(xd.data_ptr(), Rb.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(Rb[:n][mask], staged[mask])


@pytest.mark.parametrize("name,L,m", [("heisenberg", 16, 64), ("hubbard", 12, 333)])
def test_chained_steps_in_place(name, L, m):
    """New boundaries written over the old ones, and over the ket, from the ends to the middle."""
    ctx = E.Context(0)
    model, bonds, tensors, _ = make_chain(name, L, 0, seed=3, synthetic_m=m)
    chained = 0
    for left in (True, False):
        idx = E.edge_bindex(model.symm, bonds[0] if left else bonds[L])
        val = idx.edge_values()
        for p in (range(L // 2) if left else range(L - 1, L // 2, -1)):
            W, t = M.MPOHandle(model.mpo[p], model.symm), tensors[p]
            if left:
                sch, nidx = E.schedule_left_step(model.phys, bonds[p], bonds[p + 1], W, idx, True)
                ref = O.left_step(sch.plan, val, idx, t.data, t.left_paired(), nidx)
                bra = E.to_device(t.left_paired())
            else:
                sch, nidx = E.schedule_right_step(model.phys, bonds[p], bonds[p + 1], W, idx, True)
                ref = O.right_step(sch.plan, val, idx, t.data, t.data, nidx)
                bra = E.to_device(t.data)
            chained += int(E.lowering(sch.plan).chained)
            for over in ("boundary", "ket"):
                old = torch.zeros(max(len(val), len(ref)), dtype=torch.float64, device="cuda")
                old[:len(val)] = E.to_device(val)
                ket = torch.zeros(max(len(t.data), len(ref)), dtype=torch.float64, device="cuda")
                ket[:len(t.data)] = E.to_device(t.data)
                addr = idx.cohort_addresses(old.data_ptr())
                plan = E.DevicePlan(ctx, sch.plan, **({"left_addr": addr} if left else {"other_addr": addr}))
                out = old if over == "boundary" else ket
                plan.step(ket.data_ptr(), bra.data_ptr(), nidx.cohort_addresses(out.data_ptr()))
                got = out.cpu().numpy()[:len(ref)]  # the gaps between cohorts keep what was there
                assert _rel(got[ref != 0.0], ref[ref != 0.0]) <= TOL, (left, p, over)
            idx, val = nidx, ref
    assert chained >= L // 2


@pytest.mark.parametrize("large_first", [True, False])
@pytest.mark.parametrize("staged", [False, True])
def test_terms_of_a_line_are_summed_one_by_one(large_first, staged):
    """A line of two terms, one of them 2^30 times a small integer without rounding, the other a
    sum of 32 products of unit normals: each term is summed by itself, so the only rounding
    at the size of the large one is that of the sum (half a unit in the last place, 2^-23 below
    2^31; the small term's own roundings are below 2^-43).  Adding the 32 products one by one to the
    large term would round 32 times."""
    u = lambda *v: np.array(v, dtype=np.uint32)
    ls, k2, n = 8, 32, 8
    big, small = (0, 1) if large_first else (1, 0)  # column slice and boundary cohort
    plan = {
        "kind": 0, "in_size": ls * 2 * k2, "out_size": ls * n, "g_t": u(0, 2), "g_c": u(0, 1),
        "in_rows": u(ls), "in_cols": u(2 * k2), "in_off": np.array([0], np.uint64),
        "out_rows": u(ls), "out_cols": u(n), "out_off": np.array([0], np.uint64),
        "t_lb": u(0, 0), "t_col": u(0, k2), "t_ci": u(0, 1), "t_trans": np.zeros(2, np.uint8), "t_nb": u(1, 1),
        "t_brows": u(k2, k2), "t_bcols": u(n, n), "t_width": u(),
        "c_lb": u(0), "c_rb": u(0), "c_ls": u(ls), "c_rs": u(ls), "c_ci": u(0), "c_trans": np.zeros(1, np.uint8),
        "c_nsrows": u(1), "c_stripe": u(n), "c_out_ci": u(0), "c_unit": u(0, 1),
        "u_offset": u(0), "u_ms": u(n), "u_line": u(0, 1), "l_b1": u(0), "l_term": u(0, 2),
        "term_alpha": np.ones(2), "term_t": u(0, 1), "term_col": u(0, 0)}
    assert E.lowering(plan).chained
    rng = np.random.default_rng(5)
    x = np.zeros((2, ls, k2))  # the two slices
    B = np.zeros((2, k2, n))
    x[big, :, 0] = rng.integers(1, 2, ls) * 2.0 ** 30
    B[big, 0, :] = 1.0
    x[small], B[small] = rng.standard_normal((ls, k2)), rng.standard_normal((k2, n))
    ctx = E.Context(0)
    Lb = E.to_device(np.eye(ls).reshape(-1))
    Rb = E.to_device(B.transpose(0, 2, 1).reshape(-1))  # each block column-major
    p = E.DevicePlan(ctx, plan, left_addr=np.array([Lb.data_ptr()], np.uint64),
                     other_addr=np.array([Rb.data_ptr(), Rb.data_ptr() + 8 * k2 * n], np.uint64))
    if staged:
        p.set_gemm_variants(0, 0)
    xd = E.to_device(np.concatenate([x[0].T.reshape(-1), x[1].T.reshape(-1)]))
    yd = torch.zeros(ls * n, dtype=torch.float64, device="cuda")
    p.hpsi(xd.data_ptr(), yd.data_ptr())
    torch.cuda.synchronize()
    ref = sum(x[i].astype(np.longdouble) @ B[i].astype(np.longdouble) for i in (0, 1))
    err = np.abs(yd.cpu().numpy().reshape(n, ls).T - ref)
    assert float(err.max()) <= 2.0 ** -23 * (1 + 2.0 ** -15)
