"""Performance cases of the DMRG hot path: what a sweep spends its device time on.

A two-site sweep applies H·psi (alone or inside a Jacobi-Davidson solve), moves
the boundaries one site per step, splits the two-site tensor, and, for
derivatives, runs the adjoint.  The cases take each of these through its public
entry point, from a small spin chain, where launches are all there is, to an
ab-initio site problem that fills the card, in the three symmetries (U1, TwoU1,
SU2U1), in native and emulated FP64.

A case is {"op", "model", "sites", "m", "site"}:
  op     hpsi, emulated (H·psi with emulated contractions), solve, left_step,
         right_step, adjoint, batched, svd
  model  heisenberg (U1), hubbard (TwoU1), qc (SU2U1, spin-adapted)
  sites  chain length; m the bond dimension (synthetic sectors); site the first
         site of the two-site pair (the site of a boundary step)
and, for op = batched, "instances" (half Heisenberg, half Hubbard) with bond
dimensions log-uniform in [m_low, m].

The chain's structure (MPO, bond sectors, schedules) is fixed by the case, as it
is over the sweeps of one calculation; the numbers (boundaries, vectors) come
from the seed.  Boundary blocks are normal with magnitudes that fall off along
each sector's states, as the weights of a truncated state do; diagonal blocks are
symmetric, so the effective Hamiltonian is Hermitian like a real one.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "maquis-dmrg_b200"))

from dmrgb200 import _capi as capi  # noqa: E402
from dmrgb200 import dmrg as G  # noqa: E402
from dmrgb200 import engine as E  # noqa: E402
from dmrgb200 import models as M  # noqa: E402
from dmrgb200 import mps as S  # noqa: E402
from dmrgb200 import qc  # noqa: E402
from dmrgb200 import su2u1 as SU  # noqa: E402

F64 = torch.float64


def _case(name, op, model, sites, m, site, **more):
    return dict(name=name, op=op, model=model, sites=sites, m=m, site=site, **more)


def listed():
    return [
        # a small spin chain: every launch is mostly latency
        _case("hpsi_heisenberg_m64", "hpsi", "heisenberg", 32, 64, 15),
        # the flagship: middle pair of the L=64 Fermi-Hubbard chain at m=1024
        _case("hpsi_hubbard_m1024", "hpsi", "hubbard", 64, 1024, 31),
        # an ordinary off-centre pair with ragged sectors
        _case("hpsi_hubbard_m333", "hpsi", "hubbard", 20, 333, 6),
        # ab-initio, a small active space
        _case("hpsi_qc_12_m300", "hpsi", "qc", 12, 300, 5),
        # ab-initio, the largest: fills the card
        _case("hpsi_qc_20_m800", "hpsi", "qc", 20, 800, 9),
        # the ab-initio site problem with emulated contractions
        _case("emulated_qc_16_m512", "emulated", "qc", 16, 512, 7),
        # the eigen-solve of one site problem: 8 Davidson iterations
        _case("solve_hubbard_m1024", "solve", "hubbard", 64, 1024, 31),
        # moving the boundaries: lattice chain to the right, ab-initio to the left
        _case("left_step_hubbard_m1024", "left_step", "hubbard", 64, 1024, 30),
        _case("right_step_qc_12_m300", "right_step", "qc", 12, 300, 7),
        # derivatives with respect to psi and to every plan term
        _case("adjoint_qc_16_m512", "adjoint", "qc", 16, 512, 7),
        # independent site problems in one plan
        _case("batched_16_m512", "batched", "mixed", 32, 512, 15, instances=16, m_low=64),
        # the two-site split of the flagship's tensor
        _case("svd_hubbard_m1024", "svd", "hubbard", 64, 1024, 31),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["hpsi", "hpsi", "hpsi", "emulated", "solve", "left_step", "right_step", "adjoint", "batched", "svd"])
    if op == "batched":
        return dict(op=op, model="mixed", sites=2 * rng.randint(8, 16), m=log(80, 512), site=7, instances=2 * rng.randint(2, 10),
                    m_low=rng.randint(32, 72))
    model = rng.choice(["heisenberg", "hubbard", "hubbard"] if op in ("solve", "svd") else ["heisenberg", "hubbard", "qc"])
    if model == "heisenberg":
        sites, m = 2 * rng.randint(8, 32), log(32, 1024)
    elif model == "hubbard":
        sites, m = 2 * rng.randint(7, 32), log(64, 1024 if op == "svd" else 1600)
    else:
        sites, m = 2 * rng.randint(4, 8), log(64, 512)
    mid = sites // 2 - 1
    return dict(op=op, model=model, sites=sites, m=m, site=max(2, min(sites - 4, mid + rng.randint(-2, 2))))


# ---- structure (fixed by the case) ---------------------------------------------------

@functools.lru_cache(maxsize=4)
def _model(model, sites):
    if model == "heisenberg":
        return M.heisenberg(sites)
    if model == "hubbard":
        return M.fermi_hubbard(sites)
    h, eri = qc.synthetic_integrals(sites)
    return SU.quantum_chemistry(sites, sites, 0, h=h, eri=eri)


class Site:
    """Structure of one site problem: bond sectors, boundary indices, schedule."""

    def __init__(self, model, sites, m, site, kind="hpsi"):
        self.model = mod = _model(model, sites)
        phys = mod.phys
        if model == "qc":
            bonds = SU.synthetic_bonds(sites, mod.total_charge, m, 3.5)
        else:
            # the Heisenberg chain's charges are 2 Sz: a wider profile, as many sectors as a spin chain keeps
            bonds = S.synthetic_bonds(phys, sites, mod.total_charge, m, 10.0 if model == "heisenberg" else 3.5)
        self.bonds, self.site = bonds, site
        handle = lambda p: M.MPOHandle(mod.mpo[p], mod.symm)
        self.L = self.R = self.out = None
        if kind in ("hpsi", "left_step"):
            L = E.edge_bindex(mod.symm, bonds[0])
            for p in range(site):
                _, L = E.schedule_left_step(phys, bonds[p], bonds[p + 1], handle(p), L, True)
            self.L = L
        if kind in ("hpsi", "right_step"):
            R = E.edge_bindex(mod.symm, bonds[sites])
            for p in range(sites - 1, site + (1 if kind == "hpsi" else 0), -1):
                _, R = E.schedule_right_step(phys, bonds[p], bonds[p + 1], handle(p), R, True)
            self.R = R
        if kind == "hpsi":
            self.p12, self.offs = M.fuse_phys(phys, phys)
            self.W = M.MPOHandle(M.twosite_for(mod, site), mod.symm)
            self.schedule = E.schedule_hpsi(self.p12, bonds[site], bonds[site + 2], self.W, self.L, self.R)
        elif kind == "left_step":
            self.W = handle(site)
            self.schedule, self.out = E.schedule_left_step(phys, bonds[site], bonds[site + 1], self.W, self.L, True)
        elif kind == "right_step":
            self.W = handle(site)
            self.schedule, self.out = E.schedule_right_step(phys, bonds[site], bonds[site + 1], self.W, self.R, True)
        else:
            self.p12, self.offs = M.fuse_phys(phys, phys)
            self.psi = S.SiteTensor(self.p12, bonds[site], bonds[site + 2])
            self.split = G.DeviceSplitPlan(self.psi, phys, phys, self.offs)
        if kind != "svd":
            self.plan = self.schedule.plan


@functools.lru_cache(maxsize=24)
def _site(model, sites, m, site, kind):
    return Site(model, sites, m, site, kind)


def _kind(op):
    return op if op in ("left_step", "right_step", "svd") else "hpsi"


def _batch(case):
    """(model, m) of every instance: log-uniform bond dimensions, alternating models."""
    n, lo, hi = case["instances"], case["m_low"], case["m"]
    u = np.random.default_rng(6).random(n)
    return [("heisenberg" if i % 2 == 0 else "hubbard", int(round(lo * (hi / lo) ** u[i]))) for i in range(n)]


def _sites(case):
    if case["op"] == "batched":
        return [_site(mod, case["sites"], m, case["site"], "hpsi") for mod, m in _batch(case)]
    return [_site(case["model"], case["sites"], case["m"], case["site"], _kind(case["op"]))]


# ---- numbers (from the seed) -----------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


def _boundary(idx, gen):
    """Boundary values in the index's storage layout."""
    v = torch.randn(max(idx.n_elems, 1), dtype=F64, device="cuda", generator=gen)
    for ci in range(idx.n_cohorts):
        if not idx.has_storage(ci):
            continue
        o, l, r, n = int(idx.storage_off[ci]), int(idx.lsize[ci]), int(idx.rsize[ci]), int(idx.nblocks[ci])
        blk = v[o:o + l * r * n].view(n, r, l)
        wl = torch.exp(torch.arange(l, dtype=F64, device="cuda") * (-4.0 / l))
        wr = torch.exp(torch.arange(r, dtype=F64, device="cuda") * (-4.0 / r))
        blk *= (wr[:, None] * wl[None, :])
        if idx.lb[ci] == idx.rb[ci]:
            blk.copy_(0.5 * (blk + blk.transpose(1, 2)))
    return v


def _vector(rows, cols, offs, total, gen):
    """Unit vector in a block layout (padding zero)."""
    v = torch.zeros(int(total), dtype=F64, device="cuda")
    r = torch.randn(int(total), dtype=F64, device="cuda", generator=gen)
    for a, b, o in zip(rows, cols, offs):
        v[int(o):int(o) + int(a) * int(b)] = r[int(o):int(o) + int(a) * int(b)]
    return v / torch.linalg.norm(v)


def _psi(plan, gen, side="in"):
    return _vector(plan[side + "_rows"], plan[side + "_cols"], plan[side + "_off"], plan[side + "_size"], gen)


def _theta(split, gen):
    """Two-site blocks with falling singular values (eight decades, as a converged state's Schmidt spectrum)."""
    th = torch.zeros(max(split.th_elems, 1), dtype=F64, device="cuda")
    for mc in split.order:
        _, _, nr, nc, _ = split.blocks[mc]
        k = min(nr, nc)
        w = torch.exp(torch.arange(k, dtype=F64, device="cuda") * (-8.0 * math.log(10.0) / k))
        a = torch.randn(nc, k, dtype=F64, device="cuda", generator=gen)
        b = torch.randn(k, nr, dtype=F64, device="cuda", generator=gen)
        o = split.th_off[mc]
        th[o:o + nr * nc] = ((a * w) @ b / math.sqrt(nr * nc)).reshape(-1)
    return th


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = E.Context(0)
    return _ctx


class State:
    pass


def _inputs(case, seed):
    """The numbers of a case without any plan: what prepare() and exact() both start from."""
    gen = _gen(seed)
    st = State()
    st.case, st.sites = case, _sites(case)
    s0 = st.sites[0]
    if case["op"] == "svd":
        st.theta = _theta(s0.split, gen)
        return st
    st.Lb = [None if s.L is None else _boundary(s.L, gen) for s in st.sites]
    st.Rb = [None if s.R is None else _boundary(s.R, gen) for s in st.sites]
    if case["op"] in ("left_step", "right_step"):
        bonds, i = s0.bonds, s0.site
        ten = S.SiteTensor(s0.model.phys, bonds[i], bonds[i + 1])
        x = _vector(ten.rp.rows, ten.rp.cols, ten.rp.offs, ten.rp.total, gen)
        st.ket = x
        st.bra = torch.from_numpy(S.SiteTensor(s0.model.phys, bonds[i], bonds[i + 1], x.cpu().numpy()).left_paired()).cuda() \
            if case["op"] == "left_step" else x
        return st
    st.xs = [_psi(s.plan, gen) for s in st.sites]
    if case["op"] == "adjoint":
        st.w = _psi(s0.plan, gen, "out")
    return st


def prepare(case, seed):
    st = _inputs(case, seed)
    ctx, op, s0 = _context(), case["op"], st.sites[0]
    if op == "svd":
        sp = s0.split
        st.usv = torch.empty(max(sp.usv_elems, 1), dtype=F64, device="cuda")
        st.kept = torch.empty_like(st.theta)
        st.blocks, st.products = [], []
        for mc in sp.order:
            _, _, nr, nc, _ = sp.blocks[mc]
            k = min(nr, nc)
            t0, u0, s, v0 = sp.th_off[mc], sp.u_off[mc], sp.s_base + sp.s_off[mc], sp.vt_base + sp.vt_off[mc]
            u, sv, vt = st.usv[u0:u0 + nr * k], st.usv[s:s + k], st.usv[v0:v0 + k * nc]
            st.blocks.append((nr, nc, st.theta[t0:t0 + nr * nc], u, sv, vt))
            q = (k + 1) // 2  # states kept
            st.products.append((u.view(k, nr)[:q], sv[:q], vt.view(nc, k)[:, :q], st.kept[t0:t0 + nr * nc].view(nc, nr)))
        st.s = st.usv[sp.s_base:]
        return st
    laddr = [None if s.L is None else s.L.cohort_addresses(b.data_ptr()) for s, b in zip(st.sites, st.Lb)]
    raddr = [None if s.R is None else s.R.cohort_addresses(b.data_ptr()) for s, b in zip(st.sites, st.Rb)]
    if op == "batched":
        st.plan = E.BatchedPlan(ctx, [(s.plan, la, ra) for s, la, ra in zip(st.sites, laddr, raddr)])
        st.x = torch.zeros(st.plan.total_size, dtype=F64, device="cuda")
        for b, x in zip(st.plan.in_base, st.xs):
            st.x[b:b + x.numel()] = x
        st.y = torch.zeros_like(st.x)
        return st
    st.plan = E.DevicePlan(ctx, s0.plan, left_addr=laddr[0], other_addr=raddr[0])
    if op in ("left_step", "right_step"):
        st.out = torch.zeros(max(s0.out.n_elems, 1), dtype=F64, device="cuda")
        st.addr = s0.out.cohort_addresses(st.out.data_ptr())
        return st
    st.x = st.xs[0]
    st.y = torch.zeros_like(st.x)
    if op == "adjoint":
        st.galpha = torch.zeros(len(s0.plan["term_alpha"]), dtype=F64, device="cuda")
    return st


def run(st):
    op, sh = st.case["op"], torch.cuda.current_stream().cuda_stream
    if op in ("hpsi", "batched"):
        st.plan.hpsi(st.x.data_ptr(), st.y.data_ptr(), capi.PREC_FP64, sh)
        return st.y
    if op == "emulated":
        st.plan.hpsi(st.x.data_ptr(), st.y.data_ptr(), capi.PREC_FP64_EMULATED, sh)
        return st.y
    if op == "solve":
        e, _ = st.plan.solve(st.x.data_ptr(), st.y.data_ptr(), st.x.numel(), tol=0.0, max_iter=8, stream=sh)
        return {"energy": e, "x": st.y}
    if op in ("left_step", "right_step"):
        st.plan.step(st.ket.data_ptr(), st.bra.data_ptr(), st.addr, sh)
        return st.out
    if op == "adjoint":
        st.plan.adjoint(st.w.data_ptr(), st.x.data_ptr(), st.y.data_ptr(), st.galpha.data_ptr(), sh)
        return {"gx": st.y, "galpha": st.galpha}
    # the split's use: singular values for the truncation choice, and the two-site tensor of the kept
    # states (U and V alone are defined up to signs)
    E.block_svd(st.blocks, sh)
    for ut, sv, v, out in st.products:
        torch.mm(v * sv, ut, out=out)
    return {"s": st.s, "kept": st.kept}


# ---- what a pass cannot do without -------------------------------------------------------

def _stage_flops(p):
    rows = (p["t_brows"] if p["kind"] == capi.PLAN_LEFT else np.asarray(p["in_rows"])[p["t_lb"]]).astype(np.int64)
    cols = (p["t_width"] if p["kind"] == capi.PLAN_LEFT else p["t_bcols"]).astype(np.int64)
    inner = (p["t_bcols"] if p["kind"] == capi.PLAN_LEFT else p["t_brows"]).astype(np.int64)
    f1 = int((2 * rows * cols * inner * p["t_nb"]).sum())
    f3 = int((2 * p["c_ls"].astype(np.int64) * p["c_nsrows"] * p["c_rs"] * p["c_stripe"]).sum())
    return f1, f3


def work(case):
    op, sites = case["op"], _sites(case)
    if op == "svd":
        b = f = 0
        for mc in sites[0].split.order:
            _, _, nr, nc, _ = sites[0].split.blocks[mc]
            k, q = min(nr, nc), (min(nr, nc) + 1) // 2
            b += 8 * (2 * nr * nc + (nr + nc + 1) * k)
            f += 6 * max(nr, nc) * k * k + 8 * k ** 3 + 2 * nr * nc * q
        return {"bytes": b, "flops": f}
    nbytes = flops = 0
    for s in sites:
        p = s.plan
        nterm = len(p["term_alpha"])
        f1, f3 = _stage_flops(p)
        sb = max(0, s.schedule.flops - f1 - f3)
        edge = sum(i.n_elems for i in (s.L, s.R, s.out) if i is not None)
        nbytes += 8 * (int(p["in_size"]) + int(p["out_size"]) + edge + nterm)
        if op == "adjoint":
            nbytes += 8 * (int(p["in_size"]) + nterm)
            flops += 2 * f1 + f3 + 2 * sb
        else:
            flops += s.schedule.flops
    if op == "solve":
        n, k = int(sites[0].plan["in_size"]), 8
        flops = k * flops + 2 * n * (3 * k * (k + 1) // 2 + k * (k + 1) + 8 * k)
        nbytes = nbytes + 8 * n * 2 * k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    op = case["op"]
    if op == "emulated":
        return {"rel": 4e-12}  # seven 7-bit digits per operand
    if op == "solve":
        return {"rel": 1e-12}  # eight iterations amplify the rounding of the first
    if op == "svd":
        return {"rel": 3e-13}  # rounding of the rotations, over the gap at the cut
    return {"rel": 3e-14}  # sums of FP64 products in another order


# ---- the same in plain torch, 64 bits ------------------------------------------------------

class _Exec:
    """Stages of a flat plan with torch matrix products.  All matrices are column-major
    in memory, so every torch view below is the transpose of the plan's matrix."""

    def __init__(self, p, bnd1, idx1):
        self.p, self.b1, self.i1 = p, bnd1, idx1
        self.left = p["kind"] == capi.PLAN_LEFT
        rows = p["t_brows"] if self.left else np.asarray(p["in_rows"])[p["t_lb"]]
        cols = p["t_width"] if self.left else p["t_bcols"]
        size = rows.astype(np.int64) * cols * p["t_nb"]
        self.t_off = np.concatenate([[0], np.cumsum(size)])

    def _operands(self, t, x):
        p = self.p
        lb, ci, nb, tr = int(p["t_lb"][t]), int(p["t_ci"][t]), int(p["t_nb"][t]), bool(p["t_trans"][t])
        br, bc = int(p["t_brows"][t]), int(p["t_bcols"][t])
        o = int(self.i1.storage_off[ci])
        raw = self.b1[o:o + nb * br * bc]
        bt = raw.view(nb, br, bc).transpose(1, 2) if tr else raw.view(nb, bc, br)  # (nb, bcols, brows): B^T
        k = bc if self.left else int(p["in_rows"][lb])
        w = int(p["t_width"][t]) if self.left else br
        a = int(p["in_off"][lb]) + int(p["t_col"][t]) * k
        return bt, slice(a, a + w * k), (w, k)

    def create_T(self, x):
        T = torch.empty(int(self.t_off[-1]), dtype=F64, device="cuda")
        for t in range(len(self.p["t_lb"])):
            bt, sl, shape = self._operands(t, x)
            xt = x[sl].view(shape)
            T[self.t_off[t]:self.t_off[t + 1]] = ((xt @ bt) if self.left else (bt @ xt)).reshape(-1)
        return T

    def units(self, c):
        p = self.p
        for u in range(int(p["c_unit"][c]), int(p["c_unit"][c + 1])):
            l0, l1 = int(p["u_line"][u]), int(p["u_line"][u + 1])
            k0, k1 = int(p["l_term"][l0]), int(p["l_term"][l1])
            ls, ms = int(p["c_rs"][c] if self.left else p["c_ls"][c]), int(p["u_ms"][u])
            if k1 == k0:
                continue
            line = np.repeat(p["l_b1"][l0:l1], np.diff(p["l_term"][l0:l1 + 1].astype(np.int64))).astype(np.int64)
            start = self.t_off[p["term_t"][k0:k1]] + p["term_col"][k0:k1].astype(np.int64) * ls
            src, inv = np.unique(start, return_inverse=True)
            yield u, ls, ms, k0, k1, line, src, inv

    def alpha(self, c, k0, k1, line, n, inv):
        A = np.zeros((int(self.p["c_nsrows"][c]), n))
        np.add.at(A, (line, inv), self.p["term_alpha"][k0:k1])
        return torch.from_numpy(A).cuda()

    @staticmethod
    def gather(src, n):
        return torch.from_numpy(src).cuda()[:, None] + torch.arange(n, device="cuda")[None, :]

    def create_S(self, c, T):
        p = self.p
        ns, stripe = int(p["c_nsrows"][c]), int(p["c_stripe"][c])
        ls = int(p["c_rs"][c] if self.left else p["c_ls"][c])
        St = torch.zeros((ns, ls, stripe) if self.left else (stripe, ns, ls), dtype=F64, device="cuda")
        for u, ls, ms, k0, k1, line, src, inv in self.units(c):
            cells = self.alpha(c, k0, k1, line, len(src), inv) @ T[self.gather(src, ls * ms)]
            uo = int(p["u_offset"][u])
            if self.left:
                St[:, :, uo:uo + ms] = cells.view(ns, ls, ms)
            else:
                St[uo:uo + ms] = cells.view(ns, ms, ls).permute(1, 0, 2)
        return St

    def left_T(self, c, Lb, Lidx):
        """L^T of cohort c: (nsrows * ls, rs)."""
        p = self.p
        ns, ls, rs, ci = int(p["c_nsrows"][c]), int(p["c_ls"][c]), int(p["c_rs"][c]), int(p["c_ci"][c])
        o = int(Lidx.storage_off[ci])
        raw = Lb[o:o + ns * ls * rs]
        return raw.view(ns, rs, ls).transpose(1, 2).reshape(ns * ls, rs) if p["c_trans"][c] else raw.view(ns * ls, rs)

    def block(self, v, side, b):
        p = self.p
        r, c, o = int(p[side + "_rows"][b]), int(p[side + "_cols"][b]), int(p[side + "_off"][b])
        return v[o:o + r * c].view(c, r)

    def hpsi(self, x, Lb, Lidx):
        p = self.p
        T = self.create_T(x)
        y = torch.zeros(int(p["out_size"]), dtype=F64, device="cuda")
        for c in range(len(p["c_lb"])):
            St = self.create_S(c, T)
            self.block(y, "out", int(p["c_rb"][c])).add_(St.view(St.shape[0], -1) @ self.left_T(c, Lb, Lidx))
        return y

    def adjoint(self, w, x, Lb, Lidx):
        p = self.p
        T = self.create_T(x)
        gT = torch.zeros_like(T)
        ga = torch.zeros(len(p["term_alpha"]), dtype=F64, device="cuda")
        for c in range(len(p["c_lb"])):
            ns, stripe = int(p["c_nsrows"][c]), int(p["c_stripe"][c])
            Gt = (self.block(w, "out", int(p["c_rb"][c])) @ self.left_T(c, Lb, Lidx).T).view(stripe, ns, -1)
            for u, ls, ms, k0, k1, line, src, inv in self.units(c):
                uo = int(p["u_offset"][u])
                g = Gt[uo:uo + ms].permute(1, 0, 2).reshape(ns, ms * ls)
                at = self.gather(src, ls * ms)
                ga[k0:k1] = (g @ T[at].T)[torch.from_numpy(line).cuda(), torch.from_numpy(inv).cuda()]
                gT.index_add_(0, at.reshape(-1), (self.alpha(c, k0, k1, line, len(src), inv).T @ g).reshape(-1))
        gx = torch.zeros_like(x)
        for t in range(len(p["t_lb"])):
            bt, sl, shape = self._operands(t, x)
            g = gT[self.t_off[t]:self.t_off[t + 1]].view(bt.shape[0], bt.shape[1], shape[1])
            gx[sl].view(shape).add_(torch.bmm(bt.transpose(1, 2), g).sum(0))
        return {"gx": gx, "galpha": ga}

    def step(self, ket, bra, out_idx):
        p = self.p
        T = self.create_T(ket)
        out = torch.zeros(max(out_idx.n_elems, 1), dtype=F64, device="cuda")
        for c in range(len(p["c_lb"])):
            St = self.create_S(c, T)
            ns, ls, rs = int(p["c_nsrows"][c]), int(p["c_ls"][c]), int(p["c_rs"][c])
            o = int(out_idx.storage_off[int(p["c_out_ci"][c])])
            if self.left:
                got = St.view(ns * rs, -1) @ self.block(bra, "out", int(p["c_lb"][c])).T
            else:
                got = torch.matmul(self.block(bra, "out", int(p["c_rb"][c])).T, St.permute(1, 0, 2))
            out[o:o + ns * ls * rs] = got.reshape(-1)
        return out


def _lowest(A):
    """Smallest eigenpair of a symmetric matrix by cyclic Jacobi rotations from the identity,
    which also fixes the eigenvector's sign."""
    A, k = A.copy(), len(A)
    Z = np.eye(k)
    for _ in range(60):
        if np.sum(np.triu(A, 1) ** 2) <= 1e-34 * np.sum(A ** 2):
            break
        for p in range(k):
            for q in range(p + 1, k):
                if A[p, q] == 0.0:
                    continue
                tau = (A[q, q] - A[p, p]) / (2.0 * A[p, q])
                t = math.copysign(1.0, tau) / (abs(tau) + math.sqrt(1.0 + tau * tau))
                c = 1.0 / math.sqrt(1.0 + t * t)
                J = np.array([[c, t * c], [-t * c, c]])
                A[:, [p, q]] = A[:, [p, q]] @ J
                A[[p, q], :] = J.T @ A[[p, q], :]
                Z[:, [p, q]] = Z[:, [p, q]] @ J
    i = int(np.argmin(np.diag(A)))
    return A[i, i], Z[:, i]


def _davidson(matvec, x0, max_iter):
    """Jacobi-Davidson without inner solve: MGS with one refinement, Rayleigh-Ritz, t = -r + (r.u / u.u) u."""
    V, VA, Mk = [], [], np.zeros((max_iter, max_iter))
    t = x0.clone()
    for it in range(max_iter):
        tau = torch.linalg.norm(t)
        for again in range(2):
            if again and not torch.linalg.norm(t) < 0.25 * tau:
                break
            for v in V:
                t = t - torch.dot(v, t) * v
        t = t / torch.linalg.norm(t)
        V.append(t)
        VA.append(matvec(t))
        for i in range(it + 1):
            Mk[i, it] = Mk[it, i] = float(torch.dot(V[i], VA[it]))
        theta, z = _lowest(Mk[:it + 1, :it + 1])
        u = sum(float(c) * v for c, v in zip(z, V))
        r = sum(float(c) * v for c, v in zip(z, VA)) - float(theta) * u
        t = -r + torch.dot(r, u) / torch.dot(u, u) * u
    return float(theta), u


def exact(case, seed):
    st = _inputs(case, seed)
    op, s0 = case["op"], st.sites[0]
    if op == "svd":
        sp = s0.split
        sv, kept = torch.zeros(sp.usv_elems - sp.s_base, dtype=F64, device="cuda"), torch.empty_like(st.theta)
        for mc in sp.order:
            _, _, nr, nc, _ = sp.blocks[mc]
            k, q, o = min(nr, nc), (min(nr, nc) + 1) // 2, sp.th_off[mc]
            a, s, b = torch.linalg.svd(st.theta[o:o + nr * nc].view(nc, nr), full_matrices=False)
            sv[sp.s_off[mc]:sp.s_off[mc] + k] = s
            kept[o:o + nr * nc] = ((a[:, :q] * s[:q]) @ b[:q]).reshape(-1)
        return {"s": sv, "kept": kept}
    if op in ("left_step", "right_step"):
        bnd, idx = (st.Lb[0], s0.L) if op == "left_step" else (st.Rb[0], s0.R)
        return _Exec(s0.plan, bnd, idx).step(st.ket, st.bra, s0.out)
    ex = [_Exec(s.plan, r, s.R) for s, r in zip(st.sites, st.Rb)]
    if op == "batched":
        ys = [e.hpsi(x, l, s.L) for e, x, l, s in zip(ex, st.xs, st.Lb, st.sites)]
        pad = [torch.zeros(-(-y.numel() // 128) * 128, dtype=F64, device="cuda") for y in ys]
        for z, y in zip(pad, ys):
            z[:y.numel()] = y
        return torch.cat(pad)
    if op == "adjoint":
        return ex[0].adjoint(st.w, st.xs[0], st.Lb[0], s0.L)
    if op == "solve":
        e, u = _davidson(lambda v: ex[0].hpsi(v, st.Lb[0], s0.L), st.xs[0], 8)
        return {"energy": e, "x": u}
    return ex[0].hpsi(st.xs[0], st.Lb[0], s0.L)
