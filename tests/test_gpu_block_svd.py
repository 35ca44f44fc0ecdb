"""The two-site split on the device: dmrgb200_block_svd (one-sided Jacobi,
FP64) against numpy's LAPACK SVD, dmrgb200_copy_blocks against its host
definition, and split_device against the host split (svd / svd_truncate,
block_matrix/block_matrix_algorithms.h:95-113,185-298)."""
import numpy as np
import pytest

from dmrgb200 import _capi as capi
from dmrgb200 import dmrg as G
from dmrgb200 import engine as E
from dmrgb200 import models as M
from dmrgb200 import mps as S

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12

# shapes: tiny, odd, transposed, the shared-memory path and (past 200 KB of
# work) the global-scratch path
SHAPES = [(1, 1), (1, 7), (7, 1), (2, 2), (5, 3), (3, 5), (64, 64), (65, 33), (33, 65), (100, 100), (130, 130),
          (200, 120), (120, 200), (300, 17)]


def _svd_dev(mats):
    blocks, outs = [], []
    for a in mats:
        r, c = a.shape
        k = min(r, c)
        ad = torch.from_numpy(np.asfortranarray(a).reshape(-1, order="F").copy()).cuda()
        u = torch.full((max(r * k, 1),), np.nan, dtype=torch.float64, device="cuda")
        s = torch.full((max(k, 1),), np.nan, dtype=torch.float64, device="cuda")
        vt = torch.full((max(k * c, 1),), np.nan, dtype=torch.float64, device="cuda")
        blocks.append((r, c, ad, u, s, vt))
        outs.append((u, s, vt))
    E.block_svd(blocks)
    res = []
    for a, (u, s, vt) in zip(mats, outs):
        r, c = a.shape
        k = min(r, c)
        res.append((u.cpu().numpy()[:r * k].reshape(k, r).T, s.cpu().numpy()[:k], vt.cpu().numpy()[:k * c].reshape(c, k).T))
    return res


def _check(a, U, s, Vt):
    sref = np.linalg.svd(a, compute_uv=False)
    smax = max(sref[0] if sref.size else 0.0, 1e-300)
    assert np.all(np.diff(s) <= 0)
    assert np.max(np.abs(s - sref)) <= TOL * smax
    assert np.linalg.norm(U @ np.diag(s) @ Vt - a) <= TOL * max(np.linalg.norm(a), 1e-300)
    nz = s > 1e-13 * smax
    Un = U[:, nz]
    assert np.max(np.abs(Un.T @ Un - np.eye(Un.shape[1]))) <= TOL
    assert np.max(np.abs(Vt @ Vt.T - np.eye(Vt.shape[0]))) <= TOL


def test_block_svd_shapes_in_one_launch():
    rng = np.random.default_rng(0)
    mats = [rng.standard_normal(sh) for sh in SHAPES]
    for a, (U, s, Vt) in zip(mats, _svd_dev(mats)):
        _check(a, U, s, Vt)


def test_block_svd_graded_rank_deficient_and_zero_blocks():
    rng = np.random.default_rng(1)
    q1, _ = np.linalg.qr(rng.standard_normal((40, 40)))
    q2, _ = np.linalg.qr(rng.standard_normal((30, 30)))
    graded = q1[:, :30] @ np.diag(10.0 ** -np.linspace(0, 12, 30)) @ q2.T
    low = rng.standard_normal((40, 3)) @ rng.standard_normal((3, 30))
    zero = np.zeros((9, 4))
    mats = [graded, low, zero, 1e-200 * rng.standard_normal((6, 5)), 1e200 * rng.standard_normal((5, 6))]
    out = _svd_dev(mats)
    for a, (U, s, Vt) in zip(mats[:2], out[:2]):
        _check(a, U, s, Vt)
    assert np.all(out[2][1] == 0.0) and np.all(out[2][0] == 0.0)
    for a, (U, s, Vt) in zip(mats[3:], out[3:]):
        sref = np.linalg.svd(a, compute_uv=False)
        assert np.max(np.abs(s - sref)) <= TOL * sref[0]
        assert np.linalg.norm(U @ np.diag(s) @ Vt - a) <= TOL * np.linalg.norm(a)


# sizes around the register and cluster classes (32 elements per lane slot; 16 column pairs
# per CTA, 1, 2, 4 or 8 CTAs; above 256 rows the general kernel), square and not
EDGES = [(31, 31), (32, 32), (33, 33), (64, 63), (63, 64), (65, 65), (128, 127), (129, 128), (128, 129), (130, 33),
         (256, 255), (255, 256), (256, 256), (256, 2), (2, 256), (256, 1), (257, 40), (40, 257)]


@pytest.mark.parametrize("decades", [0, 8, 14])
def test_block_svd_class_edges(decades):
    """Singular values falling by `decades`: reconstruction, orthogonality of both factors
    (also of the directions of small singular values) and singular values."""
    rng = np.random.default_rng(7)
    mats = []
    for r, c in EDGES:
        k = min(r, c)
        w = 10.0 ** (-decades * np.arange(k) / max(k, 1))
        mats.append((np.linalg.qr(rng.standard_normal((r, k)))[0] * w) @ np.linalg.qr(rng.standard_normal((c, k)))[0].T)
    for a, (U, s, Vt) in zip(mats, _svd_dev(mats)):
        _check(a, U, s, Vt)
        assert np.max(np.abs(U.T @ U - np.eye(U.shape[1]))) <= TOL


def test_block_svd_column_scaling_keeps_small_values():
    """A = B diag(d) with B well conditioned and d over 40 decades: one-sided Jacobi gives the
    small singular values to relative accuracy (here within 1e-10: the condition of the
    random B, at most a few thousand, times rounding), also after the pivoted QR."""
    rng = np.random.default_rng(8)
    mats, refs = [], []
    for n in (24, 70, 150):
        q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        d = 10.0 ** (-40.0 * np.arange(n) / n)
        mats.append(q * d[rng.permutation(n)])  # orthogonal columns: the singular values are d
        refs.append(d)
    for a, d, (U, s, Vt) in zip(mats, refs, _svd_dev(mats)):
        assert np.max(np.abs(s / d - 1.0)) <= 1e-10


def test_block_svd_zero_columns_and_non_finite_blocks_take_the_general_kernel():
    """Exactly zero columns: zero singular values with zero U columns and an orthonormal V;
    a block with a NaN gives NaN and leaves the other blocks alone."""
    rng = np.random.default_rng(9)
    a = rng.standard_normal((90, 80))
    a[:, ::3] = 0.0
    bad = rng.standard_normal((40, 40))
    bad[3, 5] = np.nan
    c = rng.standard_normal((70, 70))
    (U, s, Vt), (Ub, sb, Vb), good = _svd_dev([a, bad, c])
    _check(a, U, s, Vt)
    assert np.all(U[:, s == 0.0] == 0.0) and np.sum(s == 0.0) >= 1
    assert np.any(np.isnan(sb)) or np.any(np.isnan(Ub)) or np.any(np.isnan(Vb))
    _check(c, *good)


@pytest.mark.parametrize("n", [24, 70, 150])
@pytest.mark.parametrize("decades", [130, 138, 150, 165])
def test_block_svd_vanishing_columns(n, decades):
    """Orthogonal columns scaled down to 1e-130 .. 1e-165 of the largest: squared norms that leave
    the normal range must not cost a factor its orthogonality.  The singular values (the
    scales) and both factors are right to rounding, or the call says it did not converge
    (columns below 1e-154, whose squared norms are subnormal)."""
    rng = np.random.default_rng(n)
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    d = 10.0 ** (-float(decades) * np.arange(n) / (n - 1))
    try:
        ((U, s, Vt),) = _svd_dev([q * d[rng.permutation(n)]])
    except capi.DmrgError as e:
        assert e.status == capi.NUMERIC and decades > 150
        return
    assert np.max(np.abs(s / d - 1.0)) <= TOL
    assert np.max(np.abs(U.T @ U - np.eye(n))) <= TOL and np.max(np.abs(Vt @ Vt.T - np.eye(n))) <= TOL


def test_block_svd_rejects_null_blocks():
    rows = np.array([2], dtype=np.uint32)
    nul = (capi.C.c_void_p * 1)(None)
    st = capi.lib.dmrgb200_block_svd(1, capi.ptr(rows, capi.C.c_uint32), capi.ptr(rows, capi.C.c_uint32), nul, nul,
                                     nul, nul, None)
    assert st == 1


def test_copy_blocks_against_host_definition():
    rng = np.random.default_rng(2)
    src = rng.standard_normal(5000)
    scale = rng.standard_normal(64)
    recs, off = [], 0
    for k in range(40):
        r, c = int(rng.integers(0, 9)), int(rng.integers(0, 7))
        sl = r + int(rng.integers(0, 3))
        so = int(rng.integers(0, 5000 - max(sl, 1) * max(c, 1)))
        mode = int(rng.integers(0, 3))
        recs.append((so, sl, off, max(r, 1), r, c, mode, int(rng.integers(0, 40))))
        off += max(r, 1) * max(c, 1)
    cp = E.copy_records(recs)
    ref = np.zeros(off)
    E.apply_copies(cp, src, ref, scale)
    dst = torch.zeros(off, dtype=torch.float64, device="cuda")
    E.copy_blocks(cp, torch.from_numpy(src).cuda(), dst, torch.from_numpy(scale).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy(), ref)


@pytest.mark.parametrize("name,m", [("hubbard", 10 ** 6), ("bose", 4), ("heisenberg", 10 ** 6)])
def test_split_device_matches_host_split(name, m):
    L = 6
    model = {"heisenberg": M.heisenberg(L), "hubbard": M.fermi_hubbard(L, n_up=3, n_down=3),
             "bose": M.bose_hubbard(L, N=3)}[name]
    rng = np.random.default_rng(5)
    bonds = S.allowed_sectors(model.phys, L, model.total_charge, 12)
    A = S.random_mps(model.phys, bonds, rng)
    p12, offs = M.fuse_phys(model.phys, model.phys)
    psi = G.twosite(A[2], A[3], p12, offs)
    psi_dev = E.to_device(psi.data)
    for l2r in (True, False):
        ref = G.split(psi, model.phys, model.phys, offs, m, 1e-16, l2r)
        got = G.split_device(psi_dev, psi, model.phys, model.phys, offs, m, 1e-16, l2r)
        assert got.bond == ref.bond
        assert abs(got.truncated_weight - ref.truncated_weight) <= 1e-12
        # the kept two-site tensor is gauge independent
        t_ref = G.twosite(ref.A, ref.B, p12, offs).data
        t_got = G.twosite(got.A, got.B, p12, offs).data
        assert np.linalg.norm(t_got - t_ref) <= TOL * np.linalg.norm(t_ref)
        # device copies agree with the host copies; A left-normalised (l2r) or B right-normalised
        assert np.array_equal(got.dev_A.cpu().numpy(), got.A.data)
        assert np.array_equal(got.dev_A_lp.cpu().numpy(), got.A.left_paired())
        assert np.array_equal(got.dev_B.cpu().numpy(), got.B.data)
        if l2r:
            lp = S.left_paired_layout(got.A.phys, got.A.left, got.A.right)
            for rb in range(len(got.A.right)):
                X = S.block_view(got.A.left_paired(), lp, rb)
                assert np.max(np.abs(X.T @ X - np.eye(X.shape[1]))) <= TOL
        else:
            for lb in range(len(got.B.left)):
                X = S.block_view(got.B.data, got.B.rp, lb)
                assert np.max(np.abs(X @ X.T - np.eye(X.shape[0]))) <= TOL
