"""The grouped FP64 DMMA GEMM (every autotuner variant) on single regular and
ragged problems through dmrgb200_dgemm_f64, against torch's FP64 matmul
(relative error <= 1e-13)."""
import ctypes as C

import pytest

from dmrgb200 import _capi as capi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(37, 53, 29, 0), (100, 7, 300, 3), (257, 129, 65, 1), (16, 64, 16, 0), (1, 1, 1, 0), (33, 65, 0, 0)]


@pytest.mark.parametrize("variant", range(capi.lib.dmrgb200_gemm_variant_count()))
@pytest.mark.parametrize("M,N,K,pad", SHAPES)
def test_dgemm_f64_matches_torch(variant, M, N, K, pad):
    assert torch.cuda.is_available()
    g = torch.Generator(device="cuda").manual_seed(M * 131 + N * 7 + K + variant)
    lda, ldb, ldc = M + pad, K + pad, M + 2 * pad
    A = torch.randn(max(K * lda, 1), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(max(N * ldb, 1), dtype=torch.float64, device="cuda", generator=g)
    Cm = torch.full((N * ldc,), float("nan"), dtype=torch.float64, device="cuda")
    capi.check(capi.lib.dmrgb200_dgemm_f64(M, N, K, A.data_ptr(), lda, B.data_ptr(), ldb, Cm.data_ptr(), ldc,
                                           variant, None), "dgemm_f64")
    a = A[:K * lda].view(K, lda)[:, :M].T if K else torch.zeros(M, 0, dtype=torch.float64, device="cuda")
    b = B[:N * ldb].view(N, ldb)[:, :K].T if K else torch.zeros(0, N, dtype=torch.float64, device="cuda")
    ref = a @ b
    got = Cm.view(N, ldc)[:, :M].T
    err = (got - ref).norm() / max(ref.norm(), 1e-300)
    assert float(err) <= 1e-13 or (K == 0 and float(got.abs().max()) == 0.0)
    # the padding rows of C are not written
    if pad:
        assert torch.isnan(Cm.view(N, ldc)[:, M:]).all()


def test_pinned_plan_variants_match_oracle():
    """dmrgb200_plan_set_gemm_variants: every variant pinned on both stages of an H·psi plan
    gives the oracle's H·psi (FP64, 1e-12), on the device and through the host-buffer graph
    (which is captured again after a new choice); an index out of range is rejected."""
    import numpy as np

    from dmrgb200 import engine as E
    from helpers import OracleChain, make_chain, random_psi

    model, bonds, tensors, rng = make_chain("qc", 8, 0, seed=5, synthetic_m=64)
    ch = OracleChain(model, bonds, tensors, 3)
    x = random_psi(ch.p12, ch.left, ch.right, rng).data
    want = ch.hpsi(x)
    ctx = E.Context(0)
    Lb, Rb = E.to_device(ch.Lval), E.to_device(ch.Rval)
    plan = E.DevicePlan(ctx, ch.sched.plan, left_addr=ch.Lidx.cohort_addresses(Lb.data_ptr()),
                        other_addr=ch.Ridx.cohort_addresses(Rb.data_ptr()))
    xd = E.to_device(x)
    xh = torch.tensor(x, dtype=torch.float64).pin_memory()
    yh = torch.zeros(len(want), dtype=torch.float64).pin_memory()
    n = capi.lib.dmrgb200_gemm_variant_count()
    for v in range(n):
        plan.set_gemm_variants(v, (v + 3) % n)
        yd = torch.zeros_like(xd)
        plan.hpsi(xd.data_ptr(), yd.data_ptr())
        plan.hpsi_host(xh.data_ptr(), yh.data_ptr())
        torch.cuda.synchronize()
        for got in (yd.cpu().numpy(), yh.numpy()):
            assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want), v
    with pytest.raises(capi.DmrgError) as e:
        plan.set_gemm_variants(n, 0)
    assert e.value.status == capi.INVALID_ARGUMENT


@pytest.mark.parametrize("variant", range(capi.lib.dmrgb200_gemm_variant_count()))
def test_short_k_ranges_take_nothing_from_earlier_kernels(variant):
    """K ranges of 1 to 17 (a first K step that is short, half full, full, and one more) on many
    CTAs, each after a product of NaN matrices by the same and by another variant, so that
    whatever a CTA reads of its predecessor's shared memory shows: the result is the same,
    bit for bit, every time, and torch's."""
    g = torch.Generator(device="cuda").manual_seed(variant)
    M, N = 301, 203
    nan = torch.full((M * 64 + 64 * N,), float("nan"), dtype=torch.float64, device="cuda")
    junk = torch.empty(M * N, dtype=torch.float64, device="cuda")
    n_var = capi.lib.dmrgb200_gemm_variant_count()

    def gemm(k, a, b, c, v):
        capi.check(capi.lib.dmrgb200_dgemm_f64(M, N, k, a.data_ptr(), M, b.data_ptr(), k, c.data_ptr(), M, v, None),
                   "dgemm_f64")

    for K in range(1, 18):
        A = torch.randn(K * M, dtype=torch.float64, device="cuda", generator=g)
        B = torch.randn(N * K, dtype=torch.float64, device="cuda", generator=g)
        ref = A.view(K, M).T @ B.view(N, K).T
        first = None
        for rep in range(3):
            gemm(64, nan, nan, junk, variant)
            gemm(5 + 4 * rep, nan, nan, junk, (variant + 1 + rep) % n_var)
            out = torch.full((M * N,), float("nan"), dtype=torch.float64, device="cuda")
            gemm(K, A, B, out, variant)
            # K <= 17 products of unit normals
            assert float((out.view(N, M).T - ref).norm() / ref.norm()) <= 1e-14, (K, rep)
            assert first is None or torch.equal(out, first), (K, rep)
            first = out


def test_staged_hpsi_repeats_bitwise_for_every_variant():
    """H·psi of ragged blocks (up to 36 rows, K tails of every length) through the GEMM stages:
    100 times per variant with a product of NaN matrices between, one bit pattern."""
    from dmrgb200 import engine as E
    from helpers import OracleChain, make_chain, random_psi

    model, bonds, tensors, rng = make_chain("hubbard", 14, 0, seed=3, synthetic_m=600)
    ch = OracleChain(model, bonds, tensors, 6)
    x = random_psi(ch.p12, ch.left, ch.right, rng).data
    Lb, Rb = E.to_device(ch.Lval), E.to_device(ch.Rval)
    plan = E.DevicePlan(E.Context(0), ch.sched.plan, left_addr=ch.Lidx.cohort_addresses(Lb.data_ptr()),
                        other_addr=ch.Ridx.cohort_addresses(Rb.data_ptr()))
    xd, want = E.to_device(x), ch.hpsi(x)
    nan = torch.full((512, 512), float("nan"), dtype=torch.float64, device="cuda")
    for v in range(capi.lib.dmrgb200_gemm_variant_count()):
        plan.set_gemm_variants(v, v)
        first, differ = None, torch.zeros((), dtype=torch.int64, device="cuda")
        for _ in range(100):
            nan @ nan
            yd = torch.zeros_like(xd)
            plan.hpsi(xd.data_ptr(), yd.data_ptr())
            first = yd if first is None else first
            differ += (yd != first).sum()
        assert int(differ) == 0, v
        y = first.cpu().numpy()
        assert ((y - want) ** 2).sum() ** 0.5 <= 1e-13 * (want ** 2).sum() ** 0.5, v
