"""Stages of two k-blocks of the tcgen05 product (csrc/gemm_tc.cu: K a multiple of 64, narrow tiles) against stages of one (tiles of
256 columns, pairs): odd numbers of k-blocks, parts that end inside a stage, ragged rows and columns, gate and up by one copy."""
import pytest
import torch

pytestmark = pytest.mark.gpu

WAYS = [(w, cluster, pair) for w in (256, 128, 64, 32) for cluster, pair in ((False, False), (True, False), (False, True))]


def run(Kn, parts, call):
    out = {}
    for w, cluster, pair in WAYS:
        try:
            out[(w, cluster, pair)] = call((w, parts, cluster, pair))
        except Kn.KernelError:
            pass
    return out


@pytest.mark.parametrize("M,N,K", [(17, 72, 128), (33, 520, 576), (40, 1000, 1088), (64, 130, 1984), (128, 264, 704), (129, 40, 960)])
def test_same_bits_and_64_bits(M, N, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()[:, :K]                # (rows longer than K)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    x = torch.randn(M, N, device="cuda", generator=g)
    exact = a.double() @ w.double().T
    bound = K * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)      # K additions, each cut off by at most 2^-23 of the magnitudes
    for parts in (1, 2, 3, 5):
        outs = run(Kn, parts, lambda c: Kn.gemm_tc(a, w, torch.full((M, N), float("nan"), device="cuda"), choice=c))
        first = outs.get((256, False, False))
        for way, out in outs.items():
            first = out if first is None else first
            assert bool(((out.double() - exact).abs() <= bound).all()), (parts, way)
            assert torch.equal(out, first), (parts, way)
        for way, out in run(Kn, parts, lambda c: Kn.gemm_tc(a, w, x.clone(), accumulate=True, choice=c)).items():
            assert torch.equal(out, x + first), (parts, way)
    assert Kn.tc_status() == 0


@pytest.mark.parametrize("M,ff,K", [(17, 100, 576), (64, 257, 1088), (130, 712, 704)])
def test_gated(M, ff, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(M + ff)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * ff, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    for parts in (1, 2, 3):
        outs = run(Kn, parts, lambda c: Kn.gemm_tc(a, w, torch.empty((M, ff), device="cuda", dtype=torch.bfloat16), swiglu=True, choice=c))
        gu = Kn.gemm_tc(a, w, torch.empty((M, 2 * ff), device="cuda", dtype=torch.bfloat16), choice=(128, parts, False, False))
        ref = Kn.swiglu(gu, torch.empty((M, ff), device="cuda", dtype=torch.bfloat16)).double()
        first = outs[(128, False, False)]
        assert bool(((first.double() - ref).abs() <= 2.0 ** -7 * ref.abs()).all())         # one rounding of the result apart at most
        for way, out in outs.items():
            assert torch.equal(out, first), (parts, way)
    assert Kn.tc_status() == 0
