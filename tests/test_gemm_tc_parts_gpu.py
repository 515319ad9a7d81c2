"""Parts along K of the tcgen05 product (csrc/gemm_tc.cu): they decide a sum's error and bits, and nothing else does -- the
tile's width, parts shared by a cluster or run one after the other, one CTA or a pair of them give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

WAYS = [(w, cluster, pair) for w in (256, 128, 64, 32) for cluster, pair in ((False, False), (True, False), (False, True))]


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    return a, w, torch.randn(N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)


@pytest.mark.parametrize("M,N,K,parts", [(101, 6144, 2048, 5), (257, 2048, 2048, 5), (700, 1024, 4608, 5), (200, 3072, 2048, 5),
                                         (64, 11264, 2048, 3), (1000, 2048, 5632, 2), (512, 3072, 1024, 2)])
def test_sums_are_as_exact_as_their_parts(M, N, K, parts):
    from kappai_b200.ops import kernels as Kn
    a, w, _, _ = operands(M, N, K)
    exact = a.double() @ w.double().T
    error = float((Kn.gemm_tc(a, w, torch.empty(M, N, device="cuda")).double() - exact).norm() / exact.norm())
    # the tensor core cuts a sum off at each addition of 16 products, and the n additions of a part shift it by n times that:
    # 1.65e-8 an addition was measured at one part of 128 additions, 1.5e-8 at five parts of 26; a third more is let pass, a
    # part less is not
    assert error < 1.35 * 1.65e-8 * -(-K // (16 * parts)), (error, Kn.gemm_tc_choice(M, N, K, out_dtype=torch.float32))


def ways(Kn, parts, call):
    """What ``call`` gives in every way that can run, by (cluster, pair)."""
    out = {}
    for width, cluster, pair in WAYS:
        try:
            out[(width, cluster, pair)] = call((width, parts, cluster, pair))
        except Kn.KernelError:
            pass
    return out


@pytest.mark.parametrize("M,N,K", [(17, 72, 520), (129, 520, 1032), (200, 1000, 1096), (256, 1, 1024), (257, 264, 2056), (385, 2050, 328),
                                   (1023, 515, 648)])
def test_every_way_of_running_the_parts_gives_the_same_bits(M, N, K):
    from kappai_b200.ops import kernels as Kn
    a, w, bias, x = operands(M, N, K)
    exact = a.double() @ w.double().T + bias.double()
    # at most K additions, each within 2^-23 of the magnitudes (the tensor core truncates)
    bound = K * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T) + 2.0 ** -22 * exact.abs()
    ran = set()
    for parts in (1, 2, 3, 5, 8):
        def wide(choice):
            out = torch.full((M, N + 3), 7.0, device="cuda")                  # rows that are not 16-byte aligned
            Kn.gemm_tc(a, w, out[:, :N], bias, choice=choice)
            assert bool((out[:, N:] == 7.0).all())
            return out[:, :N].clone()
        calls = [lambda c: Kn.gemm_tc(a, w, torch.full((M, N), float("nan"), device="cuda"), bias, choice=c), wide,
                 lambda c: Kn.gemm_tc(a, w, x.clone(), bias, accumulate=True, choice=c),
                 lambda c: Kn.gemm_tc(a, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), bias, choice=c),
                 lambda c: Kn.gemm_tc(a, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), bias, plain_activation="relu_squared",
                                      choice=c)]
        f32 = None
        for i, call in enumerate(calls):
            outs = ways(Kn, parts, call)
            ran |= {(cluster, pair) for _, cluster, pair in outs}
            for way, out in outs.items():
                if i == 0 and f32 is None:
                    f32 = out
                    assert bool(((f32.double() - exact).abs() <= bound).all())
                want = (f32, f32, x + f32, f32.bfloat16(), (f32.clamp(min=0) ** 2).bfloat16())[i]
                assert torch.equal(out, want), (parts, way, i)
    assert (False, False) in ran and (M <= 128 or (False, True) in ran)
    assert (True, False) in ran
    assert Kn.tc_status() == 0


@pytest.mark.parametrize("M,ff,K", [(40, 1408, 520), (200, 100, 1032), (300, 712, 1096), (513, 257, 520)])
@pytest.mark.parametrize("activation", ["silu", "relu", "gelu_tanh", "limits"])
def test_gated_ways_give_the_same_bits(M, ff, K, activation):
    from kappai_b200.ops import kernels as Kn
    a, w, bias, _ = operands(M, 2 * ff, K)
    glu = (1.5, 1.702, 1.0) if activation == "limits" else None
    for parts in (1, 2, 3):
        # the unfused path: gate and up as the product of the same parts stores them, then the row-wise kernel; both round the
        # same float32 value to bfloat16, whose last bits the two compilations of the activation may differ in
        gu = Kn.gemm_tc(a, w, torch.empty((M, 2 * ff), device="cuda", dtype=torch.bfloat16), bias, choice=(64, parts, False, False))
        ref = torch.empty((M, ff), device="cuda", dtype=torch.bfloat16)
        ref = Kn.glu_clamped(gu, ref, *glu) if glu else Kn.swiglu(gu, ref, activation)
        outs = ways(Kn, parts, lambda c: Kn.gemm_tc(a, w, torch.empty((M, ff), device="cuda", dtype=torch.bfloat16), bias, swiglu=True,
                                                    activation="silu" if glu else activation, glu=glu, choice=c))
        first = outs[(128, False, False)]
        d = (first.double() - ref.double()).abs()
        assert bool((d <= 2.0 ** -7 * ref.double().abs()).all()) and float((d > 0).double().mean()) < 1e-3
        for way, out in outs.items():
            assert torch.equal(out, first), (parts, way)
        assert M <= 128 or {w_ for w_, _, pair in outs if pair} == ({128, 256} if parts <= 2 else {128}), outs.keys()
    assert Kn.tc_status() == 0
