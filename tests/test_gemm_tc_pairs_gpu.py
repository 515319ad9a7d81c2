"""The tcgen05 product over pairs of CTAs (csrc/gemm_tc.cu, gemm_tc_pair_kernel): edges of the tiles of 256 rows, odd widths,
the last block of K, every epilogue, against float64 of the same bfloat16 operands.  The kernel is asked for by name
(``choice``), so that a test cannot pass on another; that the dispatch takes it is a test of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    z = a.double() @ w.double().T
    # float32 sums of exact products: at most K additions, each within 2^-24 of the magnitudes (the tensor core may truncate: 2^-23)
    return a, w, bias, z, K * 2.0 ** -23 * (a.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("M,N,K", [(257, 2048, 1024), (700, 3072, 136), (1030, 520, 2056), (2048, 1000, 64), (1290, 264, 200),
                                   (129, 1001, 72), (383, 130, 328)])
def test_pairs_store_accumulate_and_bias(M, N, K, width):
    from kappai_b200.ops import kernels as Kn
    a, w, bias, z, err = operands(M, N, K, M + N)
    pair = (width, 1, False, True)
    for b in (None, bias):
        y = z if b is None else z + b.double()
        one = 2.0 ** -23 * y.abs()
        f32 = Kn.gemm_tc(a, w, torch.full((M, N), float("nan"), device="cuda"), b, choice=pair)
        assert bool(((f32.double() - y).abs() <= err + one).all())
        bf = Kn.gemm_tc(a, w, torch.empty((M, N), device="cuda", dtype=torch.bfloat16), b, choice=pair)
        assert torch.equal(bf, f32.bfloat16())
        x = torch.randn(M, N, device="cuda")
        acc = Kn.gemm_tc(a, w, x.clone(), b, accumulate=True, choice=pair)
        assert torch.equal(acc, x + f32)
        act = Kn.gemm_tc(a, w, torch.empty((M, N), device="cuda", dtype=torch.bfloat16), b, plain_activation="relu_squared", choice=pair)
        assert torch.equal(act, (f32.clamp(min=0) ** 2).bfloat16())
        wide = torch.full((M, N + 3), 7.0, device="cuda")                  # rows that are not 16-byte aligned
        Kn.gemm_tc(a, w, wide[:, :N], b, choice=pair)
        assert torch.equal(wide[:, :N], f32) and bool((wide[:, N:] == 7.0).all())
    assert Kn.tc_status() == 0


@pytest.mark.parametrize("width", [256, 128])
@pytest.mark.parametrize("M,ff,K", [(512, 1408, 256), (1500, 200, 1032), (2048, 5632, 128), (129, 71, 72)])
@pytest.mark.parametrize("activation", ["silu", "relu", "gelu_tanh", "limits"])
def test_pairs_gated(M, ff, K, activation, width):
    from kappai_b200.ops import kernels as Kn
    a, w, bias, z, _ = operands(M, 2 * ff, K, ff)
    glu = (1.5, 1.702, 1.0) if activation == "limits" else None
    out = Kn.gemm_tc(a, w, torch.empty((M, ff), device="cuda", dtype=torch.bfloat16), bias, swiglu=True,
                     activation="silu" if glu else activation, glu=glu, choice=(width, 1, False, True))
    # the unfused path: gate and up as the product stores them, then the row-wise kernel; both round the same float32 value
    # to bfloat16, whose last bits the two compilations of the activation may differ in
    gu = Kn.gemm_tc(a, w, torch.empty((M, 2 * ff), device="cuda", dtype=torch.bfloat16), bias, choice=(width, 1, False, True))
    ref = torch.empty((M, ff), device="cuda", dtype=torch.bfloat16)
    ref = Kn.glu_clamped(gu, ref, *glu) if glu else Kn.swiglu(gu, ref, activation)
    d = (out.double() - ref.double()).abs()
    assert bool((d <= 2.0 ** -7 * ref.double().abs()).all()) and float((d > 0).double().mean()) < 1e-3
    assert Kn.tc_status() == 0


@pytest.mark.parametrize("N,K,gated,rows", [(6144, 2048, False, (1300, 1500, 2048)), (2048, 5632, False, (1500, 2048)), (1024, 4608, False, (2048,)),
                                            (11264, 2048, True, (1300, 2048))])
def test_the_dispatch_takes_pairs_and_rows_keep_their_bits_across_it(N, K, gated, rows):
    """Prompt steps of more than 1,024 rows (no parts along K): with the rows the choice goes from one CTA to a pair, of either width,
    and a row's bits stay."""
    from kappai_b200.ops import kernels as Kn
    a, w, bias, _, _ = operands(max(rows), N, K, N)
    n_out, dtype = (N // 2, torch.bfloat16) if gated else (N, torch.float32)
    run = lambda M: Kn.gemm_tc(a[:M], w, torch.empty(M, n_out, device="cuda", dtype=dtype), bias, swiglu=gated, split=False)
    seen, whole = set(), run(max(rows))
    for M in rows:
        assert Kn.gemm_tc_choice(M, N, K, swiglu=gated, out_dtype=dtype)[1:] == (1, False, True), M
    for M in rows + (1, 64, 128, 129, 257, 513, 700, 1025):
        width, parts, cluster, pair = Kn.gemm_tc_choice(M, N, K, swiglu=gated, split=False, out_dtype=dtype)
        seen.add(pair)
        assert parts == 1 and not cluster
        assert torch.equal(run(M), whole[:M]), (M, width, pair)
    assert seen == {False, True}
    assert Kn.tc_status() == 0
