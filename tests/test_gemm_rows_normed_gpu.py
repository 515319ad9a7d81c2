"""Products of up to 8 rows that take the RMS norm of their rows themselves (csrc/gemm_rows.cu) against the norm and the product in
64 bits, at edges of tiles, chunks of K and passes over the rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 1e-5


def exact(x, gamma, w, bias):
    """The sums in 64 bits from what the kernel multiplies (the norm kernel's rows), and the sum of the magnitudes."""
    from kappai_b200.ops import kernels as Kn
    h = Kn.rmsnorm_rows(x, gamma, EPS, torch.empty(x.shape, device="cuda", dtype=torch.bfloat16)).double()
    b = 0.0 if bias is None else bias.double()
    return h @ w.double().T + b, h.abs() @ w.double().abs().T + (0.0 if bias is None else bias.double().abs())


@pytest.mark.parametrize("M", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(2, 512), (330, 1024), (3072, 2048), (1000, 2560), (512, 4096), (16384, 512)])
def test_against_64_bits(M, N, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    x = torch.randn(M, K, device="cuda", generator=g) * torch.logspace(-2, 2, M, device="cuda")[:, None]
    gamma = 1.0 + 0.3 * torch.randn(K, device="cuda", generator=g)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    for b in (None, bias):
        want, size = exact(x, gamma, w, b)
        # K additions that each lose at most 2^-23 of what is there, the mean of squares and its root some 40 roundings
        bound = (K + 40) * 2.0 ** -23 * size
        out = Kn.gemm_rows_normed(x, gamma, EPS, w, torch.full((M, N), float("nan"), device="cuda"), b)
        assert bool(((out.double() - want).abs() <= bound).all())
        half = Kn.gemm_rows_normed(x, gamma, EPS, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), b)
        assert torch.equal(half, out.bfloat16())
        sq = Kn.gemm_rows_normed(x, gamma, EPS, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), b, plain_activation="relu_squared")
        assert torch.equal(sq, (out.clamp(min=0) ** 2).bfloat16())
        act = torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16)
        for kw in ({}, {"activation": "gelu_tanh"}, {"glu": (1.5, 1.702, 1.0)}):
            got = Kn.gemm_rows_normed(x, gamma, EPS, w, act.clone(), b, swiglu=True, **kw)
            ref = (Kn.glu_clamped(half, act.clone(), *kw["glu"]) if "glu" in kw else Kn.swiglu(half, act.clone(), kw.get("activation", "silu")))
            # one rounding of the result apart at most
            assert bool(((got.float() - ref.float()).abs() <= 2.0 ** -7 * ref.float().abs() + 1e-30).all()), kw


@pytest.mark.parametrize("M,d,K,taps", [(1, 512, 512, 3), (8, 1000, 1024, 2), (3, 2048, 4096, 4), (7, 72, 1536, 7)])
def test_conv_step(M, d, K, taps):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(d)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, gamma, w = 3.0 * rnd(M, K), 1.0 + 0.3 * rnd(K), (rnd(3 * d, K) / K ** 0.5).bfloat16()
    cw, cb, b = rnd(d, taps), rnd(d), rnd(3 * d)
    pos = torch.arange(M, device="cuda", dtype=torch.int32)
    slot = torch.arange(M, device="cuda", dtype=torch.int32).flip(0).contiguous() + 1
    state = rnd(M + 2, taps - 1, d)
    for bias, cbias in ((b, cb), (None, None)):
        p = Kn.gemm_rows_normed(x, gamma, EPS, w, torch.empty(M, 3 * d, device="cuda", dtype=torch.bfloat16), bias)
        s1, y1 = state.clone(), torch.empty(M, d, device="cuda", dtype=torch.bfloat16)
        Kn.shortconv_decode(p, cw, cbias, s1, pos, slot, y1)
        s2, y2 = state.clone(), torch.empty_like(y1)
        Kn.gemm_stream_conv_step(x, w, bias, cw, cbias, s2, pos, slot, y2, (gamma, EPS))
        assert torch.equal(y1, y2) and torch.equal(s1, s2)


def test_one_door_norms_the_rows_where_the_kernel_does_not():
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.linear import NormedRows, linear, linear_weights, linear_weights_swiglu
    g = torch.Generator(device="cuda").manual_seed(1)
    gamma = torch.rand(768, device="cuda", generator=g)
    w = torch.randn(64, 768, device="cuda", generator=g).bfloat16()
    for M in (1, 8, 9, 40):
        x = torch.randn(M, 768, device="cuda", generator=g)
        h = Kn.rmsnorm_rows(x, gamma, EPS, torch.empty(M, 768, device="cuda", dtype=torch.bfloat16))
        assert torch.equal(linear_weights(NormedRows(x, gamma, EPS), w), linear(h, w))           # (768 is no multiple of 512)
        assert torch.equal(linear_weights(NormedRows(x, gamma, EPS), w.float()), linear(h, w.float()))
        assert torch.equal(linear_weights_swiglu(NormedRows(x, gamma, EPS), w), linear_weights_swiglu(h, w))
