"""Products of up to 8 rows that take the RMS norm of their rows themselves (csrc/gemm_rows.cu): the bits of the norm kernel and the
product behind it, at edges of tiles, chunks of K and passes over the rows, and those of a row among more rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = 1e-5


def normed(Kn, x, gamma):
    return Kn.rmsnorm_rows(x, gamma, EPS, torch.empty(x.shape, device="cuda", dtype=torch.bfloat16))


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(2, 512), (330, 1024), (520, 1536), (3072, 2048), (1000, 2560), (512, 4096), (16384, 512)])
def test_the_bits_of_the_norm_and_the_product(M, N, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    x = torch.randn(M, K, device="cuda", generator=g) * torch.logspace(-2, 2, M, device="cuda")[:, None]
    gamma = 1.0 + 0.3 * torch.randn(K, device="cuda", generator=g)
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    h = normed(Kn, x, gamma)
    new = lambda n, dtype=torch.bfloat16: torch.full((M, n), float("nan"), device="cuda", dtype=dtype)
    for b in (None, bias):
        out = Kn.gemm_rows_normed(x, gamma, EPS, w, new(N, torch.float32), b)
        assert torch.equal(out, Kn.gemm_skinny(h, w, new(N, torch.float32), b))
        add = 0.0 if b is None else b.double()
        want, size = h.double() @ w.double().T + add, h.double().abs() @ w.double().abs().T + abs(add)
        assert bool(((out.double() - want).abs() <= K * 2.0 ** -23 * size).all())       # K additions, each off by 2^-23 of what is there
        assert torch.equal(Kn.gemm_rows_normed(x, gamma, EPS, w, new(N), b), Kn.gemm_skinny(h, w, new(N), b))
        assert torch.equal(Kn.gemm_rows_normed(x, gamma, EPS, w, new(N), b, plain_activation="relu_squared"),
                           Kn.gemm_skinny(h, w, new(N), b, plain_activation="relu_squared"))
        for kw in ({}, {"activation": "gelu_tanh"}, {"glu": (1.5, 1.702, 1.0)}):
            assert torch.equal(Kn.gemm_rows_normed(x, gamma, EPS, w, new(N // 2), b, swiglu=True, **kw),
                               Kn.gemm_skinny(h, w, new(N // 2), b, swiglu=True, **kw)), kw


@pytest.mark.parametrize("K", [1024, 4096])
def test_rows_of_any_size(K):
    """Squares that overflow (the norm is then zero, or NaN), infinities, NaN, subnormal values: as the norm kernel has them."""
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(K)
    x, gamma = torch.randn(8, K, device="cuda", generator=g), 1.0 + 0.3 * torch.randn(K, device="cuda", generator=g)
    x[0] = 0.0
    x[1] *= 1e25
    x[2] = 3e38
    x[3, 7] = float("inf")
    x[4, K - 1] = float("nan")
    x[5] *= 1e-39
    w = (torch.randn(40, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    got, want = (f(torch.empty(8, 40, device="cuda")) for f in (lambda o: Kn.gemm_rows_normed(x, gamma, EPS, w, o),
                                                                lambda o: Kn.gemm_skinny(normed(Kn, x, gamma), w, o)))
    assert bool((got[1] == 0).all()) and bool((got[2] == 0).all())
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got.nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("K", [1024, 2048, 2560])
def test_a_row_keeps_its_bits_when_a_ninth_joins(K):
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.linear import NormedRows, linear_weights, linear_weights_swiglu
    g = torch.Generator(device="cuda").manual_seed(K)
    x, gamma = 2.0 * torch.randn(9, K, device="cuda", generator=g), 1.0 + 0.3 * torch.randn(K, device="cuda", generator=g)
    w = (torch.randn(1024, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    h = normed(Kn, x, gamma)
    for f in (linear_weights, linear_weights_swiglu):
        nine = f(h, w)
        for M in (1, 3, 8):
            assert torch.equal(f(NormedRows(x[:M], gamma, EPS), w), nine[:M])


@pytest.mark.parametrize("M,d,K,taps", [(1, 512, 512, 3), (8, 1000, 1024, 2), (3, 2048, 4096, 4), (7, 72, 1536, 7), (2, 40, 512, 5), (5, 24, 512, 8),
                                        (4, 520, 512, 9), (8, 16, 512, 12), (1, 300, 1024, 16)])
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
        p = Kn.gemm_skinny(normed(Kn, x, gamma), w, torch.empty(M, 3 * d, device="cuda", dtype=torch.bfloat16), bias)
        s1, y1 = state.clone(), torch.empty(M, d, device="cuda", dtype=torch.bfloat16)
        Kn.shortconv_decode(p, cw, cbias, s1, pos, slot, y1)
        s2, y2 = state.clone(), torch.empty_like(y1)
        Kn.gemm_stream_conv_step(x, w, bias, cw, cbias, s2, pos, slot, y2, (gamma, EPS))
        assert torch.equal(y1, y2) and torch.equal(s1, s2)


@pytest.mark.parametrize("off", [0, 1, 2])
def test_a_norm_weight_that_is_part_of_a_larger_one(off):
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.linear import NormedRows, linear_weights
    g = torch.Generator(device="cuda").manual_seed(off)
    x, gamma = torch.randn(3, 1024, device="cuda", generator=g), torch.rand(1026, device="cuda", generator=g)[off:off + 1024]
    w = (torch.randn(72, 1024, device="cuda", generator=g) / 32).bfloat16()
    assert torch.equal(linear_weights(NormedRows(x, gamma, EPS), w), linear_weights(normed(Kn, x, gamma), w))
