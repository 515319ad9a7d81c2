"""Products of up to 8 bfloat16 rows (csrc/gemm_rows.cu): the bits of csrc/gemm_stream.cu, whose order of summation it keeps,
at edges of its tiles and rings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def both(monkeypatch, run):
    from kappai_b200.ops import kernels as Kn
    a = run()
    monkeypatch.setattr(Kn, "ROWS_MAX_M", 0)
    b = run()
    monkeypatch.undo()
    return a, b


@pytest.mark.parametrize("M", [1, 2, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 512), (7, 1024), (330, 512), (1024, 4608), (2050, 2048), (5000, 512), (16384, 512)])
def test_same_bits_as_the_streaming_kernel(monkeypatch, M, N, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()[:, :K]
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g)
    x = torch.randn(M, N, device="cuda", generator=g)
    for b in (None, bias):
        for run in (lambda: Kn.gemm_skinny(a, w, torch.empty(M, N, device="cuda"), b),
                    lambda: Kn.gemm_skinny(a, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), b),
                    lambda: Kn.gemm_skinny(a, w, torch.empty(M, N, device="cuda", dtype=torch.bfloat16), b, plain_activation="relu_squared"),
                    lambda: Kn.gemm_skinny(a, w, x.clone(), b, accumulate=True)):
            one, two = both(monkeypatch, run)
            assert torch.equal(one, two)
        if N % 2 == 0:
            for kw in ({"activation": "silu"}, {"activation": "gelu_tanh"}, {"glu": (1.5, 1.702, 1.0)}):
                one, two = both(monkeypatch, lambda: Kn.gemm_skinny(a, w, torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16), b,
                                                                    swiglu=True, **kw))
                assert torch.equal(one, two), kw
    assert Kn.stream_status() == 0


@pytest.mark.parametrize("N,K", [(65536, 1024), (40003, 512), (32768, 2048)])
def test_one_row_of_a_head_has_the_sums_of_the_register_kernel(monkeypatch, N, K):
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.linear import linear
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn(1, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    one = linear(a, w, out_dtype=torch.float32)
    monkeypatch.setattr(Kn, "USE_STREAM", False)
    two = Kn.gemm_skinny(a, w, torch.empty(1, N, device="cuda"))
    assert torch.equal(one, two)


@pytest.mark.parametrize("M,d,K,taps", [(1, 512, 512, 3), (8, 1000, 1024, 2), (3, 2048, 512, 4), (7, 72, 1536, 7)])
def test_conv_step_same_bits_and_state(monkeypatch, M, d, K, taps):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(d)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a, w = rnd(M, K).bfloat16(), (rnd(3 * d, K) / K ** 0.5).bfloat16()
    cw, cb, b = rnd(d, taps), rnd(d), rnd(3 * d)
    pos = torch.arange(M, device="cuda", dtype=torch.int32)               # row 0 starts its sequence
    slot = torch.arange(M, device="cuda", dtype=torch.int32).flip(0).contiguous() + 1
    state = rnd(M + 2, taps - 1, d)
    for bias, cbias in ((b, cb), (None, None)):
        def run():
            st, y = state.clone(), torch.empty(M, d, device="cuda", dtype=torch.bfloat16)
            Kn.gemm_stream_conv_step(a, w, bias, cw, cbias, st, pos, slot, y)
            return torch.cat([y.float().reshape(-1), st.reshape(-1)])
        one, two = both(monkeypatch, run)
        assert torch.equal(one, two)
