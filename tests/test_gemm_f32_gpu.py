"""The float32 product with 16-byte rows (csrc/gemm_simt.cu): its two kernels at the edges of their tiles, stretches and
jobs against float64, and one order of summation whatever the number of rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = (1, 2, 3, 4, 5, 8, 9, 16, 24, 25, 40, 64, 65, 130)      # few-row kernels of 1, 2, 4, 8 and 16 rows a pass, tiles of 64


@pytest.mark.parametrize("N,K", [(1, 4), (33, 252), (72, 256), (100, 260), (2050, 1024), (200, 1028), (331, 4100), (64, 9000),
                                 (5000, 512)])
def test_against_float64_and_one_order_for_every_number_of_rows(N, K):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(N * 10007 + K)
    a = torch.randn(max(ROWS), K + 4, device="cuda", generator=g)[:, :K]        # (rows longer than K)
    w = torch.randn(N, K, device="cuda", generator=g)
    bias = torch.randn(N, device="cuda", generator=g)
    exact = a.double() @ w.double().T
    # a chain of 128 FMAs, its partner, one sum a stretch of 256: each rounds at most eps/2 of the sum of magnitudes
    bound = (128 + 1 + -(-K // 256) + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T + bias.double().abs()) * 1.01
    whole = None
    for M in reversed(ROWS):
        out = Kn.gemm_nt_simt(a[:M], w, torch.full((M, N), float("nan"), device="cuda"))
        assert bool(((out.double() - exact[:M]).abs() <= bound[:M]).all()), (M, N, K)
        whole = out if whole is None else whole
        assert torch.equal(out, whole[:M]), f"{M} rows: another order of summation"
        acc = torch.ones(M, N, device="cuda")
        Kn.gemm_nt_simt(a[:M], w, acc, bias, accumulate=True)
        assert torch.equal(acc, 1.0 + (out + bias)), M
    last = Kn.gemm_nt_simt(a[-1:], w, torch.empty(1, N, device="cuda"))
    assert torch.equal(last[0], whole[-1])


def test_rows_that_are_not_16_byte_aligned_take_the_general_kernel():
    from kappai_b200.ops import kernels as Kn
    base = torch.randn(9, 130, device="cuda")
    w = torch.randn(70, 130, device="cuda")
    for a_ in (base[:, :127], base[:, 1:128], base):                            # K, address and pitch that are none
        k = a_.shape[1]
        out = Kn.gemm_nt_simt(a_, w[:, :k], torch.empty(9, 70, device="cuda"))
        exact = a_.double() @ w[:, :k].double().T
        bound = (k + 2) * 2.0 ** -24 * (a_.double().abs() @ w[:, :k].double().abs().T)
        assert bool(((out.double() - exact).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(1, 8192, 2048), (8, 4096, 4096), (40, 4096, 2048), (300, 2048, 4096)])
def test_second_operand_written_by_the_launch_in_front(M, N, K):
    """(The cast lets the launch behind it in at its start.)"""
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.linear import linear
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, device="cuda", generator=g)
    sources = [torch.randn(N, K, device="cuda", generator=g).bfloat16() for _ in range(3)]
    want = [Kn.gemm_nt_simt(a, s.float(), torch.empty(M, N, device="cuda"), w_settled=True) for s in sources]
    w = torch.zeros(N, K, device="cuda")
    torch.cuda.synchronize()
    for i in range(12):
        Kn.cast(sources[i % 3], w)
        out = Kn.gemm_nt_simt(a, w, torch.empty(M, N, device="cuda")) if i % 2 else linear(a, w)
        assert torch.equal(out, want[i % 3]), i


def test_launches_of_different_sizes_from_several_threads():
    """The kernels' limit on shared memory belongs to the function: one thread's small launch must not lower it for another's
    (of 20,000 launches a thread 970 to 2,973 failed where each set its own)."""
    import ctypes
    import threading
    from kappai_b200.ops import kernels as Kn
    from kappai_b200.ops.build import load_library
    launch = load_library("gemm_simt").kp_gemm_nt_simt
    failed, keep = [0] * 4, []
    shapes = [(8, 64, 5632), (8, 64, 1024), (8, 64, 2048), (8, 64, 4608)]                # one instantiation, 70 to 200 KB

    def work(i, args, stream):
        for _ in range(5000):
            failed[i] += launch(*args) != 0
        stream.synchronize()

    threads = []
    for i, (M, N, K) in enumerate(shapes):
        a, w, out, s = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda"), torch.empty(M, N, device="cuda"), torch.cuda.Stream()
        keep.append((a, w, out))
        args = [Kn._ptr(a), Kn._ptr(w), Kn._ptr(None), Kn._ptr(out)] + [ctypes.c_int(v) for v in (M, N, K, K, K, N, 0, 0, 0)]
        threads.append(threading.Thread(target=work, args=(i, args + [ctypes.c_void_p(s.cuda_stream)], s)))
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == [0] * 4


@pytest.mark.parametrize("M,N,K", [(5, 300, 16384), (8, 2400, 4096), (8, 2500, 36864), (33, 1100, 3076), (40, 1100, 4096), (17, 700, 7168),
                                   (64, 1100, 8192), (25, 100, 20480)])
def test_long_sums(M, N, K):
    """Where the stretches' sums leave the few-row kernels fewer warps, or none: the bits of the tiles."""
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(K)
    a, w = torch.randn(2048, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    tiles = Kn.gemm_nt_simt(a, w, torch.empty(2048, N, device="cuda"))
    assert torch.equal(Kn.gemm_nt_simt(a[:M], w, torch.empty(M, N, device="cuda")), tiles[:M])


def test_more_rows_than_a_grid_has():
    from kappai_b200.ops import kernels as Kn
    M = 16 * 65535 + 40
    a, w = torch.randn(M, 8, device="cuda"), torch.randn(8, 8, device="cuda")
    out = Kn.gemm_nt_simt(a, w, torch.empty(M, 8, device="cuda"))
    for lo in (0, M - 130):
        assert torch.equal(out[lo:lo + 130], Kn.gemm_nt_simt(a[lo:lo + 130], w, torch.empty(130, 8, device="cuda")))
