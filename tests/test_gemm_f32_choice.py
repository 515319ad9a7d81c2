"""Which kernel a float32 product runs on (csrc/gemm_simt.cu, f32_choose): a long K keeps the few-row kernels, with fewer warps
where the sums of its stretches take the room, and no grid is larger than the device takes."""
import ctypes

import pytest


def choice(M, N, K):
    from kappai_b200.ops.build import load_library
    out = (ctypes.c_int * 4)()
    assert load_library("gemm_simt").kp_gemm_f32_choice(M, N, K, out) == 0
    return tuple(out)


@pytest.mark.parametrize("M,N,K,R,MB", [(32, 4096, 3076, 4, 16), (32, 4096, 4096, 4, 16), (32, 4096, 7168, 4, 16), (64, 2048, 8192, 4, 16),
                                        (6, 4096, 16384, 2, 8), (1, 4096, 65536, 2, 1), (8, 2048, 5632, 1, 8), (16, 65536, 1024, 4, 16)])
def test_rows_kernels_take_every_k_their_sums_leave_room_for(M, N, K, R, MB):
    r, mb, warps, stages = choice(M, N, K)
    assert (r, mb) == (R, MB) and warps >= 1 and stages >= 2
    jobs = -(-K // 1024)
    assert warps * stages * (8 * R + MB) * 512 + jobs * 4 * MB * 8 * R * 4 <= 227 * 1024


@pytest.mark.parametrize("M,N,K", [(2048, 2048, 2048), (128, 2048, 12288), (96, 1024, 20480), (400, 1024, 1024), (8, 4096, 400000)])
def test_tiles(M, N, K):
    assert choice(M, N, K)[0] == 0


def test_rows_beyond_a_grid_take_tiles():
    assert choice(16 * 65535, 8, 64)[0] == 4 and choice(16 * 65535 + 1, 8, 64)[0] == 0
