"""Split-key attention of rows whose keys are one chunk: the chunk pass writes them itself, with the bits that the merge makes of
that chunk."""
import math

import numpy as np
import pytest
import torch

from test_attention_split_gpu import run_split
from test_kernels_gpu import paged_setup, rt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd,page,window", [(4, 4, 64, 16, None), (8, 4, 64, 64, None), (8, 2, 64, 8, 37), (8, 1, 64, 128, None),
                                                (6, 2, 64, 16, 100), (4, 2, 128, 16, None), (5, 1, 48, 32, 17)])
def test_the_bits_of_the_merge(dtype, H, G, hd, page, window):
    rng = np.random.default_rng(7)
    seq_lens = [1, 2, 31, 33, 64, 200, 256]
    cache, bt, _, _ = paged_setup(rng, seq_lens, page, G, hd, dtype)
    pos, seg = [n - 1 for n in seq_lens] + [100], list(range(len(seq_lens))) + [5]
    q = rt(rng.standard_normal((len(pos), H * hd)), dtype)
    one = run_split(q, cache, bt, seg, pos, 1.0 / math.sqrt(hd), window, page, H, G, hd, dtype, n_chunks=1)
    assert bool(torch.isfinite(one.float()).all())
    assert torch.equal(one, run_split(q, cache, bt, seg, pos, 1.0 / math.sqrt(hd), window, page, H, G, hd, dtype, n_chunks=3))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd,longest,chunks", [(4, 2, 64, 2000, (8, 9, 40, 64)), (3, 1, 48, 2048, (8, 9, 33)), (4, 1, 80, 1999, (8, 9, 17)),
                                                   (4, 2, 128, 2048, (8, 16, 64)), (2, 2, 64, 8500, (34, 64)), (2, 1, 128, 8500, (34, 64))])
def test_how_many_chunks_the_merge_fetches_at_a_time_changes_no_bit(dtype, H, G, hd, longest, chunks):
    rng = np.random.default_rng(8)
    seq_lens = [1, 256, 257, longest]
    cache, bt, _, _ = paged_setup(rng, seq_lens, 64, G, hd, dtype)
    pos, seg = [n - 1 for n in seq_lens], list(range(len(seq_lens)))
    q = rt(rng.standard_normal((len(pos), H * hd)), dtype)
    outs = [run_split(q, cache, bt, seg, pos, 1.0 / math.sqrt(hd), None, 64, H, G, hd, dtype, n_chunks=n) for n in chunks]
    assert bool(torch.isfinite(outs[0].float()).all())
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
