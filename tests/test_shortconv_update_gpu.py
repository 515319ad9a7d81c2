"""The convolution that writes its segments' new history itself (csrc/shortconv.cu): the bits of the forward and the update
kernel launched one after the other, for segments that begin and end anywhere in its chunks of eight rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,K", [(64, 2), (1032, 3), (2048, 3), (512, 4), (72, 5), (100, 3)])
@pytest.mark.parametrize("lens", [[1], [2], [3], [7, 1, 1, 1], [1, 2, 3, 1, 2, 9, 1, 1], [6, 2, 16, 8], [23, 4, 1], [5, 40, 3, 2, 2, 2]])
def test_forward_with_update(dtype, d, K, lens):
    from kappai_b200.ops import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(d * 100 + K)
    n, n_seg = sum(lens), len(lens)
    p = torch.randn(n, 3 * d, device="cuda", generator=g).to(dtype)
    w, b = torch.randn(d, K, device="cuda", generator=g), torch.randn(d, device="cuda", generator=g)
    i32 = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32)).cuda()
    tables = (i32(np.repeat(np.arange(n_seg), lens)), i32(np.concatenate([[0], np.cumsum(lens)])),
              i32([0 if i % 3 == 1 else 5 * i + 4 for i in range(n_seg)]), i32(np.arange(n_seg)[::-1] + 2))
    state = torch.randn(n_seg + 3, K - 1, d, device="cuda", generator=g)
    one, two = state.clone(), state.clone()
    a = Kn.shortconv_forward(p, w, b, one, *tables, torch.empty(n, d, device="cuda", dtype=dtype))
    Kn.shortconv_update_state(p, one, *tables[1:], n_seg)
    c = Kn.shortconv_forward(p, w, b, two, *tables, torch.empty(n, d, device="cuda", dtype=dtype), update=True)
    assert torch.equal(a, c) and torch.equal(one, two)
