"""What the products' dispatch says of operands that no kernel takes: no, rather than an error of its own, so that the general
kernel refuses them in its words."""
import pytest
import torch

from kappai_b200.ops import kernels as K
from kappai_b200.ops.linear import linear


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(64,), (2, 4, 64), (4, 63), (64, 4)])
def test_operands_that_are_not_rows_of_16_bytes(shape, dtype):
    a, w = torch.zeros(shape, dtype=dtype), torch.zeros(8, 64, dtype=dtype)
    if shape == (64, 4):
        a = a.t()
    assert not K.skinny_ok(a, w) and not K.tc_ok(a, w)
    assert not K.skinny_ok(w, a) and not K.tc_ok(w, a)
    with pytest.raises(K.KernelError):
        linear(a, w)


def test_operands_that_are():
    a, w = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(8, 64, dtype=torch.bfloat16)
    assert K.skinny_ok(a, w) and K.tc_ok(a, w)
    assert K.skinny_ok(a[:, :32], w[:, :32]) and not K.skinny_ok(a[:, 8:40][:, :24], w[:, :24]) and K.tc_ok(a[:, 8:32], w[:, :24])
