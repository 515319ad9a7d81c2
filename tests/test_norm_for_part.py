"""Which norms are left to the product behind them: an RMS norm's own, for a part whose forward is marked as one that takes the rows
before the norm, in bfloat16 steps of up to 8 rows; nobody else's."""
import pytest
import torch

from kappai_b200.ops.linear import NormedRows
from kappai_b200.parts.base import BuildEnv
from kappai_b200.parts.norm import LayerNorm, RMSNorm


class Marked:
    def forward(self, h):
        pass

    forward.takes_normed_rows = True


class Overridden(Marked):
    def forward(self, h):
        pass


class OtherNorm(RMSNorm):
    def forward(self, x, rows=None):
        return "its own"


def norm(cls, dtype=torch.bfloat16):
    n = cls({"size": 512, "eps": 1e-5}, BuildEnv(torch.device("cpu"), dtype, 16))
    n.weight = torch.ones(512)
    return n


def test_left_to_the_product():
    x = torch.zeros(8, 512)
    h = norm(RMSNorm).forward_for(Marked(), x)
    assert isinstance(h, NormedRows) and h.x is x and h.shape == x.shape


@pytest.mark.parametrize("cls,part,rows,dtype", [(RMSNorm, Overridden, 8, torch.bfloat16), (RMSNorm, Marked, 9, torch.bfloat16),
                                                 (RMSNorm, Marked, 8, torch.float32), (LayerNorm, Marked, 8, torch.bfloat16),
                                                 (OtherNorm, Marked, 8, torch.bfloat16)])
def test_taken_by_the_norm(monkeypatch, cls, part, rows, dtype):
    from kappai_b200.parts import norm as module
    for name in ("rmsnorm_rows", "layernorm_rows"):
        monkeypatch.setattr(module.K, name, lambda *a: "normed")
    got = norm(cls, dtype).forward_for(part(), torch.zeros(rows, 512))
    assert got == ("its own" if cls is OtherNorm else "normed")


@pytest.mark.parametrize("rows", [1, 8, 9, 999])
def test_asked_in_steps_of_few_rows_only(rows):
    """A step of more rows launches from Python and waits for it: nothing is asked there whose answer is always no."""
    from types import SimpleNamespace
    from kappai_b200.parts.block import PreNormResidualBlock
    calls = []

    class Norm:
        def forward(self, x):
            calls.append("norm")
            return "normed"

        def forward_for(self, part, x):
            calls.append("asked")
            return "left"

    class Sublayer:
        def forward(self, h, *args):
            calls.append(h)

    block = PreNormResidualBlock({}, BuildEnv(torch.device("cpu"), torch.bfloat16, 16)).assemble(Sublayer(), Sublayer(), Norm(), Norm())
    block.forward(torch.zeros(rows, 4), SimpleNamespace(n_rows=rows), None)
    assert calls == (["asked", "left"] if rows <= 8 else ["norm", "normed"]) * 2


def test_a_weight_off_its_boundary_is_left_to_the_norm_kernel():
    """The product reads the norm's weight 16 bytes at a time; the norm kernel takes any."""
    x, w = torch.zeros(3, 512), torch.zeros(64, 512, dtype=torch.bfloat16)
    whole = torch.ones(516)
    assert NormedRows(x, whole[:512], 1e-5).fusable(w) and NormedRows(x, whole[4:], 1e-5).fusable(w)
    for off in (1, 2, 3):
        assert not NormedRows(x, whole[off:off + 512], 1e-5).fusable(w)
