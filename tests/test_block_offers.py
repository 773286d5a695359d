"""What a block hands to parts that offer to take it (the residual stream to add to, a norm that is still to be formed), and that a
part which derives from such a one with a ``forward`` of its own is given neither."""
from types import SimpleNamespace

import pytest
import torch

from snowllm_b200.ops import kernels
from snowllm_b200.parts.attention import Attention
from snowllm_b200.parts.base import offered
from snowllm_b200.parts.block import PreNormBlock
from snowllm_b200.parts.ffn_dense import GatedFFN, SwiGLU
from snowllm_b200.parts.norm import RMSNorm
from snowllm_b200.parts.short_conv import ShortConv

PENDING = object()


class Norm:
    def forward(self, ctx, residual, delta=None, rows=None):
        if delta is not None:
            residual += delta
        return residual.clone()

    def before(self, ctx, residual, delta, w):
        self.forward(ctx, residual, delta)
        return PENDING


class Doubles:
    adds_to_stream = True

    def reads_pending_norm(self, *args):
        return torch.ones(1)

    def forward(self, ctx, x, *args):
        self.seen = (x is PENDING, ctx.stream is not None)
        out = torch.ones(ctx.M, 4) if x is PENDING else 2 * x
        if ctx.stream is not None:
            ctx.stream += out
            return None
        return out


class DoublesAndHalves(Doubles):
    """Works on what the part above returns."""

    def forward(self, ctx, x, *args):
        return super().forward(ctx, x, *args) * 0.25


class LoudNorm(Norm):
    def forward(self, ctx, residual, delta=None, rows=None):
        return super().forward(ctx, residual, delta) + 1


def step(part, M, norm=Norm):
    ctx = SimpleNamespace(M=M, taps=None, stream=None, tap=lambda *a: None)
    residual = torch.ones(M, 4)
    delta = PreNormBlock(part, part, norm(), norm()).forward(ctx, residual, None, None)
    assert ctx.stream is None
    return residual if delta is None else residual + delta


def test_a_part_is_given_what_it_offers_to_take():
    part = Doubles()
    assert torch.equal(step(part, 40), torch.full((40, 4), 9.0)) and part.seen == (False, True)
    step(part, kernels.PENDING_NORM_ROWS)
    assert part.seen == (True, True)


@pytest.mark.parametrize("M", [1, 40])
def test_a_part_with_a_forward_of_its_own_is_not(M):
    part = DoublesAndHalves()
    assert torch.equal(step(part, M), torch.full((M, 4), 2.25)) and part.seen == (False, False)
    loose = Doubles()
    loose.forward = lambda ctx, x, *args: torch.zeros(ctx.M, 4) if ctx.stream is None and x is not PENDING else None
    assert torch.equal(step(loose, M), torch.ones(M, 4))
    step(loose, M)


def test_nor_is_a_norm_asked_for_what_another_one_offers():
    part = Doubles()
    step(part, 1, LoudNorm)
    assert part.seen == (False, True)


def test_what_the_framework_s_own_parts_offer():
    for cls in (Attention, ShortConv, SwiGLU, GatedFFN):
        part = cls.__new__(cls)
        assert offered(part, "adds_to_stream") and offered(part, "reads_pending_norm")
    assert offered(RMSNorm.__new__(RMSNorm), "before")


def test_a_stream_that_somebody_else_looks_at_stays_where_it_is(monkeypatch):
    """A product that forms the norm in front of it moves the stream to other memory: not while a view of it is held."""
    monkeypatch.setattr(kernels, "_norm_product_sizes_ok", lambda *sizes: True)
    residual, delta, gamma = torch.zeros(2, 64), torch.ones(2, 64), torch.ones(64, dtype=torch.bfloat16)
    w = torch.zeros(4096, 64, dtype=torch.bfloat16)

    def ok(delta):
        return kernels.PendingNorm.ok(residual, delta, gamma, torch.bfloat16, w)

    experts = kernels.ExpertSum(torch.ones(4, 64), torch.arange(4, dtype=torch.int32), torch.ones(2, 2))
    assert ok(delta) and ok(experts)
    for look in (lambda: residual[0], lambda: residual.view(-1), lambda: residual.detach()):
        held = look()
        assert not ok(delta) and not ok(experts)
        assert ok(None)                                  # nothing is added: the stream is not moved
        del held
        assert ok(delta)


def test_a_delta_off_a_16_byte_boundary_is_left_to_the_norm_s_kernel(monkeypatch):
    """The norm's kernel takes such a delta an element at a time; a product that forms the norm reads 16 bytes and refuses it."""
    monkeypatch.setattr(kernels, "_norm_product_sizes_ok", lambda *sizes: True)
    residual, gamma, w = torch.zeros(2, 64), torch.ones(64, dtype=torch.bfloat16), torch.zeros(4096, 64, dtype=torch.bfloat16)
    for lead in range(5):
        delta = torch.ones(lead + 128)[lead:].view(2, 64)
        assert kernels.PendingNorm.ok(residual, delta, gamma, torch.bfloat16, w) == (lead % 4 == 0)
