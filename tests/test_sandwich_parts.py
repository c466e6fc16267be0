"""The sandwich arrangement with parts that a user registers, without a GPU: the calls that it makes of them."""
from types import SimpleNamespace

import pytest
import torch

from mdma_b200.parts.block import SandwichBlock
from mdma_b200.parts.norm import RMSNorm
from mdma_b200.spec import PartSpec

W = 8


class Sublayer:
    """Adds 2 h into a float buffer, or stores it there."""

    def __init__(self):
        self.calls = []

    def forward(self, ctx, h, y):
        self.calls.append("forward")
        y[:ctx.n_tokens] += 2 * h[:ctx.n_tokens].float()

    def produce(self, ctx, h, y, defer=False):
        self.calls.append("produce")
        y[:ctx.n_tokens] = 2 * h[:ctx.n_tokens].float()


class PlainNorm:
    """What the arrangement asks of a norm on a result, and nothing else."""

    def add_normed(self, ctx, y, x):
        x[:ctx.n_tokens] += 3 * y[:ctx.n_tokens]


class StoringNorm(PlainNorm):
    adds_stored = True

    def add_normed(self, ctx, y, x, stored=False):
        assert stored
        super().add_normed(ctx, y, x)


@pytest.mark.parametrize("norm,call", [(PlainNorm(), "forward"), (StoringNorm(), "produce")])
def test_a_norm_takes_a_sublayers_result_as_it_offers_to(norm, call):
    ctx, part = SimpleNamespace(n_tokens=3), Sublayer()
    h, x, y = torch.arange(4.0 * W).view(4, W), torch.ones(4, W), torch.full((4, W), 7.0)
    SandwichBlock._sublayer(ctx, part, norm, h, x, y)
    assert part.calls == [call]
    assert torch.equal(x[:3], 1 + 6 * h[:3]) and torch.equal(x[3], torch.ones(W))


def test_the_rms_norm_takes_stored_results_unless_it_works_in_groups():
    make = lambda **more: RMSNorm(PartSpec("rmsnorm", dict(width=W, eps=1e-5, **more)))  # noqa: E731
    assert make().adds_stored and not make(groups=2).adds_stored


def test_a_norm_in_groups_with_its_own_sum_gets_added_results():
    """The RMS norm in groups takes stored results; one derived from it that adds in its own way is asked as before."""
    class Tripled(RMSNorm):
        def add_normed(self, ctx, y, x):
            x[:ctx.n_tokens] += 3 * y[:ctx.n_tokens]

    make = lambda cls: cls(PartSpec("rmsnorm", dict(width=W, eps=1e-5, groups=2)))  # noqa: E731
    assert make(RMSNorm).completes_stored
    ctx, part = SimpleNamespace(n_tokens=3), Sublayer()
    h, x, y = torch.arange(4.0 * W).view(4, W), torch.ones(4, W), torch.full((4, W), 7.0)
    SandwichBlock._sublayer(ctx, part, make(Tripled), h, x, y)
    assert part.calls == ["forward"] and torch.equal(x[:3], 1 + 6 * h[:3])
