"""Draws from rows of many candidates (the masses of equal parts of the range of probabilities, then a sort of the part that
holds the crossing) against the cumulative distribution in float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rows(kind, rows, vocab, g):
    x = torch.randn(rows, vocab, device=DEV, generator=g)
    if kind == "flat":
        return x * 0.2
    if kind == "wide":
        return x * 4.0
    if kind == "steps":                 # few different probabilities: thousands of ties in every one
        return torch.round(x * 2) / 8
    if kind == "same":                  # all equal
        return torch.zeros_like(x)
    assert kind == "peak"
    x = x * 0.5
    x[:, 17] = 9.0
    return x


@pytest.mark.parametrize("kind", ["flat", "wide", "steps", "same", "peak"])
@pytest.mark.parametrize("vocab", [1033, 32000, 128256])
@pytest.mark.parametrize("top_p,min_p,temperature", [(0.95, 0.05, 0.8), (1.0, 0.0, 1.0), (0.3, 0.0, 1.3), (0.9999, 1e-4, 0.6), (1e-6, 0.0, 1.0), (0.9, 0.9, 1.0)])
def test_draws_lie_where_the_distribution_puts_them(kind, vocab, top_p, min_p, temperature):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(vocab + int(top_p * 1000))
    rows = 12
    logits = _rows(kind, rows, vocab, g)
    u = torch.rand(rows, device=DEV, generator=g)
    u[0], u[1] = 0.0, 1.0 - 2.0 ** -24
    tokens = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    scratch = torch.empty(ops.sample_scratch_words(rows, vocab), device=DEV)
    ops.sample(logits.contiguous(), u, tokens, scratch, temperature, top_p, min_p, 1.0, 0, impl=2)
    z = logits.double() / temperature
    p = torch.softmax(z, -1)
    top = p.amax(-1, keepdim=True)
    # float32 exponentials and sums of a vocabulary: probabilities within 1e-5 of their own size
    eps = 1e-5
    low = torch.where(p < top * min_p * (1 + eps), torch.zeros_like(p), p)        # surely there
    high = torch.where(p < top * min_p * (1 - eps), torch.zeros_like(p), p)       # possibly there
    key = logits.double() * 1.0
    ids = torch.arange(vocab, device=DEV)
    for r in range(rows):
        t = int(tokens[r])
        assert 0 <= t < vocab and float(high[r, t]) > 0, (r, t)
        ahead = (key[r] > key[r, t]) | ((key[r] == key[r, t]) & (ids < t))

        def kept(q):
            mass = float(q.sum())
            return mass if top_p >= 1.0 else min(mass, max(top_p, float(top[r])) + float(q.max()))
        before, here = float(low[r][ahead].sum()), float(p[r, t])
        # the running mass before the token is at most the target, and with the token at least the target
        most = float(u[r]) * kept(high[r])
        least = float(u[r]) * (float(low[r].sum()) if top_p >= 1.0 else min(float(low[r].sum()), top_p))
        # and the crossing itself may fall one token further where the running mass meets the target within that rounding
        slack = 2 * eps + vocab * 2.0 ** -40 + here
        assert before <= most + slack, (r, t, before, most)
        assert float(high[r][ahead].sum()) + here >= least - slack, (r, t, here, least)
        if top_p < 1.0:                  # inside the prefix that top-p keeps
            assert before < top_p + slack


def test_few_and_many_candidates_meet():
    """1,024 candidates are sorted at once, 1,025 go through the bins: the same draws on either side of the line."""
    from mdma_b200 import ops
    for n in (1024, 1025):
        logits = torch.full((64, 5000), -40.0, device=DEV)
        logits[:, :n] = torch.linspace(0, -1.5, n, device=DEV)
        u = (torch.arange(64, device=DEV) + 0.5) / 64
        tokens = torch.empty(64, dtype=torch.int32, device=DEV)
        ops.sample(logits, u, tokens, torch.empty(ops.sample_scratch_words(64, 5000), device=DEV), 1.0, 0.9, 1e-3, 1.0, 0, impl=2)
        p = torch.softmax(logits[0].double(), -1)
        cum = p.cumsum(0)
        cut = int((cum < 0.9).sum())
        want = [int((cum < float(v) * float(cum[cut])).sum()) for v in u]
        assert all(abs(a - b) <= 1 for a, b in zip(tokens.tolist(), want)), n
        assert sum(a != b for a, b in zip(tokens.tolist(), want)) <= 1 and not math.isnan(float(p.sum()))
