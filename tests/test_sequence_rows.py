"""The short convolution and the gated norm of prompts: eight rows a block, four numbers at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lengths", [(512,), (1, 2, 3, 4, 0, 9, 506), (600, 5, 1)])
@pytest.mark.parametrize("channels,dtype", [(4, torch.bfloat16), (1028, torch.float32), (4352, torch.bfloat16)])
@pytest.mark.parametrize("silu", [True, False])
def test_short_convolution(lengths, channels, dtype, silu):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(channels + len(lengths))
    T, n, taps = sum(lengths), len(lengths), 4
    proj = torch.randn(T + 1, channels + 12, device=DEV, generator=g)
    w, b = (torch.randn(channels, k, device=DEV, generator=g).to(dtype) for k in (taps, 1))
    b = b.reshape(-1).contiguous()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    start = i32([sum(lengths[:i]) for i in range(n + 1)])
    seq = i32([s for s, k in enumerate(lengths) for _ in range(k)])
    slot = torch.arange(n, dtype=torch.int32, device=DEV).flip(0).contiguous()
    state = torch.randn(n, 3 * channels + 4, device=DEV, generator=g)
    first = state.clone()
    out = torch.full((T + 1, channels), 9.0, device=DEV)
    (ops.causal_conv_silu if silu else lambda *a: ops.causal_conv_silu(*a, silu=False))(
        proj, 8, w, b, taps, channels, seq, start, slot, state, out, T, n)
    assert bool((out[T:] == 9.0).all())
    for s, k in enumerate(lengths):
        at = int(start[s])
        kept = first[slot[s], :3 * channels].double().view(3, channels)
        rows = torch.cat([kept, proj[at:at + k, 8:8 + channels].double()])
        y = b.double() + sum(rows[j:j + k] * w.double()[:, j] for j in range(taps))
        want = y * torch.sigmoid(y) if silu else y
        assert bool(((out[at:at + k] - want).abs() <= 2e-6 * (1 + want.abs()) * 4).all())        # four products and a sigmoid
        assert torch.equal(state[slot[s], :3 * channels].double().view(3, channels), rows[-3:]) or k == 0
    assert torch.equal(state[:, 3 * channels:], first[:, 3 * channels:])


@pytest.mark.parametrize("width,groups", [(516, 1), (2048, 2), (4096, 1), (8192, 1), (3 * 1032, 3)])
@pytest.mark.parametrize("rows", [256, 300])
def test_gated_norm(width, groups, rows):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(width)
    y, z = (torch.randn(rows + 1, width, device=DEV, generator=g) for _ in range(2))
    w = torch.randn(width, device=DEV, generator=g).bfloat16()
    out = torch.full((rows + 1, width), 9.0, device=DEV, dtype=torch.bfloat16)
    ops.gated_group_rmsnorm(y, z, w, out, rows, groups, 1e-5)
    v = (y[:rows].double() * z[:rows].double() * torch.sigmoid(z[:rows].double())).view(rows, groups, -1)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(rows, width) * w.double()
    assert bool(((out[:rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()) and bool((out[rows:] == 9.0).all())
