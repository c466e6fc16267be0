"""Prompts through the recurrences that are linear in their state, chunks of 64 rows side by side: against a float64 walk
row by row, at the edges of chunks, columns and quads, and against the walk row by row of the library."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


def _near(got, want, tol):
    """`tol` of each row's largest number: every output is a sum of products of order one, in float32."""
    scale = want.abs().amax(-1, keepdim=True) + 1.0
    assert torch.isfinite(got).all()
    assert bool(((got.to(F64) - want).abs() <= tol * scale).all()), float(((got.to(F64) - want).abs() / scale).max())


def _state_walk(q, k, u, decay, S):
    """S = decay_t S + k_t u_t', o_t = S' q_t; decay [T, H]; returns (o, S)."""
    out = torch.empty(u.shape, dtype=F64, device=DEV)
    for t in range(len(q)):
        S = decay[t][:, None, None] * S + k[t][:, :, None] * u[t][:, None, :]
        out[t] = torch.matmul(q[t][:, None, :], S)[:, 0]
    return out, S


LENGTHS = [(1,), (64,), (65, 3, 0, 130), (200,), (63, 128)]


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 64), (30, 70), (7, 5), (100, 130)])
@pytest.mark.parametrize("dtype,half,interleaved", [(torch.bfloat16, 0, False), (torch.float32, 3, False), (torch.bfloat16, 2, True)])
def test_linear_attention(lengths, dim, vdim, dtype, half, interleaved):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(dim * 7 + vdim + sum(lengths))
    H, T, n = 3, sum(lengths), len(lengths)
    q_col, k_col, v_col = 0, H * dim, 2 * H * dim
    width = -(-(2 * H * dim + H * vdim) // 8) * 8 + (8 if half == 0 else 3)       # a pitch that is and one that is no multiple of four
    proj = torch.randn(T + 1, width, device=DEV, generator=g).to(dtype)
    decay = torch.tensor([0.99, 0.9, 0.2], device=DEV)
    start = torch.tensor([sum(lengths[:i]) for i in range(n + 1)], dtype=torch.int32, device=DEV)
    slot = torch.arange(n, dtype=torch.int32, device=DEV).flip(0).contiguous()
    pos = torch.cat([torch.arange(x) + 5 for x in lengths]).to(DEV, torch.int32) if T else torch.zeros(1, dtype=torch.int32, device=DEV)
    freq = torch.rand(max(half, 1), device=DEV, generator=g)
    state = torch.randn(n, H * dim * vdim + 3, device=DEV, generator=g)
    first = state.clone()
    most = -(-max(lengths) // 64)
    scratch = torch.full((n * most * H * dim * vdim,), float("nan"), device=DEV)
    out = torch.full((T + 1, H * vdim), 9.0, device=DEV)
    assert ops.chunk_scan_rows(dim, vdim) == 64
    kw = dict(silu=half == 0, k_scale=0.3, inv_freq=freq if half else None, rotary_dim=2 * half, interleaved=interleaved, tok_pos=pos)
    ops.linear_attention(proj, q_col, k_col, v_col, decay, start, slot, state, out, n, H, dim, vdim, True, 64, most, scratch, **kw)
    walked, by_row = first.clone(), torch.empty_like(out)
    ops.linear_attention(proj, q_col, k_col, v_col, decay, start, slot, walked, by_row, n, H, dim, vdim, **kw)
    act = (lambda z: z * torch.sigmoid(z)) if half == 0 else (lambda z: z)

    def turn(x, t):
        if not half:
            return x
        a = pos[t, None, None].to(F64) * freq.to(F64)[:half]
        one, two = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
        y = x.clone()
        y[..., one], y[..., two] = x[..., one] * a.cos() - x[..., two] * a.sin(), x[..., two] * a.cos() + x[..., one] * a.sin()
        return y
    for s, length in enumerate(lengths):
        t = torch.arange(int(start[s]), int(start[s]) + length, device=DEV)
        rows = act(proj[t].to(F64))
        q, k = (turn(rows[:, c:c + H * dim].reshape(length, H, dim), t) for c in (q_col, k_col))
        v = rows[:, v_col:v_col + H * vdim].reshape(length, H, vdim)
        S = first[slot[s], :H * dim * vdim].to(F64).view(H, dim, vdim)
        want, S = _state_walk(q, k * 0.3, v, decay.to(F64).expand(length, H), S)
        _near(out[t], want.flatten(1), 2e-5)
        _near(state[slot[s], :H * dim * vdim], S.reshape(-1), 2e-5)
        _near(out[t], by_row[t].to(F64), 2e-5)
    assert bool((out[T:] == 9.0).all()) and torch.equal(state[:, H * dim * vdim:], first[:, H * dim * vdim:])


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("heads,groups,vdim,N", [(4, 1, 64, 128), (6, 2, 32, 64), (3, 1, 70, 30), (8, 1, 5, 7), (64, 1, 64, 128)])
def test_mamba2(lengths, heads, groups, vdim, N):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N * 7 + vdim + sum(lengths))
    draw = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    T, n, inner = sum(lengths), len(lengths), heads * vdim
    conv, proj = draw(T + 1, inner + 2 * groups * N), draw(T + 1, heads + 5)
    dt_bias, a_log, D = draw(heads).to(torch.bfloat16), draw(heads).to(torch.bfloat16), draw(heads).to(torch.bfloat16)
    start = torch.tensor([sum(lengths[:i]) for i in range(n + 1)], dtype=torch.int32, device=DEV)
    slot = torch.arange(n, dtype=torch.int32, device=DEV).flip(0).contiguous()
    floats = heads * N * vdim
    state = draw(n, floats + 4)
    first = state.clone()
    most = -(-max(lengths) // 64)
    scratch = torch.full((n * most * (floats + heads),), float("nan"), device=DEV)
    y = torch.full((T + 1, inner), 9.0, device=DEV)
    assert ops.chunk_scan_rows(N, vdim) == 64
    ops.mamba2_scan(conv, proj, 2, dt_bias, a_log, D, start, slot, state, y, n, heads, vdim, N, groups, 64, most, scratch)
    walked, by_row = first.clone(), torch.empty_like(y)
    ops.mamba2_scan(conv, proj, 2, dt_bias, a_log, D, start, slot, walked, by_row, n, heads, vdim, N, groups)
    for s, length in enumerate(lengths):
        rows = conv[start[s]:start[s] + length].to(F64)
        x = rows[:, :inner].reshape(length, heads, vdim)
        B, C = (rows[:, inner + j * groups * N:inner + (j + 1) * groups * N].reshape(length, groups, N).repeat_interleave(heads // groups, 1)
                for j in (0, 1))
        dt = torch.nn.functional.softplus(proj[start[s]:start[s] + length, 2:2 + heads].to(F64) + dt_bias.to(F64), threshold=1e9)
        S = first[slot[s], :floats].to(F64).view(heads, vdim, N).transpose(1, 2)
        want, S = _state_walk(C, B * dt[:, :, None], x, torch.exp(-torch.exp(a_log.to(F64)) * dt), S)
        want = want + D.to(F64)[:, None] * x
        _near(y[start[s]:start[s] + length], want.flatten(1), 2e-5)
        _near(state[slot[s], :floats], S.transpose(1, 2).reshape(-1), 2e-5)
        _near(y[start[s]:start[s] + length], by_row[start[s]:start[s] + length].to(F64), 2e-5)
    assert bool((y[T:] == 9.0).all()) and torch.equal(state[:, floats:], first[:, floats:])


def test_heads_beyond_the_kernels():
    from mdma_b200 import ops
    assert ops.chunk_scan_rows(129, 64) == 0 and ops.chunk_scan_rows(256, 64) == 0 and ops.chunk_scan_rows(128, 300) == 64


@pytest.mark.parametrize("chunk_rows", [0, 64])
@pytest.mark.parametrize("odd", ["dt_bias", "a_log", "d", "strided"])
def test_small_vectors_of_several_dtypes_are_refused_before_any_launch(chunk_rows, odd):
    from mdma_b200 import ops
    heads, vdim, N, T = 4, 8, 8, 70
    vectors = {name: torch.zeros(heads, device=DEV, dtype=torch.bfloat16) for name in ("dt_bias", "a_log", "d")}
    if odd == "strided":
        vectors["a_log"] = torch.zeros(2 * heads, device=DEV, dtype=torch.bfloat16)[::2]
    else:
        vectors[odd] = vectors[odd].float()
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    conv, proj = torch.zeros(T, heads * vdim + 2 * N, device=DEV), torch.zeros(T, heads, device=DEV)
    y = torch.full((T, heads * vdim), 9.0, device=DEV)
    before = ops.LAUNCHES
    with pytest.raises(AssertionError, match="one dtype"):
        ops.mamba2_scan(conv, proj, 0, vectors["dt_bias"], vectors["a_log"], vectors["d"], i32(0, T), i32(0), torch.zeros(1, heads * N * vdim, device=DEV),
                        y, 1, heads, vdim, N, 1, chunk_rows, 2, torch.zeros(2 * (heads * N * vdim + heads), device=DEV))
    assert ops.LAUNCHES == before and bool((y == 9.0).all())


@pytest.mark.parametrize("at", [0, 1, 2, 5, 8, 12, 35, 63, 64, 77, 127])
@pytest.mark.parametrize("where", ["k", "v"])
def test_a_row_that_is_not_finite_leaves_the_rows_before_it_alone_linear_attention(at, where):
    from mdma_b200 import ops
    H, dim, vdim, T = 2, 32, 70, 130
    g = torch.Generator(device=DEV).manual_seed(at)
    proj = torch.randn(T, 2 * H * dim + H * vdim, device=DEV, generator=g)
    start, slot = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([0, T], [0]))
    decay = torch.tensor([0.99, 0.2], device=DEV)
    outs = []
    for bad in (None, float("inf"), float("nan")):
        rows = proj.clone()
        if bad is not None:
            rows[at, H * dim + 3 if where == "k" else 2 * H * dim + 5] = bad
        out = torch.empty(T, H * vdim, device=DEV)
        ops.linear_attention(rows, 0, H * dim, 2 * H * dim, decay, start, slot, torch.zeros(1, H * dim * vdim, device=DEV), out, 1, H, dim,
                             vdim, True, 64, 3, torch.empty(3 * H * dim * vdim, device=DEV), silu=False)
        outs.append(out)
    assert torch.isfinite(outs[0]).all()
    for out in outs[1:]:
        assert torch.equal(out[:at], outs[0][:at]) and not torch.isfinite(out[at]).all()


@pytest.mark.parametrize("at", [0, 1, 2, 5, 8, 12, 35, 63, 64, 77, 127])
@pytest.mark.parametrize("where", ["x", "B", "dt"])
def test_a_row_that_is_not_finite_leaves_the_rows_before_it_alone_mamba2(at, where):
    from mdma_b200 import ops
    heads, vdim, N, T = 2, 70, 32, 130
    g = torch.Generator(device=DEV).manual_seed(at)
    conv, proj = torch.randn(T, heads * vdim + 2 * N, device=DEV, generator=g), torch.randn(T, heads, device=DEV, generator=g)
    start, slot = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([0, T], [0]))
    zeros = torch.zeros(heads, device=DEV)
    outs = []
    for bad in (None, float("inf"), float("nan")):
        c, p = conv.clone(), proj.clone()
        if bad is not None and where == "dt":
            p[at, 0] = bad
        elif bad is not None:
            c[at, 5 if where == "x" else heads * vdim + 3] = bad
        y = torch.empty(T, heads * vdim, device=DEV)
        ops.mamba2_scan(c, p, 0, zeros, zeros, zeros, start, slot, torch.zeros(1, heads * N * vdim, device=DEV), y, 1, heads, vdim, N, 1, 64, 3,
                        torch.empty(3 * (heads * N * vdim + heads), device=DEV))
        outs.append(y)
    assert torch.isfinite(outs[0]).all()
    for y in outs[1:]:
        assert torch.equal(y[:at], outs[0][:at]) and not torch.isfinite(y[at]).all()
