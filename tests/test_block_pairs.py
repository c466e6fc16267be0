"""The block-pair product at the edges of its token tiles (a gated tile's last columns are finished after its buffer is given
back) and where the K blocks of the last rounds are divided among all pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,N,K,mode", [(1, 512, 64, 2), (15, 300, 128, 2), (16, 256, 128, 2), (17, 256, 128, 2), (33, 256, 192, 2),
                                        (65, 512, 64, 2), (193, 256, 128, 2), (255, 256, 128, 2), (257, 19000, 128, 2), (500, 19100, 192, 2),
                                        (2385, 8192, 128, 2), (1800, 5504, 64, 2), (300, 500, 128, 0),
                                        (512, 9728, 3712, 0), (500, 9700, 3720, 1), (512, 9728, 4096, 2), (300, 9728, 3648, 1)])
def test_edges(M, N, K, mode):
    from mdma_b200 import ops, ops_tensor
    torch.manual_seed(M + N)
    a = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    w, w2 = ((torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16() for _ in range(2))
    x0 = torch.randn(M + 1, N, device=DEV)
    for _ in range(2):                          # a second call finds the scratch and its flags as the first left them
        out = x0.clone() if mode == 1 else torch.full((M + 1, N), 9.0, device=DEV, dtype=torch.bfloat16)
        keep = out[M:].clone()
        ops_tensor.gemm(a, w, out, mode, w2 if mode == 2 else None, M, bn=512, splits=1)
        ops_tensor.check_status(torch.device(DEV))
        assert torch.equal(out[M:], keep)
        ref = a.double() @ w.double().t()
        if mode == 1:                           # sums of K products of order 0.5 / sqrt(K) in float
            assert bool(((out[:M] - x0[:M].double() - ref).abs() <= 1e-5 * (1 + ref.abs())).all())
            continue
        if mode == 2:
            ref = ref / (1 + torch.exp(-ref)) * (a.double() @ w2.double().t())
        assert bool(((out[:M].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5).all())       # one rounding to bfloat16


@pytest.mark.parametrize("heads,N,K", [(1, 128, 64), (3, 40, 128), (5, 130, 64), (2, 300, 192), (4, 64, 320)])
@pytest.mark.parametrize("M", [1, 63, 65, 129, 300])
def test_one_launch_for_all_heads(heads, N, K, M):
    from mdma_b200 import ops_tensor
    torch.manual_seed(M + N)
    x = (torch.randn(M, heads * K + 16, device=DEV) * 0.5).bfloat16()[:, 8:]       # a pitch wider than the heads, an odd start
    w = (torch.randn(heads, N, K, device=DEV) * K ** -0.5).bfloat16()
    out = torch.full((M + 1, heads * N + 3), 9.0, device=DEV, dtype=torch.bfloat16)
    ops_tensor.gemm_heads(x, w, out, M)
    ops_tensor.check_status(torch.device(DEV))
    ref = torch.einsum("mhk,hnk->mhn", x[:, :heads * K].double().reshape(M, heads, K), w.double()).reshape(M, -1)
    assert bool(((out[:M, :heads * N].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all())
    assert bool((out[M:] == 9.0).all()) and bool((out[:, heads * N:] == 9.0).all())


@pytest.mark.parametrize("bn", [512, 128])
def test_gates_far_from_zero(bn):
    """Gates whose exponential nearly overflows, or does, beside inputs of any size: silu(g) is rounded before it meets u, so
    that neither a quotient by more than 2^126 nor a product of g and u beyond the floats shows.  Bound: the result's rounding
    to bfloat16 (2^-9) and the fast exponential's 2 + 1.2 |g| units of a float (2^-16 at 88)."""
    from mdma_b200 import ops, ops_tensor
    dev = torch.device("cuda:0")
    gates, ups = [-88.0, -80.0, -20.0, -1.0, 0.0, 3.0, 88.0, -1e20, -3e38], [1e30, -1e25, 1e-20, 1.0, 1e20]
    M, N, K = 300, 256, 64
    x = torch.zeros(M, K, device=dev, dtype=torch.bfloat16)
    x[:, 0] = 1.0
    w, w2 = (torch.zeros(N, K, device=dev, dtype=torch.bfloat16) for _ in range(2))
    for f in range(N):
        w[f, 0], w2[f, 0] = gates[f % 9], ups[f // 9 % 5]
    out = torch.empty(M, N, device=dev, dtype=torch.bfloat16)
    ops_tensor.gemm(x, w, out, ops.GEMM_SWIGLU, w2, M, bn=bn, splits=1)
    ops_tensor.check_status(dev)
    g, u = w[:, 0].double(), w2[:, 0].double()
    want = g / (1.0 + torch.exp(-g)) * u
    assert torch.isfinite(out).all()
    # (what is below the smallest normal float may come out as 0)
    assert bool(((out.double() - want).abs() <= 2 ** -8 * want.abs() + 2.0 ** -126 * u.abs().clamp(min=1.0)).all())


def _product(M, N, K, mode, bias, act, **forced):
    """(result, reference, bound) of a product as `forced`; partial sums are added up at once."""
    from mdma_b200 import ops, ops_tensor
    torch.manual_seed(M + N + K)
    a = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    w = (torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16()
    b = torch.randn(N, device=DEV).bfloat16() if bias else None
    x0 = torch.randn(M + 1, N, device=DEV)
    out = x0.clone() if mode == 1 else torch.full((M + 1, N), 9.0, device=DEV, dtype=torch.bfloat16)
    keep = out[M:].clone()
    ops_tensor.gemm(a, w, out, mode, None, M, bias=b, store_act=act, act=ops.ACT_GELU_TANH if act else ops.ACT_SILU, **forced)
    ops_tensor.check_status(torch.device(DEV))
    assert torch.equal(out[M:], keep)
    ref = a.double() @ w.double().t() + (b.double() if bias else 0.0)
    if mode == 1:
        return out[:M].double(), ref + x0[:M].double(), 1e-5 * (1 + ref.abs())          # sums of K products of order 0.5 / sqrt(K) in float
    if act:
        ref = torch.nn.functional.gelu(ref, approximate="tanh")
    return out[:M].double(), ref, 2.0 ** -8 * ref.abs() + 2e-5                          # one rounding to bfloat16


@pytest.mark.parametrize("M,N,K,splits", [(129, 256, 256, 2), (130, 300, 1000, 3), (256, 512, 4096, 8), (257, 260, 520, 2), (600, 1000, 1024, 4), (2048, 1024, 512, 2)])
@pytest.mark.parametrize("mode,bias,act", [(1, False, False), (1, True, False), (0, True, True)])
def test_pairs_that_divide_k(M, N, K, splits, mode, bias, act):
    got, want, tol = _product(M, N, K, mode, bias, act, bn=512, splits=splits)
    assert bool(((got - want).abs() <= tol).all())


@pytest.mark.parametrize("M,N,K,plan", [(1, 8192, 2048, (16, -2)), (8, 2752, 1024, (16, -2)), (16, 330, 1032, (16, -2)), (40, 8192, 2048, (64, 1)), (33, 300, 1024, (64, 1)), (64, 2750, 1032, (64, 1))])
def test_gated_products_of_few_tiles(M, N, K, plan):
    from mdma_b200 import ops, ops_tensor
    assert ops_tensor.gemm_plan(2, M, N, K, 148) == plan
    torch.manual_seed(M + N)
    a = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    w, w2 = ((torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16() for _ in range(2))
    ref = a.double() @ w.double().t()
    ref = ref / (1 + torch.exp(-ref)) * (a.double() @ w2.double().t())
    for forced in ({}, dict(bn=512, splits=1)):                  # as planned, and on block pairs (experts' runs of 33-64 rows)
        out = torch.full((M + 1, N), 9.0, device=DEV, dtype=torch.bfloat16)
        ops_tensor.gemm(a, w, out, ops.GEMM_SWIGLU, w2, M, **forced)
        ops_tensor.check_status(torch.device(DEV))
        assert bool((out[M:] == 9.0).all()) and bool(((out[:M].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5).all())


@pytest.mark.parametrize("N,K", [(5632, 2048), (300, 1032)])
def test_gated_runs_of_33_to_64_rows(N, K):
    """Experts side by side, some on block pairs: each gives what it gives alone."""
    from mdma_b200 import ops, ops_tensor
    torch.manual_seed(N)
    first = [0, 40, 43, 43, 107, 140, 152, 217]
    runs = len(first) - 1
    a = (torch.randn(first[-1], K, device=DEV) * 0.5).bfloat16()
    w, w2 = ((torch.randn(runs * N, K, device=DEV) * K ** -0.5).bfloat16() for _ in range(2))
    out = torch.full((first[-1] + 1, N), 9.0, device=DEV, dtype=torch.bfloat16)
    ops_tensor.gemm_runs(a, w, out, first, N, ops.GEMM_SWIGLU, w2)
    ops_tensor.check_status(torch.device(DEV))
    assert bool((out[first[-1]:] == 9.0).all())
    for r in range(runs):
        x = a[first[r]:first[r + 1]].double()
        ref = x @ w[r * N:(r + 1) * N].double().t()
        ref = ref / (1 + torch.exp(-ref)) * (x @ w2[r * N:(r + 1) * N].double().t())
        assert bool(((out[first[r]:first[r + 1]].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-5).all()), r


@pytest.mark.parametrize("M,N,K,plan", [(600, 1000, 1024, (512, 4)), (768, 2048, 8192, (512, 3)), (257, 4096, 14336, (512, 2)), (513, 1024, 520, (512, 2))])
@pytest.mark.parametrize("groups", [1, 4])
@pytest.mark.parametrize("bias", [False, True])
def test_a_norm_adds_up_what_pairs_leave(M, N, K, plan, groups, bias):
    """As planned: the pairs' parts go to the norm behind the product, added to the residual stream or onto a sublayer's result."""
    from mdma_b200 import ops, ops_tensor
    assert ops_tensor.gemm_plan(ops.GEMM_ACCUMULATE, M, N, K, 148, True) == plan
    torch.manual_seed(M + N + groups)
    a = (torch.randn(M, K, device=DEV) * 0.5).bfloat16()
    w = (torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16()
    b = torch.randn(N, device=DEV).bfloat16() if bias else None
    x, y, nw = torch.randn(M, N, device=DEV), torch.randn(M, N, device=DEV), 1 + 0.3 * torch.randn(N, device=DEV)
    want_y = y.double() + a.double() @ w.double().t() + (b.double() if bias else 0.0)
    part = want_y.view(M, groups, -1)
    normed = (part / torch.sqrt((part * part).mean(-1, keepdim=True) + 1e-5)).reshape(M, N) * nw.double()
    ops_tensor.gemm(a, w, y, ops.GEMM_ACCUMULATE, None, M, bias=b, defer=True)
    pend = ops_tensor.take_pending(y, ops.GEMM_ACCUMULATE, M)
    assert pend is not None and pend[1] == plan[1] and pend[2] == M * N
    if groups == 1:
        h = torch.empty(M, N, device=DEV)
        ops.rmsnorm(y, nw, 1e-5, h, None, M, *pend)
        got, want = h.double(), normed
    else:
        want = x.double() + normed
        ops.group_rmsnorm_add(x, y, nw, 1e-5, groups, M, *pend)
        got = x.double()
    ops_tensor.check_status(torch.device(DEV))
    # a part is K / splits products, 16 to an addition whose sum is cut to a float (2 ** -23 of sums below 2); then the parts and the rest
    tol = 1e-5 + K / plan[1] / 16 * 2.0 ** -22
    assert bool(((y.double() - want_y).abs() <= tol * (1 + want_y.abs())).all())
    assert bool(((got - want).abs() <= 4 * tol * (1 + want.abs())).all())               # the same, over the row's deviation and times w
