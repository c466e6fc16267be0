"""The two shapes of the CUDA-core products (few rows that stream a matrix, tiles of 32 rows) at the edges of their
tiles, and the experts' products made of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -24


def bound(a, w):
    """Rounding of a float32 dot product: the chains are 16 + K / 64 + 4 additions and as many products long."""
    K = a.shape[1]
    return (16 + K / 64 + 6) * EPS * (a.double().abs() @ w.double().abs().t())


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 31, 32, 33, 70])
@pytest.mark.parametrize("N,K,pitch", [(1, 4, 4), (17, 15, 15), (33, 64, 64), (40, 516, 520), (15, 1024, 1027), (130, 1100, 1100), (9, 2064, 2064), (4100, 132, 140), (4099, 70, 70), (8200, 1028, 1028)])
def test_product_edges_and_one_order_of_additions(M, N, K, pitch):
    from mdma_b200 import ops
    torch.manual_seed(M * N + K)
    a, w = torch.randn(M, pitch, device=DEV)[:, :K], torch.randn(N, K, device=DEV)
    w2 = torch.randn(N, K, device=DEV)
    out = torch.full((M + 1, N), 9.0, device=DEV)
    ops.gemm_simt(a, w, out, m=M)
    ref, tol = a.double() @ w.double().t(), bound(a, w)
    assert bool(((out[:M] - ref).abs() <= tol).all()) and bool((out[M:] == 9.0).all())
    # any row alone, and among 40 others, gives the same bits
    one, many = torch.empty(1, N, device=DEV), torch.empty(41, N, device=DEV)
    ops.gemm_simt(a[M - 1:], w, one)
    ops.gemm_simt(torch.cat([torch.randn(40, K, device=DEV), a[M - 1:]]), w, many)
    assert torch.equal(one[0], out[M - 1]) and torch.equal(many[40], out[M - 1])
    x = torch.randn(M + 1, N, device=DEV)
    x0 = x.clone()
    ops.gemm_simt(a, w, x, ops.GEMM_ACCUMULATE, m=M)
    assert torch.equal(x[:M], x0[:M] + out[:M]) and torch.equal(x[M:], x0[M:])
    gated, up = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm_simt(a, w, gated, ops.GEMM_SWIGLU, w2)
    ops.gemm_simt(a, w2, up)
    z, u = out[:M].double(), up.double()
    want = z / (1 + torch.exp(-z)) * u
    assert bool(((gated - want).abs() <= 1e-6 * (want.abs() + 1)).all())       # the same sums: expf, a division, a product


@pytest.mark.parametrize("tokens,experts,top,width,ff", [(30, 2, 2, 64, 33), (1, 6, 2, 64, 24), (9, 5, 3, 72, 40), (40, 3, 2, 100, 17), (150, 7, 4, 256, 130), (2100, 4, 4, 32, 16)])
@pytest.mark.parametrize("gated", [True, False])
def test_experts_by_expert(tokens, experts, top, width, ff, gated):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(tokens + ff)
    draw = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    h, G, U, D = draw(tokens, width), draw(experts * ff, width) * 0.1, draw(experts * ff, width) * 0.1, draw(experts * width, ff) * 0.1
    # one token's choices need not differ, one is an output without matrices
    chosen = torch.randint(0, experts + 1, (tokens, top), device=DEV, generator=g, dtype=torch.int32)
    weight = torch.rand(tokens, top, device=DEV, generator=g)
    n = tokens * top
    scratch = (torch.zeros(2 * (experts + 1), dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV),
               torch.zeros(n, width, device=DEV))
    x = draw(tokens, width)
    want = x.double()
    act = torch.zeros(n, ff, device=DEV)
    ops.experts(h, G, U if gated else None, D, chosen, weight, tokens, experts, top, ff, act, x, scratch)
    hd = h.double()
    for e in range(experts + 1):
        share = (weight.double() * (chosen == e)).sum(1, keepdim=True)
        if e == experts:
            want = want + share * hd
            continue
        z = hd @ G.double()[e * ff:(e + 1) * ff].t()
        z = z / (1 + torch.exp(-z)) * (hd @ U.double()[e * ff:(e + 1) * ff].t() if gated else 1.0)
        want = want + share * (z @ D.double()[e * width:(e + 1) * width].t())
    # two products of up to 256 and 130 terms of order one
    assert bool(((x - want).abs() <= 2e-5 * (1 + want.abs())).all())


@pytest.mark.parametrize("batch", [0, 4])
def test_a_matrix_that_the_kernel_before_writes(batch):
    """The matrix is read after its writer has ended, unless the caller says that nothing writes it (`w_fixed`)."""
    from mdma_b200 import ops
    N, K, M = 4096, 1024, 4
    sources = [torch.randn(N, K, device=DEV) for _ in range(2)]
    w = torch.zeros(N, K, device=DEV, dtype=torch.bfloat16)
    a = torch.randn(M, max(batch, 1) * K, device=DEV).bfloat16()

    def product(out, **more):
        if batch:
            ops.gemm_simt_batched(a, w.view(batch, N // batch, K), out, M, **more)
        else:
            ops.gemm_simt(a, w, out, **more)
    want = [torch.empty(M, N, device=DEV) for _ in range(2)]
    for source, out in zip(sources, want):
        w.copy_(source)
        torch.cuda.synchronize()
        product(out, w_fixed=True)
        torch.cuda.synchronize()
    outs = [torch.empty(M, N, device=DEV) for _ in range(20)]
    for i, out in enumerate(outs):
        ops.copy_rows(sources[i % 2], w, N)
        product(out)
    assert not torch.equal(*want)
    assert all(torch.equal(out, want[i % 2]) for i, out in enumerate(outs))


@pytest.mark.parametrize("M", [1, 3, 4, 5, 8])
@pytest.mark.parametrize("N,K", [(4736, 1024), (4739, 1000), (9472, 512), (9473, 20), (11000, 516), (13500, 516), (333700, 20)])
def test_matrices_larger_than_the_blocks_hold(M, N, K):
    """Blocks that walk over groups of features: the bits of a row among 40 others, which takes the tiles."""
    from mdma_b200 import ops
    torch.manual_seed(M + N + K)
    a, w, w2 = (torch.randn(n, K, device=DEV) for n in (M, N, N))
    out = torch.full((M + 1, N), 9.0, device=DEV)
    ops.gemm_simt(a, w, out, m=M, w_fixed=True)
    assert bool(((out[:M] - a.double() @ w.double().t()).abs() <= bound(a, w)).all()) and bool((out[M:] == 9.0).all())
    rows = torch.cat([a, torch.randn(40, K, device=DEV)])
    many = torch.empty(M + 40, N, device=DEV)
    ops.gemm_simt(rows, w, many)
    assert torch.equal(many[:M], out[:M])
    x = torch.randn(M, N, device=DEV)
    x0 = x.clone()
    ops.gemm_simt(a, w, x, ops.GEMM_ACCUMULATE)
    assert torch.equal(x, x0 + out[:M])
    gated, many = torch.empty(M, N, device=DEV), torch.empty(M + 40, N, device=DEV)
    ops.gemm_simt(a, w, gated, ops.GEMM_SWIGLU, w2)
    ops.gemm_simt(rows, w, many, ops.GEMM_SWIGLU, w2)
    assert torch.equal(many[:M], gated)


@pytest.mark.parametrize("M", [1, 4, 5, 8])
@pytest.mark.parametrize("gated", [False, True])
def test_streamed_products_in_a_replayed_chain(M, gated):
    """Kernels of this library write the rows that a streamed product reads, and read what it writes, several times over in one
    graph: each replay gives the bits of the tiles on its own inputs."""
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    N, K, rounds = 9473, 1024, 3
    draw = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    first, back = draw(K, K) * K ** -0.5, draw(K, N) * N ** -0.5
    ws = [(draw(N, K) * K ** -0.5, draw(N, K)) for _ in range(rounds)]
    rows, a, b = draw(M, K), torch.zeros(M, K, device=DEV), torch.zeros(M, K, device=DEV)
    outs = [torch.zeros(M, N, device=DEV) for _ in range(rounds)]

    def product(x, w, out):
        ops.gemm_simt(x, w[0], out, ops.GEMM_SWIGLU if gated else ops.GEMM_STORE, w[1] if gated else None, w_fixed=True)

    def chain():
        ops.gemm_simt(rows, first, a, w_fixed=True)
        for i in range(rounds):
            product(a, ws[i], outs[i])
            ops.gemm_simt(outs[i], back, b, w_fixed=True)
            ops.gemm_simt(b, first, a, w_fixed=True)
    chain()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    many = torch.empty(M + 40, N, device=DEV)
    for _ in range(4):
        rows.copy_(draw(M, K))
        for _ in range(3):
            graph.replay()
        x = torch.zeros(M + 40, K, device=DEV)
        ops.gemm_simt(torch.cat([rows, draw(40, K)]), first, x)
        for i in range(rounds):
            product(x, ws[i], many)
            assert torch.equal(many[:M], outs[i])
            y = torch.empty(M + 40, K, device=DEV)
            ops.gemm_simt(many, back, y)
            ops.gemm_simt(y, first, x)
