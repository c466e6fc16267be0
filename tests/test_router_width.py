"""How wide the router's blocks are: a warp an output only while every token has an SM of its own, and the same numbers either way."""
import pytest
import torch

DEV = "cuda:0"


def test_blocks_of_prompts_stay_small():
    from mdma_b200.csrc import build
    warps = build.load("core").mdma_route_warps
    assert [warps(t, 17, 148) for t in (1, 148, 149, 512, 6000)] == [17, 17, 8, 8, 8]
    assert [warps(t, 129, 148) for t in (1, 148, 149, 6000)] == [32, 32, 8, 8]
    assert warps(1, 3, 148) == warps(1, 8, 148) == 8 and warps(78, 64, 78) == 32 and warps(79, 64, 78) == 8


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("outputs,width,shared", [(16, 1024, True), (40, 264, False), (64, 1000, True), (9, 100, True)])
def test_tokens_of_a_prompt_choose_as_alone(outputs, width, shared, dtype):
    """300 tokens take blocks of eight warps, 37 of them alone wide ones: the same bits."""
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(outputs + width)
    draw = lambda *s: torch.randn(*s, device=DEV, generator=g).to(dtype)  # noqa: E731
    h, router, gate, T, top = draw(300, width), draw(outputs, width), draw(width) if shared else None, 300, 4

    def run(rows):
        n = rows.shape[0]
        chosen, weight, scale = torch.full((n, top), -7, dtype=torch.int32, device=DEV), torch.zeros(n, top, device=DEV), torch.zeros(n, device=DEV)
        ops.route(rows, router, None, gate, n, top, 1, 1, chosen, weight, scale)
        return chosen, weight, scale
    many = run(h)
    for lo in (0, 131, T - 37):
        assert all(torch.equal(a, b[lo:lo + 37]) for a, b in zip(run(h[lo:lo + 37].contiguous()), many))
    z = h.double() @ router.double().t()
    best = torch.gather(z, 1, many[0].long())
    assert bool((best >= z.topk(top, 1).values - 1e-4 * z.abs().amax(1, keepdim=True)).all())     # sums of `width` products in float
