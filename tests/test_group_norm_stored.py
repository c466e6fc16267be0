"""The norm in groups on a product that was to be stored: its partial sums are all there is of the rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width,groups", [(36, 3), (64, 1), (2048, 4), (2056, 2), (4096, 4), (4100, 5), (8192, 2), (2048, 32)])
@pytest.mark.parametrize("splits", [0, 1, 4, 9])
def test_stored_rows(width, groups, dtype, splits):
    from mdma_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(width + groups + splits)
    rows = 5
    draw = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    w, x, parts = (1 + 0.3 * draw(width)).to(dtype), draw(rows, width), draw(max(splits, 1), rows + 2, width)
    y = draw(rows, width) if splits == 0 else torch.full((rows, width), float("nan"), device=DEV)        # nobody's with partial sums
    full = (y if splits == 0 else parts[:, :rows].sum(0)).double()
    part = full.view(rows, groups, -1)
    want = x.double() + (part / torch.sqrt((part * part).mean(-1, keepdim=True) + 1e-5)).reshape(rows, width) * w.double()
    if splits:
        ops.group_rmsnorm_add(x, y, w, 1e-5, groups, rows, parts, splits, (rows + 2) * width, True)
    else:
        ops.group_rmsnorm_add(x, y, w, 1e-5, groups, rows)
    assert bool(((x - want).abs() <= 1e-5 * (1 + want.abs())).all())             # sums of up to nine floats, then of a row
    assert bool(((y - full).abs() <= 1e-5 * (1 + full.abs())).all())             # y is left complete
