"""The row kernels that take a row in 16-byte pieces, at the edges of their ranges (one piece, a ragged last warp, two, four and
six pieces a thread, the first size behind them), against 64-bit torch. Sums of a few thousand 32-bit numbers of order 1 in
another order than torch's differ by less than 1e-5 of a row's largest; a bfloat16 result by its last place, 2^-8, of the number
itself."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
TOL = {"float32": 1e-5, "bfloat16": 2.0 ** -8}


def rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float(((a - b).abs() / b.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)).max())


def draw(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,parts", [(4, 1), (132, 3), (2048, 10), (2052, 9), (4096, 5), (8192, 2), (11264, 4), (2046, 2)])
def test_layer_norm_of_partial_sums(dtype, width, parts):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(width)
    res, sums = draw(g, 5, width) + 2.0, draw(g, parts, 5, width)
    w, b = 1 + draw(g, width, scale=0.2), draw(g, width, scale=0.3)
    r, out = res.to(DEV), torch.empty(5, width, dtype=DT[dtype], device=DEV)
    ops.add_layernorm(r, ops.PartialSums(sums.to(DEV).reshape(-1), parts, 5, width), w.to(DEV), b.to(DEV), 1e-5, out)
    x = res.double() + sums.double().sum(0)
    assert rel(r, x) < 1e-6
    d = x - x.mean(-1, keepdim=True)
    want = d / (d.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
    assert rel(out.float(), want) < TOL[dtype]
    some = torch.empty(2, width, dtype=DT[dtype], device=DEV)
    ops.add_layernorm(r, None, w.to(DEV), b.to(DEV), 1e-5, some, torch.tensor([4, 0], dtype=torch.int32, device=DEV))
    assert torch.equal(some, out[[4, 0]])
