"""Latent attention of a decode step's few rows over shuffled pages, its keys cut into a few spans or into more than the join takes in
one round (32), both chunks of the latent in one CTA of eight warps, short and long cached rows.

The queries are bfloat16 numbers, so scores are exact up to 32-bit sums; a weight is rounded to bfloat16 (eight
bits: by up to 2^-8 of itself) and so is the result: |error| <= 2 * 2^-8 sum_j p_j |c_j|, and 1e-5 of it for the sums."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def latent_step(H, L, Rr, contexts, rows, window, seed):
    from tandemllm_b200.kernels import tensorcore
    from tandemllm_b200.parts.base import Runtime
    rt = Runtime(torch.device(DEV), torch.bfloat16)
    tc = tensorcore.enable(rt)
    g = torch.Generator().manual_seed(seed)
    B, Dk, page = len(contexts), L + Rr, 16
    per = -(-max(contexts) // page)
    pages = torch.randperm(B * per, generator=g).to(torch.int32).view(B, per)
    cache = torch.randn(B * per, 1, page, Dk, generator=g).to(torch.bfloat16)
    q = (torch.randn(B * rows, H, Dk, generator=g) * 2).to(torch.bfloat16).float()
    pos = [p for c in contexts for p in range(c - rows, c)]
    i32 = dict(dtype=torch.int32, device=DEV)
    step = SimpleNamespace(n_requests=B, max_rows_per_request=rows, max_context=max(contexts), host={},
                           req_of_row=torch.tensor([b for b in range(B) for _ in range(rows)], **i32),
                           row_start=torch.arange(0, B * rows + 1, rows, **i32), positions=torch.tensor(pos, **i32))
    out = torch.full((B * rows, H, L), float("nan"), dtype=torch.bfloat16, device=DEV)
    scale = Dk ** -0.5
    assert tc.attention_latent(q.to(DEV), SimpleNamespace(k=cache.to(DEV), page_size=page), pages.to(DEV), step, scale, window, out, L, rt)
    for r, p in enumerate(pos):
        b = r // rows
        keys = cache[pages[b].long(), 0].reshape(-1, Dk)[max(0, p - window + 1) if window else 0:p + 1].double().to(DEV)
        weights = torch.softmax(scale * q[r].double().to(DEV) @ keys.T, -1)
        want, room = weights @ keys[:, :L], weights @ keys[:, :L].abs()
        assert ((out[r].double() - want).abs() <= (2.0 ** -7 + 1e-5) * room).all(), (r, p)
    assert int(tc.status.item()) == 0


@pytest.mark.parametrize("H,L,Rr", [(32, 512, 64), (20, 264, 8), (4, 64, 16), (3, 300, 2)])
@pytest.mark.parametrize("window", [None, 100, 1500])
@pytest.mark.parametrize("context", [100, 250, 300, 750, 2048, 2049, 4200, 9000])
def test_one_row_over_few_and_many_spans(H, L, Rr, context, window):
    latent_step(H, L, Rr, [context], 1, window, context)


@pytest.mark.parametrize("H,L,Rr,contexts,rows,window", [(32, 512, 64, [2500, 40, 4100], 1, None), (32, 512, 64, [2500, 3000], 2, 1000),
                                                         (16, 256, 32, [5000], 4, None), (20, 264, 8, [700, 2300, 64, 33], 3, 600)])
def test_several_requests_and_rows(H, L, Rr, contexts, rows, window):
    latent_step(H, L, Rr, contexts, rows, window, len(contexts))
