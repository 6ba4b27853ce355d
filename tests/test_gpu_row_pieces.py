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


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,top,parts", [(4, 1, 1), (132, 5, 3), (2048, 6, 10), (2052, 4, 2), (4096, 9, 1), (8192, 2, 3), (8196, 3, 2),
                                             (2050, 3, 2)])
def test_norm_behind_a_branch_with_a_gate_that_is_not_computed_yet(dtype, width, top, parts):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(width + top)
    R = 3
    res, sums = draw(g, R, width), draw(g, parts, R, width)
    w, w2 = 1 + draw(g, width, scale=0.2), 1 + draw(g, width, scale=0.2)
    x, wg = draw(g, R, width, dtype=DT[dtype]), draw(g, 1, width, scale=2.0 / width ** 0.5, dtype=DT[dtype])
    rows = draw(g, 2, R * top, width)
    ids = torch.stack([torch.randperm(40, generator=g)[:top] for _ in range(R)]).to(torch.int32)
    wts, pos = torch.rand(R, top, generator=g), torch.randperm(R * top, generator=g).to(torch.int32)
    experts = ops.ExpertRows(rows.to(DEV), pos.to(DEV), ids.to(DEV), wts.to(DEV), parts=2)
    gate = torch.sigmoid((x.double() * wg.double()).sum(-1, keepdim=True))
    d = sums.double().sum(0) * gate
    for r in range(R):
        for j in range(top):
            d[r] += wts[r, j].double() * rows[:, pos[r * top + j]].double().sum(0)
    new = res.double() + w.double() * d / (d.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()
    r1, out = res.to(DEV), torch.empty(R, width, dtype=DT[dtype], device=DEV)
    ops.add_normed(r1, ops.PartialSums(sums.to(DEV).reshape(-1), parts, R, width), w.to(DEV), 1e-5, ops.RowDot(x.to(DEV), wg.to(DEV)),
                   experts, (w2.to(DEV), 1e-4, out, None))
    assert rel(r1, new) < 1e-5
    assert rel(out.float(), w2.double() * new / (new.pow(2).mean(-1, keepdim=True) + 1e-4).sqrt()) < TOL[dtype]


@pytest.mark.parametrize("width,top", [(50, 1), (2050, 6), (4094, 3), (4098, 2), (131, 0)])
def test_norm_behind_a_branch_at_widths_four_does_not_divide(width, top):
    """A number a load: the form of a step of few rows (up to two a SM, rows of up to 4096 numbers) and the other give a row the same
    bits, and those of the formula."""
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(width)
    R = 400
    res, dense = draw(g, R, width), draw(g, R, width)
    w, w2 = 1 + draw(g, width, scale=0.2), 1 + draw(g, width, scale=0.2)
    experts, d = None, dense.double()
    if top:
        rows = draw(g, R * top, width)
        ids = torch.stack([torch.randperm(40, generator=g)[:top] for _ in range(R)]).to(torch.int32)
        wts, pos = torch.rand(R, top, generator=g), torch.arange(R * top, dtype=torch.int32)
        d = d + (wts.double()[..., None] * rows.double().view(R, top, width)).sum(1)
        experts = lambda n: ops.ExpertRows(rows[:n * top].to(DEV), pos[:n * top].to(DEV), ids[:n].to(DEV), wts[:n].to(DEV))
    new = res.double() + w.double() * d / (d.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()
    made = []
    for n in (R, 3):
        r, out = res[:n].to(DEV), torch.empty(n, width, device=DEV)
        ops.add_normed(r, dense[:n].to(DEV), w.to(DEV), 1e-5, None, experts(n) if top else None, (w2.to(DEV), 1e-4, out, None))
        assert rel(r, new[:n]) < 1e-5
        assert rel(out, w2.double() * new[:n] / (new[:n].pow(2).mean(-1, keepdim=True) + 1e-4).sqrt()) < 1e-5
        made.append((r[:3], out[:3]))
    assert torch.equal(made[0][0], made[1][0]) and torch.equal(made[0][1], made[1][1])


@pytest.mark.parametrize("Hq,Hk,D,VD,rot,turn_values", [(4, 2, 16, 8, 16, False), (3, 1, 64, 64, 32, True), (16, 4, 128, 128, 128, False),
                                                        (40, 8, 128, 64, 64, True), (2, 2, 24, 16, 0, False), (4, 2, 16, 8, 8, False)])
def test_turned_heads_and_their_pages(Hq, Hk, D, VD, rot, turn_values):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(D + rot)
    R, page, pad = 5, 16, 8
    q_col, k_col = pad, pad + Hq * D
    v_col = k_col + Hk * D
    qkv = draw(g, R, v_col + Hk * VD, dtype=torch.bfloat16)
    pos, req = torch.tensor([3, 1000, 17, 250, 31]), torch.tensor([0, 1, 0, 1, 0])
    table = torch.stack([torch.randperm(64, generator=g), 64 + torch.randperm(64, generator=g)]).to(torch.int32)
    inv, inv_v = torch.rand(max(rot // 2, 1), generator=g), torch.rand(VD // 2, generator=g)
    q_out = torch.empty(R, Hq, D, dtype=torch.bfloat16, device=DEV)
    kc = torch.zeros(128, Hk, page, D, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros(128, Hk, page, VD, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    ops.qkv_rotate_store(qkv.to(DEV), q_col, k_col, v_col, inv.to(DEV) if rot else None, rot, inv_v.to(DEV) if turn_values else None,
                         pos.to(**i32), req.to(**i32), table.to(DEV), page, q_out, kc, vc, Hq, Hk, D, VD, status, rot_magnitude=0.75)
    assert int(status.item()) == 0

    def turned(x, freq, n, magnitude):              # x [R, heads, size]; angles in 32-bit as the kernel's are
        angle = (pos.float()[:, None] * freq[None, :n // 2]).double()[:, None]
        c, s = angle.cos() * magnitude, angle.sin() * magnitude
        a, b = x[..., :n // 2], x[..., n // 2:n]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., n:]], -1)

    q, k, v = (qkv[:, at:at + h * d].double().view(R, h, d) for at, h, d in ((q_col, Hq, D), (k_col, Hk, D), (v_col, Hk, VD)))
    assert rel(q_out.float(), turned(q, inv, rot, 0.75)) < TOL["bfloat16"]
    where = [(int(table[req[r], pos[r] // page]), int(pos[r] % page)) for r in range(R)]
    assert rel(torch.stack([kc[p, :, o] for p, o in where]).float(), turned(k, inv, rot, 0.75)) < TOL["bfloat16"]
    assert rel(torch.stack([vc[p, :, o] for p, o in where]).float(), turned(v, inv_v, VD, 1.0) if turn_values else v) < TOL["bfloat16"]
    assert int((kc != 0).any(-1).sum()) == R * Hk


@pytest.mark.parametrize("halves", [False, True])
@pytest.mark.parametrize("H,D,L,Rr,dims", [(1, 8, 8, 16, 16), (32, 128, 512, 64, 64), (20, 16, 520, 32, 16), (3, 0, 2048, 8, 0),
                                           (4, 16, 64, 0, 0), (2, 8, 24, 12, 8)])
def test_latent_rows_and_turned_queries(H, D, L, Rr, dims, halves):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(L + Rr)
    R, page, at, Dk = 3, 16, 16, L + Rr
    q, down = draw(g, R, H * (D + Rr), dtype=torch.bfloat16), draw(g, R, at + Dk, dtype=torch.bfloat16)
    w, inv = 1 + draw(g, L, scale=0.2), torch.rand(max(dims // 2, 1), generator=g)
    pos = torch.tensor([5, 130, 77])
    table = torch.randperm(16, generator=g).to(torch.int32)[None]
    cache = torch.zeros(16, 1, page, Dk, dtype=torch.bfloat16, device=DEV)
    qa = torch.zeros(R, H, Dk, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.latent_prepare(q.to(DEV), down.to(DEV)[:, at:], w.to(DEV), 1e-5, inv.to(DEV), dims, pos.to(DEV, torch.int32),
                       torch.zeros(R, dtype=torch.int32, device=DEV), table.to(DEV), page, cache, qa, H, D, L, Rr, status, halves)
    assert int(status.item()) == 0

    def turned(x):                                  # x [R, heads, Rr]
        n = dims // 2
        angle = (pos.float()[:, None] * inv[None, :n]).double()[:, None]
        c, s = angle.cos(), angle.sin()
        a, b = (x[..., :n], x[..., n:dims]) if halves else (x[..., 0:dims:2], x[..., 1:dims:2])
        y = x.clone()
        if halves:
            y[..., :n], y[..., n:dims] = a * c - b * s, b * c + a * s
        else:
            y[..., 0:dims:2], y[..., 1:dims:2] = a * c - b * s, b * c + a * s
        return y

    kv = down[:, at:].double()
    c = kv[:, :L] / (kv[:, :L].pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()
    got = torch.stack([cache[int(table[0, p // page]), 0, p % page] for p in pos.tolist()]).float()
    assert rel(got[:, :L], c) < TOL["bfloat16"]
    if Rr:
        assert rel(got[:, L:], turned(kv[:, None, L:])[:, 0]) < TOL["bfloat16"]
        want = turned(q.double().view(R, H, D + Rr)[..., D:])
        # (a turned number is a difference of two products and may be small beside them: held to the head's largest)
        assert rel(qa[..., L:], want) < 1e-5
    assert not qa[..., :L].any()


@pytest.mark.parametrize("n", [8, 264, 1024, 2048, 2056, 8192, 8200, 1028])
def test_norm_of_the_first_columns(n):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(n)
    x, w = draw(g, 3, n + 8 - n % 8, dtype=torch.bfloat16), 1 + draw(g, n, scale=0.2)
    out = torch.empty(3, n, dtype=torch.bfloat16, device=DEV)
    ops.rmsnorm_rows(x.to(DEV), n, w.to(DEV), 1e-5, out)
    v = x[:, :n].double()
    assert rel(out.float(), v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double()) < TOL["bfloat16"]


@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K,gate", [(16, 32, None), (24, 160, "entries"), (512, 128, None), (128, 512, "heads"), (40, 384, None), (10, 48, None)])
def test_a_product_a_head_for_a_few_rows(rows, N, K, gate):
    """32-bit sums of K products of bfloat16 numbers: 1e-5 of the row's largest in a 32-bit result, plus a last place in a bfloat16 one."""
    from tandemllm_b200.kernels import tensorcore
    from tandemllm_b200.parts.base import Runtime
    tc = tensorcore.enable(Runtime(torch.device(DEV), torch.bfloat16))
    g = torch.Generator().manual_seed(N + K + rows)
    H, pad = 3, 8
    a, w = draw(g, rows, H, K + pad, dtype=torch.bfloat16), draw(g, H, N, K, scale=K ** -0.5, dtype=torch.bfloat16)
    logits = {None: None, "entries": draw(g, rows, H * N, dtype=torch.bfloat16), "heads": draw(g, rows, H, dtype=torch.bfloat16)}[gate]
    want = torch.einsum("rhk,hnk->rhn", a[..., :K].double(), w.double())
    if gate:
        want = want * torch.sigmoid(logits.double().view(rows, H, -1))
    for dtype in ("float32", "bfloat16"):
        out = torch.zeros(rows, H, N + 4, dtype=DT[dtype], device=DEV)
        assert tc.head_linear(a.to(DEV), H * (K + pad), K + pad, w.to(DEV), out, H * (N + 4), N + 4, rows,
                              logits.to(DEV) if gate else None, gate == "heads")
        assert rel(out[..., :N].float(), want) < TOL[dtype] + 1e-5
        assert not out[..., N:].any()


@pytest.mark.parametrize("dtype,gate_dtype", [("float32", "float32"), ("bfloat16", "float32"), ("bfloat16", "bfloat16")])
@pytest.mark.parametrize("group,parts", [(260, 3), (2048, 1), (2052, 2), (4096, 1), (4100, 1), (258, 1)])
def test_norm_of_parts_times_a_gate(group, parts, dtype, gate_dtype):
    from tandemllm_b200.kernels import ops
    g = torch.Generator().manual_seed(group)
    width = group * parts
    y, w = draw(g, 3, width), 1 + draw(g, width, scale=0.2)
    gate = draw(g, 3, width + 4, dtype=DT[gate_dtype])
    for silu, weight in ((False, w), (True, None)):
        out = torch.zeros(3, width + 4, dtype=DT[dtype], device=DEV)
        ops.group_norm_gate(y.to(DEV), gate.to(DEV), width + 4, None if weight is None else weight.to(DEV), 1e-5, parts, 0.75,
                            out[:, :width], "silu" if silu else "sigmoid")
        v, z = y.double().view(3, parts, group), gate[:, :width].double()
        want = (v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).view(3, width) * (1 if weight is None else weight.double())
        want = want * (z if silu else 1) * torch.sigmoid(z) * 0.75
        assert rel(out[:, :width].float(), want) < TOL[dtype]
        assert not out[:, width:].any()


@pytest.mark.parametrize("width", [4, 1536, 2048, 2052, 2560, 4100, 8192])
def test_norm_behind_a_branch_of_many_rows(width):
    """More rows than the form for few keeps on the GPU, one dense source and none of the rest: an instantiation of its own, the same bits a row."""
    from tandemllm_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(width)
    R = 2500 if width > 512 else 160000
    res, dense = torch.randn(R, width, generator=g, device=DEV), torch.randn(R, width, generator=g, device=DEV)
    w, w2 = (1 + 0.2 * torch.randn(width, generator=g, device=DEV) for _ in range(2))
    logits = torch.randn(R, generator=g, device=DEV)
    for gate in (None, logits):
        d = dense.double() * (1 if gate is None else torch.sigmoid(gate.double())[:, None])
        new = res.double() + w.double() * d / (d.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()
        made = []
        for n in (R, 5):
            r, out = res[:n].clone(), torch.empty(n, width, dtype=torch.bfloat16, device=DEV)
            ops.add_normed(r, dense[:n].contiguous(), w, 1e-5, None if gate is None else gate[:n].contiguous(), None, (w2, 1e-4, out, None))
            made.append((r[:5], out[:5]))
            assert rel(r, new[:n]) < 1e-5
            assert rel(out.float(), w2.double() * new[:n] / (new[:n].pow(2).mean(-1, keepdim=True) + 1e-4).sqrt()) < TOL["bfloat16"]
        assert all(torch.equal(a, b) for a, b in zip(*made))


@pytest.mark.parametrize("width", [4, 1536, 2052, 2560, 8192, 11264])
def test_layer_norm_of_many_rows(width):
    """The same for the layer norm, with one source and with none."""
    from tandemllm_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(width)
    R = 2500 if width > 512 else 160000
    res, dense = torch.randn(R, width, generator=g, device=DEV) + 2, torch.randn(R, width, generator=g, device=DEV)
    w, b = (torch.randn(width, generator=g, device=DEV) for _ in range(2))
    for delta in (dense, None):
        x = res.double() + (0 if delta is None else delta.double())
        d = x - x.mean(-1, keepdim=True)
        want = d / (d.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() + b.double()
        made = []
        for n in (R, 5):
            r, out = res[:n].clone(), torch.empty(n, width, dtype=torch.bfloat16, device=DEV)
            ops.add_layernorm(r, None if delta is None else delta[:n].contiguous(), w, b, 1e-5, out)
            made.append((r[:5], out[:5]))
            assert rel(r, x[:n]) < 1e-6
            assert rel(out.float(), want[:n]) < TOL["bfloat16"]
        assert all(torch.equal(a, b) for a, b in zip(*made))
