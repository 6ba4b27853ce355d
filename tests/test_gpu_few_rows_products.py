"""The products that a step of a few rows takes straight from registers: runs of k, and the experts' grouped form over pairs without
a plan, at the edges of their chunks (32 numbers of k, 4 or 8 chunks a warp and round, 16 outputs, 8 rows, 32 and 256 pairs). Sums
of bfloat16 products in 32-bit: 1e-5 of a row's largest for rows of a few thousand numbers."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def tensor_core():
    from tandemllm_b200.kernels import tensorcore
    from tandemllm_b200.parts.base import Runtime
    return tensorcore.enable(Runtime(torch.device(DEV), torch.bfloat16))


def rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float(((a - b).abs() / b.abs().amax(dim=-1, keepdim=True).clamp_min(1e-30)).max())


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(2048, 4096), (2048, 8192), (40, 2056), (24, 11776), (9472, 2304), (512, 7168)])
def test_long_reductions_in_runs_of_k(M, N, K):
    from tandemllm_b200.kernels import ops
    tc = tensor_core()
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).to(torch.bfloat16), (torch.randn(N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    bias = torch.randn(N, generator=g)
    out = torch.empty(M, N, device=DEV)
    got = tc.linear(x.to(DEV), w.to(DEV), bias.to(DEV), out, defer=True)
    want = x.double() @ w.double().T + bias.double()
    assert rel(ops.materialize(got) if isinstance(got, ops.PartialSums) else out, want) < 1e-5


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("R,k,E", [(1, 4, 32), (5, 6, 64), (8, 4, 5), (8, 32, 64), (7, 5, 1000)])
@pytest.mark.parametrize("N,K", [(16, 32), (40, 264), (136, 1792), (24, 1536), (16, 2048)])
def test_grouped_products_of_pairs_without_a_plan(R, k, E, N, K, gated):
    from tandemllm_b200.kernels import ops, tensorcore
    tensor_core()
    k = min(k, E)
    g = torch.Generator().manual_seed(R * k + N)
    P = R * k
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(R)]).to(torch.int32)
    used = sorted(set(ids.view(-1).tolist()))       # (only the experts that are used get numbers)
    w = torch.zeros(E, (2 if gated else 1) * N, K, dtype=torch.bfloat16)
    for e in used:
        w[e] = (torch.randn(w.shape[1], K, generator=g) * K ** -0.5).to(torch.bfloat16)
    x = torch.randn(R if gated else P, K, generator=g).to(torch.bfloat16)
    out = torch.zeros(P, N, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    xd, wd, idd = x.to(DEV), w.to(DEV), ids.to(DEV)
    tensorcore._check(tensorcore.lib().tl_gemm_skinny_grouped(
        xd.data_ptr(), K, None, k if gated else 1, wd.data_ptr(), K, w.shape[1], out.data_ptr(), N, N, K, int(gated), ops.FP32, None,
        None, None, None, 0, idd.data_ptr(), P, E, status.data_ptr(), None, None, ops.stream()), "grouped")
    want = torch.empty(P, N, dtype=torch.float64)
    for p in range(P):
        y = w[int(ids.view(-1)[p])].double() @ x[p // k if gated else p].double()
        want[p] = torch.nn.functional.silu(y[:N]) * y[N:] if gated else y
    assert int(status.item()) == 0
    assert rel(out, want) < 1e-5


@pytest.mark.parametrize("R,k,E", [(1, 2, 8), (2, 3, 8), (8, 4, 40)])
@pytest.mark.parametrize("N,K", [(1024, 4096), (40, 2056), (24, 2600), (1000, 11776)])
def test_grouped_products_of_long_reductions(R, k, E, N, K):
    """The same with k above 2048, where a few CTAs have eight warps."""
    test_grouped_products_of_pairs_without_a_plan(R, k, E, N, K, False)


@pytest.mark.parametrize("M", [1, 7, 8, 9])
@pytest.mark.parametrize("inter,K", [(2368, 32), (4736, 264), (4760, 2048), (40, 264)])
def test_feed_forward_activations_in_the_products_epilogue(M, inter, K):
    """32-bit sums, activated in 32-bit and rounded once: a last place of bfloat16. Nine rows, other activations and products of
    fewer than two CTAs of 16 outputs an SM go elsewhere."""
    tc = tensor_core()
    gates, plain = (M <= 8 and -(-n // 16) >= 2 * tc.sm_count for n in (inter, 2 * inter))
    g = torch.Generator().manual_seed(M + inter)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * inter, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    z = x.double() @ w.double().T
    out = torch.empty(M, inter, dtype=torch.bfloat16, device=DEV)
    assert tc.gated_few_rows(x.to(DEV), w.to(DEV), out, 1) == gates
    if gates:
        assert rel(out, torch.nn.functional.silu(z[:, :inter]) * z[:, inter:]) < 2.0 ** -8
    got = tc.linear_act(x.to(DEV), w.to(DEV), 3)
    assert (got is not None) == plain
    if plain:
        assert rel(got, z.clamp(min=0) ** 2) < 2.0 ** -8
    assert tc.linear_act(x.to(DEV), w.to(DEV), 8) is None          # tanh: not one of the kernel's


@pytest.mark.parametrize("M", [1, 8, 33, 37, 64, 65, 127, 128])
@pytest.mark.parametrize("N,K", [(5000, 4104), (9480, 2056), (14400, 2056), (18900, 1096), (4096, 2560)])
def test_swapped_products_cut_and_uncut(M, N, K):
    """Fewer tiles than SMs: the ring as deep as it goes where k is not cut, partial sums that a kernel of its own adds where it is,
    or that are left to the consumer; last tiles, k-blocks and blocks of 16 rows that are not full. 32-bit sums of bfloat16 products, plus the rounding of a
    bfloat16 result; rows behind the last one are not written."""
    from tandemllm_b200.kernels import ops
    tc = tensor_core()
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, w = (torch.randn(n, K, generator=g, device=DEV).to(torch.bfloat16) for n in (M, N))
    w = (w.float() * K ** -0.5).to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device=DEV)
    want = x.double() @ w.double().T + bias.double()
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 1e-5 + 2.0 ** -8)):
        for defer in (False, "rounded"):
            whole = torch.full((M + 1, N), 7.0, dtype=dtype, device=DEV)
            got = tc.gemm(x, w, bias, whole[:M], defer=defer)
            assert got is None or defer
            assert rel((whole[:M] if got is None else ops.materialize(got)).float(), want) < tol, (dtype, defer)
            assert bool((whole[M] == 7).all())


@pytest.mark.parametrize("act,name", [(3, "relu2"), (1, "silu")])
@pytest.mark.parametrize("M", [1, 17, 40])
def test_swapped_grouped_products_with_an_activation(act, name, M):
    """An ungated activation in the swapped epilogue (experts without a gate), rows of a group that are not a multiple of 16."""
    from tandemllm_b200.kernels import ops
    tc = tensor_core()
    g = torch.Generator(device=DEV).manual_seed(M)
    E, N, K = 3, 264, 520
    x = torch.randn(2 * M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    ids = torch.tensor([[0]] * M + [[2]] * M, dtype=torch.int32, device=DEV)
    plan = ops.MoePlan(2 * M, E, 64, DEV).build(ids)
    out = torch.empty(2 * M, N, dtype=torch.bfloat16, device=DEV)
    tc.gemm(x, w.view(E * N, K), None, out, rows_per_group=N, plan=plan, swiglu=-act, swap=True, bn=64, n_out=N)
    z = torch.cat([x[:M].double() @ w[0].double().T, x[M:].double() @ w[2].double().T])
    want = z.clamp(min=0) ** 2 if name == "relu2" else torch.nn.functional.silu(z)
    assert rel(out.float(), want) < 1e-5 + 2.0 ** -8
