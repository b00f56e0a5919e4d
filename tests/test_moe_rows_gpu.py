"""ops.moe_experts on both sides of the line between the weight-streaming and the tcgen05 grouped kernels (ops._moe_big_rows), with experts of
few and of no rows: plain fp32 experts, and the other kernels' answer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts,top,hidden,inter,rows", [(64, 4, 1024, 1024, 15), (64, 4, 1024, 1024, 16), (64, 4, 768, 384, 23), (64, 4, 768, 384, 24),
                                                           (8, 2, 256, 256, 31), (8, 2, 256, 256, 32)])
@pytest.mark.parametrize("skewed", [False, True])
def test_both_sides_of_the_line(experts, top, hidden, inter, rows, skewed, monkeypatch):
    from nanovllm import ops
    assert ops._moe_big_rows(experts, hidden * inter) in (rows, rows + 1)
    T = rows * experts // top
    g = torch.Generator(device="cuda").manual_seed(rows)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, logits = rand(T, hidden).bfloat16(), rand(T, experts)
    if skewed:                                                 # a few experts take nearly all rows, many none
        logits[:, :top + 1] += 8
    w13, w2 = (rand(experts, 2 * inter, hidden) * hidden ** -0.5).bfloat16(), (rand(experts, hidden, inter) * inter ** -0.5).bfloat16()
    ids, weights = ops.moe_route(logits.bfloat16(), top)
    plan = ops.moe_align(ids, 0, experts)
    assert ops._moe_big(plan, hidden, inter) is (rows % 2 == 0)
    got = ops.moe_experts(x, w13, w2, ids, weights, plan).float()
    monkeypatch.setattr(ops, "_MOE_BIG_GEMM_ROWS", 1 << 30 if rows % 2 == 0 else 1)
    other = ops.moe_experts(x, w13, w2, ids, weights, plan).float()
    want = torch.zeros(T, hidden, device="cuda")
    for e in range(experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            h = (x[t].float() @ w13[e].float().T).bfloat16().float()
            h = (torch.nn.functional.silu(h[:, :inter]).bfloat16().float() * h[:, inter:]).bfloat16().float()
            want.index_add_(0, t, (h @ w2[e].float().T).bfloat16().float() * weights[t, j, None].float())
    # products and sums of bf16 roundings
    assert float((got - want).norm() / want.norm()) < 1e-2
    assert float((got - other).norm() / other.norm()) < 1e-2


@pytest.mark.parametrize("experts,ranks,tokens", [(16, 4, 256), (64, 2, 1024), (16, 2, 1500)])
def test_shares_of_the_ranks_add_up(experts, ranks, tokens):
    """Expert parallelism with skewed routing: a rank gets more rows than the ones that its kernels were chosen for, others none."""
    from nanovllm import ops
    top, hidden, inter = 4, 512, 256
    g = torch.Generator(device="cuda").manual_seed(experts)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x, logits = rand(tokens, hidden).bfloat16(), rand(tokens, experts)
    logits[:, :experts // ranks] += 8
    w13, w2 = (rand(experts, 2 * inter, hidden) * hidden ** -0.5).bfloat16(), (rand(experts, hidden, inter) * inter ** -0.5).bfloat16()
    ids, weights = ops.moe_route(logits.bfloat16(), top)
    want = ops.moe_experts(x, w13, w2, ids, weights, ops.moe_align(ids, 0, experts)).float()
    n, got, sides = experts // ranks, torch.zeros(tokens, hidden, device="cuda"), set()
    for r in range(ranks):
        plan = ops.moe_align(ids, r * n, n, experts)
        sides.add(ops._moe_big(plan, hidden, inter))
        got += ops.moe_experts(x, w13[r * n:(r + 1) * n].contiguous(), w2[r * n:(r + 1) * n].contiguous(), ids, weights, plan).float()
    assert sides == {True}
    assert float((got - want).norm() / want.norm()) < 1e-2     # sums of bf16 roundings
