"""The 32-token form of ops.linear_recurrence (csrc/seq_mixers.cu, prompt portions of bf16 models) at the edges of its
chunks and 16-token blocks, on aligned and unaligned rows, in portions with a carried state: against the recurrence in
64 bits, token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("H,G,N,V,selective,silu,pad,lens", [
    (4, 2, 128, 64, True, False, 0, [1, 15, 16, 17, 31, 32, 33]),
    (2, 2, 128, 128, False, True, 0, [63, 64, 65, 97]),
    (3, 1, 64, 64, False, False, 1, [5, 130]),             # rows that do not start on 16-byte boundaries
    (2, 1, 40, 72, True, False, 0, [33, 200]),
    (2, 2, 24, 8, False, True, 0, [47]),
    (1, 1, 128, 65, True, False, 3, [35]),
])
def test_against_64_bit_in_portions(H, G, N, V, selective, silu, pad, lens):
    from nanovllm import ops
    g = torch.Generator().manual_seed(N + V + len(lens))
    S = len(lens)
    past = [n // 2 for n in lens]                           # a first portion, then the rest: the state is carried
    state = torch.full((S + 1, H, N, V), float("nan"), device="cuda")
    slots = torch.tensor(list(range(S, 0, -1)), dtype=torch.int32, device="cuda")
    rows = {}
    for s, n in enumerate(lens):
        rows[s] = dict(q=torch.randn(n, G * N, generator=g).bfloat16(), k=(torch.randn(n, G * N, generator=g) * N ** -0.5).bfloat16(),
                       v=torch.randn(n, H * V, generator=g).bfloat16(), dt=torch.randn(n, H, generator=g).bfloat16())
    decay = torch.rand(H, generator=g) * 0.3 + 0.699
    bias, alog, skip = torch.randn(H, generator=g) * 0.5, -torch.rand(H, generator=g), torch.randn(H, generator=g)
    par = dict(dt_bias=bias.cuda(), a_log=alog.cuda(), d_skip=skip.cuda()) if selective else dict(decay=decay.cuda(), act_silu=silu)
    got = {s: [] for s in rows}
    for part in range(2):
        span = [(0, p) if part == 0 else (p, n) for p, n in zip(past, lens)]
        if part == 0 and not any(b for _, b in span):
            continue
        cu = lambda x: torch.tensor([0] + x).cumsum(0).to(torch.int32).cuda()  # noqa: E731

        def cat(name):                                       # a slice of a wider row, `pad` elements in
            x = torch.cat([rows[s][name][a:b] for s, (a, b) in enumerate(span)])
            wide = torch.zeros(len(x), x.shape[1] + 8 + pad, dtype=x.dtype)
            wide[:, pad:pad + x.shape[1]] = x
            return wide.cuda()[:, pad:pad + x.shape[1]]
        sp = ops.StepSpans(cu([b - a for a, b in span]), cu([b for _, b in span]), None, max(max(b - a for a, b in span), 16))
        o = ops.linear_recurrence(cat("q"), cat("k"), cat("v"), sp, H, G, N, V, state, slots,
                                  **(dict(par, dt=cat("dt")) if selective else par)).cpu()
        at = 0
        for s, (a, b) in enumerate(span):
            got[s].append(o[at:at + b - a])
            at += b - a
    act = (lambda x: torch.nn.functional.silu(x.float()).bfloat16().to(F64)) if silu else (lambda x: x.to(F64))
    for s, n in enumerate(lens):
        q, k, v = (act(rows[s][x]) for x in "qkv")
        step = torch.nn.functional.softplus(rows[s]["dt"].to(F64) + bias.to(F64)) if selective else torch.ones(n, H, dtype=F64)
        a = torch.exp(-torch.exp(alog.to(F64)) * step) if selective else decay.to(F64).expand(n, H)
        state64, want = torch.zeros(H, N, V, dtype=F64), torch.zeros(n, H, V, dtype=F64)
        for t in range(n):
            kt, qt = (x[t].view(G, N).repeat_interleave(H // G, 0) for x in (k, q))
            vt = v[t].view(H, V)
            state64 = a[t][:, None, None] * state64 + kt[:, :, None] * (step[t][:, None] * vt)[:, None, :]
            want[t] = torch.einsum("hn,hnv->hv", qt, state64) + (skip.to(F64)[:, None] * vt if selective else 0)
        x = torch.cat(got[s]).to(F64).view(n, H, V)
        # silu of the kernel rounds fast fp32 exponentials: one bf16 step of an operand now and then
        tol = 1e-2 if silu else 5e-6
        assert float((x - want).norm() / want.norm()) < tol, (s, n)
        kept = state[int(slots[s])].cpu().to(F64)
        assert float((kept - state64).norm() / state64.norm()) < tol, (s, n)
