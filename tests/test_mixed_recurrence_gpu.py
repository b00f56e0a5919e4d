"""ops.linear_recurrence where prompt portions stand beside single tokens (a rank-1 update each, csrc/seq_mixers.cu), below and
above the number of CTAs from which small states run with twice as many per SM; with and without a carried state, in
64 bits token by token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("H,G,N,V,selective,silu,pad,lens", [
    (4, 2, 128, 64, True, False, 0, [40, 1, 1, 17, 1]),
    (2, 2, 128, 128, False, True, 0, [1, 33, 1]),
    (3, 1, 63, 65, False, False, 1, [20, 1]),
    (2, 1, 24, 40, True, True, 0, [1, 16, 1]),
    (1, 1, 1, 8, False, False, 0, [1, 18]),
    (32, 8, 64, 64, True, False, 0, [1, 16, 2, 33, 1, 1, 5, 1, 32, 1]),
    (32, 32, 64, 64, False, True, 1, [1, 16, 2, 33, 1, 1, 5, 1, 32, 1]),
    (32, 4, 40, 100, True, False, 0, [18, 1, 1, 34, 1]),
    (60, 60, 32, 24, False, False, 0, [1, 31, 65, 1, 1]),
])
@pytest.mark.parametrize("bound", [True, False])
def test_against_64_bit(H, G, N, V, selective, silu, pad, lens, bound):
    from nanovllm import ops
    g = torch.Generator().manual_seed(N + V + H)
    S, T = len(lens), sum(lens)
    past = [(s * 7) % 3 if bound else 0 for s in range(S)]     # 0: a fresh sequence, whose slot holds another one's state
    state0 = torch.randn(S + 1, H, N, V, generator=g)
    state, slots = state0.cuda(), torch.tensor(list(range(S, 0, -1)), dtype=torch.int32, device="cuda")

    def rows(width, scale=1.0):                                # a slice of a wider row, `pad` elements in
        x = (torch.randn(T, width + 8 + pad, generator=g) * scale).bfloat16()
        return x[:, pad:pad + width], x.cuda()[:, pad:pad + width]
    (q, qd), (k, kd), (v, vd), (dt, dtd) = rows(G * N), rows(G * N, N ** -0.5), rows(H * V), rows(H)
    decay = torch.rand(H, generator=g) * 0.3 + 0.699
    bias, alog, skip = torch.randn(H, generator=g) * 0.5, -torch.rand(H, generator=g), torch.randn(H, generator=g)
    par = dict(dt=dtd, dt_bias=bias.cuda(), a_log=alog.cuda(), d_skip=skip.cuda()) if selective else dict(decay=decay.cuda(), act_silu=silu)
    cu = lambda x: torch.tensor([0] + x).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    sp = ops.StepSpans(cu(lens), cu([n + p for n, p in zip(lens, past)]), None, max(lens))
    got = ops.linear_recurrence(qd, kd, vd, sp, H, G, N, V, state if bound else None, slots if bound else None, **par).cpu().to(F64)
    act = (lambda x: torch.nn.functional.silu(x.float()).bfloat16().to(F64)) if silu and not selective else (lambda x: x.to(F64))
    # silu of the kernel rounds fast fp32 exponentials: one bf16 step of an operand now and then
    tol, at = 1e-2 if silu and not selective else 5e-6, 0
    for s, n in enumerate(lens):
        slot = int(slots[s])
        st = state0[slot].to(F64) if past[s] else torch.zeros(H, N, V, dtype=F64)
        want = torch.zeros(n, H, V, dtype=F64)
        for t in range(n):
            kt, qt = (act(x[at + t]).view(G, N).repeat_interleave(H // G, 0) for x in (k, q))
            vt = act(v[at + t]).view(H, V)
            step = torch.nn.functional.softplus(dt[at + t].to(F64) + bias.to(F64)) if selective else torch.ones(H, dtype=F64)
            a = torch.exp(-torch.exp(alog.to(F64)) * step) if selective else decay.to(F64)
            st = a[:, None, None] * st + kt[:, :, None] * (step[:, None] * vt)[:, None, :]
            want[t] = torch.einsum("hn,hnv->hv", qt, st) + (skip.to(F64)[:, None] * vt if selective else 0)
        x = got[at:at + n].view(n, H, V)
        assert float((x - want).norm() / want.norm()) < tol, (s, n)
        if bound:
            assert float((state[slot].cpu().to(F64) - st).norm() / st.norm()) < tol, (s, n)
        at += n
    if bound:
        assert torch.equal(state[0].cpu(), state0[0])          # a slot that no sequence holds
