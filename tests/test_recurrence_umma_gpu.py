"""ops.linear_recurrence in chunks of 64 tokens on the tensor cores (csrc/recurrence_umma.cu): spans around its chunks, its 16-token
blocks and the length from which it takes a span, beside spans that chunk_recurrence_kernel keeps; two heads per CTA and one,
key sizes that are padded, in two portions with a carried state, against the recurrence in 64 bits, token by token. Tolerance:
fp32 sums of a few hundred terms, as the other tests of these recurrences."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("H,G,N,V,selective,silu,lens", [
    (4, 2, 128, 64, True, False, [130, 1, 200, 95, 96, 97, 17, 0, 385]),
    (4, 1, 72, 64, True, True, [128, 191, 1]),
    (2, 2, 128, 128, False, True, [96, 1, 129, 64]),
    (2, 1, 128, 128, True, False, [257]),
    (4, 2, 64, 64, False, False, [255, 256, 257, 1, 320]),
    (2, 1, 40, 128, True, False, [321, 1, 63]),
    (2, 2, 64, 128, False, True, [449]),
])
def test_against_64_bit_in_portions(H, G, N, V, selective, silu, lens):
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(N + V + len(lens))
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    S = len(lens)
    state = torch.full((S + 1, H, N, V), float("nan"), device="cuda")
    slots = torch.tensor(list(range(S, 0, -1)), dtype=torch.int32, device="cuda")
    rows = [dict(q=rand(2 * n, G * N).bfloat16(), k=(rand(2 * n, G * N) * N ** -0.5).bfloat16(), v=rand(2 * n, H * V).bfloat16(),
                 dt=rand(2 * n, H).bfloat16()) for n in lens]
    decay = 0.699 + 0.3 * torch.rand(H, device="cuda", generator=g)
    bias, alog, skip = rand(H) * 0.5, -torch.rand(H, device="cuda", generator=g), rand(H)
    par = dict(dt_bias=bias, a_log=alog, d_skip=skip) if selective else dict(decay=decay, act_silu=silu)
    cu = lambda x: torch.tensor([0] + x).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    act = (lambda x: torch.nn.functional.silu(x.float()).bfloat16().to(F64)) if silu and not selective else (lambda x: x.to(F64))
    tol = 1e-2 if silu and not selective else 5e-6             # silu: one bf16 step of an operand now and then
    want_state = torch.zeros(S, H, N, V, dtype=F64, device="cuda")
    for part in range(2):
        at = [slice(part * n, (part + 1) * n) for n in lens]
        d = {x: torch.cat([r[x][a] for r, a in zip(rows, at)]) for x in ("q", "k", "v", "dt")}
        sp = ops.StepSpans(cu(lens), cu([n * (part + 1) for n in lens]), None, max(lens))
        o = ops.linear_recurrence(d["q"], d["k"], d["v"], sp, H, G, N, V, state, slots, **(dict(par, dt=d["dt"]) if selective else par))
        begin = 0
        for s, n in enumerate(lens):
            q, k, v = (act(rows[s][x][at[s]]) for x in "qkv")
            step = torch.nn.functional.softplus(rows[s]["dt"][at[s]].to(F64) + bias.to(F64)) if selective else torch.ones(n, H, dtype=F64, device="cuda")
            a = torch.exp(-torch.exp(alog.to(F64)) * step) if selective else decay.to(F64).expand(n, H)
            st, want = want_state[s], torch.zeros(n, H, V, dtype=F64, device="cuda")
            q, k = (x.view(n, G, N).repeat_interleave(H // G, 1) for x in (q, k))
            vx = step[:, :, None] * v.view(n, H, V)
            for t in range(n):
                st.mul_(a[t][:, None, None]).add_(k[t][:, :, None] * vx[t][:, None, :])
                want[t] = torch.matmul(q[t][:, None, :], st).squeeze(1)
            if selective:
                want += skip.to(F64)[:, None] * v.view(n, H, V)
            if n:
                x = o[begin:begin + n].to(F64).view(n, H, V)
                assert float((x - want).norm() / want.norm()) < tol, (part, s, n)
                kept = state[int(slots[s])].to(F64)
                assert float((kept - st).norm() / st.norm()) < tol, (part, s, n)
            begin += n
    assert bool(torch.isnan(state[0]).all())                   # a slot that no sequence holds


def test_the_switch_that_turns_chunks_off():
    """B200_CHUNK_RECURRENCE=0: token by token, whatever the length (the fp32 model's kernel gives the same bits for the same inputs)."""
    import os
    import subprocess
    import sys
    code = """
import sys; sys.path.insert(0, "nano-vllm-ascend_b200")
import torch
from nanovllm import ops
g = torch.Generator(device="cuda").manual_seed(1)
rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
T, H, N, V = 300, 2, 128, 128
q, k, v, decay = rand(T, H * N), rand(T, H * N), rand(T, H * V), torch.tensor([0.9, 0.99], device="cuda")
cu = torch.tensor([0, T], dtype=torch.int32, device="cuda")
sp = ops.StepSpans(cu, cu, None, T)
a, b = (ops.linear_recurrence(*t, sp, H, H, N, V, None, None, decay=decay) for t in ((q, k, v), (q.float(), k.float(), v.float())))
print("SAME" if torch.equal(a, b) else "OTHER")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for value, want in (("0", "SAME"), ("1", "OTHER")):
        done = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, B200_CHUNK_RECURRENCE=value), capture_output=True, text=True)
        assert done.stdout.split() == [want], (value, done.stdout, done.stderr[-2000:])


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("V,silu,at", [(64, False, 60), (64, False, 64), (128, True, 127), (128, False, 0), (128, False, 299)])
def test_a_value_that_is_not_finite_spoils_nothing_before_it(bad, V, silu, at):
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(at)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    lens, H, N, c = [300, 97], 2, 128, V + 5                   # a channel of the second head
    T = sum(lens)
    q, k, v, decay = rand(T, H * N), rand(T, H * N), rand(T, H * V), torch.tensor([0.9, 0.99], device="cuda")
    cu = torch.tensor([0, 300, 397], dtype=torch.int32, device="cuda")
    sp = ops.StepSpans(cu, cu, None, 300)
    slots = torch.arange(2, dtype=torch.int32, device="cuda")
    run = lambda v, s: ops.linear_recurrence(q, k, v, sp, H, 1 if V == 64 else H, N, V, s, slots, decay=decay, act_silu=silu)  # noqa: E731
    if V == 64:
        q, k = q[:, :N], k[:, :N]                              # two heads per CTA share q and k
    fine, kept = torch.zeros(2, H, N, V, device="cuda"), torch.zeros(2, H, N, V, device="cuda")
    want = run(v, fine)
    v2 = v.clone()
    v2[at, c] = bad
    got = run(v2, kept)
    spoilt = torch.zeros(T, H * V, dtype=torch.bool, device="cuda")
    spoilt[at:300, c] = True
    assert torch.equal(torch.isfinite(got), ~spoilt)
    assert torch.equal(got[~spoilt], want[~spoilt])
    column = torch.zeros_like(kept, dtype=torch.bool)
    column[0, 1, :, 5] = True
    assert not bool(torch.isfinite(kept[column]).any()) and torch.equal(kept[~column], fine[~column])
