"""ops.delta_rule over steps whose CTAs start with the longest sequences (csrc/delta_rule.cu, more CTAs than SMs): every sequence's outputs and
state are, bit for bit, those that it has alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("lens", [[5, 40, 0, 17, 40, 1, 64, 33, 2, 40, 9, 71], [12] * 32, [3, 90] + [1] * 18])
def test_same_as_alone(lens, per_head):
    from nanovllm import ops
    H, G, N, V, S, T = 8, 4, 128, 128, len(lens), sum(lens)
    g = torch.Generator(device="cuda").manual_seed(S)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1).reshape(T, G * N)  # noqa: E731
    q, k, v = unit(rand(T, G, N)), unit(rand(T, G, N)), rand(T, H * V).bfloat16()
    decay, beta = torch.sigmoid(rand(T, H if per_head else H * N) + 2), torch.sigmoid(rand(T, H))
    cu = lambda x: torch.tensor([0] + x).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    first = rand(S, H, N, V)
    past = [i % 2 for i in range(S)]                            # every other sequence carries a state on

    def run(a, b, lo, hi, state):
        spans = ops.StepSpans(cu(lens[a:b]), cu([n + p for n, p in zip(lens[a:b], past[a:b])]), None, max(lens[a:b]))
        return ops.delta_rule(q[lo:hi], k[lo:hi], v[lo:hi], decay[lo:hi], beta[lo:hi], spans, H, G, N, V, state=state,
                              state_slots=torch.arange(b - a, dtype=torch.int32, device="cuda"))
    state = first.clone()
    out, at = run(0, S, 0, T, state), 0
    for s, n in enumerate(lens):
        if n:
            own = first[s:s + 1].clone()
            assert torch.equal(out[at:at + n], run(s, s + 1, at, at + n, own)), (s, n)
            assert torch.equal(state[s], own[0]), (s, n)
        else:
            assert torch.equal(state[s], first[s])
        at += n
