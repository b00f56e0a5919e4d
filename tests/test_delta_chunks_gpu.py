"""ops.delta_rule over prompts in chunks of 64 tokens (csrc/delta_chunks.cu) against the recurrence in 64 bits, beside the token-by-token form
(csrc/delta_rule.cu) on the same inputs, and bit for bit against that form where a head is left to it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _inputs(lens, H, G, N, per_head, decay="mild", seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(lens) + N)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    T = sum(lens)
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1).reshape(T, G * N)  # noqa: E731
    q, k, v = unit(rand(T, G, N)) * N ** -0.5, unit(rand(T, G, N)), rand(T, H * N).bfloat16()
    raw = rand(T, H if per_head else H * N)
    if decay == "mild":
        gate = torch.exp(-0.3 * torch.nn.functional.softplus(raw + 1))
    elif decay == "none":
        gate = torch.ones_like(raw)
    elif decay == "edge":                                  # 2^-74 to 2^-85 over half a chunk
        gate = 0.16 + 0.04 * torch.sigmoid(raw)
    elif decay == "strong":                                # down to e^-30 a token, some exactly zero
        gate = torch.exp(-6 * torch.nn.functional.softplus(2 * raw))
        gate[raw > 2.2] = 0.0
    else:                                                  # "signed": a channel may change its sign, or grow a little
        gate = torch.where(raw > 0, 1.0, -1.0) * (0.55 + 0.5 * torch.sigmoid(raw))
    return q, k, v, gate.contiguous(), torch.sigmoid(rand(T, H)), g


def _spans(lens, past):
    from nanovllm import ops
    cu = lambda x: torch.tensor([0] + x).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    return ops.StepSpans(cu(lens), cu([n + p for n, p in zip(lens, past)]), None, max(lens))


def _call(entry, q, k, v, gate, beta, spans, H, G, N, state, slots, *extra):
    """A C entry of the delta rule: the token form (b200_delta_rule), or chunks within a workspace of a given size."""
    from nanovllm import _C, ops
    out = torch.full((q.shape[0], H * N), 7.0, device="cuda")
    cu_q, cu_k, ctx = spans.ptrs()
    args = [out.data_ptr(), q.data_ptr(), q.stride(0), k.data_ptr(), k.stride(0), v.data_ptr(), v.stride(0), gate.data_ptr(), beta.data_ptr(),
            ops._ptr(state), ops._ptr(slots), cu_q, cu_k, ctx, spans.num_seqs]
    sizes = [H, G, N, N, 1 if gate.shape[1] == H else 0, 0]
    if entry == "tokens":
        _C.check(_C.load().b200_delta_rule(*args, *sizes, ops._stream()), "b200_delta_rule")
    else:
        ws = torch.empty(extra[0], dtype=torch.uint8, device="cuda")
        _C.check(_C.load().b200_delta_rule_step(*args, spans.max_q, q.shape[0], *sizes, ws.data_ptr(), ws.numel(), ops._stream()), "b200_delta_rule_step")
    return out


def _exact(lens, past, q, k, v, gate, beta, H, G, N, first):
    T = q.shape[0]
    q, k = (x.to(F64).view(T, G, N).repeat_interleave(H // G, 1) for x in (q, k))
    v, beta = v.to(F64).view(T, H, N), beta.to(F64)
    gate = gate.to(F64).view(T, H, -1)
    o = torch.empty(T, H, N, dtype=F64, device="cuda")
    S = [(first[i].to(F64) if past[i] else torch.zeros(H, N, N, dtype=F64, device="cuda")) for i in range(len(lens))]
    at = 0
    for i, n in enumerate(lens):
        for t in range(at, at + n):
            S[i] = gate[t][..., None] * S[i]
            w = beta[t][:, None] * (v[t] - torch.matmul(k[t][:, None, :], S[i]).squeeze(1))
            S[i] = S[i] + k[t][..., None] * w[:, None, :]
            o[t] = torch.matmul(q[t][:, None, :], S[i]).squeeze(1)
        at += n
    return o.reshape(T, H * N), torch.stack(S)


def _off(x, want):
    return float((x.to(F64) - want).norm() / want.norm())


SIZES = [(4, 2, 128), (8, 4, 64)]
LENS = [[1, 63, 64, 65, 0, 130, 201], [300], [96, 128, 33]]


@pytest.mark.parametrize("H,G,N", SIZES)
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("decay", ["mild", "none", "edge", "strong", "signed"])
def test_against_64_bits(H, G, N, per_head, lens, decay):
    """No further from the result than 1.5 times the token form, or 2e-7 (a chunk sums in another order; both are 24-bit arithmetic). Strong decays
    are down to e^-30 a token, some exactly zero: one per head goes on the scores, those per channel take the blocks of 16 tokens."""
    from nanovllm import ops
    q, k, v, gate, beta, g = _inputs(lens, H, G, N, per_head, decay)
    past = [9 if i % 2 else 0 for i in range(len(lens))]
    first = torch.randn(len(lens), H, N, N, device="cuda", generator=g)
    spans, slots = _spans(lens, past), torch.arange(len(lens), dtype=torch.int32, device="cuda").flip(0).contiguous()
    want, want_S = _exact(lens, past, q, k, v, gate, beta, H, G, N, first)
    state, tokens = first.flip(0).contiguous(), first.flip(0).contiguous()
    out = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N, state, slots)
    ref = _call("tokens", q, k, v, gate, beta, spans, H, G, N, tokens, slots)
    live = [i for i, n in enumerate(lens) if n]
    for got, token, exact in ((out, ref, want), (state.flip(0)[live], tokens.flip(0)[live], want_S[live])):
        assert _off(got, exact) <= max(1.5 * _off(token, exact), 2e-7), (_off(got, exact), _off(token, exact))
    assert not torch.equal(out, ref)                       # (no head is left to tokens)
    for i, n in enumerate(lens):
        if n == 0:
            assert torch.equal(state.flip(0)[i], first[i])


@pytest.mark.parametrize("H,G,N", SIZES)
@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("decay,states", [("none", 1.0), ("signed", 1.1), ("mild", 1.2), ("edge", 1.6), ("strong", 1.6)])
def test_no_precision_is_lost(H, G, N, per_head, decay, states):
    """Outputs are as near to 64 bits as the token form's (0.8 to 0.98 of its error; half of it without decays). So are states that remember. Where the
    last token is most of a state, the token form rounds three times and a chunk five, twice by cutting off: sqrt(5 / 3) and more."""
    from nanovllm import ops
    lens, off = [700, 350], []
    for seed in (1, 2):
        q, k, v, gate, beta, g = _inputs(lens, H, G, N, per_head, decay, seed)
        first, slots = torch.randn(2, H, N, N, device="cuda", generator=g), torch.arange(2, dtype=torch.int32, device="cuda")
        spans, state, tokens = _spans(lens, [0, 9]), first.clone(), first.clone()
        want, want_S = _exact(lens, [0, 9], q, k, v, gate, beta, H, G, N, first)
        out = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N, state, slots)
        ref = _call("tokens", q, k, v, gate, beta, spans, H, G, N, tokens, slots)
        off.append([_off(out, want), _off(ref, want), _off(state, want_S), _off(tokens, want_S)])
    out, ref, state, tokens = (sum(x) / 2 for x in zip(*off))
    assert out <= 1.02 * ref and state <= states * tokens, (out / ref, state / tokens)


@pytest.mark.parametrize("H,G,N", SIZES)
@pytest.mark.parametrize("pattern", ["one channel", "second half of the channels", "one token of zeros", "each block", "2^-83"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 150])
def test_strong_decays_of_few_channels(H, G, N, pattern, n):
    """Every pair of the blocks of 16 tokens in turn, beside a sequence that does not need them: outputs of each as near to 64 bits as the token form."""
    from nanovllm import ops
    lens = [n, 130]
    q, k, v, gate, beta, g = _inputs(lens, H, G, N, False)
    marks = gate.view(n + 130, H, N)
    if pattern == "one channel":
        marks[:, 0, 5] = 1e-4
    elif pattern == "second half of the channels":
        marks[:, 1, N // 2:] = 3e-3
    elif pattern == "one token of zeros":
        marks[n // 2, :, ::3] = 0.0
    elif pattern == "each block":
        marks[::16] = 1e-30
    else:                                                  # around the line of a half chunk's decays
        marks[:32, :, 3], marks[32:, :, 3] = 2.0 ** -2.59, 2.0 ** -2.60
    first, slots = torch.randn(2, H, N, N, device="cuda", generator=g), torch.arange(2, dtype=torch.int32, device="cuda")
    spans, state, tokens = _spans(lens, [4, 0]), first.clone(), first.clone()
    want, want_S = _exact(lens, [4, 0], q, k, v, gate, beta, H, G, N, first)
    out = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N, state, slots)
    ref = _call("tokens", q, k, v, gate, beta, spans, H, G, N, tokens, slots)
    assert not torch.equal(out, ref)
    for rows in (slice(0, n), slice(n, n + 130)):          # (a few rows alone: their errors spread by a quarter)
        assert _off(out[rows], want[rows]) <= 1.3 * _off(ref[rows], want[rows])
    assert _off(state, want_S) <= 1.6 * _off(tokens, want_S)


@pytest.mark.parametrize("H,G,N", SIZES)
@pytest.mark.parametrize("with_state", [False, True])
@pytest.mark.parametrize("decay", ["mild", "strong"])
def test_any_workspace_gives_the_same(H, G, N, decay, with_state):
    """One chunk of every head at a time, a few, all: the same bits (a pass hands the state on in fp32)."""
    from nanovllm import _C
    lens = [200, 1, 130, 64, 333]
    q, k, v, gate, beta, g = _inputs(lens, H, G, N, False, decay)
    first = torch.randn(len(lens), H, N, N, device="cuda", generator=g)
    spans, slots = _spans(lens, [5, 0, 3, 0, 0] if with_state else [0] * 5), torch.arange(len(lens), dtype=torch.int32, device="cuda") if with_state else None
    whole = _C.load().b200_delta_rule_workspace_size(len(lens), max(lens), sum(lens), H, G, N, N, 0, 0)
    carry = H * N * N * 4
    chunks = sum(lens) // 64 + len(lens)
    got = []
    for n in (chunks, 5, 3, 1):
        state = first.clone() if with_state else None
        got.append((_call("step", q, k, v, gate, beta, spans, H, G, N, state, slots, carry + (whole - carry) // chunks * n), state))
    assert not torch.equal(got[0][0], _call("tokens", q, k, v, gate, beta, spans, H, G, N, first.clone() if with_state else None, slots))
    for out, state in got[1:]:
        assert torch.equal(out, got[0][0]) and (state is None or torch.equal(state, got[0][1]))


@pytest.mark.parametrize("H,G,N", SIZES)
@pytest.mark.parametrize("what", ["v inf", "k nan", "k huge", "k tiny", "g nan", "v huge", "state inf", "g two"])
@pytest.mark.parametrize("passes", [False, True])
def test_heads_left_to_tokens(H, G, N, what, passes):
    """Values that chunks cannot take: their heads (pairs of heads of 64) are what the token form gives, bit for bit, the others as without them."""
    from nanovllm import _C
    lens = [150, 200]
    q, k, v, gate, beta, g = _inputs(lens, H, G, N, False)
    first = torch.randn(2, H, N, N, device="cuda", generator=g)
    spans, slots = _spans(lens, [0, 4]), torch.arange(2, dtype=torch.int32, device="cuda")
    whole = _C.load().b200_delta_rule_workspace_size(2, 200, 350, H, G, N, N, 0, 0)
    carry, chunks = H * N * N * 4, 350 // 64 + 2
    ws = carry + (whole - carry) // chunks * (2 if passes else chunks)
    clean_state = first.clone()
    clean = _call("step", q, k, v, gate, beta, spans, H, G, N, clean_state, slots, ws)
    hit, at = [0], 150 + 70                                # head 0 of the second sequence, in its second chunk
    if what == "v inf":
        v[at, 3] = float("inf")
    elif what == "v huge":
        v[at, 3] = 1e30
    elif what == "k nan":
        k[at, 5], hit = float("nan"), list(range(H // G))
    elif what == "k huge":                                 # (its product with a reciprocal of 2^90 would be infinite)
        k[at, 5], hit = 2.0 ** 40, list(range(H // G))
    elif what == "k tiny":                                 # (low terms times decays of 2^-90 would be lost): the whole second chunk's
        k[150 + 64:150 + 128, :N] *= 2.0 ** -30
        hit = list(range(H // G))
    elif what == "g nan":
        gate[at, 5] = float("nan")
    elif what == "g two":
        gate[at, 5] = 2.5
    else:
        first[1, 0, 7, 7] = float("inf")
    state, tokens = first.clone(), first.clone()
    out = _call("step", q, k, v, gate, beta, spans, H, G, N, state, slots, ws)
    ref = _call("tokens", q, k, v, gate, beta, spans, H, G, N, tokens, slots)
    same = lambda a, b: torch.equal(a.nan_to_num(7.5, 8.5, 9.5), b.nan_to_num(7.5, 8.5, 9.5))  # noqa: E731
    if N == 64:
        hit = sorted({h ^ x for h in hit for x in (0, 1)})
    for h in range(H):
        cols = slice(h * N, (h + 1) * N)
        assert torch.equal(out[:150, cols], clean[:150, cols])
        if h in hit and not passes:
            assert same(out[150:, cols], ref[150:, cols]) and same(state[1, h], tokens[1, h])
        elif h in hit:                                     # (earlier passes may have taken chunks: another order of sums, then the same)
            for got, want in ((out[150:, cols], ref[150:, cols]), (state[1, h], tokens[1, h])):
                fine = want.isfinite()
                assert torch.equal(got.isfinite(), fine)
                size = want.where(fine, want.new_zeros(())).abs().amax(0, keepdim=True)      # (of a value column: one may be huge)
                assert bool((((got - want).abs() <= 1e-4 * want.abs() + 1e-5 * size) | ~fine).all())
        else:
            assert torch.equal(out[150:, cols], clean[150:, cols]) and torch.equal(state[1, h], clean_state[1, h])


@pytest.mark.parametrize("H,G,N", [(4, 2, 128), (8, 4, 64)])
@pytest.mark.parametrize("with_state,past", [(False, [0, 0]), (True, [0, 0]), (True, [3, 5])])
@pytest.mark.parametrize("room", [5, 1])                 # (three passes of four, or one chunk at a time)
def test_a_sequence_that_ends_and_one_that_goes_on_in_one_pass(H, G, N, with_state, past, room):
    """Two sequences of six chunks in passes of four (or one): the second pass ends the first and has the start of the other. Heads of the first, of
    the other, of both and of neither are left to tokens in that pass. A slot's earlier content is nothing to a sequence without a past. What a
    chunk does is as near to 64 bits as the token form: 2.5e-7 at most each, their difference below 1e-6."""
    from nanovllm import _C
    lens = [330, 330]
    q, k, v, gate, beta, g = _inputs(lens, H, G, N, False)
    marks = gate.view(660, H, N)                            # (a decay of two is not for chunks)
    each = H // 4
    marks[4 * 64 + 10, 0 * each:1 * each, 5] = 2.0
    marks[330 + 20, 1 * each:2 * each, 5] = 2.0
    marks[4 * 64 + 10, 2 * each:3 * each, 5] = 2.0
    marks[330 + 20, 2 * each:3 * each, 5] = 2.0
    first = torch.randn(2, H, N, N, device="cuda", generator=g)
    spans, slots = _spans(lens, past), torch.arange(2, dtype=torch.int32, device="cuda") if with_state else None
    whole = _C.load().b200_delta_rule_workspace_size(2, 330, 660, H, G, N, N, 0, 0)
    carry, chunks = H * N * N * 4, 660 // 64 + 2
    state, tokens = (first.clone(), first.clone()) if with_state else (None, None)
    for _ in range(3):
        if with_state:
            state.copy_(first)
        out = _call("step", q, k, v, gate, beta, spans, H, G, N, state, slots, carry + (whole - carry) // chunks * room)
    ref = _call("tokens", q, k, v, gate, beta, spans, H, G, N, tokens, slots)
    for h in range(H):
        cols = slice(h * N, (h + 1) * N)
        for rows in (slice(0, 256), slice(256, 330), slice(330, 458), slice(458, 660)):
            assert _off(out[rows, cols], ref[rows, cols].to(F64)) < 1e-6, (h, rows)
        if with_state:
            for s in range(2):
                assert _off(state[s, h], tokens[s, h].to(F64)) < 1e-6, (h, s)
    assert not torch.equal(out, ref)


def test_a_wait_that_runs_out_is_reported(monkeypatch):
    from types import SimpleNamespace

    from nanovllm import _C, ops
    H, G, N, lens = 8, 4, 128, [500, 129, 300]
    q, k, v, gate, beta, _ = _inputs(lens, H, G, N, False)
    spans, slots, lib = _spans(lens, [0, 0, 0]), torch.arange(3, dtype=torch.int32, device="cuda"), _C.load()
    call = lambda: ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N, torch.zeros(3, H, N, N, device="cuda"), slots)  # noqa: E731
    want = call()
    torch.cuda.synchronize()
    ops.check_waits()
    impatient = SimpleNamespace(b200_delta_rule_workspace_size=lib.b200_delta_rule_workspace_size,
                                b200_delta_rule_step=lambda *a: lib.b200_delta_rule_bounded(*a[:-1], 0, a[-1]))
    with monkeypatch.context() as m:
        m.setattr(_C, "load", lambda: impatient)
        first = call()
    torch.cuda.synchronize()
    with pytest.raises(_C.B200Error, match="ran out"):
        call()
    assert not torch.equal(first, want)
    assert torch.equal(call(), want)
    torch.cuda.synchronize()
    ops.check_waits()


def test_a_first_call_in_a_captured_graph():
    """The launches alone, workspace from the graph's pool: a replay on new inputs gives what a plain call gives."""
    from nanovllm import ops
    H, G, N, lens = 4, 2, 128, [200, 100]
    q, k, v, gate, beta, _ = _inputs(lens, H, G, N, False)
    spans = _spans(lens, [0, 0])
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            out = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N)
    torch.cuda.current_stream().wait_stream(side)
    other = _inputs(lens, H, G, N, False, seed=5)
    for a, b in zip((q, k, v, gate, beta), other[:5]):
        a.copy_(b)
    graph.replay()
    assert torch.equal(out, ops.delta_rule(*other[:5], spans, H, G, N, N))


@pytest.mark.parametrize("free", [1 << 40, 12 << 20, 3 << 20, 0])
def test_what_memory_there_is(monkeypatch, free):
    """Where the workspace that a step would like is not to be had, it takes several passes (the same bits), and without any goes token by token."""
    from nanovllm import ops
    H, G, N, lens = 4, 2, 128, [500, 129, 700]
    q, k, v, gate, beta, _ = _inputs(lens, H, G, N, False)
    spans, empty, asked = _spans(lens, [0, 0, 0]), torch.empty, []
    want = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N)

    def short(*size, **kw):
        if kw.get("dtype") == torch.uint8:
            asked.append(size[0])
            if size[0] > free:
                raise torch.OutOfMemoryError("CUDA out of memory")
        return empty(*size, **kw)
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", short)
        got = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N)
    assert (len(asked) == 1) == (free > 1 << 30)
    assert torch.equal(got, want if free else _call("tokens", q, k, v, gate, beta, spans, H, G, N, None, None))


def test_a_step_whose_workspace_is_small_takes_chunks():
    """Less than a MB, which is where a step gives up asking for less: it is asked for all the same."""
    from nanovllm import _C, ops
    H, G, N, lens = 2, 2, 64, [130]
    q, k, v, gate, beta, _ = _inputs(lens, H, G, N, False)
    spans = _spans(lens, [0])
    assert 0 < _C.load().b200_delta_rule_workspace_size(1, 130, 130, H, G, N, N, 0, 0) < 1 << 20
    out = ops.delta_rule(q, k, v, gate, beta, spans, H, G, N, N)
    assert not torch.equal(out, _call("tokens", q, k, v, gate, beta, spans, H, G, N, None, None))
