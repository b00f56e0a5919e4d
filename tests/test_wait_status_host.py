"""What the library and the runner do once a kernel has said that one of its waits ran out (the kernel's part is played by the
test, which sets the word)."""
import ctypes

import pytest


def _word():
    from nanovllm import _C
    return ctypes.cast(_C.load().b200_wait_status_word(), ctypes.POINTER(ctypes.c_int32))


def test_the_next_grouped_product_returns_the_error_once():
    from nanovllm import _C
    lib, word, one = _C.load(), _word(), ctypes.c_void_p(16)
    calls = (lambda: lib.b200_moe_gemm_gate_up_umma(one, one, one, one, None, None, 256, 64, 64, 4, 0, None),
             lambda: lib.b200_moe_gemm_down_umma(one, one, one, one, None, None, 256, 64, 128, 4, 0, None),
             lambda: lib.b200_gemm_f32out_umma(one, one, one, one, 256, 64, 128, 1, 0, None))
    for call in calls:
        word[0] = 1
        assert call() == -8 and word[0] == 0
        assert lib.b200_take_wait_status() == 0
    assert b"ran out" in lib.b200_error_string(-8)
    # arguments are still looked at first
    word[0] = 1
    assert lib.b200_moe_gemm_down_umma(one, one, one, one, one, one, 256, 64, 192, 4, 0, None) == -3
    assert lib.b200_take_wait_status() == -8 and lib.b200_take_wait_status() == 0


def test_tokens_of_a_step_whose_kernel_gave_up_are_not_returned():
    import torch
    from nanovllm import _C
    from nanovllm.engine.model_runner import ModelRunner
    assert ModelRunner._tokens(torch.tensor([3, 4])) == [3, 4]
    _word()[0] = 1
    with pytest.raises(_C.B200Error, match="not valid"):
        ModelRunner._tokens(torch.tensor([3, 4]))
    assert ModelRunner._tokens(torch.tensor([5])) == [5]


@pytest.mark.parametrize("logit_rows", [None, [1], []])
def test_what_a_decode_step_returns_is_asked_about_too(monkeypatch, logit_rows):
    """A replayed graph holds the grouped kernels, and no entry point asks for it."""
    from types import SimpleNamespace

    import torch
    from nanovllm import _C
    from nanovllm.engine.model_runner import ModelRunner
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: SimpleNamespace(synchronize=lambda: None))
    r = ModelRunner.__new__(ModelRunner)
    r.config, r.enforce_eager, r.device, r.d2h_bytes = SimpleNamespace(max_num_seqs=2), False, "cpu", 0
    r.d_out, r.h_out, r.d_logits = torch.tensor([7, 8]), torch.zeros(2, dtype=torch.int64), torch.ones(2, 3)
    given_up = [0]
    r._buckets, r._stage_decode = lambda: [2], lambda seqs, bs: 10

    def replay():
        _word()[0] = given_up[0]
    r.decode_graph = lambda bs, kv: (SimpleNamespace(replay=replay), 1)
    want = [7, 8] if logit_rows is None else None if logit_rows == [] else torch.ones(1, 3)
    same = lambda x: x == want if not isinstance(want, torch.Tensor) else torch.equal(x, want)  # noqa: E731
    assert same(r.run([object(), object()], False, logit_rows))
    given_up[0] = 1
    with pytest.raises(_C.B200Error, match="not valid"):
        r.run([object(), object()], False, logit_rows)
    given_up[0] = 0
    assert same(r.run([object(), object()], False, logit_rows))
