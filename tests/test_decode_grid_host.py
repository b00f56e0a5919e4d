"""Config.decode_attn_ctas as the decode kernels are told of it: 0 asks for one CTA per SM, and the kernels' own 0 is the library's
choice."""
import types

import pytest


@pytest.mark.parametrize("setting,rows,told", [(0, 1, 148), (0, 64, 148), (0, 256, 148), (-1, 1, 0), (-1, 96, 0), (-1, 256, 104),
                                               (72, 8, 72)])
def test_what_the_step_context_says(setting, rows, told):
    from nanovllm.config import Config
    from nanovllm.engine.model_runner import ModelRunner
    from nanovllm.utils.context import get_context, reset_context
    cfg = Config("qwen3-0.6b", kvcache_block_size=16, max_num_seqs=256, max_model_len=4096, decode_attn_ctas=setting)
    r = types.SimpleNamespace(config=cfg, shard_world=1, _num_sms=148, _kv_token_bytes=4096, enforce_eager=True, block_size=16,
                              d_slots=range(256), d_ctx=range(256), d_tables=range(256), d_state=None, state_modules=[])
    for name in ("_attn_ctas", "_grid", "_set_decode_context"):
        if hasattr(ModelRunner, name):
            setattr(r, name, types.MethodType(getattr(ModelRunner, name), r))
    r._set_decode_context(rows, rows)
    assert get_context().decode_attn_ctas == told
    r._set_decode_context(rows, rows, 0, False, r._attn_ctas(rows))      # as the two halves of a split step pass it on
    assert get_context().decode_attn_ctas == told
    reset_context()
