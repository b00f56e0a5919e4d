"""Which side of the two families of expert GEMMs ops.moe_experts takes (ops._moe_big), and which grouped kernel that side runs: a question
of the rows that the LOCAL experts can expect, not of the pairs of all ranks."""
import pytest


def _plan(tokens, top, experts, ranks=1):
    from nanovllm import ops
    local = experts // ranks
    return ops.MoePlan(tokens * top, local, 0, top, "cpu", experts)


@pytest.mark.parametrize("experts,top,hidden,inter,ranks,line", [
    (128, 8, 2048, 768, 1, 16), (128, 8, 2048, 768, 2, 16), (128, 8, 2048, 768, 4, 16), (128, 8, 2048, 768, 8, 32),
    (128, 8, 2048, 768, 16, 4),                       # 8 of 128
    (64, 4, 1024, 512, 1, 24), (64, 4, 1024, 512, 4, 24), (16, 2, 1024, 512, 1, 32), (8, 2, 2048, 1024, 1, 32),
    (64, 4, 4096, 256, 1, 32), (128, 8, 2048, 704, 1, 32), (128, 8, 1920, 768, 1, 48), (64, 4, 1152, 576, 1, 72),
    (32, 4, 1024, 512, 1, 48), (64, 8, 4096, 1792, 8, 32)])
def test_the_line_is_in_rows_of_a_local_expert(experts, top, hidden, inter, ranks, line):
    from nanovllm import ops
    for rows, side in ((line - 1, False), (line, True), (line + 1, True), (1000, True), (1, False)):
        plan = _plan(-(-rows * experts // top), top, experts, ranks)
        assert plan.local_pairs // plan.num_local == rows
        assert ops._moe_big(plan, hidden, inter) is side, rows


def test_what_moe_align_tells_the_plan():
    from nanovllm import ops
    for begin, local, experts, expected in ((0, 16, 128, 64), (112, 16, None, 64), (0, 16, None, 512), (0, 16, 16, 512)):
        assert ops.MoePlan(512, local, begin, 8, "cpu", experts).local_pairs == expected


def test_the_persistent_kernel_by_expected_pairs():
    from nanovllm import _C
    wide = _C.load().b200_moe_umma_persistent
    # 16 of 128 experts, 2048 x 768: 8 x 16 tiles of one row block each are fewer than the SMs, whatever the other ranks' pairs
    assert wide(0, 512, 16, 2048) == 0 and wide(0, 8 * 512, 16, 2048) == 1
    assert wide(1, 2048, 128, 768) == 1 and wide(1, 2047, 128, 768) == 0       # a tile per expert from 16 rows on
    assert wide(1, 4096, 128, 704) == 0 and wide(0, 4096, 128, 1920) == 0      # its bands divide the output
