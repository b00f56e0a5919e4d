"""CTAs of the tcgen05 prompt kernel that walk several work items: more items than CTA slots, lengths that leave query tiles
without rows in one item after the other, heads that come alone, in threes and in pairs, windows, and keys of 192 columns
(single-stage rings). Against a 64-bit evaluation."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64
LENS = [0, 1, 128, 129, 257, 600, 40, 0, 127, 1, 300, 2, 130, 16, 1, 513, 64, 0, 200, 5]


@pytest.fixture(autouse=True)
def _layout():
    from nanovllm import _C
    yield
    _C.load().b200_prefill_set_query_tiles(0)


@pytest.mark.parametrize("tiles", [0, 1, 2])
@pytest.mark.parametrize("H,G,DK,DV,window,keep", [(16, 16, 64, 64, 0, 0), (16, 16, 128, 128, 0, 0), (24, 8, 64, 128, 0, 0),
                                                   (24, 8, 128, 64, 0, 0), (16, 16, 128, 128, 50, 3), (24, 8, 64, 64, 190, 0),
                                                   (16, 16, 192, 128, 0, 0), (16, 8, 192, 64, 0, 0), (24, 8, 192, 128, 140, 9),
                                                   (16, 8, 128, 128, 77, 1)])
def test_several_items_per_cta(H, G, DK, DV, window, keep, tiles):
    from nanovllm import _C, ops
    _C.load().b200_prefill_set_query_tiles(tiles)
    g = torch.Generator().manual_seed(H * G + DK)
    T = sum(LENS)
    assert sum(-(-n // 256) for n in LENS) * H > 2 * 148                 # more than one round in the widest layout
    q, k, v = (torch.randn(T, h, d, generator=g).half() for h, d in ((H, DK), (G, DK), (G, DV)))
    cu = torch.tensor([0] + LENS).cumsum(0).to(torch.int32).cuda()
    got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, max(LENS), max(LENS), DK ** -0.5, G, vdim=DV,
                                  window=window, keep_first=keep).cpu().to(F64).view(T, H, DV)
    at = 0
    for n in LENS:
        if not n:
            continue
        i, j = torch.arange(n)[:, None], torch.arange(n)[None]
        hidden = (j > i) | ((i - j >= window) & (j >= keep)) if window else j > i
        qs, ks, vs = (x[at:at + n].to(F64).transpose(0, 1) for x in (q, k, v))
        ks, vs = (x.repeat_interleave(H // G, 0) for x in (ks, vs))
        p = torch.softmax((qs @ ks.transpose(1, 2) * DK ** -0.5).masked_fill(hidden, -math.inf), -1)
        # P and the result in fp16: a rounding of either is 2^-12 of values up to ~4, P V sums them
        assert float((got[at:at + n] - (p @ vs).transpose(0, 1)).abs().max()) < 4e-3, n
        at += n
