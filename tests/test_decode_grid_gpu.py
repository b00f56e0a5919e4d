"""The library's own choice of CTAs for paged decode attention (num_ctas 0) around the lines of its rule -- one, two and
three sequences, 8192 tokens of table, 15 and 16 rows, tiles of 8 heads of 128 and smaller ones -- against a 64-bit
evaluation. Few rows without a window have a kernel of their own (test_decode_small_gpu.py): a window that hides nothing keeps the same
rows to the rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [0, 4000])
@pytest.mark.parametrize("B,H,G,D,most,width", [(1, 16, 8, 128, 900, 512), (1, 16, 8, 128, 900, 513), (2, 8, 2, 128, 333, 256),
                                                (3, 16, 8, 128, 40, 8), (15, 16, 8, 128, 200, 16), (16, 16, 8, 128, 200, 16),
                                                (16, 32, 8, 64, 200, 16), (33, 16, 16, 128, 70, 8)])
def test_library_choice(B, H, G, D, most, width, window):
    from nanovllm import ops
    g = torch.Generator().manual_seed(B * D + width)
    lens = torch.randint(1, most + 1, (B,), generator=g)
    lens[0] = most
    need = [-(-int(n) // 16) for n in lens]
    order = torch.randperm(sum(need), generator=g).tolist()
    kc, vc = (torch.randn(sum(need), 16, G * D, generator=g).half() for _ in range(2))
    table = torch.full((B, width), -1, dtype=torch.int32)
    q = torch.randn(B, H, D, generator=g).half()
    for b in range(B):
        for i in range(need[b]):
            table[b, i] = order.pop()
    got = ops.paged_decode_attn(q.cuda(), kc.cuda(), vc.cuda(), table.cuda(), lens.to(torch.int32).cuda(), D ** -0.5, G, window=window).cpu().double()
    for b in range(B):
        n = int(lens[b])
        k, v = (c[table[b, :need[b]].long()].reshape(-1, G, D)[:n].double() for c in (kc, vc))
        for h in range(H):
            p = torch.softmax(k[:, h * G // H] @ q[b, h].double() * D ** -0.5, 0)
            # probabilities and the result in fp16: 2^-12 each of values below ~4
            assert float((got[b, h * D:(h + 1) * D] - p @ v[:, h * G // H]).abs().max()) < 4e-3, (b, h)


@pytest.mark.parametrize("B,H,G,D,most,width", [(1, 32, 32, 128, 500, 64), (1, 16, 16, 64, 900, 64), (2, 8, 2, 128, 700, 64),
                                                (2, 32, 8, 64, 700, 64), (1, 32, 16, 128, 300, 32)])
@pytest.mark.parametrize("window", [0, 4000])
def test_groups_and_widths_of_the_small_rule(B, H, G, D, most, width, window):
    """One or two rows: one, two and four groups of kv heads, query heads of 1024 and of 2048 output columns in a group."""
    test_library_choice(B, H, G, D, most, width, window)
