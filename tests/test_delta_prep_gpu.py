"""ops.delta_prep on both sides of the rule between its element-wise and its 16-byte form (csrc/stream_ops.cu): units per
launch, sizes that 8 divides or does not, fp32 inputs, unaligned rows; against a 64-bit evaluation."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("H,G,D,per_head,T", [(8, 4, 128, False, 127), (8, 4, 128, False, 128), (32, 16, 64, False, 63),
                                              (32, 16, 64, False, 65), (8, 4, 128, True, 1023), (8, 4, 128, True, 1024),
                                              (32, 16, 64, True, 279), (32, 16, 64, True, 280), (4, 2, 256, False, 300),
                                              (6, 2, 24, True, 1000), (3, 1, 21, False, 900), (1, 1, 8, False, 5)])
@pytest.mark.parametrize("dtype,pad", [(torch.bfloat16, 0), (torch.bfloat16, 3), (torch.float32, 0)])
def test_against_64_bit(H, G, D, per_head, T, dtype, pad):
    from nanovllm import ops
    g = torch.Generator().manual_seed(T + D)
    n = H if per_head else H * D

    def rows(width):                                         # a slice of a wider row, `pad` elements in
        x = torch.randn(T, width + 8 + pad, generator=g).to(dtype)
        return x[:, pad:pad + width], x.cuda()[:, pad:pad + width]
    (qk, qk_d), (a, a_d), (b, b_d) = rows(2 * G * D), rows(n), rows(H)
    bias, alog = torch.randn(n, generator=g), torch.randn(H, generator=g)
    got_qk, got_g, got_b = ops.delta_prep(qk_d, a_d, b_d, bias.cuda(), alog.cuda(), H, G, D, 1e-6, D ** -0.5, per_head=per_head)
    x = qk.to(F64).view(T, 2, G, D)
    x = x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) * torch.tensor([D ** -0.5, 1.0], dtype=F64)[:, None, None]
    soft = torch.nn.functional.softplus(a.to(F64) + bias.to(F64)).view(T, H, -1)
    decay = torch.exp(-torch.exp(alog.to(F64))[:, None] * soft)
    # fp32: sums of up to 256 squares, an exponential of an argument of up to ~50
    for got, want, tol in ((got_qk, x, 1e-6), (got_g, decay, 5e-6), (got_b, torch.sigmoid(b.to(F64)), 1e-6)):
        got = got.cpu().to(F64).reshape(want.shape)
        assert float((got - want).abs().max()) <= tol, float((got - want).abs().max())
