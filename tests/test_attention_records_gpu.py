"""Streaming decode attention by the number of shares a (sequence, kv head) is cut into: the records of up to three are merged by one CTA for all
heads, of more by a CTA per head, eight at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# batch x kv heads x chunks of 128 keys over 148 shares: 1 to 3 shares per head, about 4, 7 to 9, 16 and 17, one share per chunk and far more
@pytest.mark.parametrize("B,H,S", [(37, 8, 130), (37, 4, 385), (74, 1, 1100), (37, 1, 600), (18, 1, 1300), (9, 1, 2100), (9, 1, 4000), (4, 1, 1357), (1, 1, 20000)])
@pytest.mark.parametrize("G", [1, 3, 8])
def test_merge_of_shares(B, H, S, G):
    from maco_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(S)
    q = torch.randn(B, H * G, 128, device="cuda", generator=g).half()
    k = torch.randn(B, H, S, 128, device="cuda", generator=g).half()
    v = torch.randn(B, H, S, 128, device="cuda", generator=g).half()
    s = torch.einsum("bhgd,bhsd->bhgs", q.double().view(B, H, G, 128), k.double()) * 128 ** -0.5
    want = torch.einsum("bhgs,bhsd->bhgd", torch.softmax(s, -1), v.double()).reshape(B, H * G, 128)
    got = ops.attention_decode(q, k, v)
    # one rounding to fp16; fp32 sums of weights that add up to 1, of values up to about 5
    assert ((got.double() - want).abs() <= 2.0 ** -11 * want.abs() + 2.0 ** -17 * v.abs().max().double()).all()
