"""The streaming per-row selection at list sizes on both sides of its trims, on rows that keep raising the threshold."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("order", ["random", "ascending", "ties", "few_positive"])
@pytest.mark.parametrize("k,F", [(1, 8200), (31, 20000), (64, 9000), (65, 2056), (100, 8448), (200, 10000), (256, 8200)])
def test_streaming_selection(k, F, order, bf16):
    dev, T = "cuda:0", torch.bfloat16 if bf16 else torch.float32
    L, B = 2, 11
    g = torch.Generator(device=dev).manual_seed(k + F)
    z = torch.randn(L, B, F, generator=g, device=dev)
    if order == "ascending":
        z = z.sort(dim=-1).values                       # every step displaces the whole list
    elif order == "ties":
        z = (z * 2).round() / 2
    elif order == "few_positive":
        z = torch.where(torch.rand(L, B, F, generator=g, device=dev) < 0.5 * k / F, z.abs() + 0.1, -z.abs())
    z, b = z.to(T), torch.zeros(L, F, device=dev) if order == "ties" else torch.randn(L, F, generator=g, device=dev) * 0.01
    idx, val = torch.empty(L, B, k, dtype=torch.int32, device=dev), torch.empty(L, B, k, device=dev)
    fired = torch.zeros(L, (F + 31) // 32, dtype=torch.int32, device=dev)
    lib().call("clt_select_topk", z, b, idx, val, fired, B, L, F, k, bf16, stream_ptr())
    pre = z.float() + b[:, None]
    want = torch.relu(pre.topk(k, dim=-1).values)
    assert torch.equal(val.sort(dim=-1, descending=True).values, want)
    live = val > 0
    assert torch.equal(pre.gather(-1, idx.long())[live], val[live])        # each value is its feature's
    for l in range(L):
        for r in range(B):
            chosen = idx[l, r][live[l, r]]
            assert chosen.unique().numel() == chosen.numel()
    bits = torch.zeros(L, F, dtype=torch.bool, device=dev)
    for l in range(L):
        bits[l, idx[l][live[l]].long()] = True
    f = torch.arange(F, device=dev)
    got = ((fired[:, f // 32] >> (f % 32)) & 1).bool()
    assert torch.equal(got, bits)
