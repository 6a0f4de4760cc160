"""The decoder gather, one CTA per (token, target layer), against float64: row widths on both sides of its forms, list lengths
on both sides of its groups of entries."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("D", [8, 256, 264, 512, 520, 1024, 1536, 2048, 2304, 2824])
@pytest.mark.parametrize("k,cross", [(1, 1), (4, 0), (5, 1), (9, 1), (21, 0)])
def test_gather_ends_with_its_valid_slots(k, cross, D, bf16):
    dev, T = "cuda:0", torch.bfloat16 if bf16 else torch.float32
    L, B, F = 3, 2 * k + 6, 96
    P = L * (L + 1) // 2 if cross else L
    g = torch.Generator(device=dev).manual_seed(D + k)
    W = torch.randn(P, F, D, generator=g, device=dev).to(T)
    bias = torch.randn(L, D, generator=g, device=dev)
    idx = torch.randint(0, F, (L, B, k), generator=g, device=dev, dtype=torch.int32)
    val = torch.rand(L, B, k, generator=g, device=dev) + 0.1
    # rows with 0, 1, 2 .. k valid slots; what stands behind four unused ones in a row is not looked at
    n = torch.arange(B, device=dev).clamp(max=k)[None, :, None].expand(L, B, 1)
    slot = torch.arange(k, device=dev)
    val = torch.where((slot >= n) & (slot < n + 4), torch.zeros_like(val), val)
    used = torch.where(slot < n, val, torch.zeros_like(val)).double()
    recon, status = torch.empty(B, L, D, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    lib().call("clt_sparse_decoder_fwd", idx, val, None, None, B * k, W, bias, recon, B, L, D, F, k, cross, 0, bf16, status,
               stream_ptr())
    assert int(status) == 0
    for t in range(L):
        want, mag = (b[t].double().expand(B, D).clone() for b in (bias, bias.abs()))
        for s in range(t + 1) if cross else (t,):
            rows = W[t * (t + 1) // 2 + s if cross else t].double()[idx[s].long()]          # [B, k, D]
            want += (used[s][..., None] * rows).sum(1)
            mag += (used[s][..., None] * rows.abs()).sum(1)
        # an fma chain per warp and four partial sums: fewer than (t + 1) k + 5 roundings
        assert bool(((recon[:, t].double() - want).abs() <= 2.0 ** -24 * ((t + 1) * k + 5) * mag).all())
