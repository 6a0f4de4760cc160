"""clt_select_topk_export against the selection, the layout kernel and the scatter that it stands for: bit for bit."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


# whole steps of 256 columns, a ragged end alone and behind steps, fewer positive values than k, lists that overflow (equal
# values), rows that do not fill a CTA
@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("L,B,F,k,kind", [(1, 1, 8, 8, "normal"), (2, 9, 248, 16, "normal"), (3, 5, 256, 1, "normal"),
                                          (2, 17, 264, 256, "normal"), (2, 33, 8200, 64, "normal"),
                                          (1, 8, 20000, 200, "normal"), (2, 7, 4096, 32, "negative"),
                                          (2, 7, 4096, 32, "equal")])
def test_one_sweep_equals_three_passes(L, B, F, k, kind, bf16):
    g = torch.Generator(device="cuda:0").manual_seed(F + k)
    z = torch.randn(L, B, F, generator=g, device="cuda:0")
    if kind == "negative":
        z = -z.abs()
        z[:, :, 5::777] *= -1
    elif kind == "equal":
        z.fill_(0.5)
    z = z.to(torch.bfloat16 if bf16 else torch.float32)
    b = torch.zeros(L, F, device="cuda:0") if kind == "equal" else 0.02 * torch.randn(L, F, generator=g, device="cuda:0")
    new = lambda dt, *s: torch.full(s, 7, dtype=dt, device="cuda:0")
    s, status = stream_ptr(), torch.zeros(1, dtype=torch.int32, device="cuda:0")
    idx, val, pre, feat = new(torch.int32, L, B, k), new(torch.float32, L, B, k), *(new(torch.float32, B, L, F) for _ in "ab")
    lib().call("clt_select_topk_export", z, b, idx, val, pre, feat, B, L, F, k, bf16, s)
    assert torch.equal(pre, (z.float() + b[:, None]).transpose(0, 1))
    want = new(torch.float32, B, L, F)
    lib().call("clt_scatter_features", idx, val, None, want, B, L, F, k, B * k, status, s)
    assert torch.equal(feat, want) and int(status) == 0
    assert bool((val[..., 1:] <= val[..., :-1]).all())
    idx2, val2 = torch.empty_like(idx), torch.empty_like(val)
    lib().call("clt_select_topk", z, b, idx2, val2, None, B, L, F, k, bf16, s)
    assert torch.equal(val.sort(-1)[0], val2.sort(-1)[0])
    if kind != "equal":
        lib().call("clt_scatter_features", idx2, val2, None, want, B, L, F, k, B * k, status, s)
        assert torch.equal(feat, want)


# rows that each kernel of clt_select_topk takes, with every value many times over
@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("L,B,F,k", [(2, 9, 256, 8), (2, 9, 1024, 100), (2, 17, 1024, 16), (3, 9, 4096, 32), (1, 5, 8192, 64),
                                     (2, 7, 20000, 33)])
def test_ties_give_a_selection_with_the_same_values(L, B, F, k, bf16):
    """Which of equal values are taken is open; that they are k different features with the k largest values is not."""
    g = torch.Generator(device="cuda:0").manual_seed(F + k)
    z = (torch.randn(L, B, F, generator=g, device="cuda:0") * 4).round() / 4
    z = z.to(torch.bfloat16 if bf16 else torch.float32)
    b = torch.zeros(L, F, device="cuda:0")
    new = lambda dt, *s: torch.full(s, 7, dtype=dt, device="cuda:0")
    s = stream_ptr()
    got = []
    for _ in "ab":
        idx, val, pre, feat = new(torch.int32, L, B, k), new(torch.float32, L, B, k), *(new(torch.float32, B, L, F) for _ in "ab")
        lib().call("clt_select_topk_export", z, b, idx, val, pre, feat, B, L, F, k, bf16, s)
        got.append((idx, val, feat))
    assert all(torch.equal(x, y) for x, y in zip(*got))
    idx, val, feat = got[0]
    assert torch.equal(val, z.float().topk(k).values) and bool((val > 0).all())
    assert torch.equal(z.float().gather(2, idx.long()), val)
    i = idx.long().sort(-1).values
    assert bool((i[..., 1:] > i[..., :-1]).all())
    want = torch.zeros(L, B, F, device="cuda:0").scatter_(2, idx.long(), val)
    assert torch.equal(feat, want.transpose(0, 1))
    idx2, val2 = torch.empty_like(idx), torch.empty_like(val)
    lib().call("clt_select_topk", z, b, idx2, val2, None, B, L, F, k, bf16, s)
    assert torch.equal(val2.sort(-1, descending=True).values, val)
