"""The per-layer scans of the counting sort and of the dead-feature list at the ends of their rounds (8192 features) and
warps (256)."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,F", [(1, 1), (2, 31), (3, 257), (2, 8191), (1, 8192), (2, 8193), (3, 20000)])
def test_scans(L, F):
    g = torch.Generator(device="cuda:0").manual_seed(F)
    s, status = stream_ptr(), torch.zeros(1, dtype=torch.int32, device="cuda:0")
    npl = 3 * F + 5
    idx = torch.randint(0, F, (L, npl), generator=g, device="cuda:0", dtype=torch.int32)
    val = torch.rand(L, npl, generator=g, device="cuda:0") + 0.1
    val[:, ::7] = 0                                                     # unused slots
    new = lambda *shape: torch.full(shape, -1, dtype=torch.int32, device="cuda:0")
    col, cur, ent, lst, nd = new(L, F + 1), new(L, F), new(L, npl), new(L, F), new(L)
    lib().call("clt_csc_build", idx, val, col, cur, ent, npl, L, F, status, s)
    dead = (torch.rand(L, F, generator=g, device="cuda:0") < 0.3).to(torch.uint8)
    lib().call("clt_dead_compact", dead, lst, nd, L, F, s)
    for l in range(L):
        count = torch.bincount(idx[l][val[l] != 0].long(), minlength=F)
        assert int(col[l, 0]) == 0 and torch.equal(col[l, 1:].long(), count.cumsum(0))
        assert torch.equal(cur[l], col[l, 1:])                          # the fill moved every cursor to its end
        f = idx[l][ent[l, :int(col[l, -1])].long()].long()
        assert torch.equal(f, f.sort()[0])
        want = dead[l].nonzero().flatten()
        assert int(nd[l]) == want.numel() and torch.equal(lst[l, :want.numel()].long(), want)
    assert int(status) == 0
