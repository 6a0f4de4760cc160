"""The launches that stand for several small tensor operations of a step."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,code", [(torch.float16, 1), (torch.bfloat16, 2)])
@pytest.mark.parametrize("n", [1, 255, 256, 9216 + 3])
def test_cast_stats(n, dtype, code):
    src = [torch.randn(n, device="cuda:0").to(dtype) for _ in range(4)]
    out = torch.empty(4, n, device="cuda:0")
    lib().call("clt_cast_stats", *src, code, out, n, stream_ptr())
    assert torch.equal(out, torch.stack([t.float() for t in src]))


@pytest.mark.parametrize("sizes", [(1, 0, 0, 0), (3, 700001, None, 256), (None, None, None, 5), (64, 64, 64, 64)])
def test_zero4(sizes):
    arrays = [None if n is None else torch.ones(n + 1, device="cuda:0") for n in sizes]
    args = [x for t, n in zip(arrays, sizes) for x in (t, n or 0)]
    lib().call("clt_zero4", *args, stream_ptr())
    for t, n in zip(arrays, sizes):
        if t is not None:
            assert not t[:n].any() and float(t[n]) == 1.0       # and nothing behind the end
