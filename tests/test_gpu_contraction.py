"""The contraction kernels by themselves, through the C entry points, against float64 products at the sizes where
tiles, k-steps and vector loads end."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


def _rand(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda:0")


def _close(got, want, mag, k):
    """fp32: |error| of a k-long fma chain is at most k 2^-24 times the sum of the products' magnitudes; random signs
    make it about its square root."""
    bound = 2.0 ** -24 * (4.0 + 2.0 * k ** 0.5) * mag + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound).max())


# tiles are 128 x 128 and 64 x 64 (fewer than one large tile per SM), k-steps 16; odd sizes have no 16-byte rows
@pytest.mark.parametrize("L,B,D,F", [(1, 1, 1, 1), (2, 63, 17, 65), (3, 129, 64, 200), (1, 64, 15, 64), (12, 513, 64, 777),
                                     (4, 770, 48, 1027), (6, 640, 20, 1024)])
def test_fp32_products(L, B, D, F):
    g = torch.Generator(device="cuda:0").manual_seed(L * 1000 + F)
    s = stream_ptr()
    x, W = _rand(g, L, B, D), _rand(g, L, D, F)
    z = torch.empty(L, B, F, device="cuda:0")
    lib().call("clt_encoder_fwd_store", x, W, z, B, L, D, F, 0, None, s)
    _close(z, x.double() @ W.double(), x.double().abs() @ W.double().abs(), D)
    # crosslayer decoder: both operands over the concatenated sources, then its two gradients
    P = L * (L + 1) // 2
    feat, Wd, b = _rand(g, L, B, F), _rand(g, P, F, D), _rand(g, L, D)
    recon = torch.empty(B, L, D, device="cuda:0")
    lib().call("clt_decoder_dense_fwd", feat, Wd, b, recon, B, L, D, F, 1, 0, None, s)
    for t in range(L):
        blk = Wd[t * (t + 1) // 2:(t + 1) * (t + 2) // 2].double()
        fd = feat[:t + 1].double()
        _close(recon[:, t], torch.einsum("sbf,sfd->bd", fd, blk) + b[t].double(),
               torch.einsum("sbf,sfd->bd", fd.abs(), blk.abs()) + b[t].double().abs(), (t + 1) * F)
    dr = _rand(g, L, B, D)
    dW = torch.empty(P, F, D, device="cuda:0")
    lib().call("clt_decoder_dense_bwd_dw", feat, dr, dW, None, None, B, L, D, F, 1, 0, None, s)
    df = torch.empty(L, B, F, device="cuda:0")
    lib().call("clt_decoder_dense_bwd_dfeat_raw", dr, Wd, df, B, L, D, F, 1, 0, None, s)
    for t in range(L):
        for q in range(t + 1):
            p = t * (t + 1) // 2 + q
            _close(dW[p], feat[q].double().t() @ dr[t].double(), feat[q].double().abs().t() @ dr[t].double().abs(), B)
    for q in range(L):
        want = sum(dr[t].double() @ Wd[t * (t + 1) // 2 + q].double().t() for t in range(q, L))
        mag = sum(dr[t].double().abs() @ Wd[t * (t + 1) // 2 + q].double().abs().t() for t in range(q, L))
        _close(df[q], want, mag, (L - q) * D)
