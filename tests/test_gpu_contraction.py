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


# few output tiles and long chains: parts of the contraction axis run side by side; the last shape stays whole
@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("L,B,D,F,cross", [(1, 257, 768, 30000, 0), (1, 1, 64, 4096, 0), (3, 65, 264, 2504, 1),
                                           (5, 130, 64, 1368, 1), (2, 300, 320, 5000, 0), (12, 1000, 64, 512, 1),
                                           (1, 300, 1024, 496, 0)])
def test_split_decoder(L, B, D, F, cross, bf16):
    dev = "cuda:0"
    parts = lib().query("clt_decoder_dense_parts", B, L, D, F, cross, bf16, 0)
    assert (parts == 0) == (F == 496)
    g = torch.Generator(device=dev).manual_seed(F)
    P = L * (L + 1) // 2 if cross else L
    dt = torch.bfloat16 if bf16 else torch.float32
    feat, W, b = _rand(g, L, B, F).to(dt), _rand(g, P, F, D).to(dt), _rand(g, L, D)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    whole, split, again = (torch.empty(B, L, D, device=dev) for _ in range(3))
    lib().call("clt_decoder_dense_fwd", feat, W, b, whole, B, L, D, F, cross, bf16, status, stream_ptr())
    n = max(parts, 1) * B * D                               # as much as the library asks for, and no more
    for out in (split, again):
        ws = torch.full((n,), float("nan"), device=dev)     # every partial sum that is read was written
        lib().call("clt_decoder_dense_fwd_ws", feat, W, b, out, ws, n, B, L, D, F, cross, bf16, status, stream_ptr())
    assert torch.equal(split, again)
    for less in (n - 1, B * D - 1):                         # too little scratch: the unsplit chains
        small = torch.empty_like(whole)
        lib().call("clt_decoder_dense_fwd_ws", feat, W, b, small, ws, less, B, L, D, F, cross, bf16, status, stream_ptr())
        assert torch.equal(small, whole)
    assert parts or torch.equal(split, whole)
    assert int(status) == 0
    for t in range(L):
        src = slice(0, t + 1) if cross else slice(t, t + 1)
        blk = W[t * (t + 1) // 2:(t + 1) * (t + 2) // 2] if cross else W[t:t + 1]
        fd, wd = feat[src].double(), blk.double()
        want = torch.einsum("sbf,sfd->bd", fd, wd) + b[t].double()
        mag = torch.einsum("sbf,sfd->bd", fd.abs(), wd.abs()) + b[t].double().abs()
        _close(split[:, t], want, mag, fd.shape[0] * F)


def _takes_pairs(M, N, Kseg, nz):
    """csrc/gemm_tc.cuh, use_pair"""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = -(-N // 256) * nz
    single, pairs = -(-M // 128) * n, -(-M // 256) * n
    rounds, pair_rounds = -(-single // sms), -(-pairs // (sms // 2))
    return Kseg > 9 * 64 and pairs >= sms // 2 and pairs * 16 <= single * 9 and pair_rounds * 9 <= rounds * 10


# 128-row tiles and 256-row tiles of CTA pairs (`pairs`: which of encoder, feature gradient, decoder, decoder weight and
# encoder weight gradient take them), with ragged ends in every axis; contractions of a few elements, of one stage, of
# more stages than the ring holds; pairs whose second CTA has part of its 128 rows (1999) or none (2049, one row in the
# first), over several segments that each end inside a stage
@pytest.mark.parametrize("L,B,D,F,pairs", [(2, 2049, 264, 2056, ""), (1, 4000, 776, 3000, "ef"), (3, 1281, 8, 4104, "w"),
                                           (3, 1100, 64, 2312, ""), (2, 300, 520, 1032, ""), (12, 256, 256, 2048, ""),
                                           (3, 1999, 1016, 2008, "efdwx"), (3, 2049, 1016, 2008, "efdwx"),
                                           (4, 2049, 776, 1000, "efdw"), (2, 1083, 1072, 7840, "w")])
def test_bf16_products(L, B, D, F, pairs):
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(B)
    s, st = stream_ptr(), torch.zeros(1, dtype=torch.int32, device=dev)
    bf = torch.bfloat16
    P = L * (L + 1) // 2
    # the sizes are there for the forms that they take: a change of the rule has to bring others
    forms = {"e": (B, F, D, L), "f": (B, F, D, L), "d": (B, D, F, L), "w": (F, D, B, P), "x": (D, F, B, L)}
    assert "".join(k for k, m in forms.items() if _takes_pairs(*m)) == pairs
    x, W, feat, dr = (_rand(g, *n).to(bf) for n in ((L, B, D), (L, D, F), (L, B, F), (L, B, D)))
    Wd, b = _rand(g, P, F, D).to(bf), _rand(g, L, D)

    def rounded(got, want, mag, k):
        """a bf16 result is its fp32 sum rounded once more"""
        bound = 2.0 ** -24 * (4.0 + 2.0 * k ** 0.5) * mag + 2.0 ** -8 * want.abs() + 1e-30
        assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound).max())

    z, df = torch.empty(L, B, F, device=dev, dtype=bf), torch.empty(L, B, F, device=dev, dtype=bf)
    lib().call("clt_encoder_fwd_store", x, W, z, B, L, D, F, 1, st, s)
    lib().call("clt_decoder_dense_bwd_dfeat_raw", dr, Wd, df, B, L, D, F, 1, 1, st, s)
    recon = torch.empty(B, L, D, device=dev)
    lib().call("clt_decoder_dense_fwd", feat, Wd, b, recon, B, L, D, F, 1, 1, st, s)
    dW, dWe = torch.empty(P, F, D, device=dev), torch.empty(L, D, F, device=dev)
    lib().call("clt_decoder_dense_bwd_dw", feat, dr, dW, None, None, B, L, D, F, 1, 1, st, s)
    lib().call("clt_encoder_dense_bwd_dw", x, feat, dWe, B, L, D, F, 1, st, s)
    assert int(st) == 0
    mm = lambda a, w: (a.double() @ w.double(), a.double().abs() @ w.double().abs())
    for l in range(L):
        rounded(z[l], *mm(x[l], W[l]), D)
        _close(dWe[l], *mm(x[l].t(), feat[l]), B)
        blk = Wd[l * (l + 1) // 2:(l + 1) * (l + 2) // 2].reshape(-1, D)
        want, mag = mm(feat[:l + 1].transpose(0, 1).reshape(B, -1), blk)
        _close(recon[:, l], want + b[l].double(), mag + b[l].double().abs(), (l + 1) * F)
        for q in range(l + 1):
            _close(dW[l * (l + 1) // 2 + q], *mm(feat[q].t(), dr[l]), B)
        blk = torch.cat([Wd[t * (t + 1) // 2 + l] for t in range(l, L)], dim=1)
        rounded(df[l], *mm(dr[l:].transpose(0, 1).reshape(B, -1), blk.t()), (L - l) * D)


# the (Jump)ReLU and row-coefficient epilogues on the large tiles: 128 x 128 (encoder; per-layer feature gradient; weight
# gradient) and 128 x 64 (crosslayer feature gradient), with and without 16-byte rows
@pytest.mark.parametrize("L,B,D,F,cross", [(2, 1100, 648, 1160, 1), (2, 1101, 645, 1163, 0)])
def test_fp32_fused_epilogues(L, B, D, F, cross):
    dev, s = "cuda:0", stream_ptr()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sms <= -(-B // 128) * -(-F // 128) * L < 8 * sms     # the large tiles' range of sizes (csrc/gemm_simt.cuh)
    g = torch.Generator(device=dev).manual_seed(F)
    P = L * (L + 1) // 2 if cross else L
    x, W, b = _rand(g, L, B, D), _rand(g, L, D, F) * D ** -0.5, _rand(g, L, F) * 0.1
    theta, norm = (torch.rand(L, F, generator=g, device=dev) * 0.3 for _ in range(2))
    c, lam, pal, bw = 0.7, 0.3, 0.05, 0.5
    z, feat, dpre = (torch.empty(L, B, F, device=dev) for _ in range(3))
    fired, acc = torch.zeros(L, (F + 31) // 32, dtype=torch.int32, device=dev), torch.zeros(2, device=dev)
    lib().call("clt_encoder_fwd_act", x, W, b, theta, norm, z, feat, fired, acc, c, 1, 1, B, L, D, F, 0, None, s)
    _close(z, x.double() @ W.double(), x.double().abs() @ W.double().abs(), D)
    pre = z + b[:, None]                               # the kernel's own fp32 sum decides every comparison
    f32 = torch.where((pre > theta[:, None]) & (pre > 0), pre, torch.zeros_like(pre))
    assert torch.equal(feat, f32)
    i = torch.arange(F, device=dev)
    assert torch.equal(((fired[:, i // 32] >> (i % 32)) & 1).bool(), (f32 > 0).any(dim=1))
    f, n = f32.double(), norm.double()[:, None] * c
    tw = torch.tanh(f * n)
    # sums of n terms with about 1e-7 relative error each, added in fp32 groups
    assert abs(float(acc[0]) - float(torch.relu(-pre.double()).sum())) <= 4e-6 * float(acc[0])
    assert abs(float(acc[1]) - float(tw.sum())) <= 4e-6 * float(tw.sum())

    dr, Wd = _rand(g, L, B, D) * 0.1, _rand(g, P, F, D) * D ** -0.5
    dth, db, dn = (torch.zeros(L, F, device=dev) for _ in range(3))
    lib().call("clt_decoder_dense_bwd_dfeat", dr, Wd, z, b, theta, norm, dpre, dth, db, dn, bw, lam, c, pal, 1, None, B, L,
               D, F, cross, 0, None, s)
    pair = lambda t, q: t * (t + 1) // 2 + q if cross else t
    targets = lambda q: range(q, L) if cross else (q,)
    gr, mag = (torch.stack([sum(fn(dr[t].double()) @ fn(Wd[pair(t, q)].double()).t() for t in targets(q))
                            for q in range(L)]) for fn in (lambda v: v, torch.abs))
    err = 2.0 ** -24 * (4.0 + 2.0 * (L * D) ** 0.5) * mag       # of the product, as in _close
    d1 = 1 - tw * tw
    gs = gr + lam * d1 * n
    want = torch.where(pre >= 0, gs, torch.zeros_like(gs)) - pal * (pre < 0)
    assert bool(((dpre.double() - want).abs() <= err + 1e-6 * want.abs() + 1e-6).all())
    close = lambda a, w, e: bool(((a.double() - w.sum(1)).abs() <= e.sum(1) + 4e-6 * w.abs().sum(1) + 1e-6).all())
    d = pre - theta[:, None]
    rect = (d > -0.5 * bw) & ~(d > 0.5 * bw)
    slope = theta.double()[:, None] / bw
    assert close(db, want, err)
    assert close(dth, torch.where(rect, -slope * gs, torch.zeros_like(gs)), slope * err)
    assert close(dn, lam * d1 * c * f, torch.zeros_like(f))

    coef, dW = _rand(g, L, F) * 0.1, torch.empty(P, F, D, device=dev)
    lib().call("clt_decoder_dense_bwd_dw", feat, dr, dW, coef, Wd, B, L, D, F, cross, 0, None, s)
    for t in range(L):
        for q in range(t + 1) if cross else (t,):
            add = coef[q].double()[:, None] * Wd[pair(t, q)].double()
            _close(dW[pair(t, q)], f[q].t() @ dr[t].double() + add, f[q].t() @ dr[t].double().abs() + add.abs(), B)
