"""The streaming (Jump)ReLU kernels by themselves against float64, at the ends of their row groups and column blocks."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("scale", [0.3, 6.0], ids=["small", "saturating"])
@pytest.mark.parametrize("L,B,F", [(1, 1, 8), (2, 3, 1032), (3, 18, 1024), (2, 259, 88), (1, 2181, 264)])
def test_streaming_activation(L, B, F, scale, bf16):
    dev, T = "cuda:0", torch.bfloat16 if bf16 else torch.float32
    g = torch.Generator(device=dev).manual_seed(B * F)
    r = lambda *n: torch.randn(*n, generator=g, device=dev)
    z, gr, b = r(L, B, F).to(T), (r(L, B, F) * 0.1).to(T), r(L, F) * 0.1
    theta, norm = torch.rand(L, F, generator=g, device=dev) * 0.2, torch.rand(L, F, generator=g, device=dev) * scale
    c, lam, pal, bw = 0.7, 0.3, 0.05, 0.5
    s = stream_ptr()
    feat, dpre = torch.empty_like(z), torch.empty_like(z)
    fired, acc = torch.zeros(L, (F + 31) // 32, dtype=torch.int32, device=dev), torch.zeros(2, device=dev)
    dth, db, dn = (torch.zeros(L, F, device=dev) for _ in range(3))
    lib().call("clt_act_fwd", z, b, theta, norm, feat, fired, acc, c, 1, 1, B, L, F, bf16, s)
    lib().call("clt_act_bwd", gr, z, b, theta, norm, dpre, dth, db, dn, bw, lam, c, pal, 1, None, B, L, F, bf16, s)
    pre = z.float() + b[:, None]                       # the kernels' own fp32 sum decides every comparison
    f32 = torch.where((pre > theta[:, None]) & (pre > 0), pre, torch.zeros_like(pre))
    assert torch.equal(feat, f32.to(T))
    bits = (f32 > 0).any(dim=1)
    f = torch.arange(F, device=dev)
    got = ((fired[:, f // 32] >> (f % 32)) & 1).bool()
    assert torch.equal(got, bits)
    f, n = f32.double(), norm.double()[:, None] * c
    tw = torch.tanh(f * n)
    n_el = L * B * F
    # sums of n_el terms with about 1e-7 relative error each, added in fp32 groups of rows
    assert abs(float(acc[0]) - float(torch.relu(-pre.double()).sum())) <= 2e-6 * n_el ** 0.5 + 2e-6 * float(acc[0])
    assert abs(float(acc[1]) - float(tw.sum())) <= 2e-6 * float(tw.sum()) + 1e-6
    d1 = 1 - tw * tw
    gs = gr.double() + lam * d1 * n
    d = pre - theta[:, None]
    want = torch.where(pre >= 0, gs, torch.zeros_like(gs)) - pal * (pre < 0)
    tol = (2.0 ** -8 if bf16 else 1e-6) * want.abs() + 1e-6
    assert bool(((dpre.double() - want).abs() <= tol).all())
    rect = (d > -0.5 * bw) & ~(d > 0.5 * bw)
    close = lambda a, w, mag: bool(((a.double() - w).abs() <= 4e-6 * mag + 1e-6).all())
    assert close(db, want.sum(1), want.abs().sum(1))
    t = torch.where(rect, -theta.double()[:, None] / bw * gs, torch.zeros_like(gs))
    assert close(dth, t.sum(1), t.abs().sum(1))
    w = lam * d1 * c * f
    assert close(dn, w.sum(1), w.abs().sum(1))


@pytest.mark.parametrize("bf16", [0, 1])
def test_penalty_values_across_the_seam(bf16):
    """Single values of the streaming kernel's tanh on both sides of 0.7, where it leaves its polynomial for tanhf: one live
    feature, whose penalty is the whole sum.  The polynomial was fitted to 0.74 ulp, tanhf is specified to 2."""
    dev, T = "cuda:0", torch.bfloat16 if bf16 else torch.float32
    v = torch.cat([torch.logspace(-30, -2, 15), torch.linspace(0.02, 0.69, 68), torch.linspace(0.695, 0.705, 41),
                   torch.tensor([0.7, 0.71, 0.75, 1.0, 3.0, 9.0, 30.0, float("inf")])]).to(T).float().unique().to(dev)
    z = torch.full((v.numel(), 8), -1.0, dtype=T, device=dev)
    z[:, 3] = v.to(T)
    zero, one, acc = (torch.zeros(8, device=dev), torch.ones(8, device=dev), torch.zeros(v.numel(), 2, device=dev))
    feat = torch.empty(8, dtype=T, device=dev)
    for row, a in zip(z, acc):
        lib().call("clt_act_fwd", row, zero, None, one, feat, None, a, 1.0, 1, 0, 1, 1, 8, bf16, stream_ptr())
    want = torch.tanh(v.double())
    ulp = torch.ldexp(torch.ones_like(want), torch.frexp(want).exponent - 24)
    assert bool(((acc[:, 1].double() - want).abs() <= 2.0 * ulp).all())
    assert bool((acc[:, 0] == 0).all())
