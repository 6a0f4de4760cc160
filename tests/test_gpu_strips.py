"""Input preparation, loss forward and loss backward against float64, at the ends of their column blocks and row strips,
for rows that are and are not multiples of 8 columns."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import DTYPE_CODE, lib, stream_ptr

pytestmark = pytest.mark.gpu


# 256 columns to a CTA, strips of 8 to 64 rows (256 in fp32, where that gives two CTAs to an SM), 2 or 4 rows in flight per
# thread; long batches of narrow rows
@pytest.mark.parametrize("out", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,L,D", [(1, 1, 8), (9, 3, 88), (31, 2, 128), (65, 5, 72), (300, 2, 264), (2049, 1, 16),
                                   (33, 3, 20), (31, 2, 20), (9, 12, 100), (2305, 12, 768),
                                   (32769, 1, 248), (32768, 1, 248)])
def test_against_float64(B, L, D, dtype, out):
    g = torch.Generator(device="cuda:0").manual_seed(B + D)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda:0")
    batch, mu, sd = r(B, 2, L, D).to(dtype), 0.3 * r(L, D), 0.5 + r(L, D).abs()
    recon, aux, s, code, bf16 = r(B, L, D), 0.1 * r(B, L, D), stream_ptr(), DTYPE_CODE[dtype], int(out == torch.bfloat16)
    xn = torch.empty(L, B, D, dtype=out, device="cuda:0")
    lib().call("clt_prep_input", batch, code, mu, sd, xn, bf16, B, L, D, s)
    # the subtraction and the division of the same fp32 values, rounded once more to the output's type
    assert torch.equal(xn, ((batch[:, 0].float() - mu) / sd).to(out).transpose(0, 1))
    y = (batch[:, 1].double() - mu.double()) / sd.double()
    diff = recon.double() - y
    n, scale = float(B * L * D), 1 / 32
    for a in (None, aux):
        acc = torch.zeros(2, device="cuda:0")
        lib().call("clt_loss_fwd", recon, a, batch, code, mu, sd, acc, B, L, D, s)
        want = torch.stack([(diff ** 2).sum(), ((aux.double() + diff) ** 2).sum() if a is not None else diff.new_zeros(())])
        assert torch.allclose(acc.double(), want, rtol=1e-5)
        dr, da = torch.empty_like(xn), torch.empty_like(xn)
        db, gs = torch.zeros(L, D, device="cuda:0"), torch.full((1,), 3.0, device="cuda:0")
        lib().call("clt_loss_bwd", recon, a, batch, code, mu, sd, gs, scale if a is not None else 0.0, dr,
                   da if a is not None else None, bf16, db, B, L, D, s)
        ga = 2 * (aux.double() + diff) * scale * 3.0 / n if a is not None else torch.zeros_like(diff)
        gr = 2 * diff * 3.0 / n + ga
        # a few fp32 roundings of the terms (y, diff and the products), then the output's: half a bf16 step is 2^-8 of a
        # value, and no gradient is larger than its terms' magnitudes with the auxiliary share on top
        tol = (2.0 ** -8 if bf16 else 0.0) + 2.0 ** -20
        mag = recon.double().abs() + batch[:, 1].double().abs() / sd + mu.abs() / sd + aux.abs()
        mag = 2 * (1 + scale) * mag * 3.0 / n
        assert bool(((dr.transpose(0, 1).double() - gr).abs() <= tol * mag).all())
        if a is not None:
            assert bool(((da.transpose(0, 1).double() - ga).abs() <= tol * mag).all())
        assert bool(((db.double() - (gr + ga).sum(0)).abs() <= 2.0 ** -20 * 2 * mag.sum(0)).all())


def test_more_rows_than_a_grid_of_short_strips():
    """600000 rows: strips of 8 would be more than a grid has in y.  Rows of one constant, so that the sums are known."""
    B, L, D, s = 600000, 1, 8, stream_ptr()
    batch, mu, sd = torch.full((B, 2, L, D), 3.0, device="cuda:0"), torch.ones(L, D, device="cuda:0"), \
        torch.full((L, D), 2.0, device="cuda:0")
    recon, aux = torch.full((B, L, D), 1.5, device="cuda:0"), torch.full((B, L, D), -1.0, device="cuda:0")
    xn, acc = torch.empty(L, B, D, device="cuda:0"), torch.zeros(2, device="cuda:0")
    lib().call("clt_prep_input", batch, 0, mu, sd, xn, 0, B, L, D, s)
    assert bool((xn == 1.0).all())
    lib().call("clt_loss_fwd", recon, aux, batch, 0, mu, sd, acc, B, L, D, s)
    # diff = 0.5, aux + diff = -0.5; fp32 sums of 4.8 million equal terms over 148 x 8 x 256 threads
    assert torch.allclose(acc, torch.full_like(acc, 0.25 * B * L * D), rtol=1e-5)
    dr, da, db = torch.empty_like(xn), torch.empty_like(xn), torch.zeros(L, D, device="cuda:0")
    lib().call("clt_loss_bwd", recon, aux, batch, 0, mu, sd, None, 0.25, dr, da, 0, db, B, L, D, s)
    n = B * L * D
    assert torch.allclose(da, torch.full_like(da, -0.25 / n), rtol=1e-6)
    assert torch.allclose(dr, torch.full_like(dr, 0.75 / n), rtol=1e-6)
    assert torch.allclose(db, torch.full_like(db, 0.5 / D), rtol=1e-4)


@pytest.mark.parametrize("B", [256, 300, 512])
def test_fp32_bias_gradient_has_one_order_up_to_two_strips(B):
    """A batch that does not start on 16 bytes goes to the kernel with 4 columns a thread: the same bits."""
    L, D, s = 16, 2368 * (2 if B == 256 else 1), stream_ptr()
    assert -(-L * D // 256) * -(-B // 256) >= 2 * 148
    g = torch.Generator(device="cuda:0").manual_seed(B)
    r = lambda *n: torch.randn(*n, generator=g, device="cuda:0")
    mu, sd, recon, aux = 0.3 * r(L, D), 0.5 + r(L, D).abs(), r(B, L, D), r(B, L, D)
    store = r(B * 2 * L * D + 1).half()
    for a in (None, aux):
        got = []
        for off in (0, 1):
            batch = store[off:off + B * 2 * L * D] if off else store[1:].clone()
            assert (batch.data_ptr() % 16 != 0) == bool(off)
            dr, da, db = torch.empty(L, B, D, device="cuda:0"), torch.empty(L, B, D, device="cuda:0"), torch.zeros(L, D, device="cuda:0")
            lib().call("clt_loss_bwd", recon, a, batch, 1, mu, sd, None, 0.03 if a is not None else 0.0, dr,
                       da if a is not None else None, 0, db, B, L, D, s)
            got.append((dr, db, da if a is not None else dr))
        assert all(torch.equal(x, y) for x, y in zip(*got))


# one CTA's columns of a row and more, rows narrower than a CTA (powers of two and not), 16-byte rows and others
@pytest.mark.parametrize("B,L,D", [(1, 1, 1), (5, 1, 4), (1001, 1, 7), (257, 1, 16), (3000, 1, 100), (70000, 2, 8), (33, 3, 33),
                                   (129, 1, 1020), (7, 2, 512), (9, 1, 1028), (300, 12, 768)])
@pytest.mark.parametrize("offset", [0, 1])
def test_destandardize(B, L, D, offset):
    g = torch.Generator(device="cuda:0").manual_seed(B + D)
    flat = torch.randn(B * L * D + offset, generator=g, device="cuda:0")[offset:]       # (a base that is not on 16 bytes)
    mu, sd = torch.randn(L, D, generator=g, device="cuda:0"), torch.rand(L, D, generator=g, device="cuda:0") + 0.1
    out = torch.full((B * L * D + 8,), float("nan"), device="cuda:0")
    lib().call("clt_destandardize", flat, mu, sd, out, B, L, D, stream_ptr())
    want = flat.view(B, L, D).double() * sd.double() + mu.double()
    # one rounding of the exact value
    assert bool(((out[:-8].view(B, L, D).double() - want).abs() <= 2.0 ** -24 * 1.001 * want.abs() + 1e-45).all())
    assert bool(out[-8:].isnan().all())                                                 # and nothing behind the end
