"""One layer's encoder and decoder call against the launches that they stand for."""
import random

import pytest
import torch

from crosslayer_transcoder_b200 import synthetic
from crosslayer_transcoder_b200._lib import DTYPE_CODE, lib, stream_ptr

from helpers import build_module, spec_inputs


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("B,D,F", [(1, 8, 8), (1, 64, 16384), (3, 64, 248), (129, 72, 136), (257, 768, 10000), (300, 200, 264)])
def test_encoder_layer_is_bit_equal(B, D, F, bias):
    g = torch.Generator(device="cuda:0").manual_seed(F)
    x, W = torch.randn(B, D, generator=g, device="cuda:0"), torch.randn(1, D, F, generator=g, device="cuda:0").bfloat16()
    b = torch.randn(1, F, generator=g, device="cuda:0") if bias else None
    xn, z = (torch.empty(1, B, n, dtype=torch.bfloat16, device="cuda:0") for n in (D, F))
    got, want = torch.empty(B, F, device="cuda:0"), torch.empty(B, F, device="cuda:0")
    s, status = stream_ptr(), torch.zeros(1, dtype=torch.int32, device="cuda:0")
    lib().call("clt_prep_acts", x, 0, None, None, xn, 1, B, 1, D, s)
    lib().call("clt_encoder_fwd_store", xn, W, z, B, 1, D, F, 1, status, s)
    lib().call("clt_export_blf", z, b, want, B, 1, F, 1, s)
    lib().call("clt_encoder_layer_fwd", x, 0, W, b, xn, got, B, D, F, status, s)
    assert torch.equal(got, want) and int(status) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lead", [(1,), (7,), (1, 1), (2, 3), (5, 31), (3, 2, 9)])
def test_encoder_layer_through_the_module(lead, dtype):
    """Leading dimensions, 16-bit and strided inputs of ``encoder(x, layer=i)``, whose layers end inside a tile: two
    kernels, and the bits of the three launches."""
    L, D, F = 3, 72, 264
    spec = synthetic.WorkloadSpec("el", L, D, F, 8, "relu", True, True, rank_u=8, n_outlier=1)
    batch, w, la = spec_inputs(spec)
    mod = build_module(spec, w, torch.device("cuda:0"), last_active=la)
    enc, g = mod.model.encoder, torch.Generator(device="cuda:0").manual_seed(len(lead))
    wide = torch.randn(*lead, L, D, generator=g, device="cuda:0").to(dtype)
    B = wide[..., 0, 0].numel()
    for layer in range(L):
        x = wide[..., layer, :]                             # rows L * D apart
        assert x.is_contiguous() == (B == 1)
        n0 = mod._engine.launches
        got = enc(x, layer=layer)
        assert mod._engine.launches == n0 + 2 and got.shape == (*lead, F) and got.dtype == torch.float32
        xn, z = (torch.empty(1, B, n, dtype=torch.bfloat16, device="cuda:0") for n in (D, F))
        want, s, st = torch.empty(B, F, device="cuda:0"), stream_ptr(), mod._engine.status
        lib().call("clt_prep_acts", x.contiguous(), DTYPE_CODE[dtype], None, None, xn, 1, B, 1, D, s)
        lib().call("clt_encoder_fwd_store", xn, enc.W[layer].bfloat16().contiguous(), z, B, 1, D, F, 1, st, s)
        lib().call("clt_export_blf", z, enc.b[layer].detach(), want, B, 1, F, 1, s)
        assert torch.equal(got.reshape(B, F), want) and int(st) == 0


def test_parts_of_a_chain_are_no_longer_than_half_a_share():
    """A bf16 accumulator's error goes with the length of its chain, so whatever a plan fits the parts to, it does not
    make them longer (csrc/gemm_dense.cu; 64 features to a block, 128 x 256 tiles)."""
    rng, cut = random.Random(5), 0
    for _ in range(2000):
        L, cross = rng.randint(1, 12), rng.randint(0, 1)
        B, D, F = (int(10 ** rng.uniform(*e)) for e in ((0.7, 3.2), (1.8, 3.36), (2.4, 5.1)))
        blocks = [-(-F // 64) * (z + 1 if cross else 1) for z in range(L)]
        half = max(8, -(-sum(blocks) * -(-B // 128) * -(-D // 256) // (2 * 148)))
        parts = lib().query("clt_decoder_dense_parts", B, L, D, F, cross, 1, 148)
        cut += parts > 0
        assert parts == 0 or parts >= sum(-(-n // half) for n in blocks), (B, L, D, F, cross, parts)
    assert cut > 500
