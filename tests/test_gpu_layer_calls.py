"""One layer's encoder and decoder call against the launches that they stand for."""
import pytest
import torch

from crosslayer_transcoder_b200._lib import lib, stream_ptr


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("B,D,F", [(1, 64, 16384), (129, 72, 136), (257, 768, 10000), (300, 200, 264)])
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


def test_parts_fill_whole_rounds():
    """bf16 parts of a decoder chain are cut so that the last round of the chip is not begun for a few of them."""
    for B, D, K in ((257, 768, 120000), (257, 768, 50000), (100, 1024, 30000), (40, 256, 64000)):
        parts = lib().query("clt_decoder_dense_parts", B, 1, D, K, 0, 1, 148)
        tiles = -(-B // 128) * -(-D // 256)
        rounds = -(-parts * tiles // 148)
        assert parts > 1 and 1 <= rounds <= 4 and parts * tiles > 0.8 * rounds * 148, (B, D, K, parts)
