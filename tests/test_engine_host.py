"""What the engine checks on the host before it launches anything; on the CPU with the library replaced by a recorder."""
import copy
import pickle

import pytest
import torch

from crosslayer_transcoder_b200 import _lib, engine, synthetic
from crosslayer_transcoder_b200._lib import CltError

from helpers import build_module, spec_inputs

KINDS = ["jumprelu", "topk", "batchtopk", "perlayer_batchtopk"]


class _OnDevice(torch.Tensor):
    """A CPU tensor that says it is on the GPU."""
    is_cuda = True


class _Calls:
    """In the place of the library: records what would be launched."""

    def __init__(self):
        self.names, self.args = [], []

    def check_device(self):
        pass

    def call(self, name, *args):
        self.names.append(name)
        self.args.append(args)

    def query(self, name, *args):
        return 0


@pytest.fixture
def calls(monkeypatch):
    rec = _Calls()
    monkeypatch.setattr(engine, "lib", lambda: rec)
    monkeypatch.setattr(engine, "stream_ptr", lambda: 0)
    return rec


def _module(kind, dev, cross=True):
    spec = synthetic.WorkloadSpec("order", 3, 64, 128, 40, kind, cross, False, rank_u=8, n_outlier=1, k=4, k_aux=0)
    batch, w, la = spec_inputs(spec)
    mod = build_module(spec, w, dev, last_active=la)
    batch = batch.to(dev)
    mod.model.initialize_standardizers(batch)
    return mod, batch


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("first,second", [(40, 31), (31, 40), (40, 40)])
def test_earlier_step_is_refused_before_any_launch(kind, first, second, calls):
    """The backward half of a step reads the buffers that its forward half wrote; another step's forward now has them."""
    mod, batch = _module(kind, "cpu")
    batch = batch.as_subclass(_OnDevice)
    l1 = mod.training_step(batch[:first], 1)
    mod.training_step(batch[:second], 2)
    n = len(calls.names)
    with pytest.raises(CltError, match="overwritten"):
        l1.backward()
    assert len(calls.names) == n


@pytest.mark.parametrize("kind", KINDS)
def test_step_that_failed_half_way_leaves_none_to_go_backward(kind, calls):
    """The buffers belong to the step that began to write them, whether it came to its end or not."""
    mod, batch = _module(kind, "cpu")
    batch = batch.as_subclass(_OnDevice)
    l1 = mod.training_step(batch, 1)
    calls.call = lambda name, *args: (_ for _ in ()).throw(CltError("launch failed"))
    with pytest.raises(CltError, match="launch failed"):
        mod.training_step(batch[:31], 2)
    with pytest.raises(CltError, match="overwritten"):
        l1.backward()


@pytest.mark.parametrize("kind", ["jumprelu", "topk"])
@pytest.mark.parametrize("replace", ["one", "all"])
def test_replaced_decoder_blocks_are_not_answered_with_the_old_ones(kind, replace, calls):
    mod, batch = _module(kind, "cpu")
    acts = batch[:, 0].as_subclass(_OnDevice)
    dec = mod.model.decoder
    with torch.no_grad():
        mod(acts)
        if replace == "all":
            dec.load_state_dict({k: v + 1 for k, v in dec.state_dict().items()}, assign=True)
        else:
            dec.W_1 = torch.nn.Parameter(dec.W_1.detach() + 1)
        with pytest.raises(CltError, match="decoder block"):
            mod(acts)


@pytest.mark.parametrize("precision", ["bf16", "fp32"])
@pytest.mark.parametrize("tokens", [5, 200])
@pytest.mark.parametrize("layer", [-1, 3, 7])
def test_layers_that_do_not_exist_reach_the_library_as_null(layer, tokens, precision, calls):
    """(which it refuses) whatever form of the call the size takes."""
    mod, _ = _module("relu", "cpu", cross=False)
    mod.precision = precision
    rand = lambda n: torch.randn(tokens, n).as_subclass(_OnDevice)
    for part, x, name in ((mod.model.encoder, rand(64), "encoder"), (mod.model.decoder, rand(128), "decoder")):
        del calls.names[:], calls.args[:]
        part(x, layer=layer)
        i, = [i for i, n in enumerate(calls.names) if name in n]
        assert any(isinstance(a, torch.Tensor) and a.dim() > 2 and a.data_ptr() == 0 for a in calls.args[i])


# the lines of the rule: width of a step, lengths and batches from which one sweep is the faster form
@pytest.mark.parametrize("F,k,tokens,one", [(248, 64, 900, True), (256, 256, 5, True), (260, 8, 5, False), (512, 16, 1400, False),
                                            (512, 16, 1300, True), (520, 16, 700, False), (520, 16, 600, True),
                                            (520, 32, 5, False), (520, 65, 1400, True), (1024, 64, 1400, True),
                                            (1032, 16, 1400, False), (2552, 16, 1400, False), (2560, 64, 1400, True),
                                            (2568, 64, 1400, True), (8200, 64, 5, True), (8192, 257, 5, False)])
def test_forms_of_the_topk_inference(F, k, tokens, one, calls):
    L, D = 3, 64
    spec = synthetic.WorkloadSpec("forms", L, D, F, 16, "topk", False, True, rank_u=8, n_outlier=1, k=k, k_aux=0)
    batch, w, la = spec_inputs(spec)
    mod = build_module(spec, w, "cpu", last_active=la)
    mod.model.initialize_standardizers(batch)
    with torch.no_grad():
        mod(torch.zeros(tokens, L, D).as_subclass(_OnDevice))
    three = ["clt_export_blf", "clt_select_topk", "clt_scatter_features"]
    got = [n for n in calls.names if n in three or n == "clt_select_topk_export"]
    assert got == (["clt_select_topk_export"] if one else three)


@pytest.mark.parametrize("how", [copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))], ids=["deepcopy", "pickle"])
def test_module_that_has_run_can_be_copied(how, monkeypatch):
    """Weight averaging copies a module, spawned workers pickle it: the engine holds nothing of the loaded library."""
    monkeypatch.setattr(_lib._Lib, "check_device", lambda self: None)
    monkeypatch.setattr(_lib._Lib, "call", lambda self, name, *args: None)
    monkeypatch.setattr(engine, "stream_ptr", lambda: 0)
    mod, batch = _module("topk", "cpu")
    with torch.no_grad():
        mod(batch[:, 0].as_subclass(_OnDevice))
    other = how(mod)
    for a, b in zip(mod.parameters(), other.parameters()):
        assert torch.equal(a, b) and a.data_ptr() != b.data_ptr()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_last_step_still_goes_backward(kind):
    mod, batch = _module(kind, "cuda:0")
    mod.training_step(batch[:31], 1).backward()
    want = [p.grad.clone() for p in mod.parameters()]
    mod.zero_grad()
    l1 = mod.training_step(batch, 1)
    l2 = mod.training_step(batch[:31], 1)
    with pytest.raises(CltError, match="overwritten"):
        l1.backward()
    l2.backward()
    mod._engine.check_status("step order")
    for p, w in zip(mod.parameters(), want):
        # sums by atomics come in another order
        assert torch.allclose(p.grad, w, rtol=1e-4, atol=1e-6 * float(w.abs().max()) + 1e-12)
