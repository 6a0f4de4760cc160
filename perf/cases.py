"""What the speed of this framework is measured on: passes through its public entry points.

Three paths:

``step``    one training step as a training loop makes it: ``zero_grad``, ``training_step``, ``backward``,
            ``optimizer.step()`` on a batch that is already on the GPU.  The loss and every updated parameter come
            back, and from the (Jump)ReLU steps every gradient as well: a selection may keep either of two values that
            differ by a rounding error, which leaves the weights alike but not the gradients of the two features.
``infer``   the module's forward without gradients (validation): pre-activations, features and both reconstructions.
``layers``  the per-layer calls of a model whose MLPs are replaced by the transcoder: ``encoder(x, layer=i)``, the
            nonlinearity, ``decoder(features, layer=i)``, for every layer in turn.

A state is a run that is under way: parameters, optimizer and buffers exist, and two steps have been made.
"""
import math

import torch

import crosslayer_transcoder_b200.model as M
from crosslayer_transcoder_b200 import synthetic

#: Far beyond the tokens of any run here: features that start dead stay dead and no live one dies, so that every step
#: does the same work (as in the benchmark).
TOKENS_TILL_DEAD = 10 ** 12


def _case(name, path, kind, cross, bf16, L, D, F, B, **over):
    c = {"path": path, "kind": kind, "cross": cross, "bf16": bf16, "L": L, "D": D, "F": F, "B": B, "k": 0, "k_aux": 0,
         "fuse_optimizer": False, "sparsity": False, "batch": "fp16" if bf16 else "fp32"}
    c.update(over)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The test-suite's size: a debugging run, or one of many tiny transcoders.  Launches and latency.
        _case("tiny clt topk bf16", "step", "topk", True, True, 3, 64, 256, 136, k=8, k_aux=16),
        # The reference's CPU-runnable toy configuration: fp32 throughout.
        _case("toy clt jumprelu fp32", "step", "jumprelu", True, False, 12, 768, 1024, 512, sparsity=True),
        # fp32 run with per-layer batch-wide selection at odd sizes (a feature count that no tile divides).
        _case("odd plt perlayer fp32", "step", "perlayer_batchtopk", False, False, 6, 320, 2001, 777, k=16),
        # The reference's default training configuration: about 120 thousand features, dense crosslayer decoder.
        _case("default clt jumprelu bf16", "step", "jumprelu", True, True, 12, 768, 10000, 4000, sparsity=True),
        # Per-layer transcoder of the benchmark set, with the pre-activation loss.
        _case("plt jumprelu bf16", "step", "jumprelu", False, True, 12, 768, 24576, 4000),
        # Wide residual stream (four layers of the 26-layer configuration), last batch of an epoch: ragged.
        _case("wide clt jumprelu bf16", "step", "jumprelu", True, True, 4, 2304, 16384, 3001, sparsity=True),
        # The reference's TopK configuration's width, optimizer separate from backward (clipping, accumulation).
        _case("clt topk bf16", "step", "topk", True, True, 12, 768, 20000, 2047, k=16, k_aux=512),
        # The benchmark's default workload, with the decoder's optimizer update fused into backward.
        _case("large clt topk bf16", "step", "topk", True, True, 12, 768, 32768, 4000, k=32, k_aux=512,
              fuse_optimizer=True),
        # Batch-wide selection on a wide residual stream (four layers of the 16-layer configuration).
        _case("wide clt batchtopk bf16", "step", "batchtopk", True, True, 4, 2048, 16384, 8192, k=4,
              fuse_optimizer=True),
        # Validation forward of a TopK transcoder: dense pre-activations and features come back.
        _case("infer clt topk bf16", "infer", "topk", True, True, 12, 768, 10000, 1000, k=16, batch="fp32"),
        # Validation forward of a per-layer JumpReLU transcoder on a small ragged batch.
        _case("infer plt jumprelu bf16", "infer", "jumprelu", False, True, 12, 768, 24576, 333, batch="fp32"),
        # Replacement-model pass over one prompt: a few hundred tokens, layer after layer.
        _case("layers clt relu bf16", "layers", "relu", True, True, 12, 768, 10000, 257, batch="fp32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Bytes and multiplications of the case in one figure (bytes): what draw() holds below the largest listed case."""
    w = work(c)
    return w["bytes"] + w["flops"] / (250 if c["bf16"] else 15)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        path = rng.choice(["step"] * 8 + ["infer", "infer", "layers"])
        bf16 = rng.random() < 0.75
        kind = rng.choice(["jumprelu", "topk", "batchtopk", "perlayer_batchtopk", "relu"])
        if path == "layers":
            kind = "relu"
        cross = rng.random() < 0.65
        L = rng.randint(2, 12)
        # bf16 rows are 16-byte multiples; fp32 takes any feature count beside widths of 64
        if bf16:
            D, F = 8 * _log(rng, 8, 288), 8 * _log(rng, 32, 4096)
            if (D * F) % 64:
                continue
        else:
            D, F = 64 * _log(rng, 1, 20), _log(rng, 200, 8000)
        B = _log(rng, 64, 6000) if path == "step" else _log(rng, 5, 1500)
        c = _case(None, path, kind, cross, bf16, L, D, F, B)
        if kind in ("topk", "batchtopk", "perlayer_batchtopk"):
            if -(-D // 256) not in (1, 2, 3, 4, 6, 8, 9):        # the row widths that the sparse decoder takes
                continue
            c["k"] = min(_log(rng, 4, 64), F // 8)
            if path == "step":
                c["fuse_optimizer"] = F % 8 == 0 and rng.random() < 0.5
                if kind == "topk" and rng.random() < 0.75:
                    c["k_aux"] = min(512, F // 16)
        elif path == "step" and kind == "jumprelu":
            c["sparsity"] = rng.random() < 0.5
        if bf16 and path == "step":
            c["batch"] = rng.choice(["fp16", "bf16", "fp32"])
        if path != "step":
            c["batch"] = "fp32"
        # a state three times over, and the dense results of the forward passes, fit the card
        dense = 4 * B * L * F
        if _params(c) > 2.3e9 or dense > 6.5e9 or (path != "step" and dense > 2e9) or _cost(c) > most:
            continue
        return c


def _blocks(c):
    return c["L"] * (c["L"] + 1) // 2 if c["cross"] else c["L"]


def _params(c):
    L, D, F = c["L"], c["D"], c["F"]
    return L * D * F + _blocks(c) * F * D + L * F + L * D + (L * F if c["kind"] == "jumprelu" else 0)


def _returns_gradients(c):
    return c["kind"] in ("jumprelu", "relu")


def _spec(c):
    return synthetic.WorkloadSpec(
        "case", c["L"], c["D"], c["F"], c["B"], c["kind"], c["cross"], c["bf16"],
        rank_u=min(64, c["D"]), n_outlier=max(1, c["D"] // 192), lambda_sparsity=4e-4 if c["sparsity"] else 0.0,
        pre_actv_loss=3e-6 if c["kind"] == "jumprelu" else 0.0, k=c["k"], k_aux=c["k_aux"],
        aux_loss_scale=1 / 32 if c["k_aux"] else 0.0, tokens_till_dead=TOKENS_TILL_DEAD,
        dead_fraction=0.1 if c["k_aux"] else 0.0)


def _module(c, spec, dev, g):
    L, D, F = c["L"], c["D"], c["F"]
    with torch.device(dev):
        enc = M.Encoder(D, F, L)
        dec = (M.CrosslayerDecoder if c["cross"] else M.Decoder)(D, F, L)
        nl = {"jumprelu": lambda: M.JumpReLU(theta=spec.theta, bandwidth=spec.bandwidth, n_layers=L, d_features=F),
              "relu": lambda: M.ReLU(), "topk": lambda: M.PerLayerTopK(k=c["k"]),
              "batchtopk": lambda: M.BatchTopK(k=c["k"], e=spec.e),
              "perlayer_batchtopk": lambda: M.PerLayerBatchTopK(k=c["k"], e=spec.e, n_layers=L)}[c["kind"]]()
        model = M.CrossLayerTranscoder(nl, enc, dec, M.DimensionwiseInputStandardizer(L, D),
                                       M.DimensionwiseOutputStandardizer(L, D))
        with torch.no_grad():
            enc.W.uniform_(-D ** -0.5, D ** -0.5, generator=g)
            bound = (L * F) ** -0.5 if c["cross"] else F ** -0.5
            for w in dec.blocks():
                w.uniform_(-bound, bound, generator=g)
            for b in (enc.b, dec.b):
                b.normal_(0.0, 0.02, generator=g)
        common = dict(model=model, learning_rate=spec.lr, tokens_till_dead=TOKENS_TILL_DEAD, log_metrics_every=0)
        if c["kind"] in ("jumprelu", "relu"):
            mod = M.JumpReLUCrossLayerTranscoderModule(lambda_sparsity=spec.lambda_sparsity, c_sparsity=1.0,
                                                       pre_actv_loss=spec.pre_actv_loss, **common)
            mod.global_step = mod.trainer.max_steps = 1          # the sparsity penalty's ramp at its end
        elif c["kind"] == "topk":
            mod = M.TopKCrossLayerTranscoderModule(topk_aux=M.PerLayerTopK(k=c["k_aux"]),
                                                   aux_loss_scale=spec.aux_loss_scale, **common)
            if c["k_aux"]:
                # a tenth of the features is dead and, with a bias of -1, stays so
                dead = torch.rand(L, F, device=dev, generator=g) < spec.dead_fraction
                mod.last_active[dead] = 2 * TOKENS_TILL_DEAD
                with torch.no_grad():
                    enc.b[dead] = -1.0
        else:
            mod = M.CrossLayerTranscoderModule(**common)
    mod = mod.to(dev)
    mod.precision = "bf16" if c["bf16"] else "fp32"
    mod.fuse_optimizer = bool(c["fuse_optimizer"])
    return mod


def prepare(case, seed):
    c, dev = case, torch.device("cuda:0")
    spec = _spec(c)
    g = torch.Generator(device=dev).manual_seed(int(seed))
    mod = _module(c, spec, dev, g)
    dtype = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}[c["batch"]]
    # outlier channels are large: fp16 batches hold them as the reference's activation store does
    batch = synthetic.make_batch(spec, seed=int(seed) + 1, dtype=dtype, device=dev)
    mod.model.initialize_standardizers(batch)
    state = {"case": c, "mod": mod, "batch": batch, "i": 1, "opt": None}
    if c["path"] == "step":
        state["opt"] = mod.configure_optimizers()
        for _ in range(2):
            _step(state)
    elif c["path"] == "infer":
        state["acts"] = batch[:, 0].contiguous()
        del state["batch"]
    else:
        state["acts"] = mod.model.input_standardizer(batch[:, 0].contiguous()).unsqueeze(0)     # [1, tokens, L, D]
        del state["batch"]
    return state


def _step(state):
    mod, opt = state["mod"], state["opt"]
    opt.zero_grad()
    loss = mod.training_step(state["batch"], state["i"])
    loss.backward()
    opt.step()
    state["i"] += 1
    return loss


def run(state):
    c, mod = state["case"], state["mod"]
    if c["path"] == "step":
        loss = _step(state)
        out = {"loss": loss.detach(), "weights": [p.detach() for p in mod.parameters()]}
        if _returns_gradients(c):
            out["gradients"] = [p.grad for p in mod.parameters() if p.grad is not None]
        return out
    with torch.no_grad():
        if c["path"] == "infer":
            return mod(state["acts"])
        acts, model, L = state["acts"], mod.model, c["L"]
        feats = torch.empty(*acts.shape[:3], c["F"], device=acts.device)
        recons = []
        for l in range(L):
            feats[:, :, l] = model.nonlinearity(model.encoder(acts[:, :, l], layer=l), layer=l)
            recons.append(model.decoder(feats[:, :, :l + 1] if c["cross"] else feats[:, :, l], layer=l))
        return feats, recons


def work(case):
    c = case
    B, L, D, F, P, n = c["B"], c["L"], c["D"], c["F"], _blocks(c), _params(c)
    e = 2 if c["batch"] != "fp32" else 4
    sparse = c["k"] > 0
    enc = 2.0 * B * L * D * F
    dec = 2.0 * B * P * D * (c["k"] if sparse else F)
    if c["path"] == "step":
        # Adam reads and writes the weight and both moments; gradients are an output only where they are returned
        nbytes = 24.0 * n + 2.0 * B * L * D * e + (4.0 * n if _returns_gradients(c) else 0.0)
        if sparse:
            flops = enc + 2.0 * B * L * D * c["k"] + 3 * dec
            # auxiliary loss: at most k_aux of the tenth that is dead, of which about a twentieth is positive
            n_aux = min(c["k_aux"], F / 200)
            flops += 3 * 2.0 * B * P * D * n_aux + 2 * 2.0 * B * L * D * n_aux
        else:
            flops = 2 * enc + 3 * dec
        return {"bytes": nbytes, "flops": flops}
    weights = (L * D * F + P * F * D) * (2.0 if c["bf16"] else 4.0)
    if c["path"] == "infer":
        return {"bytes": weights + 4.0 * B * L * D + 8.0 * B * L * F + 8.0 * B * L * D, "flops": enc + dec}
    return {"bytes": weights + 4.0 * B * L * D + 4.0 * B * L * F + 4.0 * B * L * D, "flops": enc + dec}


def tolerance(case):
    """About four times what a step's results are off by, at reduced sizes, from the same step in another order of
    summation (bf16: the operands rounded alike, on the CPU) or in 64 bits (fp32)."""
    if case["path"] == "step" and not _returns_gradients(case):
        # Adam moves a weight of 0.03 by 1e-4 a step whichever side a rounding error puts a vanishing gradient on:
        # weights were off by 1.3e-4 (bf16) and 4e-8 (fp32; one selected entry exchanged for its equal: 4e-5)
        return {"rel": 2e-3, "max": 8e-2} if case["bf16"] else {"rel": 2e-4, "max": 2e-2}
    # encoder gradients were off by 3e-3 (bf16) and 4e-4 (fp32), because a pre-activation on its threshold falls on
    # either side; everything else by 2e-3 and 5e-7
    return {"rel": 1.2e-2, "max": 0.6} if case["bf16"] else {"rel": 1.6e-3, "max": 0.3}
