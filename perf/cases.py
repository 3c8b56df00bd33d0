"""The work that a training job hands to one GPU, as cases that can be timed and compared.

A case is a dict of plain values; ``kind`` says which public entry point it goes through:

    step     ``deepspeed.initialize`` + ``train_batch``: one optimizer step of a pipeline stage that owns
             the whole layer list (transformer decoder, masked-LM encoder or bottleneck ResNet)
    block    forward and backward of one ``TransformerBlock`` over a micro-batch, weight gradients included:
             what a middle stage does between its receive and its send
    forward  ``PipelineModule.forward`` of a stage of blocks without a graph: a redundant forward of the
             successor's layers, or a stage's warm-up forward
    head     what the last stage adds behind its blocks: LayerNorm, vocabulary projection, cross entropy,
             forward and backward
    conv     forward and backward of one convolution + batch norm (+ residual + ReLU) layer of the image network

Weights are made on the GPU from the seed (N(0, 0.02), Kaiming for convolutions, unit gains, zero biases):
the layers' own initialisation draws on the host, which takes seconds at these sizes.
"""
import math
import os

import torch

from bamboo_b200 import api, layers, models, resnet
from bamboo_b200.arena import ParamArena
from bamboo_b200.module import LayerSpec, PipelineModule

os.environ.setdefault("BAMBOO_QUIET", "1")
DEVICE = "cuda"

# a drawn case stays below the largest listed one (gpt2_medium_step: 27 TFLOP, 179 M parameters)
DRAW_FLOPS, DRAW_PARAMS = 10e12, 100e6


def listed():
    return [
        # the toy decoder that a user tries a pipeline with: hundreds of launches of a few microseconds
        {"name": "gpt_toy_step", "kind": "step", "model": "gpt", "layers": 4, "hidden": 256, "heads": 4, "ffn": 1024, "seq": 128,
         "vocab": 1024, "micro_batch": 4, "micro_batches": 4},
        # the headline workload's dimensions, depth of one of four stages plus both ends, four micro-batches
        {"name": "gpt2_medium_step", "kind": "step", "model": "gpt", "layers": 6, "hidden": 1024, "heads": 16, "ffn": 4096,
         "seq": 1024, "vocab": 50257, "micro_batch": 8, "micro_batches": 4},
        # the masked-LM encoder at its dimensions, depth of one of eight stages plus both ends
        {"name": "bert_large_step", "kind": "step", "model": "bert", "layers": 3, "hidden": 1024, "heads": 16, "ffn": 4096,
         "seq": 512, "vocab": 30522, "micro_batch": 16, "micro_batches": 4},
        # bottleneck ResNet at the widths, image size and micro-batch of the image workload, few blocks per stage
        {"name": "resnet_step", "kind": "step", "model": "resnet", "b0": 1, "b1": 2, "b2": 3, "b3": 1, "width": 64, "size": 224,
         "classes": 1000, "micro_batch": 32, "micro_batches": 2},
        # a small image job: odd image size, one block per stage, launch-bound
        {"name": "resnet_small_step", "kind": "step", "model": "resnet", "b0": 1, "b1": 1, "b2": 1, "b3": 1, "width": 32, "size": 75,
         "classes": 40, "micro_batch": 8, "micro_batches": 2},
        # one layer of the image network at its own sizes, forward and backward
        {"name": "conv_layer", "kind": "conv", "cin": 128, "cout": 128, "k": 3, "stride": 1, "relu": True, "residual": False,
         "size": 28, "micro_batch": 32},
        # one block of the 6.7B decoder: head dimension 128, hidden 4096, sequence 2048
        {"name": "gpt_6.7b_block", "kind": "block", "hidden": 4096, "heads": 32, "ffn": 16384, "seq": 2048, "micro_batch": 2,
         "causal": True},
        # sequences that no tile divides
        {"name": "ragged_block", "kind": "block", "hidden": 1024, "heads": 16, "ffn": 4096, "seq": 777, "micro_batch": 3,
         "causal": True},
        # head dimension 128 without a causal mask, one short ragged sequence per micro-batch
        {"name": "wide_head_block", "kind": "block", "hidden": 2048, "heads": 16, "ffn": 8192, "seq": 513, "micro_batch": 1,
         "causal": False},
        # the redundant forward of a quarter of the headline model for one micro-batch
        {"name": "stage_forward", "kind": "forward", "layers": 6, "hidden": 1024, "heads": 16, "ffn": 4096, "seq": 1024,
         "micro_batch": 8, "causal": True},
        # the same for the toy: the latency of a handful of launches
        {"name": "toy_forward", "kind": "forward", "layers": 2, "hidden": 256, "heads": 4, "ffn": 1024, "seq": 128,
         "micro_batch": 4, "causal": True},
        # the last stage's end on a ragged number of tokens
        {"name": "vocabulary_head", "kind": "head", "hidden": 1024, "vocab": 50257, "seq": 333, "micro_batch": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the range of its kind, odd ones among them."""
    while True:
        kind = rng.choice(["step", "step", "step", "block", "block", "conv", "forward", "head"])
        case = {"kind": kind}
        head_dim = rng.choice([64, 64, 128])
        heads = _log_int(rng, 1, 2048 // head_dim)
        shape = {"hidden": heads * head_dim, "heads": heads, "ffn": 4 * heads * head_dim, "seq": _log_int(rng, 16, 2048),
                 "micro_batch": _log_int(rng, 1, 16)}
        if kind == "step":
            model = rng.choice(["gpt", "bert", "resnet"])
            case["model"] = model
            if model == "resnet":
                case.update(b0=rng.randint(1, 3), b1=rng.randint(1, 3), b2=rng.randint(1, 3), b3=rng.randint(1, 2),
                            width=rng.choice([16, 32, 64]), size=_log_int(rng, 64, 256), classes=_log_int(rng, 10, 1000),
                            micro_batch=_log_int(rng, 8, 32), micro_batches=rng.randint(1, 3))
            else:
                case.update(layers=rng.randint(1, 4), vocab=_log_int(rng, 200, 51000), micro_batches=rng.randint(1, 4), **shape)
        elif kind == "block":
            case.update(causal=rng.random() < 0.6, **shape)
        elif kind == "forward":
            case.update(layers=rng.randint(1, 6), causal=rng.random() < 0.6, **shape)
        elif kind == "head":
            case.update(hidden=shape["hidden"], vocab=_log_int(rng, 200, 51000), seq=shape["seq"], micro_batch=shape["micro_batch"])
        else:
            case.update(cin=8 * 2 ** rng.randint(0, 8), cout=16 * 2 ** rng.randint(0, 7), k=rng.choice([1, 1, 3, 3, 7]),
                        stride=rng.choice([1, 1, 2]), relu=rng.random() < 0.7, residual=rng.random() < 0.3, size=_log_int(rng, 7, 112),
                        micro_batch=_log_int(rng, 4, 32))
        if work(case)["flops"] <= DRAW_FLOPS and _parameters(case) <= DRAW_PARAMS:
            return case


# ----------------------------------------------------------------------------------- building
def _build(specs, seed):
    """The modules of a layer list on the GPU, weights drawn there from the seed."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    mods = []
    for spec in specs:
        with torch.device("meta"):
            mod = spec.build()
        mod.to_empty(device=DEVICE)
        with torch.no_grad():
            for sub in mod.modules():
                for name, p in sub.named_parameters(recurse=False):
                    _initialise(sub, name, p, gen)
        mods.append(mod)
    return mods


def _initialise(mod, name, p, gen):
    if p.dim() == 1:
        # gains of LayerNorm (ln1_w, ln2_w, ln_weight, LayerNorm.weight) and batch norm (bn_weight) are 1, biases 0
        gain = name.startswith("ln") and name.endswith(("_w", "_weight")) or name == "bn_weight" or (
            isinstance(mod, layers.LayerNorm) and name == "weight")
        p.fill_(1.0 if gain else 0.0)
    elif isinstance(mod, resnet.ConvBN):
        p.normal_(0.0, math.sqrt(2.0 / (p.shape[0] * mod.k * mod.k)), generator=gen)
    else:
        p.normal_(0.0, 0.02, generator=gen)
        if isinstance(mod, layers.Linear):
            p[mod.out_features:] = 0.0          # rows that only pad the vocabulary


def _config(case):
    return models.TransformerConfig(layers=case["layers"], hidden=case["hidden"], heads=case["heads"], ffn=case["ffn"],
                                    seq=case["seq"], vocab=case["vocab"], causal=case["model"] == "gpt", mlm=case["model"] == "bert")


def _blocks(case):
    return (case["b0"], case["b1"], case["b2"], case["b3"])


def _activation(gen, *shape):
    return torch.randn(*shape, device=DEVICE, generator=gen).bfloat16()


def _block_specs(case, n):
    return [LayerSpec(layers.TransformerBlock, case["hidden"], case["heads"], case["ffn"], causal=case["causal"])
            for _ in range(n)]


def _conv_side(case):
    return (case["size"] + 2 * ((case["k"] - 1) // 2) - case["k"]) // case["stride"] + 1


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 1)
    kind = case["kind"]
    if kind == "step":
        return _prepare_step(case, seed, gen)
    B, state = case["micro_batch"], {"kind": kind}
    if kind == "conv":
        mods = _build([LayerSpec(resnet.ConvBN, case["cin"], case["cout"], case["k"], stride=case["stride"], relu=case["relu"])], seed)
        side = _conv_side(case)
        state["x"] = torch.relu(_activation(gen, B, case["size"], case["size"], case["cin"]))
        state["residual"] = torch.relu(_activation(gen, B, side, side, case["cout"])) if case["residual"] else None
        state["dout"] = _activation(gen, B, side, side, case["cout"]) * 0.01
    elif kind == "head":
        mods = _build([LayerSpec(layers.LayerNorm, case["hidden"]),
                       LayerSpec(layers.Linear, case["hidden"], case["vocab"], bias=False, pad_to=128)], seed)
        state["x"] = _activation(gen, B, case["seq"], case["hidden"])
        state["labels"] = torch.randint(0, case["vocab"], (B, case["seq"]), device=DEVICE, generator=gen)
        state["loss_fn"] = layers.CrossEntropyLoss(case["vocab"])
    else:
        mods = _build(_block_specs(case, case.get("layers", 1)), seed)
        state["x"] = _activation(gen, B, case["seq"], case["hidden"])
        if kind == "block":
            state["dout"] = _activation(gen, B, case["seq"], case["hidden"]) * 0.01
    if kind == "forward":
        state["module"] = PipelineModule(mods, num_stages=1, partition_method="uniform")
        state["arena"] = ParamArena(state["module"].stage_parameters(0), DEVICE, with_optimizer_state=False)
    else:
        state["mods"] = mods
        state["arena"] = ParamArena([p for m in mods for p in m.parameters()], DEVICE)
    return state


def _prepare_step(case, seed, gen):
    B, n = case["micro_batch"], case["micro_batches"]
    if case["model"] == "resnet":
        specs, loss_fn = resnet.resnet_layer_specs(_blocks(case), case["classes"], case["width"]), resnet.resnet_loss(case["classes"])
        batches = []
        for _ in range(n):
            x = torch.zeros(B, case["size"], case["size"], resnet.IN_CHANNELS, dtype=torch.bfloat16, device=DEVICE)
            x[..., :3] = _activation(gen, B, case["size"], case["size"], 3)
            batches.append((x, torch.randint(0, case["classes"], (B,), device=DEVICE, generator=gen)))
    else:
        cfg = _config(case)
        specs, loss_fn = models.transformer_layer_specs(cfg), models.transformer_loss(cfg)
        host = torch.Generator().manual_seed(seed + 2)
        batches = []
        for _ in range(n):
            tok = torch.randint(0, cfg.vocab, (B, cfg.seq + 1), generator=host)
            if cfg.mlm:
                x, y = models.mlm_mask(tok[:, :-1].contiguous(), host, cfg.vocab, mask_id=min(models.MASK_TOKEN_ID, cfg.vocab - 1))
            else:
                x, y = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
            batches.append((x.to(DEVICE), y.to(DEVICE)))
    module = PipelineModule(_build(specs, seed), num_stages=1, loss_fn=loss_fn, partition_method="uniform")
    engine, *_ = api.initialize(model=module, config={
        "train_micro_batch_size_per_gpu": B, "gradient_accumulation_steps": n, "bf16": {"enabled": True},
        "optimizer": {"type": "Adam", "params": {"lr": 1e-4}}})
    return {"kind": "step", "engine": engine, "batches": batches, "smooth": case["model"] != "resnet"}


# ----------------------------------------------------------------------------------- running
def run(state):
    kind = state["kind"]
    if kind == "step":
        engine = state["engine"]
        loss = engine.train_batch(data_iter=iter(state["batches"]))
        arena = engine.arenas[0]
        # Both moments come from the same gradients.  The second one is what a comparison can hold on to: in the
        # first, one bias element's rounding error stands against the mean of 10^8 entries that are mostly the
        # rows of tokens that did not occur.  Gradients of an image network are not compared over several
        # layers at all: an activation within bf16 rounding of zero passes its whole gradient or none of it.
        out = {"loss": loss, "weights": arena.master}
        if state["smooth"]:
            out["exp_avg_sq"] = arena.exp_avg_sq
        return out
    if kind == "forward":
        with torch.no_grad():
            return {"out": state["module"](state["x"], 0)}
    x = state["x"].detach().requires_grad_(True)
    y = x
    if kind == "conv":
        residual = None if state["residual"] is None else state["residual"].detach().requires_grad_(True)
        y = state["mods"][0](x, residual)
    else:
        for mod in state["mods"]:
            y = mod(y)
    if kind == "head":
        loss = state["loss_fn"](y, state["labels"])
        loss.backward()
        out = {"loss": loss.detach()}
    else:
        y.backward(state["dout"])
        out = {"out": y.detach()}       # (a residual's gradient is dout under the mask of out > 0)
    layers.wgrad_sync(x.device)
    return {**out, "dx": x.grad, "weight_grads": state["arena"].grad}


# ----------------------------------------------------------------------------------- what is needed, what is allowed
def _parameters(case):
    h = case.get("hidden", 0)
    block = 12 * h * h + 13 * h if case["kind"] in ("block", "forward") or case.get("model") in ("gpt", "bert") else 0
    if case["kind"] == "head":
        return h * case["vocab"] + 2 * h
    if case["kind"] in ("block", "forward"):
        return case.get("layers", 1) * block
    if case["kind"] == "conv":
        return case["cout"] * (case["k"] ** 2 * case["cin"] + 2)
    if case["model"] == "resnet":
        total, cin = 49 * 8 * case["width"], case["width"]
        for i, n in enumerate(_blocks(case)):
            m = case["width"] * 2 ** i
            total += 4 * cin * m + n * 9 * m * m + 4 * m * m + (cin * m + (n - 1) * 8 * m * m)
            cin = 4 * m
        return total + cin * case["classes"]
    return case["layers"] * block + h * (2 * case["vocab"] + case["seq"] + 2) + (h * h if case["model"] == "bert" else 0)


def _block_flops(case, causal):
    """Forward of one transformer block over the micro-batch; a causal mask halves the attention products."""
    tokens, h = case["micro_batch"] * case["seq"], case["hidden"]
    return tokens * (8 * h * h + 4 * h * case["ffn"] + 4 * case["seq"] * h * (0.5 if causal else 1.0))


def work(case):
    kind, params = case["kind"], _parameters(case)
    B = case["micro_batch"]
    if kind == "step":
        n = case["micro_batches"]
        if case["model"] == "resnet":
            flops = 3 * n * B * resnet.conv_flops_per_image(_blocks(case), case["size"], case["classes"], case["width"])
            inputs = n * B * (case["size"] ** 2 * resnet.IN_CHANNELS * 2 + 8)
        else:
            tokens = B * case["seq"]
            head = 2 * tokens * case["hidden"] * case["vocab"] + (2 * tokens * case["hidden"] ** 2 if case["model"] == "bert" else 0)
            flops = 3 * n * (case["layers"] * _block_flops(case, case["model"] == "gpt") + head)
            inputs = n * tokens * 16
        # weights and both moments in and out (fp32), the bf16 working copy in and out
        return {"bytes": inputs + params * (6 * 4 + 2 * 2), "flops": flops}
    if kind == "conv":
        outputs = B * _conv_side(case) ** 2 * case["cout"]
        # x, dx, out, dout, and the residual with its gradient
        nbytes = 2 * (2 * B * case["size"] ** 2 * case["cin"] + (4 if case["residual"] else 2) * outputs)
        return {"bytes": nbytes + params * (2 + 8), "flops": 3 * 2 * outputs * case["k"] ** 2 * case["cin"]}
    act = 2 * B * case["seq"] * case["hidden"]
    if kind == "forward":
        return {"bytes": 2 * act + 2 * params, "flops": case["layers"] * _block_flops(case, case["causal"])}
    if kind == "head":
        # x in, dx out, labels in; weights read, gradients added to
        return {"bytes": 2 * act + 8 * B * case["seq"] + params * (2 + 8), "flops": 3 * 2 * B * case["seq"] * case["hidden"] * case["vocab"]}
    return {"bytes": 4 * act + params * (2 + 8), "flops": 3 * _block_flops(case, case["causal"])}


def tolerance(case):
    """About four times what the same layers show with every product and sum done in fp32 / fp64 by the framework
    at the same rounding points (bf16 activations), over the listed cases and forty drawn ones."""
    kind = case["kind"]
    if kind == "step":
        # seen: second moments 0.010 (largest 0.61), weights 0.0004; image networks: weights 0.002, loss 0.0075
        return {"rel": 0.03, "max": 0.1 if case["model"] == "resnet" else 0.99}
    if kind == "block":
        return {"rel": 0.016, "max": 0.25}      # seen: 0.004, 0.061 (hidden 4096)
    if kind == "forward":
        return {"rel": 0.024, "max": 0.2}       # seen: 0.006, 0.044 (six blocks)
    if kind == "head":
        return {"rel": 0.003, "max": 0.06}      # seen: 0.0006, 0.014
    return {"rel": 0.014, "max": 0.99}          # seen: 0.0033, 0.45 (ReLU masks at bf16 rounding of zero)
