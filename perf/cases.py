"""The work that is timed: passes of the MoE block, of the attention block and of the language model
on one GPU, through the calls that the training script, the block benchmark and the smoke test make.

Kinds of pass
  moe_forward        MoE half of a block without gradients (serving)
  moe_train          MoE half, forward and backward, weight gradients in the flat fp32 buffers
  attention_forward  attention half without gradients
  attention_train    attention half, forward and backward
  lm_forward         language model, final hidden states of a prompt
  lm_step            language model, one whole training step with the optimizer

A pass with both halves and gradients is an ``lm_step``.  Weights are random, as the repository's own
benchmarks have them; activations, output gradients and token ids come from the seed.
"""
from __future__ import annotations

import math

import torch

from fluidmoe_b200.models.gpt import MoEGPT
from fluidmoe_b200.models.transformer import TransformerModel
from fluidmoe_b200.ops.optim import FusedAdam
from fluidmoe_b200.ops.rope import make_rope_freqs
from fluidmoe_b200.parallel.ddp import FluidDDP, FluidOptimizerWrapper
from fluidmoe_b200.parallel.scheduler import FlatGradBuffer, get_backward_scheduler
from fluidmoe_b200.tools.common import zipf_logit_prior

# Widths of the repository's presets, of the smoke test and of the training script.  ``capacity`` 0 is
# dropless routing; ``zipf`` adds the skewed expert prior of the fine-grained preset.
_SMOKE = dict(hidden=512, heads=4, kv_heads=2, ffn=768, experts=8, top_k=2, capacity=1.0, shared=0, zipf=0.0,
              act="swiglu", norm="rmsnorm")
_SCRIPT = dict(hidden=1024, heads=8, kv_heads=8, ffn=2048, experts=8, top_k=2, capacity=1.0, shared=0, zipf=0.0,
               act="gelu", norm="layernorm")
_MIXTRAL = dict(hidden=4096, heads=32, kv_heads=8, ffn=14336, experts=8, top_k=2, capacity=1.0, shared=0, zipf=0.0,
                act="swiglu", norm="rmsnorm")
_EXPERTS16 = dict(hidden=4096, heads=32, kv_heads=8, ffn=6400, experts=16, top_k=2, capacity=1.0, shared=0, zipf=0.0,
                  act="gelu", norm="layernorm")
_FINE = dict(hidden=2048, heads=16, kv_heads=16, ffn=1408, experts=64, top_k=6, capacity=0.0, shared=2, zipf=1.1,
             act="swiglu", norm="rmsnorm")
_EXPERTS64 = dict(hidden=2048, heads=16, kv_heads=16, ffn=1024, experts=64, top_k=8, capacity=1.0, shared=0, zipf=0.0,
                  act="gelu", norm="layernorm")


def _case(kind, widths, seq, batch, **more):
    c = dict(kind=kind, **widths, seq=seq, batch=batch)
    c.update(more)
    return c


def listed():
    lm = dict(layers=2, vocab=1024, moments="fp32", in_backward=False, lr=3e-4, aux=0.0, z=0.0)
    return [
        # one short prompt through the smoke test's model: launches and host work
        dict(name="lm_forward_short", **_case("lm_forward", _SMOKE, 96, 1, layers=2, vocab=1024)),
        # the smoke test's training step: a small model, many small kernels
        dict(name="lm_step_small", **_case("lm_step", _SMOKE, 256, 2, **lm)),
        # the training script at its defaults, in the GELU / LayerNorm architecture, with both router losses
        dict(name="lm_step_script", **_case("lm_step", _SCRIPT, 2048, 1, **dict(lm, vocab=32000, aux=0.01, z=0.001))),
        # the benchmark's step with one of its layers: bf16 moments, expert weights updated in the backward pass
        dict(name="lm_step_mixtral", **_case("lm_step", _MIXTRAL, 4096, 1, **dict(lm, layers=1, vocab=32000, moments="bf16",
                                                                                 in_backward=True, lr=1e-4))),
        # serving a handful of tokens: the expert weights are read once for few rows each
        dict(name="moe_forward_mixtral_64", **_case("moe_forward", _MIXTRAL, 16, 4)),
        # the benchmark's MoE layer, forward and backward
        dict(name="moe_train_mixtral", **_case("moe_train", _MIXTRAL, 4096, 1)),
        # dropless, shared experts, skewed load: a prompt of odd length, and the preset's training pass
        dict(name="moe_forward_fine_1531", **_case("moe_forward", _FINE, 1531, 1)),
        dict(name="moe_train_fine", **_case("moe_train", _FINE, 8192, 1)),
        # many small experts with a fixed capacity, GELU and LayerNorm, batch of two
        dict(name="moe_train_64experts", **_case("moe_train", _EXPERTS64, 4096, 2)),
        # attention of three prompts of odd length, as many KV heads as query heads
        dict(name="attention_forward_1117x3", **_case("attention_forward", _EXPERTS64, 1117, 3)),
        # the benchmark's attention block at the training length of one rank and at the full sequence
        dict(name="attention_train_4096", **_case("attention_train", _MIXTRAL, 4096, 1)),
        dict(name="attention_train_32768", **_case("attention_train", _MIXTRAL, 32768, 1)),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["moe_forward", "moe_train", "attention_forward", "attention_train", "lm_forward", "lm_step"])
    if kind.startswith("attention"):
        widths = rng.choice([_SMOKE, _SCRIPT, _MIXTRAL, _EXPERTS64])
        batch = rng.choice([1, 1, 2, 3])
        return _case(kind, widths, _log_uniform(rng, 48, 16384 // batch), batch)
    if kind.startswith("moe"):
        widths = rng.choice([_SMOKE, _SCRIPT, _MIXTRAL, _EXPERTS16, _FINE, _EXPERTS64])
        if kind == "moe_forward" or widths["capacity"] == 0.0:
            return _case(kind, widths, _log_uniform(rng, 32, 4096), rng.choice([1, 1, 2]))
        # fixed capacity and weight gradients: an expert's rows are a multiple of 64, as in the presets
        unit = 64 * widths["experts"] // widths["top_k"]
        return _case(kind, widths, unit * _log_uniform(rng, 1, 8192 // unit), 1)
    widths = rng.choice([_SMOKE, _SCRIPT, _FINE])
    layers = rng.choice([1, 2])
    vocab = rng.choice([1024, 4096, 32000])
    if kind == "lm_forward":
        return _case(kind, widths, _log_uniform(rng, 48, 2048), rng.choice([1, 2]), layers=layers, vocab=vocab)
    if widths["capacity"] == 0.0:
        seq = _log_uniform(rng, 200, 4096)
    else:
        seq = 256 * _log_uniform(rng, 1, 16)
    bf16 = rng.random() < 0.5
    losses = rng.random() < 0.5
    return _case(kind, widths, seq, 1, layers=layers, vocab=vocab, moments="bf16" if bf16 else "fp32", in_backward=bf16,
                 lr=3e-4, aux=0.01 if losses else 0.0, z=0.001 if losses else 0.0)


# ------------------------------------------------------------------------------------------------
def _model(case, device):
    half = dict(has_moe=False) if case["kind"].startswith("attention") else \
        dict(has_attention=False) if case["kind"].startswith("moe") else {}
    common = dict(activation_func=case["act"], norm_type=case["norm"], router_dtype=torch.float32,
                  capacity_factor=case["capacity"], num_shared_experts=case["shared"],
                  moe_combine_chunks=4, moe_dispatch_chunks=4, attn_proj_chunks=4, attn_qkv_chunks=4)
    sizes = (case["hidden"], case["heads"], case["kv_heads"], case["ffn"], case["experts"], case["top_k"])
    if case["kind"].startswith("lm"):
        model = MoEGPT(case["vocab"], case["layers"], *sizes, dtype=torch.bfloat16, device=device,
                       aux_loss_coeff=case.get("aux", 0.0), z_loss_coeff=case.get("z", 0.0), **common)
        layers = model.decoder.layers
        for name, p in model.named_parameters():
            if name.endswith("bias"):      # zero only before the first step of all
                torch.nn.init.normal_(p, std=0.02)
    else:
        model = TransformerModel(1, *sizes, dtype=torch.bfloat16, device=device, **common, **half)
        layers = model.layers
    if case["zipf"] > 0.0:
        prior = zipf_logit_prior(case["experts"], case["zipf"], device)
        for layer in layers:
            layer.set_router_bias(prior)
    return model


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    torch.manual_seed(seed)
    model = _model(case, device)
    state = dict(case=case, model=model)
    kind, seq, batch = case["kind"], case["seq"], case["batch"]
    sched = get_backward_scheduler()
    sched.enable(device)
    if kind.endswith(("train", "step")):
        # the scheduler is one per process: every state brings its own gradient buffers
        sched.shared_buffer, sched.expert_buffer = FlatGradBuffer(), FlatGradBuffer()
    if kind.startswith("lm"):
        ids = torch.randint(0, case["vocab"], (seq + 1, batch), device=device)
        state.update(ids=ids[:-1], labels=ids[1:])
        if kind == "lm_step":
            ddp = FluidDDP(None, model, sched)
            opt = FluidOptimizerWrapper(
                FusedAdam(model.parameters(), lr=case["lr"],
                          state_dtype=torch.bfloat16 if case["moments"] == "bf16" else torch.float32), sched)
            if case["in_backward"]:
                opt.fuse_into_backward()
            state.update(ddp=ddp, opt=opt)
    else:
        x = torch.randn(seq, batch, case["hidden"], dtype=torch.bfloat16, device=device)
        state.update(x=x.requires_grad_(kind.endswith("train")), rotary=None)
        if kind.startswith("attention"):
            state["rotary"] = make_rope_freqs(seq, case["hidden"] // case["heads"], device=device)
        if kind.endswith("train"):
            sched.configure_allreduce(True)
            model.setup_ar_buffer()
            state["dy"] = torch.randn(seq, batch, case["hidden"], dtype=torch.bfloat16, device=device)
    if kind.endswith(("train", "step")):
        state["buffers"] = (sched.shared_buffer, sched.expert_buffer)
    return state


def run(state):
    kind, model = state["case"]["kind"], state["model"]
    if kind == "lm_forward":
        with torch.no_grad():
            return model(state["ids"])
    if kind.endswith("forward"):
        with torch.no_grad():
            return model(state["x"], state["rotary"])
    sched = get_backward_scheduler()
    sched.shared_buffer, sched.expert_buffer = state["buffers"]
    if kind == "lm_step":
        ddp, opt = state["ddp"], state["opt"]
        ddp.zero_grad_buffer()
        loss = ddp(state["ids"], state["labels"])
        loss.backward()
        ddp.finish_grad_sync()
        opt.step()
        return dict(loss=loss.detach(), **{n: p.detach() for n, p in model.named_parameters()})
    x = state["x"]
    x.grad = None
    for p in model.parameters():
        p.grad = None
        if hasattr(p, "_ar_buf_written"):
            p._ar_buf_written = False
    y = model(x, state["rotary"])
    y.backward(state["dy"])
    sched.finish_batch()
    sched.clear_iteration()
    out = dict(y=y.detach(), dx=x.grad)
    unused = ("moe", "router", "shared", "ln2") if kind.startswith("attention") else ("qkv", "proj", "ln1")
    for name, p in model.named_parameters():
        if not name.split(".")[-1].startswith(unused):     # the other half of the block gets no gradient
            out["d_" + name] = p.main_grad
    return out


# ------------------------------------------------------------------------------------------------
def work(case):
    """Multiply-adds of the matrix products and of causal attention; inputs read once, outputs written once."""
    kind = case["kind"]
    H, F, E, k, heads, kv = (case[n] for n in ("hidden", "ffn", "experts", "top_k", "heads", "kv_heads"))
    d, seq, batch = H // heads, case["seq"], case["batch"]
    T = seq * batch
    mats = 3 if case["act"] == "swiglu" else 2
    train = kind.endswith(("train", "step"))
    moe, attention, lm = not kind.startswith("attention"), not kind.startswith("moe"), kind.startswith("lm")
    layers = case.get("layers", 1)
    flops = bytes_ = params_dense = params_expert = 0.0
    if moe:
        shared = mats * H * F * case["shared"]
        params_dense += shared + H * E + H
        params_expert += min(E, T * k) * mats * H * F
        flops += 2.0 * T * (k * mats * H * F + shared + H * E) * (3 if train else 1)
    if attention:
        proj = H * (heads + 2 * kv) * d + H * H
        params_dense += proj + H
        flops += 2.0 * T * proj * (3 if train else 1)
        flops += 2.0 * batch * float(seq) * seq * heads * d * (3.5 if train else 1)     # half of the s x s square
    flops *= layers
    weights = layers * (params_dense + params_expert)
    if lm:
        weights += 2 * case["vocab"] * H + H if kind == "lm_step" else min(T, case["vocab"]) * H + H
        if kind == "lm_step":
            flops += 2.0 * T * case["vocab"] * H * 3
            moment = 4 if case["moments"] == "fp32" else 2
            bytes_ += weights * (2 + 2 + 4 * moment) + 16 * T
        else:
            bytes_ += 2 * weights + 2 * T * H + 8 * T
    elif train:
        bytes_ += weights * (2 + 4) + 4 * 2 * T * H      # weights in, fp32 gradients out; x, dy, y, dx
    else:
        bytes_ += 2 * weights + 2 * 2 * T * H
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times what was seen on a B200.  MoE half against the same block in 64 bits (512 to 2048
    tokens, four widths): rel 0.0034, max 0.074.  Attention half against the library's attention kernels:
    rel 0.0045, max 0.036."""
    if case["kind"].startswith("moe"):
        return {"rel": 1.5e-2, "max": 0.3}
    if case["kind"].startswith("attention"):
        return {"rel": 1.8e-2, "max": 0.15}
    if case["kind"] == "lm_forward":
        # rel 0.0029, max 0.021 with the library's attention; rounding may also send a token whose logits
        # nearly tie to another expert, which changes its whole row
        return {"rel": 1.5e-2, "max": 0.8}
    # The first updates of Adam have the size lr whatever the gradient's: where rounding turns a gradient's
    # sign the weight ends 2 lr away.  With the library's attention 1.7 % of the signs of the noisiest matrix
    # (weights of 0.01) turned, which is rel 26 lr and max 200 lr; a matrix left without its update is rel 100 lr.
    return {"rel": 60.0 * case["lr"], "max": 400.0 * case["lr"]}
