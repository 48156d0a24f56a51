"""What the speed of this framework is measured on: the work that training and serving runs spend their time in, each piece through
the entry point that a program calls.

Kinds of cases (``case["kind"]``):

* ``norm``     LayerNorm / RMSNorm, forward and backward (every layer of every model, twice)
* ``attention`` flash attention, forward only (prefill of a static engine, evaluation) or forward and backward (training), on the
               packed projection output (multi-head self-attention) or on separate query / key / value views (grouped queries)
* ``paged``    one layer's attention of the continuous-batching engine: decoding tokens and portions of prompts over a paged cache
* ``layer``    a whole transformer layer in training: forward, backward, fp32 main gradients
* ``gpt``      a whole GPT model: logits of a batch, or a training pass with per-token losses and all gradients
* ``mamba``    a Mamba-2 mixer: training pass, or forward only
* ``moe``      a mixture-of-experts layer in training (fused dispatch, grouped GEMMs)
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

from megatronapp_b200 import ops
from megatronapp_b200.config.transformer_config import TransformerConfig
from megatronapp_b200.inference.dynamic import DynamicInferenceContext
from megatronapp_b200.models.gpt import GPTModel, get_gpt_layer_local_spec
from megatronapp_b200.parallel import state as ps
from megatronapp_b200.parallel.ddp import DistributedDataParallel, DistributedDataParallelConfig
from megatronapp_b200.ssm.mamba import MambaMixer
from megatronapp_b200.transformer.spec_utils import build_module

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one micro-batch of the GPT-2 125M plumbing model: the smallest call of a training step, latency and launches count
        dict(name="norm_125m", kind="norm", rows=1024, cols=768, rms=False, dtype="bf16"),
        # GPT-2 125M attention of a training step: 12 heads of 64, four sequences of 1024
        dict(name="attn_train_125m", kind="attention", train=True, packed=True, b=4, s=1024, hq=12, hkv=12, d=64, dtype="bf16"),
        # Llama-3 8B attention of a training step: grouped queries, one sequence of 4096
        dict(name="attn_train_gqa_4k", kind="attention", train=True, packed=False, b=1, s=4096, hq=32, hkv=8, d=128, dtype="bf16"),
        # prefill of a static batch of prompts of an odd length (fp16, GPT-3 1.3B heads)
        dict(name="attn_prefill_odd", kind="attention", train=False, packed=False, b=3, s=1337, hq=32, hkv=32, d=64, dtype="fp16"),
        # prefill of one long prompt, Llama-3 8B heads
        dict(name="attn_prefill_8k", kind="attention", train=False, packed=False, b=1, s=8192, hq=32, hkv=8, d=128, dtype="bf16"),
        # a decoding step of 64 running requests with contexts of 1k to 4k tokens, Llama-3 8B heads
        dict(name="decode_64", kind="paged", decode=64, chunks=0, chunk=0, ctx_min=1024, ctx_max=4096, hq=32, hkv=8, d=128, block=16, dtype="bf16"),
        # one request with a long context, the latency of a single user
        dict(name="decode_1_long", kind="paged", decode=1, chunks=0, chunk=0, ctx_min=12000, ctx_max=12000, hq=32, hkv=8, d=128, block=16, dtype="bf16"),
        # a step that carries two portions of prompts beside decoding requests
        dict(name="chunked_prefill", kind="paged", decode=24, chunks=2, chunk=500, ctx_min=500, ctx_max=3000, hq=32, hkv=8, d=128, block=16, dtype="bf16"),
        # one layer of GPT-3 6.7B, one sequence of 2048: the headline training benchmark is 32 of these
        dict(name="layer_6p7b", kind="layer", b=1, s=2048, hidden=4096, heads=32, groups=32, ffn=16384, swiglu=False, rms=False, rope=False, bias=True),
        # a small GPT model's whole training pass: embedding, layers, head, loss, gradients
        dict(name="gpt_train", kind="gpt", train=True, b=4, s=1024, layers=4, hidden=768, heads=12, vocab=50304, rope=False),
        # a Mamba-2 mixer at the width of a hybrid model, training pass
        dict(name="mamba_train", kind="mamba", train=True, b=1, s=2048, hidden=2048, d_state=128, headdim=64, groups=8),
        # a mixture-of-experts layer at half the width of Mixtral 8x7B, 8 experts, two per token, training pass
        dict(name="moe_train", kind="moe", b=2, s=2048, hidden=2048, ffn=7168, experts=8, topk=2),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["norm", "attention", "attention", "paged", "paged", "layer", "gpt", "mamba", "moe"])
    dtype = "fp16" if rng.random() < 0.2 else "bf16"
    if kind == "norm":
        return dict(kind=kind, rows=_log_int(rng, 16, 16384), cols=_log_int(rng, 256, 8192, 8), rms=rng.random() < 0.5, dtype=dtype)
    if kind == "attention":
        train, d = rng.random() < 0.5, rng.choice([64, 128])
        hkv = rng.choice([4, 8, 12, 16])
        packed = train and rng.random() < 0.5
        hq = hkv if packed else hkv * rng.choice([1, 2, 4])
        # training sequences are fixed lengths of a configuration, a quarter of them odd; prompts have any length
        s = _log_int(rng, 128, 4096, 64) if train and (packed or rng.random() < 0.75) else _log_int(rng, 100, 6000)
        b = max(1, min(rng.choice([1, 2, 4, 8]), (1 << 26) // (hq * s * d * 2)))
        return dict(kind=kind, train=train, packed=packed, b=b, s=s, hq=hq, hkv=hkv, d=d, dtype=dtype)
    if kind == "paged":
        hkv, group = rng.choice([4, 8, 12]), rng.choice([1, 2, 4, 8])
        chunks = rng.choice([0, 0, 1, 2, 4])
        return dict(kind=kind, decode=_log_int(rng, 1, 96), chunks=chunks, chunk=_log_int(rng, 16, 512) if chunks else 0,
                    ctx_min=64, ctx_max=_log_int(rng, 128, 4096), hq=hkv * group, hkv=hkv, d=rng.choice([64, 128]), block=rng.choice([16, 32]),
                    dtype=dtype)
    if kind == "layer":
        heads = rng.choice([8, 12, 16, 24])
        swiglu = rng.random() < 0.5
        return dict(kind=kind, b=rng.choice([1, 2]), s=_log_int(rng, 256, 2048, 64), hidden=heads * 128, heads=heads,
                    groups=heads // rng.choice([1, 4]) if swiglu else heads, ffn=heads * 128 * (3 if swiglu else 4), swiglu=swiglu, rms=swiglu,
                    rope=swiglu, bias=not swiglu)
    if kind == "gpt":
        heads = rng.choice([6, 8, 12])
        train = rng.random() < 0.5
        return dict(kind=kind, train=train, b=rng.choice([1, 2, 4]), s=_log_int(rng, 64, 1024, 64 if train else 1), layers=rng.choice([1, 2, 4]),
                    hidden=heads * 64, heads=heads, vocab=rng.choice([8192, 32000, 50304]), rope=rng.random() < 0.5)
    if kind == "mamba":
        return dict(kind=kind, train=rng.random() < 0.5, b=rng.choice([1, 2]), s=_log_int(rng, 64, 2048), hidden=rng.choice([512, 1024, 2048]),
                    d_state=rng.choice([64, 128]), headdim=64, groups=rng.choice([1, 8]))
    return dict(kind="moe", b=rng.choice([1, 2]), s=_log_int(rng, 64, 2048), hidden=rng.choice([512, 1024, 2048]), ffn=rng.choice([1024, 2048, 3584]),
                experts=rng.choice([4, 8, 16]), topk=rng.choice([1, 2]))


# ------------------------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, shape, dtype, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _fill(module, g):
    """Weights as at the start of training: matrices of standard deviation 0.02, scales near one, small biases."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            short = name.rsplit(".", 1)[-1]
            if short == "A_log":
                p.copy_(torch.empty(p.shape, device="cuda").uniform_(1, 8, generator=g).log())
            elif short == "dt_bias":
                dt = torch.empty(p.shape, device="cuda").uniform_(math.log(1e-3), math.log(0.05), generator=g).exp()
                p.copy_(torch.log(torch.expm1(dt)))
            elif short == "D" or (p.dim() == 1 and short in ("weight", "norm_weight")):
                p.normal_(1.0, 0.1, generator=g)
            elif "conv1d.weight" in name:
                p.normal_(0.0, 0.3, generator=g)
            elif name == "in_proj.weight":                     # step sizes stay within a factor of a few of their bias
                p.normal_(0.0, 0.5 * p.shape[1] ** -0.5, generator=g)
            else:
                p.normal_(0.0, 0.02, generator=g)
            if not hasattr(p, "tensor_model_parallel"):
                p.tensor_model_parallel = False


def _parallel_state():
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1, 1)
    torch.cuda.current_device()


def _ddp(config, module):
    return DistributedDataParallel(config, DistributedDataParallelConfig(grad_reduce_in_fp32=True), module)


def _context(c, g, seed):
    """A paged cache in the state that serving leaves it in: requests that came in turn, so that their blocks interleave."""
    r = random.Random(int(seed))
    n = c["decode"] + c["chunks"]
    # a decoding request holds its whole context; a request being prefilled holds the portions before this one
    reqs = [(int(round(c["ctx_min"] + (c["ctx_max"] - c["ctx_min"]) * (i + 0.5) / c["decode"])), 1) for i in range(c["decode"])]
    reqs += [(c["chunk"] * (i % 3), c["chunk"]) for i in range(c["chunks"])]
    r.shuffle(reqs)
    ctx, new = [L for L, _ in reqs], [m for _, m in reqs]
    blocks = sum(-(-(L + m) // c["block"]) for L, m in zip(ctx, new)) + n
    cx = DynamicInferenceContext(max(L + m for L, m in zip(ctx, new)) + 1, blocks, c["block"], max_tokens_per_step=16384, max_requests=max(n, 1))
    dev = torch.device("cuda", torch.cuda.current_device())
    for i in range(n):
        cx.add_request(str(i))
    left = list(ctx)
    while any(left):
        part = [(str(i), min(512, L)) for i, L in enumerate(left) if L]
        cx.begin_step(part, dev)
        cx.end_step()
        for i, m in part:
            left[int(i)] -= m
    work = [(str(i), new[i]) for i in range(n)]
    cx.begin_step(work, dev)
    kc, vc = cx.kv_pages(1, (c["hkv"], c["d"]), (c["hkv"], c["d"]), DTYPES[c["dtype"]])
    kc.normal_(0.0, 1.0, generator=g)
    vc.normal_(0.0, 1.0, generator=g)
    return cx, ctx, new, kc, vc


def _transformer_config(c, **kw):
    return TransformerConfig(num_layers=c.get("layers", 1), hidden_size=c["hidden"], num_attention_heads=c.get("heads", 8), params_dtype=torch.bfloat16,
                             bf16=True, hidden_dropout=0.0, attention_dropout=0.0, gradient_accumulation_fusion=True, **kw)


def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    if kind == "norm":
        dt = DTYPES[c["dtype"]]
        x = _normal(g, (c["rows"], 1, c["cols"]), dt).requires_grad_()
        gamma = (1 + _normal(g, (c["cols"],), torch.float32, 0.1)).to(dt).requires_grad_()
        beta = None if c["rms"] else _normal(g, (c["cols"],), dt, 0.1).requires_grad_()
        return dict(case=c, x=x, gamma=gamma, beta=beta, dy=_normal(g, x.shape, dt))
    if kind == "attention":
        dt, s, b, d = DTYPES[c["dtype"]], c["s"], c["b"], c["d"]
        st = dict(case=c)
        if c["packed"]:
            st["mixed"] = _normal(g, (s, b, c["hq"], 3 * d), dt).requires_grad_()
        else:
            # activations are [s, b, heads, d]; attention takes [b, heads, s, d] views of them
            st["q"], st["k"], st["v"] = (_normal(g, (s, b, h, d), dt).requires_grad_(c["train"]) for h in (c["hq"], c["hkv"], c["hkv"]))
        if c["train"]:
            st["do"] = _normal(g, (s, b, c["hq"], d), dt)
        return st
    if kind == "paged":
        cx, ctx, new, kc, vc = _context(c, g, seed)
        T, dt = sum(new), DTYPES[c["dtype"]]
        return dict(case=c, cx=cx, ctx=ctx, new=new, kc=kc, vc=vc, q=_normal(g, (T, c["hq"], c["d"]), dt),
                    k=_normal(g, (T, c["hkv"], c["d"]), dt), v=_normal(g, (T, c["hkv"], c["d"]), dt))
    _parallel_state()
    if kind == "layer":
        cfg = _transformer_config(c, num_query_groups=c["groups"], ffn_hidden_size=c["ffn"], gated_linear_unit=c["swiglu"],
                                  activation_func=F.silu if c["swiglu"] else F.gelu, add_bias_linear=c["bias"],
                                  normalization="RMSNorm" if c["rms"] else "LayerNorm")
        mod = build_module(get_gpt_layer_local_spec(), config=cfg).cuda()
        _fill(mod, g)
        rot = ops.rope_cos_sin(c["s"], c["hidden"] // c["heads"], device="cuda") if c["rope"] else None
        x = _normal(g, (c["s"], c["b"], c["hidden"]), torch.bfloat16).requires_grad_()
        return dict(case=c, mod=_ddp(cfg, mod), rot=rot, x=x, dy=_normal(g, x.shape, torch.bfloat16))
    if kind == "gpt":
        cfg = _transformer_config(c, ffn_hidden_size=4 * c["hidden"], activation_func=F.gelu)
        mod = GPTModel(cfg, get_gpt_layer_local_spec(), c["vocab"], c["s"], share_embeddings_and_output_weights=True, parallel_output=True,
                       position_embedding_type="rope" if c["rope"] else "learned_absolute").cuda()
        _fill(mod, g)
        tok = torch.randint(0, c["vocab"], (c["b"], c["s"] + 1), generator=g, device="cuda")
        pos = torch.arange(c["s"], device="cuda").unsqueeze(0).expand(c["b"], -1).contiguous()
        st = dict(case=c, tokens=tok[:, :-1].contiguous(), labels=tok[:, 1:].contiguous(), pos=pos)
        st["mod"] = _ddp(cfg, mod) if c["train"] else mod.eval()
        if c["train"]:
            st["dl"] = torch.full((c["b"], c["s"]), 1.0 / (c["b"] * c["s"]), device="cuda")
        return st
    if kind == "mamba":
        cfg = _transformer_config(c, mamba_state_dim=c["d_state"], mamba_head_dim=c["headdim"], mamba_num_groups=c["groups"])
        mod = MambaMixer(cfg, layer_number=1).cuda()
        _fill(mod, g)
        x = _normal(g, (c["s"], c["b"], c["hidden"]), torch.bfloat16).requires_grad_(c["train"])
        st = dict(case=c, x=x, mod=_ddp(cfg, mod) if c["train"] else mod.eval())
        if c["train"]:
            st["dy"] = _normal(g, x.shape, torch.bfloat16)
        return st
    cfg = _transformer_config(c, ffn_hidden_size=c["ffn"], moe_ffn_hidden_size=c["ffn"], num_moe_experts=c["experts"], moe_router_topk=c["topk"],
                              moe_router_dtype="fp32", moe_router_load_balancing_type="none", moe_token_dispatcher_type="flex",
                              moe_grouped_gemm=True, gated_linear_unit=True, activation_func=F.silu, add_bias_linear=False)
    mod = build_module(get_gpt_layer_local_spec(c["experts"], True).submodules.mlp, config=cfg).cuda()
    _fill(mod, g)
    x = _normal(g, (c["s"], c["b"], c["hidden"]), torch.bfloat16).requires_grad_()
    return dict(case=c, mod=_ddp(cfg, mod), x=x, dy=_normal(g, x.shape, torch.bfloat16))


# ------------------------------------------------------------------------------------------------------------------ one pass
def _main_grads(ddp):
    return {n: p.main_grad for n, p in ddp.module.named_parameters()}


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind == "norm":
        y = ops.layer_norm(st["x"], st["gamma"], st["beta"], 1e-5, rms=c["rms"])
        ins = [t for t in (st["x"], st["gamma"], st["beta"]) if t is not None]
        return [y, *torch.autograd.grad(y, ins, st["dy"])]
    if kind == "attention":
        scale = c["d"] ** -0.5
        if c["packed"]:
            o = ops.attention_packed_qkv(st["mixed"], scale, True).permute(2, 0, 1, 3)
            return [o, *torch.autograd.grad(o, [st["mixed"]], st["do"])]
        q, k, v = st["q"], st["k"], st["v"]
        o = ops.attention(q.permute(1, 2, 0, 3), k.permute(1, 2, 0, 3), v.permute(1, 2, 0, 3), scale, True).permute(2, 0, 1, 3)
        return [o, *torch.autograd.grad(o, [q, k, v], st["do"])] if c["train"] else [o]
    if kind == "paged":
        o = st["cx"].attend(1, st["q"], st["k"], st["v"], c["d"] ** -0.5)
        return [o, st["kc"], st["vc"]]
    if kind == "gpt" and not c["train"]:
        with torch.no_grad():
            return st["mod"](st["tokens"], st["pos"], None)
    if kind == "mamba" and not c["train"]:
        with torch.no_grad():
            return st["mod"](st["x"])[0]
    mod = st["mod"]
    mod.zero_grad_buffer()
    if kind == "gpt":
        loss = mod(st["tokens"], st["pos"], None, labels=st["labels"])
        loss.backward(st["dl"])
        return dict(loss=loss, grads=_main_grads(mod))
    x = st["x"]
    x.grad = None
    y = mod(x, rotary_pos_emb=st["rot"])[0] if kind == "layer" else mod(x)[0]
    y.backward(st["dy"])
    return dict(y=y, dx=x.grad, grads=_main_grads(mod))


# ------------------------------------------------------------------------------------------------------------------ work, tolerance
def _attn_flops(b, h, s, d, train):
    return 4.0 * b * h * d * s * (s + 1) / 2 * (3.5 if train else 1.0)


def work(case):
    c, kind = case, case["kind"]
    if kind == "norm":
        n, p = c["rows"] * c["cols"], c["cols"] * (1 if c["rms"] else 2)
        return {"bytes": 2.0 * (4 * n + 2 * p), "flops": 16.0 * n}
    if kind == "attention":
        tok = 2.0 * c["s"] * c["b"] * c["d"]
        q, kv = tok * c["hq"], tok * c["hkv"]
        moved = (2 * q + 2 * kv) if not c["train"] else (4 * q + 4 * kv)      # q k v (do) in; o (dq dk dv) out
        return {"bytes": moved, "flops": _attn_flops(c["b"], c["hq"], c["s"], c["d"], c["train"])}
    if kind == "paged":
        ctx = [c["ctx_min"] + (c["ctx_max"] - c["ctx_min"]) * (i + 0.5) / c["decode"] for i in range(c["decode"])]
        old = [c["chunk"] * (i % 3) for i in range(c["chunks"])]
        T = c["decode"] + c["chunks"] * c["chunk"]
        keys = sum(ctx) + sum(old)
        pairs = sum(ctx) + c["decode"] + sum(c["chunk"] * (L + (c["chunk"] + 1) / 2) for L in old)
        return {"bytes": 2.0 * c["d"] * (2 * keys * c["hkv"] + 2 * T * c["hq"] + 4 * T * c["hkv"]), "flops": 4.0 * pairs * c["hq"] * c["d"]}
    T = c["b"] * c["s"]
    if kind == "layer":
        dh = c["hidden"] // c["heads"]
        w = c["hidden"] * (c["hidden"] + 2 * c["groups"] * dh) + c["hidden"] ** 2 + c["hidden"] * c["ffn"] * (3 if c["swiglu"] else 2)
        return {"bytes": w * (2.0 + 4.0) + 8.0 * T * c["hidden"],
                "flops": 6.0 * w * T + _attn_flops(c["b"], c["heads"], c["s"], dh, True)}
    if kind == "gpt":
        w = c["layers"] * 12 * c["hidden"] ** 2 + c["vocab"] * c["hidden"]
        f = 2.0 * w * T + c["layers"] * _attn_flops(c["b"], c["heads"], c["s"], 64, False)
        if c["train"]:
            return {"bytes": 6.0 * w + 24.0 * T, "flops": 6.0 * w * T + c["layers"] * _attn_flops(c["b"], c["heads"], c["s"], 64, True)}
        return {"bytes": 2.0 * w + 2.0 * T * c["vocab"], "flops": f}
    if kind == "mamba":
        di, gn = 2 * c["hidden"], c["groups"] * c["d_state"]
        nh = di // c["headdim"]
        w = c["hidden"] * (2 * di + 2 * gn + nh) + di * c["hidden"]
        scan = 6.0 * di * c["d_state"] * T                                 # state update and read-out of every step
        m = 3.0 if c["train"] else 1.0
        return {"bytes": w * (6.0 if c["train"] else 2.0) + (8.0 if c["train"] else 4.0) * T * c["hidden"], "flops": m * (2.0 * w * T + scan)}
    w = 3.0 * c["hidden"] * c["ffn"]
    return {"bytes": 6.0 * w * c["experts"] + 8.0 * T * c["hidden"], "flops": 6.0 * w * T * c["topk"]}


def tolerance(case):
    """About four times the distance of the first version of each path from 64 bits (2-norms): 1.7e-3 for norms and paged attention, 2.5e-3
    for flash attention and its gradients (a sixth to an eighth of that in fp16, three more bits), 3.9e-3 to 4.5e-3 for the experts' layer,
    6e-3 for the Mamba mixer, 8e-3 for the gradients of whole layers and models."""
    kind, fp16 = case["kind"], case.get("dtype") == "fp16"
    if kind in ("norm", "paged"):
        return {"rel": 1e-3 if fp16 else 7e-3}
    if kind == "attention":
        return {"rel": 1.4e-3 if fp16 else 1e-2}
    return {"rel": {"moe": 1.8e-2, "mamba": 2.4e-2, "layer": 3e-2, "gpt": 3e-2}[kind]}


# ------------------------------------------------------------------------------------------------------------------ 64 bits
def _attn64(q, k, v, scale, do=None, visible=None):
    """``[n, d]`` of one head in 64 bits: output and, with ``do``, the three gradients.  ``visible``: keys that each query sees."""
    s = (q @ k.t()) * scale
    vis = visible if visible is not None else torch.arange(1, q.shape[0] + 1, device=q.device)
    s.masked_fill_(torch.arange(k.shape[0], device=q.device).unsqueeze(0) >= vis.unsqueeze(1), float("-inf"))
    p = torch.softmax(s, -1)
    o = p @ v
    if do is None:
        return o, None, None, None
    ds = p * (do @ v.t() - (do * o).sum(-1, keepdim=True)) * scale
    return o, ds @ k, ds.t() @ q, p.t() @ do


def _attention_module64(q, k, v, scale):
    """Differentiable causal attention on ``[s, b, h, d]`` with grouped keys."""
    s, b, h, d = q.shape
    rep = h // k.shape[2]
    k, v = (t.repeat_interleave(rep, dim=2) for t in (k, v))
    sc = torch.einsum("sbhd,tbhd->bhst", q, k) * scale
    sc = sc.masked_fill(torch.ones(s, s, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
    return torch.einsum("bhst,tbhd->sbhd", torch.softmax(sc, -1), v)


def _norm64(x, w, b, rms, eps=1e-5):
    if rms:
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w
    return F.layer_norm(x, (x.shape[-1],), w, b, eps)


def _rope64(x, cs):
    half = cs.shape[-1] // 2
    cos, sin = cs[:, :half].double()[:, None, None, :], cs[:, half:].double()[:, None, None, :]
    x0, x1 = x[..., :half], x[..., half:]
    return torch.cat([x0 * cos - x1 * sin, x1 * cos + x0 * sin], dim=-1)


def _block64(x, w, pre, heads, groups, swiglu, rms, rot):
    """One pre-norm transformer layer on ``[s, b, hidden]``; ``w``: its parameters by name."""
    g = lambda n: w.get(pre + n)  # noqa: E731
    s, b, hid = x.shape
    dh = hid // heads
    h = _norm64(x, g("input_layernorm.weight"), g("input_layernorm.bias"), rms)
    qkv = F.linear(h, g("self_attention.linear_qkv.weight"), g("self_attention.linear_qkv.bias")).view(s, b, groups, (heads // groups + 2) * dh)
    q, k, v = torch.split(qkv, [heads // groups * dh, dh, dh], dim=3)
    q = q.reshape(s, b, heads, dh)
    if rot is not None:
        q, k = _rope64(q, rot), _rope64(k, rot)
    o = _attention_module64(q, k, v, dh ** -0.5).reshape(s, b, hid)
    x = x + F.linear(o, g("self_attention.linear_proj.weight"), g("self_attention.linear_proj.bias"))
    h = _norm64(x, g("pre_mlp_layernorm.weight"), g("pre_mlp_layernorm.bias"), rms)
    h = F.linear(h, g("mlp.linear_fc1.weight"), g("mlp.linear_fc1.bias"))
    if swiglu:
        a, u = h.chunk(2, -1)
        h = F.silu(a) * u
    else:
        h = F.gelu(h, approximate="tanh")
    return x + F.linear(h, g("mlp.linear_fc2.weight"), g("mlp.linear_fc2.bias"))


def _mamba64(x, w, c):
    """Mamba-2 mixer on ``[s, b, hidden]``, the recurrence in blocks of 64 steps."""
    s, b, hid = x.shape
    di, ng, n, p = 2 * hid, c["groups"], c["d_state"], c["headdim"]
    nh = di // p
    z, xbc, dt = torch.split(F.linear(x, w["in_proj.weight"]).transpose(0, 1), [di, di + 2 * ng * n, nh], dim=-1)
    cw = w["conv1d.weight"]
    xbc = F.silu(F.conv1d(F.pad(xbc.transpose(1, 2), (cw.shape[-1] - 1, 0)), cw, w["conv1d.bias"], groups=cw.shape[0]).transpose(1, 2))
    xs, B, C = torch.split(xbc, [di, ng * n, ng * n], dim=-1)
    dt = F.softplus(dt + w["dt_bias"])
    da = dt * -torch.exp(w["A_log"])
    xs = xs.reshape(b, s, nh, p)
    B, C = (t.reshape(b, s, ng, n).repeat_interleave(nh // ng, dim=2) for t in (B, C))
    xd = xs * dt.unsqueeze(-1)
    S, ys = x.new_zeros(b, nh, p, n), []
    for i in range(0, s, 64):
        e = min(s, i + 64)
        cum = da[:, i:e].cumsum(1).transpose(1, 2)                                   # [b, h, t]
        Bc, Cc, Xc = (t[:, i:e].transpose(1, 2) for t in (B, C, xd))                 # [b, h, t, .]
        low = torch.ones(e - i, e - i, dtype=torch.bool, device=x.device).tril()
        L = torch.where(low, (cum.unsqueeze(-1) - cum.unsqueeze(-2)).masked_fill(~low, 0.0).exp(), 0.0)
        y = (Cc @ Bc.transpose(-1, -2) * L) @ Xc + cum.exp().unsqueeze(-1) * (Cc @ S.transpose(-1, -2))
        S = S * cum[..., -1].exp()[..., None, None] + (Xc * (cum[..., -1:] - cum).exp().unsqueeze(-1)).transpose(-1, -2) @ Bc
        ys.append(y.transpose(1, 2))
    y = torch.cat(ys, 1) + xs * w["D"].view(1, 1, nh, 1)
    y = (y.reshape(b, s, di) * F.silu(z)).view(b, s, ng, di // ng)
    y = (y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5)).view(b, s, di) * w["norm_weight"]
    return F.linear(y, w["out_proj.weight"]).transpose(0, 1)


def _moe64(x, w, c):
    t = x.reshape(-1, c["hidden"])
    logits = F.linear(t, w["router.weight"])
    top, idx = logits.topk(c["topk"], dim=-1)
    pr = torch.softmax(top, -1)
    f, out = c["ffn"], torch.zeros_like(t)
    for e in range(c["experts"]):
        rows, slot = (idx == e).nonzero(as_tuple=True)
        a, u = F.linear(t[rows], w["experts.weight1"][e * 2 * f:(e + 1) * 2 * f]).chunk(2, -1)
        y = F.linear(F.silu(a) * u, w["experts.weight2"][e * c["hidden"]:(e + 1) * c["hidden"]])
        out = out.index_add(0, rows, y * pr[rows, slot].unsqueeze(-1))
    return out.view(x.shape)


def exact(case, seed):
    c, st = case, prepare(case, seed)
    kind = c["kind"]
    if kind == "norm":
        ins = [t.detach().double().requires_grad_() for t in (st["x"], st["gamma"], st["beta"]) if t is not None]
        y = _norm64(ins[0], ins[1], ins[2] if len(ins) > 2 else None, c["rms"])
        return [y.detach(), *torch.autograd.grad(y, ins, st["dy"].double())]
    if kind == "attention":
        s, b, d, scale = c["s"], c["b"], c["d"], c["d"] ** -0.5
        if c["packed"]:
            q, k, v = st["mixed"].detach().split(d, dim=-1)
        else:
            q, k, v = st["q"].detach(), st["k"].detach(), st["v"].detach()
        o = torch.empty(s, b, c["hq"], d, dtype=torch.float64, device="cuda")
        dq, dk, dv = torch.empty_like(o), *(torch.zeros(s, b, c["hkv"], d, dtype=torch.float64, device="cuda") for _ in range(2))
        for i in range(b):
            for h in range(c["hq"]):
                hk = h // (c["hq"] // c["hkv"])
                r = _attn64(q[:, i, h].double(), k[:, i, hk].double(), v[:, i, hk].double(), scale, st["do"][:, i, h].double() if c["train"] else None)
                o[:, i, h] = r[0]
                if c["train"]:
                    dq[:, i, h] = r[1]
                    dk[:, i, hk] += r[2]
                    dv[:, i, hk] += r[3]
        if not c["train"]:
            return [o]
        return [o, torch.cat([dq, dk, dv], dim=-1)] if c["packed"] else [o, dq, dk, dv]
    if kind == "paged":
        cx, kc, vc = st["cx"], st["kc"].clone(), st["vc"].clone()
        kc[cx.write_slots], vc[cx.write_slots] = st["k"], st["v"]
        o = torch.empty(st["q"].shape, dtype=torch.float64, device="cuda")
        t0, rep = 0, c["hq"] // c["hkv"]
        for i, (L, m) in enumerate(zip(st["ctx"], st["new"])):
            blocks = torch.tensor(cx.seqs[str(i)].blocks, device="cuda")
            slots = (blocks.unsqueeze(1) * c["block"] + torch.arange(c["block"], device="cuda")).view(-1)[:L + m]
            vis = torch.arange(L + 1, L + m + 1, device="cuda")
            kk, vv = kc[slots].double(), vc[slots].double()
            for h in range(c["hq"]):
                o[t0:t0 + m, h] = _attn64(st["q"][t0:t0 + m, h].double(), kk[:, h // rep], vv[:, h // rep], c["d"] ** -0.5, visible=vis)[0]
            t0 += m
        return [o, kc.double(), vc.double()]
    mod = st["mod"].module if c.get("train", True) else st["mod"]
    w = {n: p.detach().double().requires_grad_(c.get("train", True)) for n, p in mod.named_parameters()}
    if kind == "gpt":
        x = F.embedding(st["tokens"], w["embedding.word_embeddings.weight"])
        rot = None
        if c["rope"]:
            inv = 1.0 / (10000.0 ** (torch.arange(0, 64, 2, dtype=torch.float64, device="cuda") / 64))
            ang = torch.outer(torch.arange(c["s"], dtype=torch.float64, device="cuda"), inv)
            rot = torch.cat([ang.cos(), ang.sin()], -1)
        else:
            x = x + F.embedding(st["pos"], w["embedding.position_embeddings.weight"])
        x = x.transpose(0, 1)
        for i in range(c["layers"]):
            x = _block64(x, w, f"decoder.layers.{i}.", c["heads"], c["heads"], False, False, rot)
        x = _norm64(x, w["decoder.final_layernorm.weight"], w["decoder.final_layernorm.bias"], False)
        logits = F.linear(x, w["embedding.word_embeddings.weight"]).transpose(0, 1)
        if not c["train"]:
            return logits
        loss = F.cross_entropy(logits.reshape(-1, c["vocab"]), st["labels"].reshape(-1), reduction="none").view(c["b"], c["s"])
        gr = torch.autograd.grad(loss, list(w.values()), st["dl"].double())
        return dict(loss=loss.detach(), grads=dict(zip(w, gr)))
    x = st["x"].detach().double().requires_grad_(c.get("train", True))
    if kind == "layer":
        y = _block64(x, w, "", c["heads"], c["groups"], c["swiglu"], c["rms"], st["rot"])
    else:
        y = _mamba64(x, w, c) if kind == "mamba" else _moe64(x, w, c)
    if not c.get("train", True):
        return y
    gr = torch.autograd.grad(y, [x, *w.values()], st["dy"].double())
    return dict(y=y.detach(), dx=gr[0], grads=dict(zip(w, gr[1:])))
