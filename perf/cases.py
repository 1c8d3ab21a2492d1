"""The measured work of this framework: training steps, embedding batches and generation requests over the package's own
presets, each through the entry points a user's program calls.

A case is a dict of plain values:
  kind    "train": one optimizer step (`train_step` over `FlatTrainEngine`)
          "embed": a batch of sequence embeddings (`Transformer.forward_embeddings`)
          "request": prompt in, greedy tokens out (`InferenceEngine.reset`, `prefill`, `decode`)
  preset  a well-known model; `layers` of its blocks (its own pattern repeats, so a part of the stack has the same work
          per block; the 7B, MoE and Mamba-1536 stacks are cut so that several copies fit one card)
  batch, seq (prompt length for a request), decode (tokens generated), optimizer, weights ("bf16" or "int4")
"""
import math

import numpy as np
import torch

from summa_b200 import mal
from summa_b200.models import Transformer
from summa_b200.models.engine import InferenceEngine
from summa_b200.models.quantized import quantize_model_int4
from summa_b200.train.engine import FlatTrainEngine, OptimConfig, train_step


def _train(name, preset, layers, batch, seq, optimizer):
    return {"name": name, "kind": "train", "preset": preset, "layers": layers, "batch": batch, "seq": seq, "optimizer": optimizer}


def _request(name, preset, layers, batch, seq, decode, weights):
    return {"name": name, "kind": "request", "preset": preset, "layers": layers, "batch": batch, "seq": seq, "decode": decode,
            "weights": weights}


def listed():
    return [
        # a smoke-sized model, as in a unit test or a first look at a recipe: launches and host work
        _train("train_tiny", "bench_tiny", 2, 8, 128, "adamw"),
        # the headline benchmark's step
        _train("train_dense", "llama_350m", 24, 8, 2048, "adamw"),
        # a fine-tune on odd lengths with the trainer's default optimizer
        _train("train_dense_odd", "llama_350m", 12, 3, 779, "muon"),
        # long-context pretraining of the hybrid stack (five Mamba blocks and one attention block of it)
        _train("train_hybrid", "hybrid_mamba_1536", 6, 2, 8192, "adamw"),
        # one micro-batch of the retriever pretraining recipe
        _train("train_retriever", "retriever_100m", 24, 27, 1024, "adamw"),
        # MoE pretraining: 64 experts, top 4
        _train("train_moe", "moe_64e_top4", 2, 4, 4096, "adamw"),
        # documents of a few hundred tokens being indexed with the MoE retriever
        {"name": "embed_moe", "kind": "embed", "preset": "retriever_200m_moe", "layers": 24, "batch": 24, "seq": 301},
        # a long prompt, one token back: time to first token with 4-bit weights
        _request("prefill_int4", "dense_7b_gqa", 8, 1, 2048, 1, "int4"),
        # one user chatting with a 4-bit model
        _request("chat_int4", "dense_7b_gqa", 8, 1, 437, 64, "int4"),
        # a full batch of short prompts on a serving box
        _request("serve_int4", "dense_7b_gqa", 8, 64, 128, 48, "int4"),
        # a few users on unquantised weights
        _request("serve_bf16", "dense_7b_gqa", 8, 6, 333, 32, "bf16"),
        # one user generating with the hybrid stack: recurrent and KV state, one token at a time
        _request("chat_hybrid", "hybrid_mamba_1536", 6, 1, 77, 24, "bf16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _batch_seq(rng, seq_lo, seq_hi, batch_hi, tokens_lo, tokens_hi):
    """Any length of the range, and as many rows as make a total of `tokens_lo .. tokens_hi` (spread over its logarithm)."""
    seq = _log_int(rng, seq_lo, seq_hi)
    total = _log_int(rng, max(tokens_lo, seq), tokens_hi)
    return max(1, min(batch_hi, total // seq)), seq


def draw(rng):
    what = rng.choice(["dense", "hybrid", "retriever", "moe", "embed", "request", "request", "request_hybrid"])
    optimizer = rng.choice(["adamw", "muon"])
    if what == "dense":
        b, s = _batch_seq(rng, 48, 2048, 64, 512, 16384)
        c = _train("", "llama_350m", rng.choice([4, 8, 12, 24]), b, s, optimizer)
    elif what == "hybrid":
        b, s = _batch_seq(rng, 256, 8192, 16, 2048, 16384)
        c = _train("", "hybrid_mamba_1536", 6, b, s, optimizer)
    elif what == "retriever":
        b, s = _batch_seq(rng, 64, 1024, 64, 2048, 27648)
        c = _train("", "retriever_100m", rng.choice([6, 12, 24]), b, s, optimizer)
    elif what == "moe":
        b, s = _batch_seq(rng, 128, 4096, 32, 1024, 16384)
        c = _train("", "moe_64e_top4", rng.choice([1, 2]), b, s, "adamw")
    elif what == "embed":
        b, s = _batch_seq(rng, 16, 512, 64, 64, 16384)
        c = {"kind": "embed", "preset": rng.choice(["retriever_100m", "retriever_200m_moe"]), "layers": 24, "batch": b, "seq": s}
    elif what == "request":
        b = _log_int(rng, 1, 64)
        c = _request("", "dense_7b_gqa", rng.choice([4, 8]), b, _log_int(rng, 16, min(2048, 8192 // b)), _log_int(rng, 2, 48),
                     rng.choice(["int4", "bf16"]))
    else:
        b = _log_int(rng, 1, 8)
        c = _request("", "hybrid_mamba_1536", 6, b, _log_int(rng, 8, 1000 // b), _log_int(rng, 4, 24), "bf16")
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs

def _model_def(case):
    cfg = mal.get_builtin_model(case["preset"])
    cfg.num_layers = case["layers"]
    cfg.max_seq_len = max(cfg.max_seq_len, case["seq"] + case.get("decode", 0) + 8)
    return cfg


def _tokens(cfg, batch, seq, gen):
    """Zipf(1.1) ids, as text has (through the inverse of the distribution: the same ids for the same seed)."""
    cdf = np.cumsum(np.arange(1, cfg.vocab_size + 1, dtype=np.float64) ** -1.1)
    u = torch.rand(batch, seq, device="cuda", generator=gen, dtype=torch.float64)
    return torch.searchsorted(torch.from_numpy(cdf / cdf[-1]).to("cuda"), u).clamp_(max=cfg.vocab_size - 1)


def _build(case, seed):
    cfg = _model_def(case)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = Transformer(cfg, init_std=0.02)
    return cfg, model, torch.Generator(device="cuda").manual_seed(seed + 1)


@torch.no_grad()
def _trained_stream(model):
    """What training leaves and a random draw does not: a token's embedding that stays visible in the residual stream, and
    branches that add to it rather than drown it."""
    model.embedding.weight.mul_(50.0)
    if model.lm_head is None:                          # tied: the logits keep their size
        model.final_norm.gamma.mul_(1 / 50)
    for name, p in model.named_parameters():
        if name.endswith(("o_proj.weight", "down_proj.weight", "out_proj.weight")) or name.endswith("down_weight"):
            p.mul_(0.25)


@torch.no_grad()
def _routers_by_token(cfg, model, gen):
    """Routers that send a token to experts of its own, as trained ones mostly do. (The routes of a random draw hang on
    the last bit of the hidden state; these do not.)"""
    V = cfg.vocab_size
    for name, p in model.named_parameters():
        if not name.endswith("router.weight"):
            continue
        H, E = p.shape
        k = next(b.ffn.moe.top_k for b in (cfg.block_for_layer(i) for i in range(cfg.num_layers)) if b.ffn.moe is not None)
        p.copy_(torch.linalg.qr(torch.randn(H, E, device="cuda", generator=gen)).Q * (0.02 * H ** 0.5))
        chosen = torch.rand(V, E, device="cuda", generator=gen).topk(k, dim=1).indices
        pull = torch.zeros(V, E, device="cuda").scatter_(1, chosen, 1.0) * (0.35 * H ** 0.5)
        model.embedding.weight[:V] += pull @ (p / (0.02 * H ** 0.5)).t()


@torch.no_grad()
def _head_by_token(cfg, model, gen):
    """A head that is sure of the next token: with the head of a random draw the two best logits are often the same number."""
    V, E = cfg.vocab_size, model.embedding.weight
    follow = torch.randperm(V, device="cuda", generator=gen)
    model.lm_head.weight[:, follow] = 0.02 * E[:V].t()


def prepare(case, seed):
    cfg, model, gen = _build(case, seed)
    _trained_stream(model)
    _routers_by_token(cfg, model, gen)
    if case["kind"] == "train":
        model.stream_dtype = torch.bfloat16
        engine = FlatTrainEngine(model, OptimConfig(lr=3e-4), muon=case["optimizer"] == "muon")
        model.train()
        at = engine.offsets
        blocks = slice(min(o for n, o in at.items() if n.startswith("layers.")), at.get("lm_head.weight", engine.numel))
        return {"kind": "train", "model": model, "engine": engine, "blocks": blocks, "tokens": _tokens(cfg, case["batch"], case["seq"] + 1, gen)}
    if case["kind"] == "embed":
        model.prepare_inference(torch.bfloat16)
        ends = torch.randint(case["seq"] // 2, case["seq"], (case["batch"],), device="cuda", generator=gen)
        return {"kind": "embed", "model": model, "tokens": _tokens(cfg, case["batch"], case["seq"], gen), "ends": ends}
    _head_by_token(cfg, model, gen)
    model.prepare_inference(torch.bfloat16)
    if case["weights"] == "int4":
        quantize_model_int4(model, include_head=True)
    return {"kind": "request", "engine": InferenceEngine(model), "prompt": _tokens(cfg, case["batch"], case["seq"], gen),
            "decode": case["decode"], "capacity": case["seq"] + case["decode"] + 8}


def run(state):
    if state["kind"] == "train":
        engine, tokens = state["engine"], state["tokens"]
        loss, norm = train_step(state["model"], engine, tokens[:, :-1], tokens[:, 1:])
        out = {"loss": loss, "norm": norm, "master": engine.master, "small": engine.small_params,
               "small_exp_avg": engine.small_exp_avg}
        if engine.muon is not None:
            out["velocity"] = dict(engine.muon.velocity)
        else:
            # The first moments of the blocks are their gradients. (Those of the two vocabulary tables are left to the
            # updated weights: a frequent token's row is a hundred times the others', and its rounding too.)
            out["exp_avg"] = engine.exp_avg[state["blocks"]]
        return out
    if state["kind"] == "embed":
        with torch.no_grad():
            return state["model"].forward_embeddings(state["tokens"], state["ends"])
    engine = state["engine"]
    engine.reset(state["prompt"].shape[0], state["capacity"])
    first = engine.prefill(state["prompt"])
    return {"first": first, "tokens": engine.decode(first, state["decode"]), "state": [vars(s) for s in engine.state.layers]}


# ------------------------------------------------------------------ what a pass cannot do without

def _shape(cfg):
    """Per token: (matrix weights used, matrix weights stored, attention layers as (q heads, kv heads, head dim), scan state
    elements), the head counted among the weights and the embedding table not."""
    H = cfg.hidden_size
    used = stored = 0
    attn, scan = [], 0
    for i in range(cfg.num_layers):
        b = cfg.block_for_layer(i)
        if b.ssm is not None:
            di, n, r = b.ssm.expand * H, b.ssm.state_dim, cfg.dt_rank(b.ssm)
            w = H * 2 * di + di * (r + 2 * n) + r * di + di * H
            scan += di * n
        else:
            hq, hk, d = b.num_heads(), b.num_kv_heads(), b.head_dim(H)
            w = H * (hq + 2 * hk) * d + hq * d * H
            attn.append((hq, hk, d))
        inter = b.ffn.hidden_dim
        one = H * inter * (3 if b.ffn.gate else 2)
        m = b.ffn.moe
        used += w + (one * m.top_k + H * m.experts if m is not None else one)
        stored += w + (one * m.experts + H * m.experts if m is not None else one)
    return used, stored, attn, scan


def work(case):
    cfg = _model_def(case)
    B, S, H, V = case["batch"], case["seq"], cfg.hidden_size, cfg.vocab_size
    used, stored, attn, scan = _shape(cfg)
    T = B * S
    head = H * V
    pairs = B * S * (S + 1) // 2                       # causal (query, key) pairs
    attn_flops = sum(4 * hq * d for hq, _, d in attn)  # per pair
    if case["kind"] == "train":
        params = stored + head * (1 if cfg.embeddings.tie_weights else 2)
        # master and two moments in and out, bf16 copy in and out; an untied embedding table is among them
        return {"bytes": params * 28 + T * 16, "flops": 3 * (2 * T * (used + head) + pairs * attn_flops) + 18 * T * scan}
    if case["kind"] == "embed":
        return {"bytes": stored * 2 + T * (8 + 2 * H) + B * H * 4, "flops": 2 * T * used + pairs * attn_flops + 6 * T * scan}
    n = case["decode"]
    per_weight = 2.0 if case["weights"] == "bf16" else 0.5 + 2 / 128
    kv = sum(2 * hk * d * 2 for _, hk, d in attn)      # bytes a cached position
    reads = sum(B * (S + t) for t in range(n)) * kv    # a decode step reads the whole cache
    rec = 2 * 4 * B * scan * n                         # and the recurrent state both ways
    return {"bytes": (n + 1) * (stored + head) * per_weight + reads + T * kv + rec,
            "flops": 2 * T * used + pairs * attn_flops + 2 * B * n * (used + head) + 2 * B * head + 6 * T * scan}


def tolerance(case):
    """Measured on shortened cases: the same step through stock PyTorch ops in bf16 differs by 0.005 (dense, AdamW and Muon),
    a computation in fp32 from the same bf16 weights by 0.003 (MoE, tiny), 0.008 (dense), 0.011 (Mamba-1536), 0.013
    (retriever), 0.011 (caches of the eighth 7B block, embeddings of the 24th block); largest single differences are
    0.03 to 0.3 of the root mean square."""
    return {"rel": 1e-2} if case["preset"] in ("moe_64e_top4", "bench_tiny") else {"rel": 2e-2}
