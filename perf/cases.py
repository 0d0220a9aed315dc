"""Measured work of the framework: single layers and blocks of the two model families, the RL loss, the optimizer,
a whole training pass and a short generation, each through the entry point that a trainer or a rollout worker calls.

Head layouts: ``hybrid`` is the full-attention layer of the Qwen3.5-0.8B shape (8 query heads, 2 key / value heads, head
dim 256), ``moe`` that of the Qwen3-30B-A3B shape (32, 4, 128).  Trainers run equal-length packed sequences of any
length; lengths that are no multiple of a tile are as common as the benchmark's 1280.
"""
import math

import torch
import torch.nn.functional as F

from cverl_b200 import ops
from cverl_b200.models.config import Qwen35TextConfig
from cverl_b200.models.decode import decode_step, prefill
from cverl_b200.models.qwen3_5 import Qwen35Model
from cverl_b200.ops import gdn, rl
from cverl_b200.ops.attention import causal_attention
from cverl_b200.ops.optim import clip_scale, sumsq
from cverl_b200.optim.adamw import AdamWOptions, FlatAdamW

HEADS = {"hybrid": (8, 2, 256), "moe": (32, 4, 128)}
GDN_HEADS, GDN_DIM = 16, 128
VOCAB = 248320          # vocabulary of the Qwen3.5-0.8B shape
HIDDEN, FFN = 1024, 3584
EPS = 1e-6
DEV = "cuda"


# ------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # loss of one small GRPO step: 64 responses of 512 tokens
        {"name": "loss_64x512", "kind": "loss", "rows": 64, "cols": 512},
        # the two norms of every layer on a training micro-batch
        {"name": "norm_train_32x1280", "kind": "norm", "tokens": 32 * 1280},
        # full-attention core of the benchmark's micro-batch, forward and backward
        {"name": "attn_train_16x1280", "kind": "attn", "heads": "hybrid", "batch": 16, "seq": 1280, "train": True},
        # the same kernels on the mixture-of-experts shape, at a length that comes from real prompts
        {"name": "attn_train_moe_4x1500", "kind": "attn", "heads": "moe", "batch": 4, "seq": 1500, "train": True},
        # prompt scoring (reference policy, prefill): forward only, short ragged sequences
        {"name": "attn_infer_24x333", "kind": "attn", "heads": "hybrid", "batch": 24, "seq": 333, "train": False},
        # Gated-DeltaNet core of the benchmark's micro-batch, forward and backward
        {"name": "gdn_train_16x1280", "kind": "gdn", "batch": 16, "seq": 1280, "train": True},
        # SwiGLU block of a dense layer
        {"name": "mlp_train_20480", "kind": "mlp", "tokens": 20480},
        # response log-probabilities under the 248,320-wide head, forward and backward
        {"name": "lmhead_train_4096", "kind": "lmhead", "rows": 4096},
        # one mixture-of-experts layer: router, dispatch, grouped GEMMs, combine
        {"name": "moe_train_4096", "kind": "moe", "tokens": 4096},
        # gradient norm, clipping and AdamW on a flat shard
        {"name": "adamw_64m", "kind": "adamw", "numel": 1 << 26},
        # a whole training pass of a two-layer hybrid model on ragged sequences (log-probabilities and gradients)
        {"name": "model_train_8x1088", "kind": "model", "batch": 8, "seq": 1088, "prompt": 256},
        # rollout: prefill of 32 prompts and the next tokens, fed as given
        {"name": "generate_32x200", "kind": "generate", "batch": 32, "seq": 200, "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loss", "norm", "attn", "attn", "attn", "gdn", "gdn", "mlp", "lmhead", "moe", "adamw", "model",
                       "generate"])
    if kind == "loss":
        return {"kind": kind, "rows": _log(rng, 8, 1024), "cols": _log(rng, 32, 1024)}
    if kind in ("norm", "mlp"):
        return {"kind": kind, "tokens": _log(rng, 64, 20480)}
    if kind == "attn":
        seq = _log(rng, 48, 3000)
        if rng.random() < 0.4:
            seq = (seq + 127) // 128 * 128
        heads = rng.choice(["hybrid", "moe"])
        room = (16 * 1280 * 1280 if heads == "hybrid" else 4 * 1500 * 1500) // (seq * seq)
        return {"kind": kind, "heads": heads, "batch": _log(rng, 1, max(1, min(64, room))), "seq": seq,
                "train": rng.random() < 0.7}
    if kind == "gdn":
        seq = 64 * _log(rng, 1, 32)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 20480 // seq)), "seq": seq, "train": rng.random() < 0.7}
    if kind == "lmhead":
        return {"kind": kind, "rows": _log(rng, 32, 4096)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 64, 4096)}
    if kind == "adamw":
        return {"kind": kind, "numel": _log(rng, 1 << 16, 1 << 26)}
    if kind == "model":
        seq = 64 * _log(rng, 4, 20)
        return {"kind": kind, "batch": _log(rng, 1, max(1, 8704 // seq)), "seq": seq,
                "prompt": rng.randint(1, seq // 2)}
    return {"kind": kind, "batch": _log(rng, 1, 64), "seq": _log(rng, 16, 400), "steps": rng.randint(1, 6)}


# ------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed * 7919 + 17)


def _bf(g, *shape, scale=1.0):
    return (torch.randn(*shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


def _config(kind):
    if kind == "moe":      # one layer of the 30B-A3B shape; the vocabulary is not used by the layer
        return Qwen35TextConfig(model_type="qwen3_moe", vocab_size=512, hidden_size=2048, num_hidden_layers=1,
                                num_attention_heads=32, num_key_value_heads=4, head_dim=128, intermediate_size=6144,
                                moe_intermediate_size=768, num_experts=128, num_experts_per_tok=8, rope_theta=1e6,
                                tie_word_embeddings=False)
    if kind == "mlp":
        return Qwen35TextConfig(vocab_size=512, num_hidden_layers=1, layer_types=["linear_attention"])
    vocab = VOCAB if kind == "generate" else 32768
    return Qwen35TextConfig(vocab_size=vocab, num_hidden_layers=2, layer_types=["linear_attention", "full_attention"])


def _model(kind, seed):
    m = Qwen35Model(_config(kind), dtype=torch.bfloat16, device=DEV, with_main_grad=kind != "generate")
    m.init_weights_on_device(seed=seed)
    return m


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case}
    if kind == "loss":
        R, C = case["rows"], case["cols"]
        lens = torch.randint(max(1, C // 16), C + 1, (R, 1), device=DEV, generator=g)
        s["mask"] = (torch.arange(C, device=DEV)[None, :] < lens).float()
        s["lp"] = -2 + 0.5 * torch.randn(R, C, device=DEV, generator=g)
        s["old"] = s["lp"] + 0.05 * torch.randn(R, C, device=DEV, generator=g)
        s["ref"] = s["lp"] + 0.1 * torch.randn(R, C, device=DEV, generator=g)
        won = (torch.rand(R, 1, device=DEV, generator=g) < 0.5).float()
        s["rewards"] = torch.zeros(R, C, device=DEV).scatter_(1, lens - 1, won)
        s["groups"] = torch.arange(R, device=DEV) // 8
    elif kind == "norm":
        T = case["tokens"]
        s["x"], s["r"] = (_bf(g, T, HIDDEN).requires_grad_(True) for _ in range(2))
        s["w"] = _bf(g, HIDDEN, scale=0.1).requires_grad_(True)
        s["w"].main_grad = torch.zeros(HIDDEN, device=DEV)
        s["dy"], s["dh"] = _bf(g, T, HIDDEN), _bf(g, T, HIDDEN)
    elif kind == "attn":
        (Hq, Hkv, D), T = HEADS[case["heads"]], case["batch"] * case["seq"]
        s["q"], s["k"], s["v"] = (_bf(g, T, h, D).requires_grad_(case["train"]) for h in (Hq, Hkv, Hkv))
        s["do"] = _bf(g, T, Hq, D)
    elif kind == "gdn":
        B, S = case["batch"], case["seq"]
        s["mixed"] = F.silu(_bf(g, B, S, 3 * GDN_HEADS * GDN_DIM)).requires_grad_(case["train"])
        s["beta"] = torch.sigmoid(torch.randn(B, S, GDN_HEADS, device=DEV, generator=g)).requires_grad_(case["train"])
        rate = 1 + 7 * torch.rand(GDN_HEADS, device=DEV, generator=g)
        s["g"] = (-rate * F.softplus(torch.randn(B, S, GDN_HEADS, device=DEV, generator=g) - 3)).requires_grad_(
            case["train"])
        s["do"] = _bf(g, B, S, GDN_HEADS, GDN_DIM)
    elif kind in ("mlp", "moe"):
        s["model"] = _model(kind, seed)
        H = s["model"].cfg.hidden_size
        s["x"] = _bf(g, case["tokens"], H).requires_grad_(True)
        s["dy"] = _bf(g, case["tokens"], H)
    elif kind == "lmhead":
        R = case["rows"]
        s["h"] = _bf(g, R, HIDDEN).requires_grad_(True)
        s["e"] = _bf(g, VOCAB, HIDDEN, scale=0.02).requires_grad_(True)
        s["e"].main_grad = torch.zeros(VOCAB, HIDDEN, device=DEV)
        s["t"] = torch.randint(0, VOCAB, (R,), device=DEV, generator=g)
        s["dlp"] = torch.randn(R, device=DEV, generator=g) / R
    elif kind == "adamw":
        n = case["numel"]
        s["p"] = _bf(g, n, scale=0.02)
        s["grad"] = 1e-3 * torch.randn(n, device=DEV, generator=g)
        s["opt"] = FlatAdamW(s["p"], AdamWOptions(lr=1e-4, weight_decay=0.01))
    elif kind in ("model", "generate"):
        s["model"] = _model(kind, seed)
        V = s["model"].cfg.vocab_size
        s["ids"] = torch.randint(1, V, (case["batch"], case["seq"]), device=DEV, generator=g)
        if kind == "model":
            s["dlp"] = torch.randn(case["batch"], case["seq"] - case["prompt"], device=DEV, generator=g) / case["batch"]
        else:
            s["next"] = torch.randint(1, V, (case["steps"], case["batch"]), device=DEV, generator=g)
    return s


# ------------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "loss":
        adv, _ = rl.fused_grpo_advantage(s["rewards"], s["mask"], s["groups"])
        metrics, grad = rl.fused_ppo_loss(s["old"], s["lp"], adv, s["mask"], s["ref"], kl_coef=0.01,
                                          kl_penalty_kind="k3")
        return adv, metrics, grad
    if kind == "norm":
        s["w"].main_grad.zero_()
        y, h = ops.add_rmsnorm(s["x"], s["r"], s["w"], EPS, 1.0)
        (dx, _) = _backward((y, h), (s["dy"], s["dh"]), s["x"], s["r"])
        return y.detach(), h.detach(), dx, s["w"].main_grad
    if kind == "attn":
        if not case["train"]:
            with torch.no_grad():
                return causal_attention(s["q"], s["k"], s["v"], case["batch"], case["seq"])
        o = causal_attention(s["q"], s["k"], s["v"], case["batch"], case["seq"])
        return (o.detach(),) + _backward((o,), (s["do"],), s["q"], s["k"], s["v"])
    if kind == "gdn":
        scale = GDN_DIM ** -0.5
        if not case["train"]:
            with torch.no_grad():
                return gdn.gated_delta_rule_packed(s["mixed"], s["beta"], s["g"], scale=scale, heads=GDN_HEADS)
        o, state = gdn.gated_delta_rule_packed(s["mixed"], s["beta"], s["g"], scale=scale, heads=GDN_HEADS)
        return (o.detach(), state.detach()) + _backward((o,), (s["do"],), s["mixed"], s["beta"], s["g"])
    if kind in ("mlp", "moe"):
        model = s["model"]
        model.flat.main_grad.zero_()
        y = model.mlp(s["x"], 0)
        return (y.detach(),) + _backward((y,), (s["dy"],), s["x"]) + tuple(w.main_grad for w in _ffn_weights(model))
    if kind == "lmhead":
        s["e"].main_grad.zero_()
        lp = ops.lmhead_logprob(s["h"], s["e"], s["t"])
        (dh,) = _backward((lp,), (s["dlp"],), s["h"])
        return lp.detach(), dh, s["e"].main_grad
    if kind == "adamw":
        sq = sumsq(s["grad"])
        s["opt"].step(s["grad"], clip=clip_scale(sq, 1.0))
        return sq, s["p"], s["opt"].parameter_shard, s["opt"].exp_avg, s["opt"].exp_avg_sq
    if kind == "model":
        model = s["model"]
        model.flat.main_grad.zero_()
        lp = model.response_logprobs(s["ids"], case["prompt"])
        lp.backward(s["dlp"])
        return (lp.detach(),) + tuple(model.param(n).main_grad for n in _grad_names(model))
    state, logits = prefill(s["model"], s["ids"], case["seq"] + case["steps"])
    out = [logits]
    for tok in s["next"]:
        out.append(decode_step(s["model"], state, tok))
    return out


def _backward(outs, grads, *leaves):
    """Backward pass as a trainer runs it: parameters collect into ``main_grad``, the leaves' gradients come back."""
    for x in leaves:
        x.grad = None
    torch.autograd.backward(outs, grads)
    return tuple(x.grad for x in leaves)


def _ffn_weights(model):
    if model.cfg.is_qwen3_moe:
        return [model.param("model.layers.0.mlp.gate.weight"), model.param("__packed_moe.layers.0.gate_up.weight"),
                model.param("__packed_moe.layers.0.down.weight")]
    return [model.fused["0.gate_up"], model.param(model.cfg.layer_root + "0.mlp.down_proj.weight")]


def _grad_names(model):
    """The matrices of the two layers, the embedding and the norms: gradients of every kind that the model has."""
    root = model.cfg.layer_root
    la, sa = root + "0.linear_attn.", root + "1.self_attn."
    return [model.cfg.embed_name, la + "in_proj_qkv.weight", la + "in_proj_z.weight", la + "out_proj.weight",
            sa + "q_proj.weight", sa + "k_proj.weight", sa + "v_proj.weight", sa + "o_proj.weight",
            root + "0.mlp.gate_proj.weight", root + "0.mlp.down_proj.weight", root + "1.mlp.up_proj.weight",
            root + "1.mlp.down_proj.weight", model.cfg.final_norm_name]


# ------------------------------------------------------------------------------------------------- its least cost
def work(case):
    kind = case["kind"]
    if kind == "loss":
        n = case["rows"] * case["cols"]
        return {"bytes": 4 * n * 7, "flops": 40 * n}
    if kind == "norm":
        n = case["tokens"] * HIDDEN
        return {"bytes": 2 * n * 7, "flops": 20 * n}
    if kind == "attn":
        (Hq, Hkv, D), B, S = HEADS[case["heads"]], case["batch"], case["seq"]
        fwd = 4 * B * Hq * D * S * (S + 1) / 2
        qo, kv = 2 * B * S * Hq * D, 2 * B * S * Hkv * D
        if not case["train"]:
            return {"bytes": 2 * qo + 2 * kv, "flops": fwd}
        return {"bytes": 4 * qo + 4 * kv, "flops": 3.5 * fwd}
    if kind == "gdn":
        n = case["batch"] * case["seq"] * GDN_HEADS
        # recurrence in chunks of 64: scores, W, U, outputs and state updates
        fwd = 2 * n * (64 * GDN_DIM * 5 + 3 * GDN_DIM * GDN_DIM)
        return {"bytes": 2 * n * GDN_DIM * (8 if case["train"] else 4) + 8 * n * (2 if case["train"] else 1),
                "flops": fwd * (3 if case["train"] else 1)}
    if kind == "mlp":
        T = case["tokens"]
        return {"bytes": 2 * (4 * T * HIDDEN) + 3 * HIDDEN * FFN * (2 + 4), "flops": 3 * 6 * T * HIDDEN * FFN}
    if kind == "moe":
        T, H, I, E, k = case["tokens"], 2048, 768, 128, 8
        used = min(E, T * k)
        return {"bytes": 2 * 4 * T * H + 3 * H * I * (2 * used + 4 * E), "flops": 3 * 6 * T * k * H * I}
    if kind == "lmhead":
        R = case["rows"]
        return {"bytes": 2 * 2 * R * HIDDEN + VOCAB * HIDDEN * (2 + 4), "flops": 3 * 2 * R * HIDDEN * VOCAB}
    if kind == "adamw":
        return {"bytes": case["numel"] * (4 + 4 + 2 + 8 + 8 + 4), "flops": 20 * case["numel"]}
    T = case["batch"] * case["seq"]
    per_token = 2 * (HIDDEN * (8224 + 2048 + 5120 + 2048) + 2 * 3 * HIDDEN * FFN)
    attn = 4 * case["batch"] * 8 * 256 * case["seq"] ** 2 / 2 + 2 * T * 16 * (64 * 128 * 5 + 3 * 128 * 128)
    weights = HIDDEN * (8224 + 2048 + 5120 + 2048) + 2 * 3 * HIDDEN * FFN
    if kind == "model":
        R = case["batch"] * (case["seq"] - case["prompt"])
        return {"bytes": (weights + 32768 * HIDDEN) * (2 + 4),
                "flops": 3 * (T * per_token + 2 * R * HIDDEN * 32768) + 3.5 * attn}
    n = case["steps"] + 1
    return {"bytes": n * (2 * (weights + VOCAB * HIDDEN) + 4 * case["batch"] * VOCAB),
            "flops": (T + case["batch"] * case["steps"]) * per_token + attn + n * 2 * case["batch"] * HIDDEN * VOCAB}


def tolerance(case):
    # bf16 results: about half a unit in the last place per rounding, a few roundings in a row
    return {"loss": {"rel": 1e-5}, "adamw": {"rel": 3e-3}, "norm": {"rel": 6e-3}, "attn": {"rel": 1.2e-2},
            "gdn": {"rel": 2e-2}, "mlp": {"rel": 1.2e-2}, "lmhead": {"rel": 1e-2}, "moe": {"rel": 1.5e-2},
            "model": {"rel": 6e-2}, "generate": {"rel": 4e-2}}[case["kind"]]


# ------------------------------------------------------------------------------------------------- 64-bit statement
def _norm64(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _attn64(q, k, v, B, S):
    T, Hq, D = q.shape
    n = Hq // k.shape[1]
    out = []
    mask = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    for b in range(B):
        r = slice(b * S, (b + 1) * S)
        kk, vv = (t[r].transpose(0, 1).repeat_interleave(n, 0) for t in (k, v))
        p = (q[r].transpose(0, 1) @ kk.transpose(1, 2)) / math.sqrt(D)
        out.append((torch.softmax(p.masked_fill(mask, float("-inf")), -1) @ vv).transpose(0, 1))
    return torch.cat(out)


def _gdn64(mixed, beta, g):
    """mixed [B, S, 3 * 16 * 128], beta, g [B, S, 16]: the recurrence, token by token."""
    B, S, _ = mixed.shape
    q, k, v = mixed.view(B, S, 3, GDN_HEADS, GDN_DIM).unbind(2)
    q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * GDN_DIM ** -0.5
    k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    e = torch.exp(g)
    state = mixed.new_zeros(B, GDN_HEADS, GDN_DIM, GDN_DIM)
    outs = []
    for t in range(S):
        state = state * e[:, t, :, None, None]
        kt = k[:, t]
        seen = torch.einsum("bhkv,bhk->bhv", state, kt)
        state = state + kt.unsqueeze(-1) * ((v[:, t] - seen) * beta[:, t].unsqueeze(-1)).unsqueeze(-2)
        outs.append(torch.einsum("bhkv,bhk->bhv", state, q[:, t]))
    return torch.stack(outs, 1), state


def _layers64(model, ids, w):
    """Final-normed hidden states [B, S, H] of the two-layer hybrid model; ``w`` maps names to 64-bit weights."""
    cfg = model.cfg
    B, S = ids.shape
    root = cfg.layer_root
    x = w[cfg.embed_name][ids.reshape(-1)]

    def mlp(h, i):
        p = f"{root}{i}.mlp."
        n = _norm64(h, 1 + w[f"{root}{i}.post_attention_layernorm.weight"])
        return h + (F.silu(n @ w[p + "gate_proj.weight"].t()) * (n @ w[p + "up_proj.weight"].t())) @ w[
            p + "down_proj.weight"].t()

    n, p = _norm64(x, 1 + w[root + "0.input_layernorm.weight"]), root + "0.linear_attn."
    mixed = (n @ w[p + "in_proj_qkv.weight"].t()).view(B, S, -1)
    conv = w[p + "conv1d.weight"].reshape(mixed.shape[-1], 4)
    mixed = F.silu(sum(F.pad(mixed, (0, 0, 3 - j, 0))[:, :S] * conv[:, j] for j in range(4)))
    beta = torch.sigmoid(n @ w[p + "in_proj_b.weight"].t()).view(B, S, GDN_HEADS)
    g = (-torch.exp(w[p + "A_log"]) * F.softplus(n @ w[p + "in_proj_a.weight"].t() + w[p + "dt_bias"])).view(
        B, S, GDN_HEADS)
    o = torch.cat([_gdn64(mixed[b:b + 8], beta[b:b + 8], g[b:b + 8])[0] for b in range(0, B, 8)])
    z = (n @ w[p + "in_proj_z.weight"].t()).view(B, S, GDN_HEADS, GDN_DIM)
    o = _norm64(o, w[p + "norm.weight"]) * F.silu(z)
    x = mlp(x + o.reshape(B * S, -1) @ w[p + "out_proj.weight"].t(), 0)

    n, p = _norm64(x, 1 + w[root + "1.input_layernorm.weight"]), root + "1.self_attn."
    q, gate = (n @ w[p + "q_proj.weight"].t()).view(-1, 8, 512).split(256, -1)
    k, v = ((n @ w[p + c + "_proj.weight"].t()).view(-1, 2, 256) for c in "kv")
    rot = cfg.rotary_dim
    freq = cfg.rope_theta ** (-torch.arange(0, rot, 2, dtype=torch.float64, device=x.device) / rot)
    ang = (torch.arange(S, dtype=torch.float64, device=x.device)[:, None] * freq).repeat(B, 1).unsqueeze(1)

    def rope(t):
        a, b, rest = t.split([rot // 2, rot // 2, 256 - rot], -1)
        return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), rest], -1)

    q, k = (rope(_norm64(t, 1 + w[p + c + "_norm.weight"])) for t, c in ((q, "q"), (k, "k")))
    o = _attn64(q, k, v, B, S) * torch.sigmoid(gate)
    x = mlp(x + o.reshape(B * S, -1) @ w[p + "o_proj.weight"].t(), 1)
    return _norm64(x, 1 + w[cfg.final_norm_name]).view(B, S, -1)


def _weights64(model, grad):
    return {n: p.detach().double().requires_grad_(grad) for n, p in model.flat.params.items()}


def exact(case, seed):
    kind, s = case["kind"], prepare(case, seed)

    def d(key, grad=False):
        return s[key].detach().double().requires_grad_(grad)

    if kind == "loss":
        mask, lp = d("mask"), d("lp", True)
        score, gid = d("rewards").mul(mask).sum(1), s["groups"]
        n = int(gid.max()) + 1
        cnt = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, gid, torch.ones_like(score))
        mean = torch.zeros_like(cnt).index_add_(0, gid, score) / cnt
        var = torch.zeros_like(cnt).index_add_(0, gid, (score - mean[gid]) ** 2) / (cnt - 1).clamp_min(1)
        single = cnt[gid] < 2
        adv = torch.where(single, score / (1 + 1e-6), (score - mean[gid]) / (var.sqrt()[gid] + 1e-6))
        adv = adv[:, None] * mask
        ratio = torch.exp((lp - d("old")).clamp(-20, 20))
        l1, l2 = -adv * ratio, -adv * ratio.clamp(0.8, 1.2)
        hi = torch.maximum(l1, l2)
        low = torch.minimum(-3.0 * adv, hi)
        tok = mask.sum()
        loss = (torch.where(adv < 0, low, hi) * mask).sum() / tok
        gap = (d("ref") - lp).clamp(-20, 20)
        kl = ((torch.exp(gap) - gap - 1).clamp(-10, 10) * mask).sum() / tok
        (grad,) = torch.autograd.grad(loss + 0.01 * kl, lp)
        frac = ((l2 > l1).double() * mask).sum() / tok
        frac_low = (((hi > -3.0 * adv) & (adv < 0)).double() * mask).sum() / tok
        ppo_kl = ((d("old") - lp) * mask).sum() / tok
        return adv, torch.stack([loss, frac, ppo_kl, frac_low, kl, tok]).detach(), grad
    if kind == "norm":
        x, r, w = d("x", True), d("r", True), d("w", True)
        h = x + r
        # the residual stream is rounded to bf16 before it is normalised
        hb = h.detach().to(torch.bfloat16).double() + (h - h.detach())
        y = _norm64(hb, 1 + w)
        dx, dw = torch.autograd.grad((y, hb), (x, w), (d("dy"), d("dh")))
        return y.detach(), hb.detach(), dx, dw
    if kind == "attn":
        q, k, v = (d(n, case["train"]) for n in "qkv")
        if not case["train"]:
            return _attn64(q, k, v, case["batch"], case["seq"])
        S, outs = case["seq"], []
        for b in range(case["batch"]):
            part = [t.detach()[b * S:(b + 1) * S].requires_grad_(True) for t in (q, k, v)]
            o = _attn64(*part, 1, S)
            outs.append((o.detach(),) + torch.autograd.grad(o, part, d("do")[b * S:(b + 1) * S]))
        return tuple(torch.cat(t) for t in zip(*outs))
    if kind == "gdn":
        if case["train"] and case["batch"] * case["seq"] > 20480:
            return None
        outs = []
        for b in range(case["batch"]):
            part = [s[n].detach()[b:b + 1].double().requires_grad_(case["train"]) for n in ("mixed", "beta", "g")]
            o, state = _gdn64(*part)
            got = (o.detach(), state.detach())
            if case["train"]:
                got += torch.autograd.grad(o, part, s["do"][b:b + 1].double())
            outs.append(got)
        return tuple(torch.cat(t) for t in zip(*outs))
    if kind == "mlp":
        gu, dn = (w.detach().double().requires_grad_(True) for w in _ffn_weights(s["model"]))
        x = d("x", True)
        a, u = (x @ gu.t()).chunk(2, -1)
        y = (F.silu(a) * u) @ dn.t()
        return (y.detach(),) + torch.autograd.grad(y, (x, gu, dn), d("dy"))
    if kind == "moe":
        gate, gu, dn = (w.detach() for w in _ffn_weights(s["model"]))
        gate, x, dy = gate.double().requires_grad_(True), d("x", True), d("dy")
        val, idx = torch.topk(x @ gate.t(), 8, -1)
        p = torch.softmax(val, -1)
        y, dgu, ddn = torch.zeros_like(dy), torch.zeros(gu.shape, device=DEV), torch.zeros(dn.shape, device=DEV)
        dxe, dp = torch.zeros_like(dy), torch.zeros_like(val)
        for e in range(gu.shape[0]):
            tok, slot = (idx == e).nonzero(as_tuple=True)
            if tok.numel() == 0:
                continue
            part = [x.detach()[tok].requires_grad_(True), gu[e].double().requires_grad_(True),
                    dn[e].double().requires_grad_(True), p.detach()[tok, slot].requires_grad_(True)]
            a, u = (part[0] @ part[1].t()).chunk(2, -1)
            o = ((F.silu(a) * u) @ part[2].t()) * part[3][:, None]
            gx, g1, g2, gp = torch.autograd.grad(o, part, dy[tok])
            y.index_add_(0, tok, o.detach())
            dxe.index_add_(0, tok, gx)
            dgu[e], ddn[e] = g1, g2
            dp[tok, slot] = gp
        gx, dgate = torch.autograd.grad(p, (x, gate), dp)
        return y, dxe + gx, dgate, dgu, ddn
    if kind == "lmhead":
        h, dlp, R = d("h"), d("dlp"), case["rows"]
        e = s["e"].detach().double()
        lp, dh, de = [], [], torch.zeros_like(e)
        for r in range(0, R, 512):
            z = torch.log_softmax(h[r:r + 512] @ e.t(), -1)
            t = s["t"][r:r + 512, None]
            lp.append(z.gather(1, t)[:, 0])
            z = -z.exp_() * dlp[r:r + 512, None]
            z.scatter_add_(1, t, dlp[r:r + 512, None])
            dh.append(z @ e)
            de.addmm_(z.t(), h[r:r + 512])
        return torch.cat(lp), torch.cat(dh), de
    if kind == "adamw":
        p, g = d("p"), d("grad")
        o = s["opt"].options
        sq = (g * g).sum()
        norm = sq.sqrt()
        g = g * (1.0 / (norm + 1e-6) if norm > 1.0 else 1.0)
        m, v = (1 - o.beta1) * g, (1 - o.beta2) * g * g
        new = p * (1 - o.lr * o.weight_decay) - o.lr * (m / (1 - o.beta1)) / ((v / (1 - o.beta2)).sqrt() + o.eps)
        return sq.view(1), new, new, m, v
    model, ids = s["model"], s["ids"]
    w = _weights64(model, kind == "model")
    if kind == "model":
        # one sequence at a time: the recurrence keeps a state per token
        P, lps = case["prompt"], []
        for b in range(case["batch"]):
            h = _layers64(model, ids[b:b + 1], w)[0, P - 1:-1]
            lp = torch.log_softmax(h @ w[model.cfg.lm_head_name].t(), -1).gather(1, ids[b, P:, None])[:, 0]
            lp.backward(s["dlp"][b].double())
            lps.append(lp.detach())
        return (torch.stack(lps),) + tuple(w[n].grad for n in _grad_names(model))
    full = torch.cat([ids, s["next"].t()], 1)
    with torch.no_grad():
        h = _layers64(model, full, w)[:, case["seq"] - 1:]
        return [h[:, j] @ w[model.cfg.lm_head_name].t() for j in range(case["steps"] + 1)]
