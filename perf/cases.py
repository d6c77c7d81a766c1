"""Requests as users of the engine send them, for timing it and for comparing its outputs between two states of the code.

A case is one batch of requests to one model through ``vllm_b200.LLM``: the model loads from a checkpoint folder, the requests are token ids,
the answers are the generated tokens and, where asked for, the log-probabilities of the five likeliest tokens at every step.  Two kinds of work
carry such an engine: prompts (thousands of tokens a step, large matrix products and whole-prompt attention) and chat (a token per request and
step, where weights and caches are read and launches count).  Both run over the mechanisms that differ most in their kernels:

    llama       grouped-query attention, gated feed-forward; bf16 or block-scaled fp8 weights
    gemma2      capped scores, every second layer with a window, norms around both blocks, capped logits
    mixtral     two of eight experts per token
    deepseek    latent attention with a rotated part, sigmoid scores in groups, many small experts beside a shared one
    qwen3next   gated delta rule beside gated attention, many small experts beside a gated shared one

Sizes are those of ``vllm_b200/benchmarks`` (widths 1024, 2048 and 4096 with heads of 128, four layers, 32000 tokens).  Weights are random, fixed
per model, of a spread that keeps every branch's share of the residual stream near that of trained models; the rows of the output matrix lean
towards one successor for each token, so that the likeliest token stands clear of the second as it does after training (the continuation is then
the same for any correct implementation) at a probability near a half.
"""
import functools
import gc
import hashlib
import json
import math
import os
import shutil
import tempfile
import weakref

import torch

VOCAB, LAYERS, HEAD, TOP = 32000, 4, 128, 5
MAX_LEN, MAX_BATCHED = 4608, 8192
# width → (query heads, kv heads, gated feed-forward)
WIDTHS = {1024: (8, 2, 2688), 2048: (16, 4, 5376), 4096: (32, 8, 10880)}
FAMILIES = ("llama", "gemma2", "mixtral", "deepseek", "qwen3next")


def _case(name, family, width, requests, low, high, new, logprobs=True, fp8=False):
    """``low`` to ``high``: tokens of a prompt; ``new``: generated tokens per request."""
    return {"name": name, "family": family, "width": width, "requests": requests, "low": low, "high": high, "new": new, "logprobs": logprobs,
            "fp8": fp8}


def listed():
    return [
        # one user types a question and waits: one short prompt, launches and latency count
        _case("llama question", "llama", 1024, 1, 23, 23, 16),
        # a busy chat server: 64 requests of ragged lengths, only the tokens are wanted
        _case("llama chat", "llama", 2048, 64, 60, 500, 32, logprobs=False),
        # the same behind block-scaled fp8 weights
        _case("llama fp8 chat", "llama", 2048, 24, 60, 500, 16, fp8=True),
        # long documents are read and answered with a word
        _case("llama documents", "llama", 4096, 4, 3500, 4100, 1),
        _case("gemma2 prompts", "gemma2", 2048, 8, 700, 1024, 2),
        _case("gemma2 chat", "gemma2", 2048, 24, 60, 900, 24),
        # classification of many texts: all prompts, one token each
        _case("mixtral prompts", "mixtral", 2048, 16, 200, 512, 1),
        _case("mixtral chat", "mixtral", 2048, 16, 40, 300, 24),
        _case("deepseek prompts", "deepseek", 2048, 8, 700, 1024, 2),
        _case("deepseek chat", "deepseek", 2048, 24, 60, 900, 24),
        _case("qwen3next prompts", "qwen3next", 2048, 8, 700, 1024, 2),
        _case("qwen3next chat", "qwen3next", 2048, 24, 60, 900, 24),
    ]


def draw(rng):
    """Any family, llama at the largest width too; prompts of 16 to 4100 tokens, at most 8192 in all; 1 to 64 requests; up to 32 new tokens."""
    family = rng.choice(FAMILIES)
    width = rng.choice((1024, 2048, 4096) if family == "llama" else (1024, 2048))
    high = int(round(math.exp(rng.uniform(math.log(16), math.log(4100)))))
    low = max(8, int(high * rng.uniform(0.3, 1.0)))
    most = max(1, min(64, MAX_BATCHED // high))
    requests = int(round(math.exp(rng.uniform(0, math.log(most)))))
    new = rng.randint(1, 3) if rng.random() < 0.5 else rng.randint(8, 32)
    fp8 = family == "llama" and rng.random() < 0.25
    c = _case("", family, width, requests, min(low, high), high, new, logprobs=rng.random() < 0.75, fp8=fp8)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ models
def _config(c):
    """config.json of a case's model."""
    H, (nh, nkv, ff) = c["width"], WIDTHS[c["width"]]
    common = dict(vocab_size=VOCAB, hidden_size=H, num_hidden_layers=LAYERS, intermediate_size=ff, num_attention_heads=nh, num_key_value_heads=nkv,
                  head_dim=HEAD, max_position_embeddings=8192, rms_norm_eps=1e-6, rope_theta=10000.0, torch_dtype="bfloat16", tie_word_embeddings=False,
                  hidden_act="silu")
    if c["family"] == "llama":
        if c["fp8"]:
            common["quantization_config"] = dict(quant_method="fp8", weight_block_size=[128, 128], activation_scheme="dynamic")
        return dict(common, architectures=["LlamaForCausalLM"], model_type="llama")
    if c["family"] == "gemma2":
        return dict(common, architectures=["Gemma2ForCausalLM"], model_type="gemma2", hidden_activation="gelu_pytorch_tanh", sliding_window=512,
                    query_pre_attn_scalar=HEAD, attn_logit_softcapping=50.0, final_logit_softcapping=30.0)
    if c["family"] == "mixtral":
        return dict(common, architectures=["MixtralForCausalLM"], model_type="mixtral", intermediate_size=H, num_local_experts=8,
                    num_experts_per_tok=2, sliding_window=None)
    E, k, eff = (16, 4, 512) if H == 1024 else (32, 6, 768)
    if c["family"] == "deepseek":
        return dict(common, architectures=["DeepseekV3ForCausalLM"], model_type="deepseek_v3", num_attention_heads=16, num_key_value_heads=16,
                    q_lora_rank=384 if H == 1024 else 1024, kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128,
                    moe_intermediate_size=eff, n_routed_experts=E, n_shared_experts=1, num_experts_per_tok=k, n_group=4, topk_group=2,
                    routed_scaling_factor=1.0, first_k_dense_replace=0, moe_layer_freq=1, norm_topk_prob=True, scoring_func="sigmoid",
                    topk_method="noaux_tc")
    return dict(common, architectures=["Qwen3NextForCausalLM"], model_type="qwen3_next", linear_num_value_heads=nh // 2, linear_num_key_heads=nh // 2,
                linear_key_head_dim=128, linear_value_head_dim=256, linear_conv_kernel_dim=4, full_attention_interval=2,
                layer_types=["linear_attention", "full_attention"] * (LAYERS // 2), num_experts=E, num_experts_per_tok=k, moe_intermediate_size=eff,
                shared_expert_intermediate_size=eff, decoder_sparse_step=1, norm_topk_prob=True, mlp_only_layers=[], attention_bias=False,
                partial_rotary_factor=0.5, rope_parameters=dict(rope_type="default", rope_theta=10000.0, partial_rotary_factor=0.5))


def _successor():
    """The token that each token leans towards."""
    g = torch.Generator().manual_seed(5)
    return torch.randperm(VOCAB, generator=g)


def _weights(c, device):
    """Checkpoint tensors by name, the same for every call."""
    f = _config(c)
    H, nh, nkv = f["hidden_size"], f["num_attention_heads"], f["num_key_value_heads"]
    gemma = c["family"] == "gemma2"
    g = torch.Generator(device=device).manual_seed(77 + H)
    w = {}

    def rnd(name, *shape, s, add=0.0, dtype=torch.bfloat16):
        w[name] = (torch.randn(*shape, generator=g, device=device) * s + add).to(dtype)

    def norm(name, n, zero=gemma or c["family"] == "qwen3next", mean=None):
        rnd(name, n, s=0.05, add=(0.0 if zero else 1.0) if mean is None else mean)

    def gated(p, ff, out=0.25):
        rnd(p + "gate_proj.weight", ff, H, s=H ** -0.5)
        rnd(p + "up_proj.weight", ff, H, s=H ** -0.5)
        rnd(p + "down_proj.weight", H, ff, s=out * ff ** -0.5)

    def experts(p, n, ff):
        for e in range(n):
            gated(f"{p}experts.{e}.", ff)

    for i in range(LAYERS):
        p = f"model.layers.{i}."
        a, m = p + "self_attn.", p + "mlp."
        norm(p + "input_layernorm.weight", H)
        if gemma:
            norm(p + "post_attention_layernorm.weight", H, mean=-0.75)
            norm(p + "pre_feedforward_layernorm.weight", H)
            norm(p + "post_feedforward_layernorm.weight", H, mean=-0.75)
        else:
            norm(p + "post_attention_layernorm.weight", H)
        if c["family"] == "deepseek":
            qr, kr = f["q_lora_rank"], f["kv_lora_rank"]
            rnd(a + "q_a_proj.weight", qr, H, s=H ** -0.5)
            norm(a + "q_a_layernorm.weight", qr)
            rnd(a + "q_b_proj.weight", nh * 192, qr, s=2 * qr ** -0.5)
            rnd(a + "kv_a_proj_with_mqa.weight", kr + 64, H, s=H ** -0.5)
            norm(a + "kv_a_layernorm.weight", kr)
            rnd(a + "kv_b_proj.weight", nh * 256, kr, s=kr ** -0.5)
            rnd(a + "o_proj.weight", H, nh * HEAD, s=0.5 * (nh * HEAD) ** -0.5)
        elif c["family"] == "qwen3next" and f["layer_types"][i] == "linear_attention":
            d, n, dk, dv = p + "linear_attn.", f["linear_num_value_heads"], 128, 256
            rnd(d + "in_proj_qkvz.weight", n * 2 * (dk + dv), H, s=H ** -0.5)
            rnd(d + "in_proj_ba.weight", 2 * n, H, s=H ** -0.5)
            rnd(d + "conv1d.weight", n * (2 * dk + dv), 1, 4, s=0.5)
            rnd(d + "dt_bias", n, s=0.5, add=-2.0, dtype=torch.float32)
            rnd(d + "A_log", n, s=0.5, dtype=torch.float32)
            norm(d + "norm.weight", dv, zero=False)
            rnd(d + "out_proj.weight", H, n * dv, s=0.5 * (n * dv) ** -0.5)
        else:
            q_out = nh * HEAD * (2 if c["family"] == "qwen3next" else 1)
            rnd(a + "q_proj.weight", q_out, H, s=2 * H ** -0.5)
            rnd(a + "k_proj.weight", nkv * HEAD, H, s=H ** -0.5)
            rnd(a + "v_proj.weight", nkv * HEAD, H, s=H ** -0.5)
            rnd(a + "o_proj.weight", H, nh * HEAD, s=0.5 * (nh * HEAD) ** -0.5)
            if c["family"] == "qwen3next":
                norm(a + "q_norm.weight", HEAD, mean=1.0)
                norm(a + "k_norm.weight", HEAD)
        if c["family"] in ("llama", "gemma2"):
            gated(m, f["intermediate_size"])
        elif c["family"] == "mixtral":
            b = p + "block_sparse_moe."
            rnd(b + "gate.weight", 8, H, s=1.5 * H ** -0.5)
            for e in range(8):
                for n, shape, s in (("w1", (H, H), 1), ("w3", (H, H), 1), ("w2", (H, H), 0.25)):
                    rnd(f"{b}experts.{e}.{n}.weight", *shape, s=s * H ** -0.5)
        else:
            n = f.get("n_routed_experts") or f["num_experts"]
            rnd(m + "gate.weight", n, H, s=1.5 * H ** -0.5)
            experts(m, n, f["moe_intermediate_size"])
            if c["family"] == "deepseek":
                rnd(m + "gate.e_score_correction_bias", n, s=0.1, dtype=torch.float32)
                gated(m + "shared_experts.", f["moe_intermediate_size"])
            else:
                gated(m + "shared_expert.", f["moe_intermediate_size"])
                rnd(m + "shared_expert_gate.weight", 1, H, s=H ** -0.5)
    norm("model.norm.weight", H)
    rnd("model.embed_tokens.weight", VOCAB, H, s=H ** -0.5 if gemma else 1.0)
    lean = torch.zeros_like(w["model.embed_tokens.weight"])
    lean[_successor().to(device)] = w["model.embed_tokens.weight"]        # row of a token: the embedding of the one that it follows
    rnd("lm_head.weight", VOCAB, H, s=H ** -0.5)
    w["lm_head.weight"] = (w["lm_head.weight"].float() + lean.float() * (14.0 / H * (H ** 0.5 if gemma else 1.0))).to(torch.bfloat16)
    if c["fp8"]:
        for name in [n for n in w if n.endswith("_proj.weight")]:
            x = w[name].float()
            r, k = (-(-s // 128) for s in x.shape)
            pad = torch.zeros(r * 128, k * 128, device=device)
            pad[:x.shape[0], :x.shape[1]] = x
            s = pad.view(r, 128, k, 128).abs().amax((1, 3)) / 448.0
            q = (pad.view(r, 128, k, 128) / s[:, None, :, None]).view(r * 128, k * 128)
            w[name] = q[:x.shape[0], :x.shape[1]].to(torch.float8_e4m3fn).contiguous()
            w[name + "_scale_inv"] = s
    return w


def _model_key(c):
    return {k: c[k] for k in ("family", "width", "fp8")}


def _checkpoint(c):
    """Folder with the model's config.json and weights; written once per machine and state of this file."""
    with open(os.path.abspath(__file__), "rb") as f:
        tag = hashlib.sha256(f.read() + json.dumps(_model_key(c), sort_keys=True).encode()).hexdigest()[:16]
    path = os.path.join(tempfile.gettempdir(), f"vllm_b200_model_{tag}")
    if not os.path.isdir(path):
        made = tempfile.mkdtemp(dir=tempfile.gettempdir())
        with open(os.path.join(made, "config.json"), "w") as f:
            json.dump(_config(c), f)
        torch.save({k: v.cpu() for k, v in _weights(c, "cuda").items()}, os.path.join(made, "pytorch_model.bin"))
        try:
            os.rename(made, path)
        except OSError:                 # another process was faster
            shutil.rmtree(made)
    return path


class _Server:
    """One engine; a program keeps it while it has requests for it."""

    def __init__(self, c):
        from vllm_b200 import LLM
        self.llm = LLM(_checkpoint(c), dtype="bfloat16", skip_tokenizer_init=True, max_model_len=MAX_LEN, max_num_seqs=64,
                       max_num_batched_tokens=MAX_BATCHED, kv_cache_memory_bytes=3 << 30, cudagraph_capture_sizes=[1, 2, 4, 8, 16, 24, 32, 48, 64],
                       multiprocess_mode=False,
                       enable_prefix_caching=False)    # the same prompts come again here: they are to be computed again

    def __del__(self):
        llm = getattr(self, "llm", None)
        if llm is not None:
            llm.shutdown()


_servers = weakref.WeakValueDictionary()       # a model's engine lives as long as a state that uses it


def _prompts(c, seed):
    g = torch.Generator().manual_seed(1000003 * seed + c["requests"])
    n = torch.randint(c["low"], c["high"] + 1, (c["requests"],), generator=g).tolist()
    return [torch.randint(0, VOCAB, (k,), generator=g).tolist() for k in n]


def prepare(case, seed):
    from vllm_b200 import SamplingParams
    key = json.dumps(_model_key(case), sort_keys=True)
    server = _servers.get(key)
    if server is None:
        gc.collect()                    # an engine of before, if any, goes first
        server = _servers[key] = _Server(case)
    return {"server": server, "prompts": [{"prompt_token_ids": p} for p in _prompts(case, seed)], "logprobs": case["logprobs"],
            "params": SamplingParams(max_tokens=case["new"], temperature=0.0, ignore_eos=True, detokenize=False,
                                     logprobs=TOP if case["logprobs"] else None)}


def run(state):
    """The generated tokens [requests, new] and, where asked for, the log-probabilities [requests, new, 5] of the likeliest tokens in order."""
    outs = [o.outputs[0] for o in state["server"].llm.generate(state["prompts"], state["params"])]
    got = {"tokens": torch.tensor([list(o.token_ids) for o in outs])}
    if state["logprobs"]:
        got["logprobs"] = torch.tensor([[sorted((p.logprob for p in step.values()), reverse=True)[:TOP] for step in o.logprobs] for o in outs])
    return got


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _active(c):
    """(parameters of a layer stack that one token meets, parameters in all), embedding and output matrices apart."""
    f = _config(c)
    H, nh, nkv, ff = f["hidden_size"], f["num_attention_heads"], f["num_key_value_heads"], f["intermediate_size"]
    gqa = H * HEAD * (2 * nh + 2 * nkv)
    if c["family"] in ("llama", "gemma2"):
        return (LAYERS * (gqa + 3 * H * ff),) * 2
    if c["family"] == "mixtral":
        return LAYERS * (gqa + 8 * H + 2 * 3 * H * H), LAYERS * (gqa + 8 * H + 8 * 3 * H * H)
    eff, k = f["moe_intermediate_size"], f["num_experts_per_tok"]
    E = f.get("n_routed_experts") or f["num_experts"]
    if c["family"] == "deepseek":
        mix = LAYERS * (H * (f["q_lora_rank"] + 576) + f["q_lora_rank"] * nh * 192 + 512 * nh * 256 + nh * HEAD * H)
    else:
        n = f["linear_num_value_heads"]
        mix = LAYERS // 2 * (gqa + H * HEAD * nh + H * n * (2 * 128 + 3 * 256 + 2))
    rest = LAYERS * H * (E + 3 * eff)
    return mix + rest + LAYERS * 3 * H * eff * k, mix + rest + LAYERS * 3 * H * eff * E


def work(case):
    """Every step reads the weights that its tokens meet and the cached tokens of its requests; every token goes through its layers."""
    c, f = case, _config(case)
    H, nh = f["hidden_size"], f["num_attention_heads"]
    n, mean, new = c["requests"], (c["low"] + c["high"]) / 2, c["new"]
    used, held = _active(c)
    E, k = (8, 2) if c["family"] == "mixtral" else (f.get("n_routed_experts") or f.get("num_experts") or 1, f["num_experts_per_tok"] if held > used else 1)
    size = 1 if c["fp8"] else 2

    def read(tokens):                    # bytes of weights that so many tokens meet
        hit = 1 - (1 - k / E) ** tokens if held > used else 1.0
        return size * (used + (held - used) * max(0.0, (hit - k / E) / (1 - k / E) if held > used else 0.0))
    full = LAYERS // 2 if c["family"] in ("qwen3next",) else LAYERS
    row = {"deepseek": 576}.get(c["family"], 2 * HEAD * f["num_key_value_heads"])          # cached values per token and layer
    per_pair = 2 * nh * (192 + 128 if c["family"] == "deepseek" else 2 * HEAD)
    state = 0 if full == LAYERS else (LAYERS - full) * f["linear_num_value_heads"] * 128 * 256
    by = read(n * mean) + n * mean * full * row * 2 + 2 * VOCAB * H + n * 4 * state
    fl = 2.0 * used * n * mean + full * per_pair * n * mean * mean / 2 + 2.0 * n * VOCAB * H + 6.0 * state * n * mean
    for s in range(1, new):
        by += read(n) + n * (mean + s) * full * row * 2 + 2 * VOCAB * H + n * 8 * state
        fl += 2.0 * used * n + full * per_pair * n * (mean + s) + 2.0 * n * VOCAB * H + 6.0 * state * n
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """16-bit activations through four layers; a token near the border of a router's choice takes another expert after another rounding."""
    if not case["logprobs"]:
        return "exact"
    return {"rel": 0.012, "max": 0.15, "differ": 0.005}


# ------------------------------------------------------------------------------------------------ 64 bits
def _norm(x, w, zero=False, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * (w + 1 if zero else w)


def _rotate(x, dims, neox=True):
    """x [T, heads, D] at positions 0 .. T - 1: the first ``dims`` dimensions are rotated."""
    T, h = x.shape[0], dims // 2
    ang = torch.arange(T, device=x.device, dtype=x.dtype)[:, None] * 10000.0 ** (-torch.arange(h, device=x.device, dtype=x.dtype) / h)
    co, si = ang.cos()[:, None], ang.sin()[:, None]
    if neox:
        a, b = x[..., :h], x[..., h:dims]
        return torch.cat([a * co - b * si, b * co + a * si, x[..., dims:]], -1)
    a, b = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([a * co - b * si, b * co + a * si], -1).flatten(-2), x[..., dims:]], -1)


def _attend(q, k, v, scale, cap=0.0, window=0):
    """q [T, H, D], k [T, G, D], v [T, G, DV] of one sequence; some rows at a time."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out, at = [], torch.arange(T, device=q.device)
    for t in range(0, T, 1024):
        qs = q[t:t + 1024].reshape(-1, G, H // G, q.shape[-1])
        s = torch.einsum("tghd,sgd->ghts", qs, k) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        gone = at[None] > at[t:t + 1024, None]
        if window:
            gone |= at[None] <= at[t:t + 1024, None] - window
        p = s.masked_fill(gone, float("-inf")).softmax(-1)
        out.append(torch.einsum("ghts,sgd->tghd", p, v).reshape(qs.shape[0], -1))
    return torch.cat(out)


def _delta_rule(q, k, v, decay, beta, lens):
    """Padded sequences [n, T, heads, ...] through S = S a (1 - b k k') + b k v', o = S' q."""
    n, T, h, dk = q.shape
    S = torch.zeros(n, h, dk, v.shape[-1], device=q.device, dtype=q.dtype)
    out = torch.empty_like(v)
    for t in range(max(lens)):
        S = S * decay[:, t, :, None, None]
        d = (v[:, t] - torch.einsum("nhkv,nhk->nhv", S, k[:, t])) * beta[:, t, :, None]
        S = S + k[:, t, :, :, None] * d[:, :, None]
        out[:, t] = torch.einsum("nhkv,nhk->nhv", S, q[:, t])
    return out


def _gelu_tanh(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _mlp(x, w, p, act, names=("gate_proj", "up_proj", "down_proj")):
    a, b, c = (w(p + n + ".weight") for n in names)
    return (act(x @ a.t()) * (x @ b.t())) @ c.t()


def _moe(c, f, x, w, p):
    silu = torch.nn.functional.silu
    if c["family"] == "mixtral":
        pw, ids = (x @ w(p + "gate.weight").t()).softmax(-1).topk(2, -1)
        pw, E, out, names = pw / pw.sum(-1, keepdim=True), 8, torch.zeros_like(x), ("w1", "w3", "w2")
    else:
        names, k, E = ("gate_proj", "up_proj", "down_proj"), f["num_experts_per_tok"], f.get("n_routed_experts") or f["num_experts"]
        logits = x @ w(p + "gate.weight").t()
        if c["family"] == "deepseek":
            s = logits.sigmoid()
            pick = (s + w(p + "gate.e_score_correction_bias")).view(len(x), f["n_group"], -1)
            kept = pick.topk(2, -1).values.sum(-1).topk(f["topk_group"], -1).indices
            gone = torch.ones(len(x), f["n_group"], dtype=torch.bool, device=x.device).scatter_(1, kept, False)
            ids = pick.masked_fill(gone[..., None], float("-inf")).flatten(1).topk(k, -1).indices
            pw, out = s.gather(1, ids), _mlp(x, w, p + "shared_experts.", silu)
        else:
            pw, ids = logits.softmax(-1).topk(k, -1)
            out = torch.sigmoid(x @ w(p + "shared_expert_gate.weight").t()) * _mlp(x, w, p + "shared_expert.", silu)
        pw = pw / pw.sum(-1, keepdim=True)
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, _mlp(x[t], w, f"{p}experts.{e}.", silu, names) * pw[t, j, None])
    return out


def _mixer(c, f, i, x, w, lens):
    """Attention or recurrence of layer i over the sequences in x (``lens`` tokens each, one after the other)."""
    p, H, nh, nkv = f"model.layers.{i}.", f["hidden_size"], f["num_attention_heads"], f["num_key_value_heads"]
    a = p + "self_attn."
    parts = functools.partial(torch.split, split_size_or_sections=lens)
    if c["family"] == "deepseek":
        q = (_norm(x @ w(a + "q_a_proj.weight").t(), w(a + "q_a_layernorm.weight")) @ w(a + "q_b_proj.weight").t()).view(-1, nh, 192)
        lat = x @ w(a + "kv_a_proj_with_mqa.weight").t()
        kv = (_norm(lat[:, :512], w(a + "kv_a_layernorm.weight")) @ w(a + "kv_b_proj.weight").t()).view(-1, nh, 256)
        out = []
        for qs, ks, ps in zip(parts(q), parts(kv), parts(lat[:, None, 512:])):
            qs = torch.cat([qs[..., :128], _rotate(qs[..., 128:], 64, False)], -1)
            kk = torch.cat([ks[..., :128], _rotate(ps, 64, False).expand(-1, nh, -1)], -1)
            out.append(_attend(qs, kk, ks[..., 128:], 192 ** -0.5))
        return torch.cat(out) @ w(a + "o_proj.weight").t()
    if c["family"] == "qwen3next" and f["layer_types"][i] == "linear_attention":
        d, n, dk, dv = p + "linear_attn.", f["linear_num_value_heads"], 128, 256
        q, k, v, z = (x @ w(d + "in_proj_qkvz.weight").t()).view(-1, n, 2 * (dk + dv)).split([dk, dk, dv, dv], -1)
        b, g = (x @ w(d + "in_proj_ba.weight").t()).view(-1, n, 2).unbind(-1)
        qkv = torch.cat([q.flatten(1), k.flatten(1), v.flatten(1)], -1)
        cw = w(d + "conv1d.weight")[:, 0]
        taps = [torch.nn.functional.pad(s, (0, 0, 3, 0)) for s in parts(qkv)]
        qkv = torch.nn.functional.silu(torch.cat([sum(s[j:len(s) - 3 + j] * cw[:, j] for j in range(4)) for s in taps]))
        q, k, v = qkv.split([n * dk, n * dk, n * dv], -1)
        unit = lambda y: y * torch.rsqrt(y.pow(2).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k, v = unit(q.view(-1, n, dk)) * dk ** -0.5, unit(k.view(-1, n, dk)), v.view(-1, n, dv)
        decay = torch.exp(-w(d + "A_log").exp() * torch.nn.functional.softplus(g + w(d + "dt_bias")))
        pad = [torch.nn.utils.rnn.pad_sequence(parts(y), batch_first=True) for y in (q, k, v, decay, b.sigmoid())]
        o = _delta_rule(*pad, lens)
        o = torch.cat([y[:m] for y, m in zip(o, lens)])
        return (_norm(o, w(d + "norm.weight")) * torch.nn.functional.silu(z)).flatten(1) @ w(d + "out_proj.weight").t()
    q = x @ w(a + "q_proj.weight").t()
    k, v = ((x @ w(a + n + ".weight").t()).view(-1, nkv, HEAD) for n in ("k_proj", "v_proj"))
    gate = None
    if c["family"] == "qwen3next":
        q, gate = q.view(-1, nh, 2 * HEAD).split([HEAD, HEAD], -1)
        q, k = _norm(q, w(a + "q_norm.weight"), True), _norm(k, w(a + "k_norm.weight"), True)
    q = q.reshape(-1, nh, HEAD)
    dims = HEAD // 2 if c["family"] == "qwen3next" else HEAD
    cap, window = f.get("attn_logit_softcapping") or 0.0, (f.get("sliding_window") or 0) if i % 2 == 0 else 0
    o = torch.cat([_attend(_rotate(qs, dims), _rotate(ks, dims), vs, HEAD ** -0.5, cap, window) for qs, ks, vs in zip(parts(q), parts(k), parts(v))])
    if gate is not None:
        o = o * torch.sigmoid(gate.flatten(1))
    return o @ w(a + "o_proj.weight").t()


def exact(case, seed):
    """The same from plain 64-bit tensors.  Tokens follow the likeliest continuation; where only they are asked for there is nothing to add."""
    if not case["logprobs"]:
        return None
    c, f, dev = case, _config(case), "cuda" if torch.cuda.is_available() else "cpu"
    held, gemma = _weights(c, dev), c["family"] == "gemma2"
    zero = gemma or c["family"] == "qwen3next"

    def w(name):
        t = held[name].double()
        s = held.get(name + "_scale_inv")
        if s is not None:
            t = t * s.double().repeat_interleave(128, 0)[:t.shape[0]].repeat_interleave(128, 1)[:, :t.shape[1]]
        return t
    nxt, seqs = _successor().tolist(), []
    for s in _prompts(c, seed):
        s = list(s)
        for _ in range(c["new"] - 1):
            s.append(nxt[s[-1]])
        seqs.append(s)
    lens = [len(s) for s in seqs]
    x = w("model.embed_tokens.weight")[torch.tensor(sum(seqs, []), device=dev)] * (f["hidden_size"] ** 0.5 if gemma else 1.0)
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        y = _mixer(c, f, i, _norm(x, w(p + "input_layernorm.weight"), zero), w, lens)
        after = w(p + "post_attention_layernorm.weight")
        x = x + (_norm(y, after, True) if gemma else y)
        h = _norm(x, w(p + "pre_feedforward_layernorm.weight"), True) if gemma else _norm(x, after, zero)
        if c["family"] == "llama":
            y = _mlp(h, w, p + "mlp.", torch.nn.functional.silu)
        elif gemma:
            y = _norm(_mlp(h, w, p + "mlp.", _gelu_tanh), w(p + "post_feedforward_layernorm.weight"), True)
        else:
            y = _moe(c, f, h, w, p + ("block_sparse_moe." if c["family"] == "mixtral" else "mlp."))
        x = x + y
    last = torch.cat([torch.arange(e - c["new"], e) for e in torch.tensor(lens).cumsum(0).tolist()]).to(dev)
    logits = _norm(x[last], w("model.norm.weight"), zero) @ w("lm_head.weight").t()
    if f.get("final_logit_softcapping"):
        logits = f["final_logit_softcapping"] * torch.tanh(logits / f["final_logit_softcapping"])
    lp = logits.log_softmax(-1)
    n = len(seqs)
    return {"tokens": lp.argmax(-1).view(n, -1).cpu(), "logprobs": lp.topk(TOP, -1).values.view(n, -1, TOP).cpu()}
