"""The work a post-training job does with this framework, as a list of measurable cases.

Every case goes through the entry points a job uses: ``InferEngine.generate`` for rollouts and ``InferEngine.step`` for
step-wise serving of layer-plan decoders, ``compute_log_probs``, ``finetune_step`` and ``rl_train_actor`` of the training
engine.  Models are the presets of the benchmark recipes and the small decoder of the smoke test, cut to a few layers: a
layer of a deep model costs the same in each place, so depth only repeats what these passes show.

``kind`` says which entry point runs:

* ``rollout``   prompts in, sampled tokens and their log-probs out (prefill, then captured decode steps);
* ``logprobs``  forward only: log-prob and entropy of every response token;
* ``sft``       masked cross-entropy, backward, AdamW;
* ``rl``        clipped policy gradient on group-normalised advantages, backward, AdamW;
* ``lora``      ``sft`` of low-rank adapters on a frozen block-fp8 base;
* ``serve``     prompt portions and then single tokens of several open requests in one batch each.
"""
import math
import random

import numpy as np
import torch
import torch.utils.checkpoint

from gcore_b200.configs.base import from_dict
from gcore_b200.configs.config import RlConfig
from gcore_b200.engine import get_training_engine
from gcore_b200.models.config import ModelConfig, from_hf_config, get_preset
from gcore_b200.models.gpt import GPTModel
from gcore_b200.models.plan_decoder import build_decoder
from gcore_b200.rollout.engine import InferEngine, RolloutWeights, SamplingParams

SMALL_VOCAB = 32768
LORA = dict(rank=64, alpha=128, targets=("linear_q_down_proj", "linear_q_up_proj", "linear_kv_down_proj",
                                         "linear_kv_up_proj", "linear_proj"))


# ------------------------------------------------------------------------------------------------------------- cases
def _case(name, kind, model, seqs, lo, hi, layers=2, vocab=SMALL_VOCAB, shape=0, samples=1, new=0, recompute="none"):
    """``seqs`` sequences of ``lo`` .. ``hi`` tokens (prompts, where tokens are generated); ``shape`` picks the lengths;
    ``samples`` per prompt and ``new`` generated or served tokens each."""
    c = dict(kind=kind, model=model, layers=layers, vocab=vocab, seqs=seqs, lo=lo, hi=hi, shape=shape, samples=samples,
             new=new, recompute=recompute)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a handful of short answers from a small model: an evaluation probe, where every launch counts
        _case("rollout_small", "rollout", "small", 4, 40, 48, new=24),
        # one group-sampled batch of the dense GRPO recipe: 8 prompts x 8 samples
        _case("rollout_group", "rollout", "qwen2.5-7b", 8, 256, 256, vocab=152064, samples=8, new=64),
        # mixture-of-experts rollout: few requests per expert
        _case("rollout_experts", "rollout", "qwen3-30b-a3b", 16, 200, 256, vocab=151936, new=48, shape=1),
        # long documents as prompts (alternating full and windowed layers with sinks), short answers
        _case("rollout_long", "rollout", "llama3-8b-swa", 3, 3001, 8000, new=32, shape=2),
        # latent attention: a small cache row shared by 128 heads
        _case("rollout_latent", "rollout", "deepseek-v3-12l", 8, 480, 512, layers=1, samples=4, new=32, shape=3),
        # log-probs of the sampled responses under the old policy, one packed micro-batch of 64 x (256 + 1024) tokens
        _case("logprobs_packed", "logprobs", "qwen2.5-7b", 9, 500, 1280, vocab=152064, shape=4),
        # the smoke-test model on 16 short sequences: optimizer and host work against small kernels
        _case("sft_small", "sft", "small", 16, 60, 72, shape=5),
        # policy update of the dense GRPO recipe on one packed micro-batch
        _case("rl_dense", "rl", "qwen2.5-7b", 9, 500, 1280, shape=6),
        # long-context supervised fine-tuning: few long documents, attention over up to 16k keys, layers recomputed
        _case("sft_long", "sft", "llama3-8b-swa", 3, 4000, 13000, shape=7, recompute="full"),
        # mixture-of-experts training: routing, ragged expert products, load-balancing loss
        _case("rl_experts", "rl", "qwen3-30b-a3b", 6, 400, 1100, layers=1, shape=8),
        # adapters on a frozen block-fp8 latent-attention base
        _case("lora_latent", "lora", "deepseek-v3-12l", 5, 300, 1000, layers=1, shape=9),
        # a layer-plan decoder served step by step: ragged prompt portions, then single tokens
        _case("serve_plan", "serve", "nafitar", 4, 700, 2500, layers=3, new=8, shape=10),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (kind, model, layers, vocabularies, sequences, tokens of a sequence, tokens of a batch, samples, new tokens)
RANGES = [
    ("rollout", "small", 2, (SMALL_VOCAB,), (1, 32), (12, 600), 4096, (1, 4), (8, 48)),
    ("rollout", "qwen2.5-7b", 2, (SMALL_VOCAB, 152064), (1, 16), (30, 1500), 8192, (1, 8), (8, 64)),
    ("rollout", "qwen3-30b-a3b", 2, (SMALL_VOCAB, 151936), (1, 32), (30, 800), 8192, (1, 1), (8, 48)),
    ("rollout", "llama3-8b-swa", 2, (SMALL_VOCAB,), (1, 4), (500, 8000), 16384, (1, 4), (8, 32)),
    ("rollout", "deepseek-v3-12l", 1, (SMALL_VOCAB,), (1, 16), (30, 1200), 8192, (1, 4), (8, 32)),
    ("logprobs", "small", 2, (SMALL_VOCAB,), (1, 64), (20, 1000), 8192, (1, 1), (0, 0)),
    ("logprobs", "qwen2.5-7b", 2, (SMALL_VOCAB, 152064), (1, 16), (60, 4000), 8192, (1, 1), (0, 0)),
    ("logprobs", "qwen3-30b-a3b", 1, (SMALL_VOCAB,), (1, 16), (60, 2000), 8192, (1, 1), (0, 0)),
    ("sft", "small", 2, (SMALL_VOCAB,), (1, 64), (20, 1000), 8192, (1, 1), (0, 0)),
    ("rl", "qwen2.5-7b", 2, (SMALL_VOCAB,), (1, 16), (60, 4000), 8192, (1, 1), (0, 0)),
    ("sft", "llama3-8b-swa", 2, (SMALL_VOCAB,), (1, 6), (300, 13000), 22000, (1, 1), (0, 0)),
    ("rl", "qwen3-30b-a3b", 1, (SMALL_VOCAB,), (1, 12), (60, 1500), 6144, (1, 1), (0, 0)),
    ("lora", "deepseek-v3-12l", 1, (SMALL_VOCAB,), (1, 12), (60, 1500), 4096, (1, 1), (0, 0)),
    ("serve", "nafitar", 3, (SMALL_VOCAB,), (1, 16), (30, 3000), 8192, (1, 1), (2, 8)),
]


def draw(rng):
    kind, model, layers, vocabs, seqs, tokens, batch, samples, new = rng.choice(RANGES)
    n = _log_uniform(rng, *seqs)
    a, b = sorted(min(_log_uniform(rng, *tokens), max(tokens[0], batch // n)) for _ in range(2))
    return _case(None, kind, model, n, a, b, layers=layers, vocab=rng.choice(vocabs), shape=rng.randrange(1 << 20),
                 samples=_log_uniform(rng, *samples), new=_log_uniform(rng, *new) if new[1] else 0,
                 recompute=rng.choice(("none", "full")) if kind in ("sft", "rl") else "none")


def _lengths(case):
    r = random.Random(case["shape"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["seqs"])]


def _prompt_part(case, n):
    """Tokens of a training sequence that are its prompt and carry no loss."""
    return 0 if case["kind"] == "sft" and case["model"] != "small" else max(1, n // 5)


def _model_config(case):
    if case["model"] == "nafitar":
        layer = dict(type="parallel", mlp=dict(ff=5632, kind="dense"), mixer=dict(
            left=dict(heads=16, kv_heads=4, dim=128, vdim=128, mask=dict(size=1024), scale=128 ** -0.5),
            right=dict(heads=8, dim=128, vdim=256, gate_cap=15.0)))
        return from_hf_config(dict(architecture="Nafitar", layers=[layer] * case["layers"], max_positions=4096,
                                   norm=dict(eps=1e-6), vocab=case["vocab"], width=2048))
    if case["model"] == "small":
        return ModelConfig(arch="qwen2", num_layers=case["layers"], hidden_size=1024, num_attention_heads=8,
                           num_kv_heads=2, head_dim=128, ffn_hidden_size=2816, vocab_size=case["vocab"], rope_theta=1e6,
                           qkv_bias=True)
    return get_preset(case["model"], num_layers=case["layers"], vocab_size=case["vocab"])


# ----------------------------------------------------------------------------------------------------------- weights
def _generator(seed, tag):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + sum(ord(c) * 31 ** (i % 7) for i, c in enumerate(tag)))
                                                      & 0x7FFFFFFF)


def _next_token(vocab, seed):
    """A permutation of the vocabulary: the token that most often follows each token."""
    return torch.randperm(vocab, generator=_generator(seed, "follows"), device="cuda")


def _weight(name, p, cfg, case, seed):
    """Values of parameter ``name`` in the shape and precision of ``p``: matrices keep the scale of their input,
    norm gains lie around one."""
    g = _generator(seed, name)
    r = torch.randn(p.shape, generator=g, device="cuda", dtype=torch.float32)
    if "layernorm" in name:
        r = 1 + 0.1 * r
    elif "sinks" in name:
        pass
    elif p.dim() == 1:
        r *= 0.1
    elif "lora_A" in name:
        r *= p.shape[-1] ** -0.5
    elif "lora_B" in name:
        r *= 0.02
    elif "word_embeddings" in name:
        pass
    elif "linear_proj" in name or "linear_fc2" in name:
        r *= (2 * cfg.num_layers * p.shape[-1]) ** -0.5
    else:
        r *= p.shape[-1] ** -0.5
    return r.to(p.dtype)


@torch.no_grad()
def _fill(model, cfg, case, seed):
    for name, p in model.named_parameters():
        if name != "output_layer.weight":
            p.copy_(_weight(name, p, cfg, case, seed))
    emb = model.embedding.word_embeddings.weight
    for name, r in model.named_parameters():
        if name.endswith("router.weight"):
            # a router that has learned something: every token carries the directions of its experts, which then stand
            # out from the others as they do after training
            g = _generator(seed, name + ".tokens")
            mine = torch.rand(emb.shape[0], r.shape[0], generator=g, device="cuda").topk(cfg.moe_top_k, -1).indices
            emb.add_((6.0 * torch.zeros(emb.shape[0], r.shape[0], device="cuda").scatter_(1, mine, 1.0) @ r).to(emb.dtype))
    head = model.output_layer.weight
    # a language model that has learned something: the embedding that leads to a token points towards its output row,
    # so that the likeliest token stands out as it does in text
    mark = torch.empty_like(head)
    mark[_next_token(head.shape[0], seed)] = emb
    a = 18.0 / math.sqrt(cfg.hidden_size)
    noise = _weight("output_layer.weight", head, cfg, case, seed)
    head.copy_(a * mark.float() * cfg.hidden_size ** -0.5 + (1 - a * a) ** 0.5 * noise.float())


def _plan_tensors(cfg, case, seed):
    """A Nafitar checkpoint."""
    w, W = cfg.hidden_size, {}

    def put(name, *shape, std=None, mean=0.0):
        std = shape[-1] ** -0.5 if std is None else std
        W[name] = (mean + std * torch.randn(*shape, generator=_generator(seed, name), device="cuda")).to(torch.bfloat16)

    put("embed", cfg.vocab_size, w, std=1.0)
    put("pos", cfg.max_position_embeddings, w, std=0.3)
    put("head", cfg.vocab_size, w)
    put("final.norm", w, std=0.1)
    for i, spec in enumerate(cfg.layer_plan.layers):
        n, a, b = f"l{i}", spec.attention, spec.memory
        qd, kd, vd = a.heads * a.dim, a.kv_heads * a.dim, b.heads * b.vdim
        for nm in ("norm1", "norm1b", "norm2", "norm2b"):
            put(f"{n}.{nm}", w, std=0.1)
        for nm, rows in (("left.q", qd), ("left.k", kd), ("right.q", b.heads * b.dim), ("right.k", b.heads * b.dim),
                         ("right.v", vd), ("right.g", vd), ("right.i", b.heads), ("right.f", b.heads)):
            put(f"{n}.mix.{nm}", rows, w)
        put(f"{n}.mix.left.q.b", qd, std=0.2)
        put(f"{n}.mix.left.k.b", kd, std=0.2)
        put(f"{n}.mix.left.o", w, qd)
        put(f"{n}.mix.right.o", w, vd)
        put(f"{n}.mix.right.norm", vd, std=0.1, mean=1.0)
        put(f"{n}.mix.right.i.b", b.heads, std=1.0)
        put(f"{n}.mix.right.f.b", b.heads, std=2.0, mean=2.0)
        put(f"{n}.mix.left.out", w, std=0.2, mean=1.0)
        put(f"{n}.mix.right.out", w, std=0.2, mean=1.0)
        put(f"{n}.mlp.gate", spec.ffn, w)
        put(f"{n}.mlp.up", spec.ffn, w)
        put(f"{n}.mlp.down", w, spec.ffn)
    return W


# ------------------------------------------------------------------------------------------------------------ inputs
def _token_lists(case, seed, extra=0):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(100, case["vocab"] - 100, (n + extra,), generator=g) for n in _lengths(case)]


def _samples(case, seed):
    g = torch.Generator().manual_seed(seed + 1)
    out = []
    for t in _token_lists(case, seed):
        n, p = t.numel(), _prompt_part(case, t.numel())
        mask = torch.zeros(n)
        mask[max(p - 1, 0):n - 1] = 1.0
        s = dict(tokens=t, prompt_length=p, mask=mask)
        if case["kind"] == "rl":
            # one advantage per response, normalised within its group
            s["advantages"] = torch.full((n,), float(torch.randn((), generator=g)))
        out.append(s)
    return out


def _training_engine(case):
    policy = dict(model_arch="qwen2", recompute=case["recompute"], without_ref=True, dynamic_mbs_target_seqlen=1 << 16,
                  without_optim=case["kind"] == "logprobs")
    if case["kind"] == "lora":
        policy.update(fp8=True, lora=dict(rank=LORA["rank"], alpha=LORA["alpha"], type="lora",
                                          target_modules=list(LORA["targets"])))
    cfg = from_dict(RlConfig, {
        "training": {"train_mbs": 1, "seed": 1234, "total_ppo_step": 1000, "per_token_loss": True},
        "policy": policy,
        "optimizer": {"lr": 1e-6, "lr_decay_style": "constant", "weight_decay": 0.01, "max_grad_norm": 1.0},
        "ppo": {"advantage_type": "grpo", "loss_func": "grpo", "grpo_kl_loss_beta": 0.0, "skip_prev_logps": True},
    })
    eng = get_training_engine(cfg.policy, cfg.optimizer, cfg.training, cfg.ppo, model_cfg=_model_config(case),
                              total_steps=1000)
    eng.setup_model_and_get_optimizer(with_ref=False)
    return eng


def prepare(case, seed):
    cfg, dev = _model_config(case), torch.device("cuda")
    st = dict(case=case)
    if case["kind"] in ("rollout", "serve"):
        longest = case["hi"] + case["new"] + 16
        if case["kind"] == "serve":
            model = build_decoder(cfg, dev).load_tensors(_plan_tensors(cfg, case, seed))
        else:
            model = GPTModel(cfg, recompute="none", device=dev)
            _fill(model, cfg, case, seed)
        requests = case["seqs"] * case["samples"]
        st["engine"] = InferEngine(cfg, RolloutWeights.from_model(model), max_running_requests=requests,
                                   max_model_len=longest, kv_block_size=64 if case["kind"] == "serve" else 16,
                                   max_prefill_tokens=1 << 20, device=dev)
        st["engine"].wake_up()
        st["tokens"] = [t.tolist() for t in _token_lists(case, seed, case["new"] if case["kind"] == "serve" else 0)]
        if case["kind"] == "rollout":
            st["params"] = SamplingParams(greedy=True, max_new_tokens=case["new"])
            # a serving engine is warm: its decode step is captured before the first request
            st["engine"].generate([[5, 6, 7]], SamplingParams(greedy=True, max_new_tokens=3))
        return st
    eng = _training_engine(case)
    _fill(eng.model, cfg, case, seed)
    if eng.optimizer is not None:
        eng.optimizer.reload_master_from_params()
    st.update(engine=eng, samples=_samples(case, seed))
    return st


def _generate(st):
    reqs = st["engine"].generate(st["tokens"], st["params"], n=st["case"]["samples"])
    return {"tokens": np.array([r.out_tokens for r in reqs], dtype=np.int64),
            "logprobs": np.array([r.out_logprobs for r in reqs], dtype=np.float32)}


def _serve(st):
    eng, new, out = st["engine"], st["case"]["new"], []
    rids = [eng.open_request() for _ in st["tokens"]]
    out.append(eng.step([(r, t[:-new]) for r, t in zip(rids, st["tokens"])], [[len(t) - new - 1] for t in st["tokens"]]))
    for k in range(new):
        out.append(eng.step([(r, [t[len(t) - new + k]]) for r, t in zip(rids, st["tokens"])], [[0]] * len(rids)))
    for r in rids:
        eng.close_request(r)
    return torch.stack(out, 1)


def run(st):
    kind = st["case"]["kind"]
    if kind == "rollout":
        return _generate(st)
    if kind == "serve":
        return _serve(st)
    eng, samples = st["engine"], [dict(s) for s in st["samples"]]
    if kind == "logprobs":
        done = eng.compute_log_probs(samples)
        return {"logprobs": torch.cat([s["logprobs"] for s in done]),
                "entropy": torch.cat([s["prev_per_token_entropies"] for s in done])}
    m = eng.rl_train_actor(samples) if kind == "rl" else eng.finetune_step(samples)
    return {"loss": m["ppo-metrics/pg_loss" if kind == "rl" else "lm_loss"],
            "grad_norm": m["policy/grad_norm" if kind == "rl" else "grad_norm"],
            "grads": {n: p.main_grad for n, p in eng.model.named_parameters() if p.requires_grad}}


# -------------------------------------------------------------------------------------------------------------- work
def _matrix_elements(case, cfg):
    """(weights that every token multiplies with, all weights of the layers)."""
    if case["model"] == "nafitar":
        per = sum(2 * (s.attention.heads + s.attention.kv_heads) * s.attention.dim * cfg.hidden_size
                  + s.memory.heads * (2 * s.memory.dim + 3 * s.memory.vdim) * cfg.hidden_size + 3 * s.ffn * cfg.hidden_size
                  for s in cfg.layer_plan.layers)
        return per, per
    full = cfg.num_parameters(include_embedding=False)
    return full - (cfg.num_parameters() - cfg.active_parameters()), full


def _attention_pairs(case, cfg, lens):
    """Query-key pairs of every layer over whole causal sequences."""
    total = 0
    for i in range(case["layers"]):
        w = 1024 if case["model"] == "nafitar" else cfg.layer_window(i)
        for n in lens:
            total += n * (n + 1) // 2 if not w or n <= w else w * (w + 1) // 2 + (n - w) * w
    return total


def _state_floats(case, cfg):
    """Numbers of recurrent state of one request."""
    return sum(s.memory.heads * s.memory.dim * s.memory.vdim for s in cfg.layer_plan.layers) \
        if case["model"] == "nafitar" else 0


def work(case):
    cfg = _model_config(case)
    active, weights = _matrix_elements(case, cfg)
    lens, new, reqs = _lengths(case), case["new"], case["seqs"] * case["samples"]
    T, V, H = sum(lens), case["vocab"], cfg.hidden_size
    dqk, dv = (cfg.qk_head_dim, cfg.v_head_dim) if cfg.use_mla else (cfg.head_dim, cfg.head_dim)
    pair = 2 * cfg.num_attention_heads * (dqk + dv)
    attention = _attention_pairs(case, cfg, lens) * pair
    row = (cfg.kv_lora_rank + cfg.qk_rope_head_dim) if cfg.use_mla else 2 * cfg.num_kv_heads * cfg.head_dim
    if case["model"] == "nafitar":
        row = cfg.num_kv_heads * cfg.head_dim
    if case["kind"] in ("rollout", "serve"):
        # prompts once; then every step reads the weights its tokens use, and the cache rows they see
        touched = weights if not cfg.is_moe else min(weights, active * reqs)
        seen = [sum(min(n + new // 2, cfg.layer_window(i) or n + new // 2, 1024 if case["model"] == "nafitar" else 1 << 30)
                    for n in lens) for i in range(case["layers"])]
        cache = sum(seen) * case["samples"] * row * 2
        steps = new - 1 if case["kind"] == "rollout" else new
        state = 8 * reqs * _state_floats(case, cfg)
        return {"flops": 2 * active * (T + reqs * steps) + attention + 2 * V * H * reqs * (steps + 1)
                + 2 * T * _state_floats(case, cfg) * 2,
                "bytes": weights * 2 + V * H * 2 + T * (H + row * case["layers"]) * 2
                + steps * (touched * 2 + V * H * 2 + cache + state)}
    scored = sum(n - 1 - max(_prompt_part(case, n) - 1, 0) for n in lens)
    head = 2 * V * H * scored
    forward = 2 * active * T + attention + head
    if case["kind"] == "logprobs":
        return {"flops": forward, "bytes": (weights + V * H) * 2 + T * H * 2 + T * 8}
    if case["kind"] == "lora":
        # the base's data gradient, no weight gradient
        return {"flops": 2 * forward + 1.5 * attention, "bytes": 2 * weights + 2 * V * H * 2 + 12 * T * H}
    params = weights + 2 * V * H
    # AdamW: gradient written and read; master weight and two moments read and written; bf16 weight read and written
    return {"flops": 3 * forward + 0.5 * attention, "bytes": params * (8 + 24 + 4) + 4 * T * H}


def tolerance(case):
    """What another order of the bf16 roundings in front of an output moves it by: the distance of these passes from the
    same in 64 bits is 0.004 for log-probs, 0.01 - 0.03 for the logits of the layer-plan decoder and 0.01 - 0.05 for the
    gradients of the layers furthest from the loss."""
    if case["kind"] == "rollout":
        return {"rel": 1.5e-2, "max": 0.5, "differ": 0.005}
    if case["kind"] == "logprobs":
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 0.03, "max": 0.99}


# ------------------------------------------------------------------------------------- the same in 64 bits, plain torch
def _norm(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, theta, interleaved):
    half = x.shape[-1] // 2
    inv = theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    ang = pos[:, None, None] * inv
    c, s = ang.cos(), ang.sin()
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend_block(q, k, v, sink, scale, window, first):
    """Rows ``first`` .. of one group of heads [h, rows, d] over one key head [keys, d]."""
    i = torch.arange(first, first + q.shape[1], device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    seen = j <= i
    if window:
        seen &= j > i - window
    s = (q @ k.T * scale).masked_fill(~seen, float("-inf"))
    m = s.amax(-1, keepdim=True).detach()
    e = torch.exp(s - m)
    den = e.sum(-1, keepdim=True)
    if sink is not None:
        den = den + torch.exp(sink[:, None, None] - m)
    return (e / den) @ v


def _checkpoint(f, *a):
    return torch.utils.checkpoint.checkpoint(f, *a, use_reentrant=False)


def _attention(q, k, v, bounds, scale, window, sinks):
    """q [T, H, d], k / v [T, G, d]: causal attention inside each sequence."""
    H, G = q.shape[1], k.shape[1]
    seqs = []
    for a, b in bounds:
        heads = []
        for g in range(G):
            hs = slice(g * (H // G), (g + 1) * (H // G))
            qg, kg, vg = q[a:b, hs].transpose(0, 1), k[a:b, g], v[a:b, g]
            rows = [_checkpoint(_attend_block, qg[:, r:r + 2048], kg[:min(r + 2048, b - a)], vg[:min(r + 2048, b - a)],
                                None if sinks is None else sinks[hs], scale, window, r) for r in range(0, b - a, 2048)]
            heads.append(torch.cat(rows, 1))
        seqs.append(torch.cat(heads, 0).transpose(0, 1))
    return torch.cat(seqs)


def _e4m3(x, rows):
    """Values after a round trip through e4m3 with one scale per block of ``rows`` x 128; gradients pass straight through."""
    n, k = x.shape
    blocks = torch.nn.functional.pad(x.detach(), (0, 0, 0, -n % rows)).view(-1, rows, k // 128, 128)
    scale = blocks.abs().amax((1, 3), keepdim=True).clamp_min(1e-10) / 448
    back = (blocks / scale).float().to(torch.float8_e4m3fn).double() * scale
    return x + (back.reshape(-1, k)[:n] - x).detach()


def _adapted(W, name, x):
    y = (_e4m3(x, 1) if "fp8" in W else x) @ W[name + ".weight"].T
    if name + ".lora.lora_A" in W:
        y = y + (x @ W[name + ".lora.lora_A"].T) @ W[name + ".lora.lora_B.0"].T * (LORA["alpha"] / LORA["rank"])
    return y


def _latent_attention(W, n, cfg, x, pos, bounds):
    T, h, eps = x.shape[0], cfg.num_attention_heads, cfg.rms_norm_eps
    dn, dr, dv, C = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.kv_lora_rank
    ql = _norm(_adapted(W, n + "linear_q_down_proj", x), W[n + "q_layernorm.weight"], eps)
    q = _adapted(W, n + "linear_q_up_proj", ql).view(T, h, dn + dr)
    kv = _adapted(W, n + "linear_kv_down_proj", x)
    up = _adapted(W, n + "linear_kv_up_proj", _norm(kv[:, :C], W[n + "kv_layernorm.weight"], eps)).view(T, h, dn + dv)
    kr = _rotate(kv[:, None, C:], pos, cfg.rope_theta, cfg.rope_interleaved).expand(T, h, dr)
    q = torch.cat([q[..., :dn], _rotate(q[..., dn:], pos, cfg.rope_theta, cfg.rope_interleaved)], -1)
    o = _attention(q, torch.cat([up[..., :dn], kr], -1), up[..., dn:], bounds, (dn + dr) ** -0.5, 0, None)
    return _adapted(W, n + "linear_proj", o.reshape(T, h * dv))


def _grouped_attention(W, n, cfg, x, pos, bounds, window):
    T, D, hq, hk = x.shape[0], cfg.head_dim, cfg.num_attention_heads, cfg.num_kv_heads
    qkv = x @ W[n + "linear_qkv.weight"].T
    if cfg.qkv_bias:
        qkv = qkv + W[n + "linear_qkv.bias"]
    q, k, v = qkv.view(T, hq + 2 * hk, D).split([hq, hk, hk], 1)
    if cfg.qk_layernorm:
        q = _norm(q, W[n + "q_layernorm.weight"], cfg.rms_norm_eps)
        k = _norm(k, W[n + "k_layernorm.weight"], cfg.rms_norm_eps)
    q, k = (_rotate(t, pos, cfg.rope_theta, False) for t in (q, k))
    o = _attention(q, k, v, bounds, D ** -0.5, window, W.get(n + "sinks"))
    return o.reshape(T, hq * D) @ W[n + "linear_proj.weight"].T


def _gated(x, fc1, fc2, fp8=False):
    g, u = ((_e4m3(x, 1) if fp8 else x) @ fc1.T).chunk(2, -1)
    y = torch.nn.functional.silu(g) * u
    return (_e4m3(y, 1) if fp8 else y) @ fc2.T


def _experts(W, n, cfg, x):
    E, K = cfg.num_experts, cfg.moe_top_k
    p = torch.softmax(x @ W[n + "router.weight"].T, -1)
    w, idx = torch.topk(p, K, -1)
    w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(E):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            y = y.index_add(0, t, w[t, slot, None] * _gated(x[t], W[n + "experts.linear_fc1.weight"][e],
                                                            W[n + "experts.linear_fc2.weight"][e]))
    load = torch.bincount(idx.reshape(-1), minlength=E) * (E / (K * x.shape[0]))
    return y, cfg.moe_aux_loss_coef * (load * p.mean(0)).sum()


def _hidden(W, cfg, tokens, pos, bounds):
    """Final-normed hidden states of packed sequences and the routers' balancing loss."""
    x, aux = W["embedding.word_embeddings.weight"][tokens], 0.0

    def layer(x, i):
        n = f"decoder.layers.{i}."
        h = _norm(x, W[n + "input_layernorm.weight"], cfg.rms_norm_eps)
        a = n + "self_attention."
        x = x + (_latent_attention(W, a, cfg, h, pos, bounds) if cfg.use_mla else
                 _grouped_attention(W, a, cfg, h, pos, bounds, cfg.layer_window(i)))
        h = _norm(x, W[n + "pre_mlp_layernorm.weight"], cfg.rms_norm_eps)
        if cfg.layer_is_moe(i):
            y, b = _experts(W, n + "mlp.", cfg, h)
            return x + y, b
        return x + _gated(h, W[n + "mlp.linear_fc1.weight"], W[n + "mlp.linear_fc2.weight"], "fp8" in W), x.new_zeros(())

    for i in range(cfg.num_layers):
        x, b = _checkpoint(layer, x, i)
        aux = aux + b
    return _norm(x, W["decoder.final_layernorm.weight"], cfg.rms_norm_eps), aux


def _scores(h, head, targets):
    z = torch.log_softmax(h @ head.T, -1)
    return z.gather(-1, targets[:, None])[:, 0], -(z.exp() * z).sum(-1)


def _weights64(case, seed, grad):
    """The weights that ``prepare`` makes, and (``grad``) which of them are trained."""
    cfg = _model_config(case)
    if case["kind"] in ("rollout", "logprobs"):
        model = GPTModel(cfg, recompute="none", device=torch.device("cuda"))
    else:
        model = _training_engine(case).model
    _fill(model, cfg, case, seed)
    W = {}
    for n, p in model.named_parameters():
        w = p.detach().double()
        if case["kind"] == "lora" and ".linear_" in n and "lora_" not in n:
            w, W["fp8"] = _e4m3(w, 128), w.new_ones(())   # the frozen base is stored in block fp8
        W[n] = w.requires_grad_(grad and p.requires_grad)
    return cfg, W


def _packed(lists):
    tokens = torch.cat(lists).cuda()
    pos = torch.cat([torch.arange(len(t)) for t in lists]).cuda().double()
    ends = np.cumsum([len(t) for t in lists]).tolist()
    return tokens, pos, list(zip([0] + ends[:-1], ends))


def _exact_rollout(case, seed):
    cfg, W = _weights64(case, seed, False)
    follows, new = _next_token(case["vocab"], seed), case["new"]
    prompts = _token_lists(case, seed)

    def extend(t, n):
        t = t.tolist()
        for _ in range(n):
            t.append(int(follows[t[-1]]))
        return torch.tensor(t)

    seqs = [extend(p, new) for p in prompts]
    for _ in range(8):   # the guess is the likeliest successor of each token; corrected where the model says otherwise
        tokens, pos, bounds = _packed(seqs)
        h, _ = _hidden(W, cfg, tokens, pos, bounds)
        rows = torch.cat([torch.arange(b - new - 1, b - 1) for _, b in bounds]).cuda()
        z = torch.log_softmax(h[rows] @ W["output_layer.weight"].T, -1).view(len(seqs), new, -1)
        best, again = z.argmax(-1).cpu(), False
        for k, s in enumerate(seqs):
            wrong = (best[k] != s[-new:]).nonzero()
            if len(wrong):
                w = int(wrong[0])
                seqs[k] = extend(torch.cat([s[:len(s) - new + w], best[k][w:w + 1]]), new - w - 1)
                again = True
        if not again:
            break
    lp = z.amax(-1).repeat_interleave(case["samples"], 0)
    return {"tokens": torch.stack([s[-new:] for s in seqs]).repeat_interleave(case["samples"], 0), "logprobs": lp}


def _exact_training(case, seed):
    train = case["kind"] != "logprobs"
    cfg, W = _weights64(case, seed, train)
    samples = _samples(case, seed)
    lists = [s["tokens"] for s in samples]
    pad = -sum(len(t) for t in lists) % 8     # the engine fills a packed batch up with a masked sequence
    tokens, pos, bounds = _packed(lists + [torch.zeros(pad, dtype=torch.long)] * (pad > 0))
    mask = torch.cat([s["mask"] for s in samples] + [torch.zeros(pad)]).cuda().double()
    targets = torch.roll(tokens, -1)
    with torch.set_grad_enabled(train):
        h, aux = _hidden(W, cfg, tokens, pos, bounds)
        at = mask.nonzero()[:, 0]
        parts = [_checkpoint(_scores, h[c], W["output_layer.weight"], targets[c]) for c in at.split(1024)]
        lp, ent = (torch.cat([p[k] for p in parts]) for k in (0, 1))
    if not train:
        out = [torch.zeros(tokens.numel(), dtype=torch.float64, device="cuda").index_copy(0, at, t) for t in (lp, ent)]
        n = tokens.numel() - pad
        return {"logprobs": out[0][:n], "entropy": out[1][:n]}
    if case["kind"] == "rl":
        adv = torch.cat([s["advantages"] for s in samples]).cuda().double()
        adv = torch.cat([adv, adv.new_zeros(pad)])[at]
        loss = -(adv * torch.exp(lp - lp.detach())).mean()
    else:
        loss = -lp.mean()
    trained = {n: w for n, w in W.items() if w.requires_grad}
    # the training engine's batch is one micro-batch: the balancing loss joins with weight one
    grads = dict(zip(trained, torch.autograd.grad(loss + aux, list(trained.values()))))
    norm = math.sqrt(sum(float(g.square().sum()) for g in grads.values()))
    return {"loss": float(loss), "grad_norm": norm, "grads": grads}


def _plan_attention(W, n, a, h):
    T, H, G, d = h.shape[0], a.heads, a.kv_heads, a.dim
    q = (h @ W[n + ".q"].T + W[n + ".q.b"]).view(T, H, d)
    k = (h @ W[n + ".k"].T + W[n + ".k.b"]).view(T, G, d)
    dist = torch.arange(T, device=h.device)[:, None] - torch.arange(T, device=h.device)
    hidden, out = (dist < 0) | (dist >= a.window), []
    for i in range(H):
        s = q[:, i] @ k[:, i // (H // G)].T * a.scale - 2.0 ** (-8.0 * (i + 1) / H) * dist
        out.append(torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ k[:, i // (H // G)])
    return torch.stack(out, 1).reshape(T, H * d) @ W[n + ".o"].T


def _plan_memory(W, n, m, h, eps):
    """Gated matrix memory, every output as a weighted sum over the earlier values."""
    T, H, d, dv, cap = h.shape[0], m.heads, m.dim, m.vdim, m.gate_cap
    q = (h @ W[n + ".q"].T).view(T, H, d) * d ** -0.5
    k, v = (h @ W[n + ".k"].T).view(T, H, d), (h @ W[n + ".v"].T).view(T, H, dv)
    gi, gf = (cap * torch.tanh((h @ W[n + f".{g}"].T + W[n + f".{g}.b"]) / cap) for g in "if")
    F = torch.nn.functional.logsigmoid(gf).cumsum(0)
    later, out = torch.ones(T, T, dtype=torch.bool, device=h.device).triu(1), []
    for a in range(H):
        D = (F[:, None, a] - F[None, :, a] + gi[None, :, a]).masked_fill(later, float("-inf"))
        mx = torch.maximum(D.amax(-1), F[:, a])
        P = torch.exp(D - mx[:, None]) * (q[:, a] @ k[:, a].T)
        out.append((P @ v[:, a]) / (torch.maximum(P.sum(-1).abs(), torch.exp(-mx)) + 1e-6)[:, None])
    y = _norm(torch.stack(out, 1), 1.0, eps).reshape(T, H * dv) * W[n + ".norm"] * torch.sigmoid(h @ W[n + ".g"].T)
    return y @ W[n + ".o"].T


def _exact_serve(case, seed):
    cfg, new, rows = _model_config(case), case["new"], []
    W = {n: t.double() for n, t in _plan_tensors(cfg, case, seed).items()}
    eps = cfg.rms_norm_eps
    for t in _token_lists(case, seed, new):
        t = t.cuda()
        x = W["embed"][t] + W["pos"][:len(t)]
        for i, spec in enumerate(cfg.layer_plan.layers):
            n = f"l{i}"
            h = _norm(x, 1 + W[n + ".norm1"], eps)
            a = _norm(_plan_attention(W, n + ".mix.left", spec.attention, h), W[n + ".mix.left.out"], eps)
            b = _norm(_plan_memory(W, n + ".mix.right", spec.memory, h, eps), W[n + ".mix.right.out"], eps)
            x = x + _norm(0.5 * (a + b), 1 + W[n + ".norm1b"], eps)
            h = _norm(x, 1 + W[n + ".norm2"], eps)
            y = (torch.nn.functional.silu(h @ W[n + ".mlp.gate"].T) * (h @ W[n + ".mlp.up"].T)) @ W[n + ".mlp.down"].T
            x = x + _norm(y, 1 + W[n + ".norm2b"], eps)
        rows.append(_norm(x[-new - 1:], 1 + W["final.norm"], eps) @ W["head"].T)
    return torch.stack(rows)


def exact(case, seed):
    with torch.random.fork_rng():
        if case["kind"] in ("rollout", "serve"):
            with torch.no_grad():
                return _exact_rollout(case, seed) if case["kind"] == "rollout" else _exact_serve(case, seed)
        return _exact_training(case, seed)
