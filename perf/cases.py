"""What a user of the framework runs: training steps, scoring of rollouts and generation, through the public entry points.

Four kinds of case, each over the decoder families the framework trains:

  sft       one optimizer step of `PeftTrainer.train` on token batches (full weights, or LoRA adapters on a frozen base)
  grpo      one optimizer step of the RL trainer on a micro-batch of scored rollouts (`algo_core.grpo_loss_fn`)
  score     log-probs and entropies of finished rollouts without gradients (`rl.common.compute_per_token_logps`)
  generate  a call of `PagedEngine`: prompts in, sampled tokens and their log-probs out

Models have the sizes of a preset with fewer layers, and a smaller vocabulary where the whole one would outweigh the few
layers. Weights and inputs are drawn here, from the seed alone, on the GPU; `exact` computes the same in 64 bits with plain
torch, from the same weights and inputs.

Generation needs a model that knows what comes next, as a trained one does: with random weights alone the best two tokens
are often closer than bf16 rounding, and one flipped token changes all that follow. So the output matrix leans, for each
token, towards the embedding of the token before it in a fixed random order.
"""
from __future__ import annotations

import math
import random

import torch
from torch.utils.checkpoint import checkpoint

PAD, EOS = 0, -1
LR, B1, B2, EPS = 1e-6, 0.9, 0.95, 1e-8
BETA = 0.04

# widths of the presets (`ModelConfig.<name>()`): D model, F feed-forward, N heads, K key / value heads, H head width
_SIZES = {
    "tiny_llama": dict(D=256, F=1024, N=4, K=2, H=64, theta=1e4, eps=1e-6),
    "qwen2p5_0p5b": dict(D=896, F=4864, N=14, K=2, H=64, theta=1e6, eps=1e-6, bias=True, tied=True),
    "deepseek_r1_distill_qwen_1p5b": dict(D=1536, F=8960, N=12, K=2, H=128, theta=1e6, eps=1e-6, bias=True),
    "llama3p2_3b": dict(D=3072, F=8192, N=24, K=8, H=128, theta=5e5, eps=1e-5, tied=True),
    "llama3p1_8b": dict(D=4096, F=14336, N=32, K=8, H=128, theta=5e5, eps=1e-5),
    "qwen3_8b": dict(D=4096, F=12288, N=32, K=8, H=128, theta=1e6, eps=1e-6, qk_norm=True),
    "gemma2_9b": dict(D=3584, F=14336, N=16, K=8, H=256, theta=1e4, eps=1e-6, tied=True, one=True, gelu=True, post=True,
                      embed_scale=True, cap=50.0, final_cap=30.0, window=4096),
    "qwen3_30b_a3b": dict(D=2048, F=768, N=32, K=4, H=128, theta=1e6, eps=1e-6, qk_norm=True, experts=128, top=8),
}


def listed():
    return [
        # the smallest training step: the CPU-sized decoder of the tests and examples on a GPU; launches and host work
        dict(name="sft_tiny", kind="sft", model="tiny_llama", layers=2, vocab=1024, batch=2, seq=64, prompt=16, accum=1),
        # fine-tuning of a small model on packed rows of odd length (several examples a row), biases, 64-wide heads
        dict(name="sft_packed_small", kind="sft", model="qwen2p5_0p5b", layers=4, vocab=32768, batch=3, seq=777, prompt=0,
             accum=1, packed=True),
        # the benchmark's micro-batches (2 x 2048 tokens, loss behind a prompt of 512) with gradient accumulation
        dict(name="sft_8b", kind="sft", model="llama3p1_8b", layers=4, vocab=32768, batch=2, seq=2048, prompt=512, accum=2),
        # long documents: one row of 16384 tokens
        dict(name="sft_long", kind="sft", model="qwen3_8b", layers=2, vocab=32768, batch=1, seq=16384, prompt=0, accum=1),
        # adapters on a frozen base with soft-capped, 256-wide heads, as in preference tuning: rows of prompt + response
        dict(name="lora_gemma2", kind="sft", model="gemma2_9b", layers=2, vocab=32768, batch=4, seq=1001, prompt=500, accum=1,
             rank=16),
        # GRPO micro-batch: 8 rollouts of one prompt, 256 + 768 tokens, ragged at both ends
        dict(name="grpo_8b", kind="grpo", model="qwen3_8b", layers=2, vocab=32768, batch=8, seq=1024, prompt=256, accum=1),
        # the same for a mixture of experts, with the sampler's routing replayed
        dict(name="grpo_moe", kind="grpo", model="qwen3_30b_a3b", layers=1, vocab=32768, batch=8, seq=1024, prompt=256, accum=1),
        # log-probs of rollouts under the reference or old policy
        dict(name="score_8b", kind="score", model="qwen3_8b", layers=4, vocab=32768, batch=16, seq=1024, prompt=256),
        # one short question to a small model, greedy: latency of a call
        dict(name="chat_small", kind="generate", model="deepseek_r1_distill_qwen_1p5b", layers=8, vocab=151936, batch=1,
             prompt=37, new=24, sampled=False),
        # rollouts: 64 running sequences, sampled with top-k and top-p over the whole vocabulary
        dict(name="rollout_64", kind="generate", model="qwen3_8b", layers=4, vocab=151936, batch=64, prompt=256, new=48,
             sampled=True),
        # long prompts, first token only: what a caller of the server waits for
        dict(name="first_token_4k", kind="generate", model="llama3p1_8b", layers=4, vocab=128256, batch=8, prompt=4096, new=1,
             sampled=False),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case. Rows and lengths are spread over their logarithm, odd ones included, up to the listed totals."""
    kind = rng.choice(["sft", "sft", "lora", "grpo", "score", "generate", "generate"])
    if kind in ("sft", "lora"):
        model = rng.choice(["tiny_llama", "qwen2p5_0p5b", "llama3p2_3b", "llama3p1_8b", "qwen3_8b"]) if kind == "sft" else \
            rng.choice(["gemma2_9b", "llama3p1_8b", "qwen3_8b"])
        seq = _log(rng, 64, 16384 if kind == "sft" else 4096)
        rows = max(1, 8192 // seq)
        case = dict(kind="sft", model=model, layers=rng.randint(1, 2), vocab=rng.choice([1024, 8192, 32768]),
                    batch=_log(rng, 1, rows), seq=seq, prompt=rng.choice([0, seq // 4]), accum=rng.choice([1, 1, 2]))
        if kind == "lora":
            case["rank"] = rng.choice([8, 16, 32])
        elif rng.random() < 0.4:
            case["packed"], case["prompt"] = True, 0
        return case
    if kind in ("grpo", "score"):
        model = rng.choice(["qwen2p5_0p5b", "llama3p1_8b", "qwen3_8b"] + (["qwen3_30b_a3b"] if kind == "grpo" else []))
        seq = _log(rng, 96, 4096)
        return dict(kind=kind, model=model, layers=1 if model == "qwen3_30b_a3b" else rng.randint(1, 2),
                    vocab=rng.choice([8192, 32768]), batch=_log(rng, 1, max(1, min(64, 8192 // seq))), seq=seq,
                    prompt=max(8, int(seq * rng.uniform(0.1, 0.6))), **({"accum": 1} if kind == "grpo" else {}))
    model = rng.choice(["deepseek_r1_distill_qwen_1p5b", "llama3p1_8b", "qwen3_8b"])
    prompt = _log(rng, 5, 4096)
    batch = _log(rng, 1, max(1, min(128, 16384 // prompt)))
    return dict(kind="generate", model=model, layers=rng.randint(2, 4), vocab=rng.choice([32768, 151936]), batch=batch,
                prompt=prompt, new=rng.choice([1, 8, 16, 32]), sampled=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ weights and inputs
def _gen(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt) % (1 << 62))


def _shapes(case):
    """(name, shape, standard deviation or None for a norm, "bias" for a bias), in the order of the model's parameters."""
    s, V, L = _SIZES[case["model"]], case["vocab"], case["layers"]
    D, F, N, K, H = s["D"], s["F"], s["N"], s["K"], s["H"]
    deep = 0.02 / math.sqrt(2 * L)
    tied = s.get("tied", False)
    # for generation the embedding outweighs what the layers add, so that the last hidden state tells its token
    out = [("embed_tokens", (V, D), 0.02 if tied else 3.0 if case["kind"] == "generate" else 1.0)]
    if not tied:
        out.append(("lm_head", (V, D), 0.02))
    for i in range(L):
        p = f"layers.{i}."
        out.append((p + "input_layernorm.weight", (D,), None))
        for name, o, k, std in (("q_proj", N * H, D, 0.02), ("k_proj", K * H, D, 0.02), ("v_proj", K * H, D, 0.02),
                                ("o_proj", D, N * H, deep)):
            out.append((p + f"self_attn.{name}.weight", (o, k), std))
            if s.get("bias") and name != "o_proj":
                out.append((p + f"self_attn.{name}.bias", (o,), "bias"))
        if s.get("qk_norm"):
            out += [(p + "self_attn.q_norm.weight", (H,), None), (p + "self_attn.k_norm.weight", (H,), None)]
        out.append((p + "post_attention_layernorm.weight", (D,), None))
        if "experts" in s:
            E = s["experts"]
            out += [(p + "mlp.gate_proj", (E, F, D), 0.02), (p + "mlp.up_proj", (E, F, D), 0.02),
                    (p + "mlp.down_proj", (E, D, F), deep), (p + "mlp.router.weight", (E, D), 0.02)]
        else:
            out += [(p + "mlp.gate_proj.weight", (F, D), 0.02), (p + "mlp.up_proj.weight", (F, D), 0.02),
                    (p + "mlp.down_proj.weight", (D, F), deep)]
        if s.get("post"):
            out += [(p + "post_attn_norm.weight", (D,), None), (p + "post_ffw_norm.weight", (D,), None)]
    out.append(("norm.weight", (D,), None))
    return out


def _weights(case, seed):
    """Every parameter by name, bf16."""
    g, s, w = _gen(seed, 1), _SIZES[case["model"]], {}
    for name, shape, std in _shapes(case):
        t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
        if std is None:
            t.normal_(0.0 if s.get("one") else 1.0, 0.1, generator=g)
        else:
            t.normal_(0.0, 0.1 if std == "bias" else std, generator=g)
        w[name] = t
    if case["kind"] == "generate":
        head, emb, nxt = w["lm_head"], w["embed_tokens"], _follower(case, seed)
        # the follower's logit against the sum over all others: enough for top-p 0.95 to keep it alone, or well ahead of the next.
        # A last hidden state lies at a cosine of about 0.93 from the embedding of its token.
        rest = math.log(case["vocab"]) + 0.5 * s["D"] * 0.02 ** 2
        lean = (rest + (6.0 if case["sampled"] else -1.0)) / (0.93 * math.sqrt(s["D"]))
        for a in range(0, case["vocab"], 16384):       # in slices: no 32-bit copy of the whole matrix
            rows = nxt[a:a + 16384]
            e = emb[a:a + 16384].float()
            head[rows] = (head[rows].float() + lean * e / e.norm(dim=1, keepdim=True)).to(torch.bfloat16)
    return w


def _follower(case, seed):
    """The token that the model holds for most likely after each token."""
    return torch.randperm(case["vocab"], generator=_gen(seed, 2), device="cuda")


def _adapters(case, seed):
    """LoRA factors by projection name: A [r, in], B [out, r]."""
    g, out = _gen(seed, 3), {}
    for name, shape, _ in _shapes(case):
        if name.endswith("_proj.weight"):
            a = torch.empty(case["rank"], shape[1], device="cuda").normal_(0.0, 1.0 / math.sqrt(shape[1]), generator=g)
            b = torch.empty(shape[0], case["rank"], device="cuda").normal_(0.0, 0.02, generator=g)
            out[name[:-len(".weight")]] = (a.bfloat16(), b.bfloat16())
    return out


def _lengths(case, seed, low, high, n):
    """n row lengths between two fractions' bounds, the longest among them."""
    r = random.Random(int(seed) * 7919 + 11)
    v = [r.randint(max(1, low), max(1, high)) for _ in range(n)]
    v[r.randrange(n)] = max(1, high)
    return v


def _batches(case, seed):
    """SFT micro-batches: tokens int32 [B, T], mask fp32 [B, T], and segment ids / positions where rows are packed."""
    out = []
    B, T, V = case["batch"], case["seq"], case["vocab"]
    for m in range(case["accum"]):
        g = _gen(seed, 100 + m)
        toks = torch.randint(1, V, (B, T), generator=g, device="cuda", dtype=torch.int32)
        mask = torch.zeros(B, T, device="cuda")
        mask[:, case["prompt"]:] = 1
        b = {"input_tokens": toks, "input_mask": mask}
        if case.get("packed"):
            r = random.Random(int(seed) * 31 + m)
            seg, pos = torch.zeros(B, T, dtype=torch.int32), torch.zeros(B, T, dtype=torch.int32)
            for i in range(B):
                at, k = 0, 1
                while at < T:
                    n = min(T - at, r.randint(max(1, T // 6), max(1, T // 2)))
                    seg[i, at:at + n], pos[i, at:at + n] = k, torch.arange(n, dtype=torch.int32)
                    at, k = at + n, k + 1
            b["segment_ids"], b["positions"] = seg.cuda(), pos.cuda()
            mask[:, 1:] *= (b["segment_ids"][:, 1:] == b["segment_ids"][:, :-1]).float()      # nothing predicts a first token
        out.append(b)
    return out


def _rollouts(case, seed):
    """Left-padded prompts, right-padded completions, their mask, advantages and reference log-probs."""
    B, P, C, V = case["batch"], case["prompt"], case["seq"] - case["prompt"], case["vocab"]
    g = _gen(seed, 200)
    ids = torch.randint(1, V, (B, P + C), generator=g, device="cuda")
    pl = torch.tensor(_lengths(case, seed, P // 2, P, B), device="cuda")[:, None]
    cl = torch.tensor(_lengths(case, seed + 1, C // 3, C, B), device="cuda")[:, None]
    prompt = torch.where(torch.arange(P, device="cuda")[None] >= P - pl, ids[:, :P], PAD)
    cmask = (torch.arange(C, device="cuda")[None] < cl).to(torch.int32)
    r = {"prompt": prompt, "completion": torch.where(cmask > 0, ids[:, P:], PAD), "mask": cmask,
         "advantages": torch.randn(B, generator=g, device="cuda"),
         "ref": -math.log(V) + torch.randn(B, C, generator=g, device="cuda")}
    s = _SIZES[case["model"]]
    if "experts" in s:
        scores = torch.rand(B * (P + C) * case["layers"], s["experts"], generator=g, device="cuda")
        r["routed"] = scores.topk(s["top"], dim=1).indices.view(B, P + C, case["layers"], s["top"])
    return r


def _prompts(case, seed):
    P = case["prompt"]
    g = torch.Generator().manual_seed(int(seed) + 5)
    return [torch.randint(1, case["vocab"], (n,), generator=g).tolist()
            for n in _lengths(case, seed, P // 4 if case["batch"] > 1 else P, P, case["batch"])]


class _Ids:
    """Token ids in place of text."""

    def encode(self, text, **_):
        return [int(t) for t in text.split()]

    def decode(self, ids, **_):
        return ""

    def bos_id(self):
        return None

    def eos_id(self):
        return EOS

    def pad_id(self):
        return PAD


# --------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    from tunix_b200 import lora, optim
    from tunix_b200.common.configs import CacheConfig, TrainingConfig
    from tunix_b200.generate.engine import PagedEngine
    from tunix_b200.models.config import get_config
    from tunix_b200.models.transformer import create_model
    from tunix_b200.rl import algo_core
    from tunix_b200.rl.algorithm_config import GRPOConfig
    from tunix_b200.rl.common import TrainExample
    from tunix_b200.rl.trainer import Trainer
    from tunix_b200.sft.peft_trainer import PeftTrainer

    longest = case.get("seq", 0) or case["prompt"] + case["new"]
    cfg = get_config(case["model"]).replace(num_layers=case["layers"], vocab_size=case["vocab"], dtype=torch.bfloat16,
                                            max_position=longest + 64)
    model = create_model(cfg, device="cuda", init=False)
    weights = _weights(case, seed)
    own = dict(model.named_parameters())
    if list(own) != list(weights):
        raise RuntimeError("the model's parameters are not those of the case")
    with torch.no_grad():
        for name, p in own.items():
            p.copy_(weights[name])
    del weights
    if case.get("rank"):
        lora.apply_lora_to_model(model, lora.LoraProvider(module_path=r".*_proj", rank=case["rank"], alpha=2.0 * case["rank"]))
        with torch.no_grad():
            for name, (a, b) in _adapters(case, seed).items():
                mod = model.get_submodule(name)
                mod.lora_a.copy_(a)
                mod.lora_b.copy_(b)
    if case["kind"] == "score":
        return {"kind": "score", "model": model.eval(), **_rollouts(case, seed)}
    if case["kind"] == "generate":
        cache = (longest + 63) // 64 * 64 + 64
        engine = PagedEngine(model, _Ids(), CacheConfig(cache, cfg.num_layers, cfg.num_kv_heads, cfg.head_dim), page_size=64,
                             max_running_requests=case["batch"], prefix_caching=False)
        how = dict(temperature=0.9, top_k=50, top_p=0.95) if case["sampled"] else dict(temperature=0.0)
        return {"kind": "generate", "engine": engine, "prompts": _prompts(case, seed), "call": dict(
            max_generation_steps=case["new"], max_prompt_length=case["prompt"], return_logprobs=True, eos_tokens=[EOS],
            seed=int(seed) & 0xFFFF, pad_output=True, **how)}
    tc = TrainingConfig(eval_every_n_steps=10 ** 9, max_steps=None, gradient_accumulation_steps=case["accum"],
                        pbar_description=None, resume_from_checkpoint_on_init=False)
    opt = optim.AdamW(LR, b1=B1, b2=B2, eps=EPS, weight_decay=0.0, max_grad_norm=1.0)
    if case["kind"] == "grpo":
        trainer = Trainer(model, opt, tc)
        conf = GRPOConfig(beta=BETA, num_generations=2)
        trainer.with_loss_fn(lambda m, train_example: algo_core.grpo_loss_fn(m, train_example, conf, PAD, EOS), has_aux=True)
        trainer.with_gen_model_input_fn(lambda ex: {"train_example": ex})
        r = _rollouts(case, seed)
        batches = [TrainExample(prompt_ids=r["prompt"], prompt_mask=(r["prompt"] != PAD).to(torch.int32),
                                completion_ids=r["completion"], completion_mask=r["mask"], advantages=r["advantages"],
                                ref_per_token_logps=r["ref"], routed_experts=r.get("routed"))]
    else:
        trainer = PeftTrainer(model, opt, tc)
        trainer.is_managed_externally = True
        batches = _batches(case, seed)
    return {"kind": "train", "trainer": trainer, "batches": batches}


def run(state):
    if state["kind"] == "train":
        trainer = state["trainer"]
        trainer.train(state["batches"])
        opt = trainer.optimizer
        return {"mu": opt.m, "master": opt.buffers.master}      # running mean of the gradients, and the 32-bit weights
    if state["kind"] == "score":
        from tunix_b200.rl.common import compute_per_token_logps
        logp, ent = compute_per_token_logps(state["model"], state["prompt"], state["completion"], PAD, EOS,
                                            completion_mask=state["mask"], return_entropy=True)
        return {"logp": logp, "entropy": ent}
    out = state["engine"](prompt_token_ids=state["prompts"], **state["call"])
    return {"tokens": torch.from_numpy(out.tokens), "logprobs": torch.tensor(out.logprobs)}


# ------------------------------------------------------------------------------------------------- work and tolerance
def _matrix_params(case):
    """(parameters in the layers, those among them that a token passes, parameters of the vocabulary matrices, of one)."""
    s, layer, passed = _SIZES[case["model"]], 0, 0
    for name, shape, std in _shapes(case):
        if name.startswith("layers."):
            n = math.prod(shape)
            layer += n
            if len(shape) > 1:
                passed += n * s["top"] // s["experts"] if len(shape) == 3 else n
    one = case["vocab"] * s["D"]
    return layer, passed, one * (1 if s.get("tied") else 2), one


def work(case):
    s = _SIZES[case["model"]]
    layers, passed, vocab, head = _matrix_params(case)
    L, NH, KH = case["layers"], s["N"] * s["H"], s["K"] * s["H"]
    if case["kind"] == "generate":
        B, P, n = case["batch"], case["prompt"], case["new"]
        toks = B * (0.625 * P if B > 1 else P)
        att = 4 * L * NH * B * ((0.43 * P * P if B > 1 else P * P) / 2 + (n - 1) * (0.625 * P + n / 2))
        fl = 2 * passed * (toks + B * (n - 1)) + 2 * head * B * n + att
        by = n * 2 * (layers + head) + 2 * B * n * s["D"] + 4 * L * KH * (toks + B * (n - 1) * (0.625 * P + n / 2))
        return {"bytes": by, "flops": fl}
    B, T = case["batch"], case["seq"]
    if case.get("packed"):
        pairs = B * T * T / 6
    else:
        w = s.get("window", 0)
        pairs = B * T * T / 2 if not w or w >= T else B * (T * w - w * w / 2)      # the longer of the alternating layers
    toks = B * T
    scored = B * (T - case["prompt"])
    fwd = 2 * passed * toks + 2 * head * scored + 4 * L * NH * pairs
    if case["kind"] == "score":
        return {"bytes": 2 * (layers + head) + 2 * toks * s["D"] + 8 * scored, "flops": fwd}
    if case.get("rank"):
        r = case["rank"]
        ad = sum(r * sum(shape) for name, shape, _ in _shapes(case) if name.endswith("_proj.weight"))
        fl = (2 * fwd + 4 * L * NH * pairs + 6 * ad * toks) * case["accum"]
        return {"bytes": 2 * (layers + vocab) + 28 * ad + 2 * toks * s["D"], "flops": fl}
    # weights 2 + 2 bytes, master and both moments 12 + 12
    return {"bytes": 28 * (layers + vocab) + 8 * toks * case["accum"], "flops": 3 * fwd * case["accum"]}


def tolerance(case):
    # measured against `exact`: gradients are off by 0.3 to 1.5 %, log-probs by 0.1 %, those of generated tokens by 0.2 to 0.7 %
    if case["kind"] == "generate":
        return {"rel": 0.025, "max": 0.5, "differ": 0.005}
    if case["kind"] == "score":
        return {"rel": 0.004, "max": 0.05}
    return {"rel": 0.03, "max": 0.9}


# -------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm64(x, w, s):
    w = w + 1.0 if s.get("one") else w
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + s["eps"]) * w


def _rotate64(x, pos, s):
    """x [T, heads, H], pos [T]"""
    half = s["H"] // 2
    inv = s["theta"] ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    ang = pos.double()[:, None] * inv
    c, sn = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * sn, b * c + a * sn], -1)


def _heads64(q, k, v, seg, s, window):
    """Query heads of one key / value head: q [T, G, H], k, v [T, H] -> [T, G, H]"""
    T = q.shape[0]
    i = torch.arange(T, device=q.device)
    see = (i[None] <= i[:, None]) & (seg[None] == seg[:, None])
    if window:
        see &= i[None] > i[:, None] - window
    out = []
    for h in range(q.shape[1]):
        z = q[:, h] @ k.t() * (s["H"] ** -0.5)
        if s.get("cap"):
            z = s["cap"] * torch.tanh(z / s["cap"])
        out.append(torch.softmax(z.masked_fill(~see, float("-inf")), -1) @ v)
    return torch.stack(out, 1)


def _act64(x, s):
    return torch.nn.functional.gelu(x, approximate="tanh") if s.get("gelu") else torch.nn.functional.silu(x)


def _layer64(x, w, p, pos, seg, routed, s, local, scale, grad):
    """One decoder layer on x [B, T, D]."""
    B, T, D = x.shape
    N, K, H = s["N"], s["K"], s["H"]

    def proj(name, y):
        o = y @ w[p + name + ".weight"].t()
        if p + name + ".bias" in w:
            o = o + w[p + name + ".bias"]
        if p + name + ".lora_a" in w:
            o = o + scale * (y @ w[p + name + ".lora_a"].t()) @ w[p + name + ".lora_b"].t()
        return o

    h = _norm64(x, w[p + "input_layernorm.weight"], s)
    q = proj("self_attn.q_proj", h).view(B, T, N, H)
    k = proj("self_attn.k_proj", h).view(B, T, K, H)
    v = proj("self_attn.v_proj", h).view(B, T, K, H)
    if s.get("qk_norm"):
        q, k = _norm64(q, w[p + "self_attn.q_norm.weight"], s), _norm64(k, w[p + "self_attn.k_norm.weight"], s)
    rows = []
    for b in range(B):
        qb, kb = _rotate64(q[b], pos[b], s), _rotate64(k[b], pos[b], s)
        G = N // K
        one = []
        for j in range(K):
            part = (qb[:, j * G:(j + 1) * G], kb[:, j], v[b, :, j], seg[b], s, s.get("window", 0) if local else 0)
            if grad and T > 4096:                       # head by head, recomputed in the backward pass
                one += [checkpoint(_heads64, part[0][:, g:g + 1], *part[1:], use_reentrant=False) for g in range(G)]
            else:
                one.append(checkpoint(_heads64, *part, use_reentrant=False) if grad else _heads64(*part))
        rows.append(torch.cat(one, 1))
    a = proj("self_attn.o_proj", torch.stack(rows).reshape(B, T, N * H))
    x = x + (_norm64(a, w[p + "post_attn_norm.weight"], s) if s.get("post") else a)
    h = _norm64(x, w[p + "post_attention_layernorm.weight"], s)
    if "experts" in s:
        flat = h.reshape(B * T, D)
        prob = torch.softmax(flat @ w[p + "mlp.router.weight"].t(), -1)
        idx = routed.reshape(B * T, -1)
        wt = prob.gather(1, idx)
        wt = wt / wt.sum(-1, keepdim=True)
        y = torch.zeros_like(flat)
        for e in range(s["experts"]):
            t, j = (idx == e).nonzero(as_tuple=True)
            r = flat[t]
            u = _act64(r @ w[p + "mlp.gate_proj"][e].t(), s) * (r @ w[p + "mlp.up_proj"][e].t())
            y = y.index_add(0, t, wt[t, j][:, None] * (u @ w[p + "mlp.down_proj"][e].t()))
        m = y.view(B, T, D)
    else:
        m = proj("mlp.down_proj", _act64(proj("mlp.gate_proj", h), s) * proj("mlp.up_proj", h))
    return x + (_norm64(m, w[p + "post_ffw_norm.weight"], s) if s.get("post") else m)


def _hidden64(w, case, tokens, pos, seg, routed=None, grad=False):
    s = _SIZES[case["model"]]
    x = w["embed_tokens"][tokens.long()]
    if s.get("embed_scale"):
        x = x * math.sqrt(s["D"])
    for i in range(case["layers"]):
        local = "window" in s and i % 2 == 0
        r = None if routed is None else routed[:, :, i]
        args = (x, w, f"layers.{i}.", pos, seg, r, s, local, 2.0, grad)
        x = checkpoint(_layer64, *args, use_reentrant=False) if grad else _layer64(*args)
    return _norm64(x, w["norm.weight"], s)


def _scores64(h, w, case, targets):
    """(log p(target), entropy) per row of h [rows, D]."""
    s = _SIZES[case["model"]]
    z = h @ w.get("lm_head", w["embed_tokens"]).t()
    if s.get("final_cap"):
        z = s["final_cap"] * torch.tanh(z / s["final_cap"])
    z = torch.log_softmax(z, -1)
    return z.gather(1, targets.long()[:, None])[:, 0], -(z.exp() * z).sum(-1)


def _logp64(h, w, case, targets, grad=False):
    h, t = h.reshape(-1, h.shape[-1]), targets.reshape(-1)
    parts = []
    for a in range(0, h.shape[0], 2048):
        args = (h[a:a + 2048], w, case, t[a:a + 2048])
        parts.append(checkpoint(_scores64, *args, use_reentrant=False) if grad else _scores64(*args))
    return tuple(torch.cat([p[j] for p in parts]).view(targets.shape) for j in (0, 1))


def _positions(mask):
    return (mask.cumsum(-1) - 1).clamp(min=0)


def exact(case, seed):
    try:
        return _exact(case, seed)
    finally:
        torch.cuda.empty_cache()


def _exact(case, seed):
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    if case["kind"] == "generate":
        with torch.no_grad():
            return _generated64(w, case, seed)
    if case["kind"] in ("grpo", "score"):
        r = _rollouts(case, seed)
        ids = torch.cat([r["prompt"], r["completion"]], 1)
        seg = torch.cat([(r["prompt"] != PAD).int(), r["mask"]], 1)
    if case["kind"] == "score":
        with torch.no_grad():
            h = _hidden64(w, case, ids, _positions(seg), seg)
            logp, ent = _logp64(h[:, case["prompt"] - 1:-1], w, case, r["completion"])
            return {"logp": logp, "entropy": ent}
    train = list(w)
    if case.get("rank"):
        train = []
        for name, _, _ in _shapes(case):
            base = name[:-len(".weight")]
            if name.endswith("_proj.weight"):
                a, b = _adapters_of(case, seed)[base]
                w[base + ".lora_a"], w[base + ".lora_b"] = a, b
                train += [base + ".lora_a", base + ".lora_b"]
    for n in train:
        w[n].requires_grad_(True)
    if case["kind"] == "grpo":
        # first step on fresh rollouts: the ratio is one and its gradient that of the log-prob
        h = _hidden64(w, case, ids, _positions(seg), seg, r.get("routed"), grad=True)
        logp, _ = _logp64(h[:, case["prompt"] - 1:-1], w, case, r["completion"], grad=True)
        m = r["mask"].double()
        per = (BETA - r["advantages"].double()[:, None]) * logp * m
        (per.sum(1) / m.sum(1).clamp(min=1)).sum().backward()
        den = float((m.sum(1) > 0).sum())
    else:
        den = 0.0
        for b in _batches(case, seed):
            toks = b["input_tokens"]
            B, T = toks.shape
            pos = b["positions"] if "positions" in b else torch.arange(T, device="cuda")[None].expand(B, T)
            seg = b["segment_ids"] if "segment_ids" in b else torch.ones(B, T, device="cuda")
            h = _hidden64(w, case, toks, pos, seg, grad=True)
            logp, _ = _logp64(h[:, :-1], w, case, toks[:, 1:], grad=True)
            m = b["input_mask"][:, 1:].double()
            (-(logp * m).sum()).backward()
            den += float(m.sum())
    grads = {n: w[n].grad / max(den, 1e-8) for n in train}
    total = math.sqrt(sum(float(g.square().sum()) for g in grads.values()))
    mu, master = [], []
    for n in train:
        g = (grads[n] / max(total, 1.0)).reshape(-1)
        step = g / (g.abs() + EPS)                                  # first step: both moments are unbiased at once
        gap = (-g.numel()) % 128                                    # a parameter starts at a multiple of 128
        mu.append(torch.nn.functional.pad((1 - B1) * g, (0, gap)))
        master.append(torch.nn.functional.pad(w[n].detach().reshape(-1) - LR * step, (0, gap)))
    return {"mu": torch.cat(mu), "master": torch.cat(master)}


def _adapters_of(case, seed):
    return {n: (a.double(), b.double()) for n, (a, b) in _adapters(case, seed).items()}


def _generated64(w, case, seed):
    """Row by row: the chain of most likely followers is fed as a whole, and the best token at each place is what a greedy
    run, or one whose top-p keeps the best token alone, generates."""
    nxt, n = _follower(case, seed).cpu(), case["new"]
    temp = 0.9 if case["sampled"] else 1.0
    toks, lps = [], []
    for row in _prompts(case, seed):
        ids = list(row)
        for _ in range(n - 1):
            ids.append(int(nxt[ids[-1]]))
        t = torch.tensor(ids, device="cuda")[None]
        one = torch.ones_like(t)
        h = _hidden64(w, case, t, _positions(one), one)[0, len(row) - 1:]
        z = torch.log_softmax(h @ w["lm_head"].t() / temp, -1)
        best = z.max(-1)
        toks.append(best.indices)
        lps.append(best.values)
    return {"tokens": torch.stack(toks), "logprobs": torch.stack(lps)}
