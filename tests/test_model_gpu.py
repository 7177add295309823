"""Whole-model checks on the GPU: native bf16 forward/backward against the fp32 CPU reference path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _models(cfg_kw):
    from tunix_b200.models.config import ModelConfig
    from tunix_b200.models.transformer import create_model
    base = dict(num_layers=2, vocab_size=2048, embed_dim=256, hidden_dim=768, num_heads=4, head_dim=64,
                num_kv_heads=2, max_position=512)
    base.update(cfg_kw)
    cfg32 = ModelConfig(**base, dtype=torch.float32)
    ref = create_model(cfg32, seed=0)
    cfg16 = cfg32.replace(dtype=torch.bfloat16)
    gpu = create_model(cfg16, device=torch.device("cuda"), seed=1)
    with torch.no_grad():
        for (n, p), (_, q) in zip(ref.named_parameters(), gpu.named_parameters()):
            p.copy_(q.float().cpu())
    return ref, gpu


FAMILIES = {
    "llama": dict(family="llama3"),
    "qwen2": dict(family="qwen2", qkv_bias=True),
    "qwen3": dict(family="qwen3", qk_norm=True, head_dim=128),
    "gemma2": dict(family="gemma2", norm_add_one=True, embed_scale=True, activation="gelu", weight_tying=True,
                   attn_logit_softcap=50.0, final_logit_softcap=30.0, sliding_window=64,
                   layer_pattern=("local", "global"), post_norms=True, head_dim=256, num_heads=2, num_kv_heads=1),
}


@pytest.mark.parametrize("family", list(FAMILIES))
def test_forward_backward_matches_reference(family):
    from tunix_b200 import _lib
    from tunix_b200.sft.peft_trainer import _default_loss_fn
    ref, gpu = _models(FAMILIES[family])
    torch.manual_seed(0)
    toks = torch.randint(0, 2048, (2, 192))
    mask = torch.ones(2, 192)
    mask[:, :50] = 0
    out_ref = _default_loss_fn(ref, toks, mask)
    out_ref.loss.value().backward()
    out_gpu = _default_loss_fn(gpu, toks.cuda(), mask.cuda())
    out_gpu.loss.value().backward()
    _lib.raise_if_kernel_error()
    assert abs(out_gpu.loss.value().item() - out_ref.loss.value().item()) < 3e-2
    checked = 0
    for (n, p), (_, q) in zip(ref.named_parameters(), gpu.named_parameters()):
        if p.grad is None:
            continue
        g_ref, g = p.grad, q.grad.float().cpu()
        denom = g_ref.norm().item()
        if denom < 1e-8:
            continue
        rel = (g - g_ref).norm().item() / denom
        assert rel < 8e-2, (n, rel)
        checked += 1
    assert checked > 5


GEMMA4 = {
    "ple_shared": dict(num_layers=8, per_layer_input_dim=64, num_kv_shared_layers=4, kv_shared_hidden_dim=1536, num_kv_heads=1),
    "k_eq_v_wide_global": dict(num_layers=4, k_eq_v_global=True, num_global_kv_heads=1, num_kv_heads=2, global_head_dim=512),
    "moe": dict(num_layers=4, num_experts=8, num_experts_per_tok=2, moe_hidden_dim=128, num_kv_heads=2),
}


@pytest.mark.parametrize("case", list(GEMMA4))
def test_gemma4_forward_backward_matches_reference(case):
    """Gemma 4 text decoder in bf16 on the CUDA ops (flash attention for 64/128-wide heads, reference attention for
    the 512-wide global heads, grouped GEMMs for the experts) against the same weights in fp32 on the CPU."""
    from tunix_b200 import _lib
    from tunix_b200.models.gemma4 import Gemma4Config
    from tunix_b200.models.transformer import create_model
    from tunix_b200.sft.peft_trainer import _default_loss_fn
    kw = dict(vocab_size=2048, embed_dim=256, hidden_dim=768, num_heads=4, head_dim=64, global_head_dim=128,
              sliding_window=64, max_position=512, layer_pattern=("local", "local", "local", "global"))
    kw.update(GEMMA4[case])
    cfg32 = Gemma4Config._base(**kw, dtype=torch.float32)
    ref = create_model(cfg32, seed=0)
    gpu = create_model(cfg32.replace(dtype=torch.bfloat16), device=torch.device("cuda"), seed=1)
    with torch.no_grad():
        # the softmax scale is 1 and q, k are unit-RMS: with all-ones norm scales the scores have a standard
        # deviation of sqrt(H) and the softmax is close to an arg-max, which no bf16 / fp32 comparison survives;
        # a q-norm scale of 1/8 gives the scores of a trained model
        for n, q in gpu.named_parameters():
            if n.endswith("q_norm.weight"):
                q.fill_(0.125)
        for (n, p), (_, q) in zip(ref.named_parameters(), gpu.named_parameters()):
            p.copy_(q.float().cpu())
    torch.manual_seed(0)
    toks = torch.randint(0, 2048, (2, 192))
    mask = torch.ones(2, 192)
    mask[:, :50] = 0
    out_ref = _default_loss_fn(ref, toks, mask)
    out_ref.loss.value().backward()
    out_gpu = _default_loss_fn(gpu, toks.cuda(), mask.cuda())
    out_gpu.loss.value().backward()
    _lib.raise_if_kernel_error()
    assert abs(out_gpu.loss.value().item() - out_ref.loss.value().item()) < 3e-2
    checked = 0
    for (n, p), (_, q) in zip(ref.named_parameters(), gpu.named_parameters()):
        if p.grad is None or "router" in n or "per_expert" in n:      # routing flips on bf16 near-ties
            continue
        denom = p.grad.norm().item()
        if denom < 1e-8:
            continue
        rel = (q.grad.float().cpu() - p.grad).norm().item() / denom
        assert rel < (0.3 if case == "moe" else 0.12), (n, rel)
        checked += 1
    assert checked > 5


def test_smoke_entry():
    import __graft_entry__ as ge
    ge.smoke()


@pytest.mark.parametrize("how", ["subclass", "instance"])
def test_losses_call_a_replaced_token_logprobs_as_it_is_declared(how):
    """A model whose `token_logprobs` has been replaced, by a method or function that knows nothing of rows to pass over, trains as it did: the
    losses hand it every target and no further argument."""
    from tunix_b200.models.config import ModelConfig
    from tunix_b200.models.transformer import Transformer, create_model
    from tunix_b200.rl.common import compute_per_token_logps
    from tunix_b200.sft.peft_trainer import _default_loss_fn
    cfg = ModelConfig(num_layers=2, vocab_size=2048, embed_dim=256, hidden_dim=768, num_heads=4, head_dim=64, num_kv_heads=2, max_position=512,
                      dtype=torch.bfloat16)
    model = create_model(cfg, device=torch.device("cuda"), seed=0)
    seen = []

    class Own(type(model)):
        def token_logprobs(self, hidden, targets, *, temperature=1.0, want_entropy=False, chunk=None):
            seen.append(int(targets.min()))
            return Transformer.token_logprobs(self, hidden, targets, temperature=temperature, want_entropy=want_entropy, chunk=chunk)
    toks = torch.randint(3, 200, (2, 40), device="cuda")
    mask = torch.ones_like(toks)
    mask[:, :11] = 0
    want = _default_loss_fn(model, toks, mask)
    if how == "subclass":
        model.__class__ = Own
    else:
        model.token_logprobs = Own.token_logprobs.__get__(model)
    got = _default_loss_fn(model, toks, mask)
    assert float((got.loss.value() - want.loss.value()).detach().abs()) < 1e-4
    lp = compute_per_token_logps(model, toks[:, :20], toks[:, 20:], 0, -1, completion_mask=mask[:, :20], stop_gradient=False, skip_masked=True)
    assert lp.shape == (2, 20) and len(seen) == 2 and min(seen) >= 3
