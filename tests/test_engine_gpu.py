"""Paged engine (paged KV, CUDA-graphed decode) against the dense-cache Sampler, and kernel-level checks."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


class Tok:
    def encode(self, s):
        return [3 + (ord(c) % 200) for c in s]

    def decode(self, ids):
        return " ".join(str(int(i)) for i in ids)

    def bos_id(self):
        return 1

    def eos_id(self):
        return 2

    def pad_id(self):
        return 0


def _model(**kw):
    from tunix_b200.models.config import ModelConfig
    from tunix_b200.models.transformer import create_model
    base = dict(family="qwen3", num_layers=2, vocab_size=512, embed_dim=256, hidden_dim=512, num_heads=4, head_dim=64,
                num_kv_heads=2, qk_norm=True, dtype=torch.bfloat16, max_position=512)
    base.update(kw)
    return create_model(ModelConfig(**base), device=torch.device("cuda"), seed=0)


@pytest.mark.parametrize("page", [16, 64])          # 64-token pages are staged by TMA, smaller ones gathered by cp.async
@pytest.mark.parametrize("N,KH,H,window,softcap", [(8, 2, 128, 0, 0.0), (4, 4, 64, 0, 0.0), (16, 2, 256, 0, 30.0),
                                                   (8, 1, 128, 100, 0.0), (32, 2, 128, 0, 0.0)])
def test_paged_decode_kernel_matches_reference(N, KH, H, window, softcap, page):
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as K
    torch.manual_seed(0)
    B, max_pages = 5, 640 // page
    lens = torch.tensor([1, 17, 300, 600, 255], device="cuda", dtype=torch.int32)
    num_pages = B * max_pages
    kp = torch.randn(num_pages, page, KH * H, device="cuda", dtype=torch.bfloat16)
    vp = torch.randn_like(kp)
    perm = torch.randperm(num_pages, device="cuda").int().view(B, max_pages)
    big = torch.randn(B, N * H + 64, device="cuda", dtype=torch.bfloat16)      # q rows with a stride, as the engine passes them
    q = big[:, :N * H].view(B, N, H)
    slots = torch.arange(B, device="cuda", dtype=torch.int32)
    out = K.paged_decode(q, kp, vp, perm, slots, lens, num_kv_heads=KH, page_size=page, max_ctx=640, scale=1 / math.sqrt(H),
                         window=window, softcap=softcap)
    for split in (64, 128, 256, 512, 640):   # the context split per CTA only changes the schedule (640: one split, no combine)
        again = K.paged_decode(q, kp, vp, perm, slots, lens, num_kv_heads=KH, page_size=page, max_ctx=640,
                               scale=1 / math.sqrt(H), window=window, softcap=softcap, split_tokens=split)
        assert torch.allclose(again.float(), out.float(), atol=2e-2, rtol=2e-2), split
    _lib.raise_if_kernel_error()
    for b in range(B):
        L = int(lens[b])
        idx = torch.arange(L, device="cuda")
        rows = perm[b][idx // page].long() * page + idx % page
        k = kp.view(-1, KH, H)[rows].float()
        v = vp.view(-1, KH, H)[rows].float()
        kk = k.repeat_interleave(N // KH, dim=1)
        vv = v.repeat_interleave(N // KH, dim=1)
        s = torch.einsum("nh,lnh->nl", q[b].float(), kk) / math.sqrt(H)
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if window:
            s = s.masked_fill(idx[None] < L - window, float("-inf"))
        ref = torch.einsum("nl,lnh->nh", torch.softmax(s, -1), vv)
        assert torch.allclose(out[b].float(), ref, atol=2e-2, rtol=2e-2), b


@pytest.mark.parametrize("H,qk_norm", [(128, True), (64, False), (256, True)])
def test_qkv_post_matches_separate_kernels(H, qk_norm):
    from tunix_b200.ops import kernels as K
    torch.manual_seed(1)
    n_tok, N, KH, page, max_pages = 7, 4, 2, 16, 8
    qkv = torch.randn(n_tok, (N + 2 * KH) * H, device="cuda", dtype=torch.bfloat16)
    ref = qkv.clone()
    pos = torch.tensor([0, 5, 17, -1, 33, 100, 2], device="cuda", dtype=torch.int32)
    slots = torch.arange(n_tok, device="cuda", dtype=torch.int32)
    table = torch.randperm(n_tok * max_pages, device="cuda").int().view(n_tok, max_pages)
    kp = torch.zeros(n_tok * max_pages, page, KH * H, device="cuda", dtype=torch.bfloat16)
    vp = torch.zeros_like(kp)
    kp2, vp2 = kp.clone(), vp.clone()
    qw = torch.randn(H, device="cuda", dtype=torch.bfloat16) if qk_norm else None
    kw = torch.randn(H, device="cuda", dtype=torch.bfloat16) if qk_norm else None
    inv = 1.0 / (10000.0 ** (torch.arange(0, H // 2, device="cuda").float() / (H // 2)))
    ang = torch.arange(128, device="cuda").float()[:, None] * inv[None]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    K.qkv_post(qkv, slots, pos, qw, kw, 1e-6, False, cos, sin, table, page, kp, vp, N, KH, H)
    q = ref[:, :N * H].reshape(n_tok * N, H)
    k = ref[:, N * H:(N + KH) * H].reshape(n_tok * KH, H)
    v = ref[:, (N + KH) * H:].contiguous()
    if qk_norm:
        q, _ = K.rmsnorm_fwd(q.contiguous(), qw, 1e-6, want_rstd=False)
        k, _ = K.rmsnorm_fwd(k.contiguous(), kw, 1e-6, want_rstd=False)
    q, k = q.reshape(n_tok, N, H).contiguous(), k.reshape(n_tok, KH, H).contiguous()
    cpos = pos.clamp(min=0)
    K.rope_(q, cpos, cos, sin)
    K.rope_(k, cpos, cos, sin)
    K.kv_write(k.view(n_tok, -1), v, slots, pos, table, page, kp2, vp2)
    valid = pos >= 0
    assert torch.allclose(qkv[:, :N * H].view(n_tok, N, H)[valid].float(), q[valid].float(), atol=2e-2, rtol=2e-2)
    assert torch.allclose(kp.float(), kp2.float(), atol=2e-2, rtol=2e-2)
    assert torch.equal(vp, vp2)


@pytest.mark.parametrize("M,N,K_", [(8, 4096, 512), (64, 1024, 4096), (100, 12288, 256), (64, 24576, 512), (32, 151936, 256),
                                    (128, 6144, 1024), (17, 5000, 320)])
def test_small_m_gemm_tiles(M, N, K_):
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as K
    torch.manual_seed(1)
    A = torch.randn(M, K_, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K_, device="cuda", dtype=torch.bfloat16)
    out = K.gemm(A, B, out_dtype=torch.float32)
    _lib.raise_if_kernel_error()
    ref = A.float() @ B.float().t()
    assert ((out - ref).norm() / ref.norm()).item() < 2e-3
    # tile widths picked at run time (176, 208, 48, ...) must respect the epilogue options and the tile's column limit
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    out2 = K.gemm(A, B, bias=bias, residual=res)
    _lib.raise_if_kernel_error()
    want = ref + bias.float() + res.float()
    assert ((out2.float() - want).norm() / want.norm()).item() < 6e-3


@pytest.mark.parametrize("M,N,K_", [(64, 4096, 4096), (64, 4096, 12288), (200, 6144, 4096), (17, 1000, 2048), (256, 24576, 1024),
                                    (300, 512, 8192)])
def test_splitk_gemm_with_epilogue(M, N, K_):
    """Skinny problems take the cluster split-K kernel; bias, residual, alpha, fp32 accumulate and ragged edges."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as K
    torch.manual_seed(2)
    A = torch.randn(M, K_, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K_, device="cuda", dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t()
    out = K.gemm(A, B, bias=bias, residual=res, alpha=0.5)
    _lib.raise_if_kernel_error()
    want = 0.5 * ref + bias.float() + res.float()
    assert ((out.float() - want).norm() / want.norm()).item() < 6e-3
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    K.gemm(A, B, out=acc, accumulate=True)
    _lib.raise_if_kernel_error()
    assert ((acc - (ref + 1)).norm() / (ref + 1).norm()).item() < 2e-3
    strided = torch.zeros(M, N + 8, device="cuda", dtype=torch.bfloat16)
    K.gemm(A, B, out=strided[:, 8:])
    _lib.raise_if_kernel_error()
    assert ((strided[:, 8:].float() - ref).norm() / ref.norm()).item() < 6e-3 and float(strided[:, :8].abs().sum()) == 0.0


@pytest.mark.parametrize("graph", [False, True])
def test_engine_matches_dense_sampler_greedy(graph):
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    from tunix_b200.generate.sampler import Sampler
    model = _model()
    cc = CacheConfig(cache_size=256, num_layers=2, num_kv_heads=2, head_dim=64)
    prompts = [[1, 5, 9, 77, 30], [1, 200, 3], [1] + list(range(10, 40)), [1, 8]]
    dense = Sampler(model, Tok(), cc)(prompt_token_ids=prompts, max_generation_steps=24, return_logprobs=True, eos_tokens=[2])
    eng = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=3, use_cuda_graph=graph, check_every=4)
    paged = eng(prompt_token_ids=prompts, max_generation_steps=24, return_logprobs=True, eos_tokens=[2])
    _lib.raise_if_kernel_error()
    agree = 0
    for a, b, la, lb in zip(dense.tokens, paged.tokens, dense.logprobs, paged.logprobs):
        n = min(len(a), len(b))
        same = int((np.asarray(a[:n]) == np.asarray(b[:n])).sum())
        agree += same
        # log-probs of the first token come from identical prefill math
        assert abs(la[0] - lb[0]) < 5e-2
    total = sum(min(len(a), len(b)) for a, b in zip(dense.tokens, paged.tokens))
    assert agree / total > 0.9, (agree, total)       # bf16 near-ties may flip an argmax late in a sequence


def test_engine_sampling_reproducible_and_wave_independent():
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    eng = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4)
    p = [[1, 4, 5, 6], [1, 9, 9], [1, 7], [1, 3, 3, 3, 3]]
    a = eng(prompt_token_ids=p, max_generation_steps=12, temperature=1.0, top_p=0.95, seed=5, return_logprobs=True, eos_tokens=[2])
    b = eng(prompt_token_ids=p, max_generation_steps=12, temperature=1.0, top_p=0.95, seed=5, return_logprobs=True, eos_tokens=[2])
    c = eng(prompt_token_ids=p, max_generation_steps=12, temperature=1.0, top_p=0.95, seed=6, return_logprobs=True, eos_tokens=[2])
    assert all(np.array_equal(x, y) for x, y in zip(a.tokens, b.tokens))
    assert any(not np.array_equal(x, y) for x, y in zip(a.tokens, c.tokens))
    assert eng.pool.free_pages == eng.pool.num_pages


@pytest.mark.parametrize("M,N,K_", [(64, 6144, 4096), (64, 4096, 12288), (8, 24576, 512), (128, 5000, 320), (1, 1024, 256),
                                    (200, 4096, 8192), (33, 151936, 128)])
def test_packed_weight_gemm(M, N, K_):
    """Decode-size GEMMs against a weight re-tiled for streaming: persistent kernel at run-time widths and the
    cluster split-K kernel (width 256), with the epilogue options and ragged edges."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as K
    torch.manual_seed(3)
    A = torch.randn(M, K_, device="cuda", dtype=torch.bfloat16)
    W = torch.randn(N, K_, device="cuda", dtype=torch.bfloat16) * 0.05
    pw = K.PackedWeight(W)
    ref = A.float() @ W.float().t()
    out = K.gemm_packed(A, pw, out_dtype=torch.float32)
    _lib.raise_if_kernel_error()
    assert ((out - ref).norm() / ref.norm()).item() < 2e-3
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    out2 = K.gemm_packed(A, pw, bias=bias, residual=res, alpha=0.5)
    _lib.raise_if_kernel_error()
    want = 0.5 * ref + bias.float() + res.float()
    assert ((out2.float() - want).norm() / want.norm()).item() < 6e-3
    W2 = torch.randn_like(W) * 0.05
    pw.refresh(W2)
    out3 = K.gemm_packed(A, pw, out_dtype=torch.float32)
    _lib.raise_if_kernel_error()
    ref3 = A.float() @ W2.float().t()
    assert ((out3 - ref3).norm() / ref3.norm()).item() < 2e-3


def test_engine_packed_weights_match_unpacked():
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    prompts = [[1, 5, 9, 77, 30], [1, 200, 3], [1] + list(range(10, 30))]
    plain = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4, pack_weights=False)
    packed = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4, pack_weights=True)
    packed.pack_min_rows = 0            # pack every projection of the tiny model
    a = plain(prompt_token_ids=prompts, max_generation_steps=16, return_logprobs=True, eos_tokens=[2])
    b = packed(prompt_token_ids=prompts, max_generation_steps=16, return_logprobs=True, eos_tokens=[2])
    _lib.raise_if_kernel_error()
    assert packed._packed is not None and all(v is not None for d in packed._packed for v in d.values())
    same = sum(int((np.asarray(x[:min(len(x), len(y))]) == np.asarray(y[:min(len(x), len(y))])).sum()) for x, y in zip(a.tokens, b.tokens))
    total = sum(min(len(x), len(y)) for x, y in zip(a.tokens, b.tokens))
    assert same / total > 0.9, (same, total)
    # weights changed in place are picked up by the next call
    with torch.no_grad():
        for p in model.parameters():
            p.mul_(0.5)
    a2 = plain(prompt_token_ids=prompts, max_generation_steps=8, return_logprobs=True, eos_tokens=[2])
    b2 = packed(prompt_token_ids=prompts, max_generation_steps=8, return_logprobs=True, eos_tokens=[2])
    for la, lb in zip(a2.logprobs, b2.logprobs):
        assert abs(la[0] - lb[0]) < 5e-2


@pytest.mark.parametrize("family", [dict(qk_norm=True), dict(qk_norm=False, qkv_bias=True), dict(family="gemma2", post_norms=True, qk_norm=False)])
def test_engine_few_sequences_round_behind_every_norm(family):
    """Decode steps of one to four sequences of wide layers: log-probs bit for bit those of a model whose norms have to run by themselves."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model(hidden_dim=8192, **family)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if p.dim() == 1:
                p.add_(0.3 * torch.randn(p.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(len(name))).to(p.dtype))
    prompts = [[1, 5, 9, 77, 30], [1, 200, 3], [1] + list(range(10, 30)), [7, 8]]
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    for n in (1, 2, 4):
        run = lambda: PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4)(  # noqa: E731
            prompt_token_ids=prompts[:n], max_generation_steps=20, return_logprobs=True, eos_tokens=[511])
        got = run()
        hooks = [m.register_forward_hook(lambda *a: None) for layer in model.layers for m in layer.modules() if type(m).__name__ == "RMSNorm"]
        want = run()
        for h in hooks:
            h.remove()
        _lib.raise_if_kernel_error()
        for t, u, x, y in zip(got.tokens, want.tokens, got.logprobs, want.logprobs):
            assert list(t) == list(u) and list(x) == list(y)


@pytest.mark.parametrize("n", [1, 3, 6])
def test_engine_short_calls_and_few_sequences_read_packed_weights(n, monkeypatch):
    """Calls of few steps and of few sequences multiply by packed weights as longer ones do, and so round alike; first tokens alone pack the
    head, and a call after that packs the layers."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    from tunix_b200.ops import kernels as K
    model = _model(hidden_dim=8192, vocab_size=1024)
    prompts = [[1, 5, 9, 77, 30], [1, 200, 3], [1] + list(range(10, 30)), [7, 8], [9, 9, 4], [100]][:n]
    seen, real = [], K.gemm_packed
    monkeypatch.setattr(K, "gemm_packed", lambda x, pw, **kw: (seen.append(pw.N), real(x, pw, **kw))[1])
    eng = PagedEngine(model, Tok(), CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64), page_size=16, max_running_requests=8)
    eng.pack_min_rows = 1024
    outs = []
    for steps, widths in ((1, {1024}), (4, {1024, 16384}), (20, {1024, 16384}), (1, {1024})):
        seen.clear()
        outs.append(eng(prompt_token_ids=prompts, max_generation_steps=steps, return_logprobs=True, eos_tokens=[1023]))
        assert set(seen) == widths
    _lib.raise_if_kernel_error()
    for out, steps in zip(outs, (1, 4, 20, 1)):
        for t, u, x, y in zip(out.tokens, outs[2].tokens, out.logprobs, outs[2].logprobs):
            assert list(t) == list(u)[:steps] and list(x) == list(y)[:steps]
    with torch.no_grad():                # weights changed in place reach the buffers of a call for first tokens too
        model.head_weight().mul_(0.5)
    fresh = PagedEngine(model, Tok(), CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64), page_size=16, max_running_requests=8)
    fresh.pack_min_rows = 1024
    for steps in (1, 4):
        got, want = (e(prompt_token_ids=prompts, max_generation_steps=steps, return_logprobs=True, eos_tokens=[1023]) for e in (eng, fresh))
        assert [list(x) for x in got.logprobs] == [list(x) for x in want.logprobs]


def test_engine_continuous_batching_matches_single_batch():
    """More requests than slots: finished sequences hand their slot to waiting ones; greedy results equal those of
    an engine that runs all requests side by side, and every page returns to the pool."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(0)
    prompts = [[1] + rng.integers(3, 500, size=int(n)).tolist() for n in (4, 9, 2, 17, 6, 30, 3, 12, 5)]
    wide = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=16, check_every=4)
    ref = wide(prompt_token_ids=prompts, max_generation_steps=24, return_logprobs=True, eos_tokens=[2])
    # end-of-sequence ids taken from what the model actually emits, so that sequences stop at different steps
    eos = sorted({2, int(ref.tokens[0][3]), int(ref.tokens[4][9]), int(ref.tokens[7][1])})
    ref = wide(prompt_token_ids=prompts, max_generation_steps=24, return_logprobs=True, eos_tokens=eos)
    lens = [len(t) for t in ref.tokens]
    assert min(lens) < 24 and max(lens) > min(lens)
    for graph in (True, False):
        narrow = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=3, check_every=4, use_cuda_graph=graph)
        out = narrow(prompt_token_ids=prompts, max_generation_steps=24, return_logprobs=True, eos_tokens=eos)
        _lib.raise_if_kernel_error()
        same = total = 0
        for a, b, la, lb in zip(ref.tokens, out.tokens, ref.logprobs, out.logprobs):
            n = min(len(a), len(b))
            same += int((np.asarray(a[:n]) == np.asarray(b[:n])).sum())
            total += max(len(a), len(b))
            assert abs(la[0] - lb[0]) < 5e-2
        assert same / total > 0.9, (same, total)
        assert narrow.pool.free_pages == narrow.pool.num_pages
    # a single generated token per request never enters the decode loop
    one = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=2)(prompt_token_ids=prompts, max_generation_steps=1,
                                                                               eos_tokens=[2])
    assert [len(t) for t in one.tokens] == [1] * len(prompts)
    assert [int(t[0]) for t in one.tokens] == [int(t[0]) for t in ref.tokens]


def test_engine_server_mode_joins_requests_and_pauses_for_weight_updates():
    from concurrent.futures import ThreadPoolExecutor
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import EngineServer, PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(1)
    prompts = [[1] + rng.integers(3, 500, size=int(n)).tolist() for n in (4, 9, 2, 17, 6, 30, 3, 12)]
    limits = [20, 5, 12, 20, 1, 8, 20, 3]
    ref = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=8)(
        prompt_token_ids=prompts, max_generation_steps=20, max_prompt_length=32, return_logprobs=True, eos_tokens=[2])
    eng = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=3, check_every=4)
    with EngineServer(eng, max_new_tokens=20, max_prompt_length=32, eos_tokens=[2]) as srv:
        with ThreadPoolExecutor(4) as ex:            # one prompt per call, from several threads at once
            res = list(ex.map(lambda a: srv.generate(a[0], a[1], timeout=120), zip(prompts, limits)))
        same = total = 0
        for (toks, lps), want, wlp, lim in zip(res, ref.tokens, ref.logprobs, limits):
            n = min(lim, len(want))
            assert len(toks) == n and len(lps) == n
            same += int((toks == np.asarray(want[:n])).sum())
            total += n
            assert abs(float(lps[0]) - wlp[0]) < 5e-2
        assert same / total > 0.9, (same, total)
        assert srv.admitted == len(prompts)
        # weight update between requests: drain, change the weights in place, resume
        assert srv.pause(timeout=60)
        with torch.no_grad():
            for p in model.parameters():
                p.mul_(0.5)
        torch.cuda.synchronize()
        srv.resume()
        toks, lps = srv.generate(prompts[3], 6, timeout=120)
        want = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=2)(
            prompt_token_ids=[prompts[3]], max_generation_steps=6, max_prompt_length=32, return_logprobs=True, eos_tokens=[2])
        assert abs(float(lps[0]) - want.logprobs[0][0]) < 5e-2 and int(toks[0]) == int(want.tokens[0][0])
    _lib.raise_if_kernel_error()
    assert eng.pool.free_pages == eng.pool.num_pages
    with pytest.raises(RuntimeError):
        srv.submit([1, 2, 3])


def test_tiered_page_pool_round_trip_on_device():
    """Pages offloaded to pinned host memory and loaded back keep their contents, on the pool's own stream, while
    the pools adopted are plain device tensors like the engine's K / V page pools."""
    from tunix_b200.experimental.generate.tiered_page_pool import PageLocation, TieredPagePool
    dev = torch.device("cuda")
    g = torch.Generator(device="cuda").manual_seed(0)
    pools = {n: torch.randn(16, 64, 2, 128, device=dev, generator=g).to(torch.bfloat16) for n in ("k", "v")}
    pool = TieredPagePool(["k", "v"], (64, 2, 128), torch.bfloat16, 16, 8, device=dev, device_pages=pools)
    ids = pool.allocate_device_pages(16)
    want = {n: {p: pools[n][pool.page_idx(p)].clone() for p in ids} for n in pools}
    out = ids[2:10]
    pool.offload(out)
    assert pool.num_free_device_pages == 8 and all(pool.page_location(p) is PageLocation.HOST for p in out)
    assert pool.host["k"].is_pinned()
    for n in pools:                                         # the freed slots get overwritten before the pages return
        pools[n][torch.tensor([i for i in range(16) if i not in pool.device_indices([p for p in ids if p not in out])],
                              device=dev)] = 0
    pool.load(out[::-1])
    torch.cuda.synchronize()
    for n in pools:
        for p in ids:
            assert torch.equal(pools[n][pool.page_idx(p)], want[n][p]), (n, p)
    assert pool.bytes_offloaded == pool.bytes_loaded == 8 * 2 * 64 * 2 * 128 * 2


def test_http_front_end_and_model_client_over_the_real_engine():
    """The serving path end to end on the device: HTTP request -> engine server -> paged engine's captured decode
    step -> answer, greedy, compared with the same prompts generated by the engine directly; token-id prompts and
    log-probs through the model client; counters on /metrics."""
    import asyncio
    import json
    import urllib.request
    from concurrent.futures import ThreadPoolExecutor
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import EngineServer, PagedEngine
    from tunix_b200.generate.openai_server import serve
    from tunix_b200.rl.agentic.http_model_client import HTTPModelClient
    model, tok = _model(), Tok()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(3)
    prompts = [[1] + rng.integers(3, 200, size=int(n)).tolist() for n in (5, 11, 3, 20, 8, 14)]
    ref = PagedEngine(model, tok, cc, page_size=16, max_running_requests=8)(
        prompt_token_ids=prompts, max_generation_steps=10, max_prompt_length=32, return_logprobs=True, eos_tokens=[2])
    eng = PagedEngine(model, tok, cc, page_size=16, max_running_requests=4, check_every=4)
    with EngineServer(eng, max_new_tokens=10, max_prompt_length=32, eos_tokens=[2]) as srv, serve(srv, tok, model_name="tiny") as http:
        def post(ids):
            body = json.dumps({"prompt": ids, "max_tokens": 10, "logprobs": True}).encode()
            with urllib.request.urlopen(urllib.request.Request(http.url + "/v1/completions", data=body), timeout=120) as r:
                return json.loads(r.read())
        with ThreadPoolExecutor(6) as ex:
            answers = list(ex.map(post, prompts))
        same = total = 0
        for ans, want, wlp in zip(answers, ref.tokens, ref.logprobs):
            got = ans["choices"][0]["logprobs"]["tokens"]
            n = min(len(got), len(want))
            assert n >= 1 and ans["choices"][0]["text"] == tok.decode(got)
            same += sum(int(a == int(b)) for a, b in zip(got[:n], want[:n]))
            total += n
            assert abs(ans["choices"][0]["logprobs"]["token_logprobs"][0] - float(wlp[0])) < 5e-2
        assert same / total > 0.9, (same, total)
        client = HTTPModelClient(http.url, route_key="ep0")
        out = asyncio.run(client(prompt_token_ids=prompts[1], max_tokens=4))
        assert out["tokens"][0] == int(ref.tokens[1][0]) and len(out["logprobs"]) == len(out["tokens"]) <= 4
        with urllib.request.urlopen(http.url + "/metrics", timeout=30) as r:
            text = r.read().decode()
        assert "tunix_b200_http_requests_total 7" in text
    _lib.raise_if_kernel_error()
    assert eng.pool.free_pages == eng.pool.num_pages


def test_engine_prefix_cache_shares_prompt_pages_between_generations():
    """Eight generations of one prompt (a GRPO group): the prompt is prefilled once, the other seven reuse its full
    pages and compute only the tail; greedy outputs equal those of an engine without the cache, and a second call
    with the same prompt (a follow-up) hits the pages the first one left behind."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=256, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(1)
    pa = [1] + rng.integers(3, 500, size=69).tolist()          # 70 tokens: 4 full pages of 16 + a tail of 6
    pb = [1] + rng.integers(3, 500, size=31).tolist()          # 32 tokens: exactly 2 pages (the last token is recomputed)
    prompts = [pa] * 8 + [pb] * 3
    plain = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=16, prefix_caching=False)
    ref = plain(prompt_token_ids=prompts, max_generation_steps=12, return_logprobs=True, eos_tokens=[2])
    eng = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=16)
    out = eng(prompt_token_ids=prompts, max_generation_steps=12, return_logprobs=True, eos_tokens=[2])
    _lib.raise_if_kernel_error()
    assert eng.pool.hit_tokens == 7 * 64 + 2 * 32 and eng.pool.prompt_tokens == 8 * 70 + 3 * 32
    same = total = 0
    for a, b, la, lb in zip(ref.tokens, out.tokens, ref.logprobs, out.logprobs):
        n = min(len(a), len(b))
        same += int((np.asarray(a[:n]) == np.asarray(b[:n])).sum())
        total += max(len(a), len(b))
        assert abs(la[0] - lb[0]) < 5e-2
    assert same / total > 0.9, (same, total)
    assert eng.pool.free_pages == eng.pool.num_pages           # cached pages are evictable: nothing is lost
    hits = eng.pool.hit_tokens
    again = eng(prompt_token_ids=[pa + [int(t) for t in out.tokens[0][:10]]], max_generation_steps=4, eos_tokens=[2])
    # the 70 prompt tokens and the 10 generated ones fill five pages, all published when the first call finished
    assert eng.pool.hit_tokens - hits == 80 and len(again.tokens[0]) >= 1


def test_engine_small_pool_queues_and_preempts_instead_of_failing():
    """A pool far smaller than slots x full length: requests wait for pages, and when the running sequences outgrow the
    pool the youngest goes back to the queue. Every request is still answered, with the greedy tokens of a roomy engine."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(2)
    prompts = [[1] + rng.integers(3, 500, size=int(n)).tolist() for n in (20, 35, 18, 40, 25, 30)]
    roomy = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=6, prefix_caching=False)
    ref = roomy(prompt_token_ids=prompts, max_generation_steps=48, eos_tokens=[-1])
    # 14 pages = 224 tokens: three prompts fit at first, none of the six reaches 40 + 48 tokens side by side
    tight = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=6, num_pages=14, check_every=4, prefix_caching=False)
    out = tight(prompt_token_ids=prompts, max_generation_steps=48, eos_tokens=[-1])
    _lib.raise_if_kernel_error()
    assert tight.preemptions > 0
    same = total = 0
    for a, b in zip(ref.tokens, out.tokens):
        assert len(b) == 48
        same += int((np.asarray(a) == np.asarray(b)).sum())
        total += 48
    assert same / total > 0.9, (same, total)
    assert tight.pool.free_pages == 14
    with pytest.raises(RuntimeError, match="cannot hold"):
        PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=2, num_pages=2)(
            prompt_token_ids=[prompts[3]], max_generation_steps=4, eos_tokens=[-1])


def test_engine_chunked_prefill_forbidden_tokens_and_final_softcap():
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    from tunix_b200.generate.sampler import Sampler
    model = _model(final_logit_softcap=20.0)
    cc = CacheConfig(cache_size=256, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(3)
    prompts = [[1] + rng.integers(3, 500, size=int(n)).tolist() for n in (100, 37, 64)]
    whole = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4, prefix_caching=False)
    a = whole(prompt_token_ids=prompts, max_generation_steps=10, return_logprobs=True, eos_tokens=[2])
    pieces = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4, prefix_caching=False, prefill_chunk=32)
    b = pieces(prompt_token_ids=prompts, max_generation_steps=10, return_logprobs=True, eos_tokens=[2])
    _lib.raise_if_kernel_error()
    for x, y, lx, ly in zip(a.tokens, b.tokens, a.logprobs, b.logprobs):
        assert int(x[0]) == int(y[0]) and abs(lx[0] - ly[0]) < 5e-2        # the prompt's last hidden state is the same
    # the soft-capped log-probability of the first token equals the dense sampler's
    dense = Sampler(model, Tok(), cc)(prompt_token_ids=prompts, max_generation_steps=2, return_logprobs=True, eos_tokens=[2])
    for ld, la in zip(dense.logprobs, a.logprobs):
        assert abs(ld[0] - la[0]) < 5e-2
    # forbidden ids never come out, and the rest of the distribution is renormalised without them
    banned = sorted({int(t) for row in a.tokens for t in row})[:6]
    c = whole(prompt_token_ids=prompts, max_generation_steps=10, return_logprobs=True, eos_tokens=[2], forbidden_tokens=banned)
    assert not ({int(t) for row in c.tokens for t in row} & set(banned))
    d = Sampler(model, Tok(), cc)(prompt_token_ids=prompts, max_generation_steps=2, return_logprobs=True, eos_tokens=[2],
                                  forbidden_tokens=banned)
    for ld, lc, td, tc_ in zip(d.logprobs, c.logprobs, d.tokens, c.tokens):
        assert int(td[0]) == int(tc_[0]) and abs(ld[0] - lc[0]) < 5e-2


def test_engine_decodes_a_mixture_of_experts_model_like_the_dense_sampler():
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    from tunix_b200.generate.sampler import Sampler
    model = _model(num_experts=8, num_experts_per_tok=2, moe_hidden_dim=128, hidden_dim=128)
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    prompts = [[1, 5, 9, 77, 30], [1, 200, 3], [1] + list(range(10, 40))]
    dense = Sampler(model, Tok(), cc)(prompt_token_ids=prompts, max_generation_steps=12, return_logprobs=True, eos_tokens=[2])
    for graph in (False, True):
        eng = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=4, use_cuda_graph=graph)
        out = eng(prompt_token_ids=prompts, max_generation_steps=12, return_logprobs=True, eos_tokens=[2])
        _lib.raise_if_kernel_error()
        same = total = 0
        for a, b, la, lb in zip(dense.tokens, out.tokens, dense.logprobs, out.logprobs):
            n = min(len(a), len(b))
            same += int((np.asarray(a[:n]) == np.asarray(b[:n])).sum())
            total += n
            assert abs(la[0] - lb[0]) < 6e-2
        assert same / total > 0.85, (graph, same, total)


def test_tensor_parallel_decode_matches_whole_model(tmp_path):
    """The paged engine on a model sliced over 2 ranks (o / down projections summed over the group, kv heads split over
    the ranks' page pools) against the engine on the whole model."""
    import json
    import os
    import subprocess
    import sys
    if torch.cuda.device_count() < 2:
        pytest.skip("needs at least 2 GPUs")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = str(tmp_path / "res.json")
    env = dict(os.environ, NCCL_NVLS_ENABLE="0")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", "29733", os.path.join(root, "tests", "engine_tp_worker.py"), out]
    res = subprocess.run(cmd, capture_output=True, text=True, timeout=600, env=env)
    assert res.returncode == 0, res.stdout[-3000:] + res.stderr[-3000:]
    for r in json.load(open(out)):
        for g in (0, 1):
            assert r[f"agree_graph{g}"] > 0.9, r           # bf16 near-ties may flip an argmax late in a sequence
            assert r[f"first_lp_graph{g}"] < 5e-2, r
            assert r[f"ranks_equal_graph{g}"], r
            assert r[f"sampled_agree_graph{g}"] > 0.6, r    # a flipped draw changes the rest of that sequence


@pytest.mark.parametrize("family,window", [("qwen3", 0), ("gemma2", 48)])
@pytest.mark.parametrize("pack", [131072, 150])             # one call of the attention kernel, and several
def test_packed_prefill_matches_padded(family, window, pack):
    """Prompts end to end give every prompt the hidden state and the pages that rows padded to the longest give it."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    kw = dict(sliding_window=window, layer_pattern=("local", "global"), attn_logit_softcap=50.0, post_norms=True) if window else {}
    model = _model(family=family, qk_norm=not window, **kw)
    cfg = model.config
    lens, rng = [5, 64, 200, 1, 129], np.random.RandomState(0)
    rows = [rng.randint(3, 500, n) for n in lens]
    slots, P, out = list(range(len(lens))), max(lens), {}
    for name in ("padded", "packed"):
        eng = PagedEngine(model, Tok(), CacheConfig(256, cfg.num_layers, cfg.num_kv_heads, cfg.head_dim), page_size=16,
                          max_running_requests=len(lens), prefix_caching=False)
        eng.PACK_TOKENS = pack
        with torch.no_grad():
            eng._fuse_all()
            eng._ensure_pool(len(lens))
            for s, r in zip(slots, rows):
                eng.pool.open(s, r.tolist(), 1)
            eng.pool.sync_table()
            for pool in eng.pool.k + eng.pool.v:
                pool.zero_()
            if name == "packed":
                h = eng._prefill_packed(rows, slots, [0, 0, 7, 0, 0])
            else:
                toks = torch.zeros(len(lens), P, dtype=torch.int64, device="cuda")
                for i, r in enumerate(rows):
                    toks[i, P - len(r):] = torch.from_numpy(r).cuda()
                n = torch.tensor(lens, device="cuda")
                seg = (torch.arange(P, device="cuda")[None] >= (P - n)[:, None]).int()
                pos = (seg.cumsum(-1) - 1).clamp(min=0).int()
                h = eng._prefill(toks, pos, seg, torch.tensor(slots, dtype=torch.int32, device="cuda"), None,
                                 torch.tensor([0, 0, 7, 0, 0], dtype=torch.int32, device="cuda"))
        _lib.raise_if_kernel_error()
        out[name] = [h] + [torch.cat([p.view(-1, p.shape[-1])[torch.tensor(
            [pg * 16 + o for pg in eng.pool.pages_of(s) for o in range(16)], device="cuda")] for s in slots])
            for p in eng.pool.k + eng.pool.v]
    for i, (a, b) in enumerate(zip(out["packed"], out["padded"])):
        # the same products in bf16; key blocks of another start round other weights
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 2e-2
        if i:                                               # nothing is written that the padded form does not write
            assert torch.equal((a != 0).any(1), (b != 0).any(1))


def test_biased_projections_decode_fused_like_one_by_one(monkeypatch):
    """q, k and v with biases as one product per layer, before and after the biases were changed from outside."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model(family="qwen2", qk_norm=False, qkv_bias=True, head_dim=64)
    with torch.no_grad():
        for layer in model.layers:
            for proj in (layer.self_attn.q_proj, layer.self_attn.k_proj, layer.self_attn.v_proj):
                proj.bias.normal_(0, 0.5)
    cc = CacheConfig(cache_size=128, num_layers=2, num_kv_heads=2, head_dim=64)
    rng = np.random.default_rng(3)
    prompts = [[1] + rng.integers(3, 500, size=n).tolist() for n in (9, 30, 17)]
    call = dict(prompt_token_ids=prompts, max_generation_steps=4, eos_tokens=[-1], return_logprobs=True)
    fused = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=3, prefix_caching=False)
    apart = PagedEngine(model, Tok(), cc, page_size=16, max_running_requests=3, prefix_caching=False)
    plain = PagedEngine._fused_weight
    monkeypatch.setattr(apart, "_fused_weight", lambda mods, bias=False: plain(mods))
    for _ in range(2):
        a, b = fused(**call), apart(**call)
        assert all(w is not None for w in fused._wqkv) and all(w is None for w in apart._wqkv)
        # first tokens come from the prefill, which both share; those behind it from decode steps that round alike up to the
        # order of bf16 sums
        for x, y in zip(a.logprobs, b.logprobs):
            assert abs(x[0] - y[0]) < 1e-6 and abs(x[1] - y[1]) < 5e-2
        with torch.no_grad():
            model.layers[0].self_attn.k_proj.bias.add_(1.0)
    _lib.raise_if_kernel_error()


def test_deleted_cache_gives_the_decode_graph_back():
    """No private memory pool of the engine outlives `delete_cache`; captures before and after it give the same tokens."""
    import gc
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine

    def pools():
        gc.collect()
        torch.cuda.empty_cache()
        return {s["segment_pool_id"] for s in torch.cuda.memory_snapshot()}

    model = _model()
    before = pools()
    eng = PagedEngine(model, Tok(), CacheConfig(128, 2, 2, model.config.head_dim), page_size=16, max_running_requests=2)
    call = dict(prompt_token_ids=[[1, 5, 9, 4], [1, 7]], max_generation_steps=12, eos_tokens=[-1])
    outs = []
    for _ in range(3):
        outs += [eng(**call).tokens, eng(**call).tokens]
        assert pools() - before
        eng.delete_cache()
        assert not pools() - before
        eng.reinitialize_cache()
    assert all(all(np.array_equal(a, b) for a, b in zip(o, outs[0])) for o in outs)


def test_decode_graph_kept_from_call_to_call():
    """A later call steps the last one's graph only where it would capture the same: its tokens are those of a new engine for other seeds,
    weights changed in place, weights that have moved, other lengths, a hooked layer and forbidden tokens, and back again."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()
    make = lambda: PagedEngine(model, Tok(), CacheConfig(128, 2, 2, 64), page_size=16, max_running_requests=3, prefix_caching=False)  # noqa: E731
    eng, captured = make(), []
    capture = eng._capture_step
    eng._capture_step = lambda st: captured.append(1) or capture(st)
    rng = np.random.default_rng(4)
    prompts = [[1] + rng.integers(3, 500, size=n).tolist() for n in (9, 30, 17, 5)]

    def check(captures, steps=24, **kw):
        kw = dict(prompt_token_ids=prompts, max_generation_steps=steps, eos_tokens=[2], return_logprobs=True, temperature=1.0, top_k=20,
                  top_p=0.9, **kw)
        captured.clear()
        a, b = eng(**kw), make()(**kw)
        assert all(np.array_equal(x, y) for x, y in zip(a.tokens, b.tokens)) and a.logprobs == b.logprobs
        assert len(captured) == captures
        return a
    first = check(1, seed=5)
    again = check(0, seed=6)
    assert any(not np.array_equal(x, y) for x, y in zip(first.tokens, again.tokens))
    check(0, seed=5)
    check(0, seed=-1)
    with torch.no_grad():
        model.layers[1].mlp.down_proj.weight.mul_(-1.0)
        model.layers[0].self_attn.q_proj.weight.mul_(0.5)
    check(0, seed=5)
    for p in model.parameters():
        p.data = p.data.clone()
    check(1, seed=5)
    check(0, seed=7)
    check(1, steps=9, seed=5)
    check(1, seed=5, forbidden_tokens=[int(first.tokens[0][0])])
    check(1, seed=5)
    handle = model.layers[0].mlp.down_proj.register_forward_hook(lambda m, i, o: o * 2.0)
    check(1, seed=5)
    handle.remove()
    check(1, seed=5)
    model.layers[0].self_attn.window = 4
    check(1, seed=5)
    _lib.raise_if_kernel_error()


def test_kept_decode_graph_reads_refreshed_packed_weights():
    """The graph of the last call steps packed buffers that a call refreshes in place: weights changed between two calls that share it, a call for
    first tokens alone in between (which refreshes the head and nothing else), and one whose buffers are new."""
    from tunix_b200 import _lib
    from tunix_b200.common.configs import CacheConfig
    from tunix_b200.generate.engine import PagedEngine
    model = _model()

    def make(packs=True):
        eng = PagedEngine(model, Tok(), CacheConfig(128, 2, 2, 64), page_size=16, max_running_requests=3, prefix_caching=False, pack_weights=packs)
        eng.pack_min_rows = 0
        return eng
    eng, captured = make(), []
    capture = eng._capture_step
    eng._capture_step = lambda st: captured.append(1) or capture(st)
    rng = np.random.default_rng(4)
    prompts = [[1] + rng.integers(3, 500, size=n).tolist() for n in (9, 30, 17)]

    def run(e, steps):
        return e(prompt_token_ids=prompts, max_generation_steps=steps, eos_tokens=[2], return_logprobs=True)

    def check(captures, steps=24):
        captured.clear()
        a, b, plain = run(eng, steps), run(make(), steps), run(make(False), steps)
        assert eng._packed_on and all(pw is not None for src in eng._packed for pw in src.values()) or steps == 1
        assert all(np.array_equal(x, y) for x, y in zip(a.tokens, b.tokens)) and a.logprobs == b.logprobs
        assert len(captured) == captures
        for t, u, x, y in zip(a.tokens, plain.tokens, a.logprobs, plain.logprobs):
            n = next((i for i, (p, q) in enumerate(zip(t, u)) if p != q), len(t))         # a near tie may part the two
            assert n > 0 and np.allclose(x[:n], y[:n], atol=5e-2)
        return a
    first = check(1)
    assert any(len(t) > 4 for t in first.tokens)
    check(0)
    for names in (("gate_proj", "up_proj"), ("q_proj", "o_proj"), ("down_proj",), ("lm_head", "embed_tokens")):
        with torch.no_grad():
            for name, p in model.named_parameters():
                if any(n in name for n in names):
                    p.mul_(-0.7)
        if names == ("down_proj",):
            check(0, steps=1)             # (a call of other numbers ends the kept graph)
        changed = check(int(names == ("down_proj",)))
        assert changed.logprobs != first.logprobs
        first = changed
    eng._packed = None
    check(1)
    _lib.raise_if_kernel_error()
