"""Grouped-GEMM mixture-of-experts path against a per-expert fp32 PyTorch reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(x, wts, idx, gw, uw, dw):
    T, D = x.shape
    out = torch.zeros(T, D, dtype=torch.float32, device=x.device)
    for t_k in range(idx.shape[1]):
        for e in range(gw.shape[0]):
            sel = idx[:, t_k] == e
            if sel.any():
                xs = x[sel].float()
                h = torch.nn.functional.silu(xs @ gw[e].float().t()) * (xs @ uw[e].float().t())
                out[sel] += wts[sel, t_k, None].float() * (h @ dw[e].float().t())
    return out


@pytest.mark.parametrize("T,E,k,D,Fd", [(300, 8, 2, 128, 192), (64, 16, 4, 256, 64), (1000, 4, 1, 192, 320)])
def test_experts_forward_backward(T, E, k, D, Fd):
    from tunix_b200 import _lib
    from tunix_b200.ops import moe
    torch.manual_seed(0)
    dev = "cuda"
    x = (torch.randn(T, D, device=dev) * 0.5).to(torch.bfloat16).requires_grad_()
    gw = (torch.randn(E, Fd, D, device=dev) * 0.08).to(torch.bfloat16).requires_grad_()
    uw = (torch.randn(E, Fd, D, device=dev) * 0.08).to(torch.bfloat16).requires_grad_()
    dw = (torch.randn(E, D, Fd, device=dev) * 0.08).to(torch.bfloat16).requires_grad_()
    logits = torch.randn(T, E, device=dev)
    if E == 16:
        logits[:, 5] = -1e9       # an expert nobody picks
    wts, idx = torch.topk(torch.softmax(logits, -1), k, -1)
    wts = wts.detach().requires_grad_()
    res = torch.randn(T, D, device=dev).to(torch.bfloat16)
    out = moe.experts(x, wts, idx, gw, uw, dw, residual=res)
    _lib.raise_if_kernel_error()
    dout = torch.randn(T, D, device=dev).to(torch.bfloat16)
    out.backward(dout)
    _lib.raise_if_kernel_error()
    xr, wr = x.detach().float().requires_grad_(), wts.detach().clone().requires_grad_()
    gr, ur, dr = (w.detach().float().requires_grad_() for w in (gw, uw, dw))
    ref = _ref(xr, wr, idx, gr, ur, dr) + res.float()
    ref.backward(dout.float())

    def rel(a, b):
        return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-6)).item()
    assert rel(out, ref) < 1e-2
    assert rel(x.grad, xr.grad) < 2e-2
    assert rel(wts.grad, wr.grad) < 2e-2
    assert rel(gw.grad, gr.grad) < 2e-2 and rel(uw.grad, ur.grad) < 2e-2 and rel(dw.grad, dr.grad) < 2e-2


def test_moe_model_trains_and_matches_fallback():
    from tunix_b200.models.config import ModelConfig
    from tunix_b200.models.transformer import create_model
    cfg = ModelConfig(family="qwen3", num_layers=2, vocab_size=512, embed_dim=128, hidden_dim=256, num_heads=4, head_dim=32,
                      num_kv_heads=2, qk_norm=True, dtype=torch.bfloat16, max_position=256, num_experts=8,
                      num_experts_per_tok=2, moe_hidden_dim=64)
    model = create_model(cfg, device=torch.device("cuda"), seed=0)
    toks = torch.randint(0, 512, (2, 64), device="cuda")
    logits = model(toks)[0] if isinstance(model(toks), tuple) else model(toks)
    layer = model.layers[0].mlp
    x = torch.randn(128, 128, device="cuda").to(torch.bfloat16)
    w, idx = torch.topk(torch.softmax(torch.randn(128, 8, device="cuda"), -1), 2, -1)
    from tunix_b200.parallel import moe_dispatch
    fast = moe_dispatch.expert_forward(layer, x, w, idx)
    slow = _ref(x, w, idx, layer.gate_proj, layer.up_proj, layer.down_proj)
    assert ((fast.float() - slow).norm() / slow.norm()).item() < 1e-2
    loss = logits.float().logsumexp(-1).mean()
    loss.backward()
    assert all(p.grad is not None and torch.isfinite(p.grad.float()).all() for p in layer.parameters())


@pytest.mark.parametrize("T,E,k,D,Fd,acc", [(2100, 4, 2, 320, 384, None), (1100, 4, 1, 256, 320, torch.bfloat16), (1500, 3, 2, 512, 256, torch.float32)])
def test_experts_on_sm_pairs(T, E, k, D, Fd, acc):
    """Enough rows an expert for the products on SM pairs: segments of an odd number of 128 rows, an expert without rows, columns that end
    inside a tile, gradients of their own and added to what is there."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as K
    from tunix_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    x = (rnd(T, D) * 0.5).to(torch.bfloat16).requires_grad_()
    ws = [(rnd(E, *s) * 0.08).to(torch.bfloat16).requires_grad_() for s in ((Fd, D), (Fd, D), (D, Fd))]
    assert K.moe_on_pairs(T * k, E, Fd, D, *ws)
    logits = rnd(T, E)
    logits[:, 1] = -1e9 if k < E - 1 else -2.0            # an expert nobody picks
    wts, idx = torch.topk(torch.softmax(logits, -1), k, -1)
    wts = wts.detach().requires_grad_()
    if acc is not None:
        for w in ws:
            w.main_grad = torch.full(w.shape, 0.5, device="cuda", dtype=acc)
    out = moe.experts(x, wts, idx, *ws)
    dout = rnd(T, D).to(torch.bfloat16)
    out.backward(dout)
    _lib.raise_if_kernel_error()
    xr, wr, *rs = (t.detach().double().requires_grad_() for t in (x, wts, *ws))
    sel = torch.nn.functional.one_hot(idx, E).double() * wr[..., None]
    ref = sum(sel[:, :, e].sum(1, keepdim=True) * ((torch.nn.functional.silu(xr @ rs[0][e].t()) * (xr @ rs[1][e].t())) @ rs[2][e].t())
              for e in range(E))
    ref.backward(dout.double())

    def rel(a, b):
        return ((a.double() - b).norm() / (b.norm() + 1e-6)).item()
    assert rel(out, ref) < 1e-2 and rel(x.grad, xr.grad) < 1e-2 and rel(wts.grad, wr.grad) < 1e-2
    for w, r in zip(ws, rs):
        assert rel(w.grad, r.grad) < 1e-2 if acc is None else rel(w.main_grad, r.grad + 0.5) < 1e-2


@pytest.mark.parametrize("T,E,k,D,Fd", [(1024, 8, 2, 256, 320), (1500, 4, 2, 1536, 256)])
def test_experts_on_sm_pairs_without_gradients(T, E, k, D, Fd, monkeypatch):
    """Nothing is kept for a backward that nobody asks for, and the result is the same bit for bit: no gradients, or none wanted of any input."""
    from tunix_b200.ops import moe
    kept, real = [], moe.K.gemm_grouped_glu

    def spy(*a, **kw):
        out = real(*a, **kw)
        kept.append(out[1] is not None and out[2] is not None)
        return out
    monkeypatch.setattr(moe.K, "gemm_grouped_glu", spy)
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *n: (0.1 * torch.randn(*n, device="cuda", generator=g)).bfloat16()  # noqa: E731
    x, ws = 5 * rnd(T, D), [rnd(E, Fd, D), rnd(E, Fd, D), rnd(E, D, Fd)]
    wts, idx = torch.topk(torch.softmax(torch.randn(T, E, device="cuda", generator=g), -1), k, -1)
    plain = moe.experts(x, wts, idx, *ws)
    grads = [w.clone().requires_grad_() for w in ws]
    want = moe.experts(x, wts, idx, *grads)
    with torch.no_grad():
        again = moe.experts(x, wts, idx, *grads)
    assert kept == [False, True, False] and torch.equal(plain, want) and torch.equal(again, want)
    want.sum().backward()
    assert all(w.grad is not None and bool(w.grad.isfinite().all()) for w in grads)



def test_row_tiles_cover_every_segment_once():
    """The planned tiles of 128 and 256 rows against the segments, empty ones and an odd number of 128 rows among them."""
    import numpy as np
    from tunix_b200.ops import kernels as K
    sizes = [0, 128, 384, 0, 256, 1280, 128] + [128 * (i % 4) for i in range(120)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    seg = torch.tensor(off, dtype=torch.int32, device="cuda")
    for kw, bm, bn in (({}, 128, 256), ({"pairs": True}, 256, 256), ({"pairs": True, "glu": True}, 256, 128)):
        tl = K.moe_tiles_rows(seg, int(off[-1]), 640, 192, 640, **kw)
        n = int(tl.count)
        d = tl.desc[:n * 32].cpu().numpy().view(np.int32).reshape(n, 8)
        want = [(off[e] + m, c, min(off[e] + m + bm, off[e + 1]), 0, 3, e * 640) for e in range(len(sizes)) for m in range(0, sizes[e], bm)
                for c in range(0, 640, bn)]
        assert n <= tl.max_tiles and [tuple(r[:6]) for r in d.tolist()] == [tuple(int(v) for v in w) for w in want]
