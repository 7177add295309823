"""Numerics of the sm_100a kernels against plain PyTorch fp32 references."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _k():
    from tunix_b200.ops import kernels
    return kernels


def _check_status():
    from tunix_b200 import _lib
    _lib.raise_if_kernel_error()


def _rel_err(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (256, 512, 128), (384, 1024, 4096), (200, 264, 72),
                                   (1000, 136, 520), (4096, 4096, 1024)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    k = _k()
    torch.manual_seed(0)
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t()
    a = A.t().contiguous() if a_mn else A
    b = B.t().contiguous() if b_mn else B
    out = k.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    _check_status()
    assert _rel_err(out, ref) < 1e-2
    out32 = k.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32)
    _check_status()
    assert _rel_err(out32, ref) < 2e-3


def test_gemm_epilogues():
    k = _k()
    torch.manual_seed(1)
    M, N, K = 512, 768, 256
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    ref = 0.5 * (A.float() @ B.float().t()) + bias.float() + res.float()
    out = k.gemm(A, B, bias=bias, residual=res, alpha=0.5)
    assert _rel_err(out, ref) < 1e-2
    acc = torch.ones(M, N, device="cuda", dtype=torch.float32)
    k.gemm(A, B, out=acc, accumulate=True)
    assert _rel_err(acc, A.float() @ B.float().t() + 1.0) < 2e-3
    # strided output: write into the right half of a wider buffer
    wide = torch.zeros(M, 2 * N, device="cuda", dtype=torch.bfloat16)
    k.gemm(A, B, out=wide[:, N:])
    assert _rel_err(wide[:, N:], A.float() @ B.float().t()) < 1e-2
    assert wide[:, :N].abs().max().item() == 0
    _check_status()


@pytest.mark.parametrize("rows,D,add_one", [(37, 256, False), (1024, 4096, False), (300, 3584, True), (4096, 128, False),
                                             (64, 8192, False), (5, 1536, True)])
def test_rmsnorm(rows, D, add_one):
    k = _k()
    torch.manual_seed(2)
    x = torch.randn(rows, D, device="cuda", dtype=torch.bfloat16)
    w = (torch.randn(D, device="cuda") * 0.1 + (0.0 if add_one else 1.0)).to(torch.bfloat16)
    dy = torch.randn(rows, D, device="cuda", dtype=torch.bfloat16)
    xf = x.float().requires_grad_(True)
    wf = w.float().requires_grad_(True)
    rstd_ref = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-6)
    yref = xf * rstd_ref * (wf + (1.0 if add_one else 0.0))
    yref.backward(dy.float())
    y, rstd = k.rmsnorm_fwd(x, w, 1e-6, add_one)
    assert _rel_err(y, yref) < 1e-2
    dx, dw = k.rmsnorm_bwd(dy, x, w, rstd, add_one)
    assert _rel_err(dx, xf.grad) < 1e-2
    assert _rel_err(dw, wf.grad) < 1e-2


def test_rope_roundtrip_and_reference():
    k = _k()
    torch.manual_seed(3)
    tokens, heads, H = 513, 6, 128
    x = torch.randn(tokens, heads, H, device="cuda", dtype=torch.bfloat16)
    pos = torch.randint(0, 2048, (tokens,), device="cuda", dtype=torch.int32)
    inv = 1.0 / (10000.0 ** (torch.arange(0, H // 2, device="cuda", dtype=torch.float64) * 2 / H))
    ang = torch.arange(2048, device="cuda", dtype=torch.float64)[:, None] * inv[None]
    cos, sin = ang.cos().float().contiguous(), ang.sin().float().contiguous()
    xf = x.float()
    c = cos[pos.long()][:, None, :]
    s = sin[pos.long()][:, None, :]
    x1, x2 = xf[..., : H // 2], xf[..., H // 2:]
    ref = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1)
    y = k.rope_(x.clone(), pos, cos, sin)
    assert _rel_err(y, ref) < 1e-2
    back = k.rope_(y.clone(), pos, cos, sin, backward=True)
    assert _rel_err(back, x) < 2e-2


@pytest.mark.parametrize("kind", [0, 1])
def test_glu(kind):
    k = _k()
    torch.manual_seed(4)
    rows, F = 333, 1024
    g = torch.randn(rows, F, device="cuda", dtype=torch.bfloat16)
    u = torch.randn(rows, F, device="cuda", dtype=torch.bfloat16)
    dh = torch.randn(rows, F, device="cuda", dtype=torch.bfloat16)
    gf, uf = g.float().requires_grad_(True), u.float().requires_grad_(True)
    act = torch.nn.functional.silu(gf) if kind == 0 else torch.nn.functional.gelu(gf, approximate="tanh")
    href = act * uf
    href.backward(dh.float())
    h = k.glu_fwd(g, u, kind)
    assert _rel_err(h, href) < 1e-2
    dg, du = k.glu_bwd(dh, g, u, kind)
    assert _rel_err(dg, gf.grad) < 1.5e-2
    assert _rel_err(du, uf.grad) < 1.5e-2


def test_embedding():
    k = _k()
    torch.manual_seed(5)
    V, D, T = 1000, 256, 777
    table = torch.randn(V, D, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    out = k.embedding_fwd(ids, table, scale=2.0)
    assert _rel_err(out, table[ids.long()].float() * 2.0) < 1e-2
    dout = torch.randn(T, D, device="cuda", dtype=torch.bfloat16)
    dtable = torch.zeros_like(table)
    k.embedding_bwd(ids, dout, dtable, scale=2.0)
    ref = torch.zeros(V, D, device="cuda").index_add_(0, ids.long(), dout.float() * 2.0)
    assert _rel_err(dtable, ref) < 2e-2


@pytest.mark.parametrize("softcap,temp", [(0.0, 1.0), (30.0, 0.7)])
def test_logsoftmax_and_dlogits(softcap, temp):
    k = _k()
    torch.manual_seed(6)
    rows, V = 65, 5003
    raw = (torch.randn(rows, V, device="cuda") * 4).requires_grad_(True)
    tg = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
    tg[3] = -1
    z = raw
    if softcap > 0:
        z = softcap * torch.tanh(z / softcap)
    z = z / temp
    lsm = torch.log_softmax(z, -1)
    logp_ref = lsm.gather(1, tg.clamp(min=0).long()[:, None])[:, 0] * (tg >= 0)
    ent_ref = -(lsm.exp() * lsm).sum(-1)
    gl = torch.randn(rows, device="cuda")
    ge = torch.randn(rows, device="cuda")
    ((logp_ref * gl).sum() + (ent_ref * ge).sum()).backward()
    logp, lse, ent = k.logsoftmax_gather(raw.detach(), tg, softcap=softcap, temperature=temp, want_entropy=True)
    assert torch.allclose(logp, logp_ref.detach(), atol=2e-3, rtol=1e-3)
    assert torch.allclose(ent, ent_ref.detach(), atol=2e-3, rtol=1e-3)
    d = k.dlogits(raw.detach(), tg, lse, ent, gl, ge, softcap=softcap, temperature=temp)
    assert _rel_err(d, raw.grad) < 1.5e-2


def test_adamw_matches_torch():
    k = _k()
    torch.manual_seed(7)
    n = 100003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    ref_p = p.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    p32, m, v = p.clone(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    p16 = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    for step in range(1, 4):
        gs = g * step
        ref_p.grad = gs.clone()
        opt.step()
        k.adamw(p32, m, v, gs.to(torch.bfloat16).float(), p16, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8,
                weight_decay=0.1, step=step)
    # torch applies decay as p *= (1 - lr*wd) before the Adam step; optax adds wd*p to the update.
    # The two differ at O(lr^2 * wd), far below this tolerance.
    assert _rel_err(p32, ref_p.detach()) < 2e-3
    assert _rel_err(p16, p32) < 5e-3
    ss = torch.zeros(1, device="cuda")
    k.sumsq(g, ss)
    assert abs(ss.item() - g.pow(2).sum().item()) / g.pow(2).sum().item() < 1e-4


@pytest.mark.parametrize("M,N,K_,a_mn,b_mn", [(2048, 2048, 512, False, False), (4096, 1536, 1024, False, True),
                                              (2304, 2048, 768, True, True), (2000, 2100, 320, False, False),
                                              (8192, 4096, 4096, False, False)])
def test_gemm_cta_pair_tiles(M, N, K_, a_mn, b_mn):
    """Problems with a wave of 256 x 256 tiles run on CTA pairs (tcgen05.mma.cta_group::2): layouts, ragged edges,
    bias / residual / alpha, fp32 accumulation into an existing buffer."""
    k = _k()
    torch.manual_seed(5)
    A = torch.randn((K_, M) if a_mn else (M, K_), device="cuda", dtype=torch.bfloat16)
    B = (torch.randn((K_, N) if b_mn else (N, K_), device="cuda") * 0.05).to(torch.bfloat16)
    ref = (A.float().t() if a_mn else A.float()) @ (B.float() if b_mn else B.float().t())
    out = k.gemm(A, B, a_mn=a_mn, b_mn=b_mn)
    _check_status()
    assert _rel_err(out, ref) < 5e-3
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    out2 = k.gemm(A, B, a_mn=a_mn, b_mn=b_mn, bias=bias, residual=res, alpha=0.25)
    _check_status()
    assert _rel_err(out2, 0.25 * ref + bias.float() + res.float()) < 5e-3
    acc = torch.full((M, N), 2.0, device="cuda", dtype=torch.float32)
    k.gemm(A, B, a_mn=a_mn, b_mn=b_mn, out=acc, accumulate=True)
    _check_status()
    assert _rel_err(acc, ref + 2.0) < 2e-3


@pytest.mark.parametrize("shape,block", [((256, 512), 64), ((100, 72), 32), ((3, 50), 64)])
def test_nf4_dequant_kernel_matches_reference(shape, block):
    from tunix_b200.lora import NF4Weight
    torch.manual_seed(3)
    w = torch.randn(*shape, device="cuda", dtype=torch.bfloat16)
    q = NF4Weight(w, block)
    got = q.dequantize()
    _check_status()
    cpu = NF4Weight(w.cpu(), block).dequantize()
    assert got.shape == w.shape and torch.allclose(got.float().cpu(), cpu.float(), atol=1e-2, rtol=1e-2)
    assert (got.float() - w.float()).abs().mean() < 0.15


@pytest.mark.parametrize("rows,V,D,softcap,temp", [(512, 5000, 256, 0.0, 1.0), (1024, 33000, 512, 30.0, 0.7), (300, 128256, 128, 0.0, 1.0)])
def test_fused_lm_head_logprobs_match_reference(rows, V, D, softcap, temp):
    """The log-softmax epilogue of the two-SM GEMM (no logits in memory) against fp32 PyTorch, forward and backward."""
    from tunix_b200.ops import functional as F
    torch.manual_seed(9)
    h = (torch.randn(rows, D, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(V, D, device="cuda") * 0.1).to(torch.bfloat16).requires_grad_()
    tg = torch.randint(0, V, (rows,), device="cuda")
    tg[::17] = -1                                                  # ignored positions
    logp, ent = F.lm_head_logprobs(h, w, tg, softcap=softcap, temperature=temp, want_entropy=True)
    _check_status()
    z = h.detach().float() @ w.detach().float().t()
    if softcap:
        z = softcap * torch.tanh(z / softcap)
    z = z / temp
    ref_lp = torch.log_softmax(z, -1).gather(-1, tg.clamp(min=0)[:, None]).squeeze(-1)
    ref_lp = torch.where(tg >= 0, ref_lp, torch.zeros_like(ref_lp))
    p = torch.softmax(z, -1)
    ref_ent = -(p * torch.log_softmax(z, -1)).sum(-1)
    assert torch.allclose(logp, ref_lp, atol=3e-2, rtol=2e-2), float((logp - ref_lp).abs().max())
    assert torch.allclose(ent, ref_ent, atol=3e-2, rtol=2e-2)
    g = torch.randn(rows, device="cuda")
    g2 = torch.randn(rows, device="cuda") * 0.3
    ((logp * g).sum() + (ent * g2).sum()).backward()          # both gradient terms of the fused epilogue
    _check_status()
    hr = h.detach().float().requires_grad_()
    wr = w.detach().float().requires_grad_()
    zr = hr @ wr.t()
    if softcap:
        zr = softcap * torch.tanh(zr / softcap)
    lsm = torch.log_softmax(zr / temp, -1)
    lp2 = lsm.gather(-1, tg.clamp(min=0)[:, None]).squeeze(-1)
    ent2 = -(lsm.exp() * lsm).sum(-1)
    ((torch.where(tg >= 0, lp2, torch.zeros_like(lp2)) * g).sum() + (ent2 * g2).sum()).backward()
    assert _rel_err(h.grad, hr.grad) < 3e-2 and _rel_err(w.grad, wr.grad) < 3e-2


@pytest.mark.parametrize("M,N,K,r", [(2048, 4096, 1024, 16), (2304, 2560, 520, 8), (4096, 2048, 2048, 64), (2048, 4096, 512, 72),
                                     (128, 256, 64, 16)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_with_second_segment(M, N, K, r, b_mn):
    """A @ B^T + A2 @ B2^T in one launch (adapter rank r as extra k-blocks; the last shape falls back to two GEMMs)."""
    k = _k()
    torch.manual_seed(11)
    A = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    B = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    A2 = torch.randn(M, r, device="cuda", dtype=torch.bfloat16)
    B2 = torch.randn(N, r, device="cuda", dtype=torch.bfloat16) * 4
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    res = torch.randn(M, N, device="cuda", dtype=torch.bfloat16)
    ref = A.float() @ B.float().t() + A2.float() @ B2.float().t()
    b, b2 = (B.t().contiguous(), B2.t().contiguous()) if b_mn else (B, B2)
    out = k.gemm_ext(A, b, A2, b2, b_mn=b_mn)
    _check_status()
    assert _rel_err(out, ref) < 1e-2
    # the low-rank part alone must be right too (it is small next to the main product)
    low = out.float() - (A.float() @ B.float().t())
    assert _rel_err(low, A2.float() @ B2.float().t()) < 0.2
    out = k.gemm_ext(A, b, A2, b2, b_mn=b_mn, bias=bias, residual=res)
    _check_status()
    full = ref + bias.float() + res.float()
    assert _rel_err(out, full) < 1e-2
    assert torch.allclose(out.float(), full, atol=0.02 * full.abs().max().item(), rtol=2e-2)


@pytest.mark.parametrize("with_bias,with_res", [(False, False), (True, True)])
def test_lora_linear_matches_fp32(with_bias, with_res):
    """Fused LoRA projection (forward, input gradient, adapter gradients) against fp32 PyTorch."""
    from tunix_b200.ops import functional as F
    torch.manual_seed(5)
    M, D, O, r, s = 2048, 1024, 3072, 16, 2.0
    x = (torch.randn(4, M // 4, D, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(O, D, device="cuda") * 0.05).to(torch.bfloat16)
    a = (torch.randn(r, D, device="cuda") * 0.05).to(torch.bfloat16).requires_grad_()
    b = (torch.randn(O, r, device="cuda") * 0.2).to(torch.bfloat16).requires_grad_()
    bias = (torch.randn(O, device="cuda") * 0.1).to(torch.bfloat16).requires_grad_() if with_bias else None
    res = (torch.randn(4, M // 4, O, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_() if with_res else None
    y = F.lora_linear(x, w, bias, a, b, s, res)
    g = torch.randn_like(y)
    y.backward(g)
    _check_status()
    xf, af, bf = (t.detach().float().requires_grad_() for t in (x, a, b))
    yf = xf @ w.float().t() + s * (xf @ af.t()) @ bf.t()
    if with_bias:
        yf = yf + bias.detach().float()
    if with_res:
        yf = yf + res.detach().float()
    yf.backward(g.float())
    assert _rel_err(y, yf) < 1e-2
    assert _rel_err(x.grad, xf.grad) < 1e-2
    assert _rel_err(a.grad, af.grad) < 2e-2
    assert _rel_err(b.grad, bf.grad) < 2e-2
    if with_res:
        assert torch.equal(res.grad, g)
    if with_bias:
        assert _rel_err(bias.grad, g.float().sum((0, 1))) < 1e-2


def test_qlora_linear_keeps_no_expanded_weight():
    """A LoRA projection over an NF4 base: same values and gradients as the projection over the expanded weight, and
    between forward and backward nothing of the size of the expanded weight stays allocated."""
    from tunix_b200 import lora
    from tunix_b200.models.transformer import Linear
    torch.manual_seed(2)
    D, O = 2048, 4096
    lin = Linear(D, O, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        lin.weight.normal_(0, 0.05)

    class _M(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.proj = lin

    m = _M()
    lora.apply_lora_to_model(m, lora.LoraProvider(rank=16, alpha=32.0, weight_qtype="nf4", module_path=".*proj"))
    with torch.no_grad():
        lin.lora_b.normal_(0, 0.05)
    w_full = lin.quant.dequantize().float()
    x = (torch.randn(2, 1024, D, device="cuda") * 0.5).to(torch.bfloat16).requires_grad_()
    y = lin(x)                                   # first call allocates the shared scratch
    del y
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    y = lin(x)
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated() - before
    weight_bytes = D * O * 2
    # y itself (2 * 1024 * O * 2 bytes) plus the rank-16 intermediate, but no [O, D] bf16 tensor
    assert held < 2 * 1024 * O * 2 + weight_bytes // 4, (held, weight_bytes)
    g = torch.randn_like(y)
    y.backward(g)
    _check_status()
    xf = x.detach().float().requires_grad_()
    af, bf = lin.lora_a.detach().float().requires_grad_(), lin.lora_b.detach().float().requires_grad_()
    yf = xf @ w_full.t() + lin.lora_scale * (xf @ af.t()) @ bf.t()
    yf.backward(g.float())
    assert _rel_err(y, yf) < 1e-2 and _rel_err(x.grad, xf.grad) < 1e-2
    assert _rel_err(lin.lora_a.grad, af.grad) < 2e-2 and _rel_err(lin.lora_b.grad, bf.grad) < 2e-2


@pytest.mark.parametrize("M,F,D,kind", [(64, 12288, 1024, "silu"), (16, 1408, 512, "gelu"), (200, 2816, 256, "silu"), (256, 4096, 512, "silu")])
def test_packed_gemm_with_gated_epilogue(M, F, D, kind):
    """Fused gate / up projection on a pre-tiled, row-interleaved weight with act(gate) * up in the epilogue."""
    k = _k()
    torch.manual_seed(4)
    x = (torch.randn(M, D, device="cuda") * 0.5).to(torch.bfloat16)
    w = (torch.randn(2 * F, D, device="cuda") * 0.05).to(torch.bfloat16)
    pw = k.PackedWeight(w, glu=True)
    out = k.gemm_packed(x, pw, glu=k.GLU_SILU if kind == "silu" else k.GLU_GELU)
    _check_status()
    z = x.float() @ w.float().t()
    g, u = z[:, :F], z[:, F:]
    act = torch.nn.functional.silu(g) if kind == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    ref = act * u
    assert out.shape == (M, F)
    assert _rel_err(out, ref) < 1e-2
    assert torch.allclose(out.float(), ref, atol=0.02 * ref.abs().max().item() + 1e-3, rtol=3e-2)


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K_", [(1, 8), (5, 264), (1030, 1536), (2050, 520), (72, 4104)])
def test_gemm_few_rows(M, N, K_):
    """Products of up to four rows: remainders of the row groups and of the steps over K, every epilogue."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(8)
    draw = lambda r, c: torch.randn(r, c + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :c]  # noqa: E731
    a, b, res = draw(M, K_), draw(N, K_), draw(M, N)
    bias = torch.randn(N, device="cuda", generator=g).to(torch.bfloat16)
    want = a.double() @ b.double().t()
    # sums of K_ products in 32 bits: 2^-24 a term, far below the norm of the sum
    assert _rel_err(k.gemm(a, b, out_dtype=torch.float32), want) < 1e-5
    full = 0.5 * want + bias.double() + res.double()
    assert _rel_err(k.gemm(a, b, bias=bias, residual=res, alpha=0.5), full) < 4e-3
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 4e-3)):
        out = torch.ones(M, N + 3, device="cuda", dtype=dtype)[:, :N]
        assert _rel_err(k.gemm(a, b, out=out, accumulate=True), want + 1) < tol
    _check_status()


@pytest.mark.parametrize("rows", [1, 3, 1301])
@pytest.mark.parametrize("D", [8, 64, 72, 128, 136, 256, 264, 4096, 4104, 8192, 8200, 16384, 16392])
def test_rmsnorm_widths(rows, D):
    """Widths on both sides of every kernel's limit, rows that lie apart, dx added to what is there."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(7)
    draw = lambda: torch.randn(rows, D + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :D]  # noqa: E731
    x, dy, base = draw(), draw(), draw()
    w = torch.randn(D, device="cuda", generator=g).to(torch.bfloat16)
    y, rstd = k.rmsnorm_fwd(x, w, 1e-6, True)
    into = base.clone()
    dx, dw = k.rmsnorm_bwd(dy, x, w, rstd, True, dx_accumulate_into=into)
    xd, dd, wd = x.double(), dy.double(), w.double() + 1
    rs = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6)
    gx = dd * wd
    want = base.double() + rs * (gx - xd * rs * (gx * xd * rs).mean(-1, keepdim=True))
    # one rounding to bf16: 2^-9 of a value
    assert _rel_err(y, xd * rs * wd) < 4e-3 and _rel_err(dx, want) < 4e-3
    assert _rel_err(dw, (dd * xd * rs).sum(0)) < 1e-5          # 32-bit sums over the rows
    _check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("tokens,D", [(1, 8), (37, 264), (300, 10)])
def test_embedding_bwd_tables(tokens, D, dtype):
    """Both tables, rows of whole 16-byte pieces and by pairs; ids outside the table are left out."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(10)
    ids = torch.randint(-1, 41, (tokens,), device="cuda", generator=g, dtype=torch.int32)
    dout = torch.randn(tokens, D, device="cuda", generator=g).to(torch.bfloat16)
    table = torch.zeros(40, D, device="cuda", dtype=dtype)
    k.embedding_bwd(ids, dout, table, scale=0.5)
    ok = (ids >= 0) & (ids < 40)
    want = torch.zeros(40, D, device="cuda").index_add_(0, ids[ok].long(), 0.5 * dout.float()[ok])
    # up to some 20 terms a row: a bf16 rounding each where the table is bf16
    assert _rel_err(table, want) < (2e-2 if dtype == torch.bfloat16 else 1e-6)
    _check_status()


@pytest.mark.parametrize("tokens,heads,H,gap", [(1, 1, 16, 0), (33, 3, 64, 64), (70, 5, 128, 0), (129, 4, 256, 8), (20, 6, 40, 0), (9, 4, 64, 4)])
def test_rope_widths(tokens, heads, H, gap):
    """Head groups that are not full, rows that lie apart, and sizes without whole 16-byte pieces (H = 40, a gap of 4)."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(tokens, heads * H + gap, device="cuda", generator=g).to(torch.bfloat16)
    v = x[:, :heads * H].unflatten(1, (heads, H))
    pos = torch.randint(0, 50, (tokens,), device="cuda", generator=g, dtype=torch.int32)
    ang = torch.randn(50, H // 2, device="cuda", generator=g)
    c, s = ang.cos()[pos.long()][:, None], ang.sin()[pos.long()][:, None]
    a, b = v.float()[..., :H // 2], v.float()[..., H // 2:]
    want, rest = torch.cat([a * c - b * s, b * c + a * s], -1), x[:, heads * H:].clone()
    k.rope_(v, pos, ang.cos(), ang.sin())
    assert _rel_err(v, want) < 4e-3 and torch.equal(x[:, heads * H:], rest)
    _check_status()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (4099, 1), (5_000_003, 0), (5_000_003, 3)])
def test_sumsq_tails(n, off, dtype):
    """Lengths that are not whole vectors, and a start that is not aligned to one."""
    k = _k()
    x = torch.randn(n + off, device="cuda", generator=torch.Generator(device="cuda").manual_seed(11)).to(dtype)[off:]
    out = torch.full((1,), 2.0, device="cuda")
    k.sumsq(x, out)
    want = 2.0 + x.double().square().sum().item()
    assert abs(out.item() - want) < 1e-5 * want                # 32-bit partial sums


@pytest.mark.parametrize("D", [8, 128, 264, 4096, 16392])
def test_rmsnorm_weight_gradient_alone(D):
    """Without dx the entry point asks for no weight and no 16-byte alignment of x and dy."""
    from tunix_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(12)
    rows, ld = 37, D + 6
    x, dy = (torch.randn(rows * ld + 2, device="cuda", generator=g).to(torch.bfloat16)[2:].view(rows, ld)[:, :D] for _ in range(2))
    assert x.data_ptr() % 16 == 4
    rstd = torch.rand(rows, device="cuda", generator=g) + 0.5
    dw = torch.zeros(D, device="cuda")
    rc = _lib.cuda().tb_rmsnorm_bwd(dy.data_ptr(), ld, x.data_ptr(), ld, 0, rstd.data_ptr(), 0, 0, dw.data_ptr(), rows, D, 0.0, 0,
                                    _lib.stream_ptr())
    assert rc == 0
    assert _rel_err(dw, (dy.double() * x.double() * rstd.double()[:, None]).sum(0)) < 1e-5      # 32-bit sums over the rows


@pytest.mark.parametrize("gap,off", [(0, 0), (4, 0), (3, 0), (4, 1)])
@pytest.mark.parametrize("M,N", [(2048, 1536), (1999, 1560), (2311, 1533)])
def test_scaled_sums_into_fp32(M, N, gap, off):
    """Large products added to fp32 with a factor: whole 32-column blocks as reductions, remainders of rows and columns, and results
    without 16-byte rows (a gap of 3, an offset of 1), as the epilogue before."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(14)
    K_ = 256
    a = torch.randn(K_, (M + 7) // 8 * 8, device="cuda", generator=g).to(torch.bfloat16)[:, :M]
    b = torch.randn(K_, (N + 7) // 8 * 8, device="cuda", generator=g).to(torch.bfloat16)[:, :N]
    buf = torch.randn(M * (N + gap) + off, device="cuda", generator=g)
    before, out = buf.clone(), buf[off:].view(M, N + gap)[:, :N]
    want = out.double() - 0.375 * (a.double().t() @ b.double())
    k.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, alpha=-0.375)
    _check_status()
    # sums of K_ products in 32 bits
    assert _rel_err(out, want) < 1e-6
    rest = torch.ones(M, N + gap, dtype=torch.bool, device="cuda")
    rest[:, :N] = False
    assert torch.equal(buf[off:].view(M, N + gap)[rest], before[off:].view(M, N + gap)[rest])
    assert torch.equal(buf[:off], before[:off])


@pytest.mark.parametrize("M,N,K_", [(1, 32768, 4096), (1, 32776, 4096), (2, 16384, 4096), (2, 16392, 4096), (3, 4096, 4096), (4, 4104, 4096),
                                    (3, 12288, 1024), (4, 12296, 1024)])
def test_gemm_few_rows_at_the_limits(M, N, K_):
    """The largest weights of the few-row kernel, and the next size, which the tensor cores take."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(15)
    a, b = (torch.randn(r, K_, device="cuda", generator=g).to(torch.bfloat16) for r in (M, N))
    want = torch.cat([a.double() @ p.double().t() for p in b.split(4096)], 1)
    assert _rel_err(k.gemm(a, b, out_dtype=torch.float32), want) < 1e-5      # sums of K_ products in 32 bits
    _check_status()


@pytest.mark.parametrize("rows,D", [(4095, 64), (4099, 8), (4099, 128), (4099, 136), (8191, 72), (8195, 8), (8195, 64), (8195, 72), (8195, 128),
                                    (8195, 136), (16383, 264), (16389, 512), (513, 2304), (512, 2304), (3000, 4104), (9, 16384), (2049, 16384),
                                    (8195, 3584), (8191, 3584)])
def test_rmsnorm_rows_and_frozen_weights(rows, D):
    """Numbers of rows on both sides of every kernel's limit, with and without a gradient of the weight."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(16)
    draw = lambda: torch.randn(rows, D + 8, device="cuda", generator=g).to(torch.bfloat16)[:, :D]  # noqa: E731
    x, dy, base = draw(), draw(), draw()
    w = torch.randn(D, device="cuda", generator=g).to(torch.bfloat16)
    y, rstd = k.rmsnorm_fwd(x, w, 1e-6)
    xd, dd, wd = x.double(), dy.double(), w.double()
    rs = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6)
    gx = dd * wd
    want = rs * (gx - xd * rs * (gx * xd * rs).mean(-1, keepdim=True))
    dx, dw = k.rmsnorm_bwd(dy, x, w, rstd)
    frozen, none = k.rmsnorm_bwd(dy, x, w, rstd, want_dw=False)
    into = base.clone()
    k.rmsnorm_bwd(dy, x, w, rstd, want_dw=False, dx_accumulate_into=into)
    assert none is None
    # one rounding to bf16: 2^-9 of a value; 32-bit sums over the rows
    assert _rel_err(y, xd * rs * wd) < 4e-3 and _rel_err(dx, want) < 4e-3 and _rel_err(frozen, want) < 4e-3
    assert _rel_err(into, base.double() + want) < 4e-3 and _rel_err(dw, (dd * xd * rs).sum(0)) < 1e-5
    _check_status()


@pytest.mark.parametrize("tokens,heads,H,gap", [(5461, 3, 48, 16), (5462, 3, 48, 16), (2050, 5, 64, 8), (1030, 32, 64, 0), (300, 30, 128, 0),
                                                (129, 41, 256, 8), (9000, 4, 64, 4)])
def test_rope_of_many_heads(tokens, heads, H, gap):
    """Sizes of the vector kernel, from the smallest on: head groups that are not full, rows that lie apart or without 16-byte pieces."""
    test_rope_widths(tokens, heads, H, gap)


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("tokens,N,KH,H,gap", [(1, 1, 1, 64, 0), (37, 14, 2, 64, 0), (130, 4, 5, 128, 24), (1000, 32, 8, 128, 0), (67, 16, 8, 256, 8)])
def test_qk_rope(tokens, N, KH, H, gap, norm):
    """Head groups that are not full, rows that lie apart, one token, more units than one round of blocks takes; forward and backward."""
    k = _k()
    g = torch.Generator(device="cuda").manual_seed(13)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)  # noqa: E731
    xs = [rnd(tokens, n * H + gap)[:, :n * H] for n in (N, KH)]
    ws = [1 + 0.2 * rnd(H), 1 + 0.2 * rnd(H)] if norm else [None, None]
    ds = [rnd(tokens, n * H) for n in (N, KH)]
    pos = torch.randint(0, 50, (tokens,), device="cuda", generator=g, dtype=torch.int32)
    ang = torch.randn(50, H // 2, device="cuda", generator=g)
    cos, sin = ang.cos(), ang.sin()
    want, leaves = [], []
    for x, w in zip(xs, ws):
        x = x.double().unflatten(1, (-1, H)).requires_grad_()
        w = None if w is None else w.double().requires_grad_()
        leaves.append((x, w))
        y = x if w is None else x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * (w + 1)
        c, s = cos.double()[pos.long()][:, None], sin.double()[pos.long()][:, None]
        a, b = y[..., :H // 2], y[..., H // 2:]
        want.append(torch.cat([a * c - b * s, b * c + a * s], -1).flatten(1))
    yq, yk, rq, rk = k.qk_rope(*xs, H, pos, cos, sin, wq=ws[0], wk=ws[1], eps=1e-6, add_one=True, want_rstd=norm)
    # a rounding to bf16 is at most 2^-8 of a value, about 1.7e-3 in the norm of many; behind a norm there are two (2.4e-3)
    tol = 3e-3 if norm else 2e-3
    assert _rel_err(yq, want[0]) < tol and _rel_err(yk, want[1]) < tol
    torch.autograd.backward(want, [d.double() for d in ds])
    if norm:
        dxq, dxk, dwq, dwk = k.qk_rope_bwd(*ds, *xs, H, pos, cos, sin, *ws, rq, rk, True)
        assert _rel_err(dwq, leaves[0][1].grad) < 1e-4 and _rel_err(dwk, leaves[1][1].grad) < 1e-4      # 32-bit sums
        assert k.qk_rope_bwd(*ds, *xs, H, pos, cos, sin, *ws, rq, rk, True, want_dw=False)[2] is None
    else:
        dxq, dxk, _, _ = k.qk_rope(*ds, H, pos, cos, sin, backward=True)
    assert _rel_err(dxq, leaves[0][0].grad.flatten(1)) < 2e-3 and _rel_err(dxk, leaves[1][0].grad.flatten(1)) < 2e-3
    again = [x.clone() for x in xs]
    k.qk_rope(*again, H, pos, cos, sin, wq=ws[0], wk=ws[1], eps=1e-6, add_one=True, out=again)          # over its inputs
    assert torch.equal(again[0], yq) and torch.equal(again[1], yk)
    assert k.qk_rope(xs[0], rnd(tokens, KH * H + 4)[:, :KH * H], H, pos, cos, sin) is None              # rows without 16-byte pieces
    _check_status()


@pytest.mark.parametrize("tokens,N,KH,H", [(3, 4, 2, 64), (1037, 16, 16, 64), (130, 8, 4, 128), (2100, 32, 4, 128), (700, 12, 8, 256)])
def test_qk_rope_norms_like_the_norms_own_kernel(tokens, N, KH, H):
    """1 / rms of every head bit for bit, in each of the norm's kernels for these widths; where the rotation runs by vectors (16384 units of
    4 heads and 16 columns) the rotated rows too."""
    k = _k()
    pos = torch.arange(tokens, device="cuda", dtype=torch.int32) % 50
    ang = _normal(50, H // 2, seed=3)
    xs = [3 * _normal(tokens, n * H, seed=n) for n in (N, KH)]
    xs, ws = [x.bfloat16() for x in xs], [(1 + 0.2 * _normal(H, seed=7 + i)).bfloat16() for i in (0, 1)]
    got = k.qk_rope(*xs, H, pos, ang.cos(), ang.sin(), wq=ws[0], wk=ws[1], eps=1e-6, want_rstd=True)
    for n, x, w, y, rstd in zip((N, KH), xs, ws, got[:2], got[2:]):
        rows, want = k.rmsnorm_fwd(x.view(-1, H), w, 1e-6)
        assert torch.equal(rstd, want)
        if tokens * (H // 16) * ((n + 3) // 4) >= 16384:
            assert torch.equal(y, k.rope_(rows.view(tokens, n, H), pos, ang.cos(), ang.sin()).view(tokens, -1))
    _check_status()


@pytest.mark.parametrize("tokens,N,KH,H", [(5, 3, 1, 64), (2000, 14, 2, 64), (4100, 14, 2, 64), (1023, 8, 4, 128), (513, 32, 8, 128),
                                           (255, 17, 4, 256)])
@pytest.mark.parametrize("backward", [False, True])
def test_qk_rope_rotates_like_the_rotations_own_kernels(tokens, N, KH, H, backward):
    """Bit for bit, on both sides of the 16384 units of 4 heads and 16 columns that divide the rotation's kernels, for either tensor."""
    k = _k()
    pos = torch.arange(tokens, device="cuda", dtype=torch.int32) % 500
    ang = _normal(500, H // 2, seed=3)
    xs = [_normal(tokens, n * H, seed=n).bfloat16() for n in (N, KH)]
    got = k.qk_rope(*xs, H, pos, ang.cos(), ang.sin(), backward=backward)
    for n, x, y in zip((N, KH), xs, got):
        assert torch.equal(y, k.rope_(x.view(tokens, n, H).clone(), pos, ang.cos(), ang.sin(), backward=backward).view(tokens, -1))
    _check_status()


@pytest.mark.parametrize("qk_norm", [False, True])
def test_model_joint_rotation_matches_separate(qk_norm):
    """The attention layer with the joint kernel and, made to by a hook or by a refusing kernel, with norm and rotation one by one."""
    from tunix_b200.models.config import ModelConfig
    from tunix_b200.models.transformer import Attention
    from tunix_b200.ops import functional as F
    cfg = ModelConfig(family="qwen3", num_layers=1, vocab_size=64, embed_dim=128, hidden_dim=128, num_heads=4, head_dim=64, num_kv_heads=2,
                      qk_norm=qk_norm, dtype=torch.bfloat16, max_position=64)
    att = Attention(cfg, 0, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    with torch.no_grad():
        for p in att.parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=g) * 0.1 + (1.0 if p.dim() == 1 else 0.0))
    x = torch.randn(2, 33, 128, device="cuda", generator=g).to(torch.bfloat16)
    pos = torch.arange(33, device="cuda", dtype=torch.int32)[None].expand(2, 33).contiguous()
    ang = torch.randn(64, 32, device="cuda", generator=g)
    def run():
        leaf = x.clone().requires_grad_()
        y, _ = att(leaf, pos, (ang.cos(), ang.sin()))
        return [y.detach(), *torch.autograd.grad(y.float().pow(2).sum(), [leaf, *att.parameters()])]
    joint, sep = run(), None
    real, F.qk_rope = F.qk_rope, lambda *a, **k: None
    try:
        sep = run()
    finally:
        F.qk_rope = real
    assert torch.equal(joint[0], sep[0])                               # the same roundings forward
    for a, b in zip(joint[1:], sep[1:]):
        assert _rel_err(a, b) < 2e-2, (a.shape, _rel_err(a, b))        # a few roundings to bf16 apart
    _check_status()


def _normal(*shape, seed):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("M,N,K_,gap", [(2065, 1300, 320, 4), (2065, 1300, 320, 8), (2048, 1536, 256, 0), (5000, 776, 264, 24)])
def test_gemm_result_blocks(M, N, K_, gap):
    """Results of the two-SM kernel in blocks of 32 rows and 128 bytes: edges inside a block, rows that lie apart (1308 bf16 columns
    are no whole 16-byte pieces and leave by a lane a row), every way the results leave, and nothing written beside them."""
    k = _k()
    a, b = _normal(M, K_, seed=1).bfloat16(), _normal(N, K_, seed=2).bfloat16()
    bias, res = _normal(N, seed=3).bfloat16(), _normal(M, N, seed=4).bfloat16()
    want = a.double() @ b.double().t()
    for dtype, tol in ((torch.bfloat16, 2e-3), (torch.float32, 1e-5)):       # one rounding; sums of K_ products in 32 bits
        for what in ("plain", "epilogue", "sum"):
            wide = torch.full((M, N + gap), 3.0, device="cuda", dtype=dtype)
            out = wide[:, :N]
            if what == "plain":
                k.gemm(a, b, out=out)
                ref = want
            elif what == "epilogue":
                k.gemm(a, b, out=out, bias=bias, residual=res, alpha=0.5)
                ref = 0.5 * want + bias.double() + res.double()
            else:
                k.gemm(a, b, out=out, accumulate=True, alpha=-0.25)
                ref = 3.0 - 0.25 * want
            assert _rel_err(out, ref) < tol, (dtype, what)
            assert bool((wide[:, N:] == 3.0).all())
    _check_status()


@pytest.mark.parametrize("M,N,Ks", [(2065, 1304, (320, 136, 64)), (2065, 1304, (64, 8, 320)), (300, 72, (128, 64, 72))])
@pytest.mark.parametrize("b_mn", [False, True])
def test_gemm_sum_of_three_products(M, N, Ks, b_mn):
    """Contractions that end inside a k-block, in any of the products; the last size is left to one GEMM a product."""
    k = _k()
    xs = [_normal(M, K_, seed=i).bfloat16() for i, K_ in enumerate(Ks)]
    ws = [_normal(*((K_, N) if b_mn else (N, K_)), seed=9 + i).bfloat16() for i, K_ in enumerate(Ks)]
    want = sum(x.double() @ (w.double() if b_mn else w.double().t()) for x, w in zip(xs, ws))
    out = k.gemm_ext(*(t for p in zip(xs, ws) for t in p), b_mn=b_mn)
    assert _rel_err(out, want) < (2e-3 if M > 300 else 5e-3)                 # one rounding, or one a product
    _check_status()


@pytest.mark.parametrize("kind", ["silu", "gelu"])
@pytest.mark.parametrize("M,F_,D", [(2065, 1288, 1544), (4096, 768, 1536), (2065, 1288, 320)])
def test_gated_products(M, F_, D, kind):
    """The activation in the epilogue of the products in front of it; the last size is left to separate kernels."""
    from tunix_b200.ops import functional as F
    k = _k()
    x, wg, wu = _normal(M, D, seed=1).bfloat16(), 0.05 * _normal(F_, D, seed=2), 0.05 * _normal(F_, D, seed=3)
    wg, wu, wd = wg.bfloat16(), wu.bfloat16(), (0.1 * _normal(D, F_, seed=4)).bfloat16()
    res, dy = _normal(M, D, seed=5).bfloat16(), _normal(M, D, seed=6).bfloat16()
    kd = k.GLU_SILU if kind == "silu" else k.GLU_GELU
    act = torch.nn.functional.silu if kind == "silu" else lambda t: torch.nn.functional.gelu(t, approximate="tanh")
    g, u = x.double() @ wg.double().t(), x.double() @ wu.double().t()
    kept, bare = k.gemm_glu(x, wg, wu, kd, keep=True), k.gemm_glu(x, wg, wu, kd)
    assert (kept is None) == (D < 1536) and (bare is None) == (D < 1536)
    # gate, up and the result are rounded to bf16, each by about 1.7e-3 in the norm of many, a gate's by up to 1.5 of that behind the
    # activation (3.6e-3 in all); the hardware tanh of the GELU adds an error of up to 5e-4 of a gate
    tol = 4e-3 if kind == "silu" else 6e-3
    if kept is not None:
        assert _rel_err(kept[0], act(g) * u) < tol and _rel_err(kept[1], g) < 2e-3 and _rel_err(kept[2], u) < 2e-3
        assert torch.equal(bare[0], kept[0]) and bare[1] is None
    leaves = [t.clone().requires_grad_() for t in (x, wg, wu, wd, res)]
    out = F.gated_mlp(*leaves[:4], kind, leaves[4])
    ref = [t.double().requires_grad_() for t in (x, wg, wu, wd, res)]
    want = (act(ref[0] @ ref[1].t()) * (ref[0] @ ref[2].t())) @ ref[3].t() + ref[4]
    assert _rel_err(out, want) < 6e-3
    out.backward(dy)
    want.backward(dy.double())
    for a, b in zip(leaves, ref):
        assert _rel_err(a.grad, b.grad) < 1e-2, a.shape                      # gate, up and hidden rows rounded to bf16 on the way
    _check_status()


@pytest.mark.parametrize("kind", ["silu", "gelu"])
@pytest.mark.parametrize("M,F_,D", [(2065, 1288, 1544), (4096, 768, 1536)])
def test_gated_products_round_like_separate_kernels(M, F_, D, kind):
    """The epilogue's activation is that of gate and up as they leave, bit for bit: dense, kept or not, and grouped by experts."""
    k = _k()
    kd = k.GLU_SILU if kind == "silu" else k.GLU_GELU
    x, wg, wu = (_normal(M, D, seed=1).bfloat16(), (0.05 * _normal(F_, D, seed=2)).bfloat16(), (0.05 * _normal(F_, D, seed=3)).bfloat16())
    h, g, u = k.gemm_glu(x, wg, wu, kd, keep=True)
    assert torch.equal(h, k.glu_fwd(g, u, kd)) and torch.equal(h, k.gemm_glu(x, wg, wu, kd)[0])
    seg = torch.tensor([0, 384, 384, 640], dtype=torch.int32, device="cuda")
    gate, up = (_normal(3 * 320, 512, seed=s).bfloat16() for s in (4, 5))
    tiles = k.moe_tiles_rows(seg, 640, 320, 512, 320, pairs=True, glu=True)
    h, g, u = k.gemm_grouped_glu(x[:640, :512].contiguous(), gate, up, tiles, kd)
    assert torch.equal(h, k.glu_fwd(g, u, kd))
    _check_status()


@pytest.mark.parametrize("rows,D", [(1, 64), (77, 896), (300, 4096), (40, 6144), (9, 12288)])
@pytest.mark.parametrize("frozen", [False, True])
def test_rmsnorm_with_the_streams_gradient(rows, D, frozen):
    """The norm's gradient and the one that passes it by, in one kernel, against their sum; in the kernels for narrow, wide and widest rows."""
    from tunix_b200.ops import functional as F
    x, w = _normal(rows, D, seed=1).bfloat16(), (1 + 0.1 * _normal(D, seed=2)).bfloat16()
    dy, dres = _normal(rows, D, seed=3).bfloat16(), _normal(rows, D, seed=4).bfloat16()
    leaf, wl = x.clone().requires_grad_(), w.clone().requires_grad_(not frozen)
    y, kept = F.rmsnorm_keep(leaf, wl, 1e-6)
    torch.autograd.backward([y, kept], [dy, dres])
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    yd = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
    torch.autograd.backward([yd, xd * 1.0], [dy.double(), dres.double()])
    assert _rel_err(y, yd) < 2e-3 and torch.equal(kept, x) and _rel_err(leaf.grad, xd.grad) < 2e-3       # one rounding
    assert frozen or _rel_err(wl.grad, wd.grad) < 4e-3
    _check_status()


@pytest.mark.parametrize("M", [2065, 70])
def test_joint_projections(M):
    """Three projections of one input, with and without biases, into gradients of their own and into `main_grad`."""
    from tunix_b200.ops import functional as F
    D, outs = 328, (1024, 264, 264)
    x = _normal(M, D, seed=1).bfloat16()
    ws = [(0.1 * _normal(o, D, seed=2 + i)).bfloat16() for i, o in enumerate(outs)]
    bs = [_normal(outs[0], seed=7).bfloat16(), None, _normal(outs[2], seed=8).bfloat16()]
    dys = [_normal(M, o, seed=20 + i).bfloat16() for i, o in enumerate(outs)]
    leaf = x.clone().requires_grad_()
    wl = [w.clone().requires_grad_() for w in ws]
    bl = [None if b is None else b.clone().requires_grad_() for b in bs]
    wl[1].main_grad = torch.ones_like(wl[1], dtype=torch.float32)
    ys = F.joint_linear(leaf, list(zip(wl, bl)))
    torch.autograd.backward(ys, dys)
    for y, w, b in zip(ys, ws, bs):
        assert _rel_err(y, x.double() @ w.double().t() + (0 if b is None else b.double())) < 2e-3
    # a rounding a product (1.7e-3 each in the norm), or one in all
    assert _rel_err(leaf.grad, sum(d.double() @ w.double() for d, w in zip(dys, ws))) < 5e-3
    for i, (w, d) in enumerate(zip(wl, dys)):
        want = d.double().t() @ x.double()
        if i == 1:
            assert w.grad is None and w.grad_added_to_main_grad and _rel_err(w.main_grad, want + 1) < 1e-5
        else:
            assert _rel_err(w.grad, want) < 2e-3
    assert _rel_err(bl[0].grad, dys[0].double().sum(0)) < 2e-3 and bl[1] is None
    _check_status()


@pytest.mark.parametrize("M,N,K_", [(5, 6144, 4096), (16, 1000, 520), (33, 136, 2056), (64, 4096, 12288), (4004, 16, 3584), (2056, 24, 1000),
                                    (16, 3584, 4004), (776, 64, 512), (48, 9000, 640)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_with_a_short_side(M, N, K_, a_mn, b_mn):
    """One side of at most 64: the other in tiles of 128 with the contraction over a cluster; ragged tiles, columns and k-blocks, every layout
    and way the result leaves, and more tiles than clusters (left to the other kernels)."""
    k = _k()
    up8 = lambda n: (n + 7) // 8 * 8  # noqa: E731
    def operand(rows, mn, seed):          # strides are multiples of 8 whatever the sizes
        t = _normal(*((K_, up8(rows)) if mn else (rows, up8(K_))), seed=seed).bfloat16()
        return t[:, :rows] if mn else t[:, :K_]
    a, b = operand(M, a_mn, 1), operand(N, b_mn, 2)
    want = (a.double().t() if a_mn else a.double()) @ (b.double() if b_mn else b.double().t())
    bias, res = _normal(N, seed=3).bfloat16(), _normal(M, N, seed=4).bfloat16()
    kw = dict(a_mn=a_mn, b_mn=b_mn)
    assert _rel_err(k.gemm(a, b, **kw), want) < 2e-3                         # one rounding
    assert _rel_err(k.gemm(a, b, out_dtype=torch.float32, **kw), want) < 1e-5                 # sums of K_ products in 32 bits
    assert _rel_err(k.gemm(a, b, bias=bias, residual=res, alpha=0.5, **kw), 0.5 * want + bias.double() + res.double()) < 2e-3
    for dtype, tol in ((torch.bfloat16, 2e-3), (torch.float32, 1e-5)):
        wide = torch.full((M, N + 3), 2.0, device="cuda", dtype=dtype)
        k.gemm(a, b, out=wide[:, :N], accumulate=True, **kw)
        assert _rel_err(wide[:, :N], want + 2.0) < tol and bool((wide[:, N:] == 2.0).all())
    _check_status()


@pytest.mark.parametrize("M,N,K_", [(64, 4096, 12288), (5, 4096, 8192), (16, 1536, 8960), (33, 3590, 14336), (48, 800, 9000), (17, 4096, 4096),
                                    (64, 2304, 4104), (64, 9472, 4096)])
def test_gemm_of_a_few_rows_sums_the_same_partial_products(M, N, K_):
    """Bit for bit what the kernel for higher problems gives (the same rows among 65, which it takes from K = 8192 on, or the product scaled by
    two, which it takes always), whatever the rows, ragged columns and k-blocks and way out."""
    k = _k()
    a, b = _normal(65, K_, seed=1).bfloat16(), _normal(N, K_, seed=2).bfloat16()
    bias, res, base = _normal(N, seed=3).bfloat16(), _normal(65, N, seed=4).bfloat16(), _normal(65, N, seed=5).bfloat16()
    for kw in (dict(), dict(bias=bias), dict(bias=bias, residual=res), dict(out_dtype=torch.float32)):
        cut = {key: v[:M] if key == "residual" else v for key, v in kw.items()}
        got = k.gemm(a[:M], b, **cut)
        assert torch.equal(2 * got, k.gemm(a[:M], b, alpha=2.0, **{key: v if key == "out_dtype" else 2 * v for key, v in cut.items()}))
        if K_ >= 8192:
            assert torch.equal(got, k.gemm(a, b, **kw)[:M])
    got, two = base[:M].clone(), 2 * base[:M]
    assert torch.equal(2 * k.gemm(a[:M], b, out=got, accumulate=True), k.gemm(a[:M], b, out=two, accumulate=True, alpha=2.0))
    _check_status()


@pytest.mark.parametrize("rows,V,D,share,chunk", [(4094, 2048, 512, 0.6, 2048), (2250, 5000, 264, 0.5, 1000), (3000, 4096, 256, 0.0, 2048),
                                                  (2048, 2304, 256, 1.0, 2048), (5000, 3080, 384, 0.02, 2048)])
@pytest.mark.parametrize("softcap,want_ent", [(0.0, True), (30.0, False)])
def test_head_over_the_rows_that_count(rows, V, D, share, chunk, softcap, want_ent, monkeypatch):
    """Log-probs, entropies and gradients of the rows with a target; none, all, few rows, chunks that are no whole blocks of 64, a last
    chunk with the one before, gradients added to what is there. The other rows hold values that would spoil any sum they took part in."""
    from tunix_b200.ops import functional as F
    monkeypatch.setattr(F, "_SCORED_MIN", 0)
    g = torch.Generator(device="cuda").manual_seed(rows)
    h, w = torch.randn(rows, D, device="cuda", generator=g).bfloat16(), (0.2 * torch.randn(V, D, device="cuda", generator=g)).bfloat16()
    tg = torch.randint(0, V, (rows,), device="cuda", generator=g)
    tg[torch.rand(rows, device="cuda", generator=g) >= share] = -1
    on = tg >= 0
    bad = h.clone()
    bad[~on] = float("nan")
    leaf, wl = bad.clone().requires_grad_(), w.clone().requires_grad_()
    wl.main_grad = torch.ones(V, D, device="cuda")
    logp, ent = F.lm_head_logprobs(leaf, wl, tg, softcap=softcap, temperature=0.8, want_entropy=want_ent, chunk=chunk, skip_ignored=True)
    assert type(logp.grad_fn).__name__ == "_LmHeadScoredFnBackward"
    z = h.double() @ w.double().t()
    hd, wd = h.double().requires_grad_(), w.double().requires_grad_()
    z = hd @ wd.t()
    z = (softcap * torch.tanh(z / softcap) if softcap else z) / 0.8
    lsm = torch.log_softmax(z, -1)
    ref = torch.where(on, lsm.gather(1, tg.clamp(min=0)[:, None])[:, 0], 0.0)
    ref_e = torch.where(on, -(lsm.exp() * lsm).sum(-1), 0.0)
    wa, we = torch.randn(rows, device="cuda", generator=g), torch.randn(rows, device="cuda", generator=g)
    (logp * wa + (ent * we if want_ent else 0.0)).sum().backward()
    (ref * wa.double() + (ref_e * we.double() if want_ent else 0.0)).sum().backward()
    assert bool((logp[~on] == 0).all()) and (not want_ent or bool((ent[~on] == 0).all()))
    if share:
        # 32-bit softmax of sums over bf16 rows; the capped score's tanh is off by 5e-4 of the cap
        tol = 1e-4 if not softcap else 4e-3
        assert _rel_err(logp, ref) < tol and (not want_ent or _rel_err(ent, ref_e) < tol)
        assert _rel_err(leaf.grad[on], hd.grad[on]) < 1e-2              # dz rounded to bf16 on the way
    assert bool((leaf.grad[~on] == 0).all()) and _rel_err(wl.main_grad, wd.grad + 1) < 1e-2 and wl.grad is None
    _check_status()


@pytest.mark.parametrize("count", [0, 1, 64, 700, 2048, 2049, 2500, 4094])
@pytest.mark.parametrize("off", [0, 2048])
def test_products_that_end_at_a_number_on_the_device(count, off):
    """`gemm_limited` at sizes that the kernel takes: rows (tiles past the limit stay as they are) and contractions that end inside a block
    of 64, on its edge, before the chunk and past it, over operands that are NaN behind the zeros up to the block's end; a contraction of
    nothing leaves what it would add to alone, the sign of its zeros too."""
    k = _k()
    M, N, K_ = 2046, 2560, 1536
    n = max(0, min(M, count - off))
    limit = torch.tensor([count], dtype=torch.int32, device="cuda")
    a, b = _normal(M, K_, seed=1).bfloat16(), (0.1 * _normal(K_, N, seed=2)).bfloat16()
    out = torch.full((M, N), -7.0, device="cuda", dtype=torch.bfloat16)
    assert k.gemm_limited(a, b, out, limit, off, b_mn=True)
    assert n == 0 or _rel_err(out[:n], a[:n].double() @ b.double()) < 2e-3
    assert bool((out[-(-n // 256) * 256:] == -7.0).all())
    x, y = _normal(M, N, seed=3).bfloat16(), (0.1 * _normal(M, K_, seed=4)).bfloat16()
    x[n:] = y[n:] = 0
    x[n + 63:] = y[n + 63:] = float("nan")
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 3e-3)):
        for start in (-0.0, 1.0):
            out = torch.full((N, K_), start, device="cuda", dtype=dtype)
            assert k.gemm_limited(x, y, out, limit, off, a_mn=True, b_mn=True, accumulate=True, contraction=True)
            if n:
                assert _rel_err(out, x[:n].double().t() @ y[:n].double() + start) < tol
            else:
                assert bool((out == start).all()) and bool((out.signbit() == (start == 0)).all())
    out = torch.full((N, K_), 5.0, device="cuda")
    assert k.gemm_limited(x, y, out, limit, off, a_mn=True, b_mn=True, contraction=True)
    assert _rel_err(out, x[:n].double().t() @ y[:n].double()) < 1e-5 if n else bool((out == 0).all())
    _check_status()


@pytest.mark.parametrize("count", [0, 1, 700, 2111, 4094])
@pytest.mark.parametrize("held", [False, True])
def test_head_over_the_rows_that_count_on_sm_pairs(count, held, monkeypatch):
    """The head at sizes where every product runs on SM pairs, with a gradient kept in 32 bits or not: the second chunk empty, ending inside a
    block, or full."""
    from tunix_b200.ops import functional as F
    rows, V, D = 4094, 8192, 3072
    monkeypatch.setattr(F, "_SCORED_MIN", 0)
    ran, real = [], F.K.gemm_limited
    monkeypatch.setattr(F.K, "gemm_limited", lambda *a, **kw: (ran.append(real(*a, **kw)), ran[-1])[1])
    g = torch.Generator(device="cuda").manual_seed(count)
    h, w = torch.randn(rows, D, device="cuda", generator=g).bfloat16(), (0.05 * torch.randn(V, D, device="cuda", generator=g)).bfloat16()
    tg = torch.randint(0, V, (rows,), device="cuda", generator=g)
    on = torch.zeros(rows, dtype=torch.bool, device="cuda")
    on[torch.randperm(rows, device="cuda", generator=g)[:count]] = True
    tg[~on] = -1
    bad = h.clone()
    bad[~on] = float("nan")
    leaf, wl = bad.requires_grad_(), w.clone().requires_grad_()
    if held:
        wl.main_grad = torch.ones(V, D, device="cuda")
    logp, _ = F.lm_head_logprobs(leaf, wl, tg, chunk=2048, skip_ignored=True)
    wa = torch.randn(rows, device="cuda", generator=g)
    (logp * wa).sum().backward()
    assert ran == [True] * 4
    z = h[on].double() @ w.double().t()
    lsm = torch.log_softmax(z, -1)
    assert bool((logp[~on] == 0).all()) and bool((leaf.grad[~on] == 0).all())
    dz = -lsm.exp()
    dz[torch.arange(count, device="cuda"), tg[on]] += 1
    dz *= wa[on].double()[:, None]
    dw = dz.t() @ h[on].double()
    got = wl.main_grad - 1 if held else wl.grad
    if count:
        assert _rel_err(logp[on], lsm.gather(1, tg[on][:, None])[:, 0]) < 1e-4
        assert _rel_err(leaf.grad[on], dz @ w.double()) < 1e-2 and _rel_err(got, dw) < 1e-2          # dz rounded to bf16 on the way
    else:
        assert bool((got == 0).all())
    _check_status()


@pytest.mark.parametrize("M,N,K_", [(256, 11264, 256), (256, 11008, 256), (255, 32768, 512), (2816, 1024, 248), (2816, 1024, 256), (1100, 2304, 4096)])
def test_the_head_asks_the_kernels_own_rule(M, N, K_, monkeypatch):
    """`two_sm_takes` says what a limited product of these sizes does, also where a switch has changed since the kernels read it."""
    k = _k()
    a, b, limit = _normal(M, K_, seed=1).bfloat16(), _normal(N, K_, seed=2).bfloat16(), torch.tensor([M], dtype=torch.int32, device="cuda")
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    k.gemm(a, b)
    for switch in (None, "TUNIX_B200_NO_2CTA"):
        if switch:
            monkeypatch.setenv(switch, "1")
        assert k.two_sm_takes(M, N, K_) == k.gemm_limited(a, b, out, limit, 0)
    _check_status()


@pytest.mark.parametrize("M,F_,D", [(300, 2816, 8192), (512, 3072, 9000), (300, 2816, 4096), (513, 2816, 8192)])
def test_gated_products_sum_like_separate_products(M, F_, D):
    """Gate and up bit for bit those of the two products, also where these are sums of several parts (which the joint launch leaves to them)."""
    k = _k()
    x, wg, wu = _normal(M, D, seed=1).bfloat16(), (0.05 * _normal(F_, D, seed=2)).bfloat16(), (0.05 * _normal(F_, D, seed=3)).bfloat16()
    out = k.gemm_glu(x, wg, wu, k.GLU_SILU, keep=True)
    assert (out is None) == (M <= 512 and D >= 8192)
    if out is not None:
        assert torch.equal(out[1], k.gemm(x, wg)) and torch.equal(out[2], k.gemm(x, wu))
    _check_status()
