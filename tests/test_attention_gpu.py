"""tcgen05 flash attention (forward and backward) against an fp32 PyTorch reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def ref_attention(q, k, v, scale, causal, window, softcap, seg_q, seg_k):
    B, Tq, N, H = q.shape
    Tk, KH = k.shape[1], k.shape[2]
    G = N // KH
    qf = q.float().permute(0, 2, 1, 3)
    kf = k.float().permute(0, 2, 1, 3).repeat_interleave(G, dim=1)
    vf = v.float().permute(0, 2, 1, 3).repeat_interleave(G, dim=1)
    s = torch.einsum("bnqh,bnkh->bnqk", qf, kf) * scale
    if softcap > 0:
        s = softcap * torch.tanh(s / softcap)
    qpos = torch.arange(Tq, device=q.device)[:, None] + (Tk - Tq)
    kpos = torch.arange(Tk, device=q.device)[None, :]
    mask = torch.ones(Tq, Tk, dtype=torch.bool, device=q.device)
    if causal:
        mask &= kpos <= qpos
    if window > 0:
        mask &= kpos > qpos - window
    mask = mask[None, None].expand(B, 1, Tq, Tk)
    if seg_q is not None:
        mask = mask & (seg_q[:, None, :, None] == seg_k[:, None, None, :])
    s = s.masked_fill(~mask, float("-inf"))
    p = torch.softmax(s, dim=-1)
    p = torch.nan_to_num(p, nan=0.0)
    o = torch.einsum("bnqk,bnkh->bnqh", p, vf)
    return o.permute(0, 2, 1, 3)


CASES = [
    # B, Tq, Tk, N, KH, H, causal, window, softcap, segs
    (1, 128, 128, 1, 1, 128, True, 0, 0.0, False),
    (2, 256, 256, 4, 2, 128, True, 0, 0.0, False),
    (2, 200, 200, 4, 1, 64, True, 0, 0.0, False),
    (1, 512, 512, 4, 2, 128, True, 96, 0.0, False),
    (1, 384, 384, 2, 1, 256, True, 0, 50.0, False),
    (2, 320, 320, 4, 2, 128, True, 0, 0.0, True),
    (1, 64, 320, 4, 4, 128, True, 0, 0.0, False),
    (1, 256, 256, 2, 2, 128, False, 0, 0.0, False),
    (1, 1024, 1024, 8, 2, 128, True, 0, 0.0, False),
    # two query tiles per CTA: ragged last tile, a window narrower than a tile, more keys than queries, segments with a
    # soft-cap, no causal mask
    (1, 448, 448, 2, 1, 128, True, 0, 0.0, False),
    (2, 300, 300, 2, 2, 64, True, 64, 0.0, False),
    (1, 384, 640, 4, 2, 128, True, 0, 0.0, False),
    (1, 512, 512, 2, 1, 128, True, 0, 30.0, True),
    (1, 640, 640, 2, 2, 64, False, 0, 0.0, False),
]


def _make(B, Tq, Tk, N, KH, H, segs):
    torch.manual_seed(0)
    q = torch.randn(B, Tq, N, H, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(B, Tk, KH, H, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(B, Tk, KH, H, device="cuda", dtype=torch.bfloat16)
    seg_q = seg_k = None
    if segs:
        cuts = torch.tensor([0, Tk // 3, Tk // 3 + 70, Tk], device="cuda")
        seg_k = torch.bucketize(torch.arange(Tk, device="cuda"), cuts[1:], right=True).int()[None].expand(B, Tk).contiguous() + 1
        seg_q = seg_k[:, Tk - Tq:].contiguous()
    return q, k, v, seg_q, seg_k


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-9)).item()


def _close(a, b, what=""):
    """Element-wise, next to the norm: a handful of wrong elements cannot hide in a large tensor."""
    a, b = a.float(), b.float()
    tol = 0.03 * b.abs().max().item() + 1e-6
    bad = (a - b).abs() > tol + 0.05 * b.abs()
    assert not bad.any(), (what, int(bad.sum()), (a - b).abs().max().item(), tol)


@pytest.mark.parametrize("two_tile", [False, True])
@pytest.mark.parametrize("case", CASES)
def test_attention_forward(case, two_tile, monkeypatch):
    """Both forward kernels: one 128-row query tile per CTA (the default) and two tiles per CTA (opt-in)."""
    if two_tile and (case[5] > 128 or case[1] <= 128):
        pytest.skip("the two-tile kernel serves head dims up to 128 and more than 128 query rows")
    monkeypatch.setenv("TUNIX_B200_ATTN_TWO_TILE", "1" if two_tile else "0")
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    B, Tq, Tk, N, KH, H, causal, window, softcap, segs = case
    q, k, v, seg_q, seg_k = _make(B, Tq, Tk, N, KH, H, segs)
    scale = 1.0 / math.sqrt(H)
    o, lse = k_.attn_fwd(q, k, v, scale=scale, causal=causal, window=window, softcap=softcap, seg_q=seg_q, seg_k=seg_k)
    _lib.raise_if_kernel_error()
    ref = ref_attention(q, k, v, scale, causal, window, softcap, seg_q, seg_k)
    assert _rel(o, ref) < 2e-2, _rel(o, ref)
    _close(o, ref, "o")
    # log-sum-exp of every row that sees at least one key
    s_ = torch.einsum("bqnh,bknh->bnqk", q.float(), k.float().repeat_interleave(N // KH, dim=2)) * scale
    if softcap > 0:
        s_ = softcap * torch.tanh(s_ / softcap)
    qpos = torch.arange(Tq, device="cuda")[:, None] + (Tk - Tq)
    kpos = torch.arange(Tk, device="cuda")[None, :]
    m = torch.ones(Tq, Tk, dtype=torch.bool, device="cuda")
    if causal:
        m &= kpos <= qpos
    if window > 0:
        m &= kpos > qpos - window
    m = m[None, None].expand(B, 1, Tq, Tk)
    if seg_q is not None:
        m = m & (seg_q[:, None, :, None] == seg_k[:, None, None, :])
    want = torch.logsumexp(s_.masked_fill(~m, float("-inf")), dim=-1)
    seen = torch.isfinite(want)
    assert torch.allclose(lse[seen], want[seen], atol=2e-2, rtol=1e-3)


@pytest.mark.parametrize("case", CASES)
def test_attention_backward(case):
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    B, Tq, Tk, N, KH, H, causal, window, softcap, segs = case
    q, k, v, seg_q, seg_k = _make(B, Tq, Tk, N, KH, H, segs)
    scale = 1.0 / math.sqrt(H)
    do = torch.randn(B, Tq, N, H, device="cuda", dtype=torch.bfloat16)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = ref_attention(qf, kf, vf, scale, causal, window, softcap, seg_q, seg_k)
    ref.backward(do.float())
    o, lse = k_.attn_fwd(q, k, v, scale=scale, causal=causal, window=window, softcap=softcap, seg_q=seg_q, seg_k=seg_k)
    dq, dk, dv = k_.attn_bwd(do, q, k, v, o, lse, scale=scale, causal=causal, window=window, softcap=softcap,
                             seg_q=seg_q, seg_k=seg_k)
    _lib.raise_if_kernel_error()
    assert _rel(dv, vf.grad) < 3e-2, ("dv", _rel(dv, vf.grad))
    assert _rel(dk, kf.grad) < 3e-2, ("dk", _rel(dk, kf.grad))
    assert _rel(dq, qf.grad) < 3e-2, ("dq", _rel(dq, qf.grad))
    _close(dv, vf.grad, "dv")
    _close(dk, kf.grad, "dk")
    _close(dq, qf.grad, "dq")


def _segments(layout, B, Tq, Tk):
    g = torch.Generator().manual_seed(3)
    if layout == "whole_blocks":                # boundaries on block edges: listed blocks hold one id
        seg = (torch.arange(Tk) // 128).expand(B, Tk)
    elif layout == "mixed":                     # ids in no order, negative ones among them: every block is compared
        seg = torch.randint(-2, 3, (B, Tk), generator=g)
    elif layout == "pads":                      # padding on both sides of a row, a row of padding alone
        seg = torch.zeros(B, Tk, dtype=torch.long)
        seg[0, 37:Tk - 70] = 1
    else:                                       # "unseen": the ids of some queries occur in no key
        seg = (torch.arange(Tk) // 100).expand(B, Tk)
    seg_k = seg.to(torch.int32).contiguous().cuda()
    seg_q = seg_k[:, Tk - Tq:].contiguous()
    if layout == "unseen":
        seg_q = torch.where(seg_q == 2, 1 << 20, seg_q).int().contiguous()
    return seg_q, seg_k


@pytest.mark.parametrize("H", [64, 128, 256])
@pytest.mark.parametrize("window", [0, 150])
@pytest.mark.parametrize("layout", ["whole_blocks", "mixed", "pads", "unseen"])
def test_segment_blocks(layout, window, H):
    """Key blocks that the segment ids leave out, let pass unseen, or have compared element by element."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    B, Tq, Tk, N, KH = 2, 509, 573, 4, 2
    q, k, v, _, _ = _make(B, Tq, Tk, N, KH, H, False)
    seg_q, seg_k = _segments(layout, B, Tq, Tk)
    do = torch.randn(B, Tq, N, H, device="cuda", dtype=torch.bfloat16)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = ref_attention(qf, kf, vf, H ** -0.5, True, window, 0.0, seg_q, seg_k)
    ref.backward(do.float())
    kw = dict(scale=H ** -0.5, causal=True, window=window, seg_q=seg_q, seg_k=seg_k)
    o, lse = k_.attn_fwd(q, k, v, **kw)
    grads = k_.attn_bwd(do, q, k, v, o, lse, **kw)
    _lib.raise_if_kernel_error()
    # bf16 operands (2^-9 each) in sums of products: the bounds of the tests above
    assert _rel(o, ref) < 2e-2
    _close(o, ref, "o")
    for name, got, want in zip(("dq", "dk", "dv"), grads, (qf.grad, kf.grad, vf.grad)):
        assert _rel(got, want) < 3e-2, (name, _rel(got, want))
        _close(got, want, name)


def test_segments_past_the_block_list():
    """More key blocks than the list of a tile holds."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    Tq, Tk = 64, 64 * 2048 + 100
    q, k, v, _, _ = _make(1, Tq, Tk, 1, 1, 64, False)
    seg_k = (torch.arange(Tk, device="cuda") // 50000).int()[None].contiguous()
    seg_q = torch.full((1, Tq), 1, dtype=torch.int32, device="cuda")
    seg_q[0, 40:] = 2
    o, _ = k_.attn_fwd(q, k, v, scale=0.125, causal=False, seg_q=seg_q, seg_k=seg_k)
    _lib.raise_if_kernel_error()
    ref = ref_attention(q, k, v, 0.125, False, 0, 0.0, seg_q, seg_k)
    assert _rel(o, ref) < 2e-2


@pytest.mark.parametrize("H", [64, 128])
def test_gradients_of_rollouts_repeat(H):
    """Rows padded at both ends make the warps of a block run apart (they fetch segment ids on their own): what the kernels sum in a
    fixed order is the same bit for bit in every run."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    B, T, N, KH = 8, 1024, 16, 4
    q, k, v, _, _ = _make(B, T, T, N, KH, H, False)
    do = torch.randn(B, T, N, H, device="cuda", dtype=torch.bfloat16)
    at = torch.arange(T, device="cuda")[None]
    seg = ((at >= 23 * torch.arange(B, device="cuda")[:, None]) & (at < T - 61 * torch.arange(B, device="cuda")[:, None])).int().contiguous()
    first = None
    for _ in range(40):
        o, lse = k_.attn_fwd(q, k, v, scale=H ** -0.5, seg_q=seg, seg_k=seg)
        _, dk, dv = k_.attn_bwd(do, q, k, v, o, lse, scale=H ** -0.5, seg_q=seg, seg_k=seg)
        got = (o, lse, dk, dv)
        first = first or [t.clone() for t in got]
        assert all(torch.equal(a, b) for a, b in zip(got, first))
    _lib.raise_if_kernel_error()


def test_backward_past_32768_query_tiles():
    """More query tiles than the block numbers of a segment list count: every query meets the keys once."""
    from tunix_b200 import _lib
    from tunix_b200.ops import kernels as k_
    Tq, Tk, H = 64 * 32768 + 130, 40, 64
    q, k, v, _, _ = _make(1, Tq, Tk, 1, 1, H, False)
    do = torch.randn(1, Tq, 1, H, device="cuda", dtype=torch.bfloat16)
    kw = dict(scale=H ** -0.5, causal=False)
    o, lse = k_.attn_fwd(q, k, v, **kw)
    dq, dk, dv = k_.attn_bwd(do, q, k, v, o, lse, **kw)
    _lib.raise_if_kernel_error()
    qf, kf, vf, df = (t[0, :, 0].float() for t in (q, k, v, do))
    p = (qf @ kf.T * H ** -0.5).softmax(-1)
    ds = p * (df @ vf.T - (df * (p @ vf)).sum(-1, keepdim=True)) * H ** -0.5
    # the bounds of the tests above
    for name, got, want in (("dq", dq, ds @ kf), ("dk", dk, ds.T @ qf), ("dv", dv, p.T @ df)):
        assert _rel(got[0, :, 0], want) < 3e-2, (name, _rel(got[0, :, 0], want))
    assert _rel(dq[0, -130:, 0], (ds @ kf)[-130:]) < 3e-2


@pytest.mark.parametrize("H,off,gap", [(128, 0, 0), (128, 2, 0), (64, 0, 2), (96, 0, 0), (30, 2, 6)])
def test_delta_rows(H, off, gap):
    """Row sums of dO * O of rows without whole 16-byte pieces, and of head sizes that the attention kernels do not take."""
    from tunix_b200 import _lib
    B, T, N = 2, 37, 3
    g = torch.Generator(device="cuda").manual_seed(13)
    ld = N * H + gap
    o, do = (torch.randn(B * T * ld + off, device="cuda", generator=g).to(torch.bfloat16)[off:].view(B, T, ld)[..., :N * H] for _ in range(2))
    delta = torch.empty(B, N, T, device="cuda")
    rc = _lib.cuda().tb_attn_delta(o.data_ptr(), ld, do.data_ptr(), ld, delta.data_ptr(), B, T, N, H, _lib.stream_ptr())
    assert rc == 0
    want = (o.double() * do.double()).unflatten(-1, (N, H)).sum(-1).transpose(1, 2)
    assert ((delta.double() - want).norm() / want.norm()).item() < 1e-6          # 32-bit sums of up to 128 terms
