"""Fused sampling kernel against the PyTorch reference filter."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_greedy_and_logprob():
    from tunix_b200.ops import sampling_kernels as S
    torch.manual_seed(0)
    z = torch.randn(33, 50257, device="cuda")
    tok, lp = S.sample(z, 0.0, None, None, 0, 0, want_logprob=True)
    assert torch.equal(tok, z.argmax(-1))
    ref = torch.log_softmax(z, -1).gather(1, tok[:, None])[:, 0]
    assert torch.allclose(lp, ref, atol=1e-4)


@pytest.mark.parametrize("top_k,top_p", [(None, None), (20, None), (None, 0.8), (50, 0.9)])
def test_samples_stay_in_kept_set_and_follow_distribution(top_k, top_p):
    from tunix_b200.generate import sampling
    from tunix_b200.ops import sampling_kernels as S
    torch.manual_seed(1)
    V, temp = 2000, 0.8
    row = torch.randn(1, V, device="cuda") * 2
    z = row.expand(4096, V).contiguous()
    kept = torch.isfinite(sampling.filter_logits(row, temp, top_p, top_k))[0]
    tok, lp = S.sample(z, temp, top_p, top_k, seed=11, step=3, want_logprob=True)
    assert kept[tok].float().mean().item() > 0.995          # threshold ties may differ by one token
    ref_p = torch.softmax(sampling.filter_logits(row, temp, top_p, top_k), -1)[0]
    emp = torch.bincount(tok, minlength=V).float() / tok.numel()
    top = ref_p.topk(5).indices
    assert torch.allclose(emp[top], ref_p[top], atol=0.03)
    ref_lp = torch.log_softmax(row / temp, -1)[0][tok]
    assert torch.allclose(lp, ref_lp, atol=1e-4)
    tok2, _ = S.sample(z, temp, top_p, top_k, seed=11, step=3)
    assert torch.equal(tok, tok2)                             # same (seed, step) -> same draw
    tok3, _ = S.sample(z, temp, top_p, top_k, seed=11, step=4)
    assert not torch.equal(tok, tok3)
    assert tok.unique().numel() > 1                           # rows draw independently


def _kept(z, temp, top_k, top_p):
    """The filter in 64 bits: e = exp(z / temp - max) at least the largest multiple of 2^-26 that keeps top_k tokens, then the
    largest that keeps a mass of top_p among them. Also where rounding in 32 bits may decide otherwise."""
    e = torch.exp((z.double() / temp) - (z.double() / temp).max(-1, keepdim=True).values)
    u = 2.0 ** -26
    lo = torch.zeros(e.shape[0], 1, dtype=torch.float64, device=z.device)
    if top_k:
        lo = (e.topk(top_k, -1).values[:, -1:] / u).floor() * u
    keep = e >= lo
    if top_p:
        s, _ = torch.where(keep, e, 0.0).sort(-1, descending=True)
        need = (s.cumsum(-1) >= top_p * s.sum(-1, keepdim=True)).float().argmax(-1, keepdim=True)
        lo = torch.maximum(lo, (s.gather(-1, need) / u).floor() * u)
    return e >= lo * (1 - 1e-5) - 1e-7, e


@pytest.mark.parametrize("shape", ["flat", "peaked", "ties", "forbidden"])
@pytest.mark.parametrize("V", [3, 1023, 32771, 151936])
@pytest.mark.parametrize("top_k,top_p", [(1, None), (50, 0.95), (None, 0.95), (None, 0.9999), (40000, 0.5)])
def test_filtered_draws_for_any_split_of_the_row(shape, V, top_k, top_p):
    """Rows are split over 8, 4, 2 or 1 thread blocks by the batch size; the draw of a row does not depend on it."""
    from tunix_b200.ops import sampling_kernels as S
    if top_k and top_k >= V:
        top_k = 2
    torch.manual_seed(V)
    B, temp = 300, 0.9
    z = torch.randn(B, V, device="cuda") * {"flat": 0.01, "peaked": 4.0}.get(shape, 1.5)
    if shape == "ties":
        z = (z * 2).round() / 2
    forbidden = None
    if shape == "forbidden":
        forbidden = torch.arange(0, V - 1, 2, dtype=torch.int32, device="cuda")
    ref = z.clone()
    if forbidden is not None:
        ref[:, forbidden.long()] = float("-inf")
    kept, _ = _kept(ref, temp, top_k, top_p)
    want = torch.log_softmax(ref.double() / temp, -1)
    whole = None
    for n in (300, 100, 60, 5, 1):
        tok, lp = S.sample(z[:n].clone(), temp, top_p, top_k, seed=7, step=2, want_logprob=True, forbidden=forbidden)
        whole = tok if whole is None else whole
        assert torch.equal(tok, whole[:n])
        assert kept[:n].gather(1, tok[:, None]).all()
        # 32-bit exponentials (2 ulp) and sums of up to 151936 terms in blocks: a relative error of the sum below 1e-5
        assert (lp - want[:n].gather(1, tok[:, None])[:, 0]).abs().max().item() < 1e-4


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_values_that_are_not_finite(value):
    """An infinite logit is drawn, rows of nothing but -inf give token 0, and a NaN is never drawn."""
    from tunix_b200.ops import sampling_kernels as S
    z = torch.zeros(2, 9000, device="cuda")
    z[0, 77] = value
    if value == float("-inf"):
        z[1] = value
    for top_k, top_p in ((None, None), (30, 0.9), (None, 0.9)):
        tok, _ = S.sample(z.clone(), 1.0, top_p, top_k, seed=1, step=1, want_logprob=True)
        if value == float("inf"):
            assert tok[0].item() == 77
        else:
            assert tok[0].item() != 77
        if value == float("-inf"):
            assert tok[1].item() == 0


@pytest.mark.parametrize("temp", [1e-4, 1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("top_k,top_p", [(1, None), (50, 0.95), (None, 0.95), (None, 0.9999), (3000, 0.5)])
def test_filtered_draws_at_low_temperatures(temp, top_k, top_p):
    """z / temperature up to 4e8, where the rounding of a product is many nats: no weight lies above the best token's, which leads by
    more than the draw's noise and is always the one, and log-probs are those of 64 bits. Rows on 1, 2, 4 and 8 thread blocks."""
    from tunix_b200.ops import sampling_kernels as S
    for V, B in ((5000, 40), (9000, 40), (151936, 300), (151936, 60), (151936, 5)):
        g = torch.Generator(device="cuda").manual_seed(B)
        z = torch.rand(B, V, device="cuda", generator=g) * 30 + 9.9
        best = torch.randint(0, V, (B,), device="cuda", generator=g)
        # the others end at 39.9: at least 0.1 / 1e-4 nats of lead against 23 of noise
        z.scatter_(1, best[:, None], 40 + torch.rand(B, 1, device="cuda", generator=g))
        tok, lp = S.sample(z, temp, top_p, top_k, seed=3, step=1, want_logprob=True)
        assert torch.equal(tok, best), (V, B)
        want = torch.log_softmax(z.double() / torch.tensor(temp, dtype=torch.float32).item(), -1).gather(1, best[:, None])[:, 0]
        # a weight's exponent is off by 2^-23 of itself, which nothing within 20 nats of the best token sees; sums as above
        assert (lp - want).abs().max().item() < 1e-4, (V, B)


@pytest.mark.parametrize("temp", [0.6, 0.9, 1.0, 1.3])
@pytest.mark.parametrize("weights,top_k,top_p,n_kept,crowd", [
    ((1.0, 0.97), 2, None, 2, None), ((0.9, 0.4, 0.3, 0.25, 0.2, 0.1), 5, None, 5, None),
    ((0.9, 0.1), None, 0.95, 2, None), ((0.55, 0.3, 0.15), None, 0.8, 2, None), ((0.55, 0.3, 0.15), None, 0.9, 3, None),
    ((0.5, 0.3, 0.2), 3, 0.75, 2, None),
    # more candidates than the list holds, so that the halvings run over the row: behind the k-th token in its own bin, or of no weight
    ((1.0, 0.8, 0.6), 3, None, 3, (0.594, 0.599)), ((0.5, 0.3, 0.2), 2500, 0.75, 2, (1e-6, 2e-6))])
def test_every_kept_token_is_drawn(weights, top_k, top_p, n_kept, crowd, temp):
    """The k-th token, or the one that completes the mass, comes as often as its weight says, at any rounding of z / temperature."""
    from tunix_b200.ops import sampling_kernels as S
    rows, draws, V = 256, 128, 16384
    g = torch.Generator(device="cuda").manual_seed(5)
    w = torch.tensor(weights, dtype=torch.float64, device="cuda")
    base = torch.rand(rows, 1, device="cuda", generator=g, dtype=torch.float64) * 20 + 10
    z = torch.full((rows, V), -60.0, dtype=torch.float64, device="cuda")
    at = torch.rand(rows, V, device="cuda", generator=g).argsort(-1)
    z.scatter_(1, at[:, :len(weights)], base + temp * w.log())
    if crowd:
        c = torch.linspace(*crowd, 3000, dtype=torch.float64, device="cuda")
        z.scatter_(1, at[:, len(weights):len(weights) + 3000], base + temp * c.log())
    z = z.float()
    kept = at[:, :n_kept]
    p = (z.double().gather(1, kept) / temp).softmax(-1)
    n = torch.zeros(rows, V, device="cuda")
    for step in range(draws):
        tok, _ = S.sample(z, temp, top_p, top_k, seed=17, step=step)
        n[torch.arange(rows, device="cuda"), tok] += 1
    n = n.gather(1, kept)
    assert (n.sum(1) == draws).all()                          # nothing else is drawn
    # counts of independent draws: 6 standard deviations over at most 1280 of them
    assert ((n - draws * p).abs() <= 6 * (draws * p * (1 - p)).sqrt()).all()
    assert ((n.sum(0) - draws * p.sum(0)).abs() <= 5 * (draws * (p * (1 - p)).sum(0)).sqrt()).all()
