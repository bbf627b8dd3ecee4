"""The flash attention kernels at the places where their pipelines can go wrong, against the fp32 reference."""
import pytest
import torch

from dew_b200 import ops
from dew_b200.ops import library as L

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def rel_err(a, b):
    a, b = a.double(), b.double()
    return float((a - b).norm() / b.norm().clamp_min(1e-12))


@pytest.mark.parametrize("S,docs,seed", [(2048, 6, 0), (2048, 6, 1), (4096, 9, 2), (4096, 40, 3)])
def test_flash_packed_documents_of_uneven_work(S, docs, seed):
    """Documents cut at arbitrary places: the warps of a query tile have unequal work (some rows of a key tile are masked element by element, some rescale,
    some do neither), so fast ones run a tile ahead of slow ones.  bf16 results of fp32 sums: a rounding of the probabilities (2^-9) and one of the result."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    B, Hq, Hkv, D = 2, 8, 2, 128
    # scores that grow along the row make the running maximum move, as trained attention does
    grow = torch.linspace(0.5, 4.0, S, device=DEV)[None, :, None, None]
    q, k, v = (torch.randn(B, S, h, D, generator=g, device=DEV) for h in (Hq, Hkv, Hkv))
    q, k, v = q.bfloat16(), (k * grow).bfloat16(), v.bfloat16()
    seg = torch.ones(B, S, dtype=torch.int32)
    r = torch.Generator().manual_seed(seed)
    for row in seg:
        for cut in (torch.randperm(S - 1, generator=r)[: docs - 1] + 1).tolist():
            row[cut:] += 1
    seg = seg.to(DEV)
    out = ops.attention(q, k, v, segment_ids=seg, kernel="sm100_flash")
    L.check_status()
    assert all(torch.equal(out, ops.attention(q, k, v, segment_ids=seg, kernel="sm100_flash")) for _ in range(5))
    assert rel_err(out, ops.attention_reference(q.float(), k.float(), v.float(), segment_ids=seg)) < 6e-3


def truth(q, k, v, causal, scale):
    """Attention in 64 bits, the causal mask aligned at the last query and key; -> output, log-sum-exp (natural), with a graph where the operands have one."""
    S, T, rep = q.shape[1], k.shape[1], q.shape[2] // k.shape[2]
    s = torch.einsum("bshd,bthd->bhst", q, k.repeat_interleave(rep, 2)) * scale
    if causal:
        s = s.masked_fill(~torch.ones(S, T, dtype=torch.bool, device=q.device).tril(T - S), float("-inf"))
    return torch.einsum("bhst,bthd->bshd", torch.softmax(s, -1), v.repeat_interleave(rep, 2)), torch.logsumexp(s, -1)


# query tiles alone (no more than there are SMs), two heads of a key head, and neighbouring rows (odd numbers of heads a key head, odd numbers of tiles); more items than
# CTAs; lengths that end inside a tile; more keys than queries
@pytest.mark.parametrize("B,S,T,Hq,Hkv,D,causal", [(1, 128, 128, 1, 1, 128, True), (1, 8, 8, 2, 1, 64, True), (2, 200, 200, 4, 2, 128, False), (2, 640, 640, 30, 30, 64, True),
                                                   (1, 1152, 1152, 17, 17, 128, True), (3, 384, 384, 32, 8, 64, False), (1, 2048, 2048, 12, 4, 128, True),
                                                   (1, 128, 640, 160, 80, 64, True), (2, 264, 1000, 40, 8, 128, True)])
def test_flash_forward_pairs_of_tiles(B, S, T, Hq, Hkv, D, causal):
    """The probabilities are rounded to bf16 (2^-9 each, independent) and so is the result; the log-sum-exp is made of fp32 sums of fp32 products of bf16 operands."""
    from dew_b200.ops.flash import flash_fwd
    g = torch.Generator(device=DEV).manual_seed(S + Hq)
    q, k, v = (torch.randn(B, n, h, D, generator=g, device=DEV).bfloat16() for n, h in ((S, Hq), (T, Hkv), (T, Hkv)))
    out, lse = flash_fwd(q, k, v, causal, D ** -0.5)
    L.check_status()
    want, want_lse = truth(q.double(), k.double(), v.double(), causal, D ** -0.5)
    assert rel_err(out, want) < 2.0 ** -8
    assert float((lse.double() - want_lse).abs().max()) < 1e-5 * max(1.0, float(want_lse.abs().max()))


@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal", [(1, 64, 1, 1, 128, True), (1, 192, 4, 1, 64, False), (1, 192, 2, 2, 128, True), (2, 640, 30, 15, 64, True), (1, 1152, 18, 6, 128, True),
                                                 (2, 256, 96, 32, 128, False)])
def test_flash_backward_tiles(B, S, Hq, Hkv, D, causal):
    """Lengths that end in the middle of a tile of queries (their statistics are half there), more query tiles than CTAs, several heads a key head.  Weights and their
    gradients are rounded to bf16 (2^-9 each) in front of the products, the results once more."""
    from dew_b200.ops.flash import flash_bwd, flash_fwd
    g = torch.Generator(device=DEV).manual_seed(S + Hq)
    q, k, v, do = (torch.randn(B, S, h, D, generator=g, device=DEV).bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    out, lse = flash_fwd(q, k, v, causal, D ** -0.5)
    got = flash_bwd(do, q, k, v, out, lse, causal, D ** -0.5)
    again = flash_bwd(do, q, k, v, out, lse, causal, D ** -0.5)
    L.check_status()
    leaves = [x.double().requires_grad_() for x in (q, k, v)]
    want = torch.autograd.grad(truth(*leaves, causal, D ** -0.5)[0], leaves, do.double())
    for a, b, w in zip(got, again, want):
        assert torch.equal(a, b)
        assert rel_err(a, w) < 2.0 ** -7


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("gap", [0, 8, 16, 24])
def test_flash_gradients_into_rows_of_any_alignment(D, gap):
    """Rows that start on a 16-byte boundary only, all of them or every second one, get the same bits, and what lies between them is left alone."""
    from dew_b200.ops.flash import flash_bwd, flash_fwd
    g = torch.Generator(device=DEV).manual_seed(gap)
    B, S, Hq, Hkv = 1, 192, 4, 2
    q, k, v, do = (torch.randn(B, S, h, D, generator=g, device=DEV).bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    out, lse = flash_fwd(q, k, v, True, D ** -0.5)
    want = flash_bwd(do, q, k, v, out, lse, True, D ** -0.5)
    wide = [torch.full((B, S, h, D + gap), 7.0, device=DEV, dtype=torch.bfloat16) for h in (Hq, Hkv, Hkv)]
    first = gap // 2 // 8 * 8
    flash_bwd(do, q, k, v, out, lse, True, D ** -0.5, grads=[w[..., first:first + D] for w in wide])
    L.check_status()
    for a, w in zip(want, wide):
        assert torch.equal(w[..., first:first + D], a)
        assert bool((w[..., :first] == 7).all()) and bool((w[..., first + D:] == 7).all())


# one key tile (the second half has none), two, an odd number; rows and keys that end inside a tile; keys before and behind the queries; rows that one half sees nothing
# of, and rows that see nothing; a second wave of items; one row fewer and more than the line to pairs
@pytest.mark.parametrize("B,S,T,Hq,Hkv,D,causal", [(1, 128, 128, 1, 1, 128, True), (1, 64, 384, 2, 2, 64, False), (2, 384, 640, 2, 1, 128, True), (1, 200, 333, 4, 2, 64, True),
                                                   (1, 333, 200, 2, 2, 128, True), (1, 1100, 1100, 8, 8, 64, False), (1, 1024, 1024, 37, 37, 64, True), (1, 896, 896, 37, 37, 128, True),
                                                   (1, 2000, 2000, 12, 4, 128, True)])
@pytest.mark.parametrize("sinks", [False, True])
def test_flash_halves_of_a_rows_keys(B, S, T, Hq, Hkv, D, causal, sinks):
    from dew_b200.ops.flash import NONE, Variants, flash_fwd
    g = torch.Generator(device=DEV).manual_seed(S + T)
    q, k, v = (torch.randn(B, n, h, D, generator=g, device=DEV).bfloat16() for n, h in ((S, Hq), (T, Hkv), (T, Hkv)))
    sink = torch.randn(Hq, generator=g, device=DEV)
    out, lse = flash_fwd(q, k, v, causal, D ** -0.5, var=Variants(sinks=sink) if sinks else NONE)
    L.check_status()
    scores = torch.einsum("bshd,bthd->bhst", q.double(), k.double().repeat_interleave(Hq // Hkv, 2)) * D ** -0.5
    if causal:
        scores = scores.masked_fill(torch.ones(S, T, dtype=torch.bool, device=DEV).triu(T - S + 1), float("-inf"))
    with_sink = torch.cat([scores, sink.double()[None, :, None, None].expand(B, Hq, S, 1)], -1) if sinks else scores
    want_lse = torch.logsumexp(with_sink, -1)
    weights = (scores - want_lse[..., None]).exp().nan_to_num(0.0)
    # a rounding of the probabilities (2^-9) and one of the result
    assert rel_err(out, torch.einsum("bhst,bthd->bshd", weights, v.double().repeat_interleave(Hq // Hkv, 2))) < 2.0 ** -8
    seen = want_lse.isfinite()
    assert float((lse.double() - want_lse)[seen].abs().max()) < 1e-5 * max(1.0, float(want_lse[seen].abs().max())) and bool((lse[~seen] == float("-inf")).all())


# few tiles, where both halves of a CTA share a row's keys: one key tile, two, an odd number, and the lines up to two tiles an SM; kept first tiles, in the walk of one half or
# of both, beside a window that starts in every place of a tile; documents that end inside a tile, of a few tokens, and padding behind the last
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(1, 100, 2, 1, 64), (1, 256, 3, 3, 128), (2, 640, 4, 2, 64), (1, 1100, 5, 1, 128), (2, 768, 16, 16, 64), (6, 384, 16, 16, 64), (1, 896, 32, 8, 128),
                                          (2, 128, 100, 100, 64)])
@pytest.mark.parametrize("kind,causal", [(kind, True) for kind in ("window", "keep", "keep many", "chunk", "softcap", "gain", "sigmoid", "packed", "packed short", "packed and padded",
                                                                  "window and documents", "sinks and window")] + [(kind, False) for kind in ("window", "chunk", "softcap", "packed")])
def test_flash_variants_of_few_tiles(B, S, Hq, Hkv, D, kind, causal):
    from dew_b200.ops.flash import Variants, flash_fwd
    g = torch.Generator(device=DEV).manual_seed(S + Hq)
    q, k, v = (torch.randn(B, S, h, D, generator=g, device=DEV).bfloat16() for h in (Hq, Hkv, Hkv))
    at = torch.arange(S, device=DEV)
    lengths = torch.tensor([37, 3, 130, 1, 200, 129, 64], device=DEV)
    docs = {"packed": at // 300 + 1, "packed short": torch.repeat_interleave(torch.arange(1, 8, device=DEV), lengths).repeat(S // 564 + 1)[:S] + at // 564 * 7,
            "packed and padded": torch.where(at < S - 90, at // 200 + 1, torch.zeros_like(at)), "window and documents": at // 250 + 1}
    kw = dict(window=dict(window=77), keep=dict(window=70, keep=4), chunk=dict(chunk=96), softcap=dict(softcap=5.0), gain=dict(gain=torch.rand(Hq, generator=g, device=DEV) + 0.5),
              sigmoid=dict(sigmoid=torch.randn(Hq, generator=g, device=DEV)), **{"keep many": dict(window=130, keep=300), "window and documents": dict(window=200),
                                                                                 "sinks and window": dict(window=200, sinks=torch.randn(Hq, generator=g, device=DEV))}).get(kind, {})
    if kind in docs:
        kw["segments"] = docs[kind].to(torch.int32)[None].expand(B, S).contiguous()
    out, lse = flash_fwd(q, k, v, causal, D ** -0.5, need_lse=kind != "sigmoid", var=Variants(**kw))
    L.check_status()
    scores = torch.einsum("bshd,bthd->bhst", q.double(), k.double().repeat_interleave(Hq // Hkv, 2)) * D ** -0.5
    if "gain" in kw:
        scores = scores * kw["gain"].double()[:, None, None]
    if "softcap" in kw:
        scores = kw["softcap"] * torch.tanh(scores / kw["softcap"])
    seen = torch.ones(S, S, dtype=torch.bool, device=DEV)
    if causal:
        seen &= at[None] <= at[:, None]
    if "window" in kw:
        seen &= (at[None] > at[:, None] - kw["window"]) | (at[None] < kw.get("keep", 0))
    if "chunk" in kw:
        seen &= at[None] >= at[:, None] // kw["chunk"] * kw["chunk"]
    if "segments" in kw:
        seen = seen & (kw["segments"][0][None] == kw["segments"][0][:, None])
    if kind == "sigmoid":
        weights = torch.sigmoid(scores + kw["sigmoid"].double()[:, None, None]) * seen
    else:
        scores = scores.masked_fill(~seen, float("-inf"))
        both = torch.cat([scores, kw["sinks"].double()[None, :, None, None].expand(B, Hq, S, 1)], -1) if "sinks" in kw else scores
        want_lse = torch.logsumexp(both, -1)
        weights = (scores - want_lse[..., None]).exp()
        # fp32 sums of fp32 products of bf16 operands; a soft cap's tanh is good to 2^-22 of the cap
        assert float((lse.double() - want_lse).abs().max()) < 1e-5 * max(1.0, float(want_lse.abs().max()))
    # a rounding of the weights (2^-9) and one of the result
    assert rel_err(out, torch.einsum("bhst,bthd->bshd", weights, v.double().repeat_interleave(Hq // Hkv, 2))) < 2.0 ** -8


# more items than CTAs, of neighbouring rows (which start at different key tiles) and of two heads: kept first tiles in front of a window, in the walk of one tile or of both
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(2, 1280, 17, 17, 64), (2, 1152, 24, 4, 128), (1, 2176, 22, 2, 64)])
@pytest.mark.parametrize("kind", ["window", "keep", "keep many", "chunk", "softcap", "sigmoid", "packed", "packed short", "packed and padded", "window and documents"])
def test_flash_variants_of_several_items_a_cta(B, S, Hq, Hkv, D, kind):
    test_flash_variants_of_few_tiles(B, S, Hq, Hkv, D, kind, True)


def test_variants_of_few_tiles_take_no_longer():
    """Sixteen tiles with factors of the heads' scores, one multiplication a score, against the same without (1.07 times; 1.64 with half of a CTA idle)."""
    from dew_b200.ops.flash import NONE, Variants, flash_fwd
    q, k, v = (torch.randn(1, 2048, 1, 128, device=DEV).bfloat16() for _ in range(3))
    took = []
    for var in (NONE, Variants(gain=torch.ones(1, device=DEV))):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            torch.cuda._sleep(1000000)                           # (the launches are enqueued by the time the first one starts)
            a.record()
            for _ in range(10):
                flash_fwd(q, k, v, True, 128 ** -0.5, need_lse=False, var=var)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        took.append(sorted(times)[3])
    assert took[1] < 1.35 * took[0], took


@pytest.mark.parametrize("D", [64, 128])
def test_flash_backward_of_saturated_caps(D):
    """Scores of seven to nine caps, whose capped values have derivatives of 1e-6 and less: these hold to fp32 relative to themselves, not to 1; then a rounding of the scores'
    gradients to bf16 (2^-9), and one of the results."""
    from dew_b200.ops.flash import Variants, flash_bwd, flash_fwd
    g = torch.Generator(device=DEV).manual_seed(D)
    S = 256
    q, k = torch.zeros(1, S, 2, D, device=DEV), torch.zeros(1, S, 1, D, device=DEV)
    q[..., 0] = 8
    k[..., 0] = (torch.randint(0, 2, (1, S, 1), generator=g, device=DEV) * 2 - 1) * (7 + 2 * torch.rand(1, S, 1, generator=g, device=DEV)) / 8 * D ** 0.5
    q, k = q.bfloat16(), k.bfloat16()
    v, do = (torch.randn(1, S, h, D, generator=g, device=DEV).bfloat16() for h in (1, 2))
    var = Variants(softcap=1.0)
    out, lse = flash_fwd(q, k, v, True, D ** -0.5, var=var)
    _, dk, _ = flash_bwd(do, q, k, v, out, lse, True, D ** -0.5, var=var)
    L.check_status()
    leaves = [x.double().requires_grad_() for x in (q, k, v)]
    scores = torch.tanh(torch.einsum("bshd,bthd->bhst", leaves[0], leaves[1].repeat_interleave(2, 2)) * D ** -0.5)
    scores = scores.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=DEV).tril(), float("-inf"))
    want, = torch.autograd.grad(torch.einsum("bhst,bthd->bshd", torch.softmax(scores, -1), leaves[2].repeat_interleave(2, 2)), leaves[1:2], do.double())
    # (of the keys' gradient: the queries' is a sum over keys that nearly cancels where the derivatives are alike)
    assert rel_err(dk[..., 0], want[..., 0]) < 2.0 ** -7
