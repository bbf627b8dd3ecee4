"""The work this framework's speed is measured on.

Eight kinds of work, each through the entry point a user's program calls: the sequence operations of a training step (attention, gated delta rule, Mamba-2 state
space) with all their gradients, a mixture-of-experts feed-forward, whole training steps of decoders and of a diffusion transformer, a denoising call as a sampler
makes it, and a served decoder's prompts and generation steps.  ``listed`` are the configurations of this repository (its benchmark, recipes, examples and tests)
cut to a few layers; ``draw`` spreads the same kinds over their ranges.

``exact`` restates every kind in 64 bits with plain torch.
"""
import math

import torch
import torch.nn.functional as F

import dew_b200  # noqa: F401  (the package before its parts)
from dew_b200 import ops
from dew_b200.models import CausalTransformer, SimpleDiT
from dew_b200.models.causal_transformer import Mixture
from dew_b200.nn.kv_cache import KVCache
from dew_b200.nn.moe import SparseMLP
from dew_b200.objectives.base import Step
from dew_b200.objectives.lm import LMObjective
from dew_b200.ops import scan
from dew_b200.sampling.text import RowBatch

DEV = "cuda"
BF16 = torch.bfloat16
PAGE = 64


def listed():
    return [
        # one attention layer of the dense 8 B configuration on a microbatch of two sequences, forward and backward
        dict(name="attention_train", kind="attention", batch=2, seq=4096, heads=32, kv=8, dim=128, causal=True),
        # a layer of 64-wide heads on short rows, as fine-tuning has them
        dict(name="attention_short", kind="attention", batch=8, seq=512, heads=32, kv=8, dim=64, causal=True),
        # the gated delta rule of a layer of the hybrid configuration on a microbatch of two sequences
        dict(name="delta_train", kind="delta", batch=2, seq=8192, heads=16, key_heads=16),
        # the state space scan of a Mamba-2 layer of width 2048 (64 heads of 64, state 128, one group)
        dict(name="ssd_train", kind="ssd", batch=2, seq=4096, heads=64, groups=1),
        # a feed-forward of the mixture-of-experts configuration (block-scaled fp8 experts) on two sequences
        dict(name="experts_train", kind="experts", tokens=8192, width=2048, experts=64, top_k=6, ff=1408, shared=2816, fp8=True),
        # the byte-level decoder that the examples train: launches and host work
        dict(name="lm_bytes_train", kind="lm", batch=16, seq=128, width=128, heads=2, kv=2, dim=64, ff=256, layers=4, vocab=256),
        # a decoder of width 2048 on a microbatch of two sequences
        dict(name="lm_train", kind="lm", batch=2, seq=4096, width=2048, heads=16, kv=4, dim=128, ff=5632, layers=4, vocab=32768),
        # a class-conditional diffusion transformer of width 768 on 64 images of 256 patches
        dict(name="dit_train", kind="dit", train=True, batch=64, grid=16, patch=2, channels=4, width=768, heads=12, layers=4),
        # one denoising call on four images of the diffusion recipe's size, as every step of a sampler makes it
        dict(name="dit_denoise", kind="dit", train=False, batch=4, grid=16, patch=4, channels=3, width=384, heads=6, layers=4),
        # sixteen prompts of 128 to 2048 tokens entering the cache of two layers of the dense 8 B configuration
        dict(name="prompts", kind="prompts", rows=16, shortest=128, longest=2048, width=4096, heads=32, kv=8, dim=128, ff=14336, layers=2, vocab=32768),
        # one generation step of 128 requests in flight, prompts of 128 to 2048 tokens behind them
        dict(name="step_many", kind="step", rows=128, shortest=128, longest=2048, width=4096, heads=32, kv=8, dim=128, ff=14336, layers=2, vocab=32768),
        # one generation step of a single request to a small decoder
        dict(name="step_one", kind="step", rows=1, shortest=512, longest=512, width=1024, heads=8, kv=4, dim=128, ff=2816, layers=8, vocab=32000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "delta", "ssd", "experts", "lm", "dit", "prompts", "step"])
    if kind == "attention":
        dim, kv, group = rng.choice([64, 128]), rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4])
        causal = rng.random() < 0.8
        seq = _log(rng, 128, 12288)
        if rng.random() < 0.8:
            seq = max(128, seq // 128 * 128)
        return dict(kind=kind, batch=rng.randint(1, max(1, min(8, 12288 // seq))), seq=seq, heads=kv * group, kv=kv, dim=dim, causal=causal)
    if kind == "delta":
        key_heads, rep = rng.choice([1, 2, 4, 8, 16]), rng.choice([1, 1, 2])
        seq = _log(rng, 64, 8192)
        return dict(kind=kind, batch=rng.randint(1, max(1, min(4, 16384 // seq))), seq=seq, heads=min(16, key_heads * rep), key_heads=key_heads)
    if kind == "ssd":
        groups, per = rng.choice([1, 1, 2, 4]), rng.choice([2, 8, 16])
        seq = _log(rng, 64, 4096)
        return dict(kind=kind, batch=rng.randint(1, max(1, min(4, 8192 // seq))), seq=seq, heads=groups * per, groups=groups)
    if kind == "experts":
        return dict(kind=kind, tokens=_log(rng, 64, 8192), width=256 * rng.randint(2, 8), experts=rng.choice([8, 16, 64]), top_k=rng.randint(1, 6),
                    ff=128 * rng.randint(2, 11), shared=rng.choice([0, 1024]), fp8=rng.random() < 0.5)
    if kind == "lm":
        dim, kv = rng.choice([64, 128]), rng.choice([1, 2, 4])
        heads = kv * rng.choice([1, 2, 4])
        seq = _log(rng, 64, 4096)
        if rng.random() < 0.7:
            seq = max(128, seq // 128 * 128)
        return dict(kind=kind, batch=rng.randint(1, max(1, min(16, 8192 // seq))), seq=seq, width=heads * dim, heads=heads, kv=kv, dim=dim, ff=128 * rng.randint(1, 24),
                    layers=rng.randint(1, 4), vocab=rng.choice([256, 1000, 8192, 32768]))
    if kind == "dit":
        heads = rng.randint(2, 12)
        return dict(kind=kind, train=rng.random() < 0.6, batch=_log(rng, 1, 64), grid=rng.choice([8, 12, 16]), patch=rng.choice([2, 4]), channels=rng.choice([3, 4]),
                    width=64 * heads, heads=heads, layers=rng.randint(1, 4))
    kv, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4])
    longest = _log(rng, 64, 2048)
    return dict(kind=kind, rows=_log(rng, 1, 16 if kind == "prompts" else 128), shortest=rng.randint(16, longest), longest=longest, width=128 * rng.randint(4, 24), heads=kv * group,
                kv=kv, dim=128, ff=256 * rng.randint(2, 40), layers=rng.randint(1, 4), vocab=rng.choice([1000, 8192, 32768]))


# --------------------------------------------------------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=DEV) * std).to(dtype)


def _attention_inputs(case, seed):
    g = _gen(seed)
    B, S, H, G, D = (case[k] for k in ("batch", "seq", "heads", "kv", "dim"))
    return dict(q=_normal(g, B, S, H, D), k=_normal(g, B, S, G, D), v=_normal(g, B, S, G, D), do=_normal(g, B, S, H, D))


def _delta_inputs(case, seed):
    """What a layer hands the recurrence: unit q and k, the logarithm of a decay per head and token, write strengths."""
    g = _gen(seed)
    B, T, H, K = (case[k] for k in ("batch", "seq", "heads", "key_heads"))
    rate = torch.rand(H, generator=g, device=DEV) * 15 + 1
    dt = torch.exp(torch.rand(H, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
    a = torch.randn(B, T, H, generator=g, device=DEV) * 0.5 + torch.log(torch.expm1(dt))
    return dict(q=F.normalize(_normal(g, B, T, K, 128, dtype=torch.float32), dim=-1).to(BF16), k=F.normalize(_normal(g, B, T, K, 128, dtype=torch.float32), dim=-1).to(BF16),
                v=_normal(g, B, T, H, 128), g=-rate * F.softplus(a), beta=torch.sigmoid(torch.randn(B, T, H, generator=g, device=DEV)), do=_normal(g, B, T, H, 128))


def _ssd_inputs(case, seed):
    g = _gen(seed)
    B, T, H, G = (case[k] for k in ("batch", "seq", "heads", "groups"))
    bias = torch.exp(torch.rand(H, generator=g, device=DEV) * math.log(100.0) + math.log(1e-3))
    dt = F.softplus(torch.randn(B, T, H, generator=g, device=DEV) * 0.5 + torch.log(torch.expm1(bias)))
    return dict(x=_normal(g, B, T, H, 64), dt=dt, A=-(torch.rand(H, generator=g, device=DEV) * 15 + 1), Bm=_normal(g, B, T, G, 128, std=0.5), Cm=_normal(g, B, T, G, 128, std=0.5),
                D=torch.ones(H, device=DEV) + 0.1 * torch.randn(H, generator=g, device=DEV), dy=_normal(g, B, T, H, 64))


def _expert_weights(case, seed):
    g = _gen(seed)
    d, E, f, s = (case[k] for k in ("width", "experts", "ff", "shared"))
    w = {"router.weight": _normal(g, E, d, std=d ** -0.5, dtype=torch.float32), "experts.gate_up": _normal(g, E, 2 * f, d, std=0.02), "experts.down": _normal(g, E, d, f, std=0.02)}
    if s:
        w.update({"shared.gate_up_proj.weight": _normal(g, 2 * s, d, std=0.02), "shared.down_proj.weight": _normal(g, d, s, std=0.02)})
    return w


def _expert_inputs(case, seed):
    g = _gen(seed + 7)
    return _normal(g, 1, case["tokens"], case["width"]), _normal(g, 1, case["tokens"], case["width"])


def _decoder_weights(case, seed):
    g = _gen(seed)
    d, H, G, D, f, V = (case[k] for k in ("width", "heads", "kv", "dim", "ff", "vocab"))
    near_one = lambda n: (1 + 0.1 * torch.randn(n, generator=g, device=DEV)).to(BF16)
    w = {"embed.weight": _normal(g, V, d, std=0.5)}
    for i in range(case["layers"]):
        w.update({f"layers.{i}.input_norm.weight": near_one(d), f"layers.{i}.mixer.qkv_proj.weight": _normal(g, (H + 2 * G) * D, d, std=d ** -0.5),
                  f"layers.{i}.mixer.o_proj.weight": _normal(g, d, H * D, std=(H * D) ** -0.5), f"layers.{i}.post_norm.weight": near_one(d),
                  f"layers.{i}.mlp.gate_up_proj.weight": _normal(g, 2 * f, d, std=d ** -0.5), f"layers.{i}.mlp.down_proj.weight": _normal(g, d, f, std=f ** -0.5)})
    w.update({"final_norm.weight": near_one(d), "head.weight": _normal(g, V, d, std=d ** -0.5)})
    return w


def _decoder(case, seed, length):
    model = CausalTransformer(vocab_size=case["vocab"], emb_features=case["width"], num_layers=case["layers"], num_heads=case["heads"], num_kv_heads=case["kv"], head_dim=case["dim"],
                              mlp_features=case["ff"], max_seq_len=length, qk_norm=False, tie_embeddings=False, norm_eps=1e-5, dtype=BF16, device=DEV)
    model.load_state_dict(_decoder_weights(case, seed))
    return model


def _token_rows(case, seed):
    return torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=_gen(seed + 7), device=DEV)


def _prompt_rows(case, seed):
    """Token rows and their lengths, between the shortest and the longest."""
    r = torch.Generator().manual_seed(seed + 3)
    lengths = torch.randint(case["shortest"], case["longest"] + 1, (case["rows"],), generator=r)
    lengths[0] = case["longest"]
    tokens = torch.randint(0, case["vocab"], (case["rows"], case["longest"]), generator=_gen(seed + 7), device=DEV)
    return tokens, lengths.to(DEV)


CLASSES = 1000


def _dit_weights(case, seed):
    """Weights of every layer of full size: those that training starts at zero as well."""
    g = _gen(seed)
    d, c = case["width"], case["patch"] ** 2 * case["channels"]
    lin = lambda name, n_out, n_in: {f"{name}.weight": _normal(g, n_out, n_in, std=n_in ** -0.5), f"{name}.bias": _normal(g, n_out, std=0.02)}
    w = {**lin("embed.proj", d, c), **lin("conditioning.t1", d, d), **lin("conditioning.t2", d, d), "conditioning.classes.weight": _normal(g, CLASSES + 1, d, std=0.5)}
    for i in range(case["layers"]):
        p = f"blocks.{i}."
        w.update({**lin(p + "attn.qkv_proj", 3 * d, d), **lin(p + "attn.o_proj", d, d), **lin(p + "mlp.fc1", 4 * d, d), **lin(p + "mlp.fc2", d, 4 * d)})
        w.update({p + "ada_proj.weight": _normal(g, 6 * d, d, std=0.5 * d ** -0.5), p + "ada_proj.bias": _normal(g, 6 * d, std=0.02)})
    w.update({"output.ada_proj.weight": _normal(g, 2 * d, d, std=0.5 * d ** -0.5), "output.ada_proj.bias": _normal(g, 2 * d, std=0.02), **lin("output.out", c, d)})
    return w


def _dit_inputs(case, seed):
    g = _gen(seed + 7)
    side = case["grid"] * case["patch"]
    images = lambda: torch.randn(case["batch"], side, side, case["channels"], generator=g, device=DEV)
    return images(), torch.rand(case["batch"], generator=g, device=DEV), torch.randint(0, CLASSES, (case["batch"],), generator=g, device=DEV), images()


# --------------------------------------------------------------------------------------------------------------- the passes


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind in ("attention", "delta", "ssd"):
        t = {"attention": _attention_inputs, "delta": _delta_inputs, "ssd": _ssd_inputs}[kind](case, seed)
        leaves = {"attention": ("q", "k", "v"), "delta": ("q", "k", "v", "g", "beta"), "ssd": ("x", "dt", "A", "Bm", "Cm", "D")}[kind]
        s.update({n: x.requires_grad_() if n in leaves else x for n, x in t.items()}, leaves=leaves)
    elif kind == "experts":
        mix = Mixture(experts=case["experts"], top_k=case["top_k"], expert_features=case["ff"], shared_features=case["shared"], fp8=case["fp8"])
        s["model"] = SparseMLP(case["width"], mix, case["ff"], dtype=BF16, device=DEV)
        s["model"].load_state_dict(_expert_weights(case, seed))
        s["x"], s["dy"] = _expert_inputs(case, seed)
        s["x"].requires_grad_()
    elif kind == "lm":
        s["model"] = _decoder(case, seed, case["seq"])
        s["objective"] = LMObjective(s["model"], case["seq"])
        s["batch"] = {"tokens": _token_rows(case, seed)}
    elif kind == "dit":
        s["model"] = SimpleDiT(patch_size=case["patch"], emb_features=case["width"], num_layers=case["layers"], num_heads=case["heads"], input_channels=case["channels"],
                               output_channels=case["channels"], num_classes=CLASSES, dtype=BF16, device=DEV)
        s["model"].load_state_dict(_dit_weights(case, seed))
        s["x"], s["t"], s["labels"], s["target"] = _dit_inputs(case, seed)
    else:
        model = _decoder(case, seed, case["longest"] + 256).eval()
        s["tokens"], s["lengths"] = _prompt_rows(case, seed)
        # room for 256 more tokens a row, as a request that generates needs
        s["rows"] = RowBatch(model, case["rows"], case["longest"] + 256, kv_cache=KVCache(page_size=PAGE))
        if kind == "step":
            s["rows"].prefill(s["tokens"], s["lengths"])
            s["next"] = torch.randint(0, case["vocab"], (case["rows"], 1), generator=_gen(seed + 9), device=DEV)
            s["positions"] = s["lengths"][:, None].clone()
    return s


def _parameter_gradients(s):
    out = {n: p.grad for n, p in s["model"].named_parameters()}
    s["model"].zero_grad(set_to_none=True)
    return out


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "attention":
        o = ops.attention(s["q"], s["k"], s["v"], causal=case["causal"])
        return [o, *torch.autograd.grad(o, [s[n] for n in s["leaves"]], s["do"])]
    if kind == "delta":
        o, last = scan.chunk_gated_delta_rule(s["q"], s["k"], s["v"], s["g"], s["beta"])
        return [o, last, *torch.autograd.grad(o, [s[n] for n in s["leaves"]], s["do"])]
    if kind == "ssd":
        y, last = scan.ssd(s["x"], s["dt"], s["A"], s["Bm"], s["Cm"], s["D"])
        return [y, last, *torch.autograd.grad(y, [s[n] for n in s["leaves"]], s["dy"])]
    if kind == "experts":
        y = s["model"](s["x"])
        y.backward(s["dy"])
        dx, s["x"].grad = s["x"].grad, None
        return dict(y=y, dx=dx, **_parameter_gradients(s))
    if kind == "lm":
        loss = s["objective"].loss(None, s["batch"], Step(train=True, device=DEV))[0].value()
        loss.backward()
        return dict(loss=loss, **_parameter_gradients(s))
    if kind == "dit":
        conditions = {"label": s["labels"]}
        if not case["train"]:
            with torch.no_grad():
                return s["model"](s["x"], s["t"], conditions)
        out = s["model"](s["x"], s["t"], conditions, train=True)
        (0.5 * (out - s["target"]) ** 2).mean().backward()
        return dict(out=out, **_parameter_gradients(s))
    if kind == "prompts":
        logits, store = s["rows"].prefill(s["tokens"], s["lengths"]), s["rows"].store
        return dict(logits=logits, keys=store.k[:, : store.pages], values=store.v[:, : store.pages])      # (behind the last page: what nobody reads)
    return s["rows"].forward(s["next"], s["positions"])[:, 0]


# --------------------------------------------------------------------------------------------------------------- what a pass cannot do without


def _pairs(case):
    """Visible (query, key) pairs of a row."""
    S = case["seq"]
    return S * (S + 1) / 2 if case["causal"] else S * S


def _decoder_sizes(case):
    d, H, G, D, f = (case[k] for k in ("width", "heads", "kv", "dim", "ff"))
    return case["layers"] * ((H + 2 * G) * D * d + H * D * d + 3 * f * d), case["vocab"] * d


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, S, H, G, D = (case[k] for k in ("batch", "seq", "heads", "kv", "dim"))
        return {"bytes": 2 * B * S * D * (4 * H + 4 * G), "flops": 14 * B * H * D * _pairs(case)}
    if kind == "delta":
        B, T, H, K = (case[k] for k in ("batch", "seq", "heads", "key_heads"))
        # per token and head: reading the state, writing it, and the products inside a chunk of 64, three times (forward, and two of them backward)
        return {"bytes": B * T * (128 * 2 * (4 * K + 4 * H) + 4 * 4 * H) + 4 * B * H * 128 * 128, "flops": 3 * B * T * H * (2 * 2 * 128 * 128 + 2 * 128 * 64 * 3)}
    if kind == "ssd":
        B, T, H, G = (case[k] for k in ("batch", "seq", "heads", "groups"))
        return {"bytes": 2 * B * T * (64 * H * 4 + 128 * G * 4) + 4 * B * T * H * 2 + 4 * B * H * 64 * 128, "flops": 3 * B * T * H * (2 * 2 * 64 * 128 + 2 * 64 * 64)}
    if kind == "experts":
        T, d, E, k, f, s = (case[n] for n in ("tokens", "width", "experts", "top_k", "ff", "shared"))
        weights = min(E, T * k) * 3 * f * d + 3 * s * d
        return {"bytes": 2 * 4 * T * d + 2 * 2 * weights + 8 * E * d, "flops": 6 * T * d * (3 * k * f + 3 * s + E)}
    if kind == "lm":
        T, S = case["batch"] * case["seq"], case["seq"]
        layers, head = _decoder_sizes(case)
        return {"bytes": 2 * 2 * (layers + 2 * head) + 8 * T, "flops": 6 * T * (layers + head) + 14 * case["layers"] * case["heads"] * case["dim"] * T * (S + 1) / 2}
    if kind == "dit":
        d, n, L, B, c = case["width"], case["grid"] ** 2, case["layers"], case["batch"], case["patch"] ** 2 * case["channels"]
        weights = L * 18 * d * d + 4 * d * d + 2 * c * d
        flops = 2 * B * (n * (12 * L * d * d + 2 * c * d) + 6 * L * d * d + 4 * d * d) + 4 * B * L * n * n * d
        return {"bytes": 2 * weights * (2 if case["train"] else 1) + 4 * B * n * c * (3 if case["train"] else 2), "flops": flops * (3 if case["train"] else 1)}
    layers, head = _decoder_sizes(case)
    mean = (case["shortest"] + case["longest"]) / 2
    R, kv = case["rows"], 2 * 2 * case["layers"] * case["kv"] * case["dim"]
    if kind == "prompts":
        return {"bytes": 2 * (layers + head) + kv * R * mean + 2 * R * case["vocab"], "flops": 2 * R * (mean * layers + head) + 2 * case["layers"] * case["heads"] * case["dim"] * R * mean * mean}
    return {"bytes": 2 * (layers + head) + kv * R * mean + 2 * R * case["vocab"], "flops": 2 * R * (layers + head) + 4 * case["layers"] * case["heads"] * case["dim"] * R * mean}


def tolerance(case):
    """bf16 operands and results with fp32 sums: the distance between this path and the same path with its sums in another order is a few parts in a thousand
    for one operation and up to twice that through a stack of layers."""
    return {"rel": {"attention": 0.01, "delta": 0.02, "ssd": 0.02, "experts": 0.02, "lm": 0.03, "dit": 0.03, "prompts": 0.02, "step": 0.02}[case["kind"]]}


# --------------------------------------------------------------------------------------------------------------- the same in 64 bits


def _attend64(q, k, v, causal):
    """One row, one head: ``q, k, v [S, D]``."""
    s = (q @ k.t()) * q.shape[-1] ** -0.5
    if causal:
        s = s.masked_fill(~torch.ones(s.shape, dtype=torch.bool, device=s.device).tril(), float("-inf"))
    return torch.softmax(s, -1) @ v


def _exact_attention(case, seed):
    t = _attention_inputs(case, seed)
    rep = case["heads"] // case["kv"]
    out, dq, dk, dv = (torch.zeros(t[n].shape, dtype=torch.float64, device=DEV) for n in ("q", "q", "k", "v"))
    for b in range(case["batch"]):
        for h in range(case["heads"]):
            q, k, v = (x.double().requires_grad_() for x in (t["q"][b, :, h], t["k"][b, :, h // rep], t["v"][b, :, h // rep]))
            o = _attend64(q, k, v, case["causal"])
            gq, gk, gv = torch.autograd.grad(o, (q, k, v), t["do"][b, :, h].double())
            out[b, :, h], dq[b, :, h] = o.detach(), gq
            dk[b, :, h // rep] += gk
            dv[b, :, h // rep] += gv
    return [out, dq, dk, dv]


def _chunks64(x, n):
    """``[B, T, H, ...] -> [B, H, chunks, n, ...]`` with zeros behind the last token."""
    x = x.transpose(1, 2)
    pad = -x.shape[2] % n
    if pad:
        x = torch.cat([x, x.new_zeros(*x.shape[:2], pad, *x.shape[3:])], 2)
    return x.reshape(*x.shape[:2], -1, n, *x.shape[3:])


def _decays64(g):
    """``exp`` of the sums of ``g`` between two tokens of a chunk, from the chunk's start, and to its end."""
    c = g.cumsum(-1)
    low = torch.ones(g.shape[-1], g.shape[-1], dtype=torch.bool, device=g.device).tril()
    between = (c[..., :, None] - c[..., None, :]).masked_fill(~low, float("-inf")).exp()
    return between, c.exp(), (c[..., -1:] - c).exp()


def _exact_delta(case, seed):
    t = _delta_inputs(case, seed)
    leaves = [t[n].double().requires_grad_() for n in ("q", "k", "v", "g", "beta")]
    rep, T = case["heads"] // case["key_heads"], case["seq"]
    q, k, v, g, beta = leaves
    q, k = (_chunks64(x.repeat_interleave(rep, 2), 64) for x in (q, k))
    v, g, beta = (_chunks64(x, 64) for x in (v, g, beta))
    between, start, end = _decays64(g)
    eye = torch.eye(64, dtype=torch.float64, device=DEV)
    mixed = (beta[..., None] * (k @ k.transpose(-1, -2)) * between).tril(-1)
    u, w = (torch.linalg.solve_triangular(eye + mixed, x, upper=False) for x in (beta[..., None] * v, (beta * start)[..., None] * k))
    scores = (q @ k.transpose(-1, -2)) * between * 128 ** -0.5
    S, out = torch.zeros(case["batch"], case["heads"], 128, 128, dtype=torch.float64, device=DEV), []
    for c in range(v.shape[2]):
        new = u[:, :, c] - w[:, :, c] @ S
        out.append(128 ** -0.5 * start[:, :, c, :, None] * (q[:, :, c] @ S) + scores[:, :, c] @ new)
        S = start[:, :, c, -1, None, None] * S + (end[:, :, c, :, None] * k[:, :, c]).transpose(-1, -2) @ new
    o = torch.cat(out, 2)[:, :, :T].transpose(1, 2)
    grads = torch.autograd.grad(o, leaves, t["do"].double())
    return [o.detach(), S.detach(), *grads]


def _exact_ssd(case, seed):
    t = _ssd_inputs(case, seed)
    leaves = [t[n].double().requires_grad_() for n in ("x", "dt", "A", "Bm", "Cm", "D")]
    x, dt, A, Bm, Cm, D = leaves
    rep, T = case["heads"] // case["groups"], case["seq"]
    xs, gs = _chunks64(x * dt[..., None], 64), _chunks64(dt * A, 64)
    bs, cs = (_chunks64(m.repeat_interleave(rep, 2), 64) for m in (Bm, Cm))
    S, out = torch.zeros(case["batch"], case["heads"], 64, 128, dtype=torch.float64, device=DEV), []
    for c in range(xs.shape[2]):
        between, start, end = _decays64(gs[:, :, c])
        b, m, v = bs[:, :, c], cs[:, :, c], xs[:, :, c]
        out.append(((m @ b.transpose(-1, -2)) * between) @ v + start[..., None] * (m @ S.transpose(-1, -2)))
        S = start[..., -1, None, None] * S + (v * end[..., None]).transpose(-1, -2) @ b
    y = torch.cat(out, 2)[:, :, :T].transpose(1, 2) + x * D[:, None]
    grads = torch.autograd.grad(y, leaves, t["dy"].double())
    return [y.detach(), S.detach(), *grads]


def _glu64(x, gate_up, down):
    a, b = (x @ gate_up.t()).chunk(2, -1)
    return (F.silu(a) * b) @ down.t()


def _exact_experts(case, seed):
    w = {n: x.double().requires_grad_() for n, x in _expert_weights(case, seed).items()}
    x, dy = (a.double()[0] for a in _expert_inputs(case, seed))
    x.requires_grad_()
    p = torch.softmax(x @ w["router.weight"].t(), -1)
    top, ids = p.topk(case["top_k"], -1)
    top = top / top.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(case["experts"]):
        rows, place = (ids == e).nonzero(as_tuple=True)
        y = y.index_add(0, rows, top[rows, place, None] * _glu64(x[rows], w["experts.gate_up"][e], w["experts.down"][e]))
    if case["shared"]:
        y = y + _glu64(x, w["shared.gate_up_proj.weight"], w["shared.down_proj.weight"])
    names = list(w)
    grads = torch.autograd.grad(y, [x] + [w[n] for n in names], dy)
    return dict(y=y.detach()[None], dx=grads[0][None], **dict(zip(names, grads[1:])))


def _rms64(x, weight):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * weight


def _rotate64(x):
    """``[S, H, D]`` turned by its positions, halves against each other."""
    S, _, D = x.shape
    angle = torch.outer(torch.arange(S, dtype=torch.float64, device=DEV), 10000.0 ** (-torch.arange(0, D, 2, dtype=torch.float64, device=DEV) / D))
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., : D // 2], x[..., D // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _decoder64(case, w, ids, kept=None):
    """One row of token ids through the decoder; the normed hidden states.  ``kept`` receives every layer's keys and values."""
    H, G, D = case["heads"], case["kv"], case["dim"]
    h = F.embedding(ids, w["embed.weight"])
    for i in range(case["layers"]):
        p = f"layers.{i}."
        qkv = (_rms64(h, w[p + "input_norm.weight"]) @ w[p + "mixer.qkv_proj.weight"].t()).view(-1, H + 2 * G, D)
        qk, v = _rotate64(qkv[:, : H + G]), qkv[:, H + G:]
        if kept is not None:
            kept.append((qk[:, H:], v))
        o = torch.stack([_attend64(qk[:, j], qk[:, H + j // (H // G)], v[:, j // (H // G)], True) for j in range(H)], 1)
        h = h + o.reshape(-1, H * D) @ w[p + "mixer.o_proj.weight"].t()
        h = h + _glu64(_rms64(h, w[p + "post_norm.weight"]), w[p + "mlp.gate_up_proj.weight"], w[p + "mlp.down_proj.weight"])
    return _rms64(h, w["final_norm.weight"])


def _exact_lm(case, seed):
    w = {n: x.double().requires_grad_() for n, x in _decoder_weights(case, seed).items()}
    total, names = 0.0, list(w)
    grads = [torch.zeros_like(w[n]) for n in names]
    tokens = _token_rows(case, seed)
    for row in tokens:                       # a row at a time
        loss = F.cross_entropy(_decoder64(case, w, row[:-1]) @ w["head.weight"].t(), row[1:], reduction="sum") / (tokens.shape[0] * case["seq"])
        for a, b in zip(grads, torch.autograd.grad(loss, [w[n] for n in names])):
            a += b
        total += float(loss.detach())
    return dict(loss=torch.tensor(total, dtype=torch.float64, device=DEV), **dict(zip(names, grads)))


def _exact_served(case, seed):
    w = {n: x.double() for n, x in _decoder_weights(case, seed).items()}
    tokens, lengths = _prompt_rows(case, seed)
    if case["kind"] == "step":
        more = torch.randint(0, case["vocab"], (case["rows"], 1), generator=_gen(seed + 9), device=DEV)
        return torch.stack([_decoder64(case, w, torch.cat([tokens[r, :n], more[r]]))[-1] @ w["head.weight"].t() for r, n in enumerate(lengths.tolist())])
    room = -(-(case["longest"] + 256) // PAGE) * PAGE
    keys, values = (torch.zeros(case["layers"], case["rows"], room, case["kv"], case["dim"], dtype=torch.float64, device=DEV) for _ in range(2))
    out = []
    for r, n in enumerate(lengths.tolist()):
        kept = []
        out.append(_decoder64(case, w, tokens[r, :n], kept)[-1] @ w["head.weight"].t())
        for i, (k, v) in enumerate(kept):
            keys[i, r, :n], values[i, r, :n] = k, v
    pages = lambda t: t.reshape(case["layers"], -1, PAGE, case["kv"], case["dim"])
    return dict(logits=torch.stack(out), keys=pages(keys), values=pages(values))


def _dit64(case, w, x, t, labels):
    d, n, p, H, B = case["width"], case["grid"], case["patch"], case["heads"], x.shape[0]
    lin = lambda name, a: a @ w[name + ".weight"].t() + w[name + ".bias"]
    norm = lambda a: (a - a.mean(-1, keepdim=True)) * torch.rsqrt(a.var(-1, unbiased=False, keepdim=True) + 1e-6)
    change = lambda a, shift, scale: norm(a) * (1 + scale[:, None]) + shift[:, None]
    axis = torch.outer(torch.arange(n, dtype=torch.float64, device=DEV), 10000.0 ** (-torch.arange(d // 4, dtype=torch.float64, device=DEV) / (d // 4)))
    axis = torch.cat([axis.sin(), axis.cos()], 1)
    place = torch.cat([axis[:, None].expand(n, n, -1), axis[None].expand(n, n, -1)], -1).reshape(n * n, d)
    patches = x.double().reshape(B, n, p, n, p, -1).permute(0, 1, 3, 2, 4, 5).reshape(B, n * n, -1)
    h = lin("embed.proj", patches) + place
    angle = t.double()[:, None] * 16.0 * torch.exp(-math.log(10000.0) * torch.arange(d // 2, dtype=torch.float64, device=DEV) / (d // 2))
    c = lin("conditioning.t2", F.silu(lin("conditioning.t1", torch.cat([angle.cos(), angle.sin()], -1)))) + w["conditioning.classes.weight"][labels]
    for i in range(case["layers"]):
        b = f"blocks.{i}."
        s1, k1, g1, s2, k2, g2 = lin(b + "ada_proj", F.silu(c)).chunk(6, -1)
        q, k, v = lin(b + "attn.qkv_proj", change(h, s1, k1)).view(B, n * n, 3, H, d // H).permute(2, 0, 3, 1, 4)
        o = torch.softmax(q @ k.transpose(-1, -2) * (d // H) ** -0.5, -1) @ v
        h = h + g1[:, None] * lin(b + "attn.o_proj", o.transpose(1, 2).reshape(B, n * n, d))
        h = h + g2[:, None] * lin(b + "mlp.fc2", F.gelu(lin(b + "mlp.fc1", change(h, s2, k2)), approximate="tanh"))
    shift, scale = lin("output.ada_proj", F.silu(c)).chunk(2, -1)
    y = lin("output.out", change(h, shift, scale))
    return y.reshape(B, n, n, p, p, -1).permute(0, 1, 3, 2, 4, 5).reshape(x.shape)


def _exact_dit(case, seed):
    x, t, labels, target = _dit_inputs(case, seed)
    w = {n: a.double() for n, a in _dit_weights(case, seed).items()}
    if not case["train"]:
        return _dit64(case, w, x, t, labels)
    names = list(w)
    for a in w.values():
        a.requires_grad_()
    grads, outs = [torch.zeros_like(w[n]) for n in names], []
    for i in range(0, case["batch"], 16):    # sixteen images at a time
        sl = slice(i, i + 16)
        out = _dit64(case, w, x[sl], t[sl], labels[sl])
        for a, b in zip(grads, torch.autograd.grad((0.5 * (out - target[sl].double()) ** 2).sum() / target.numel(), [w[n] for n in names])):
            a += b
        outs.append(out.detach())
    return dict(out=torch.cat(outs), **dict(zip(names, grads)))


def exact(case, seed):
    return {"attention": _exact_attention, "delta": _exact_delta, "ssd": _exact_ssd, "experts": _exact_experts, "lm": _exact_lm, "dit": _exact_dit,
            "prompts": _exact_served, "step": _exact_served}[case["kind"]](case, seed)
