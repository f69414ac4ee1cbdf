"""The work a user of this framework has it do, as cases that can be timed: sizes, inputs, one pass, its result.

Kinds of pass (``case["kind"]``), each through the entry point that a program calls:

``prefill``   api.vq_attention_prefill on rotated queries and keys: codes, aggregates, fused attention
``layer``     attn_vq.dispatch_attn_impl on raw q / k / v of one attention layer and an empty cache (what the module's
              forward does for a prompt): rotations, codes, aggregates, attention, cache state
``step``      api.vq_attention_decode: one token per sequence over a window cache and far aggregates
``generate``  attn_vq.dispatch_attn_impl once per token on a filled cache: 128 tokens, so exactly one block leaves the window
``dropin``    fused_vq_attn.vq_attn_forward on the arguments of the interface it mirrors (sorted prefix sums and row indexes)

Distributions: q, k, v ~ N(0, 1), codebook entries ~ N(0, D^-1/2) as in the benchmark's workloads; codes of real keys, so
that counts and value sums are those of a real sequence.
"""
from __future__ import annotations

import math

import torch

from vqtree_b200 import api, attn_vq, fused_vq_attn

BLOCK = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # ---- the smallest calls: launches and host work count
        # the attention module's self-test shape: two heads of 64, fp16, 511 tokens, one codebook of 128
        dict(name="layer_511_fp16", kind="layer", dtype="fp16", B=1, Hq=2, Hkv=2, D=64, L=511, W=256, M=1, K=128),
        # four chat prompts shorter than the window: the short-sequence path, nothing is quantised
        dict(name="layer_300_short", kind="layer", dtype="bf16", B=4, Hq=32, Hkv=8, D=128, L=300, W=1024, M=4, K=256),
        # the naive path's full-precision shape: eight heads of 64, 1024 tokens, window 128
        dict(name="prefill_1k_fp32", kind="prefill", dtype="fp32", B=1, Hq=8, Hkv=8, D=64, L=1024, W=128, M=2, K=256, rerope=False),
        # one conversation generating 128 tokens, 7B shape
        dict(name="generate_b1", kind="generate", dtype="bf16", B=1, Hq=32, Hkv=32, D=128, L=4096, W=1024, M=4, K=256),
        # ---- ordinary ones
        # eight long conversations, grouped-query heads, generating 128 tokens each
        dict(name="generate_b8_gqa", kind="generate", dtype="bf16", B=8, Hq=32, Hkv=8, D=128, L=8192, W=2048, M=8, K=256),
        # one decode step of sixteen sequences at context 32768: 1152 window rows, 127 of them on the constant-position query
        dict(name="step_b16_32k", kind="step", dtype="bf16", B=16, Hq=32, Hkv=32, D=128, n_valid=1152, n_bd=127, M=4, K=256),
        # 7B attention over 8192 tokens, plain RoPE
        dict(name="prefill_8k", kind="prefill", dtype="bf16", B=1, Hq=32, Hkv=32, D=128, L=8192, W=1024, M=4, K=256, rerope=False),
        # a half-precision model's layer on a prompt of odd length, ONE codebook of 1024 codes per head
        dict(name="layer_5001_fp16", kind="layer", dtype="fp16", B=1, Hq=32, Hkv=32, D=128, L=5001, W=1024, M=1, K=1024),
        # a program written for the interface that is mirrored: its own preparation, this framework's attention
        dict(name="dropin_8k", kind="dropin", dtype="bf16", B=1, Hq=32, Hkv=32, D=128, L=8192, W=1024, M=1, K=1024),
        # ---- the large ones
        # the headline workload: 7B attention at 32768 tokens, plain RoPE
        dict(name="prefill_32k", kind="prefill", dtype="bf16", B=1, Hq=32, Hkv=32, D=128, L=32768, W=1024, M=4, K=256, rerope=False),
        # ReRoPE with four codebooks of 512 codes, two sequences of 16384 tokens
        dict(name="rerope_16k_k512", kind="prefill", dtype="bf16", B=2, Hq=32, Hkv=32, D=128, L=16384, W=512, M=4, K=512, rerope=True),
        # a grouped-query layer on two prompts of 131072 tokens, eight codebooks
        dict(name="layer_131k_gqa", kind="layer", dtype="bf16", B=2, Hq=32, Hkv=8, D=128, L=131072, W=2048, M=8, K=256),
    ]


# ------------------------------------------------------------------------------------------- more of the same ranges

_MOST_FLOPS = 1.0e13      # of one drawn pass; the largest listed case has about 2e13
_MOST_SNAPSHOTS = 8.0e9   # bytes of per-block value sums that a drawn prefill forms; the largest listed case: 8.5e9


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _blocks(c):
    return max(0, -(-c["L"] // BLOCK) - c["W"] // BLOCK - 1)


def _fits(c):
    w = work(c)
    if c["kind"] in ("step", "generate"):
        return w["bytes"] < (5.0e8 if c["kind"] == "step" else 1.2e10)
    snapshots = c["B"] * c["Hkv"] * _blocks(c) * c["M"] * c["K"] * c["D"] * SIZE[c["dtype"]]
    # full precision runs on the regular cores: its drawn sizes stay small
    return w["flops"] < (4.0e10 if c["dtype"] == "fp32" else _MOST_FLOPS) and snapshots < _MOST_SNAPSHOTS


def draw(rng):
    while True:
        kind = rng.choice(["prefill", "prefill", "layer", "layer", "step", "generate", "dropin"])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"]) if kind != "dropin" else rng.choice(["bf16", "fp16"])
        D = rng.choice([64, 128, 128])
        Hkv = rng.choice([2, 4, 8, 8, 16, 32])
        G = 1 if kind == "dropin" else rng.choice([1, 1, 2, 4, 8])
        M, K = rng.choice([(1, 128), (1, 1024), (2, 128), (2, 256), (4, 256), (4, 256), (8, 256), (4, 512)])
        if kind == "dropin":
            M, K = 1, rng.choice([128, 256, 512, 1024])
        if Hkv * G > 64:
            continue
        c = dict(kind=kind, dtype=dtype, B=rng.choice([1, 1, 2, 4, 8]), Hq=Hkv * G, Hkv=Hkv, D=D, M=M, K=K)
        W = rng.choice([128, 256, 512, 1024, 2048])
        if kind == "step":
            n_valid = W + rng.randint(0, BLOCK - 1) + 1
            c.update(B=_log_int(rng, 1, 32), n_valid=n_valid, n_bd=n_valid - W - 1)
        else:
            c.update(W=W, L=_log_int(rng, 200, 100000 if kind in ("prefill", "layer") else 20000))
            if kind == "dropin":
                c["L"] = -(-c["L"] // BLOCK) * BLOCK     # the mirrored preparation knows whole blocks only
            if kind in ("dropin", "generate") and _blocks(c) < 1:
                continue
            if kind == "prefill":
                c["rerope"] = rng.random() < 0.5
        if _fits(c):
            return c


# ------------------------------------------------------------------------------------------- what a program has in hand

def _randn(g, *shape, dtype, scale=1.0):
    """Normal values rounded to dtype, a gigabyte of single precision at a time."""
    out = torch.empty(shape, dtype=dtype, device="cuda")
    flat = out.view(-1)
    step = 1 << 28
    for i in range(0, flat.numel(), step):
        n = min(step, flat.numel() - i)
        flat[i:i + n] = torch.randn(n, generator=g, device="cuda") * scale
    return out


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000003) + 17)


def _codebooks(g, c):
    cb = _randn(g, c["Hkv"], c["M"], c["K"], c["D"], dtype=torch.float32, scale=c["D"] ** -0.25)
    return cb, cb.reshape(c["Hkv"], c["M"] * c["K"], c["D"]).to(DTYPES[c["dtype"]])


def _prepare_prefill(c, g):
    dt, W = DTYPES[c["dtype"]], c["W"]
    q = _randn(g, c["B"], c["Hq"], c["L"], c["D"], dtype=dt)
    k = _randn(g, c["B"], c["Hkv"], c["L"], c["D"], dtype=dt)
    v = _randn(g, c["B"], c["Hkv"], c["L"], c["D"], dtype=dt)
    cb, act = _codebooks(g, c)
    if c["rerope"]:
        q1, q2, k1 = api.rope_qk(q, k, const_pos=W + 1, n_pos=max(c["L"], W + 2))
        k3 = k
    else:
        q1, _, k1 = api.rope_qk(q, k, n_pos=c["L"])
        q2, k3 = q1, k1
    return dict(q1=q1, q2=q2, k1=k1, k3=k3, v=v, cb=cb, act=act)


def _prepare_layer(c, g):
    # [B,L,H,D] storage seen as [B,H,L,D]: the layout that a layer's projections leave
    dt = DTYPES[c["dtype"]]
    q = _randn(g, c["B"], c["L"], c["Hq"], c["D"], dtype=dt).transpose(1, 2)
    k = _randn(g, c["B"], c["L"], c["Hkv"], c["D"], dtype=dt).transpose(1, 2)
    v = _randn(g, c["B"], c["L"], c["Hkv"], c["D"], dtype=dt).transpose(1, 2)
    cb, _ = _codebooks(g, c)
    pos = torch.arange(c["L"], device="cuda")[None].expand(c["B"], -1)
    return dict(q=q, k=k, v=v, cb=cb, pos=pos)


def _prepare_step(c, g):
    dt, B, Hkv, D, MK = DTYPES[c["dtype"]], c["B"], c["Hkv"], c["D"], c["M"] * c["K"]
    q1, q2 = _randn(g, B, c["Hq"], D, dtype=dt), _randn(g, B, c["Hq"], D, dtype=dt)
    k1, k3, v = (_randn(g, B, Hkv, c["n_valid"], D, dtype=dt) for _ in range(3))
    _, act = _codebooks(g, c)
    # about 32000 keys spread over each codebook's codes, some of which have no member
    cnt = torch.poisson(torch.full((B, Hkv, MK), 32000.0 / c["K"], device="cuda"), generator=g)
    cnt[torch.rand(B, Hkv, MK, generator=g, device="cuda") < 0.05] = 0
    vsum = (_randn(g, B, Hkv, MK, D, dtype=torch.float32) * cnt.sqrt()[..., None]).to(dt)
    return dict(q1=q1, q2=q2, k1=k1, k3=k3, v=v, act=act, cnt=cnt, vsum=vsum, ws=api.decode_workspace(B, c["Hq"], Hkv, D, "cuda"))


def _prepare_generate(c, g):
    s = _prepare_layer(c, g)
    cache = attn_vq.VectorQuantizedReRoPECache(c["W"], s["cb"])
    attn_vq.dispatch_attn_impl(s["q"], s["k"], s["v"], s["pos"], cache, kv_seq_len=c["L"])
    dt = DTYPES[c["dtype"]]
    new = [tuple(_randn(g, c["B"], h, 1, c["D"], dtype=dt) for h in (c["Hq"], c["Hkv"], c["Hkv"])) for _ in range(BLOCK)]
    return dict(cache=cache, new=new)


def _prepare_dropin(c, g):
    """The arguments of the mirrored interface: per-code running value sums in sorted order and, per block and code, the row
    of the last member so far."""
    s = _prepare_prefill(dict(c, rerope=True), g)
    dt, B, H, L, D, K = DTYPES[c["dtype"]], c["B"], c["Hkv"], c["L"], c["D"], c["K"]
    codes = api.assign_codes(s["k3"], s["cb"], out_dtype=torch.int64)[..., 0]
    nb = L // BLOCK
    cnt = torch.zeros(B, H, nb, K, device="cuda")
    cnt.scatter_add_(3, codes.view(B, H, nb, BLOCK), torch.ones(B, H, nb, BLOCK, device="cuda"))
    cnt = cnt.cumsum(2)
    order = torch.argsort(codes, dim=2, stable=True)
    total = torch.gather(s["v"].float(), 2, order[..., None].expand(-1, -1, -1, D)).double().cumsum(2)
    start = cnt[:, :, -1].cumsum(2) - cnt[:, :, -1]                          # first sorted row of every code
    first = torch.gather(start, 2, torch.gather(codes, 2, order)).long()     # ... of every row's own code
    before = torch.cat([torch.zeros(B, H, 1, D, dtype=total.dtype, device="cuda"), total], 2)
    v_vq = torch.zeros(B, H, L + 1, D, dtype=dt, device="cuda")
    v_vq[:, :, :L] = (total - torch.gather(before, 2, first[..., None].expand(-1, -1, -1, D))).to(dt)
    vi = torch.where(cnt > 0, start[:, :, None] + cnt - 1, float(L)).long()
    return dict(s, cnt=cnt, v_vq=v_vq, vi=vi)


def prepare(case, seed):
    g = _generator(seed)
    make = dict(prefill=_prepare_prefill, layer=_prepare_layer, step=_prepare_step, generate=_prepare_generate, dropin=_prepare_dropin)
    return dict(make[case["kind"]](case, g), case=case)


# ------------------------------------------------------------------------------------------- one pass

def run(s):
    c = s["case"]
    if c["kind"] == "prefill":
        return api.vq_attention_prefill(s["q1"], s["q2"], s["k1"], s["k3"], s["v"], s["cb"], c["W"], codebook_act=s["act"])
    if c["kind"] == "layer":
        # an empty cache per prompt, as a program makes one; what the prompt leaves in it comes back beside the output
        cache = attn_vq.VectorQuantizedReRoPECache(c["W"], s["cb"])
        out = attn_vq.dispatch_attn_impl(s["q"], s["k"], s["v"], s["pos"], cache, kv_seq_len=c["L"])
        return dict(out=out, counts=cache.key_cache[0], sums=cache.value_cache[0], keys=cache.key_buffers[0], values=cache.value_buffers[0])
    if c["kind"] == "step":
        return api.vq_attention_decode(s["q1"], s["q2"], s["k1"], s["k3"], s["v"], s["act"], s["cnt"], s["vsum"], n_valid=c["n_valid"],
                                       n_bd=c["n_bd"], workspace=s["ws"])
    if c["kind"] == "generate":
        cache = s["cache"]
        out = [attn_vq.dispatch_attn_impl(q, k, v, None, cache) for q, k, v in s["new"]]
        return dict(out=torch.cat(out, 1), counts=cache.key_cache[0], sums=cache.value_cache[0])
    return fused_vq_attn.vq_attn_forward(s["q1"], s["q2"], s["k1"], s["act"], s["cnt"], s["k3"], s["v"], s["v_vq"], s["vi"], c["W"])


# ------------------------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    c, size = case, SIZE[case["dtype"]]
    B, Hq, Hkv, D, MK = c["B"], c["Hq"], c["Hkv"], c["D"], c["M"] * c["K"]
    books = Hkv * MK * D
    if c["kind"] in ("step", "generate"):
        # window keys and values, value sums and counts, the codebooks once; queries and outputs
        tokens = 1 if c["kind"] == "step" else BLOCK
        rows = c["n_valid"] if c["kind"] == "step" else c["W"] + BLOCK // 2
        moved = B * Hkv * (2 * rows * D * size + MK * (D * size + 4)) + books * size + 2 * B * Hq * D * size
        return dict(bytes=tokens * moved, flops=tokens * 4.0 * B * Hq * D * (rows + MK))
    L, W = c["L"], c["W"]
    act = (2 * Hq + 2 * Hkv) * B * L * D * size
    i = torch.arange(L, dtype=torch.int64)
    short = c["kind"] == "layer" and L <= W + BLOCK
    bd = torch.zeros_like(i) if short else (i - W).clamp(min=0) // BLOCK * BLOCK
    far = int((bd > 0).sum())
    flops = 4.0 * D * B * Hq * (int((i - bd + 1).sum()) + far * MK)
    if far and c["kind"] != "dropin":
        flops += 2.0 * D * MK * B * Hkv * L      # a score of every key against every code
    moved = act + (books * 4 if far else 0)
    if c["kind"] == "layer":
        keep = L - max(0, L - W) // BLOCK * BLOCK
        moved += B * Hkv * (MK * (D + 1) * 4 + 3 * keep * D * size)          # the state left behind: sums, counts, window
    if c["kind"] == "prefill" and c["rerope"]:
        moved += (Hq + Hkv) * B * L * D * size   # both rotations of the queries, both kinds of keys
    if c["kind"] == "dropin":
        moved += (Hq + Hkv + Hkv) * B * L * D * size + B * Hkv * (L // BLOCK) * MK * 12
    return dict(bytes=moved, flops=flops)


def tolerance(case):
    """Four times the distance to the same attention in 64 bits (or, at the large sizes, to the single-precision kernel)."""
    return {
        "bf16": {"rel": 1e-2, "max": 2e-1},       # seen: 2.4e-3, 4.8e-2 (weights, sums and outputs rounded to 8 bits)
        "fp16": {"rel": 1.2e-3, "max": 2e-2},     # seen: 2.8e-4, 4.7e-3
        "fp32": {"rel": 2e-6, "max": 2e-5},       # seen: 2.8e-7, 4.3e-6
    }[case["dtype"]]
