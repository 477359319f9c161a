"""The work that users of this package have it do, as cases that can be prepared, run and timed.

A case is a dict of plain values.  ``kind`` says which public entry point a pass goes through:

  prefill    VecAttention_prefill on device tensors: one attention layer of a long prompt or of a video model
  vision     customize_prefill_attention with metric "vecattention" and a vision span: one layer of a vision-language
             model whose prompt has text before and after the video
  full       customize_prefill_attention with metric "full": the dense layers of a mixed configuration
  qk_hidden  qk_norm_rope: RMSNorm over the hidden size and rotary embedding of Q and K of a video-DiT layer
  qk_heads   qk_head_norm_rope: the same with a norm per head, on (B, H, L, 128) tensors with the text tokens last
  host       VecAttention_prefill_host: q, k and v start in pinned host memory and the result ends there

The path has one direction (prefill; there is no backward and no decode), two data types (bf16, fp16), two heights of the
query tile (64, 128) and the options that the models' configurations set: causal or not, grouped-query heads, a threshold
per call or per head, the size of the key-block groups, and the layout of the tensors.
"""
import math
from types import SimpleNamespace

import torch

import vecattention_b200 as va
from vecattention_b200.preattn import as_heads, qk_head_norm_rope, qk_norm_rope

D = 128  # head size of every model the path serves

# What the inputs look like, and the thresholds that keep a tenth or so of the keys on them.  The kept share is a
# property of the distribution and of the rule's block sizes, so work() can state it without running anything.
#   stripes: N(0, 1) with 1 % of the keys moved along a direction that every query shares (sinks and vertical stripes)
#   frames:  N(0, 0.5^2), K of rank 16 within each frame of 3600 tokens plus noise, 2 % stripe keys (video latents)
# (values, k_local_size, group_k_block) -> ((threshold, kept share), ...)
RULES = {
    ("stripes", 16, 16): ((0.840, 0.10), (0.870, 0.07)),
    ("stripes", 16, 1): ((0.880, 0.21),),
    ("stripes", 128, 1): ((0.845, 0.10),),
    ("frames", 16, 8192): ((0.879, 0.09), (0.894, 0.05)),
}


def _rule(values, bk, g, i=0):
    th, keep = RULES[values, bk, g][i]
    return {"values": values, "bk": bk, "g": g, "threshold": th, "keep": keep}


def listed():
    return [
        # one small layer: four heads, 2048 tokens; what is left of a call when there is hardly any work in it
        dict(name="short_2k", kind="prefill", dtype="bf16", heads=4, kv_heads=4, tokens=2048, pq=64, causal=False,
             chunk=32768, layout="bhsd", per_head=False, **_rule("stripes", 16, 16)),
        # an ordinary long prompt of a language model with 28 query heads on 4 KV heads: a ragged length, fp16,
        # thresholds per head, the configuration object's own block sizes and chunk
        dict(name="prompt_9k_fp16", kind="prefill", dtype="fp16", heads=28, kv_heads=4, tokens=9001, pq=64, causal=True,
             chunk=8192, layout="bhsd", per_head=True, **_rule("stripes", 16, 1)),
        # the README's quick-use call: 32 heads, 32 K tokens
        dict(name="quick_use_32k", kind="prefill", dtype="bf16", heads=32, kv_heads=32, tokens=32768, pq=64, causal=False,
             chunk=32768, layout="bhsd", per_head=False, **_rule("stripes", 16, 16)),
        # the operator's default arguments (128-row query tiles, 128-key blocks, causal, chunks of 16 K rows)
        dict(name="defaults_32k", kind="prefill", dtype="bf16", heads=32, kv_heads=32, tokens=32768, pq=128, causal=True,
             chunk=16384, layout="bhsd", per_head=False, **_rule("stripes", 128, 1)),
        # long-video prefill of a vision-language model: 28 query heads on 4 KV heads, 64 K tokens, causal
        dict(name="long_video_64k", kind="prefill", dtype="bf16", heads=28, kv_heads=4, tokens=65536, pq=64, causal=True,
             chunk=65536, layout="bhsd", per_head=False, **_rule("stripes", 16, 16)),
        # one GPU's share of a 40-head video-DiT layer whose heads are split over eight GPUs: 21 frames of 3600 tokens,
        # in the (B, S, H*D) storage that the projections leave
        dict(name="video_shard_75k", kind="prefill", dtype="bf16", heads=5, kv_heads=5, tokens=75600, pq=64, causal=False,
             chunk=32768, layout="bshd", per_head=False, **_rule("frames", 16, 8192)),
        # a whole video-DiT layer: 24 heads, 33 frames of 3600 tokens; the largest call
        dict(name="video_119k", kind="prefill", dtype="bf16", heads=24, kv_heads=24, tokens=118800, pq=64, causal=False,
             chunk=32768, layout="bhsd", per_head=False, **_rule("frames", 16, 8192)),
        # a prompt with a short text, a video and a question: dense rows around a sparse span, through the dispatcher
        dict(name="vision_20k", kind="vision", dtype="bf16", heads=28, kv_heads=4, tokens=20011, pq=64, causal=True,
             chunk=65536, begin=15, end=19900, **_rule("stripes", 16, 16)),
        # a dense layer through the same dispatcher
        dict(name="dense_8k", kind="full", dtype="bf16", heads=28, kv_heads=4, tokens=8192, causal=True),
        # what a video-DiT layer does to Q and K before attention: 40 heads (hidden size 5120), 75 600 tokens
        dict(name="qk_hidden_75k", kind="qk_hidden", dtype="bf16", heads=40, tokens=75600, text=0),
        # the per-head form of it: 24 heads, 118 800 video tokens and 256 text tokens
        dict(name="qk_heads_119k", kind="qk_heads", dtype="bf16", heads=24, tokens=119056, text=256),
        # activations kept in host memory: eight heads of 32 K tokens through the copy pipeline
        dict(name="host_8h_32k", kind="host", dtype="bf16", heads=8, kv_heads=8, tokens=32768, pq=64, causal=False,
             chunk=32768, **_rule("stripes", 16, 16)),
    ]


# ---- drawn cases --------------------------------------------------------------------------------------------------------
def _tokens(rng, lo, hi):
    """A length spread over the logarithm of its range: half of them whole query tiles, half of them any number."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.5 else max(lo, n // 128 * 128)


def draw(rng):
    most = work(next(c for c in listed() if c["name"] == "video_119k"))["flops"]
    while True:
        kind = rng.choice(["prefill"] * 5 + ["vision", "full", "qk_hidden", "qk_heads", "host"])
        dtype = rng.choice(["bf16", "bf16", "fp16"])
        if kind in ("qk_hidden", "qk_heads"):
            heads = rng.choice([12, 16, 24, 40])
            case = dict(kind=kind, dtype=dtype, heads=heads, tokens=_tokens(rng, 1000, 119056), text=rng.choice([0, 77, 256]))
        elif kind == "full":
            heads, kv = rng.choice([(28, 4), (16, 16), (32, 8)])
            case = dict(kind=kind, dtype=dtype, heads=heads, kv_heads=kv, tokens=_tokens(rng, 500, 16384), causal=True)
        else:
            frames = kind == "prefill" and rng.random() < 0.3
            wide = not frames and kind == "prefill" and rng.random() < 0.3
            causal = kind == "vision" or (kind == "prefill" and not frames and rng.random() < 0.6)
            if causal:
                heads, kv = rng.choice([(28, 4), (32, 8), (16, 16), (32, 32), (7, 1)])
            else:
                heads = kv = rng.choice([3, 4, 5, 8, 12, 24, 32, 40])
            # (a whole-sequence group keeps more of a shorter sequence: video layers have tens of thousands of tokens)
            lo, hi = (50000, 118800) if frames else (1500, {"prefill": 118800, "vision": 65536, "host": 65536}[kind])
            bk, g = (16, 8192) if frames else rng.choice([(128, 1)] if wide else [(16, 16), (16, 16), (16, 1)])
            values = "frames" if frames else "stripes"
            case = dict(kind=kind, dtype=dtype, heads=heads, kv_heads=kv, tokens=_tokens(rng, lo, hi),
                        pq=128 if wide else 64, causal=causal, chunk=rng.choice([8192, 16384, 32768, 65536]),
                        **_rule(values, bk, g, rng.randrange(len(RULES[values, bk, g]))))
            if kind == "prefill":
                case.update(layout=rng.choice(["bhsd", "bhsd", "bshd"]), per_head=rng.random() < 0.3)
            if kind == "vision":
                case["begin"] = rng.randrange(0, min(300, case["tokens"] // 8))
                case["end"] = case["tokens"] - rng.randrange(0, min(600, case["tokens"] // 8))
        need = work(case)
        if need["flops"] <= most and need["bytes"] <= 3e9:
            return case


# ---- inputs -------------------------------------------------------------------------------------------------------------
def _dtype(case):
    return {"bf16": torch.bfloat16, "fp16": torch.float16}[case["dtype"]]


def _qkv(case, seed):
    """q (1, H, S, D), k and v (1, Hkv, S, D) in the case's data type, and its layout."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, kv, s = case["heads"], case["kv_heads"], case["tokens"]
    frames = case.get("values") == "frames"
    sigma, share = (0.5, 0.02) if frames else (1.0, 0.01)
    bshd = case.get("layout") == "bshd"

    def empty(n):
        if bshd:
            return as_heads(torch.empty(1, s, n * D, dtype=_dtype(case), device="cuda"), n)
        return torch.empty(1, n, s, D, dtype=_dtype(case), device="cuda")

    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    q, k, v = empty(h), empty(kv), empty(kv)
    for i in range(kv):
        u = randn(D)
        u = u / u.norm()
        key = randn(s, D)
        if frames:
            nf = math.ceil(s / 3600)
            low = torch.bmm(randn(nf, 3600, 16), randn(nf, 16, D)).reshape(nf * 3600, D)[:s] / 4.0
            key = 0.8 * low + 0.6 * key
        key = sigma * key
        key[torch.randperm(s, generator=g, device="cuda")[: max(1, int(share * s))]] += 3.0 * sigma * u
        if case["causal"]:
            key[:4] += 3.0 * sigma * u  # attention sink
        k[0, i] = key
        v[0, i] = sigma * randn(s, D)
        for j in range(i * (h // kv), (i + 1) * (h // kv)):
            q[0, j] = sigma * (randn(s, D) + u)
    return q, k, v


def _angles(tokens):
    """Angles of a rotary embedding: token position times 64 frequencies."""
    freq = 10000.0 ** (-torch.arange(0, D, 2, dtype=torch.float32, device="cuda") / D)
    return torch.outer(torch.arange(tokens, dtype=torch.float32, device="cuda"), freq)


def prepare(case, seed):
    kind, st = case["kind"], SimpleNamespace(case=case)
    if kind in ("qk_hidden", "qk_heads"):
        g = torch.Generator(device="cuda").manual_seed(seed)
        h, s, dt = case["heads"], case["tokens"], _dtype(case)
        shape, width = ((1, s, h * D), h * D) if kind == "qk_hidden" else ((1, h, s, D), D)
        st.q, st.k = (torch.randn(shape, generator=g, device="cuda", dtype=dt) for _ in range(2))
        st.wq, st.wk = ((1 + 0.1 * torch.randn(width, generator=g, device="cuda")).to(dt) for _ in range(2))
        a = _angles(s - case["text"])
        a = a if kind == "qk_hidden" else a.repeat_interleave(2, dim=1)
        st.cos, st.sin = a.cos().contiguous(), a.sin().contiguous()
        return st
    st.q, st.k, st.v = _qkv(case, seed)
    if kind == "prefill":
        st.threshold = torch.full((case["heads"],), case["threshold"], device="cuda") if case["per_head"] else case["threshold"]
    elif kind == "vision":
        # one row of thresholds per layer, as tuned configurations have them
        st.config = va.FastPrefillConfig(metric="vecattention", threshold=torch.full((4, case["heads"]), case["threshold"], device="cuda"),
                                         block_size_q=case["pq"], block_size_k=case["bk"], group_k_block=case["g"],
                                         chunk_size=case["chunk"], vision_start_position=case["begin"],
                                         vision_end_position=case["end"], output_time=False)
        st.layer = SimpleNamespace(layer_idx=2)
    elif kind == "full":
        st.config = va.FastPrefillConfig(metric="full", output_time=False)
        st.layer = SimpleNamespace(layer_idx=0)
    elif kind == "host":
        st.q, st.k, st.v = (t.cpu().pin_memory() for t in (st.q, st.k, st.v))
        st.out, st.staging = torch.empty_like(st.q).pin_memory(), {}
    return st


# ---- one pass -----------------------------------------------------------------------------------------------------------
def run(st):
    c = st.case
    if c["kind"] == "prefill":
        return va.VecAttention_prefill(st.q, st.k, st.v, st.threshold, c["pq"], c["bk"], c["g"], c["causal"], c["chunk"])
    if c["kind"] in ("vision", "full"):
        return va.customize_prefill_attention(st.layer, st.q, st.k, st.v, causal=c["causal"], config=st.config)
    if c["kind"] == "qk_hidden":
        return qk_norm_rope(st.q, st.k, st.wq, st.wk, 1e-6, st.cos, st.sin, c["text"], heads=c["heads"])
    if c["kind"] == "qk_heads":
        return qk_head_norm_rope(st.q, st.k, st.wq, st.wk, 1e-6, st.cos, st.sin, c["text"])
    return va.VecAttention_prefill_host(st.q, st.k, st.v, c["threshold"], c["pq"], c["bk"], c["g"], c["causal"], c["chunk"],
                                        out=st.out, staging=st.staging)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def _sparse_pairs(case, rows):
    """(query row, key) pairs of rows [0, rows) that the selection leaves: the kept share of the keys that a row's query
    tile may select, and under the causal rule the first and the diagonal tile."""
    if not case["causal"]:
        return rows * case["tokens"] * case["keep"]
    pq = case["pq"]
    diagonal = rows * pq / 2
    return diagonal + max(0, rows - pq) * pq + max(0.0, rows * rows / 2 - rows * 1.5 * pq) * case["keep"]


def work(case):
    h, s, kind = case["heads"], case["tokens"], case["kind"]
    if kind in ("qk_hidden", "qk_heads"):
        table = (s - case["text"]) * (D // 2 if kind == "qk_hidden" else D) * 4
        weights = 2 * 2 * (h * D if kind == "qk_hidden" else D)
        # a multiplication-addition for the sum of squares, two products, and three operations of the rotation
        return {"bytes": 2 * (2 * s * h * D * 2) + 2 * table + weights, "flops": 7 * 2 * s * h * D}
    bytes_ = 2 * (2 * h + 2 * case["kv_heads"]) * s * D
    if kind == "full":
        return {"bytes": bytes_, "flops": 4 * D * h * s * s / 2}
    end, begin = case.get("end", s), case.get("begin", 0)
    pairs = _sparse_pairs(case, end) - (_sparse_pairs(case, begin) if begin else 0)
    pairs += begin * begin / 2 + (s * s - end * end) / 2  # the dense rows before and after a vision span
    estimate = 2 * D * math.ceil(end / case["pq"]) * (end / 2 if case["causal"] else s)  # pooled Q times every key
    return {"bytes": bytes_, "flops": h * (4 * D * pairs + estimate)}


def tolerance(case):
    """Results are 16-bit; the probabilities and the weighted sums' operands are 16-bit too.  bf16 has 8 significant
    bits and fp16 has 11."""
    if case["kind"] in ("qk_hidden", "qk_heads"):
        return {"rel": 5e-3 if case["dtype"] == "bf16" else 1e-3}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


# ---- the results in 64 bits -------------------------------------------------------------------------------------------------
MOST_PAIRS = 6e10  # (query, key) pairs of all heads above which the 64-bit result takes too long


def _selected(q, k, threshold, pq, bk, g, causal, chunk):
    """Keep mask (query tiles, keys) of one head.  The pooled queries are 16-bit values by the operator's definition;
    everything after them is 64-bit."""
    s, n = k.shape[0], math.ceil(q.shape[0] / pq)
    pad = n * pq - q.shape[0]
    pooled = torch.nn.functional.pad(q.double(), (0, 0, 0, pad)).view(n, pq, D).sum(1)
    rows = torch.full((n, 1), float(pq), dtype=torch.float64, device=q.device)
    rows[-1] -= pad
    pooled = ((pooled / rows).to(q.dtype).float() * (1.0 / math.sqrt(D))).to(q.dtype)
    est = pooled.double() @ k.double().t()
    blocks = math.ceil(s / bk)
    groups = math.ceil(blocks / g)
    tops = torch.full((n, groups * g * bk), -math.inf, dtype=torch.float64, device=q.device)
    tops[:, :s] = est
    if causal:
        tops[:, :pq] = -math.inf
    tops = tops.view(n, groups * g, bk).amax(-1).view(n, groups, g).cummax(-1).values.view(n, -1)
    keep = est - math.log(threshold + 1e-9) >= tops.repeat_interleave(bk, dim=1)[:, :s]
    if causal:  # the first tile and the diagonal one are dense; a chunk's every 64th tile loses most of the tile before its own
        tile = torch.arange(n, device=q.device)
        end = tile * pq
        end = torch.where(tile % (chunk // pq) % 64 == 0, torch.minimum(end, (tile - 1) * pq + bk), end)[:, None]
        key = torch.arange(s, device=q.device)[None]
        tile = tile[:, None]
        keep = (keep & (key >= pq) & (key < end)) | (key < pq) | ((key >= tile * pq) & (key < (tile + 1) * pq))
    return keep


def _attend(q, k, v, keep, pq, causal, row0=0):
    """Softmax attention of one head's rows row0, row0 + 1, ...; keep: their tiles' keys, or None for all."""
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    k, v = k.double(), v.double()
    step = max(pq, int(1e8) // k.shape[0] // pq * pq)
    for a in range(0, q.shape[0], step):
        x = q[a:a + step].double() @ k.t() / math.sqrt(D)
        n = x.shape[0]
        if keep is not None:
            x.masked_fill_(~keep[a // pq:(a + n + pq - 1) // pq].repeat_interleave(pq, dim=0)[:n], -math.inf)
        if causal:
            row = torch.arange(row0 + a, row0 + a + n, device=q.device)[:, None]
            x.masked_fill_(torch.arange(k.shape[0], device=q.device)[None] > row, -math.inf)
        out[a:a + n] = torch.softmax(x, dim=-1) @ v
    return out


def _normed_rotated(x, w, cos, sin, per_head, text):
    """RMSNorm of the last dimension, then the rotation of (even, odd) pairs of every token that has angles."""
    x = x.double()
    x = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    if per_head:
        cos, sin = cos[:, ::2].double(), sin[:, ::2].double()
        turned = x[:, :, :x.shape[2] - text]
    else:
        x = x.view(x.shape[0], x.shape[1], -1, D).transpose(1, 2)
        cos, sin = cos.double(), sin.double()
        turned = x[:, :, text:]
    even, odd = turned[..., ::2], turned[..., 1::2]
    turned[..., ::2], turned[..., 1::2] = even * cos - odd * sin, odd * cos + even * sin
    return x


def exact(case, seed):
    kind, h, s = case["kind"], case["heads"], case["tokens"]
    if kind not in ("qk_hidden", "qk_heads") and h * s * s > MOST_PAIRS:
        return None
    st = prepare(case, seed)
    if kind in ("qk_hidden", "qk_heads"):
        return tuple(_normed_rotated(x, w, st.cos, st.sin, kind == "qk_heads", case["text"]) for x, w in ((st.q, st.wq), (st.k, st.wk)))
    out = torch.empty(st.q.shape, dtype=torch.float64, device="cuda")
    begin, end = case.get("begin", 0), 0 if kind == "full" else case.get("end", s)
    for i in range(h):
        q, (k, v) = st.q[0, i].cuda(), (x[0, i // (h // case["kv_heads"])].cuda() for x in (st.k, st.v))
        if end:
            keep = _selected(q[:end], k[:end], case["threshold"], case["pq"], case["bk"], case["g"], case["causal"], case["chunk"])
            out[0, i, :end] = _attend(q[:end], k[:end], v[:end], keep, case["pq"], case["causal"])
        if begin:
            out[0, i, :begin] = _attend(q[:begin], k, v, None, 64, True)
        if end < s:
            out[0, i, end:] = _attend(q[end:], k, v, None, 64, True, end)
    return out
