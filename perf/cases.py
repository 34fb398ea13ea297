"""The work that a program built on this package has it do, as timed cases.

Every case is one pass through public entry points (``ops``, ``MixedLoraLinear``, ``add_lora``, the operator-level
functions of ``kernels``, the paged cache of ``kvcache``, ``rms_norm``) on inputs that are on the GPU already.  A
case is a dict of plain values; ``prepare`` makes its inputs from a seed, ``run`` does one pass and returns what it
computes, ``work`` says what the pass cannot do without and ``tolerance`` how far two correct implementations of
it may be apart.

Kinds of cases
  layer     every LoRA projection of one transformer layer through the calls that take several projections at a
            time: both plans, dV/dX, forward, dA/dB - or plan and forward only where the batch trains nothing
  linear    one layer's projections through the ``MixedLoraLinear`` modules, base product included; with train
            requests in the batch also their backward through autograd
  add_lora  the autograd function alone, forward and backward
  operator  the two operator calls (shrink, expand) of one projection
  decode    one attention step of a decode batch over the paged cache: append, then attention
  prefill   the same for prompts: the keys and values into the cache, then causal attention
  rms       RMSNorm forward and backward
"""
from __future__ import annotations

import math

import numpy as np
import torch

from loquetier_b200 import kernels, kvcache, ops
from loquetier_b200.kernel_utils import BatchLenInfo, add_lora, rms_norm
from loquetier_b200.mixed_lora import MixedLoraContext, MixedLoraLinear, NamedLoraLayer
from loquetier_b200.segments import wants_grouped_plan

SCALE = 2.0   # alpha / r
THETA = 500000.0
HEAD = 128
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # One training-and-serving step of a layer: seven projections, segment lengths of a heavy-tailed mix,
        # a quarter of the tokens in fine-tune segments.
        dict(name="layer_mixed", kind="layer", proj="all", hidden=4096, inter=14336, kv=1024, tokens=8192, seg="zipf",
             ft=0.25, rank=16, adapters=128, dtype="bf16", len_seed=3000),
        # A fine-tuning-only step at a large rank: long segments, all of them trained.
        dict(name="layer_finetune_r64", kind="layer", proj="updown", hidden=4096, inter=14336, kv=0, tokens=32768,
             seg="2048", ft=1.0, rank=64, adapters=64, dtype="bf16", len_seed=5000),
        # A large decode batch in arrival order: one token per request, many adapters.
        dict(name="decode_adapters", kind="layer", proj="updown", hidden=4096, inter=11008, kv=0, tokens=1024, seg="1",
             ft=0.0, rank=32, adapters=256, dtype="bf16", len_seed=4000),
        # A decode step of a small server through the modules: latency and launches count.
        dict(name="linear_decode", kind="linear", proj="all", hidden=4096, inter=14336, kv=1024, trains=0, train_len=0,
             prefills=0, prefill_len=0, decodes=64, rank=16, adapters=32, dtype="bf16", len_seed=6000),
        # A unified step through the modules: two fine-tune requests, a few prompts and some decode tokens.
        dict(name="linear_train", kind="linear", proj="attn", hidden=4096, inter=0, kv=1024, trains=2, train_len=512,
             prefills=4, prefill_len=150, decodes=32, rank=8, adapters=8, dtype="bf16", len_seed=6100),
        # The autograd function on a q projection: two fine-tune segments, prompts and decode tokens, fp16.
        dict(name="add_lora_fp16", kind="add_lora", h_in=4096, h_out=4096, trains=2, train_len=1024, prefills=4,
             prefill_len=512, decodes=64, rank=16, adapters=32, dtype="fp16", len_seed=2000),
        # The smallest call: operator granularity, a hundred tokens in four segments, narrow layers.
        dict(name="operator_small", kind="operator", h_in=256, h_out=256, tokens=105, segments=4, rank=8, adapters=3,
             dtype="fp16", len_seed=1000),
        # A full decode batch over long contexts, then a few requests over short ones.
        dict(name="attn_decode", kind="decode", batch=128, ctx_lo=512, ctx_hi=4096, kv_heads=8, group=4, page=16,
             dtype="bf16", len_seed=9000),
        dict(name="attn_decode_few", kind="decode", batch=5, ctx_lo=70, ctx_hi=3000, kv_heads=8, group=4, page=16,
             dtype="fp16", len_seed=9100),
        # A batch of ordinary prompts, then two long ones with wider groups and larger pages.
        dict(name="attn_prefill", kind="prefill", prompts=32, len_lo=256, len_hi=2048, kv_heads=8, group=4, page=16,
             dtype="bf16", len_seed=9000),
        dict(name="attn_prefill_long", kind="prefill", prompts=2, len_lo=4001, len_hi=7999, kv_heads=8, group=8, page=32,
             dtype="fp16", len_seed=9200),
        # The norm in front of the projections of a long training batch.
        dict(name="rms_norm_train", kind="rms", rows=32768, cols=4096, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "linear", "linear", "add_lora", "operator", "decode", "decode",
                       "prefill", "prefill", "rms"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    seed = rng.randrange(1 << 20)
    if kind == "layer":
        hidden = 64 * rng.randint(16, 80)
        inter = 16 * int(hidden * rng.uniform(2.5, 3.5) / 16)
        what = rng.choice(["mixed", "finetune", "decode"])
        base = dict(kind=kind, hidden=hidden, inter=inter, dtype=dtype, len_seed=seed)
        if what == "mixed":
            return dict(base, proj="all", kv=hidden // 4, tokens=_log(rng, 64, 8192), seg="zipf",
                        ft=rng.choice([0.0, 0.25, 0.5]), rank=rng.choice([8, 16, 32, 64]), adapters=_log(rng, 4, 128))
        if what == "finetune":
            return dict(base, proj="updown", kv=0, tokens=_log(rng, 500, 20000), seg=str(_log(rng, 100, 2048)), ft=1.0,
                        rank=rng.choice([8, 16, 64, 128]), adapters=64)
        return dict(base, proj="updown", kv=0, tokens=_log(rng, 8, 1024), seg="1", ft=0.0,
                    rank=rng.choice([8, 16, 32, 64]), adapters=_log(rng, 2, 256))
    if kind == "linear":
        hidden = 64 * rng.randint(16, 64)
        train = rng.random() < 0.5
        return dict(kind=kind, proj="attn" if train else "all", hidden=hidden, inter=0 if train else 16 * (hidden // 5),
                    kv=hidden // 4, trains=rng.randint(1, 3) if train else 0, train_len=_log(rng, 40, 512) if train else 0,
                    prefills=rng.randint(0, 4), prefill_len=_log(rng, 10, 400), decodes=_log(rng, 1, 256),
                    rank=rng.choice([8, 16, 32]), adapters=rng.randint(4, 32), dtype=dtype, len_seed=seed)
    if kind == "add_lora":
        return dict(kind=kind, h_in=64 * rng.randint(8, 96), h_out=64 * rng.randint(8, 96), trains=rng.randint(1, 4),
                    train_len=_log(rng, 30, 1024), prefills=rng.randint(0, 4), prefill_len=_log(rng, 10, 700),
                    decodes=_log(rng, 1, 200), rank=rng.choice([8, 16, 32, 64]), adapters=rng.randint(4, 32), dtype=dtype,
                    len_seed=seed)
    if kind == "operator":
        return dict(kind=kind, h_in=8 * _log(rng, 16, 1000), h_out=8 * _log(rng, 16, 1000), tokens=_log(rng, 10, 4000),
                    segments=_log(rng, 1, 200), rank=rng.choice([8, 16, 32, 64]), adapters=_log(rng, 1, 64), dtype=dtype,
                    len_seed=seed)
    if kind == "decode":
        hi = _log(rng, 100, 8000)
        batch = min(_log(rng, 1, 256), max(1, 300000 // hi))
        return dict(kind=kind, batch=batch, ctx_lo=max(1, hi // rng.randint(2, 12)), ctx_hi=hi,
                    kv_heads=rng.choice([4, 8]), group=rng.choice([1, 4, 8]), page=rng.choice([8, 16, 32]), dtype=dtype,
                    len_seed=seed)
    if kind == "prefill":
        hi, N, G = _log(rng, 30, 6000), rng.choice([4, 8]), rng.choice([1, 4, 8])
        prompts = min(_log(rng, 1, 64), max(1, 40000 // hi), max(1, int(4.7e9 / (N * G * hi * hi))))
        return dict(kind=kind, prompts=prompts, len_lo=max(1, hi // rng.randint(1, 8)), len_hi=hi, kv_heads=N, group=G,
                    page=rng.choice([16, 32, 64]), dtype=dtype, len_seed=seed)
    return dict(kind=kind, rows=_log(rng, 1, 32768), cols=8 * rng.randint(64, 768), dtype=dtype)


# ---------------------------------------------------------------------------
# what a case is made of
# ---------------------------------------------------------------------------

def _projections(c):
    """(h_in, h_out) of the case's projections."""
    h, f, kv = c["hidden"], c["inter"], c["kv"]
    attn = [(h, h), (h, kv), (h, kv), (h, h)]
    return {"attn": attn, "updown": [(h, f), (f, h)], "all": attn + [(h, f), (h, f), (f, h)]}[c["proj"]]


def _layer_batch(c):
    """Segment lengths, adapter per segment and number of leading fine-tune segments."""
    rng = np.random.default_rng(c["len_seed"])
    total, lens = c["tokens"], []
    while sum(lens) < total:
        n = int(min(2048, rng.zipf(1.2))) if c["seg"] == "zipf" else int(c["seg"])
        lens.append(min(n, total - sum(lens)))
    want, train, rest = int(round(c["ft"] * total)), [], []
    for n in lens:   # the first tokens are trained; a segment across the line is cut there
        take = min(n, want - sum(train))
        if take > 0:
            train.append(take)
        if n > take:
            rest.append(n - take)
    # a trained adapter appears once in the trained part
    ids = [int(v) for v in rng.permutation(c["adapters"])[:len(train)]] if len(train) <= c["adapters"] \
        else [int(v) for v in rng.integers(0, c["adapters"], size=len(train))]
    ids += [int(v) for v in rng.integers(0, c["adapters"], size=len(rest))]
    return train + rest, ids, len(train)


def _request_batch(c):
    """Lengths and adapters of the segments train | prompts | decode of a request batch, and the prompts'
    lengths.  Decode tokens come sorted by adapter, equal neighbours merged, as a batch assembler hands them on."""
    rng = np.random.default_rng(c["len_seed"])
    lens = [c["train_len"] - int(rng.integers(0, 1 + c["train_len"] // 8)) for _ in range(c["trains"])]
    ids = [int(v) for v in rng.permutation(c["adapters"])[:c["trains"]]]
    prompts = [max(1, int(rng.integers(c["prefill_len"] // 2, 2 * c["prefill_len"] + 1))) for _ in range(c["prefills"])]
    lens += prompts
    ids += sorted(int(v) for v in rng.integers(0, c["adapters"], size=len(prompts)))
    for a in sorted(int(v) for v in rng.integers(0, c["adapters"], size=c["decodes"])):
        if len(ids) > c["trains"] + len(prompts) and ids[-1] == a:
            lens[-1] += 1
        else:
            ids.append(a)
            lens.append(1)
    return lens, ids, prompts


def _operator_batch(c):
    rng = np.random.default_rng(c["len_seed"])
    n = min(c["segments"], c["tokens"])
    cuts = sorted(int(v) for v in rng.permutation(c["tokens"] - 1)[:n - 1] + 1)
    bounds = [0] + cuts + [c["tokens"]]
    return [b - a for a, b in zip(bounds[:-1], bounds[1:])], [int(v) for v in rng.integers(0, c["adapters"], size=n)]


def _lengths(c):
    """Context lengths of a decode batch or prompt lengths of a prefill batch."""
    rng = np.random.default_rng(c["len_seed"])
    lo, hi = (c["ctx_lo"], c["ctx_hi"]) if c["kind"] == "decode" else (c["len_lo"], c["len_hi"])
    return [int(v) for v in rng.integers(lo, hi + 1, size=c["batch"] if c["kind"] == "decode" else c["prompts"])]


class _Maker:
    """Seeded tensors of one case."""

    def __init__(self, c, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.dev).manual_seed(seed)
        self.dt = DTYPES[c["dtype"]]

    def randn(self, *shape, scale=1.0):
        return (torch.randn(shape, generator=self.g, device=self.dev, dtype=torch.float32) * scale).to(self.dt)

    def empty(self, *shape, dtype=None):
        return torch.empty(shape, device=self.dev, dtype=dtype or self.dt)

    def ints(self, v, dtype=torch.int32):
        return torch.tensor(v, dtype=dtype, device=self.dev)

    def table(self, tensors):
        return self.ints([t.data_ptr() for t in tensors], torch.int64)

    def adapter(self, n, rank, h_in, h_out):
        """n adapters' A [rank, h_in] and B [h_out, rank]."""
        return self.randn(n, rank, h_in, scale=h_in ** -0.5), self.randn(n, h_out, rank, scale=0.02)


def _starts(lens):
    return [0] + [int(v) for v in np.cumsum(np.asarray(lens, dtype=np.int64))]


# ---------------------------------------------------------------------------
# prepare and run, kind by kind
# ---------------------------------------------------------------------------

def _prepare_layer(c, m):
    lens, ids, ntrain = _layer_batch(c)
    bounds = _starts(lens)
    T, n, r = bounds[-1], bounds[ntrain], c["rank"]
    s = dict(T=T, n=n, r=r, n_ad=c["adapters"], seg=m.ints(bounds), ids=m.ints(ids), ids_host=ids, lens=lens,
             scale=torch.full((c["adapters"],), SCALE, dtype=torch.float32, device=m.dev), projs=[])
    if n:
        s.update(part=m.ints(bounds[:ntrain + 1]), part_ids=m.ints(ids[:ntrain]))
    for hi, ho in _projections(c):
        A, B = m.adapter(c["adapters"], r, hi, ho)
        p = dict(x=m.randn(T, hi), A=A, B=B, wa=m.table(list(A)), wb=m.table(list(B)), y=m.empty(T, ho),
                 v=m.empty(T, r), h_in=hi, h_out=ho)
        if n:
            p.update(go=m.randn(n, ho), dx=m.empty(n, hi), dv=m.empty(n, r), dA=m.empty(ntrain, r, hi),
                     dB=m.empty(ntrain, ho, r))
            p.update(dA_t=m.table(list(p["dA"])), dB_t=m.table(list(p["dB"])))
        s["projs"].append(p)
    s["set"] = ops.ProjSet(s["projs"])
    return s


def _run_layer(s):
    group = wants_grouped_plan(s["lens"], s["ids_host"])
    seg_ids = s["ids"] if group else None
    r = s["r"]
    if not s["n"]:
        plan = ops.Plan(s["seg"], s["T"], seg_ids=seg_ids, n_table=s["n_ad"])
        ops.fwd_multi(s["set"], plan, r, seg_ids=s["ids"], seg_scale=s["scale"])
        return [p["y"] for p in s["projs"]]
    plan, pplan = ops.plan_pair(s["seg"], s["T"], s["part"], s["n"], seg_ids_a=seg_ids, n_table_a=s["n_ad"])
    ops.bwd_dx_multi(s["set"], pplan, r, part_ids=s["part_ids"], part_scale=s["scale"])
    ops.fwd_multi(s["set"], plan, r, seg_ids=s["ids"], seg_scale=s["scale"], independent=True)
    ops.wgrad_pair_multi(s["set"], s["part"], pplan, r, part_ids=s["part_ids"], part_scale=s["scale"], n_table=s["n_ad"])
    return [[p[k] for k in ("y", "dx", "dA", "dB")] for p in s["projs"]]


def _prepare_linear(c, m):
    lens, ids, prompts = _request_batch(c)
    bounds = _starts(lens)
    T, ntrain = bounds[-1], c["trains"]
    ctx = MixedLoraContext()
    s = dict(ctx=ctx, lens=lens, ids=ids, train_idx=ids[:ntrain], lora_len=m.ints(lens), segment=m.ints(bounds),
             blen=BatchLenInfo([(1, n) for n in lens[:ntrain]], prompts, c["decodes"], [], m.dev), mods=[], params=[])
    for hi, ho in _projections(c):
        base = torch.nn.Linear(hi, ho, bias=False, dtype=m.dt, device="meta")
        base.weight = torch.nn.Parameter(m.randn(ho, hi, scale=0.02), requires_grad=False)
        A, B = m.adapter(c["adapters"], c["rank"], hi, ho)
        ads = [NamedLoraLayer("a%d" % i, A[i], B[i], torch.nn.Identity(), SCALE) for i in range(c["adapters"])]
        lin = MixedLoraLinear(ctx, base, ads, c["rank"], m.dt)
        lin.set_trainable(s["train_idx"])
        params = [lin.get_parameter("lora-%d-%s" % (i, k)) for i in s["train_idx"] for k in "AB"]
        x = m.randn(T, hi)
        s["mods"].append((lin, x.requires_grad_(ntrain > 0), m.randn(T, ho) if ntrain else None, params))
    return s


def _run_linear(s):
    s["ctx"].update(s["blen"], s["ids"], s["lora_len"], s["segment"], s["train_idx"])
    if not s["train_idx"]:
        with torch.no_grad():
            return [lin(x) for lin, x, _, _ in s["mods"]]
    out = []
    for lin, x, go, params in s["mods"]:
        for t in [x] + params:
            t.grad = None
        y = lin(x)
        y.backward(go)
        out.append([y.detach(), x.grad] + [p.grad for p in params])
    return out


def _prepare_add_lora(c, m):
    lens, ids, _ = _request_batch(c)
    bounds = _starts(lens)
    T, ntrain = bounds[-1], c["trains"]
    A, B = m.adapter(c["adapters"], c["rank"], c["h_in"], c["h_out"])
    ws = [torch.nn.Parameter(w) for i in ids[:ntrain] for w in (A[i], B[i])]
    return dict(A=A, B=B, ws=ws, x=m.randn(T, c["h_in"]).requires_grad_(True), go=m.randn(T, c["h_out"]),
                wa=m.table([A[i] for i in ids]), wb=m.table([B[i] for i in ids]), s=m.ints(bounds), r=c["rank"],
                shape=(T, c["h_out"]), tp=bounds[:ntrain + 1])


def _run_add_lora(s):
    for t in [s["x"]] + s["ws"]:
        t.grad = None
    y = add_lora.apply(s["shape"], s["x"], s["wa"], s["wb"], s["s"], s["r"], s["tp"][-1], s["tp"], *s["ws"])
    y.backward(s["go"])
    return [y.detach(), s["x"].grad] + [w.grad for w in s["ws"]]


def _prepare_operator(c, m):
    lens, ids = _operator_batch(c)
    A, B = m.adapter(c["adapters"], c["rank"], c["h_in"], c["h_out"])
    return dict(A=A, B=B, x=m.randn(c["tokens"], c["h_in"]), v=m.empty(c["tokens"], c["rank"]),
                y=m.empty(c["tokens"], c["h_out"]), wa=m.table([A[i] for i in ids]), wb=m.table([B[i] for i in ids]),
                s=m.ints(_starts(lens)),
                tmp=m.empty(kernels.smlm_forward_cutlass_tmp_size(len(lens)), dtype=torch.uint8))


def _run_operator(s):
    kernels.smlm_forward_cutlass(s["v"], s["x"], s["wa"], s["s"], s["tmp"], False)
    kernels.smlm_forward_cutlass(s["y"], s["v"], s["wb"], s["s"], s["tmp"], False)
    return [s["v"], s["y"]]


def _prepare_attention(c, m):
    lens = _lengths(c)
    N, G, D = c["kv_heads"], c["group"], HEAD
    pages = sum(-(-n // c["page"]) for n in lens)
    pool = kvcache.KvPool(2, N, D, c["page"], m.dt, m.dev, pages_per_slab=pages)
    caches = [kvcache.KvCache(pool, n) for n in lens]
    for slab in pool._slabs:
        slab.normal_(generator=m.g)
    rows = len(lens) if c["kind"] == "decode" else sum(lens)
    return dict(pool=pool, caches=caches, kv=kvcache.BatchedKvCache(caches), indptr=m.ints(_starts(lens)),
                q=m.randn(rows, N * G, D), k=m.randn(rows, N, D), v=m.randn(rows, N, D))


def _run_decode(s):
    kvcache.append_kv(s["kv"], s["k"], s["v"], 1)
    return [kvcache.batch_decode(s["q"], s["kv"], THETA, 1)] + s["pool"]._slabs


def _run_prefill(s):
    kvcache.init_kv(s["kv"], s["k"], s["v"], s["indptr"], 1)
    return [kvcache.batch_prefill(s["q"], s["indptr"], s["kv"], THETA, 1)] + s["pool"]._slabs


def _prepare_rms(c, m):
    w = 1.0 + 0.1 * torch.randn(c["cols"], generator=m.g, device=m.dev)
    return dict(x=m.randn(c["rows"], c["cols"], scale=1.5).requires_grad_(True), w=torch.nn.Parameter(w.to(m.dt)),
                go=m.randn(c["rows"], c["cols"]))


def _run_rms(s):
    s["x"].grad = s["w"].grad = None
    o = rms_norm.apply(s["x"], s["w"], 1e-5)
    o.backward(s["go"])
    return [o.detach(), s["x"].grad, s["w"].grad]


_KINDS = {
    "layer": (_prepare_layer, _run_layer), "linear": (_prepare_linear, _run_linear),
    "add_lora": (_prepare_add_lora, _run_add_lora), "operator": (_prepare_operator, _run_operator),
    "decode": (_prepare_attention, _run_decode), "prefill": (_prepare_attention, _run_prefill),
    "rms": (_prepare_rms, _run_rms),
}


def prepare(case, seed):
    make, go = _KINDS[case["kind"]]
    return go, make(case, _Maker(case, seed))


def run(state):
    go, s = state
    return go(s)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _lora_work(T, n, hi, ho, r, used, used_ft):
    """Bytes and operations of one projection's update over T rows, n of them trained: x and y and every adapter in
    use once; for the trained rows gO and dX once (x is read above, v and dV stay inside) and their gradients once."""
    b = 2 * (T * (hi + ho) + used * r * (hi + ho))
    b += 2 * (n * (hi + ho) + used_ft * r * (hi + ho))
    return b, 2 * r * (hi + ho) * (T + 2 * n)


def work(case):
    c, kind = case, case["kind"]
    b = f = 0
    if kind == "layer":
        lens, ids, nt = _layer_batch(c)
        for hi, ho in _projections(c):
            d = _lora_work(sum(lens), sum(lens[:nt]), hi, ho, c["rank"], len(set(ids)), nt)
            b, f = b + d[0], f + d[1]
    elif kind in ("linear", "add_lora"):
        lens, ids, _ = _request_batch(c)
        T, n = sum(lens), sum(lens[:c["trains"]])
        for hi, ho in (_projections(c) if kind == "linear" else [(c["h_in"], c["h_out"])]):
            d = _lora_work(T, n, hi, ho, c["rank"], len(set(ids)), c["trains"])
            b, f = b + d[0], f + d[1]
            if n:   # gO and the gradient of x are there for every row
                b += 2 * (T - n) * (hi + ho)
            if kind == "linear":   # the base product, and in training the gradient through it
                b, f = b + 2 * hi * ho, f + 2 * T * hi * ho * (2 if n else 1)
    elif kind == "operator":
        lens, ids = _operator_batch(c)
        T, r, h = sum(lens), c["rank"], c["h_in"] + c["h_out"]
        b, f = 2 * (T * h + 2 * T * r + len(set(ids)) * r * h), 2 * T * r * h
    elif kind == "decode":
        lens, N, G = _lengths(c), c["kv_heads"], c["group"]
        rows = len(lens)
        # every key and value once, q and o once, the new keys and values read and written
        b = 2 * HEAD * (2 * sum(lens) * N + 2 * rows * N * G + 2 * rows * N)
        f = 4 * HEAD * N * G * sum(lens)
    elif kind == "prefill":
        lens, N, G = _lengths(c), c["kv_heads"], c["group"]
        rows = sum(lens)
        # q and o once, the keys and values read once and written to the cache once; visible keys only
        b = 2 * HEAD * (2 * rows * N * G + 4 * rows * N)
        f = 4 * HEAD * N * G * sum(n * (n + 1) // 2 for n in lens)
    else:
        rows, cols = c["rows"], c["cols"]
        b, f = 2 * (4 * rows * cols + 2 * cols), 10 * rows * cols   # x, gO read, o, dX written; w, dW
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Against the same pass in 64 bits the outputs are off by a relative 2.3e-3 (the projections), 3.4e-3 (attention) and
    1.7e-3 (the norm) in bf16, and by 3.0e-4 and 4.3e-4 in fp16: the rounding of the rank-r intermediates, of rotated
    keys and softmax weights, and of the results.  Single values are off by up to 3e-2 in bf16 and 5e-3 in fp16, in units
    of the larger of the value and the result's root mean square.  Stated is four times that."""
    if case["dtype"] == "fp16":
        return {"rel": 1.7e-3, "max": 2e-2}
    return {"rel": 7e-3, "max": 2e-2} if case["kind"] == "rms" else {"rel": 1.3e-2, "max": 1.2e-1}
