"""Decode attention at the sizes where its tiles and ranges end.  Tolerance: keys, softmax weights
and results are rounded to 16 bits once each (2^-9 relative in bf16), scores and sums are fp32; three such roundings of
values of order one stay below rtol = atol = 1e-2."""
import numpy as np
import pytest
import torch

from helpers import assert_close
from oracle import attention_oracle as A

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
THETA = 10000.0


def _cache(seed, seqlens, N, P, dtype):
    pages, indptr, last = A.make_cache(seed, seqlens, 1, N, P, 128, dtype)
    pd = [p.to(DEV).contiguous() for p in pages]
    dev = dict(keep=pd, ptrs=torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device=DEV),
               ind=torch.tensor(indptr, dtype=torch.int32, device=DEV),
               last=torch.tensor(last, dtype=torch.int32, device=DEV))
    return (pages, indptr, last), dev


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group,batch", [(1, 3), (4, 3), (8, 2), (4, 60), (2, 65), (8, 57), (1, 127), (1, 128), (1, 129)])
def test_decode_at_the_edges_of_tiles_ranges_and_ranks(dtype, group, batch):
    """Tiles of 16 keys, a warp's step of 64, the rotation computed afresh every 1024 keys; small batches are cut into
    ranges.  Equal lengths, empty requests and batches that are no multiple of four are among them, and a page table with
    entries that no request uses."""
    from loquetier_b200 import kvcache
    N, P = 8, 16
    edge = [1023, 1024, 1025, 2100, 15, 16, 17, 63, 64, 65, 0, 1, 128, 129, 64, 0, 17]
    seqlens = (edge * 4 + [3, 20] * 40)[:batch] if batch > 3 else [1025, 2100, 17][:batch]
    host, d = _cache(50 + group + batch, seqlens, N, P, dtype)
    q = torch.randn((batch, N * group, 128), generator=torch.Generator().manual_seed(batch)).to(dtype)
    ptrs = d["ptrs"]
    padded = torch.cat([ptrs, ptrs[:1].expand(max(0, 97 * batch - ptrs.numel()))]).contiguous()
    outs = []
    for table in ((ptrs, ptrs) if batch <= 3 else (ptrs, padded)):
        o = torch.full(q.shape, float("nan"), dtype=dtype, device=DEV)
        word = torch.zeros(1, dtype=torch.int32, device=DEV)
        kvcache.batch_decode_into(o, q.to(DEV), table, d["ind"], d["last"], 1, 0, N, THETA, P, status_word=word)
        assert int(word.item()) == 0
        outs.append(o)
    assert torch.equal(outs[0], outs[1])   # merged in a fixed order
    assert_close(outs[0], A.batch_decode(q, *host, 0, THETA), what=f"group {group} batch {batch}")


def test_decode_scores_that_grow_along_the_sequence():
    """Keys scaled up with their position: the maxima are raised again and again, in every warp and range."""
    from loquetier_b200 import kvcache
    N, group, P, L = 1, 4, 16, 900
    (pages, indptr, last), d = _cache(77, [L], N, P, torch.float16)
    for i, pg in enumerate(pages):
        pg[:, 0] *= 1.0 + 0.1 * i
        d["keep"][i].copy_(pg)
    q = (torch.randn((1, group, 128), generator=torch.Generator().manual_seed(78)) * 1.5).to(torch.float16)
    o = torch.empty(q.shape, dtype=q.dtype, device=DEV)
    kvcache.batch_decode_into(o, q.to(DEV), d["ptrs"], d["ind"], d["last"], 1, 0, N, THETA, P)
    assert_close(o, A.batch_decode(q, pages, indptr, last, 0, THETA), what="raised maxima")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group,batch", [(4, 60), (8, 57), (1, 130)])
def test_decode_weight_of_a_key_that_dominates_late_is_not_rounded(dtype, group, batch):
    """Softmax weights are rounded to 16 bits relative to the largest score met so far, so the key that sets it has the
    weight one exactly, in whatever tile it comes.  One key in the second tile of its warp dominates, by 1 to 7.9 in the
    base-2 score; its value is the only one that is not zero.  Query and key lie in a dimension that this rope base does
    not turn and their product is exact, so the result is known in float64 and is off by its own rounding only: half a
    unit of the storage type (and 2^-18 relative for the fp32 exponential, sums and reciprocal)."""
    from loquetier_b200 import kvcache
    N, P, L, at, dim = 8, 16, 192, 69, 63
    bits, k = (8, 16.0) if dtype == torch.bfloat16 else (11, 16.0)
    qscale = 1.4426950408889634 / 128 ** 0.5
    g = torch.Generator().manual_seed(group)
    cand = (torch.rand(20000, generator=g, dtype=torch.float64) * 6.9 + 1.0).div(k * qscale).to(dtype).double()
    scaled = cand * qscale
    cand = cand[((scaled * (1 + 1e-5)).to(dtype) == (scaled * (1 - 1e-5)).to(dtype))]   # its rounding is beyond doubt
    q1 = cand[torch.randperm(cand.numel(), generator=g)[:batch * N * group]].view(batch, N * group)
    q = torch.zeros((batch, N * group, 128), dtype=dtype)
    q[:, :, dim] = q1.to(dtype)
    npg = L // P
    pages = torch.zeros((batch * npg, 1, 2, N, P, 128), dtype=dtype)
    v = torch.randn((batch, N, 128), generator=g).to(dtype)
    for b in range(batch):
        pg = pages[b * npg + at // P, 0]
        pg[0, :, at % P, dim] = k
        pg[1, :, at % P] = v[b]
    pd = pages.to(DEV)
    ptrs = torch.tensor([p.data_ptr() for p in pd], dtype=torch.int64, device=DEV)
    ind = torch.arange(0, (batch + 1) * npg, npg, dtype=torch.int32, device=DEV)
    last = torch.full((batch,), P, dtype=torch.int32, device=DEV)
    o = torch.empty(q.shape, dtype=dtype, device=DEV)
    kvcache.batch_decode_into(o, q.to(DEV), ptrs, ind, last, 1, 0, N, 1e30, P)
    w = torch.exp2((q1 * qscale).to(dtype).double() * k)
    want = (w / (w + (L - 1))).unsqueeze(-1) * v.double().repeat_interleave(group, dim=1)
    half = torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(2.0 ** -14))) - bits)   # half a unit in the last place
    assert ((o.cpu().double() - want).abs() <= half * 1.0001 + want.abs() * 2.0 ** -18).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch", [4, 60])   # cut into ranges, and not
def test_decode_not_a_number_shows_in_the_heads_it_enters(dtype, batch):
    """A NaN or an infinity in one query head or one key makes the heads that see it NaN - never zeros, which would pass
    for a result - and leaves all others as they are."""
    from loquetier_b200 import kvcache
    N, group, P, L = 8, 4, 16, 600
    _, d = _cache(90 + batch, [L] * batch, N, P, dtype)
    q = torch.randn((batch, N * group, 128), generator=torch.Generator().manual_seed(91)).to(dtype)
    run = lambda: kvcache.batch_decode_into(torch.empty(q.shape, dtype=dtype, device=DEV), q.to(DEV), d["ptrs"], d["ind"],
                                            d["last"], 1, 0, N, THETA, P)
    clean = run()
    assert torch.isfinite(clean.float()).all()
    bad = torch.zeros(q.shape[:2], dtype=torch.bool, device=DEV)
    q[1, 5, 17] = float("nan")                                     # one query head
    bad[1, 5] = True
    npg = -(-L // P)
    d["keep"][2 * npg + 300 // P][0, 0, 3, 300 % P, 9] = float("nan")   # one key of request 2, kv head 3
    bad[2, 3 * group:4 * group] = True
    d["keep"][3 * npg][0, 0, 6, :, 40] = float("inf")              # a whole tile of keys of request 3, kv head 6
    bad[3, 6 * group:7 * group] = True
    o = run()
    assert torch.isnan(o[bad].float()).all()
    assert torch.equal(o[~bad], clean[~bad])


@pytest.mark.parametrize("spare", [0, 1, 3000])
def test_decode_ranges_follow_the_requests_and_not_the_page_table(spare):
    """A page table may be longer than the pages in use (a captured step keeps its arguments).  The ranges a request is
    cut into are seen from the states parked in the workspace: as many as its length asks for, with any table."""
    from loquetier_b200 import kvcache
    from loquetier_b200.cabi import lib
    N, group, P, REC = 8, 4, 16, 132
    seqlens = [1024, 2000, 40, 600]
    host, d = _cache(61, seqlens, N, P, torch.bfloat16)
    batch = len(seqlens)
    q = torch.randn((batch, N * group, 128), generator=torch.Generator().manual_seed(62)).to(torch.bfloat16)
    head = lib.smlm_b200_batch_decode_ticket_bytes(batch, N)
    ws = torch.zeros(lib.smlm_b200_batch_decode_workspace_bytes(batch, N * group, N), dtype=torch.uint8, device=DEV)
    ws[head:].view(torch.float32).fill_(float("nan"))
    table = torch.cat([d["ptrs"], d["ptrs"][:1].expand(spare)]).contiguous()
    o = torch.empty(q.shape, dtype=q.dtype, device=DEV)
    kvcache.batch_decode_into(o, q.to(DEV), table, d["ind"], d["last"], 1, 0, N, THETA, P, workspace=ws)
    parked = ~torch.isnan(ws[head:].view(torch.float32).view(batch, N * group, -1, REC)[..., 0])
    splits = parked.shape[2]
    assert splits == min(16, -(-3 * 148 // (batch * N)))
    for b, n in enumerate(seqlens):
        tiles = -(-n // 16)
        per = max(4, -(-tiles // splits))
        want = -(-tiles // per)
        want = 0 if want == 1 else want   # one range is not parked
        assert (parked[b].sum(-1) == want).all(), (n, want)
    assert_close(o, A.batch_decode(q, *host, 0, THETA), what="long table")


@pytest.mark.parametrize("batch", [56, 57, 128, 129, 160, 191, 192])
@pytest.mark.parametrize("lens", ["uneven", "equal", "one long"])
def test_decode_longest_first_does_not_show(batch, lens):
    """From 56 requests of 8 kv heads to 192 the requests go by length if they hold 96 tiles each on average and one of
    them 5/4 of the mean.  The same requests in a batch of 193 go in batch order: equal results bit for bit.  Empty and
    equal requests among them; pages are shared between requests, which a cache of prefixes does too."""
    from loquetier_b200 import kvcache
    N, group, P, dtype = 8, 1, 16, torch.bfloat16
    edge = [0, 1, 17, 4100, 1600, 1600, 3000, 2999, 64, 2500, 4100, 1023, 3300]
    seqlens = {"uneven": (edge * 15)[:batch], "equal": [1600] * batch, "one long": [1600] * (batch - 1) + [2100]}[lens]
    while sum(-(-n // P) for n in seqlens) * P < 96 * 16 * batch:   # raise the mean over the line
        seqlens[seqlens.index(min(v for v in seqlens if v > 64))] = 4000
    assert lens == "equal" or max(seqlens) * batch > 1.25 * sum(seqlens)
    more = seqlens + [1600] * (193 - batch)
    g = torch.Generator().manual_seed(batch)
    pool = torch.randn((400, 1, 2, N, P, 128), generator=g).to(dtype)
    dev = pool.to(DEV)
    pick = [torch.randint(0, 400, (-(-n // P),), generator=g).tolist() for n in more]
    q = torch.randn((193, N * group, 128), generator=g).to(dtype)

    def run(lengths):
        idx = [i for p in pick[:len(lengths)] for i in p]
        ind = torch.tensor([0] + np.cumsum([-(-n // P) for n in lengths]).tolist(), dtype=torch.int32, device=DEV)
        last = torch.tensor([A.last_page_offset_of(n, P) if n else 0 for n in lengths], dtype=torch.int32, device=DEV)
        table = torch.tensor([dev[i].data_ptr() for i in range(400)], dtype=torch.int64, device=DEV)[idx]
        o = torch.full((len(lengths), N * group, 128), float("nan"), dtype=dtype, device=DEV)
        word = torch.zeros(1, dtype=torch.int32, device=DEV)
        kvcache.batch_decode_into(o, q[:len(lengths)].to(DEV), table, ind, last, 1, 0, N, THETA, P, status_word=word)
        assert int(word.item()) == 0
        return o.cpu()

    o = run(seqlens)
    assert torch.equal(o, run(more)[:batch])
    some = [0, 1, 2, 3, batch - 1]
    host = [pool[i] for b in some for i in pick[b]]
    ind = [0] + np.cumsum([len(pick[b]) for b in some]).tolist()
    last = [A.last_page_offset_of(seqlens[b], P) if seqlens[b] else 0 for b in some]
    assert_close(o[some], A.batch_decode(q[some], host, ind, last, 0, THETA), what=f"{lens} {batch}")
