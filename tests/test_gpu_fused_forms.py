"""The two forms of the fused kernel at ranks 17 to 64, against the oracle: small and ragged batches, which take the wide
form except where the narrow one can split their pieces further, and batches with enough pieces for the narrow form; alone,
grouped, several projections at a time, and split over clusters.  Tolerance: v and y are rounded to 16 bits (2^-9
relative in bf16) after fp32 sums, and y carries v's rounding: rtol = atol = 1e-2 as for the other forward tests."""
import pytest
import torch

from oracle import smlm_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rank", [24, 32, 40, 64])
@pytest.mark.parametrize("rm", [False, True])
@pytest.mark.parametrize("lens", [[1] * 9, [8] * 6, [8] * 5 + [9], [64, 65, 1, 17, 130], [0, 3, 0, 0, 5], [9] * 150])
@pytest.mark.parametrize("split", [0, 1, 2, 4])
def test_forms_on_either_side_of_the_rule(dtype, rank, rm, lens, split):
    from gpu_util import check_forward
    from loquetier_b200 import ops
    ids = [(3 * i) % 4 for i in range(len(lens))]
    prev = ops.set_cluster_split(split)
    try:
        # the widths end in partial steps of 256 and 512 columns, slabs of 512 and 1024, and half a k16 step
        c = O.make_case(90 + rank, lens, ids, 4, 1304, 2056, rank, dtype, is_row_major=rm)
        check_forward(c)
        check_forward(c, scale=[2.0, 0.5, 1.25, 1.0], indexed=True)
    finally:
        ops.set_cluster_split(prev)


# every kind of row block: whole, half and ragged ones, pieces of 64 rows with a rest, and short segments that share
# adapters, so that a grouped plan gathers them.  36 rows a segment: never the tcgen05 kernel at this rank.
PATTERN = [8, 16, 40, 64, 65, 130, 1, 3, 7, 30]


def _ctas_per_sm(lens, jobs, n_table=None):
    """What the rule counts (unsplit): a segment as its rows / 64 and half a piece."""
    segs = len(lens) if n_table is None else min(len(lens), n_table)
    return max(segs, sum(lens) / 64 + segs / 2) * jobs / 148


@pytest.mark.parametrize("dtype,rank,rm,split", [
    (torch.bfloat16, 64, False, 0), (torch.float16, 64, False, 2), (torch.float16, 64, True, 4), (torch.bfloat16, 64, True, 1),
    (torch.bfloat16, 40, False, 4), (torch.float16, 40, True, 0), (torch.bfloat16, 32, True, 2), (torch.float16, 32, False, 4),
    (torch.float16, 32, True, 0), (torch.bfloat16, 24, False, 1)])
def test_narrow_form_whole_and_ragged_blocks(dtype, rank, rm, split):
    """One projection: one pointer per segment, then gathered by 40 adapters with a scale, then added to a result."""
    from gpu_util import check_forward
    from loquetier_b200 import ops
    n_ad, lens = 40, PATTERN * 44
    ids = [(7 * i) % n_ad for i in range(len(lens))]
    assert _ctas_per_sm(lens, 1) >= 1.75 and _ctas_per_sm(lens, 1, n_ad) >= 1.75   # both calls take the narrow form
    prev = ops.set_cluster_split(split)
    try:
        # partial steps of 128 and 256 columns, partial slabs of 256 and 512
        c = O.make_case(70 + rank, lens, ids, n_ad, 712, 1096, rank, dtype, is_row_major=rm)
        check_forward(c)
        check_forward(c, scale=[(2.0, 0.5, 1.25, 1.0)[i % 4] for i in range(n_ad)], indexed=True)
        y0 = torch.randn((sum(lens), 1096), generator=torch.Generator().manual_seed(rank)).to(dtype)
        check_forward(c, accumulate=True, y_init=y0, indexed=True)
    finally:
        ops.set_cluster_split(prev)


@pytest.mark.parametrize("dtype,rank", [(torch.bfloat16, 64), (torch.float16, 64), (torch.bfloat16, 32), (torch.float16, 40)])
@pytest.mark.parametrize("grouped", [False, True])
def test_narrow_form_seven_projections(dtype, rank, grouped):
    """A layer's projections in one launch, forward (gathered or not) and dV/dX."""
    from gpu_util import ptr_table
    from helpers import assert_close
    from loquetier_b200 import ops
    dev = torch.device("cuda:0")
    n_ad, lens = 24, PATTERN * 7
    ids = [(5 * i) % n_ad for i in range(len(lens))]
    assert _ctas_per_sm(lens, 7) >= 2.25 and _ctas_per_sm(lens, 7, n_ad) >= 2.25   # the narrow form, with either plan
    T = sum(lens)
    cases = [O.make_case(300 + i, lens, ids, n_ad, hi, ho, rank, dtype)
             for i, (hi, ho) in enumerate([(520, 520), (520, 136), (520, 136), (520, 520), (520, 1320), (520, 1320), (1320, 520)])]
    seg = torch.tensor(cases[0]["seg"], dtype=torch.int32, device=dev)
    idt = torch.tensor(ids, dtype=torch.int32, device=dev)
    projs, keep = [], []
    for c in cases:
        wa, wb = [w.to(dev) for w in c["wa"]], [w.to(dev) for w in c["wb"]]
        keep.append((wa, wb))
        nan = lambda n: torch.full((T, n), float("nan"), dtype=dtype, device=dev)
        projs.append(dict(x=c["x"].to(dev), go=c["go"].to(dev), y=nan(c["h_out"]), v=nan(rank), dx=nan(c["h_in"]), dv=nan(rank),
                          wa=ptr_table(wa), wb=ptr_table(wb)))
    ps = ops.ProjSet(projs)
    plan = ops.Plan(seg, T, seg_ids=idt, n_table=n_ad) if grouped else ops.Plan(seg, T)
    parts = ops.Plan(seg, T)
    ops.fwd_multi(ps, plan, rank, seg_ids=idt)
    ops.bwd_dx_multi(ps, parts, rank, part_ids=idt)
    torch.cuda.synchronize()
    plan.raise_if_failed()
    parts.raise_if_failed()
    for c, p in zip(cases, projs):
        wa, wb = [c["wa"][i] for i in ids], [c["wb"][i] for i in ids]
        y, v = O.add_lora_forward((T, c["h_out"]), c["x"], wa, wb, c["seg"], rank, round_v=True)
        assert_close(p["v"].cpu(), v, what="v")
        assert_close(p["y"].cpu(), y.to(torch.float32), what="y")
        dv = torch.cat([c["go"][a:b].float() @ w.float() for a, b, w in zip(c["seg"], c["seg"][1:], wb)]).to(dtype)
        dx = torch.cat([dv[a:b].float() @ w.float() for a, b, w in zip(c["seg"], c["seg"][1:], wa)])
        assert_close(p["dv"].cpu(), dv, what="dv")
        assert_close(p["dx"].cpu(), dx, what="dx")
