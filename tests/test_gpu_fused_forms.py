"""The two forms of the fused kernel at ranks 17 to 64: batches on either side of the rule (rows per segment) and at
it, alone, grouped, and split over clusters, against the oracle.  Tolerance: v and y are rounded to 16 bits (2^-9
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
