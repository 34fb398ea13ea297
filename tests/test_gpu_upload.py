"""Small host arrays written to the device through kernel parameters: exact at the sizes where the launch changes
(128 and 896 words) and where the copy takes over, in stream order, and under capture."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n", [0, 1, 63, 64, 65, 127, 128, 129, 447, 448, 449, 896, 897, 2048, 2049])
def test_device_ints_holds_the_values(dtype, n):
    from loquetier_b200 import ops
    top = (1 << 31) - 1 if dtype == torch.int32 else (1 << 62)
    vals = [(-1) ** i * ((i * 2654435761) % top) for i in range(n)]
    t = ops.device_ints(vals, dtype, DEV)
    assert t.dtype == dtype and t.device == DEV and t.tolist() == vals


def test_upload_follows_the_stream_and_can_be_captured():
    from loquetier_b200 import ops
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        a = ops.device_ints([1, 2, 3], torch.int64, DEV)
        b = a + 1
    side.synchronize()
    assert b.tolist() == [2, 3, 4]
    out = torch.zeros(3, dtype=torch.int64, device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c = ops.device_ints([7, 8, 9], torch.int64, DEV)
        out.copy_(c)
    graph.replay()
    torch.cuda.synchronize()
    assert out.tolist() == [7, 8, 9]


def test_workspace_tickets_survive_shapes_on_either_side_of_the_smallest_head():
    """Weight gradients of a few and of many partitions in turn through the cached workspace: the head of tickets stands
    still for small shapes and moves (and is cleared) for large ones; a stale ticket would leave a gradient unmerged."""
    from loquetier_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)

    def grads(npart, rows, hi, ho, rank):
        n = npart * rows
        rnd = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
        x, go, v, dv = rnd(n, hi), rnd(n, ho), rnd(n, rank), rnd(n, rank)
        dA = torch.full((npart, rank, hi), float("nan"), dtype=torch.bfloat16, device=DEV)
        dB = torch.full((npart, ho, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
        part = torch.arange(0, n + 1, rows, dtype=torch.int32, device=DEV)
        tab = lambda w: torch.tensor([t.data_ptr() for t in w], dtype=torch.int64, device=DEV)
        ops.wgrad_pair(tab(list(dA)), tab(list(dB)), dv, x, v, go, part, ops.Plan(part, n), rank)
        f = lambda t: t.double().view(npart, rows, -1)
        want_a = torch.matmul(f(dv).transpose(1, 2), f(x))
        want_b = torch.matmul(f(go).transpose(1, 2), f(v))
        for got, want in ((dA, want_a), (dB, want_b)):
            # one rounding of the result to bf16 (2^-9) on top of fp32 sums of `rows` products
            assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + 1e-4 * rows).all()

    for npart, rows, hi, ho, rank in ((2, 300, 512, 256, 8), (300, 40, 2048, 2048, 16), (3, 700, 1024, 512, 64),
                                      (300, 70, 2048, 1024, 64), (2, 300, 512, 256, 8), (300, 40, 2048, 2048, 16)):
        grads(npart, rows, hi, ho, rank)
