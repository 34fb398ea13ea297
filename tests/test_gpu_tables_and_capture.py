"""Device arrays that outlive the call which fills them, and calls under stream capture.

A module's pointer tables are read on whatever stream runs it, so they are complete when the module is; arrays that
describe one batch, and workspaces, must not be left behind half made by a capture, which records launches and runs
none."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _module(n_ad, rank=8, h_in=64, h_out=96, is_scaled=False):
    from loquetier_b200.mixed_lora import MixedLoraContext, MixedLoraLinear, NamedLoraLayer
    g = torch.Generator(device=DEV).manual_seed(n_ad)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
    base = nn.Linear(h_in, h_out, bias=False, dtype=torch.bfloat16, device=DEV)
    ads = [NamedLoraLayer(f"a{i}", rnd(rank, h_in), rnd(h_out, rank), nn.Identity(), None if is_scaled else 0.5 + i)
           for i in range(n_ad)]
    ctx = MixedLoraContext()
    return ctx, base, ads, lambda: MixedLoraLinear(ctx, base, ads, rank, torch.bfloat16, is_scaled=is_scaled)


@pytest.mark.parametrize("is_scaled", [False, True])
def test_a_modules_tables_are_complete_on_return(is_scaled):
    """Built on a stream that is still busy; read on another one without waiting for the first."""
    _, _, ads, make = _module(5, is_scaled=is_scaled)
    _, _, more, _ = _module(6, is_scaled=is_scaled)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    want = lambda mod, k: [getattr(a, k).data_ptr() for a in mod.adapters]
    with torch.cuda.stream(side):
        torch.cuda._sleep(300_000_000)   # about 0.15 s
        lin = make()
    for add in (False, True):
        if add:
            with torch.cuda.stream(side):
                torch.cuda._sleep(300_000_000)
                lin.add_adapter(more[5])
        assert lin.wa_ptrs.tolist() == want(lin, "wa") and lin.wb_ptrs.tolist() == want(lin, "wb")
        if not is_scaled:
            assert lin.scaling_f32.tolist() == [float(torch.tensor(a.scaling).to(torch.bfloat16)) for a in lin.adapters]
    side.synchronize()


def _batch(ctx, lens, ids, trains, train_idx):
    from loquetier_b200.kernel_utils import BatchLenInfo
    seg = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    blen = BatchLenInfo([(1, n) for n in lens[:trains]], [], sum(lens[trains:]), [], DEV)
    ctx.update(blen, ids, torch.tensor(lens, dtype=torch.int32, device=DEV), seg, train_idx)


@pytest.mark.parametrize("trains", [0, 2])
def test_the_first_forward_of_a_batch_is_refused_under_capture(trains):
    """It builds the batch's plans and index arrays, which later forwards use outside the graph as well; under capture
    nothing of it would have run.  The batch is as before afterwards, and a captured forward after an eager one works."""
    ctx, _, _, make = _module(4)
    lin = make()
    lin.set_trainable([0, 1])
    lens, ids = [20, 30, 1, 1], [0, 1, 2, 3]
    _batch(ctx, lens, ids, trains, [0, 1][:trains])
    x = torch.randn((sum(lens), 64), device=DEV).to(torch.bfloat16)
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad():
        lin.base_layer(x)   # (the base product's library is set up)
        with pytest.raises(RuntimeError, match="captur"):
            with torch.cuda.graph(graph):
                lin(x)
        assert ctx._dev == {}
        want = lin(x)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = lin(x)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("kind", ["linear", "add_lora"])
def test_a_backward_is_refused_under_capture(kind):
    """It writes the addresses of this call's gradients and weights to the device; a graph would keep them.  The same
    backward runs afterwards outside the capture."""
    from loquetier_b200.kernel_utils import add_lora
    ctx, _, ads, make = _module(4)
    lens, ids = [20, 30, 1, 1], [0, 1, 2, 3]
    x = torch.randn((sum(lens), 64), device=DEV).to(torch.bfloat16).requires_grad_(True)
    go = torch.randn((sum(lens), 96), device=DEV).to(torch.bfloat16)
    lin = make()
    lin.set_trainable([0, 1])
    params = [lin.get_parameter(f"lora-{i}-{k}") for i in (0, 1) for k in "AB"]
    _batch(ctx, lens, ids, 2, [0, 1])
    tab = lambda k: torch.tensor([getattr(ads[i], k).data_ptr() for i in ids], dtype=torch.int64, device=DEV)
    seg = torch.tensor([0, 20, 50, 51, 52], dtype=torch.int32, device=DEV)
    wa, wb = tab("wa"), tab("wb")

    def forward():
        if kind == "linear":
            return lin(x)
        return add_lora.apply((sum(lens), 96), x, wa, wb, seg, 8, 50, [0, 20, 50], *params)

    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        want = torch.autograd.grad(forward(), [x] + params, go)
        y = forward()
        with pytest.raises(RuntimeError, match="captur"):
            with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=side):
                torch.autograd.grad(y, [x] + params, go, retain_graph=True)
        got = torch.autograd.grad(y, [x] + params, go)
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_a_workspace_made_under_capture_is_cleared_before_its_first_eager_use():
    """The zeros of a workspace that a capture allocates are recorded there; until a replay its memory holds anything."""
    from loquetier_b200 import kvcache, ops
    N, group, P = 8, 4, 16
    g = torch.Generator(device=DEV).manual_seed(3)
    pool = torch.randn((400, 1, 2, N, P, 128), generator=g, device=DEV).to(torch.bfloat16)

    def decode(batch, pages):
        ptrs = torch.tensor([pool[i].data_ptr() for i in range(batch * pages)], dtype=torch.int64, device=DEV)
        ind = torch.arange(0, (batch + 1) * pages, pages, dtype=torch.int32, device=DEV)
        last = torch.full((batch,), P, dtype=torch.int32, device=DEV)
        q = torch.randn((batch, N * group, 128), generator=g, device=DEV).to(torch.bfloat16)
        o = torch.full_like(q, float("nan"))
        return o, lambda: kvcache.batch_decode_into(o, q, ptrs, ind, last, 1, 0, N, 1e4, P)

    def wgrad(npart, rows, hi, ho, rank):
        n = npart * rows
        rnd = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)
        x, go, v, dv = rnd(n, hi), rnd(n, ho), rnd(n, rank), rnd(n, rank)
        out = torch.full((npart, rank * (hi + ho)), float("nan"), dtype=torch.bfloat16, device=DEV)
        part = torch.arange(0, n + 1, rows, dtype=torch.int32, device=DEV)
        tab = lambda off: torch.tensor([o.data_ptr() + 2 * off for o in out], dtype=torch.int64, device=DEV)
        tA, tB, plan = tab(0), tab(rank * hi), ops.Plan(part, n)
        return out, lambda: ops.wgrad_pair(tA, tB, dv, x, v, go, part, plan, rank)

    # the first of each pair needs the larger workspace
    for caches, a, b in (((kvcache._WORKSPACES,), decode(4, 80), decode(3, 60)),
                         ((ops._WORKSPACES,), wgrad(3, 700, 1024, 512, 16), wgrad(2, 600, 512, 256, 8))):
        want = []
        for out, run in (a, b):
            run()
            torch.cuda.synchronize()
            want.append(out.clone())
            out.fill_(float("nan"))
        for cache in caches:
            cache.clear()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            a[1]()
        for ws in caches[0].values():
            ws.fill_(1)                      # what memory holds that nothing has cleared
        for out, run in (b, a):
            run()
        torch.cuda.synchronize()
        assert torch.equal(a[0], want[0]) and torch.equal(b[0], want[1])
        a[0].fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(a[0], want[0])


def test_device_ints_takes_what_torch_tensor_takes():
    from loquetier_b200 import ops
    for vals in ([True, False], [1.0, 2.0, -3.0], [torch.tensor(4), torch.tensor(5)], torch.tensor([6, 7]), (8, 9)):
        for dtype in (torch.int32, torch.int64):
            assert ops.device_ints(vals, dtype, DEV).tolist() == torch.tensor(list(vals), dtype=dtype).tolist()
    for bad, dtype in (([1 << 31], torch.int32), ([1 << 63], torch.int64), (["a"], torch.int32), ([None], torch.int32)):
        with pytest.raises((RuntimeError, TypeError, ValueError, OverflowError)) as want:
            torch.tensor(bad, dtype=dtype, device=DEV)
        with pytest.raises(want.type):
            ops.device_ints(bad, dtype, DEV)
