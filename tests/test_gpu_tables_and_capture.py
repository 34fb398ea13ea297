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
