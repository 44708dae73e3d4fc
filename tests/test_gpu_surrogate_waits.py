"""An expired wait in any warp of the surrogate's tcgen05 kernels is reported: the block leaves
together, the device status reads TIPT_ERR_TIMEOUT (6) whichever warp it was, and the next
launch gives the usual result."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import surrogate as S  # noqa: E402


@pytest.mark.parametrize("warp", [1, 7])
@pytest.mark.parametrize("call", ["forward", "grad"])
def test_reported(warp, call):
    assert L.device_status(clear=True) == 0
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    net = S.SurrogateNet()
    x = torch.randn(200, 6, device="cuda", generator=g)
    t = torch.rand(200, 20, device="cuda", generator=g)
    run = (lambda: net.forward(x)) if call == "forward" else (lambda: net.grad(x, t))
    ref = run().clone()
    L.test_expire_wait(warp)
    run()
    torch.cuda.synchronize()
    assert L.device_status(clear=True) == 6
    assert torch.equal(run(), ref)
    assert L.device_status() == 0
