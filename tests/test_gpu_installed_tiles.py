"""An installed tile shape takes the automatic call to the marching kernel, also where the rule for
the automatic shapes takes the generic one (32^3): a withheld plane of the next marching launch
then expires (status 6), and without a shape it does not.  The results stay those of the generic
kernel, bit for bit, for both fields and the integrators."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402
from thermal_inflation_phase_transition_b200._common import poly_source  # noqa: E402

SHAPE = (32, 32, 32)
VS = poly_source(-0.2, 0.0, 0.3)


@pytest.fixture(autouse=True)
def _restore():
    yield
    L.test_withhold_plane(-1)
    L.set_march_tiles(0, 0, 0)
    L.device_status(clear=True)


def fields(n, storage="f32c"):
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    f = [torch.randn(SHAPE, dtype=torch.float64, device="cuda", generator=g) for _ in range(n)]
    return f if storage == "f64" else [x.float() if storage == "f32" else RF.to_f32c(x) for x in f]


def step(storage):
    f = fields(2, storage)
    o = [torch.empty_like(x) for x in f]
    RF.rk2_step_table_into(*f, *o, 0.05, 1.0, 1.0, 1.0, 1.0, VS, noise_scale=0.3, noise_step=1)
    torch.cuda.synchronize()
    return o


@pytest.mark.parametrize("tiles,status", [((0, 0, 0), 0), ((4, 0, 0), 6), ((0, 16, 0), 6), ((0, 0, 3), 6)])
def test_route(tiles, status):
    assert L.device_status(clear=True) == 0
    L.set_march_tiles(*tiles)
    L.test_withhold_plane(1)
    step("f32c")
    assert L.device_status(clear=True) == status


@pytest.mark.parametrize("tiles", [(4, 8, 3), (8, 5, 4)])
def test_same_bits(tiles):
    def runs():
        out = [x for st in ("f64", "f32", "f32c") for x in step(st)]
        c = fields(4)
        o = [torch.empty_like(x) for x in c]
        CF.rk2_step_table_into(c, o, 0.05, 1.0, 1.0, 1.0, 1.0, VS, eps4=1e-3, noise_scale=0.3)
        r = fields(2)
        RF.baoab_step_table(*r, 0.05, 1.0, 1.0, 1.0, 1.0, None, 0.0, 0.0, 0, 0.3, 2, vpoly=(-0.2, 0.0, 0.3))
        return out + o + r
    ref = runs()
    L.set_march_tiles(*tiles)
    for a, b in zip(runs(), ref):
        assert torch.equal(a, b)
