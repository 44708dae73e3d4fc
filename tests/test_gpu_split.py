"""The marching kernels' equal shares of the work against the generic kernel, bit for bit, at
shapes where a CTA's share is less than a plane run, spans several tiles, or ends inside one;
beside them shapes that keep the round-robin items.  Every storage, the thermal source, both
fields and the integrators."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

# (planes, rows, row length): few units; many short tiles; long runs; 300+ items
SHAPES = [(3, 8, 32), (5, 96, 64), (70, 16, 64), (61, 64, 128), (33, 4, 512), (150, 12, 256),
          (40, 512, 32), (1, 256, 64)]


@pytest.fixture(autouse=True)
def _restore():
    yield
    L.set_kernel_policy(0)


def state(shape, storage, n, seed=5):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f = [torch.randn(shape, dtype=torch.float64, device="cuda", generator=g).mul_(0.6).add_(0.3)
         for _ in range(n)]
    if storage == "f64":
        return f
    return [x.float() if storage == "f32" else RF.to_f32c(x) for x in f]


def table():
    x = np.linspace(0.0, 3.0, 1024)
    return torch.from_numpy(0.1 * x ** 3 - 0.147 * x ** 2 - 0.01 * x).cuda(), 0.0, 1023 / 3.0, 1024


def both(run):
    out = []
    for policy in (1, 2):
        L.set_kernel_policy(policy)
        out.append(run())
    torch.cuda.synchronize()
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert L.device_status() == 0


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["f64", "f32", "f32c"])
def test_real_step(shape, storage):
    def run():
        f = state(shape, storage, 2)
        t = [torch.empty_like(x) for x in f]
        for n in range(2):
            RF.rk2_step_table(*f, 0.05, 1.0, 1.0, 1.0, None, *t, 1.0, *table(), noise_scale=0.3,
                              noise_step=n, seed=2)
        return f
    both(run)


@pytest.mark.parametrize("shape", SHAPES[:6])
@pytest.mark.parametrize("storage", ["f64", "f32", "f32c"])
def test_real_thermal(shape, storage):
    def run():
        f = state(shape, storage, 2)
        t = [torch.empty_like(x) for x in f]
        RF.rk2_fused_single_pass(*f, 0.05, 1.0, 1.0, 7350.0, 7349.0, 1000.0, 1e-24, 1000.0, 1e6,
                                 1.09, 1.05, 1.09, 1.05, 0.3, 4, *t, 1.0)
        return f
    both(run)


@pytest.mark.parametrize("shape", SHAPES)
def test_complex_step(shape):
    def run():
        f = state(shape, "f32c", 4)
        t = [torch.empty_like(x) for x in f]
        for n in range(2):
            CF.rk2_step_table(*f, 0.05, 1.0, 1.0, 1.0, None, None, *t, 1.0, *table(), eps4=1e-3,
                              noise_scale=0.3, noise_step=n, seed=2)
        return f
    both(run)


@pytest.mark.parametrize("shape", SHAPES[:6])
@pytest.mark.parametrize("method", ["overdamped", "baoab"])
def test_integrators(shape, method):
    def real():
        f = state(shape, "f32c", 2)
        if method == "baoab":
            RF.baoab_step_table(*f, 0.05, 1.0, 1.0, 1.0, 1.0, *table(), 0.3, 3)
            return f
        RF.overdamped_euler_step_table(f[0], 0.05, 1.0, 1.0, 1.0, 1.0, *table(), 0.3, 3)
        return f[:1]

    def cplx():
        f = state(shape, "f32c", 4)
        if method == "baoab":
            CF.baoab_step_table(*f, 0.05, 1.0, 1.0, 1.0, 1.0, *table(), 0.3, 3)
            return f
        CF.overdamped_euler_step_table(*f[:2], 0.05, 1.0, 1.0, 1.0, 1.0, *table(), 0.3, 3)
        return f[:2]
    both(real)
    both(cplx)
