"""The generic stage's column walk at the shapes where it can go wrong: fewer than 256 sites a
plane and just more, one plane (2-D), more chunks than planes, rows of one site, slabs of planes
with a site offset -- every storage, both fields -- against the FP64 oracle and, for a slab,
against the whole lattice.  Tolerances as the parity tests': FP64 1e-13, float32 2e-6 and
compensated FP32 2e-6 (complex 5e-6) of the field's scale after one step."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402
from thermal_inflation_phase_transition_b200._common import (  # noqa: E402
    ptr, step_params, stream_handle, table_source)
from thermal_inflation_phase_transition_b200.slab import Slab  # noqa: E402

SHAPES = [(1, 1, 3), (2, 5, 51), (3, 16, 16), (33, 15, 17), (1, 257, 3), (40, 1, 257), (17, 255, 1),
          (150, 9, 31), (35, 37, 90)]
TOL = {"f64": 1e-13, "f32": 2e-6, "f32c": 2e-6}


@pytest.fixture(autouse=True)
def _generic():
    L.set_kernel_policy(1)
    yield
    L.set_kernel_policy(0)


def to(x, storage):
    t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    return t if storage == "f64" else (t.float() if storage == "f32" else RF.to_f32c(t))


def val(t):
    return (RF.from_f32c(t) if t.dim() == 4 else t.double()).cpu().numpy()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["f64", "f32", "f32c"])
def test_real(shape, storage):
    rng = np.random.default_rng(3)
    f = [rng.normal(0.5, 0.6, shape), rng.normal(0.0, 0.3, shape)]
    tab, tmin, dinv = O.build_table(lambda x: O.toy_vprime(x, 1.0), 0.0, 3.0, 4096)
    g = [to(x, storage) for x in f]
    a, b = (val(x).copy() for x in g)
    O.rk2_step_table(a, b, 0.05, 1.0, 1.0, 1.0, None, np.empty(shape), np.empty(shape), 1.0, tab,
                     tmin, dinv, 4096, noise_scale=0.3, noise_step=5)
    rng_ = RF.PhiRange()
    RF.rk2_step_table(*g, 0.05, 1.0, 1.0, 1.0, None, torch.empty_like(g[0]), torch.empty_like(g[1]),
                      1.0, torch.from_numpy(tab).cuda(), tmin, dinv, 4096, noise_scale=0.3,
                      noise_step=5, phi_range=rng_)
    for got, ref in ((val(g[0]), a), (val(g[1]), b)):
        assert np.abs(got - ref).max() <= TOL[storage] * max(1.0, np.abs(ref).max())
    lo, hi, bad = RF.PhiRange.decode(rng_.last.cpu())
    v = val(g[0])
    assert not bad and lo <= v.min() and hi >= v.max()
    assert lo >= np.nextafter(np.float32(v.min()), np.float32(-9)) and \
        hi <= np.nextafter(np.float32(v.max()), np.float32(9))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["f64", "f32", "f32c"])
def test_complex(shape, storage):
    rng = np.random.default_rng(4)
    f = [rng.normal(0.4, 0.5, shape) for _ in range(2)] + [rng.normal(0, 0.3, shape) for _ in range(2)]
    tab, tmin, dinv = O.build_table(lambda x: O.toy_vprime(x, 1.0), 0.0, 4.0, 4096)
    g = [to(x, storage) for x in f]
    ref = [val(x).copy() for x in g]
    O.rk2_step_table_complex(*ref, 0.05, 1.0, 1.0, 1.0, None, None, *(np.empty(shape) for _ in range(4)), 1.0, tab,
                             tmin, dinv, 4096, eps4=1e-3, noise_scale=0.3, noise_step=5)
    CF.rk2_step_table(*g, 0.05, 1.0, 1.0, 1.0, None, None, *[torch.empty_like(x) for x in g], 1.0,
                      torch.from_numpy(tab).cuda(), tmin, dinv, 4096, eps4=1e-3, noise_scale=0.3,
                      noise_step=5)
    tol = 5e-6 if storage == "f32c" else TOL[storage]
    for x, r in zip(g, ref):
        assert np.abs(val(x) - r).max() <= tol * max(1.0, np.abs(r).max())


@pytest.mark.parametrize("storage", ["f64", "f32c"])
def test_slab_planes(storage):
    nx, ny, nz = 37, 9, 30
    rng = np.random.default_rng(6)
    f = [to(rng.normal(0.5, 0.6, (nx, ny, nz)), storage), to(rng.normal(0, 0.3, (nx, ny, nz)), storage)]
    x = np.linspace(0.0, 3.0, 512)
    vs = table_source(torch.from_numpy(O.toy_vprime(x, 1.0)).cuda(), 0.0, 511 / 3.0, 512)
    out = [torch.empty_like(t) for t in f]
    RF.rk2_step_table_into(*f, *out, 0.05, 1.0, 1.0, 1.0, 1.0, vs, noise_scale=0.3, noise_step=2, seed=1)
    for r in range(2):
        sl = Slab((nx, ny, nz), rank=r, world=2)
        n, lo = sl.nx_local, sl.i_lo
        loc = [sl.scatter(t) for t in f] + [sl.empty(storage, "cuda") for _ in range(2)]
        L.call("tipt_rk2_step_table_slab", L.TIPT_F64 if storage == "f64" else L.TIPT_F32C,
               *[ptr(t) for t in loc], n, ny, nz, lo, nx,
               step_params(0.05, 1.0, 1.0, 1.0, 1.0, 0.3, 2, 1), vs, stream_handle())
        d = 1 if storage == "f32c" else 0
        for a, b in zip(loc[2:], out):
            assert torch.equal(sl.interior(a), b.narrow(d, lo, n))
