"""BAOAB and overdamped kernels on the column walk at the edges of its split: one plane, planes
that are no multiple of the chunk, rows shorter and longer than a block's 256 sites, more items
than resident blocks.  Against the oracle's simultaneous-update restatement."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import integrators as I  # noqa: E402
from oracle import oracle as O  # noqa: E402
from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

DEV = "cuda"
DT, DX, MU, IA2, GAMMA, ETA, NS = 0.05, 0.9, 1.1, 0.95, 0.8, 1.3, 0.3
SHAPES = [(1, 7, 5), (2, 3, 300), (3, 1, 1), (17, 16, 16), (35, 13, 21), (75, 64, 257)]
# the bounds of the integrators' own tests, for one step
TOL = {"f64": 1e-12, "f32": 3e-6, "f32c": 5e-6}


@pytest.fixture(autouse=True)
def generic():
    L.set_kernel_policy(1)
    yield
    L.set_kernel_policy(0)


def _dev(a, storage):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    if storage == "f32c":
        return RF.to_f32c(t)
    return t.float() if storage == "f32" else t


def _host(t, storage):
    if storage == "f32c":
        return RF.from_f32c(t).cpu().numpy()
    return t.double().cpu().numpy()


@pytest.mark.parametrize("storage", ["f64", "f32", "f32c"])
@pytest.mark.parametrize("shape", SHAPES)
def test_alt_steps(shape, storage):
    tab, tmin, dinv = O.build_table(lambda x: O.toy_vprime(x, 1.01), 0.0, 4.0, 2048)
    tabd = torch.from_numpy(tab).to(DEV)
    rng = np.random.default_rng(sum(shape))
    # exactly float32 start values, so that every storage starts where the oracle does
    f0 = [rng.normal(m, 0.5, shape).astype(np.float32).astype(np.float64)
          for m in (0.5, 0.4, 0.0, 0.1)]
    a = (MU, IA2, tab, tmin, dinv, 2048, NS, 3)
    d = (MU, IA2, tabd, tmin, dinv, 2048, NS, 3)
    want, got = [], []
    want.append(I.overdamped_step_table(f0[0], DT, DX, ETA, *a, seed=4))
    t = _dev(f0[0], storage)
    RF.overdamped_euler_step_table(t, DT, DX, ETA, *d, hash_seed=4)
    got.append(t)
    want += I.baoab_step_table(f0[0], f0[2], DT, DX, GAMMA, *a, seed=5)
    ts = [_dev(f0[0], storage), _dev(f0[2], storage)]
    RF.baoab_step_table(*ts, DT, DX, GAMMA, *d, hash_seed=5)
    got += ts
    want += I.complex_overdamped_step_table(f0[0], f0[1], DT, DX, ETA, *a, seed=6)
    ts = [_dev(x, storage) for x in f0[:2]]
    CF.overdamped_euler_step_table(*ts, DT, DX, ETA, *d, hash_seed=6)
    got += ts
    want += I.complex_baoab_step_table(*f0, DT, DX, GAMMA, *a, seed=7)
    ts = [_dev(x, storage) for x in f0]
    CF.baoab_step_table(*ts, DT, DX, GAMMA, *d, hash_seed=7)
    got += ts
    torch.cuda.synchronize()
    assert len(want) == len(got) == 9
    for t, r in zip(got, want):
        assert np.abs(_host(t, storage) - r).max() <= TOL[storage] * np.abs(r).max()
