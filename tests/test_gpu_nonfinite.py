"""Infinite and NaN momenta in float32 storage (beside denormal and signed-zero ones), with the
field itself finite: the midpoint phi~ = phi + h1 pi carries them to the six neighbours through
the Laplacian.  Non-finite outputs at the oracle's sites and nowhere else, the finite ones within
the parity tests' 2e-6 of the field's scale; the real field's kernels agree bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import oracle as O  # noqa: E402
from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

SHAPE = (8, 8, 32)
BAD = {"inf": np.inf, "-inf": -np.inf, "nan": np.nan, "denormal": 1e-42, "-0": -0.0}


def momentum(rng, bad):
    pi = rng.normal(0.0, 0.3, SHAPE).astype(np.float32)
    for site in ((0, 0, 0), (3, 4, 9), (6, 7, 31)):   # no common neighbours
        pi[site] = bad
    return pi


def check(got, ref):
    fin = np.isfinite(ref)
    assert np.array_equal(np.isfinite(got), fin)
    assert np.abs(got[fin] - ref[fin]).max() <= 2e-6 * max(1.0, np.abs(ref[fin]).max())


def same_bits(a, b):
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(
        torch.nan_to_num(a, nan=0.0).view(torch.int32), torch.nan_to_num(b, nan=0.0).view(torch.int32))


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("eta", [0.0, 1.0])
def test_real(bad, eta):
    rng = np.random.default_rng(8)
    phi = rng.normal(0.5, 0.6, SHAPE).astype(np.float32)
    pi = momentum(rng, BAD[bad])
    tab, tmin, dinv = O.build_table(lambda x: O.toy_vprime(x, 1.0), 0.0, 3.0, 4096)
    a, b = phi.copy(), pi.copy()
    tmp = [np.empty(SHAPE, np.float32) for _ in range(2)]
    O.rk2_step_table(a, b, 0.05, 1.0, eta, 1.0, None, *tmp, 1.0, tab, tmin, dinv, 4096)
    out = []
    for policy in (1, 2, 0):
        g = [torch.from_numpy(x).cuda() for x in (phi, pi)]
        L.set_kernel_policy(policy)
        try:
            RF.rk2_step_table(*g, 0.05, 1.0, eta, 1.0, None, *[torch.empty_like(x) for x in g], 1.0,
                              torch.from_numpy(tab).cuda(), tmin, dinv, 4096)
        finally:
            L.set_kernel_policy(0)
        for got, ref in zip(g, (a, b)):
            check(got.cpu().numpy(), ref)
        out.append(g)
    for g in out[1:]:
        assert same_bits(g[0], out[0][0]) and same_bits(g[1], out[0][1])


@pytest.mark.parametrize("bad", sorted(BAD))
@pytest.mark.parametrize("which", [0, 1])
def test_complex(bad, which):
    rng = np.random.default_rng(9)
    f = [rng.normal(0.4, 0.5, SHAPE).astype(np.float32) for _ in range(2)]
    m = [rng.normal(0.0, 0.3, SHAPE).astype(np.float32) for _ in range(2)]
    m[which] = momentum(rng, BAD[bad])
    f += m
    tab, tmin, dinv = O.build_table(lambda x: O.toy_vprime(x, 1.0), 0.0, 4.0, 4096)
    ref = [x.astype(np.float64) for x in f]
    O.rk2_step_table_complex(*ref, 0.05, 1.0, 1.0, 1.0, None, None, *(np.empty(SHAPE) for _ in range(4)),
                             1.0, tab, tmin, dinv, 4096, eps4=1e-3)
    g = [torch.from_numpy(x).cuda() for x in f]
    CF.rk2_step_table(*g, 0.05, 1.0, 1.0, 1.0, None, None, *[torch.empty_like(x) for x in g], 1.0,
                      torch.from_numpy(tab).cuda(), tmin, dinv, 4096, eps4=1e-3)
    for x, r in zip(g, ref):
        check(x.cpu().numpy().astype(np.float64), r)
