"""The inline thermal V' where its reciprocal-square-root form hands over to the one with the
clamps: zero and tiny fields and couplings (x = 0, x < 1e-20), a negative squared mass, arguments
beyond the splines, huge, infinite and NaN fields.  One FP64 step of isolated sites against the
formula (R:2228-2262) in numpy; tolerance 1e-11 of the result's size, as the fixtures' (the
spline's cubic cancels to about 1e-13 of its terms)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import thermal as OT  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402
from thermal_inflation_phase_transition_b200.thermal import ThermalPotential  # noqa: E402

T = 7350.0
CASES = {"script": (1.0e6, 1.09, 1.05, 1.09, 1.05), "massless": (0.0, 1.09, 0.0, 1.09, 0.0),
         "negative": (-4.0e5, 1.09, 0.0, 0.3, 0.2), "no fermion": (1.0e6, 1.09, 1.05, 0.0, 0.0)}


@pytest.mark.parametrize("form", ["inline", "field"])
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("policy", [1, 2])
def test_clamps(form, case, policy):
    from thermal_inflation_phase_transition_b200 import _lib as L
    bms, gb, gbg, gf, gfg = CASES[case]
    x = np.array([0.0, -0.0, 1e-30, -1e-25, 1e-18, 1e-12, 3.0, -500.0, 580.0, -581.0, 7350.0,
                  9.0e5, -9.6e5, 1.0e6, 1e8, -1e20, 1e60])
    phi = np.zeros((1, 8, 3 * 32))
    phi[0, 4, :3 * x.size:3] = x
    tp = ThermalPotential(device="cuda")
    kw = dict(lam=1e-24, mphi=1000.0, bosonMassSquared=bms, bosonCoupling=gb,
              bosonGaugeCoupling=gbg, fermionCoupling=gf, fermionGaugeCoupling=gfg)
    f = OT.vprime_inline if form == "inline" else OT.vprime_field
    with np.errstate(all="ignore"):
        ref = f(phi, T, tp.cb, tp.cf, 0.0, 100.0 / 255, **kw)
    # pi' of a step with inv_a2 = 0, h -> 0: pi' = -dt V'(phi) to O(dt^2 pi) = 0 at pi = 0
    p, v = torch.from_numpy(phi).cuda(), torch.zeros(phi.shape, dtype=torch.float64, device="cuda")
    po, vo = torch.empty_like(p), torch.empty_like(v)
    L.set_kernel_policy(policy)
    try:
        RF.rk2_step_table_into(p, v, po, vo, 1.0, 1.0, 0.0, 1.0, 0.0, tp.source(T, form=form, **kw))
    finally:
        L.set_kernel_policy(0)
    got = -vo.cpu().numpy()       # V' at phi + h1 pi = phi
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(got))
    scale = np.abs(phi) ** 3 * 1e-24 + np.abs(phi) * (1e6 + T * T) + 1e-300
    assert (np.abs(got - ref)[fin] <= 1e-11 * scale[fin]).all()


def test_bad_fields():
    phi = torch.full((4, 8, 32), 100.0, dtype=torch.float64, device="cuda")
    phi[1, 2, 3], phi[2, 5, 7] = float("nan"), float("inf")
    v = torch.zeros_like(phi)
    po, vo = torch.empty_like(phi), torch.empty_like(phi)
    src = ThermalPotential(device="cuda").source(T)
    RF.rk2_step_table_into(phi, v, po, vo, 1.0, 1.0, 0.0, 1.0, 0.0, src)
    bad = ~torch.isfinite(vo)
    # the two sites and, through the Laplacian (0 times a non-finite sum), their neighbours
    want = torch.zeros_like(bad)
    for i, j, k in ((1, 2, 3), (2, 5, 7)):
        want[i, j, k] = True
        for d in (-1, 1):
            want[(i + d) % 4, j, k] = want[i, (j + d) % 8, k] = want[i, j, (k + d) % 32] = True
    assert torch.equal(bad, want)
