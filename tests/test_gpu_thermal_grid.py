"""The inline thermal V' on spline grids that start below zero, at arguments next to their top:
there x - x_min rounds to the grid's whole length and only the clamp keeps the segment inside the
splines.  (The unclamped segment of these arguments is checked to be nseg.)  One FP64 step of
isolated sites against the formula in numpy; tolerance 1e-9 of the result's size, from the
cubic's terms (|x - x_i| < 1.3e6 known to 1e-10, coefficients of order 1 in (x - x_i) / h)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import thermal as OT  # noqa: E402
from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

T = 7350.0
X_MIN, H, NSEG = -6484841.752939573, 1296969.4245733782, 5
KW = dict(lam=0.0, mphi=0.0, bosonMassSquared=0.0, bosonCoupling=1.0, bosonGaugeCoupling=0.0,
          fermionCoupling=1.0, fermionGaugeCoupling=0.0)


@pytest.mark.parametrize("form", [0, 1])
def test_top_of_a_grid_from_below_zero(form):
    top = X_MIN + H * NSEG
    x = top * (1.0 - np.array([2e-12, 1e-11, 1e-9, 1e-6, 0.1, 0.5, -1e-13, -1e-9, -0.5]))
    # x_f = phi / (sqrt(2) T) and x_b = sqrt(phi^2 / 2 + T^2 / 4) / T: the fermion's argument is x,
    # and the boson's for the second half of the fields
    ph = np.concatenate([np.sqrt(2.0) * T * x, np.sqrt(2.0 * np.maximum((x * T) ** 2 - T * T / 4, 0.0))])
    assert int((x[0] - X_MIN) * (1.0 / H)) == NSEG
    phi = np.zeros((1, 8, 3 * 32))
    phi[0, 4, :3 * ph.size:3] = ph
    rng = np.random.default_rng(4)
    cb, cf = (rng.normal(size=(4, NSEG)) / H ** np.array([3, 2, 1, 0])[:, None] for _ in range(2))
    spl = torch.from_numpy(np.ascontiguousarray(np.concatenate([cb, cf]))).cuda()
    th = L.Thermal(0.0, 0.0, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, 1.0, X_MIN, H, NSEG, form, spl.data_ptr())
    src = L.VSource(L.VP_THERMAL, 0, None, 0.0, 0.0, 0, 0, 0.0, 0.0, T, 0.0, 0.0, 0.0, C.addressof(th))
    f = OT.vprime_field if form else OT.vprime_inline
    ref = f(phi, T, cb, cf, X_MIN, H, **KW)
    p = torch.from_numpy(phi).cuda()
    v, po, vo = (torch.zeros_like(p) for _ in range(3))
    for policy in (1, 2):
        L.set_kernel_policy(policy)
        try:
            RF.rk2_step_table_into(p, v, po, vo, 1.0, 1.0, 0.0, 1.0, 0.0, src)
        finally:
            L.set_kernel_policy(0)
        got = -vo.cpu().numpy()
        scale = T ** 4 / (2 * np.pi ** 2) * np.abs(phi) / (T * T) + 1e-300
        assert (np.abs(got - ref) <= 1e-9 * scale).all()
