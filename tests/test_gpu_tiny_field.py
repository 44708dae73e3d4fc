"""Complex fields smaller than the projection's floor of 1e-30 (C:2137-2150): V' is taken at
rho itself and only the division by rho is floored, so phi_a V'(rho) / 1e-30 has to keep its
quadratic fall.  One step without the Laplacian (inv_a2 = 0) against the oracle; tolerances as
the parity tests' (FP64 1e-13, float32 2e-6), relative to the result."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import complex_steps as OC  # noqa: E402
from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200._common import table_source  # noqa: E402

SHAPE = (4, 6, 8)
SIZES = [1e-29, 2e-30, 1.0000001e-30, 9.999999e-31, 3e-31, 1e-31, 1e-34, 1e-37]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("step", ["rk2", "overdamped"])
def test_below_the_floor(dtype, step):
    rng = np.random.default_rng(3)
    size = np.resize(np.array(SIZES), np.prod(SHAPE)).reshape(SHAPE)
    a = rng.uniform(0.0, 2.0 * np.pi, SHAPE)
    f = [torch.from_numpy(size * np.cos(a)).to(dtype), torch.from_numpy(size * np.sin(a)).to(dtype)]
    # V'(rho) = rho on a table from 0: the force is phi_a rho / 1e-30 below the floor
    n = 64
    tab = np.arange(n, dtype=np.float64)
    q1, q2 = (x.double().numpy() for x in f)
    ref = OC.table_force(tab, 0.0, 1.0, n)(q1, q2)
    g = [x.cuda() for x in f]
    t = torch.from_numpy(tab).cuda()
    if step == "rk2":
        z = [torch.zeros_like(x) for x in g]
        o = [torch.empty_like(x) for x in g + z]
        CF.rk2_step_table_into((*g, *z), o, 1.0, 1.0, 0.0, 1.0, 0.0, table_source(t, 0.0, 1.0, n))
        got = [-x.cpu().double().numpy() for x in o[2:]]
    else:
        CF.overdamped_euler_step_table(*g, 1.0, 1.0, 1.0, 1.0, 0.0, t, 0.0, 1.0, n, 0.0, 0)
        got = [q - x.cpu().double().numpy() for q, x in zip((q1, q2), g)]
    tol = 1e-13 if dtype == torch.float64 else 2e-6
    for x, r, q in zip(got, ref, (q1, q2)):
        # the overdamped step adds the force to the field, in the field's precision
        scale = np.abs(r) if step == "rk2" else np.abs(r) + np.abs(q)
        assert (np.abs(x - r) <= tol * scale + (1e-45 if dtype == torch.float32 else 0.0)).all()
