"""The tcgen05 gradient at the edges of its 64-row tiles, against the mma.sync kernel: one row,
one less and one more than a tile and than two, several tiles, more tiles than SMs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from oracle import mlp as M  # noqa: E402
from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import surrogate as S  # noqa: E402


@pytest.mark.parametrize("rows", [1, 16, 63, 64, 65, 127, 129, 1000, 9601])
def test_gradient_tiles(rows):
    """Both kernels round the same operands to BF16 and accumulate in FP32; an accumulation
    order that differs can flip a BF16 rounding (2^-8 of one activation), so layers agree to
    2^-8 in norm and the losses, a few activations deep, to 2^-8 of their scale."""
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, 6)).astype(np.float32)
    t = rng.uniform(0.1, 1.0, (rows, M.TGT_COLS)).astype(np.float32)
    p = M.init_params(rows)
    lay, _ = M.layout()
    for (_, b, _, fo) in lay:
        p[b:b + fo] = rng.normal(0, 0.2, fo)
    p[lay[3][1] + 17:lay[3][1] + 32] = 0.0
    net = S.SurrogateNet(p)
    out = {}
    try:
        for pol in (1, 2):
            L.call("tipt_mlp_set_policy", pol)
            loss = torch.full((rows,), float("nan"), dtype=torch.float32, device="cuda")
            out[pol] = (net.grad(x, t, loss_rows=loss).clone(), loss)
    finally:
        L.call("tipt_mlp_set_policy", 0)
    (g1, l1), (g2, l2) = out[1], out[2]
    tol = 2.0 ** -8
    assert float((l1 - l2).abs().max()) <= tol * float(l1.abs().max())
    for (w, b, _, fo) in lay:
        for sl in (slice(w, b), slice(b, b + fo)):
            assert float((g1[sl] - g2[sl]).norm()) <= tol * float(g1[sl].norm())
    assert L.device_status(clear=True) == 0
