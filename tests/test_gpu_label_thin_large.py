"""Thin lattices with more tiles of the usual shapes than are resident at once: the tile shapes made
for them, one lattice at least per shape and past its end, against scipy.ndimage.label."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
ndimage = pytest.importorskip("scipy.ndimage")

pytestmark = pytest.mark.gpu

from test_gpu_label_tiles import reference  # noqa: E402
from thermal_inflation_phase_transition_b200 import labels as LB  # noqa: E402

SHAPES = [(1, 1, 50001), (60000, 1, 1), (1, 3, 40100), (5, 1, 40050), (2, 2, 45000), (3, 2, 41000),
          (11000, 1, 40), (10500, 1, 5), (1, 80001, 2), (10400, 3, 4), (3, 40010, 4), (10300, 2, 19)]


@pytest.mark.parametrize("shape", SHAPES)
def test_thin(shape):
    rng = np.random.default_rng(sum(shape))
    for n, density in enumerate((0.1, 0.55, 0.9, 1.0)):
        periodic = bool(n & 1)
        f = rng.uniform(0.1, 1.0, shape) * np.where(rng.uniform(size=shape) < density, 1.0, 0.05)
        t = torch.from_numpy(f).cuda()
        lab, cnt = LB.label(t if n % 2 else t.float(), 0.08, periodic=periodic)
        ref, nref = reference(np.abs(f if n % 2 else f.astype(np.float32)) > 0.08, periodic)
        assert cnt == nref
        assert np.array_equal(lab.cpu().numpy(), ref)
