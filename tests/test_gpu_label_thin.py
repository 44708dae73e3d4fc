"""The labeller's tiles for lattices that are thin in two directions (rows of several 32-site
segments, or many short rows), one lattice at least per tile shape and past its end, open and
periodic, from sparse masks to full ones: label arrays equal to scipy.ndimage.label's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytest.importorskip("scipy.ndimage")

pytestmark = pytest.mark.gpu

from test_gpu_label_tiles import reference  # noqa: E402
from thermal_inflation_phase_transition_b200 import labels as LB  # noqa: E402

SHAPES = [(1, 1, 5000), (5000, 1, 1), (1, 4100, 1), (1, 3, 3000), (3, 3000, 1), (1, 8, 1025),
          (5, 1, 2000), (2, 1, 4500), (2, 2, 3000), (3, 2, 1600), (500, 1, 40), (3000, 1, 5),
          (1, 3000, 3), (3000, 2, 1), (900, 3, 4), (3, 700, 4), (2000, 2, 2), (1, 1, 2), (600, 1, 19),
          (1, 1, 2048), (2, 1, 20)]


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_thin(shape, periodic):
    rng = np.random.default_rng(sum(shape))
    for n, density in enumerate((0.1, 0.4, 0.6, 0.85, 0.97, 1.0)):
        f = rng.uniform(0.1, 1.0, shape) * np.where(rng.uniform(size=shape) < density, 1.0, 0.05)
        t = torch.from_numpy(f).cuda()
        lab, cnt = LB.label(t if n % 2 else t.float(), 0.08, periodic=periodic)
        ref, nref = reference(np.abs(f if n % 2 else f.astype(np.float32)) > 0.08, periodic)
        assert cnt == nref
        assert np.array_equal(lab.cpu().numpy(), ref)
