"""The tiled labeller at the extents where its tiles end (8 planes, 8 or 32 rows, 8 or 32
sites; 64 rows of a single plane; chunks of 8192 sites), open and periodic, below, at and above
the percolation threshold, and on one long winding path: label arrays equal to
scipy.ndimage.label's, joined across the boundary and renumbered in raster order when
periodic."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
ndimage = pytest.importorskip("scipy.ndimage")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import labels as LB  # noqa: E402

SHAPES = [(7, 9, 31), (8, 8, 32), (9, 17, 33), (17, 64, 8), (16, 33, 19), (5, 70, 20), (3, 2, 7),
          (1, 130, 65), (200, 130, 1), (300, 1, 1), (2, 2, 2), (33, 40, 97), (1, 64, 32),
          (64, 64, 2)]


def reference(mask, periodic):
    lab, n = ndimage.label(mask)
    if not periodic:
        return lab, n
    root = np.arange(n + 1)

    def find(x):
        while root[x] != x:
            x = root[x]
        return x
    for d in range(mask.ndim):
        a, b = np.take(lab, 0, d).ravel(), np.take(lab, -1, d).ravel()
        for u, v in set(zip(a.tolist(), b.tolist())):
            if u and v:
                u, v = find(u), find(v)
                root[max(u, v)] = min(u, v)
    flat = np.array([find(x) for x in range(n + 1)])[lab]
    roots = np.unique(flat[flat > 0])     # ordered by first voxel already
    new = np.zeros(n + 1, np.int64)
    new[roots] = np.arange(1, roots.size + 1)
    return new[flat], roots.size


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("density", [0.15, 0.33, 0.6, 1.0])
@pytest.mark.parametrize("periodic", [False, True])
def test_tiles_equal_scipy(shape, density, periodic):
    rng = np.random.default_rng(sum(shape))
    f = rng.uniform(0.0, 1.0, shape).astype(np.float32) * rng.choice([-1, 1], shape).astype(np.float32)
    thr = 1.0 - density - (0.1 if density == 1.0 else 0.0)
    ref, nref = reference(np.abs(f.astype(np.float64)) > thr, periodic)
    for t in (torch.from_numpy(f).cuda(), torch.from_numpy(f.astype(np.float64)).cuda()):
        lab, n = LB.label(t, thr, periodic=periodic)
        assert n == nref
        np.testing.assert_array_equal(lab.cpu().numpy(), ref)


@pytest.mark.parametrize("shape", [(1, 129, 200), (65, 1, 130), (90, 150, 1)])
def test_one_winding_path(shape):
    """Every second row masked, joined at alternating ends: one component."""
    f = np.zeros([n for n in shape if n > 1])
    f[::2] = 1.0
    f[1::4, -1] = 1.0
    f[3::4, 0] = 1.0
    f = f.reshape(shape)
    ref, nref = ndimage.label(f > 0.5)
    lab, n = LB.label(torch.from_numpy(f).cuda(), 0.5)
    assert n == nref
    np.testing.assert_array_equal(lab.cpu().numpy(), ref)
