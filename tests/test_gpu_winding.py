"""Winding kernels at the sizes and values where they can go wrong: widths around the
31-column warps and the 24-site switch between the two kernels, row and plane remainders, and
edges whose phase difference is +-pi to the last bit, zero, signed zero, tiny, huge or NaN
(the FP32 cross product must leave those to the phases).  Integers: equal to the wrap rule
d - 2 pi m of C:2683-2744 on FP64 phases of the same atan2 (its last bit decides these edges)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import complex_field as CF  # noqa: E402
from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

SHAPES = [(17, 5, 24), (16, 4, 31), (33, 7, 32), (5, 9, 62), (1, 6, 63), (3, 1, 40), (2, 2, 25),
          (20, 18, 23), (18, 17, 7), (40, 70, 1), (1, 1, 64), (4, 3, 96)]


def hard_fields(shape, seed):
    """Smooth strings with exactly opposite, aligned, zero and extreme neighbours sown in."""
    rng = np.random.default_rng(seed)
    a, b = (rng.standard_normal(shape).astype(np.float32).astype(np.float64) for _ in range(2))
    fa, fb = a.reshape(-1), b.reshape(-1)
    n = fa.size
    for q in range(0, n - 1, 3):
        kind = (q // 3) % 12
        s = np.float32(rng.uniform(0.25, 4.0))
        if kind == 0:        # exactly opposite: the difference is +-pi, rounded
            fa[q + 1], fb[q + 1] = -fa[q], -fb[q]
        elif kind == 1:      # opposite up to a scale that rounds
            fa[q + 1], fb[q + 1] = np.float32(-s * fa[q]), np.float32(-s * fb[q])
        elif kind == 2:      # on the cut
            fa[q], fb[q] = -abs(fa[q]), 0.0
        elif kind == 3:
            fa[q], fb[q] = -abs(fa[q]), -0.0
        elif kind == 4:
            fa[q], fb[q] = abs(fa[q]), -0.0
        elif kind == 5:
            fa[q], fb[q] = 0.0, 0.0
        elif kind == 6:
            fa[q], fb[q] = -0.0, -0.0
        elif kind == 7:      # next to the cut
            fa[q], fb[q], fa[q + 1], fb[q + 1] = 1.0, 1e-30, -1.0, -1e-20
        elif kind == 8:
            fa[q] *= 1e-25
            fb[q] *= 1e-25
        elif kind == 9:
            fa[q] *= 1e25
            fb[q] *= 1e25
        elif kind == 10:
            fb[q + 1] = np.nextafter(np.float32(-fb[q]), np.float32(0.0))
            fa[q + 1] = -fa[q]
        elif kind == 11 and q % 2:
            fa[q] = np.nan
    return a, b


def by_phases(phi1, phi2):
    """(site windings, int8 windings of the XY, XZ, YZ plaquettes) from every phase."""
    th = torch.atan2(phi2, phi1)

    def wrap(d):
        return (d > np.pi).to(torch.int8) - (d < -np.pi).to(torch.int8)
    e = [wrap(th.roll(-1, d) - th) for d in range(3)]
    w3 = torch.stack([-(e[p] + e[q].roll(-1, p) - e[p].roll(-1, q) - e[q])
                      for p, q in ((0, 1), (0, 2), (1, 2))])
    return w3.sum(0).float(), w3


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("storage", ["f32", "f64", "f32c"])
def test_winding_hard_edges(shape, storage):
    a, b = hard_fields(shape, shape[2])
    with np.errstate(invalid="ignore"):
        a, b = a.astype(np.float32).astype(np.float64), b.astype(np.float32).astype(np.float64)
        if storage == "f64":    # values that FP32 rounds (exactly opposite ones stay so)
            a, b = a * (1 + 2.0 ** -40), b * (1 + 2.0 ** -40)
    ta, tb = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    if storage == "f32c":       # hi + lo of a zero is +0
        w, w3 = by_phases(ta + 0.0, tb + 0.0)
    else:
        w, w3 = by_phases(ta, tb)
    w, w3 = w.cpu().numpy(), w3.cpu().numpy()
    if storage == "f32":
        ta, tb = ta.float(), tb.float()
    elif storage == "f32c":
        ta, tb = RF.to_f32c(ta), RF.to_f32c(tb)
    r = CF.compute_winding_number_full(ta, tb, pierced_cap=3 * a.size)
    assert np.array_equal(r.w_site.cpu().numpy(), w)
    assert np.array_equal(r.w3.cpu().numpy(), w3)
    assert r.counts.tolist()[:4] == [int((w3[o] != 0).sum()) for o in range(3)] + [int((w != 0).sum())]
    listed = np.sort(r.pierced[:r.counts[4]].cpu().numpy().view(np.uint32))
    o, s = np.nonzero(w3.reshape(3, -1))
    assert np.array_equal(listed, np.sort((s * 3 + o).astype(np.uint32)))
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    assert np.array_equal(CF.compute_winding_number(ta, tb, out).cpu().numpy(), w)
