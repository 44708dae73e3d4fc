"""The ensemble's count of converted sites on single blocks (small replicas; middling ones, many of
them) and on clusters (few middling ones), aligned and misaligned slices, against numpy."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200._common import ptr, stream_handle  # noqa: E402

# replicas' extents: small and uneven; 320 and 20 of about 20,000 sites
SETS = {"small": [(1, 1, 1), (1, 3, 5), (8, 8, 8), (1, 128, 128), (1, 97, 101), (17, 16, 15)] * 40,
        "many": [(20, 31, 33)] * 320, "few": [(20, 31, 33)] * 20}


@pytest.mark.parametrize("storage", ["f64", "f32c"])
@pytest.mark.parametrize("name", sorted(SETS))
@pytest.mark.parametrize("pad", [0, 1])
def test_counts(storage, name, pad):
    shapes = SETS[name]
    reps = (L.Replica * len(shapes))()
    off = 0
    for r, (a, b, c) in enumerate(shapes):
        reps[r] = L.Replica(a, b, c, 0, 0, 0, off, 0.0, 0.0, 0.0, 0.0, 0)
        off += a * b * c + (r % 3 if pad else -(a * b * c) % 4)
    n_total = off
    rng = np.random.default_rng(7)
    val = rng.normal(1.0, 0.3, n_total)
    val[::97] = np.nan
    if storage == "f64":
        phi, held = torch.from_numpy(val).cuda(), val
    else:
        hi = val.astype(np.float32)
        lo = np.where(np.isnan(val), np.float32(0), (val - hi).astype(np.float32))
        phi = torch.from_numpy(np.stack([hi, lo])).cuda()
        held = hi.astype(np.float64) + lo.astype(np.float64)
    R = len(shapes)
    dev_reps = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).cuda()
    active = torch.ones(R, dtype=torch.int32, device="cuda")
    n_active = torch.tensor([R], dtype=torch.int32, device="cuda")
    first = torch.full((R,), -1, dtype=torch.int64, device="cuda")
    frac = torch.full((R,), -1.0, dtype=torch.float64, device="cuda")
    L.call("tipt_ensemble_observe", L.TIPT_F64 if storage == "f64" else L.TIPT_F32C, ptr(phi),
           n_total, ptr(dev_reps), R, ptr(active), ptr(n_active), 1.0, 0.49, 0.5, 17, None, 0,
           ptr(first), ptr(frac), stream_handle())
    torch.cuda.synchronize()
    want = np.array([(held[q.offset:q.offset + q.n0 * q.n1 * q.n2] > 1.0).sum() /
                     float(q.n0 * q.n1 * q.n2) for q in reps])
    np.testing.assert_array_equal(frac.cpu().numpy(), want)
    np.testing.assert_array_equal(first.cpu().numpy(), np.where(want > 0.49, 17, -1))
    np.testing.assert_array_equal(active.cpu().numpy(), (want <= 0.5).astype(np.int32))
    assert int(n_active) == int((want <= 0.5).sum())
