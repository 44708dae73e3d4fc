"""Blocks shared out inside the ensemble: the cluster that counts a replica (aligned and
misaligned slices, remainders of 16 bytes, one site, many passes) against numpy, and chunks
shared between blocks (chunk lengths from one block to many, odd extents) bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import ensemble as EN  # noqa: E402
from thermal_inflation_phase_transition_b200._common import ptr, stream_handle  # noqa: E402

SHAPES = [(1, 1, 1), (1, 1, 3), (1, 5, 7), (3, 16, 16), (1, 127, 129), (31, 33, 35), (64, 64, 64)]


@pytest.mark.parametrize("storage", ["f64", "f32c"])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_observe_counts(storage, shift):
    reps = (L.Replica * len(SHAPES))()
    off = shift
    for r, (a, b, c) in enumerate(SHAPES):
        reps[r] = L.Replica(a, b, c, 0, 0, 0, off, 0.0, 0.0, 0.0, 0.0, 0)
        off += a * b * c + (shift and r % 3)
    n_total = off + 5
    rng = np.random.default_rng(shift)
    val = rng.normal(1.0, 0.3, n_total)
    val[::97] = np.nan
    if storage == "f64":
        phi = torch.from_numpy(val).cuda()
        held = val
    else:
        hi = val.astype(np.float32)
        lo = np.where(np.isnan(val), np.float32(0), (val - hi).astype(np.float32))
        phi = torch.from_numpy(np.stack([hi, lo])).cuda()
        held = hi.astype(np.float64) + lo.astype(np.float64)
    R = len(SHAPES)
    dev_reps = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).cuda()
    active = torch.ones(R, dtype=torch.int32, device="cuda")
    n_active = torch.tensor([R], dtype=torch.int32, device="cuda")
    first = torch.full((R,), -1, dtype=torch.int64, device="cuda")
    frac = torch.full((R,), -1.0, dtype=torch.float64, device="cuda")
    L.call("tipt_ensemble_observe", L.TIPT_F64 if storage == "f64" else L.TIPT_F32C, ptr(phi),
           n_total, ptr(dev_reps), R, ptr(active), ptr(n_active), 1.0, 0.45, 0.5, 17, None, 0,
           ptr(first), ptr(frac), stream_handle())
    torch.cuda.synchronize()
    want = np.array([(held[q.offset:q.offset + q.n0 * q.n1 * q.n2] > 1.0).sum() /
                     float(q.n0 * q.n1 * q.n2) for q in reps])
    np.testing.assert_array_equal(frac.cpu().numpy(), want)
    np.testing.assert_array_equal(first.cpu().numpy(), np.where(want > 0.45, 17, -1))
    np.testing.assert_array_equal(active.cpu().numpy(), (want <= 0.5).astype(np.int32))
    assert int(n_active) == int((want <= 0.5).sum())


@pytest.mark.parametrize("storage", ["f64", "f32c"])
def test_shared_chunks(storage):
    """use_march off: every replica on the work-list; on: the 3-D classes on the
    work-list kernel, or under policy 2 on the marching stage; the graph's branches against one stream."""
    specs = [EN.ReplicaSpec(s, 1.0, 0.7, seed=n) for n, s in
             enumerate([(16, 16, 16), (31, 7, 9), (128, 128, 1), (50, 49, 1), (96, 32, 33)])]
    out = []
    for chunk, march, graphs, policy in (
            (1 << 20, False, False, 0), (8192, False, True, 0), (250, False, True, 0),
            (8192, True, True, 0), (8192, True, False, 0), (8192, True, True, 2),
            (8192, True, False, 2)):
        L.set_kernel_policy(policy)
        try:
            e = EN.Ensemble(specs, storage=storage, chunk_sites=chunk, use_march=march,
                            check_every=4, retire_frac=0.51, stop_frac=0.01)
            first = e.run(12, use_graphs=graphs)
        finally:
            L.set_kernel_policy(0)
        out.append((first, e.frac.cpu().numpy(), e.phi[0].clone(), e.pi[0].clone()))
    for o in out[1:]:
        np.testing.assert_array_equal(out[0][0], o[0])
        np.testing.assert_array_equal(out[0][1], o[1])
        for r in range(len(specs)):
            n, off = int(e.sizes[r]), int(e.offsets[r])
            for x, y in zip(out[0][2:], o[2:]):
                assert torch.equal(x[..., off:off + n], y[..., off:off + n])


@pytest.mark.parametrize("policy", [0, 2])
def test_class_skips_and_reports_misaligned_replica(policy):
    """A replica of a class whose offset is no multiple of 4 sites is left alone and reported,
    whichever kernel the class takes; the others step."""
    e = EN.Ensemble([EN.ReplicaSpec((8, 16, 64), 1.0, 0.05, seed=n) for n in range(3)],
                    storage="f32c", check_every=2)
    _, rids, act, n_act = e._march[0]
    reps = (L.Replica * 3).from_buffer_copy(e._reps.cpu().numpy().tobytes())
    reps[1].offset -= 1                     # inside the buffer
    bad = torch.frombuffer(bytearray(bytes(reps)), dtype=torch.uint8).cuda()
    out = []
    try:
        for table, entry in ((bad, "march"), (e._reps, "list")):
            phi, pi = torch.full_like(e.phi[0], -7.0), torch.full_like(e.pi[0], -7.0)
            args = (ptr(e.phi[0]), ptr(e.pi[0]), ptr(phi), ptr(pi), e.n_total, ptr(table))
            L.set_kernel_policy(policy)
            if entry == "march":
                L.call("tipt_ensemble_step_march", *args, ptr(rids), 3, None, 8, 16, 64,
                       ptr(e.active), e._sp, None, 0, stream_handle())
                assert L.device_status(clear=True) == 3  # TIPT_ERR_ALIGN
            else:
                chunks = (L.Chunk * 3)(*[L.Chunk(r, 8192, 0) for r in range(3)])
                dev = torch.frombuffer(bytearray(bytes(chunks)), dtype=torch.uint8).cuda()
                L.call("tipt_ensemble_step", L.TIPT_F32C, *args, ptr(dev), 3, ptr(e.active),
                       e._sp, None, 0, stream_handle())
            torch.cuda.synchronize()
            out.append((phi, pi))
    finally:
        L.set_kernel_policy(0)
        L.device_status(clear=True)
    for x, y in zip(*out):
        assert torch.equal(x[:, :8192], y[:, :8192]) and torch.equal(x[:, 16384:], y[:, 16384:])
        assert bool((x[:, 8192:16384] == -7.0).all())
