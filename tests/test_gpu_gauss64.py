"""The FP64 Box-Muller transform of the hash at the arguments where it can go wrong: keys whose
first uniform is 0, below and at the 1e-12 clamp, at every edge of the logarithm's table
intervals and next to 1 (the hash is inverted to find them), beside random keys; the cosine
through the key's z, both branches through the noise field.  Against 80-bit long double.

Tolerance: 4 ulp of z, from 0.75 ulp of -2 ln u1 (halved by the square root), 2 ulp of the
cosine (its argument is rounded once) and 0.5 ulp of the product; the 2-norm of the error over
random keys stays below 8.5e-17 of z's, what CUDA's log, sqrt and cos give."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402

M = (1 << 64) - 1


def unshift(y, k):
    x = y
    for _ in range(64 // k + 1):
        x = y ^ (x >> k)
    return x


def key_of(x):
    """The key whose first mix is x (u1 = (x >> 11) 2^-53)."""
    x = unshift(x, 31) * pow(0x94D049BB133111EB, -1, 1 << 64) & M
    x = unshift(x, 27) * pow(0xBF58476D1CE4E5B9, -1, 1 << 64) & M
    return unshift(x, 30)


def edge_keys():
    m1 = [0, 1, 2, 9006, 9007, 9008, 9009, (1 << 53) - 1, (1 << 53) - 2, (1 << 52), (1 << 52) - 1]
    for e in (14, 30, 52, 53):            # the table's interval edges, and below them
        m1 += [(q << (e - 8)) - d for q in range(128, 257) for d in (0, 1) if e > 8]
    rng = np.random.default_rng(2)
    low = rng.integers(0, 1 << 11, len(m1))
    return np.array([key_of((m % (1 << 53)) << 11 | int(b)) for m, b in zip(m1, low)], np.uint64)


def parts(u1, u2):
    r = np.sqrt(-2 * np.log(u1.astype(np.longdouble)))
    a = (6.283185307179586 * u2).astype(np.longdouble)
    return r * np.cos(a), r * np.sin(a)


def test_z_of_keys():
    rng = np.random.default_rng(1)
    keys = np.concatenate([edge_keys(), rng.integers(0, 1 << 63, 500000).astype(np.uint64)])
    u1, u2, z = (t.cpu().numpy() for t in RF.hash_rng_pair(torch.from_numpy(keys.view(np.int64)).cuda()))
    assert u1.min() == 1e-12 and u1.max() == 1 - 2.0 ** -53
    ref, _ = parts(u1, u2)
    err = np.abs((z - ref).astype(np.float64))
    assert (err / np.spacing(np.abs(ref.astype(np.float64)))).max() <= 4
    n = edge_keys().size
    assert np.linalg.norm(err[n:]) <= 8.5e-17 * np.linalg.norm(ref[n:].astype(np.float64))


@pytest.mark.parametrize("component", [0, 1])
def test_noise_field_branches(component):
    shape, step, mul = (61, 67, 65), 77, RF.K_PASS2
    out = torch.empty(shape, dtype=torch.float64, device="cuda")
    RF.generate_noise_field(out, 1.0, step, component=component)
    site = torch.arange(out.numel(), dtype=torch.int64, device="cuda")
    u1, u2, _ = (t.cpu().numpy() for t in RF.hash_rng_pair((site * mul) ^ step))
    ref = parts(u1, u2)[component]
    err = np.abs((out.cpu().numpy().ravel() - ref).astype(np.float64))
    assert (err / np.spacing(np.abs(ref.astype(np.float64)))).max() <= 4
    assert np.linalg.norm(err) <= 8.5e-17 * np.linalg.norm(ref.astype(np.float64))
