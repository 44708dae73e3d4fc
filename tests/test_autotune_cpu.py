"""What the autotuner times: the default call as the library takes it by itself, then every tile
shape on the marching kernel, each with its own planes and stages; the settings are restored."""
import pytest

torch = pytest.importorskip("torch")

from thermal_inflation_phase_transition_b200 import _lib as L  # noqa: E402
from thermal_inflation_phase_transition_b200 import autotune as AT  # noqa: E402


@pytest.mark.parametrize("field", ["real", "complex"])
def test_default_is_the_default_call(monkeypatch, field):
    now = {"policy": 0, "tiles": (9, 9, 5), "kseg": 7}    # left over from an earlier use
    timed = []
    monkeypatch.setattr(L, "set_kernel_policy", lambda p: now.update(policy=p))
    monkeypatch.setattr(L, "set_march_tiles", lambda *t: now.update(tiles=t))
    monkeypatch.setattr(L, "set_march_kseg", lambda k: now.update(kseg=k))
    monkeypatch.setattr(AT, "_state", lambda *a: None)

    def clock(*a):
        timed.append((now["policy"], now["tiles"], now["kseg"]))
        return 1.0 / len(timed)
    monkeypatch.setattr(AT, "_time", clock)
    shape = (64, 16, 256)
    res = AT.tune(shape, persist=False, device="cpu", field=field)
    assert timed[0] == (0, (0, 0, 0), 0) and res["default_ms"] == 1.0
    cands = AT.candidates(shape, field)
    assert [(t, k) for _, t, k in timed[1:]] == [(c[:3], c[3] if len(c) > 3 else 0) for c in cands]
    assert {p for p, _, _ in timed[1:]} == {2}
    assert now == {"policy": 0, "tiles": (0, 0, 0), "kseg": 0}
    assert res["best"] == list(cands[-1])
