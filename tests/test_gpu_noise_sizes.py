"""The noise field's one-site and two-site launches give the same numbers: prefixes of one field
of 1024 x 200 x 2 sites, at the sizes where the launch changes (1024 sites an SM) and at the
smallest, both storages and components."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from thermal_inflation_phase_transition_b200 import real_field as RF  # noqa: E402


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("component", [0, 1])
def test_prefixes(dtype, component):
    def field(n):
        t = torch.full((1, 1, n), float("nan"), dtype=dtype, device="cuda")
        RF.generate_noise_field(t, 0.5, 9, component=component)
        return t.view(-1)
    line = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    whole = field(2 * line + 77)
    assert bool(torch.isfinite(whole).all())
    for n in (1, 2, 255, 257, line - 1, line, line + 1, line + 255, 2 * line):
        assert torch.equal(field(n), whole[:n])
