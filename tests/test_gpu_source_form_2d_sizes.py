"""2-D grids on either side of the source form's size rule (700,000 nodes, 256 columns), with extents at the edges of the
phi pass's windows of columns (382 inner columns a block): stepping the state against stepping the stored populations that a
checkpoint holds; a read of f on another stream beside a step; captured steps."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_captured_steps import _capture  # noqa: E402
from test_gpu_captured_steps import _same as _same_fields  # noqa: E402
from test_gpu_read_populations import _equal, _same, _solver  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


@pytest.mark.parametrize("grid", [(2735, 256), (2734, 256), (2800, 255), (1840, 382), (1831, 383), (916, 765), (4, 180000),
                                  (3, 233335)])
def test_source_form_2d_matches_stored_populations(grid):
    a, b = _solver(grid, torch.float32), _solver(grid, torch.float32)
    for _ in range(4):
        a.run(1)
        b.run(1)
        f = a.f
        b.load_state_dict(b.state_dict())  # b holds populations from here
        assert _equal(f, b.f)
    assert torch.isfinite(a.phi).float().mean() > 0.9
    _same(a, b)


def test_reading_f_on_another_stream_beside_a_step():
    a, b = _solver((1831, 383), torch.float32), _solver((1831, 383), torch.float32)
    side = torch.cuda.Stream()
    for _ in range(4):
        a.run(2)
        b.run(2)
        want = b.f
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            f = a.f
        a.run(1)
        b.run(1)
        torch.cuda.synchronize()
        assert _equal(f, want)
    _same(a, b)


@pytest.mark.parametrize("warm", [1, 2])
def test_replays_between_other_calls(warm):
    a, b = _solver((1831, 383), torch.float32), _solver((1831, 383), torch.float32)
    a.run(warm)
    g = _capture(a)
    b.run(warm)
    g.replay()
    g.replay()
    b.run(4)
    _same_fields(a, b)
    a.run(2)
    g.replay()
    at = a.state_dict()
    g.replay()
    a.load_state_dict(at)
    g.replay()
    b.run(6)
    _same_fields(a, b)
