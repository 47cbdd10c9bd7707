"""Steps captured into a CUDA graph and replayed, against the same steps made by calls: whatever form the state had when
they were captured (stored populations right after the first step, else the source form), and whatever was done to it
between the replays: more steps, a read of f, a checkpoint restored, the fused kernel, the autotuner, new initial fields.
Batches of larger grids likewise, and captured read-outs of f and g."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_batch_streams import GRIDS, _sets  # noqa: E402
from test_gpu_read_populations import _equal, _solver  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _capture(s, n=2):
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.run(n)
    return g


def _same(a, b):
    for s in (a, b):
        s._cache.clear()  # a replay does not tell the solver
    for x, y in zip(a.fields("phi", "u", "P", "mu_phi") + [a.f, a.g], b.fields("phi", "u", "P", "mu_phi") + [b.f, b.g]):
        assert _equal(x, y)


CASES = [((18, 33), torch.float32), ((18, 33), torch.float64), ((18, 20), torch.float32),
         ((14, 17, 18), torch.float32), ((14, 17, 18), torch.float16), ((14, 17, 18), torch.float64)]


@pytest.mark.parametrize("warm", [1, 2, 3])
@pytest.mark.parametrize("grid,dtype", CASES)
def test_replays_between_other_calls(grid, dtype, warm):
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    a.run(warm)
    g = _capture(a)
    b.run(warm)
    for _ in range(2):
        g.replay()
        b.run(2)
    _same(a, b)  # reads f
    g.replay()
    b.run(2)
    _same(a, b)
    a.run(2)
    g.replay()
    b.run(4)
    _same(a, b)
    at = a.state_dict()
    g.replay()
    a.load_state_dict(at)
    g.replay()
    b.run(2)
    _same(a, b)
    a.run(1)
    a.run(1)
    b.run(2)
    _same(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_replays_around_the_fused_kernel_and_the_autotuner(dtype):
    grid = (14, 17, 18)
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    for s in (a, b):
        s.run(2)
    g = _capture(a)
    for s in (a, b):
        s.set_tile(4, 4, 9)
        s.run(2)
    fused = _capture(a)
    for s in (a, b):
        s.set_tile(0, 0, 0)
    g.replay()
    b.run(2)
    _same(a, b)
    fused.replay()
    b.set_tile(4, 4, 9)
    b.run(2)
    b.set_tile(0, 0, 0)
    _same(a, b)
    a.run(2)
    a.autotune(reps=1)
    a.set_tile(0, 0, 0)
    g.replay()
    b.run(4)
    _same(a, b)
    a.autotune(reps=1)  # of a state that the last replay left
    a.set_tile(0, 0, 0)
    a.run(2)
    b.run(2)
    _same(a, b)


@pytest.mark.parametrize("grid,dtype", [CASES[0], CASES[3], CASES[4]])
def test_replays_after_new_initial_fields(grid, dtype):
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    phi, u = a.phi.clone(), a.u.clone()
    a.run(2)
    g = _capture(a)
    g.replay()
    for s in (a, b):
        s.init_fields(phi, u)
        s.run(2)
    g.replay()
    b.run(2)
    _same(a, b)
    a.inject_droplet((5.0,) * len(grid), 3.0, 4.0)
    b.inject_droplet((5.0,) * len(grid), 3.0, 4.0)
    for s in (a, b):
        s.run(3)
    _same(a, b)


@pytest.mark.parametrize("grid,dtype", [((14, 17, 18), torch.float32), ((101, 97, 53), torch.float32),
                                        ((101, 97, 53), torch.float16), ((1831, 383), torch.float32)])
def test_replays_of_a_read_out(grid, dtype):
    a, b = _solver(grid, dtype), _solver(grid, dtype)
    for s in (a, b):
        s.run(3)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f, pg = a.f, a.g
    for stored in (False, True, False):
        if stored:
            a.load_state_dict(a.state_dict())  # populations from here to the next step
        else:
            for s in (a, b):
                s.run(2)
        f.fill_(float("nan"))
        g.replay()
        assert _equal(f, b.f) and _equal(pg, b.g)
        assert bool(torch.isfinite(f).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_replays_of_a_batch_on_streams(dtype):
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(GRIDS[:3], dtype)
    batch = AllenCahnBatch(mixed)
    batch.run(1)
    g = _capture(batch)
    for _ in range(2):
        g.replay()
    batch.run(2)
    for s in mixed:
        s._cache.clear()
        assert s.f is not None
    g.replay()
    torch.cuda.synchronize()
    for s in alone:
        s.run(9)
    for x, y in zip(alone, mixed):
        _same(x, y)
    batch.close()
