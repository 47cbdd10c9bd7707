"""Batches of larger grids, whose cases step through the kernels of a grid alone on several streams, against
stepping each case alone: bit-identical phi, u, populations and scalars.  More cases than streams and fewer, a
tau_h != 1 case, a mean extent on either side of the size rule, a caller's stream, and a change to the cooperative
form and back; the batch autotuner leaves the state unchanged."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from lbm.impact import ImpactCase, impact_config, impact_inputs  # noqa: E402

GRIDS = [(48, 48, 48), (64, 48, 40), (40, 61, 47), (96, 40, 32), (51, 47, 49), (50, 46, 50)]
KINDS = ["flat", "ridge", "convex", "concave", "ridge", "flat"]


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return built_lib


def _solver(i, grid, dtype, tau_h=None):
    from lbm.fe_ac_solver import AllenCahnSolver
    case = ImpactCase(i, grid, KINDS[i], 7.0, 100.0 + 12.0 * i, -0.04, 0)
    cfg = impact_config(case, "cuda")
    if tau_h is not None:
        cfg.tau_h = tau_h
    solid, frac, C, u = impact_inputs(case)
    s = AllenCahnSolver(cfg, dtype=dtype, geo_amplification=1.5, geometric_wetting=True)
    s.set_solid(solid, frac)
    s.init_fields(C, u)
    return s


def _sets(grids, dtype, n=2):
    taus = [None, 0.57, None, None, None, None]
    return [[_solver(i, g, dtype, taus[i]) for i, g in enumerate(grids)] for _ in range(n)]


def _same(a, m):
    for x, y in zip(a, m):
        assert torch.equal(x.phi, y.phi) and torch.equal(x.u, y.u)
        assert torch.equal(x.f, y.f) and torch.equal(x.g, y.g)
        assert x.scalars() == y.scalars()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("grids", [GRIDS, GRIDS[:1], GRIDS[:3], [(47, 47, 47), (48, 48, 48)]],
                         ids=["six", "one", "three", "below"])
def test_batch_on_streams_matches_cases_alone(dtype, grids):
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(grids, dtype)
    for s in alone:
        s.run(8)
    b = AllenCahnBatch(mixed)
    for n in (1, 4, 3):
        b.run(n)
    _same(alone, mixed)
    b.close()


def test_batch_on_streams_orders_with_the_callers_stream():
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(GRIDS[:3], torch.float32)
    b = AllenCahnBatch(mixed)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    for s in alone:
        s.run(7)
    b.run(3, stream=st)
    mixed[0].run(2, stream=st)  # a case alone between two batch calls
    alone[0].run(2)
    b.run(4, stream=st)
    torch.cuda.current_stream().wait_stream(st)
    _same(alone, mixed)


def test_batch_on_streams_changes_to_the_cooperative_form_and_back():
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(GRIDS[:3], torch.float32)
    for s in alone:
        s.run(9)
    b = AllenCahnBatch(mixed)
    b.run(3)
    b.set_cooperative(True)
    b.run(2)
    b.set_cooperative(False)
    b.run(1)
    per, ms = b.autotune(reps=2)
    assert per in (1, 2, 4, 8, 12, 16, 24, 32) and ms > 0
    b.run(3)
    _same(alone, mixed)
