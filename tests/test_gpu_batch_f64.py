"""Batches of float64 grids against stepping each case alone: the same bits, scalars included (the sum of phi, and with
it the mass correction, is rounded per block of a case)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_batch_streams import _same, _sets  # noqa: E402

GRIDS = [(24, 24, 20), (40, 33, 27), (51, 47, 49)]


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


@pytest.mark.parametrize("coop", [True, False])
def test_float64_batch_matches_cases_alone(coop):
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(GRIDS, torch.float64)
    b = AllenCahnBatch(mixed)
    b.set_cooperative(coop)
    for n in (1, 4):
        b.run(n)
    for s in alone:
        s.run(5)
    for s in (alone[1], mixed[1]):
        s.set_launch_shape(1, 128)  # of a case's own: the batch follows it
    b.run(2)
    b.autotune(reps=1)
    b.run(2)
    for s in alone:
        s.run(4)
    _same(alone, mixed)
    b.close()
