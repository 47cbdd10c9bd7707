"""Batches of small grids through the table kernels, in source form or in stored populations by the rule on their
sizes and tau_h, against stepping each case alone: the same bits, over cases that step alone in between, a read of f, the
cooperative form and the autotuner."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_batch_streams import KINDS, _same, _solver  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _lib(built_lib):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _sets(grids, taus, dtype):
    return [[_solver(i % len(KINDS), g, dtype, t) for i, (g, t) in enumerate(zip(grids, taus))] for _ in range(2)]


SETS = {
    "source": ([(24, 24, 20), (30, 25, 33), (16, 16, 16)], [None] * 3),
    "tau mix": ([(24, 24, 20), (30, 25, 33), (16, 16, 16)], [None, 0.57, None]),
    "tau alone": ([(24, 24, 20), (30, 25, 33)], [0.57, 0.6]),
    "many small": ([(32, 32, 32)] * 31, [None] * 31),  # 1.02e6 nodes of a mean below 40,000
    "very many small": ([(32, 32, 32)] * 92, [None] * 92),  # 3.01e6: float in source form again
    "one too small": ([(96, 96, 64), (96, 64, 64), (24, 24, 24)], [None] * 3),  # of a mean for the streams
    "sizes apart": ([(96, 64, 32), (24, 24, 24), (17, 40, 21)], [None] * 3),
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("name", SETS)
def test_table_batch_matches_cases_alone(name, dtype):
    from lbm.batch import AllenCahnBatch
    alone, mixed = _sets(*SETS[name], dtype)
    for s in alone:
        s.run(16)
    b = AllenCahnBatch(mixed)
    for n in (1, 4, 1):
        b.run(n)
    for s in mixed:
        s.run(1)  # each alone: in source form where tau_h allows it
    b.run(3)
    assert mixed[0].f is not None
    b.set_cooperative(True)
    b.run(2)
    b.set_cooperative(False)
    b.autotune(reps=1)
    b.run(4)
    _same(alone, mixed)
    b.close()


def test_autotuners_leave_alone_what_reaches_no_kernel():
    """The nodes per thread of the phi pass over stored populations, in source form."""
    from lbm.batch import AllenCahnBatch
    s = _solver(0, (24, 24, 20), torch.float32)
    s.run(3)
    s.set_launch_shape(11, 128)
    s.autotune(reps=1)
    assert s.launch_shape()[0] == 11
    cases = [_solver(i, (24, 24, 20), torch.float32) for i in range(3)]
    b = AllenCahnBatch(cases)
    b.run(3)
    per = b.launch_shape()[0]
    for _ in range(4):
        assert b.autotune(reps=1)[0] == per
    b.close()


def test_cooperative_form_leaves_the_update_block_of_the_two_launches():
    from lbm.batch import AllenCahnBatch
    cases = [_solver(i, (24, 24, 20), torch.float32) for i in range(2)]
    b = AllenCahnBatch(cases)
    before = b.launch_shape()
    b.set_cooperative(True)
    assert b.launch_shape()[1] == 256
    b.run(2)
    b.autotune(reps=1)
    b.set_cooperative(False)
    assert b.launch_shape()[1] == before[1]
    b.run(2)
    b.close()
