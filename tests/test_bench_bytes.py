"""bench.py's algorithmic bytes per node of every form of the step, counted by hand."""
import bench


def test_bytes_per_node():
    a = bench.alg_bytes
    # source form: g, u, S, previous phi read and written, u and previous phi read by both kernels
    assert a("fp32") == (224, 33, 193)
    assert a("fp16") == (148, 33, 117)
    assert a("fp32", two_d=True) == (124, 25, 101)
    # stored populations (the paired layout, small or narrow 2-D grids)
    assert a("fp32", source=False) == (336, 81, 257)
    assert a("fp16", source=False) == (188, 47, 143)
    assert a("fp32", two_d=True, source=False) == (168, 41, 129)
    # one kernel
    assert a("fp32", fused=True) == (336, None, 337)
    assert a("fp16", fused=True) == (184, None, 185)
    # mu: 4 + 4, its gradient 4 + 12, both read again: 4 + 12; class bytes of the two kernels
    assert a("fp32", gmu=True) == (224 + 40, 33, 193 + 42)
    assert a("fp32", source=False, gmu=True) == (336 + 40, 81, 257 + 42)
    assert a("fp32", two_d=True, source=False, gmu=True) == (168 + 32 + 36, 41, 129 + 34 + 36)


def test_form_of_the_workloads():
    f = bench.source_form
    assert f(False, 150, 150 * 150 * 107, False, False) and f(False, 128, 128 ** 3, False, True)
    assert not f(False, 150, 150 * 150 * 108, True, False)
    assert f(True, 1024, 2048 * 1024, False, False) and not f(True, 1024, 2048 * 1024, False, True)
    assert not f(True, 255, 10 ** 6, False, False) and not f(True, 256, 699904, False, False)
