"""The step kernels read state arrays that the kernel before them in the stream writes while their own blocks may be
resident, and update u in place: ld.global.nc and __ldg, whose data has to stay unwritten while the kernel runs, have no
place in their loads, nor an asm statement that the compiler may move across the wait or a store."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pytorch-lbm_gb300", "csrc")
FILES = ("lbm_kernels.cu", "lbm_pair.cuh", "lbm_phis.cuh", "lbm_kernels2d.cu")


def _code(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def test_state_loads_are_coherent_and_ordered():
    for name in FILES:
        src = _code(name)
        assert "ld.global.nc" not in src, name
        # the case descriptors (written by a copy, in plain stream order) are all that __ldg reads
        ldg = re.findall(r"__ldg\(([^)]*)\)", src)
        assert ldg == (["a + i"] if name == "lbm_kernels.cu" else []), (name, ldg)
        loads = re.findall(r'asm( volatile)?\("(ld\.global[^"]*)"', src)
        assert all(vol for vol, _ in loads), [op for vol, op in loads if not vol]
