"""Rules on the CUDA sources that no single run can show broken."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "litetopk_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_dependent_launches_do_not_read_through_the_read_only_path():
    # a kernel that waits with pdl_wait() is alive while its predecessors still write: ld.global.nc
    # (__ldg) would take what they write to be constant
    files = [f for f in sorted(CSRC.glob("*.cu*")) if f.name != "common.cuh" and "pdl_wait()" in _code(f)]
    assert {f.name for f in files} >= {"attn_fp8.cu", "mla_bf16.cuh", "index_topk.cu", "prefill.cu", "union_qm.cu"}
    for f in files:
        assert "__ldg(" not in _code(f) and ".nc" not in _code(f), f.name


def test_a_kernels_shared_memory_limit_does_not_depend_on_the_call():
    # two threads that set a kernel's limit to their own sizes can leave it below what one of them has
    # recorded; every caller sets the same one
    calls = [c for f in sorted(CSRC.glob("*.cu*"))
             for c in re.findall(r"cudaFuncSetAttribute\(([^;{]*)", _code(f)) if "MaxDynamicSharedMemorySize" in c]
    assert calls
    for c in calls:
        assert not re.search(r"\b(bytes|dyn|smem)\b", c), c


def test_a_kernel_with_swizzled_tiles_rounds_or_checks_its_shared_memory_base():
    # the declared alignment of dynamic shared memory is no promise about its address at run time
    found = 0
    for f in sorted(CSRC.glob("*.cu*")):
        for body in _code(f).split("extern __shared__ __align__(1024)")[1:]:
            found += 1
            assert re.search(r"\+ 1023u?\) & ~1023u?|& 1023u?\) != 0\)", body[:900]), f.name
    assert found >= 5
