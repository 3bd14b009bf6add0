"""Tensor memory is taken at run time and tcgen05.alloc blocks until columns are free, so a CTA that holds columns must
never wait for a CTA that may still be asking for them: two clusters that share two SMs in opposite order, or a launch and
its successor, would wait for each other for good.  Read off the kernels' sources, since the hang itself must not be run."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "aginfer_b200" / "csrc" / "kernels"
EVENTS = re.compile(r"\b(tmem_alloc|tmem_free|cluster_arrive|cluster_wait|grid_dependency_\w+)\(")


def body_events(name: str) -> list[str]:
    """The calls of interest of a kernel's body in source order (the bodies run straight down), without comments and
    without the definitions of the helpers."""
    source = re.sub(r"//[^\n]*", "", (KERNELS / name).read_text())
    source = re.sub(r"__device__ __forceinline__ \w+ \w+\([^\n]*\) \{[^\n]*(?:\n[^}\n]*;)*\n?\}", "", source)
    return [m.group(1) for m in EVENTS.finditer(source)]


@pytest.mark.parametrize("name", ["gemm_tk.cuh", "gemm_tc.cuh", "gemm_tc_persist.cuh", "gemm_tcs.cuh"])
def test_no_cta_waits_for_another_one_that_may_lack_tensor_memory(name):
    events = body_events(name)
    held = allocated = arrived_early = False
    for event in events:
        if event == "tmem_alloc":
            held = allocated = True
        elif event == "tmem_free":
            held = False
        elif event == "cluster_arrive":
            arrived_early = not allocated
        elif event == "cluster_wait":
            # allowed while holding: a barrier that every rank reaches without tensor memory of its own
            assert not held or arrived_early, f"{name}: cluster barrier with columns held"
        elif "release" in event or event == "grid_dependency_wait":
            # successors start (and may take columns) only when every CTA of this launch has its own
            assert allocated, f"{name}: successors released before the allocation"
    assert allocated and not held
