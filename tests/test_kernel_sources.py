"""Rules of the device code that no run on one GPU can show, read from the sources."""
import re
from pathlib import Path

CUDA = Path(__file__).resolve().parent.parent / "nexus_b200" / "csrc" / "cuda"


def _kernels():
    for path in sorted(CUDA.glob("*.cu")):
        text = path.read_text()
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            yield path.name, text[a:b]


def test_a_kernel_has_its_tensor_memory_before_it_lets_a_dependent_start():
    """A dependent that took tensor memory first would wait for the kernel in front, which waits for that memory."""
    seen = 0
    for name, body in _kernels():
        alloc = body.find("tmem_alloc(")
        trigger = [m.start() for m in re.finditer(r"pdl_launch_dependents\(\)|pdl_trigger\(\)", body)]
        if alloc >= 0 and trigger:
            seen += 1
            assert min(trigger) > body.index("__syncthreads();", alloc), name
    assert seen >= 5
