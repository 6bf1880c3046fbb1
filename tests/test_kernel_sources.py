"""Rules of the device code that no run on one GPU can show, read from the sources."""
import re
import subprocess
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


def test_function_attributes_are_set_for_each_device(tmp_path):
    """Dynamic shared memory above the default is allowed per device: no process-wide flag stands before it."""
    for path in sorted(CUDA.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"static bool \w+ = false;", text):
            assert "cudaFuncSetAttribute" not in text[m.end(): m.end() + 400], path.name
    (tmp_path / "once.cpp").write_text("""
        #include "once_per_device.h"
        #include <cstdio>
        int main() {
          nx::OncePerDevice once;
          int runs[66] = {0};
          auto work = [&](int d) { return ++runs[d] == 1 && d == 3 ? -2 : 0; };      // device 3 fails the first time
          const int devices[] = {0, 1, 0, 1, 3, 3, 3, 63, 63, 65, 65};
          for (int d : devices) std::printf("%d ", once(d, work));
          std::printf("| %d %d %d %d %d", runs[0], runs[1], runs[3], runs[63], runs[65]);
        }""")
    subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(tmp_path / "once"), str(tmp_path / "once.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "once")], check=True, capture_output=True, text=True).stdout
    assert out == "0 0 0 0 -2 0 0 0 0 0 0 | 1 1 2 1 2"
