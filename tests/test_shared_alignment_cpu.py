"""Kernels read and clear dynamic shared memory in 16-byte vectors, and the
compiler places it behind a kernel's static arrays by its declared alignment: so
every declaration asks for 16 bytes or more."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencl-sdk_gb300", "csrc")


def test_dynamic_shared_memory_is_aligned():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            for number, line in enumerate(f, 1):
                if "extern __shared__" not in line:
                    continue
                found += 1
                m = re.search(r"extern __shared__ __align__\((\d+)\)", line)
                assert m and int(m[1]) >= 16, f"{name}:{number}: {line.strip()}"
    assert found > 10
