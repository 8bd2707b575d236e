"""The messages of device error words and the wait limit (octree-cuda_gb300/csrc/kernels.h, compiled with the host
compiler): every bit has a message, so that no failed build is taken for a good one."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PROGRAM = r"""
#include <cstdio>
#include "kernels.h"
int main() {
    for (int k = 0; k < 32; ++k) {
        const char* m = oc::device_error_message(1u << k);
        if (!m || !*m) return 1 + k;
    }
    if (oc::device_error_message(0)) return 40;
    // no unit is given less than a second; the largest cloud's limit does not wrap
    if (oc::unit_wait_limit(0, 0) < (1ll << 31) || oc::unit_wait_limit(0, 0xFFFFFFFFull) < (1ll << 41)) return 41;
    return oc::unit_wait_limit(oc::kDebugNoWait, 1000) < 0 ? 0 : 42;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.exists(CUDA_INC), reason="no host compiler or CUDA headers")
def test_every_error_bit_has_a_message(tmp_path):
    src = tmp_path / "errors.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "errors"
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "octree-cuda_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
