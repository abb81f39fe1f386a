"""The calls that keep temporary device memory between calls, before and after cudaDeviceReset: the same
results, and what was kept under the context that is gone is given back. tests/workspace_harness.cu (the
library's source included whole, built with nvcc) runs in a process of its own, whose device state the reset ends."""
import ctypes
import json
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
SOURCE = HERE / "workspace_harness.cu"
CSRC = HERE.parent / "sadcs_b200" / "csrc"
BUILT = HERE / "_build" / "libworkspace_harness.so"

# A run of one character: its suffix array and LCP array are known, and the calls keep memory (12n bytes).
CHILD = """
import ctypes, json, sys
import numpy as np

library = ctypes.CDLL(sys.argv[1])
n, resets = 32 << 20, 2
text = np.full(n, 97, np.uint8)
sa = np.arange(n - 1, -1, -1, dtype=np.uint32)
lcp, bwt = np.zeros(n, np.uint32), np.zeros(n, np.uint8)
left = np.zeros(resets + 2, np.int64)
point = lambda a: a.ctypes.data_as(ctypes.c_void_p)
status = library.reset_rounds(point(text), ctypes.c_int64(n), point(sa), point(lcp), point(bwt), resets, point(left))
same = bool(np.array_equal(lcp, np.arange(n)) and np.array_equal(bwt, text))
print(json.dumps({"status": status, "same": same, "left": left.tolist()}))
"""


def harness():
    newest = max(p.stat().st_mtime for p in [SOURCE, *CSRC.iterdir()])
    if not BUILT.exists() or BUILT.stat().st_mtime < newest:
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not Path(nvcc).exists():
            pytest.skip("nvcc is needed to build the workspace harness")
        BUILT.parent.mkdir(exist_ok=True)
        tmp = BUILT.with_suffix(".so.tmp")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-Xcompiler", "-fPIC",
                        "-shared", "-o", str(tmp), str(SOURCE)], check=True)
        tmp.replace(BUILT)
    return BUILT


def test_harness_builds():
    assert hasattr(ctypes.CDLL(str(harness())), "reset_rounds")


@pytest.mark.gpu
def test_calls_after_a_device_reset():
    done = subprocess.run([sys.executable, "-c", CHILD, str(harness())], capture_output=True, text=True, cwd=HERE.parent,
                          timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    result = json.loads(done.stdout.strip().splitlines()[-1])
    assert result["status"] == 0 and result["same"]
    left = result["left"]
    kept = left[-1] - left[-2]
    assert kept > 12 * (32 << 20) // 2, left  # the pool keeps memory between calls
    # without the replacement every reset would leave another pool's memory behind
    assert min(left[1:-1]) > left[0] - kept // 2, left
