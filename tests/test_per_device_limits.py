"""The kernels' limits on dynamic shared memory are raised once per kernel and device (host logic, no GPU)."""

from __future__ import annotations

import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mini_gpt_inference_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "per_device.h"
int main() {
    PerDeviceLimits limits;
    int a = 0, b = 0, calls = 0, answer = 0;
    auto raise = [&](const void* kernel, int device, int bytes) {
        return limits.raise(kernel, device, bytes, [&] { ++calls; return answer; });
    };
    auto expect = [&](int said, int made, int want_said, int want_made) {
        if (said != want_said || made != want_made) { std::printf("said %d, %d calls\n", said, made); return 1; }
        calls = 0;
        return 0;
    };
    int bad = 0;
    int r = raise(&a, 0, 100); bad += expect(r, calls, 0, 1);
    r = raise(&a, 0, 100); bad += expect(r, calls, 0, 0);      // once per device ...
    r = raise(&a, 1, 100); bad += expect(r, calls, 0, 1);      // ... and kernel
    r = raise(&b, 1, 100); bad += expect(r, calls, 0, 1);
    r = raise(&a, 0, 200); bad += expect(r, calls, 0, 1);      // more than it was raised to
    r = raise(&a, 0, 150); bad += expect(r, calls, 0, 0);      // and never lowered again
    answer = 2;
    r = raise(&b, 0, 100); bad += expect(r, calls, 2, 1);      // a refusal is answered and not kept
    answer = 0;
    r = raise(&b, 0, 100); bad += expect(r, calls, 0, 1);
    return bad;
}
"""


def test_limits_are_held_per_kernel_and_device(tmp_path):
    (tmp_path / "limits.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "limits"), str(tmp_path / "limits.cpp")], check=True)
    done = subprocess.run([str(tmp_path / "limits")], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def test_every_kernel_file_asks_through_them():
    for path in sorted(CSRC.glob("*.cu*")):
        calls = re.findall(r"cudaFuncSetAttribute", path.read_text())
        assert len(calls) == (path.name == "common.cuh"), f"{path.name} sets a limit by itself"
