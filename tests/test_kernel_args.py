"""Sizes of the structs that kernels take by value (CPU only).  A struct
argument above 128 bytes is read from parameter memory at each use instead of
being held in registers, which cost the group kernel up to a fifth of its rate:
the common data side stays within that, whatever one kernel adds for itself."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "jw_types.h"
int main() { std::printf("%zu", sizeof(pfb::JwIO)); }
"""


def test_common_data_side_fits_registers(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-I", os.path.join(ROOT, "pfsolve_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    assert int(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout) <= 128
