"""A kernel's launch limits are kept per device (csrc/tws_limits.h), on the CPU
against a stand-in for the driver: a process that steps grids on a second device
raises the limits there too."""
from __future__ import annotations

import glob
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "terrainwatersim_gb300", "csrc")


def test_limits_are_kept_per_device(tmp_path):
    exe = str(tmp_path / "limits_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "limits_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert r.returncode == 0, r.stdout


def test_no_launcher_keeps_limits_of_its_own():
    """The shared memory limit is raised through KernelLimits, or at every use (the
    resident kernel)."""
    callers = [os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu"))
               if re.search(r"cudaFuncSetAttribute", open(f).read())]
    assert sorted(callers) == ["tws_resident.cu", "tws_step.cu"]
