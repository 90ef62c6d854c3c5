"""The builds' fork onto side streams (side_streams.h): every way out of a
call joins it back to the caller's stream; the streams are the process's, as
many for 512 handles as for four, lent to one call at a time and kept with a
capture until it ends; they have the caller's priority.  Host logic: the harness runs it against stand-ins for
the CUDA calls."""

import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_side_streams(tmp_path):
    exe = tmp_path / "h"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(REPO, "felizjueves_b200", "csrc"),
                    "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    os.path.join(REPO, "tests", "side_streams_harness.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
