"""PageRank's packed lists are made by worker threads when a model is opened: none of them may need memory of its own, as
an allocation that fails there ends the process instead of the call (tests/cpp/pack_lists.cu, on the CPU)."""
import glob
import os
import subprocess

from gpreempt_b200 import build as gpx_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_packing_allocates_on_the_calling_thread_only(tmp_path):
    gpx_build.build()
    exe = str(tmp_path / "pack_lists")
    objects = [o for o in sorted(glob.glob(os.path.join(gpx_build.OBJDIR, "*.o"))) if os.path.basename(o) != "graphwl.o"]
    res = subprocess.run([gpx_build.nvcc(), *[f for f in gpx_build.NVCC_FLAGS if f != "-lineinfo"], "-I", gpx_build.CSRC,
                          *[os.path.join(ROOT, "tests", "cpp", f) for f in ("pack_lists.cu", "first_thread_new.cpp")], *objects, "-o", exe, "-lpthread", "-ldl", "-lrt"],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and "PASS" in res.stdout, (res.returncode, res.stdout, res.stderr)
