"""Kernels that claim two tiles ahead hand the claims to their warps through slots of shared memory.  On the CPU: the
order of a kernel's stores, barriers and reads with a warp as late as the barriers let it be (tests/cpp/claim_slots.cu)."""
import os
import re
import subprocess

import pytest

from gpreempt_b200 import build as gpx_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpreempt_b200", "csrc")
KERNELS = {"layernorm": ("transformer.cu", "layernorm_kernel"), "miniweather_x": ("miniweather.cu", "miniweather_x_kernel")}


@pytest.fixture(scope="module")
def late_reads(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("slots") / "claim_slots")
    res = subprocess.run([gpx_build.nvcc(), *[f for f in gpx_build.NVCC_FLAGS if f != "-lineinfo"], "-I", CSRC,
                          os.path.join(ROOT, "tests", "cpp", "claim_slots.cu"), "-o", exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return lambda kernel, tiles: int(subprocess.run([exe, kernel, str(tiles)], capture_output=True, text=True, check=True).stdout)


@pytest.mark.parametrize("kernel", sorted(KERNELS))
def test_a_late_warp_reads_its_own_claims(late_reads, kernel):
    assert [late_reads(kernel, tiles) for tiles in (1, 2, 3, 4, 7, 40)] == [0] * 6


@pytest.mark.parametrize("kernel", sorted(KERNELS))
def test_the_kernel_uses_those_slots(kernel):
    file, name = KERNELS[kernel]
    with open(os.path.join(CSRC, file)) as fp:
        text = fp.read()
    body = text[text.index("\n" + name + "("):]
    body = body[:body.index("\n}\n")]
    uses = re.findall(r"s_tile\[([^\]]*(?:\([^)]*\))?[^\]]*)\]", body)
    assert uses.count("kClaimSlots") == 1 and len(uses) > 4
    assert all(u == "kClaimSlots" or u.startswith("claim_slot(") for u in uses), uses
