"""Groups of warps that map the blocks of a ring in turn.  On the CPU: copies that land in any order and barriers that are
waited for by parity (tests/cpp/ring_rounds.cu)."""
import os
import re
import subprocess

import pytest

from gpreempt_b200 import build as gpx_build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpreempt_b200", "csrc")
# Rings of the layers behind an affine map: two planes 3 and 4, one plane 6 and 8, and what a cluster's landing area leaves.
RINGS = [(3, 2), (4, 2), (6, 2), (8, 2), (6, 3), (8, 3)]


@pytest.fixture(scope="module")
def rounds(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rounds") / "ring_rounds")
    res = subprocess.run([gpx_build.nvcc(), *[f for f in gpx_build.NVCC_FLAGS if f != "-lineinfo"], "-I", CSRC,
                          os.path.join(ROOT, "tests", "cpp", "ring_rounds.cu"), "-o", exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return lambda *args: [int(v) for v in subprocess.run([exe, *map(str, args)], capture_output=True, text=True, check=True).stdout.split()]


@pytest.mark.parametrize("stages,groups", RINGS)
@pytest.mark.parametrize("blocks", [1, 2, 11, 77])
def test_no_block_is_mapped_before_it_has_landed(rounds, stages, groups, blocks):
    assert rounds(stages, groups, blocks, 2) == [0, 0]


def test_the_wait_is_what_keeps_the_rounds_apart(rounds):
    assert rounds(3, 2, 77, 0)[0] > 0 and rounds(8, 3, 77, 0)[0] > 0
    assert rounds(3, 2, 77, 1) == rounds(8, 3, 77, 1) == [0, 0]


def test_the_kernel_makes_that_wait():
    with open(os.path.join(CSRC, "cgemm_tcgen05.cu")) as fp:
        text = re.sub(r"//[^\n]*", "", fp.read())
    turn = text[text.index("if (turn == group) {"):]
    before = turn[:turn.index("ctl->full[stage]")]
    assert re.search(r"ring_rounds_skipped\(nst, Cfg::kAffGroups\)\s*&&[^;]*mbar_wait\(smem_u32\(&ctl->ready\[stage\]\), phase \^ 1,", before)
