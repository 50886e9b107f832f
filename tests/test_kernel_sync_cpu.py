"""Synchronisation that a run on the hardware does not show to be missing, read off the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpreempt_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as fp:
        return re.sub(r"//[^\n]*", "", fp.read())


def test_partial_sums_of_other_ctas_are_waited_for_at_cluster_scope():
    waits = re.findall(r"(\w*mbar\w*wait\w*)\(smem_u32\(&ctl->landed\)", _source("cgemm_tcgen05.cu"))
    assert waits == ["mbar_wait_cluster"]


def test_warps_meet_ahead_of_instructions_for_whole_warps():
    """Loads of accumulators inside loops whose bodies end in stores that only lanes with a row make, and waits of the
    cluster's barrier: __syncwarp stands before each, with no branch of single lanes in between."""
    for name, first in (("cgemm_tcgen05.cu", r"tmem_ld_32x16\(t_acc \+ c, u\);|tmem_ld_32x16\(t_acc \+ c, t16\);|cluster_wait\(\);"),
                        ("conv3x3_tcgen05.cu", r"tmem_ld_32x32\(t_acc, l\);|tmem_ld_32x32\(t_acc \+ 32 \* half, m\);")):
        text = _source(name)
        found = list(re.finditer(first, text))
        assert len(found) == {"cgemm_tcgen05.cu": 4, "conv3x3_tcgen05.cu": 2}[name]
        for m in found:
            before = text[:m.start()].rstrip().splitlines()[-6:]
            at = max((i for i, line in enumerate(before) if "__syncwarp();" in line), default=None)
            assert at is not None, (name, m.group(0), before)
            assert not any("lane" in line or "live" in line or "valid" in line for line in before[at + 1:]), before
