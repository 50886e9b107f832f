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
