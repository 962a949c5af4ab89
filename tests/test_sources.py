"""The library is one file that replicas on several GPUs load, so its tensor loads
stay with the CTA that issues them: none delivers to other CTAs of a cluster (the
arrivals of a multiply's commit may)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gputools_gb300", "csrc")


def test_no_load_to_other_ctas_of_a_cluster():
    files = glob.glob(os.path.join(CSRC, "*.cu*"))
    loads = 0
    for f in files:
        with open(f) as fh:
            text = fh.read()
        for asm in re.findall(r"asm volatile\((.*?)\);", text, re.S):
            if "cp.async.bulk" in asm:
                loads += 1
                assert "multicast" not in asm, f
    assert loads >= 2
