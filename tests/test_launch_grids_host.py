"""Grids follow the device: no kernel file writes a number of SMs into a launch."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "streamsim_gb300", "csrc")


def test_no_sm_count_in_the_code():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//.*", "", f.read())
        assert not re.search(r"\b(148|152|160)\b", code), name
