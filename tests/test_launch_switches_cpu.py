"""Every launch that may be a dependent one takes the engine's switch (MLQ_PDL), none a constant."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "maxlq_b200", "csrc")


def test_dependent_launches_follow_the_switch():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for m in re.finditer(r"\blaunch_pdl\(\s*([A-Za-z_0-9]+)", open(path).read()):
            if m.group(1) == "bool":  # the definition
                continue
            seen += 1
            assert m.group(1) in ("pdl", "pdl_"), (path, m.group(0))
    assert seen >= 3
