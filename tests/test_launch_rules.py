"""Launch rules and grids that count blocks per SM ask the device for its SMs: no kernel source carries a GPU's SM count."""
import glob
import os
import re

from conftest import ROOT


def test_no_source_carries_an_sm_count():
    files = glob.glob(os.path.join(ROOT, "probabilistic_mapping_b200", "csrc", "*.c*")) + \
        glob.glob(os.path.join(ROOT, "probabilistic_mapping_b200", "csrc", "*.h"))
    assert len(files) > 15
    for f in files:
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(f).read(), flags=re.S)
        assert not re.search(r"(?<![\w.])148(?![\w.])", code), f
