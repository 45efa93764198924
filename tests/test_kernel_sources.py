"""A rule on the kernels' sources that no run can show to be broken."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aristos_b200", "csrc")


def test_no_load_promises_read_only_data():
    """Kernels become resident while the one in front still writes (programmatic launches), so none of them may read
    activations, weights or bookkeeping through the read-only path."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        assert not re.search(r"__ldg\s*\(|ld\.global(\.\w+)*\.nc\b|__restrict__", code), path
