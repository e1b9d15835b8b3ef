"""What the library's sources may not hold."""
import glob
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "jupiterncsm_gb300", "csrc", "*.c*"))
                 + glob.glob(os.path.join(ROOT, "jupiterncsm_gb300", "csrc", "*.h")) + [os.path.join(ROOT, "bench.py")])


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_load_to_several_ctas(path):
    """The benchmark runs the same library on several GPUs, where a load that one CTA issues for all CTAs of its
    cluster is not to be used."""
    with open(path) as f:
        assert "multi" + "cast" not in f.read()
