"""Rules of the kernels' launches that no result shows, read out of the sources (no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cinnamon_b200", "csrc")
SOURCES = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read()) for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def test_shared_memory_limits_are_set_on_every_device():
    """A function's attributes belong to a device: set once per process, a second device's launches of the kernel are refused."""
    for name, text in SOURCES.items():
        for m in re.finditer(r"call_once", text):
            assert "cudaFuncSetAttribute" not in text[m.start():text.index("});", m.start())], name
