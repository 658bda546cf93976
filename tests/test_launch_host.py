"""Every launch that may start before the kernel ahead of it has ended follows
HPCG_B200_PDL: wherever the sources set the launch attribute for it, what is handed
to the launch depends on pdl_enabled()."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ATTRIBUTE = "cudaLaunchAttributeProgrammaticStreamSerialization;"


def test_early_launches_follow_the_knob():
    found = 0
    for path in glob.glob(os.path.join(ROOT, "hpcg_b200", "csrc", "*.cu*")):
        text = open(path).read()
        for m in re.finditer(re.escape(ATTRIBUTE), text):
            found += 1
            count = re.search(r"numAttrs = ([^;]*);", text[m.end():])
            assert count and "pdl" in count.group(1), os.path.basename(path)
    assert found >= 1
