"""Function attributes and constant tables belong to a device: what notes that they are set is one flag
per device, read from the sources."""
import glob
import os
import re

from conftest import ROOT


def test_flags_are_per_device():
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "emerge_gb300", "csrc", "*.cu*"))):
        for line in open(path):
            m = re.match(r"\s*(?:static\s+)?bool\s+(?:g_)?\w*(?:attr|ready)\w*\s*(\[\d+\])?\s*=", line)
            if m:
                assert m.group(1), f"{os.path.basename(path)}: {line.strip()}"
                seen += 1
    assert seen >= 5
