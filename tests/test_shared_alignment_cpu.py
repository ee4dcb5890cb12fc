"""Dynamic shared memory is read and written 16 bytes at a time (float4, double2, cp.async): its
declarations say so, so that the place of the segment behind the static arrays does not matter."""
import glob
import os
import re

import build_lib


def test_dynamic_shared_memory_is_aligned():
    found = 0
    for path in glob.glob(os.path.join(build_lib.CSRC, "*.cu*")):
        for line in open(path):
            m = re.search(r"extern\s+__shared__\s+(.*?)\w+\[\]", line)
            if not m:
                continue
            found += 1
            align = re.search(r"__align__\((\d+)\)", m.group(1))
            ok = int(align.group(1)) >= 16 if align else m.group(1).split()[-1] in ("double2", "float4", "uint4")
            assert ok, "%s: %s" % (os.path.basename(path), line.strip())
    assert found >= 10
