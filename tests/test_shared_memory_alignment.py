"""Dynamic shared memory that a kernel divides up as bytes declares the alignment
of the widest access to it (16 bytes); a plain byte array promises only one."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ves2dpy_gb300", "csrc")


def test_byte_arrays_declare_their_alignment():
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            for line, text in enumerate(f, 1):
                if re.search(r"extern\s+__shared__.*\b(unsigned )?char\b", text):
                    found += 1
                    m = re.search(r"__align__\((\d+)\)", text)
                    assert m and int(m.group(1)) >= 16, f"{os.path.basename(path)}:{line}"
    assert found > 10
