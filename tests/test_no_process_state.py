"""The library keeps its state in handles: handles of several devices, driven by
several threads of one process, share no mutable variable.  (What a kernel is
allowed to take of shared memory, for one, is set per device.)"""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paris-git_b200", "csrc")


def test_no_mutable_static_variables():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        for no, line in enumerate(open(path), 1):
            # a static variable: a name followed by an initialiser, an array bound or a semicolon, not by a parameter list
            m = re.match(r"\s*static\s+(?!assert|cast|const\b|constexpr\b|inline\b)[\w:<>,\s*&]+?\b\w+\s*(=|;|\[)", line)
            if m and "__shared__" not in line:
                found.append(f"{os.path.basename(path)}:{no}: {line.strip()}")
    assert not found, found
