"""State that host functions keep between calls is shared by contexts on several
threads: every function-local static variable of the library's sources stands
beside the mutex or once-flag that guards it.  (Checked in the source.)"""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_statics_are_guarded():
    found = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "wsclean_b200", "csrc", "*"))):
        if not path.endswith((".cu", ".cuh", ".cpp", ".h")):
            continue
        lines = open(path).read().splitlines()
        for i, line in enumerate(lines):
            # a variable: indented, not const, no parameter list before = or ;
            m = re.match(r"\s+static (?!const|__|inline)([^()]*?)\s*(=[^;]*)?;", line)
            if not m or "{" in line and "(" in line.split("{")[0]:
                continue
            found += 1
            near = "\n".join(lines[max(0, i - 2):i + 3])
            assert re.search(r"static std::(mutex|once_flag)\b", near), (path, i + 1, line)
    assert found >= 4
