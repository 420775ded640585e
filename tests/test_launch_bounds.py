"""Every launch bound of the kernels (MB_*, resident blocks per SM) is a
default that -D on the command line overrides, as the tuned headers promise and
disco_b200/autotune.py relies on."""
import os
import re

import disco_b200 as db

CSRC = os.path.join(os.path.dirname(os.path.abspath(db.__file__)), "csrc")


def test_bounds_can_be_given_on_the_command_line():
    found = set()
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            guards = []                        # the open #if levels' "not defined" names
            for line in f:
                if m := re.match(r"\s*#\s*if(?:n?def)?\b\s*(.*)", line):
                    guards.append(m.group(1).strip() if "ifndef" in line else "")
                elif re.match(r"\s*#\s*endif\b", line):
                    guards.pop()
                elif m := re.match(r"\s*#\s*define\s+(MB_\w+)\s", line):
                    assert m.group(1) in guards, (name, line)
                    found.add(m.group(1))
            assert not guards, name
    assert {"MB_UPDATE", "MB_MHD_FLUX", "MB_CT_EDGES", "MB_CT_FACES", "MB_CT_LINE", "MB_CT_UPDATE"} <= found
