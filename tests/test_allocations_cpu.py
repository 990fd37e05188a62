"""The transfer pool's idle memory is given up when an allocation of the library fails, so
every device allocation goes through the one function that does so."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scp3_b200", "csrc")


def test_device_allocations_go_through_one_function():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh", ".cpp", ".h")):
            for line in open(os.path.join(CSRC, name)):
                if re.search(r"\bcudaMalloc(Async|Managed)?\s*\(", line.split("//")[0]):
                    found.append(name)
    assert found == ["internal.h", "internal.h"], found      # first try and second
