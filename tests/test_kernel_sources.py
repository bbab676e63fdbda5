"""Rules of the kernel sources that no run can show to be broken."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flaggems_b200", "csrc")


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def test_operands_are_not_read_through_the_read_only_path():
    # Kernels may start before the one that writes their operands has ended (fg_launch).
    for name in _sources():
        assert not re.findall(r"__ldg\b|__restrict__|ld\.global\.nc", _code(name)), name

