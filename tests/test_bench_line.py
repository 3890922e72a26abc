"""The benchmark's result line stands on a line of its own in a pipe, behind
whatever the C library had printed and not yet flushed.
"""

import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, sys
sys.path.insert(0, {root!r})
import bench
printf = ctypes.CDLL(None).printf
for i in range({lines}):  # the buffer is flushed in the middle of a line
    printf(b"LB system '(null)' initialised for 24 * 25 * 26 lattice\\n")
bench.emit({{"value": 1.5, "config": {{"a": [1, 2]}}}})
printf(b"Signalling implemented, process id = 7\\n")
"""


@pytest.mark.parametrize("lines", [1, 75, 200, 500])
def test_result_starts_a_line(lines):
    out = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, lines=lines)], capture_output=True, text=True,
                         check=True).stdout
    found = [json.loads(s) for s in out.splitlines() if s.startswith("{")]
    assert found == [{"value": 1.5, "config": {"a": [1, 2]}}]
    assert out.count("LB system") == lines and out.endswith("process id = 7\n")
