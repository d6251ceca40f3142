"""Device allocations that fail: what has another way takes it, what has none
returns an error and can be called again.  The failures come from a stand-in for
cudaMalloc (no_room.py), each case in a process of its own.

Bars: the two ways of a Gram-Schmidt or a pairing contraction differ by their own
errors, the bars of the block tests (1e-13 FP64, 1e-11 mixed); behind the pairing
step's eigensolver 1e-9."""
import subprocess
import sys
from pathlib import Path

import pytest

import no_room

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", sorted(no_room.CASES))
def test_no_room(built, case):
    r = subprocess.run([sys.executable, no_room.__file__, case], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr
