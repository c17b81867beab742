"""The smoke entry point, in a process of its own: the launches it asserts are counted from the process's start."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_smoke():
    run = subprocess.run([sys.executable, "__graft_entry__.py", "smoke"], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-4000:]
