"""New handles after a context reset work as the first ones did: what the
library keeps per process (scratch pool, kernels' shared-memory limits) is not
carried over from the ended context. Run in a child process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("handles", ["kept", "destroyed"])
def test_new_handles_after_a_reset(gpu, handles):
    child = os.path.join(os.path.dirname(os.path.abspath(__file__)), "context_reset_child.py")
    r = subprocess.run([sys.executable, child, handles], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
