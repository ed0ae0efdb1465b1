"""A ridge launch whose blocks give up waiting for one another is an error for
every caller, never a partial result: the debug library's limit on the polls of a
wait is lowered until waits run out (tests/ridge_give_up.py, in an interpreter of
its own with that library)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_launches_that_give_up(nb):
    from numbacs_gb300 import build
    env = dict(os.environ, NBCS_LIB=build.build(check=True))
    r = subprocess.run([sys.executable, os.path.join(HERE, "ridge_give_up.py")],
                       capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, (r.stdout + r.stderr)[-3000:]
    assert "gave up: all" in r.stdout
