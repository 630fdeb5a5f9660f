"""Lifetime of the MoE workspace handle, on the CPU (a null handle: nothing is allocated)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("keep", ["w = h()", "moe.keep = h()", "import builtins; builtins.keep = h()", "h()"])
def test_a_workspace_that_outlives_the_interpreter_is_left_quietly(keep):
    """A program may end with a workspace, or a tensor on its memory, still referenced."""
    code = ("import ctypes as C\nfrom xccl_b200.ops import moe\nh = lambda: moe._Workspace(C.c_void_p())\n"
            f"{keep}\nprint('end')")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, PYTHONPATH=str(ROOT)), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("end")
    assert "Exception ignored" not in r.stderr, r.stderr
