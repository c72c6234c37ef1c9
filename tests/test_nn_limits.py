"""Sizes beyond the weight gradient's limits: the workspace query answers for every
argument (tomo_nn_wgrad refuses the call afterwards).  In a child process, since a
division by zero would end it; no GPU needed."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

LIB = Path(__file__).resolve().parents[1] / "iterative_tomographic_reconstruction_algorithms_b200" / "libtomo_nn.so"


@pytest.mark.parametrize("args", ["1, 65536, 65536, 8, 8, 9", "1, 65536, 65536, 8, 8, 1", "4, 32768, 32768, 8, 8, 9",
                                  "2147483647, 2147483647, 2147483647, 8, 8, 9", "1, 0, 0, 8, 8, 9"])
def test_wgrad_workspace_answers(args):
    if not LIB.exists():
        pytest.skip("libtomo_nn.so is not built")
    code = (f"import ctypes; l = ctypes.CDLL({str(LIB)!r}); l.tomo_nn_wgrad_workspace.restype = ctypes.c_size_t; "
            f"print(l.tomo_nn_wgrad_workspace({args}))")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and int(r.stdout) > 0, (r.returncode, r.stderr[-300:])
