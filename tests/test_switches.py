"""The measurement switches of the environment, through the entry points that report a call's scratch and workspace.
``LQ_GEMV_MAX_M`` is read once per process, hence the child processes.  No GPU is needed."""

import os
import subprocess
import sys

import pytest

PROBE = ("from liquidgemm_b200._lib import lib; import ctypes; p = (ctypes.c_size_t * 3)(); "
         "print([(lib.lq_linear_plan(256, m, 4096, 4096, 0, p), p[0] > 0)[1] for m in (1, 2)])")


@pytest.mark.parametrize("limit,two_launches", [(None, [False, False]), ("4", [False, False]), ("1", [False, True]), ("0", [True, True])])
def test_gemv_limit_reaches_the_quantising_form(limit, two_launches):
    """Its tokens need scratch exactly where the quantiser is a launch of its own."""
    env = {k: v for k, v in os.environ.items() if k != "LQ_GEMV_MAX_M"}
    if limit is not None:
        env["LQ_GEMV_MAX_M"] = limit
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", PROBE], env=env, cwd=root, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == str(two_launches)


@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (200, 1024, 4096)])
def test_i8_pair_switch_keeps_the_persistent_kernel(monkeypatch, M, N, K):
    """The streaming kernel cuts these layers and needs a workspace for it; the persistent kernel needs none."""
    from liquidgemm_b200._lib import lib
    monkeypatch.delenv("LQ_I8_PAIR", raising=False)
    assert lib.lq_i8_workspace_bytes(M, N, K) > 0
    monkeypatch.setenv("LQ_I8_PAIR", "0")
    assert lib.lq_i8_workspace_bytes(M, N, K) == 0
