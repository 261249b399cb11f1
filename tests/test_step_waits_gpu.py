"""The bounded waits of the tcgen05 kernels: what a wait that runs out leaves behind. Each test is a process of its own, since the count stays."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu


def _run(code):
    r = subprocess.run([sys.executable, "-c", "import ctypes, torch\nfrom omchat_b200 import seqlib\nn = ctypes.c_uint(7)\nL = seqlib.load()\n"
                        "out = torch.full((4,), 9, dtype=torch.int32, device='cuda')\n" + code], capture_output=True, text=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1])
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.split("\n")


def test_a_wait_that_runs_out_refuses_the_next_and_lets_drains_finish():
    got = _run("print(L.omc_step_wait_failures(ctypes.byref(n)), n.value)\n"
               "print(L.omc_step_wait_selfcheck(out.data_ptr(), torch.cuda.current_stream().cuda_stream), out.tolist())\n"
               "print(L.omc_step_wait_failures(ctypes.byref(n)), n.value)\n"
               "print(torch.ones(3, device='cuda').sum().item())")
    assert got[:4] == ["0 0", "0 [0, 0, 0, 1]", "0 1", "3.0"]
