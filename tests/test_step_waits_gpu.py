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


def test_a_wait_that_ran_out_is_reported():
    """By the next launch of a kernel that has such waits, and to who replays a graph by seqlib.check_waits; kernels without them still run."""
    got = _run("x, y = torch.ones(64, 128, dtype=torch.bfloat16, device='cuda'), torch.zeros(64, 64, device='cuda')\n"
               "g = torch.cuda.CUDAGraph()\n"
               "with torch.cuda.graph(g):\n    seqlib.linear(x, x, y)\n"       # the first launch of the process: captured
               "g.replay(); torch.cuda.synchronize(); seqlib.check_waits(); print(L.omc_step_wait_failed(), y[0, 0].item())\n"
               "L.omc_step_wait_selfcheck(out.data_ptr(), torch.cuda.current_stream().cuda_stream); torch.cuda.synchronize()\n"
               "print(L.omc_step_wait_failed())\n"
               "for f in (seqlib.check_waits, lambda: seqlib.linear(x, x, y)):\n"
               "    try:\n        f(); print('no error')\n"
               "    except seqlib.OmcError as e:\n        print('ran out' in str(e))\n"
               "z = torch.ones(64, 64, device='cuda'); seqlib.linear(z, z, y); print(y[0, 0].item())\n")
    assert got[:5] == ["0 128.0", "1", "True", "True", "64.0"]


def test_the_lanes_of_a_warp_have_one_answer():
    """Half of them wait for a phase that has come: they too go the way of the others, or the warp's next barrier would wait for ever."""
    got = _run("out = torch.full((32,), 9, dtype=torch.int32, device='cuda')\n"
               "print(L.omc_step_wait_warp_selfcheck(out.data_ptr(), torch.cuda.current_stream().cuda_stream), out.tolist() == [0] * 32)\n"
               "print(L.omc_step_wait_failures(ctypes.byref(n)), n.value)\n")
    assert got[:2] == ["0 True", "0 1"]
