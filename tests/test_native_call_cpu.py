"""csrc/call.cpp puts arguments where the C entries expect them, and leaves to ctypes what it does not know."""
import ctypes
import subprocess
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest
import torch

from omchat_b200 import lib, native, seqlib

KINDS = {"P": (c_void_p, "const void*"), "I": (c_int, "int"), "L": (c_longlong, "long long"), "F": (c_float, "float")}


def _library(tmp_path, signature):
    """int f(<signature>, void* seen): every argument as a double into seen, in order."""
    args = "".join(f"{KINDS[k][1]} a{i}, " for i, k in enumerate(signature))
    body = "".join(f"s[{i}] = (double){'(long long)' if k == 'P' else ''}a{i};" for i, k in enumerate(signature))
    src = tmp_path / "f.c"
    src.write_text(f"int f({args}void* seen) {{ double* s = seen; {body} return {len(signature)}; }}\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-O1", str(src), "-o", str(tmp_path / "f.so")], check=True)
    return native.Entries(ctypes.CDLL(str(tmp_path / "f.so")), {"f": (c_int, [KINDS[k][0] for k in signature] + [c_void_p])})


@pytest.mark.parametrize("signature", ["", "F", "PIL", "PLPPLIIIIIPFLF", "".join(seqlib._P is t and "P" or {c_int: "I", c_longlong: "L", c_float: "F"}[t]
                                                                                  for t in seqlib.SIGNATURES["omc_linear_state_scan"][1]),
                                       "IF" * 8 + "L" * 30, "F" * 9])      # one float more than there are registers: by ctypes
def test_arguments_arrive(tmp_path, signature):
    entries = _library(tmp_path, signature)
    gen = torch.Generator().manual_seed(len(signature))
    seen = torch.full((len(signature) + 1,), -7.0, dtype=torch.float64)
    held, args, want = [], [], []
    for i, k in enumerate(signature):
        if k == "P":
            held.append(torch.zeros(3))
            args.append([None, held[-1], held[-1].data_ptr()][i % 3])
            want.append([0.0, float(held[-1].data_ptr()), float(held[-1].data_ptr())][i % 3])
        elif k == "F":
            args.append(float(torch.randn(1, generator=gen)) if i % 2 else 3)
            want.append(float(torch.tensor(args[-1], dtype=torch.float32)))
        else:
            args.append(int(torch.randint(-2 ** 31, 2 ** 31, (1,), generator=gen)) if k == "I" else (1 << 40) - i)
            want.append(float(args[-1]))
    for out in (seen, seen.data_ptr(), ctypes.c_void_p(seen.data_ptr())):     # the last is none of the kinds that go straight through
        seen.fill_(-7.0)
        assert entries.f(*args, out) == len(signature)
        assert seen[:-1].tolist() == want and seen[-1] == -7.0
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        entries.f(*args)
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        entries.f(*args, object())


def test_tensors_that_are_not_on_the_gpu_are_refused():
    with pytest.raises(lib.OmcError, match="no CPU fallback"):
        lib._need_cuda(None, torch.zeros(1))
    assert lib._need_cuda() is None and lib._need_cuda(None) is None


def test_the_compiled_calls_are_used():
    if native.module() is None:
        pytest.skip("no compiler or Python headers")
    assert type(seqlib.load().omc_linear).__name__ == "Entry" and type(lib.load().omc_gemm_bf16).__name__ == "Entry"
