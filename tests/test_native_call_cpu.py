"""csrc/call.cpp puts arguments where the C entries expect them, and leaves to ctypes what it does not know."""
import ctypes
import subprocess
import sys
from ctypes import c_float, c_int, c_longlong, c_void_p

import pytest
import torch

from omchat_b200 import build, lib, native, seqlib

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
                                       "IF" * 8 + "L" * 23, "L" * 39, "IF" * 8 + "L" * 30, "F" * 9])   # the last two by ctypes: more arguments, and one float more, than there are places
def test_arguments_arrive(tmp_path, signature):
    entries = _library(tmp_path, signature)
    if build.ensure_call() is not None:
        assert (type(entries.f).__name__ == "Entry") == (signature.count("F") <= 8 and len(signature) < 40)
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
    if build.ensure_call() is None:
        pytest.skip("no compiler or Python headers")
    assert type(seqlib.load().omc_linear).__name__ == "Entry" and type(lib.load().omc_gemm_bf16).__name__ == "Entry"


def test_a_failed_build_is_said_once(tmp_path, monkeypatch):
    """ctypes does the calls then, and the compiler's reason is not lost."""
    def fail(**kw):
        raise RuntimeError("g++ failed for call.cpp:\n\ncall.cpp:7:1: error: nothing of the kind\n  7 | x\ncompilation terminated.\n")
    monkeypatch.setattr(native, "_module", None)
    monkeypatch.setattr(native, "_tried", False)
    monkeypatch.setattr(build, "ensure_call", fail)
    with pytest.warns(RuntimeWarning, match="nothing of the kind") as said:
        entries = _library(tmp_path, "PI")
        assert native.module() is None and native.need_cuda(lib.OmcError)() is None
    assert len(said) == 1
    seen = torch.zeros(3, dtype=torch.float64)
    assert type(entries.f).__name__ != "Entry" and entries.f(None, 5, seen) == 2 and seen.tolist() == [0.0, 5.0, 0.0]


def test_the_import_compiles_nothing(tmp_path):
    """A fresh checkout: the first library that is loaded builds the calls, not the import; the checks of tensors work before and after."""
    code = ("import subprocess, sys, pathlib\n"
            "from omchat_b200 import build\n"
            f"build.LIBDIR = pathlib.Path({str(tmp_path)!r}); build.CALL_LIB = build.LIBDIR / 'omc_call.so'\n"
            "assert 'omchat_b200.lib' not in sys.modules\n"
            "real, ran = subprocess.run, []\n"
            "def run(*a, **k):\n    ran.append(a)\n    return real(*a, **k)\n"
            "subprocess.run = run\n"
            "import torch\nfrom omchat_b200 import lib, native, seqlib\n"
            "def refused():\n    try:\n        seqlib._need_cuda(torch.zeros(1))\n    except lib.OmcError as e:\n        return 'no CPU fallback' in str(e)\n"
            "assert not ran and refused()\n"
            "native.module()\n"
            "assert len(ran) == (native.module() is not None) and refused()\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=build.PKG.parent)
    assert r.returncode == 0, r.stderr[-2000:]
