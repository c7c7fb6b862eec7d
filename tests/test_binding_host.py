"""The host path of layers.py (native/binding.cpp) beside a library of the same name that does nothing but wait, and where it has
to give an error."""
import os
import subprocess
import sys

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "crucible_strix_halo_b200")

# cr_proj_gemm waits, ten seconds at most, until another thread has set `flag`; the other entry points are not called.
STUB = r"""
#include <unistd.h>
volatile int flag = 0, seen = -1;
int cr_proj_gemm() { for (int i = 0; i < 10000 && !flag; ++i) usleep(1000); seen = flag; return 0; }
int cr_gdn_step() { return 1; }
int cr_qsa_step() { return 1; }
int cr_gdn_prefill() { return 1; }
int cr_qsa_prefill() { return 1; }
const char* cr_last_error() { return ""; }
"""

UNLOCKED = r"""
import ctypes, importlib.machinery, importlib.util, sys, threading, time, torch
torch.cuda.current_stream()
loader = importlib.machinery.ExtensionFileLoader("_binding", sys.argv[1] + "/_binding.so")
binding = importlib.util.module_from_spec(importlib.util.spec_from_loader("_binding", loader))
stub = ctypes.CDLL(sys.argv[1] + "/libcrucible_attn.so")
def other():
    time.sleep(0.2)                                   # the call is waiting by now
    ctypes.c_int.in_dll(stub, "flag").value = 1
t = threading.Thread(target=other)
t.start()
binding.proj_gemm(torch.zeros(1, 64), torch.zeros(32, 64), [torch.zeros(1, 32)])
t.join()
assert ctypes.c_int.in_dll(stub, "seen").value == 1, "no other thread ran during the call"
"""


@pytest.mark.gpu
def test_calls_release_the_interpreter_lock(tmp_path):
    """Another Python thread runs while a call is inside the library.  (Host memory only; the GPU is needed for its stream.)"""
    (tmp_path / "stub.c").write_text(STUB)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "libcrucible_attn.so"), str(tmp_path / "stub.c")], check=True)
    with open(os.path.join(PKG, "_binding.so"), "rb") as f:
        (tmp_path / "_binding.so").write_bytes(f.read())
    r = subprocess.run([sys.executable, "-c", UNLOCKED, str(tmp_path)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


def _without_gpu(code):
    """Runs `code` in a process of its own that sees no GPU; it prints what it has to say."""
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="", PYTHONPATH=os.path.dirname(PKG))
    r = subprocess.run([sys.executable, "-c", "import torch\nfrom crucible_strix_halo_b200 import _binding, layers\n" + code], capture_output=True,
                       text=True, timeout=300, env=env)
    assert r.returncode == 0, "status %d\n%s" % (r.returncode, r.stderr[-2000:])
    return r.stdout.split()


@pytest.mark.parametrize("call", ["_binding.current_stream()", "layers.proj_gemm(torch.zeros(1, 64).bfloat16(), torch.zeros(32, 64).bfloat16(), [torch.zeros(1, 32)])"])
def test_no_gpu_is_an_exception(call):
    assert _without_gpu("try:\n    %s\nexcept RuntimeError:\n    print('refused')" % call) == ["refused"]


@pytest.mark.parametrize("x,out,error", [((1, 64), (0,), "IndexError"), ((1, 64), (0, 4, 8), "IndexError"), ((1, 64), (), "IndexError"),
                                         ((1, 8, 8), (1, 32), "ValueError"), ((64,), (1, 32), "ValueError"), ((), (1, 32), "ValueError")])
def test_projection_shapes_that_are_refused(x, out, error):
    """Outputs without rows that are not matrices (the width is looked up in the first row), and inputs that are not matrices."""
    code = "try:\n    layers.proj_gemm(torch.zeros(%s).bfloat16(), torch.zeros(32, 64).bfloat16(), [torch.zeros(%s)])\nexcept %s:\n    print('refused')"
    assert _without_gpu(code % (x, out, error)) == ["refused"]
