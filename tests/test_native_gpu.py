"""The host path of the kernel calls (csrc_host/native.cpp) on a second copy of the module that is bound to a stub library."""
import ctypes
import importlib.machinery
import importlib.util
import shutil
import subprocess
import threading
import time

import pytest
import torch

from based_b200 import _capi

pytestmark = pytest.mark.gpu

STUB = """
#include <unistd.h>
static volatile int started, released;
int has_started(void) { return started; }
void release(void) { released = 1; }
/* waits for release() from another thread, two seconds at most */
int based_gated_act(void) { started = 1; for (int i = 0; i < 2000 && !released; ++i) usleep(1000); return released ? 0 : 77; }
"""


@pytest.fixture()
def stub(tmp_path):
    src, lib, copy = tmp_path / "stub.c", tmp_path / "libstub.so", tmp_path / "_native.so"
    src.write_text(STUB + "".join(f"int {n}(void) {{ return 0; }}\n" for n in _capi.SIGNATURES if n != "based_gated_act"))
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src)], check=True)
    shutil.copy(_capi.native_path(), copy)
    loader = importlib.machinery.ExtensionFileLoader("_native", str(copy))
    module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("_native", str(copy), loader=loader))
    loader.exec_module(module)
    module.bind(str(lib))
    return module, ctypes.CDLL(str(lib))


def test_other_threads_run_while_a_launch_waits(stub):
    module, lib = stub

    def other():
        while not lib.has_started():
            time.sleep(0.001)
        lib.release()

    x = torch.zeros(1, 16, device="cuda")
    t = threading.Thread(target=other)
    t.start()
    code = module.gated_act(x, x, x, 1, 8, 16, 16, 16, 0, 0)
    lib.release()
    t.join()
    assert code == 0


def test_errors_after_a_call_and_before_one(stub):
    module, lib = stub
    x = torch.zeros(1, 16, device="cuda")
    with pytest.raises(TypeError, match="at least one CUDA tensor"):
        module.gated_act(0, 0, 0, 1, 8, 16, 16, 16, 0, 0)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        module.gated_act(x.cpu(), x, x, 1, 8, 16, 16, 16, 0, 0)
    lib.release()
    assert module.gated_act(x, x, x, 1, 8, 16, 16, 16, 0, 0) == 0
