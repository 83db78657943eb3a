"""The host path of the kernel calls (csrc_host/native.cpp), in part on a second copy of the module that is bound to a stub
library, and chains of programmatic launches."""
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


def _launchers():
    from based_b200 import ops
    g = torch.Generator("cuda").manual_seed(0)
    r = lambda *s, dtype=torch.bfloat16: torch.randn(*s, generator=g, device="cuda").to(dtype)
    W, n, B = 64, 32, 2
    rg = [r(W // n, 2, n, n), r(W), r(W), r(W, dtype=torch.float32)]
    x, w, o = r(2, 64), r(16, 64), r(2, 16)
    q, k, v, y = r(1, 2, 70, 16, dtype=torch.float32), r(1, 2, 70, 16, dtype=torch.float32), r(1, 2, 70, 16, dtype=torch.float32), r(1, 2, 70, 16, dtype=torch.float32)
    cache, h, ctx = r(B, 8, 2, 2, 16), r(B, 1, 2, 16), r(B, 1, 2, 16)
    u, out, S, ring, taps = r(B, 16, W), r(B, 16, W), r(B, W, dtype=torch.float32), r(B, 4, W), r(W, 4)
    return {
        "decode_linear": lambda: ops.decode_linear(x, w, out=o),
        "linattn_prefill": lambda: ops.linattn_prefill(q, k, v, out=y, return_state=False),
        "swa_decode": lambda: ops.swa_decode(h, h, h, cache, 3, 4, out=ctx),
        "rglru_gated": lambda: ops.rglru_gated(u, u, *rg, S, pos=0, out=out),
        "rglru_step": lambda: ops.rglru_step(u[:, 0], u[:, 1], taps, None, ring, *rg, S, pos=1, out=out[:, 0]),
    }


@pytest.mark.parametrize("name", ["decode_linear", "linattn_prefill", "swa_decode", "rglru_gated", "rglru_step"])
def test_a_refused_launch_leaves_no_error_behind(name):
    """A launch into a capture that has been invalidated (by waiting for its stream) is refused by the runtime; the calls after it
    answer for themselves."""
    from based_b200 import ops
    launch = _launchers()[name]
    launch()                                    # first uses load modules and set attributes
    other, gate = torch.randn(2, 32, device="cuda"), torch.empty(2, 16, device="cuda")
    torch.cuda.synchronize()
    rt, s = ctypes.CDLL("libcudart.so.12"), torch.cuda.Stream()
    stream, graph = ctypes.c_void_p(s.cuda_stream), ctypes.c_void_p()
    with torch.cuda.stream(s):
        assert rt.cudaStreamBeginCapture(stream, 2) == 0
        assert rt.cudaStreamSynchronize(stream) != 0
        try:
            with pytest.raises(_capi.BasedLibraryError):
                launch()
        finally:
            rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
            rt.cudaGetLastError()
    got = ops.gated_act(other, out=gate)
    assert torch.equal(got, gate)
    torch.cuda.synchronize()


class Drained:
    """The extension module with the device drained after every call."""

    def __init__(self, module):
        self.module = module

    def __getattr__(self, name):
        fn = getattr(self.module, name)

        def call(*args):
            code = fn(*args)
            torch.cuda.synchronize()
            return code
        return call


def _tensors(x):
    if torch.is_tensor(x):
        return [x]
    return [t for y in (x.values() if isinstance(x, dict) else x) for t in _tensors(y)]


@pytest.mark.parametrize("stack,B", [("based", 1), ("based", 16), ("based", 20), ("razesun", 3), ("vubenex", 1), ("vubenex", 17)])
def test_chains_equal_the_same_launches_one_at_a_time(stack, B, monkeypatch):
    """Prompt, portions and decode steps, whose kernels start under the ones before them, give to the bit the logits and states
    of the same calls with nothing in flight between them."""
    if stack == "based":
        from test_model_gpu import _small_model
        m = _small_model(seed=11)
    elif stack == "razesun":
        from test_razesun_gpu import build
        m = build("mixed", torch.bfloat16)[2]
    else:
        import vubenex_models
        from test_vubenex_gpu import build
        m = build(vubenex_models.configs()["wide"], torch.bfloat16)[1]
    g = torch.Generator().manual_seed(B)
    pieces = [40] + [1] * 8 if stack == "based" else [40, 24, 1, 1, 16] + [1] * 6
    ids = torch.randint(0, 90, (B, sum(pieces)), generator=g).cuda()

    @torch.inference_mode()
    def run():
        ip = m.new_inference_params(B, sum(pieces))
        for t in _tensors(ip.key_value_memory_dict):
            t.zero_()
        out, at = [], 0
        for n in pieces:
            out.append(m.advance(ids[:, at:at + n], ip))
            at += n
        return out + _tensors(ip.key_value_memory_dict)

    real = _capi.native()
    with monkeypatch.context() as patch:
        patch.setattr(_capi, "native", lambda: Drained(real))
        want = run()
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(run(), want, strict=True))
