"""Rules of the CUDA sources that a compiler does not check and a run shows only by chance."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "based_b200", "csrc", "*.cu")))
# Read-only loads that stay: weights and tables, which no kernel of the library writes.
WEIGHT_LOADS = {
    "decode_linear.cu": {"wr[i] + ko"},
    "gated_conv.cu": {"src + q"},                                                            # taps
    "rglru.cu": {"w + k * 32 + 8 * t"},
    "short_conv.cu": {"src + q"},                                                            # taps
    "swa_simt.cu": {f"r{t} + (size_t){at} * half + c" for t in ("cos", "sin") for at in ("pos", "l")},   # rotary tables
    "token_side.cu": {"p"},
}
TABLES = {"rcos", "rsin"}


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def _programmatic(path):
    return "launch_pdl(" in _code(path)


def _argument(code, at):
    """The text between the parenthesis at ``at`` and its partner."""
    depth = 0
    for i in range(at, len(code)):
        depth += (code[i] == "(") - (code[i] == ")")
        if depth == 0:
            return code[at + 1:i]


@pytest.mark.parametrize("path", [p for p in SOURCES if _programmatic(p)], ids=os.path.basename)
def test_programmatic_kernels_read_activations_coherently(path):
    """A block of a programmatic launch may be resident while the kernel that writes its inputs still runs: the read-only path
    (ld.global.nc, __ldg, a const __restrict__ parameter) is for weights and tables only."""
    code, name = _code(path), os.path.basename(path)
    assert not re.findall(r"ld\.global\.nc[.\w]*", code)
    for m in re.finditer(r"__ldg\(", code):
        arg = _argument(code, m.end() - 1)
        arg = re.sub(r"^reinterpret_cast<const uint4\*>\((.*)\)$", r"\1", arg)
        assert arg in WEIGHT_LOADS.get(name, ()), arg
    for m in re.finditer(r"__global__[^;{]*?(\w+)\(([^;{]*)\)\s*\{", code):
        body = code[m.end():code.find("__global__", m.end()) if "__global__" in code[m.end():] else len(code)]
        if "pdl_wait()" not in body[:600]:
            continue
        assert set(re.findall(r"\bconst\s+\w+\*\s*__restrict__\s+(\w+)", m.group(2))) <= TABLES, m.group(1)


@pytest.mark.parametrize("path", [p for p in SOURCES if "tmem_st" in open(p).read()], ids=os.path.basename)
def test_tmem_hand_overs_between_warps_are_fenced(path):
    """Accesses to TMEM are ordered between threads by the tcgen05 fences around what the threads meet at, not by the barrier: a named
    barrier between reads of TMEM and writes of it has one before the arrival and one behind the wait."""
    code = re.sub(r"\s+", " ", _code(path))
    for m in re.finditer(r'asm volatile\("bar\.(sync|arrive)[^;]*;[^;]*;', code):
        later = code[m.end():].split("__global__")[0]
        writes, waits = later.find("tmem_st"), min((x for x in (later.find("mbar_"), later.find("__syncthreads")) if x >= 0), default=len(later))
        if not 0 <= writes < waits:
            continue                     # what is behind it does not write TMEM before the threads meet again
        alone = m.group(1) == "arrive" or "bar.arrive" in code
        if m.group(1) == "arrive" or not alone:
            assert code[:m.start()].rstrip().endswith("fence_before_sync();"), m.group(0)
        if m.group(1) == "sync":
            assert later.lstrip().startswith("fence_after_sync();"), m.group(0)
