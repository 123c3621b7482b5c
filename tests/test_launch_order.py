"""Kernels of a pass start before their predecessor in the stream has ended (programmatic dependent launch) and are ordered by
griddepcontrol.wait alone. What the sources have to keep for that, checked on their text: every kernel launched that way waits, and
none reads through the read-only path (__ldg, ld.global.nc, const __restrict__), which is defined only for memory that nothing
writes while the kernel is resident and whose loads the compiler may move ahead of the wait."""
from __future__ import annotations

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "comfyui-backend-but-rust_b200", "csrc")


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.inl"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _kernels():
    """name -> (parameter list, body) of every __global__ function."""
    out = {}
    for _, text in _sources():
        for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += (text[i] == "{") - (text[i] == "}")
                i += 1
            out[m.group(1)] = (m.group(2), text[m.end():i])
    return out


def _launched_early():
    """Kernels named in a launch_pdl call, directly or through a variable of the same function."""
    names = set()
    for name, text in _sources():
        if name == "common.cuh":       # where the launchers are defined
            continue
        kernels = set(re.findall(r"\b(\w+_kernel)\b", text))
        for m in re.finditer(r"launch_pdl(?:_cluster)?\(\s*(\w+)", text):
            if m.group(1) in kernels:
                names.add(m.group(1))
            elif m.group(1) == "kern":
                start = text.rindex("auto kern =", 0, m.start())
                names |= set(re.findall(r"\b(\w+_kernel)\b", text[start:text.index(";", start)]))
    return names


def test_every_kernel_launched_early_waits():
    kernels, early = _kernels(), _launched_early()
    assert {"quant_rows_kernel", "gemm_i8_pair_kernel", "gemm_w6a8_rows_kernel", "skinny_gemm_kernel", "w6_requant_regs_kernel"} <= early
    for name, (_, body) in kernels.items():        # and nobody waits for a launch that is not of this kind
        assert ("pdl_wait()" in body) == (name in early), name


def test_successors_are_let_in_only_when_a_kernel_is_nearly_done():
    """A trigger at a kernel's start places the successor's CTAs beside the running kernel, on whatever SMs it leaves idle (a
    small quantizer after a GEMM: all of it on twenty SMs). GEMMs leave the trigger to the end of their CTAs; where a kernel has
    one, it comes after its wait and its loads."""
    for name, (_, body) in _kernels().items():
        if "pdl_trigger()" not in body:
            continue
        assert "gemm" not in name, name
        at = body.index("pdl_trigger()")
        assert body.index("pdl_wait()") < at and max(body.find("gload("), body.find("load32<")) < at, name
        assert "gload(" in body[:at] or "load32<" in body[:at], name


def test_no_read_only_loads_in_kernels_that_start_early():
    for name, text in _sources():
        assert "__ldg(" not in text and "ld.global.nc" not in text and ".nc." not in text, name
    kernels = _kernels()
    for name in _launched_early():
        params, body = kernels[name]
        assert "__restrict__" not in params + body, name
