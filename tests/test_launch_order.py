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


# ---- the same rules through the functions that kernels call ----------------------------------------------------------------------

def _device_functions():
    """name -> [(qualifiers, parameter list, body)] of every __device__ function; overloads and specialisations side by side."""
    out = {}
    for _, text in _sources():
        for m in re.finditer(r"((?:__noinline__\s+)?__device__[^;{}()]*?)\b(\w+)\s*\(((?:[^(){}]|\((?:[^()]|\([^()]*\))*\))*)\)\s*(?:const\s*)?\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += (text[i] == "{") - (text[i] == "}")
                i += 1
            out.setdefault(m.group(2), []).append((m.group(1), m.group(3), text[m.end():i]))
    return out


def _followed(body, functions, out_of_line=False, stack=()):
    """A body with the bodies of the functions it calls in place of the calls, in the order of the text; those of functions out of line
    only on demand (what they do, they do beside the kernel's common path)."""
    def put(m):
        name = m.group(1)
        if name not in functions or name in stack:
            return m.group(0)
        inner = [_followed(b, functions, out_of_line, stack + (name,)) for q, _, b in functions[name] if out_of_line or "__noinline__" not in q]
        return m.group(2) + "( {" + " ".join(inner) + "} "
    return re.sub(r"\b(\w+)((?:\s*<[^;(){}<>]*(?:<[^;(){}<>]*>[^;(){}<>]*)*>)?\s*)\(", put, body)


_NAMES = ("pdl_wait", "pdl_trigger", "gload")      # stay as they are in the text


def _order_of(kernels, functions):
    """What breaks the rules for kernels that start early or let a successor in, and the kernels that have a trigger."""
    functions = {n: f for n, f in functions.items() if n not in _NAMES}
    wrong, with_trigger = [], []
    for name in sorted(_launched_early()):
        params, body = kernels[name]
        text = _followed(body, functions)
        whole = _followed(body, functions, out_of_line=True)
        if "__restrict__" in whole or "__ldg(" in whole:
            wrong.append((name, "a read through the read-only path"))
        loads = [m.start() for m in re.finditer(r"\bgload\(|\bload32<", text)]
        if "pdl_wait()" not in text or (loads and loads[0] < text.index("pdl_wait()")):
            wrong.append((name, "a load before the wait"))
        if "pdl_trigger()" not in text:
            continue
        with_trigger.append(name)
        if "gemm" in name:
            wrong.append((name, "a GEMM with a trigger"))
        at = text.index("pdl_trigger()")
        if at < text.index("pdl_wait()") or not loads or loads[0] > at:
            wrong.append((name, "a trigger before the wait and the rows"))
        if re.search(r"\bload32<|\bgload\(reinterpret_cast<const (?:uint4|float4)\*>\(x|\bgload\((?:x|up|aux|in)\b", text[at:]):
            wrong.append((name, "rows requested behind the trigger"))
    return wrong, with_trigger


def test_successors_are_let_in_behind_the_loads_of_called_functions_too():
    """The rules above hold for what a kernel does in the functions it calls: the row quantizers wait in the kernel, load in one function and let
    their successor in from there or from the next."""
    kernels, functions = _kernels(), _device_functions()
    wrong, with_trigger = _order_of(kernels, functions)
    assert not wrong, wrong
    assert {"quant_direct_kernel", "quant_norm_kernel", "sd_quant_fast_kernel", "w6_decode32_kernel"} <= set(with_trigger), with_trigger


def test_a_trigger_out_of_order_is_noticed():
    """The check above on sources with a mistake in them: it looks at the functions that matter."""
    def planted(name, change, kernel=False):
        kernels, functions = _kernels(), _device_functions()
        if kernel:
            params, body = kernels[name]
            assert change(body) != body
            kernels[name] = (params, change(body))
        else:
            before = functions[name]
            functions[name] = [(q, p, change(b)) for q, p, b in before]
            assert functions[name] != before, name
        return {n for n, _ in _order_of(kernels, functions)[0]}
    first = lambda b: " pdl_trigger(); " + b
    assert "quant_direct_kernel" in planted("direct_values", first)
    assert "quant_norm_kernel" in planted("norm_values", first)
    for k in ("quant_direct_kernel", "quant_norm_kernel"):
        assert k in planted(k, first, kernel=True)
        assert k in planted(k, lambda b: b.replace("pdl_wait();", "pdl_trigger(); pdl_wait();", 1), kernel=True)
    assert "quant_direct_kernel" in planted("direct_values", lambda b: b.replace("elementwise_prologue<", "gload(x); elementwise_prologue<"))
    assert "gemm_i8_pair_kernel" in planted("drain_values", first)
    assert "quant_direct_kernel" in planted("load32", lambda b: "const T* __restrict__ y = x; " + b)
    assert "quant_norm_kernel" in planted("norm_lane", lambda b: "gload(x); " + b)


def test_functions_out_of_line_are_given_their_warp_mask():
    """Which lanes a partial warp has is read once, at a kernel's start. Read again in a called function it would be whichever lanes the
    compiler happens to have there together."""
    functions = _device_functions()
    inside = {n: _followed(b, functions, out_of_line=True) for n, forms in functions.items() for q, _, b in forms if "__noinline__" in q}
    assert {"direct_again", "norm_again"} <= set(inside)
    assert [n for n, text in inside.items() if "__activemask(" in text] == []
