"""Kernels that may start before the kernel ahead of them has finished (they call `chain_wait`) must not treat what that kernel writes
as constant: no `const __restrict__` inputs and no `__ldg`, in the kernel or in the device functions it calls. The rotary
tables, written once when an engine is set up, are the exception. Read from the sources; needs no GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parameter_golf_b200", "csrc")
TABLES = {"cosT", "sinT", "c4", "s4"}


def _functions(path):
    """{name: (parameter text, body text)} of the functions of a source file."""
    src = re.sub(r"//[^\n]*", "", open(path).read())
    out = {}
    for m in re.finditer(r"\b(\w+)\(", src):
        depth, i = 1, m.end()
        while depth and i < len(src):
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        j = re.match(r"\s*(const\s*)?\{", src[i:])
        if not j or m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            continue
        start = k = i + j.end()
        depth = 1
        while depth and k < len(src):
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        out.setdefault(m.group(1), (src[m.end():i - 1], src[start:k - 1]))
    return out


def _chained():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            fns = _functions(os.path.join(CSRC, f))
            for name, (params, body) in fns.items():
                if "chain_wait()" in body:
                    yield f, name, fns


CASES = list(_chained())


def test_the_chained_kernels_are_found():
    names = {n for _, n, _ in CASES}
    assert {"gemm_tcgen05_kernel", "attn_fwd_kernel", "attn_bwd_fused_kernel", "mix_norm_fwd_kernel", "mix_norm_bwd2_kernel", "xsa_bwd64_kernel",
            "qk_norm_rope_bwd64_acc_kernel"} <= names
    launched = set()
    for f in os.listdir(CSRC):
        if f.endswith(".cu"):
            launched |= set(re.findall(r"launch_chained\([^;]*?\b(\w+_kernel)\b", open(os.path.join(CSRC, f)).read()))
    assert launched <= names                                  # whoever may start early waits


@pytest.mark.parametrize("file,name", [(f, n) for f, n, _ in CASES])
def test_a_chained_kernel_reads_no_predecessor_output_as_constant(file, name):
    fns = next(x for f, n, x in CASES if (f, n) == (file, name))
    todo, seen = [name], set()
    while todo:
        fn = todo.pop()
        if fn in seen:
            continue
        seen.add(fn)
        params, body = fns[fn]
        for p in params.split(","):
            if "const" in p.split("*")[0] and "__restrict__" in p:
                assert re.findall(r"\w+", p)[-1] in TABLES, (fn, p.strip())
        for arg in re.findall(r"__ldg\(((?:[^()]|\([^()]*\))*)\)", body):
            assert TABLES & set(re.findall(r"\w+", arg)), (fn, arg)
        todo += [g for g in re.findall(r"\b(\w+)\s*(?:<[^;(]*>)?\(", body) if g in fns]
