"""Kernels that may begin before the kernel in front of them has finished (csrc/common.cuh: pdl_wait): what their pointers
promise the compiler, read from the sources. Only what is fixed while kernels run may be declared free of writes; the
read-only path that the promise opens is not ordered behind the wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm_infer_engine_b200", "csrc")


def _kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        start = text.find("{", m.start())
        head = text[m.start():start]
        if start < 0 or ";" in head:
            continue
        close = head.rfind(")")
        depth, i = 0, close
        while True:
            depth += (head[i] == ")") - (head[i] == "(")
            if depth == 0:
                break
            i -= 1
        depth, end = 0, start
        while True:
            depth += (text[end] == "{") - (text[end] == "}")
            end += 1
            if depth == 0:
                break
        yield re.search(r"(\w+)\s*$", head[:i]).group(1), " ".join(head[i + 1:close].split()), text[start:end]


SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


@pytest.mark.parametrize("source", SOURCES)
def test_inputs_of_waiting_kernels_are_plain_pointers(source):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    for name, params, body in _kernels(text):
        if "pdl_wait()" not in body:
            continue
        for p in params.split(","):
            assert not ("const" in p and "__restrict__" in p), f"{source}: {name}({p.strip()})"
            if "LLMIE_WEIGHT" in p:
                assert p.strip().startswith("const "), f"{source}: {name} writes {p.strip()}"
        assert "__ldg(" not in body, f"{source}: {name}"
    for m in re.finditer(r"struct (\w*Args)\s*\{(.*?)\n\};", text, re.S):
        assert "__restrict__" not in m.group(2), f"{source}: {m.group(1)}"


def test_the_sources_were_read():
    """The reader above finds the kernels (an empty list would pass the test of every file)."""
    found = []
    for source in SOURCES:
        with open(os.path.join(CSRC, source)) as f:
            found += [n for n, _, body in _kernels(f.read()) if "pdl_wait()" in body]
    assert len(found) >= 80 and {"causal_conv_kernel", "conv_qk_store8_kernel", "skinny_gemm_kernel"} <= set(found)
