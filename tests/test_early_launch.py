"""Kernels that start while their predecessor drains read what it writes only
after their wait: by plain loads through pointers that promise the compiler
nothing (__ldg and restricted parameters may be read before the wait)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "reef3d_b200", "csrc")
# grid tables, written once at creation
TABLES = {"dxn", "dyn", "dzn"}
# device code that stage kernels inline, and the fields it reads
FIELDS = {"stencil_f64.cuh": "fuvw", "cell_f32.cuh": "fuvw"}


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def kernels(text):
    """(name, parameters, body) of every kernel."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params, start = text[m.end():at - 1], text.index("{", at)
        end, depth = start + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), params, text[start:end]


def early():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            out += [(f, *k) for k in kernels(source(f)) if "step_wait()" in k[2]]
    return out


def test_early_kernels_are_found():
    assert {k[1] for k in early()} >= {"dt_kernel", "volume_reduce_kernel", "fluid_kernel", "io_level_kernel",
                                       "io_ghost_kernel", "relax_kernel", "stage_kernel", "stage_kernel32"}


@pytest.mark.parametrize("kernel", early(), ids=lambda k: k[1])
def test_no_promise_about_written_memory(kernel):
    _, name, params, body = kernel
    held = {re.split(r"\W+", p.strip())[-1] for p in params.split(",") if "__restrict__" in p}
    assert held <= TABLES, (name, held - TABLES)
    for arg in re.findall(r"__ldg\(([^;]*?)\)", body):
        assert re.match(r"g\.\w+", arg), (name, arg)
    first = body.index("step_wait()")
    assert not re.search(r"\w\[", body[:first]), f"{name} reads memory before its wait"


@pytest.mark.parametrize("name", sorted(FIELDS))
def test_fields_by_plain_loads(name):
    text = source(name)
    for f in FIELDS[name]:
        assert not re.search(rf"__ldg\(\(?{f}\b", text), (name, f)
    for fn in ("conv_L", "reini_L"):
        params = re.search(rf"{fn}\(([^)]*)\)", text).group(1)
        assert "__restrict__" not in params, (name, fn)
