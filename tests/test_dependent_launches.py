"""The kernels that are launched as programmatic dependents (they begin with
pdl_wait()), checked in their source.

Such a kernel may be resident while the kernels before it still write, so
what those write is not constant for its lifetime: it must not be taken as
`const T *__restrict__`, which promises the compiler just that (and lets it
read through the non-coherent path, or early). Only the caller's own inputs,
which are complete before the call's first kernel, may be.
"""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "pypo_gb300" / "csrc"

#: inputs of the entry points, written by no kernel of a call's chain
CALLER = {"src7", "cur", "tgt7", "cot"}

KERNEL = re.compile(r"__global__[^;{}]*?\b(\w+_kernel)\s*\(([^{};]*)\)\s*\{(.*?)^\}", re.S | re.M)


def dependents():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for name, params, body in KERNEL.findall(text):
            if "pdl_wait();" in body:
                yield name, [p.strip() for p in params.split(",")], body


def test_every_dependent_kernel_is_seen():
    waits = sum(re.sub(r"//[^\n]*", "", p.read_text()).count("pdl_wait();") for p in CSRC.glob("*.cu"))
    assert waits > 10 and len(list(dependents())) == waits


def test_written_buffers_are_not_declared_constant():
    wrong = [f"{name}: {p}" for name, params, _ in dependents() for p in params
             if "const" in p and "__restrict__" in p and p.split("__restrict__")[-1].strip() not in CALLER]
    assert not wrong, wrong


def test_nothing_is_read_before_the_wait():
    """Ahead of pdl_wait(): declarations and index arithmetic only, no access through a pointer parameter."""
    for name, params, body in dependents():
        head = body.split("pdl_wait();")[0]
        ptrs = [re.split(r"[\s*]", p)[-1] for p in params if "*" in p]
        assert not [p for p in ptrs if re.search(rf"\*\s*{p}\b|\b{p}\s*(\[|->)", head)], name
