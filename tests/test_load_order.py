"""Population loads of the early-starting step kernels must stay behind their
griddepcontrol.wait, or a step reads what the step before is still writing.
The compiler keeps volatile asm in order with the wait (volatile asm itself)
and may move any other asm that it takes for a function of its operands.  So
the loads of the storage formats must use cache intrinsics that the toolkit
defines as volatile asm; those of __half and __nv_bfloat16 are not."""
import re
from pathlib import Path

import pytest

from flow_anizotropy_b200.build import CSRC, nvcc

POINTER = {"StoreF64": "double", "StoreF32": "float", "StoreF16": "__half", "StoreBF16": "__nv_bfloat16"}


def _struct(name):
    text = (CSRC / "d3q19.cuh").read_text()
    return re.search(r"struct %s \{(.*?)\n\};" % name, text, re.S).group(1)


def _loads(body):
    """(function, type that its __ldcs reads, None for the format's own) per load function."""
    for fn in ("ld", "ld2"):
        m = re.search(r" %s\(const T \*p[^)]*\)\s*\{(.*?)\}" % fn, body, re.S)
        if m:
            for arg in re.findall(r"__ldcs\((.*)", m.group(1)):
                c = re.match(r"reinterpret_cast<const ([\w ]+?) ?\*>\(p\)", arg)
                yield fn, c.group(1) if c else None


def _volatile_types():
    hpp = Path(nvcc()).resolve().parent.parent / "include" / "sm_32_intrinsics.hpp"
    if not hpp.exists():
        pytest.skip("no CUDA headers beside nvcc")
    return set(re.findall(r"__ldcs\(const ([\w ]+?) ?\*ptr\) \{[^}]*?asm volatile", hpp.read_text()))


@pytest.mark.parametrize("store", list(POINTER))
def test_population_loads_are_volatile(store):
    volatile = _volatile_types()
    loads = list(_loads(_struct(store)))
    assert loads
    for fn, typ in loads:
        assert (typ or POINTER[store]) in volatile, f"{store}::{fn}"


@pytest.mark.parametrize("source", ["k2d.cu", "step3d_slots.cuh", "k3d_reduce.cu"])
def test_no_restrict_across_the_wait(source):
    """An ordinary load stays behind the wait because the wait may write any
    memory; a __restrict__ pointer declared before it would promise that what
    it points to is written through it alone."""
    code = re.sub(r"//.*", "", (CSRC / source).read_text())
    assert "pdl_wait()" in code and "__restrict__" not in code
