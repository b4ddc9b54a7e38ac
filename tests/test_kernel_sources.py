"""Loads from global memory in inline assembly are volatile, and 16-bit scalars do not go through the __ldg overloads of
cuda_fp16.h / cuda_bf16.h (asm statements that are not): the compiler may evaluate either ahead of the bounds test in front
of it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mflux_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


def test_loads_in_assembly_are_volatile():
    found = 0
    for src in SOURCES:
        for m in re.finditer(r"asm\s*(volatile)?\s*\(\s*\"([^\"]*)", src.read_text()):
            if re.search(r"\bld(u)?\.(global|shared|weak|relaxed|acquire)|\bld\.param|prefetch", m.group(2)):
                found += 1
                assert m.group(1), f"{src.name}: {m.group(2)[:60]}"
    assert found


def test_no_16_bit_ldg():
    for src in SOURCES:
        assert not re.search(r"__ldg\((static_cast|reinterpret_cast)<const (__half|__nv_bfloat16)", src.read_text()), src.name
