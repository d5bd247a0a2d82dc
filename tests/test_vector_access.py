"""Arrays that kernels read or write through wider pointers say so in their declaration: a plain array of floats is aligned to four bytes,
which holds only for as long as the compiler keeps it in registers."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "echokv_b200" / "csrc"
VECTOR = r"(?:V|float2|float4|uint2|uint4|int2|int4)"


DECLARATION = re.compile(r"^\s*(?:(?:__shared__|static|const) )*(__align__\(\d+\) )?(?:__half|__nv_bfloat16|float|uint8_t|unsigned char|uint16_t|uint32_t|int) (\w.*?);")


def unaligned(text: str) -> list[str]:
    """Names of arrays accessed through a pointer to vectors whose declaration, the last one ahead of the access, has no alignment."""
    aligned, found = {}, set()
    for line in text.splitlines():
        m = DECLARATION.match(line)
        for name in re.findall(r"(?:^|, )(\w+)\[", re.sub(r"\([^()]*\)", "", m.group(2))) if m else ():
            aligned[name] = bool(m.group(1))
        found |= {n for n in re.findall(r"reinterpret_cast<(?:const )?" + VECTOR + r"\*>\(&?(\w+)(?:\[[^\]]*\])*\)", line) if aligned.get(n) is False}
    return sorted(found)


def test_the_search_finds_one():
    assert unaligned("  float lt = 0.f, sum[VEC];\n  *reinterpret_cast<const V*>(sum);") == ["sum"]
    assert unaligned("  float t[W][VEC];\n  *reinterpret_cast<V*>(t[i]) = x;") == ["t"]
    assert unaligned("  __align__(16) float sum[VEC];\n  *reinterpret_cast<const V*>(sum);") == []


@pytest.mark.parametrize("file", sorted(f.name for f in CSRC.glob("*.cu*")))
def test_local_arrays_behind_vector_accesses_are_aligned(file):
    assert unaligned((CSRC / file).read_text()) == []
