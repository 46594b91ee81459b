"""Tables and shared arrays that kernels access by wider words than their
elements declare the alignment that this takes (read off the sources: nothing
else places them on such a boundary, and a misaligned access faults)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bzip2gpu_b200" / "csrc"

WIDE = {"uint16_t": 2, "uint32_t": 4, "uint64_t": 8, "uint2": 8, "uint4": 16, "int4": 16,
        "float4": 16, "ulonglong2": 16}


def _source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _table_alignment(src, table):
    """The declared alignment of a __device__ or __constant__ table's type."""
    kind = re.search(r"__(?:device|constant)__ (?:const )?(\w+) %s\b" % table, src).group(1)
    m = re.search(r"struct (?:alignas\((\d+)\) )?%s\b" % kind, src)
    return int(m.group(1) or 4)


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_tables_read_by_wider_words_are_aligned(name):
    src = _source(name)
    for word, table in re.findall(r"reinterpret_cast<const (\w+) \*>\(&(c_\w+)\.", src):
        assert _table_alignment(src, table) >= WIDE[word], (name, table, word)
