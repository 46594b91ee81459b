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


def _shared_arrays(src):
    """name -> the smallest alignment among its __shared__ declarations."""
    res = {}
    for align, kind, names in re.findall(
            r"__shared__ (?:__align__\((\d+)\) )?(\w+) ([^;]+);", src):
        own = {"uint8_t": 1, "uint16_t": 2, "int16_t": 2, "uint64_t": 8, "int64_t": 8}.get(kind, 4)
        for v in re.findall(r"(\w+)\s*\[", re.sub(r"\[[^\]]*\]", "[", names)):
            res[v] = min(res.get(v, 1 << 10), max(own, int(align or 0)))
    return res


# shared arrays that kernels reach by wider words through another pointer or a
# function: (file, array, bytes)
THROUGH = [("decode.cu", "lists", 4),  # k_dec_syms: lst; k_dec_emit: lists[w]
           ("decode.cu", "sb", 4),     # load_segments
           ("rle1.cu", "tbl", 16),     # crc_word_table_fill
           ("mtf.cu", "tab", 4), ("pack.cu", "sy", 16), ("huffman.cu", "heap_s", 16)]


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_shared_arrays_read_by_wider_words_are_aligned(name):
    src = _source(name)
    for v, n in [(v, n) for f, v, n in THROUGH if f == name]:
        assert _shared_arrays(src)[v] >= n, (name, v, n)
    for part in re.split(r"__global__|__device__", src):  # function by function
        arrays = _shared_arrays(part)
        for word, v in re.findall(r"reinterpret_cast<(?:const )?(\w+) \*>\(&?(\w+)", part):
            if v in arrays and word in WIDE:
                assert arrays[v] >= WIDE[word], (name, v, word)
