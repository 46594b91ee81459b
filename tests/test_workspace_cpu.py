"""A slab workspace is two allocations, one on the device and one page-locked
(read off the sources): the calls for single stages make one each time, and
allocating its arrays one by one cost them more than a short stage does."""
import re
from pathlib import Path

SRC = Path(__file__).resolve().parents[1] / "bzip2gpu_b200" / "csrc" / "engine.cu"


def test_a_workspace_is_two_allocations():
    src = re.sub(r"//[^\n]*", "", SRC.read_text())
    assert len(re.findall(r"\bcudaMalloc\(", src)) == 1
    assert len(re.findall(r"\bcudaMallocHost\(", src)) == 1
