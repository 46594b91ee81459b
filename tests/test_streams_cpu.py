"""The library's streams keep the default priority (read off the sources): it
is the lowest there is, so with any other one a program's own kernels on
ordinary streams would wait behind all of the library's, and stage times taken
by events on streams of different priority would count waiting for others."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "bzip2gpu_b200" / "csrc"


def test_no_stream_outranks_the_callers():
    for p in sorted(CSRC.glob("*.cu")):
        src = re.sub(r"//[^\n]*", "", p.read_text())
        assert "StreamCreateWithPriority" not in src, p.name


def test_workspaces_are_zeroed_on_the_stream_that_uses_them():
    # a memset on the default stream does not order the work on the library's streams
    src = (CSRC / "engine.cu").read_text()
    assert "cudaMemset(" not in src and "cudaMemsetAsync(device_, 0, to_zero_, st)" in src
