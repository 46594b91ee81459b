"""Loops with barriers are left by all threads of a block together (read off
the sources): a `break` must not depend on a shared variable, since a thread
that is ahead may already write the next value while one that is behind still
reads it; the decision comes with the barrier (__syncthreads_or) or from
registers that all threads hold alike."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bzip2gpu_b200" / "csrc"


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_no_loop_exit_reads_a_shared_flag(name):
    src = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for part in re.split(r"__global__|__device__", src):  # function by function
        shared = set()
        for names in re.findall(r"__shared__ (?:__align__\(\d+\) )?\w+ ([^;]+);", part):
            shared |= set(re.findall(r"\b[A-Za-z_]\w*", re.sub(r"\[[^\]]*\]", "", names)))
        for cond in re.findall(r"\bif \(([^;{}]*)\) (?:\{\s*)?break;", part):
            assert not shared & set(re.findall(r"\b[A-Za-z_]\w*", cond)), (name, cond)
