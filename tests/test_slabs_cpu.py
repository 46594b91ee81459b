"""How a call's blocks are shared out over slabs (csrc/slabs.h, host code)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
MB = 1_000_000


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    exe = tmp_path_factory.mktemp("slabs") / "slabs"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'bzip2gpu_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "slabs.cpp"), "-o", str(exe)], check=True)

    def run(rows):
        r = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, x)) for x in rows),
                           check=True, capture_output=True, text=True)
        return [int(x) for x in r.stdout.split()]
    return run


def test_short_blocks_do_not_cut_a_small_call(counts):
    # (blocks, bytes) that 16 blocks a slab alone would cut in four
    rows = [(64, 64_000), (100, MB), (64, 6_400_000), (200, 20 * MB), (67, 20 * MB)]
    assert counts([(n, b, 4, d) for n, b in rows for d in (0, 1)]) == [1] * 10


def test_full_blocks(counts):
    sizes = [1, 14, 28, 29, 57, 86, 87, 116, 300, 1300]
    rows = [(-(-s * MB // 900_000), s * MB, 4, 1) for s in sizes]
    assert counts(rows) == [1, 1, 1, 2, 2, 2, 3, 4, 4, 4]
    # host input is cut sooner, and takes several slabs per worker later
    rows = [(-(-s * MB // 900_000), s * MB, 4, 0) for s in (28, 29, 70, 71, 93, 94)]
    assert counts(rows) == [1, 2, 2, 3, 3, 4]
    assert counts([(n, n * 900_000, 4, 0) for n in (128, 512, 1023, 1024, 1536)]) == [4, 4, 4, 8, 12]


def test_few_long_blocks_stay_together(counts):
    # the bzip2 split's blocks can hold 45 MB of zeros each
    assert counts([(12, 540 * MB, 4, 1), (15, 675 * MB, 4, 1), (32, 1440 * MB, 4, 1)]) == [1, 1, 2]


def test_workers_bound_the_count(counts):
    assert counts([(384, 345 * MB, w, 1) for w in (1, 2, 3, 4)]) == [1, 2, 3, 4]
