"""How a call's blocks are shared out over slabs (csrc/slabs.h, host code)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
MB = 1_000_000


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("slabs") / "slabs"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'bzip2gpu_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "slabs.cpp"), "-o", str(exe)], check=True)

    def run(rows, *args):
        r = subprocess.run([str(exe), *args], input="\n".join(" ".join(map(str, x)) for x in rows),
                           check=True, capture_output=True, text=True)
        return [[int(x) for x in ln.split()] for ln in r.stdout.splitlines()]
    return run


@pytest.fixture(scope="module")
def counts(program):
    return lambda rows: [x[0] for x in program(rows)]


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


@pytest.mark.parametrize("n,length", [(500, 300), (200, 1001), (1000, 1001), (1000, 1), (7, 16)])
@pytest.mark.parametrize("slabs", [1, 2, 3, 4])
def test_a_queue_makes_the_slabs_it_is_meant_to(program, n, length, slabs):
    # lengths that are no multiples of 16 take more room than they have bytes
    sizes = program([(n, length, slabs, 1024)], "queue")[0]
    assert sum(sizes) == n and len(sizes) == slabs
    assert max(sizes) - min(sizes) <= slabs


def test_a_slab_takes_at_most_its_blocks(program):
    assert program([(1000, 500, 1, 384), (5, 16, 4, 1), (0, 16, 4, 1)], "queue") == [
        [384, 384, 232], [1, 1, 1, 1, 1], []]
