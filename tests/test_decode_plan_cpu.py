"""The decoder's launch shapes (csrc/decode_plan.h, host code without CUDA):
they follow the batch's own blocks and cover them."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CAP = 1200000


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    exe = tmp_path_factory.mktemp("plan") / "decode_plan"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'bzip2gpu_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "decode_plan.cpp"), "-o", str(exe)], check=True)

    def run(what, *args):
        r = subprocess.run([str(exe), what, *map(str, args)], check=True, capture_output=True,
                           text=True)
        return [[int(x) for x in ln.split()] for ln in r.stdout.splitlines()]
    return run


SIZES = [1, 2, 63, 64, 65, 1000, 4095, 4096, 4097, 8191, 8192, 8193, 100000, 599999, 600000,
         600001, 600100, 650000, 900000, 1199999, CAP]


def test_column_grids_cover_every_block(plan):
    for m, (lf, walk, gather, repeat, unrle) in zip(SIZES, plan("grids", *SIZES)):
        assert lf == -(-m // 4096) and unrle == -(-m // 8192) and 1 <= repeat <= 16
        # the batch's other blocks are no longer than m: the most walkers of any
        step = [64 if x <= CAP // 2 else 128 for x in (m, min(m, CAP // 2))]
        most = max(-(-x // s) + 1 for x, s in zip((m, min(m, CAP // 2)), step))
        assert walk * 128 >= most and gather * 128 >= most + m // 64


def test_short_blocks_take_few_ctas(plan):
    # grids of the largest block were 293, 74, 220, 16 and 147 CTAs for each
    assert plan("grids", 1000) == [[1, 1, 1, 1, 1]]
    assert plan("chunks", 2400) == [[1]] and plan("crc", 1000) == [[1]]
    # 1,563 + 1 walkers, 1,562 more pool chunks
    assert plan("grids", 100000) == [[25, 13, 25, 16, 13]]


def test_chunk_and_crc_grids(plan):
    assert plan("chunks", 1, 160, 50 * 32 * 4, 50 * 18002, 1 << 40) == [[1], [1], [2], [141], [141]]
    assert plan("crc", 0, 1, 4096, 4097, 31 * 4096, 45_900_000) == [[1], [1], [1], [2], [31], [32]]


def test_jump_tiles_are_those_of_the_blocks(plan):
    assert plan("tiles", 1, 4095, 4096, 8192) == [[0, 1, 2, 4, 7]]
    # many short blocks and a long one, and garbage after the last block that
    # counts as its own: a CTA per tile, where a rectangle of the longest block's
    # tiles for every block was 4,096 x 24,415; a block has at most 18,307,033 bits
    short = [2400] * 4095
    assert plan("tiles", *short, 1_400_000)[0][-1] == 4095 + 342
    assert plan("tiles", *short, 100_000_000)[0][-1] == 4095 + 18_307_033 // 4096 + 1


TEXT, SHORT, NOISE = 1_400_000, 155_000, 7_250_000


@pytest.mark.parametrize("bits", [TEXT, SHORT, NOISE, 40_000])
def test_the_blocks_in_all_decide_whatever_their_size(plan, bits):
    # up to 125 times the longest block, and 3 tiles a block
    tiles = bits // 4096 + 1
    most = 125 * tiles // (tiles - 3)
    assert plan("jumps", 1 << 30, *[bits] * most)[1] == [1]
    assert plan("jumps", 1 << 30, *[bits] * (most + 1))[1] == [0]


def test_short_blocks_take_jumps(plan):
    assert plan("jumps", 1 << 30, *[2400] * 4096)[1] == [1]
    assert plan("jumps", 1 << 30, *[10_000] * 4000)[1] == [1]
    assert plan("jumps", 1 << 30, *[14_000] * 2000, TEXT)[1] == [1]  # beside a long one


def test_jumps_run_in_pieces_of_whole_blocks(plan):
    # 51,200 tiles a piece: 28 blocks of 1,771 tiles
    assert plan("jumps", 51200, *[NOISE] * 28) == [[0, 28], [1]]
    assert plan("jumps", 51200, *[NOISE] * 40) == [[0, 28, 40], [1]]
    assert plan("jumps", 51200, *[NOISE] * 57) == [[0, 28, 56, 57], [0]]
    assert plan("jumps", 51200, *[TEXT] * 150)[1] == [0]
    assert plan("jumps", 1770, NOISE) == [[], [0]] and plan("jumps", 1771, NOISE) == [[0, 1], [1]]
    assert plan("jumps", 3, 1, 4096, 4096, 1) == [[0, 2, 4], [1]]
