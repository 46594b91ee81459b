"""The BWT's group sort at its edges: groups of equal 4-byte prefixes around
the run lengths of its merges (8, 16, ..), around the longest that fit a tile with
a step of 512 (3584, above which a block goes on by radix sort) and across tiles; long repeats (many
rounds), equal rotations, and blocks of both kinds in one slab.  The suffix
array equals the oracle's exactly; streams equal the oracle's byte for byte."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import oracle

pytestmark = pytest.mark.gpu


def _groups(sizes, seed, tail=3):
    """Per size k: k copies of one 4-byte string, each followed by noise."""
    rng = np.random.default_rng(seed)
    units = []
    for q, k in enumerate(sizes):
        head = np.array([128 + q % 64, 200 + q // 64, 129 + q % 50, 190], np.uint8)
        for _ in range(k):
            units.append(np.concatenate([head, rng.integers(0, 120, tail).astype(np.uint8)]))
    order = rng.permutation(len(units))
    return np.concatenate([units[i] for i in order])


def _check(torch, a):
    d = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    assert np.array_equal(B.bwt(d).cpu().numpy(), oracle.bwt(a))


@pytest.mark.parametrize("k", [2, 7, 8, 9, 15, 16, 17, 63, 64, 65, 1023, 1025, 2047, 2048, 2049, 3583, 3584, 3585,
                               4095, 4097, 9000])
def test_group_sizes(torch_cuda, k):
    _check(torch_cuda, _groups([k, 3, 1, 5], k))


def test_many_groups_across_tiles(torch_cuda):
    rng = np.random.default_rng(3)
    _check(torch_cuda, _groups(rng.integers(1, 300, 300).tolist(), 4))
    _check(torch_cuda, _groups([2048, 2047, 2, 2048, 1, 2046, 3, 3584], 5))


@pytest.mark.parametrize("period,copies", [(1, 5000), (2, 4100), (17, 2048), (17, 2049),
                                           (1000, 9), (3001, 3), (40000, 2)])
def test_equal_rotations_and_long_repeats(torch_cuda, period, copies):
    unit = np.random.default_rng(period).integers(0, 256, period).astype(np.uint8)
    a = np.tile(unit, copies)
    _check(torch_cuda, a)
    _check(torch_cuda, np.concatenate([a, np.array([7, 9], np.uint8)]))


@pytest.mark.parametrize("m", [1, 2, 3, 5, 4095, 4096, 4097, 8193])
def test_small_alphabets_and_lengths(torch_cuda, m):
    for k in (1, 2, 3):
        _check(torch_cuda, np.random.default_rng(m + k).integers(0, k, m).astype(np.uint8))


def test_both_kinds_of_blocks_in_one_slab(torch_cuda):
    rng = np.random.default_rng(8)
    parts = [np.tile(rng.integers(0, 256, 17), 2000), rng.integers(0, 256, 34000),
             _groups([300, 20, 4, 2, 2], 1)[:2000], rng.integers(0, 2, 34000),
             np.tile(rng.integers(0, 256, 5000), 7), np.zeros(34000, np.int64)]
    a = np.concatenate([np.resize(p, 34000) for p in parts]).astype(np.uint8)
    assert B.compress(a, 9, 34000) == oracle.compress(a, 9, 34000)
