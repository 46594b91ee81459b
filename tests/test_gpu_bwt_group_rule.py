"""Which blocks sort their groups in shared memory: those whose active groups
are short (at most 2,048 rotations and 512 on average), and of the others those
that fit (3,584) while the slab holds few of their rotations; the rest goes on
by radix sort.  Read off the count of radix scatter launches (the first sort
has four), with the stream compared with the oracle's."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import oracle

pytestmark = pytest.mark.gpu


def _repeat(copies, length=899_000):
    """A block with groups of `copies` rotations that stay together for many rounds."""
    period = length // copies
    unit = np.random.default_rng(period).integers(0, 256, period).astype(np.uint8)
    return np.concatenate([np.tile(unit, copies), np.array([7, 9], np.uint8)])


def _few_long(k, n=3000):
    """A block with one group of k rotations among n groups of 3."""
    rng = np.random.default_rng(k)
    heads = [np.array([250, 251, 252, 253], np.uint8)] * k
    for q in range(n):
        heads += [np.array([150 + q % 90, 200 + q // 90, 160, 170], np.uint8)] * 3
    return np.concatenate([np.concatenate([heads[i], rng.integers(0, 120, 3).astype(np.uint8)])
                           for i in rng.permutation(len(heads))])


@pytest.mark.parametrize("make,k,blocks,radix", [
    (_repeat, 2, 2, False), (_repeat, 400, 8, False), (_repeat, 500, 8, False),
    (_repeat, 540, 8, True), (_repeat, 540, 6, False), (_repeat, 1000, 8, True),
    (_repeat, 1100, 3, True), (_repeat, 1100, 2, False), (_repeat, 2000, 3, True),
    (_repeat, 2100, 2, True), (_repeat, 2100, 1, False), (_repeat, 3500, 2, True),
    (_repeat, 3584, 1, False), (_repeat, 3700, 1, True),
    (_few_long, 1900, 8, False), (_few_long, 2060, 8, False), (_few_long, 3700, 1, True)])
def test_radix_sort_where_groups_are_long(torch_cuda, make, k, blocks, radix):
    one = make(k)
    a = np.tile(one, blocks)
    B.set_timing(True)
    try:
        got = B.compress(a, 9, one.size)
        scatters = B.last_stats()["scatter_launches"]
    finally:
        B.set_timing(False)
    # the blocks are alike: the oracle codes one
    part, bits, fold, _ = oracle.compress_part(one, one.size)
    assert got == oracle.assemble([part] * blocks, [bits] * blocks, [fold] * blocks, [1] * blocks)
    assert (scatters > 4) == radix, scatters
