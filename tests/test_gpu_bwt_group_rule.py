"""Which blocks sort their groups in shared memory: those whose active groups
are short, at most 2,048 rotations and 512 on average; the others go on by
radix sort.  Read off the count of radix scatter launches (the first sort has
four), with the stream compared with the oracle's."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import oracle

pytestmark = pytest.mark.gpu


def _repeat(period, copies):
    """Groups of `copies` rotations that stay together for many rounds."""
    unit = np.random.default_rng(period).integers(0, 256, period).astype(np.uint8)
    return np.concatenate([np.tile(unit, copies), np.array([7, 9], np.uint8)])


def _few_long(k, n):
    """One group of k rotations among n groups of 3."""
    rng = np.random.default_rng(k)
    heads = [np.array([250, 251, 252, 253], np.uint8)] * k
    for q in range(n):
        heads += [np.array([150 + q % 90, 200 + q // 90, 160, 170], np.uint8)] * 3
    return np.concatenate([np.concatenate([heads[i], rng.integers(0, 120, 3).astype(np.uint8)])
                           for i in rng.permutation(len(heads))])


@pytest.mark.parametrize("make,args,radix", [
    (_repeat, (1500, 2), False), (_repeat, (100, 400), False), (_repeat, (100, 500), False),
    (_repeat, (100, 540), True), (_repeat, (100, 1000), True), (_repeat, (50, 3500), True),
    (_few_long, (1900, 3000), False), (_few_long, (2040, 3000), False),
    (_few_long, (2060, 3000), True), (_few_long, (3500, 3000), True)])
def test_radix_sort_where_groups_are_long(torch_cuda, make, args, radix):
    a = make(*args)
    B.set_timing(True)
    try:
        got = B.compress(a, 9)
        scatters = B.last_stats()["scatter_launches"]
    finally:
        B.set_timing(False)
    assert got == oracle.compress(a, 9)
    assert (scatters > 4) == radix, scatters
