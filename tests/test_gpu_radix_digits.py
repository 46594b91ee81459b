"""The radix sort's digit counts at their edges: blocks of a few bytes (shorter
than the 3 bytes the first pass looks ahead), of one tile of 4096 more or less,
of one group of 16 tiles more or less, blocks whose groups start anywhere in a
slab, 8- and 9-bit digits, separate keys and values (over 2^21 rotations), and digits that all items share, so that a pass is
left out and the next counts the items themselves.  Suffix arrays and streams
equal the oracle's exactly."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import oracle

pytestmark = pytest.mark.gpu


def _text(m, symbols, seed):
    """m bytes of few symbols with repeats, so that rounds follow the first sort."""
    rng = np.random.default_rng(seed)
    unit = rng.integers(0, symbols, max(1, min(m, 700))).astype(np.uint8)
    a = np.tile(unit, m // len(unit) + 1)[:m]
    at = rng.integers(0, m, max(1, m // 3000))
    a[at] = rng.integers(0, symbols, len(at))
    return a


@pytest.mark.parametrize("m", [2, 3, 4, 15, 16, 17, 4093, 4094, 4095, 4096, 4097, 4098, 4099, 4100,
                               65535, 65536, 65537, 65539, 131072, 131073, 200003, 263000, 600001,
                               (1 << 21) + 5])
def test_sizes(torch_cuda, m):
    for symbols in (1, 2, 251):
        a = _text(m, symbols, m)
        d = torch_cuda.from_numpy(a).cuda()
        assert np.array_equal(B.bwt(d).cpu().numpy(), oracle.bwt(a)), symbols


@pytest.mark.parametrize("block", [3000, 4096, 65536, 70000, 140001])
def test_groups_start_anywhere(torch_cuda, block):
    parts = [_text(50000 + 7 * block // 3, 2 + 60 * k, k) for k in range(4)]
    a = np.concatenate(parts + [np.zeros(3 * block + 1, np.uint8)] + parts[:1])
    assert B.compress(a, 9, block) == oracle.compress(a, 9, block, threads=8)
