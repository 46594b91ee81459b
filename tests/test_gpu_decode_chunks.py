"""The decoder's parallel entropy decode at its edges: symbol counts around a
50-symbol group, a 32-group chunk (1600 symbols) and a CTA's four chunks;
zero runs across chunk ends; codes longer than the lookup tables; alphabets of
one and of 256 bytes.  The oracle is libbz2 (its stream in, the input out)."""
import bz2

import numpy as np
import pytest

import bzip2gpu_b200 as B

pytestmark = pytest.mark.gpu


def _noise(n, k, seed):
    """n bytes over k values without 4 equal in a row (so about n symbols)."""
    a = np.random.default_rng(seed).integers(0, k, n)
    a[3::4] = (a[2::4][: a[3::4].size] + 1) % k
    return a.astype(np.uint8)


@pytest.mark.parametrize("n", [1, 2, 48, 49, 50, 51, 99, 1598, 1599, 1600, 1601, 3199, 3201,
                               6399, 6400, 6401, 899_981])
@pytest.mark.parametrize("k", [2, 7, 256])
def test_symbol_counts(torch_cuda, n, k):
    a = _noise(n, k, n + k).tobytes()
    assert B.decompress(bz2.compress(a, 9)) == a


@pytest.mark.parametrize("period", [1, 2, 3, 50, 257, 1600])
def test_zero_runs_across_chunks(torch_cuda, period):
    # a repeated string leaves long runs of equal last-column bytes
    rng = np.random.default_rng(period)
    unit = rng.integers(0, 256, period).astype(np.uint8)
    a = np.concatenate([np.tile(unit, 600_000 // period + 1)[:600_000], _noise(5000, 256, 1)])
    assert B.decompress(bz2.compress(a.tobytes(), 9)) == a.tobytes()


def test_long_codes(torch_cuda):
    # geometric frequencies: code lengths from 1 to the format's longest
    rng = np.random.default_rng(5)
    a = np.minimum(rng.geometric(0.5, 800_000) - 1, 255).astype(np.uint8)
    a = np.concatenate([a, np.arange(256, dtype=np.uint8)])
    rng.shuffle(a)
    assert B.decompress(bz2.compress(a.tobytes(), 9)) == a.tobytes()


def test_many_small_blocks(torch_cuda):
    a = _noise(300_000, 200, 9)
    s = B.compress(a, 9, 777)
    assert B.decompress(s) == a.tobytes()
