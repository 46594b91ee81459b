"""Code lengths at the heap's edges: alphabets around each heap depth and both
ends of the range, with tied, skewed and over-long (length-limited) counts.
Lengths, codes and selectors equal the oracle's exactly."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import oracle

pytestmark = pytest.mark.gpu


def _symbols(alpha, kind, seed):
    """RLE2 symbols 0 .. alpha - 2 and the end-of-block symbol alpha - 1."""
    rng = np.random.default_rng(seed)
    n = 30_000
    if kind == "ties":
        s = np.arange(n) % (alpha - 1)
    elif kind == "uniform":
        s = rng.integers(0, alpha - 1, n)
    elif kind == "skewed":
        s = np.minimum(rng.geometric(0.08, n) - 1, alpha - 2)
    else:  # Fibonacci counts: codes longer than the limit
        f = [1, 1]
        while len(f) < min(alpha - 1, 24):
            f.append(f[-1] + f[-2])
        s = np.repeat(np.arange(len(f)), f)
        rng.shuffle(s)
    return np.append(s, alpha - 1).astype(np.uint16)


@pytest.mark.parametrize("kind", ["ties", "uniform", "skewed", "fibonacci"])
@pytest.mark.parametrize("alpha", [3, 4, 5, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130,
                                   254, 255, 256, 257, 258])
def test_code_lengths(torch_cuda, alpha, kind):
    s = _symbols(alpha, kind, alpha)
    d = torch_cuda.from_numpy(s.view(np.int16).copy()).cuda()
    ln, code, sel, ng = B.huffman_build(d, alpha - 2)
    rl, rc, rs, rng = oracle.huffman_build(s, alpha - 2)[:4]
    assert ng == rng and np.array_equal(sel, rs)
    assert np.array_equal(ln[:ng, :alpha], rl[:ng, :alpha])
    assert np.array_equal(code[:ng, :alpha], rc[:ng, :alpha])
