"""The fused selector's counts at their edges: streams shorter than one 16-byte
piece of symbols, of one group and one tile of 128 groups more or less, of more
tiles than the GPU has SMs (so that a CTA prefetches its next one), and groups that
repeat one symbol, two in turn, or hold the largest ones.  The bound is that of the
fused selector's comparison with the oracle: both round the same values to bf16
and differ in the order of 32-bit sums, at most 256 terms a layer, far below 2e-3
of the logits' size."""
import numpy as np
import pytest

import bzip2gpu_b200 as B
import bzip2gpu_b200.selector as S
import oracle.mlp as M

pytestmark = pytest.mark.gpu


def _check(torch, syms, seed):
    P = S.init_params(seed)
    P[S.OFF_B1:S.OFF_W2] = np.random.default_rng(seed).normal(0, 0.1, S.HID)
    lg, sel = B.selector_logits(torch.from_numpy(syms.astype(np.int16)).cuda(),
                                torch.from_numpy(P).cuda())
    lg, sel = lg.cpu().numpy(), sel.cpu().numpy()
    c, n = M.features(M.groups_of_stream(syms))
    ze = M.logits(P, c, n, emulate=True)
    assert lg.shape == ze.shape
    assert np.abs(lg - ze).max() <= 2e-3 * max(1.0, float(np.abs(ze).max()))
    assert np.array_equal(sel, lg.argmax(1))


@pytest.mark.parametrize("s", [1, 3, 4, 7, 8, 9, 49, 50, 51, 53, 100, 6399, 6400, 6401, 6407, 12851,
                               6400 * 150 + 31])
def test_lengths(torch_cuda, s):
    _check(torch_cuda, np.random.default_rng(s).integers(0, 258, s), s % 97)


@pytest.mark.parametrize("kind", ["one", "two", "pairs", "largest", "skewed"])
def test_repeated_symbols(torch_cuda, kind):
    i = np.arange(128 * 50 + 77)
    syms = {"one": i * 0 + 5, "two": i % 2 * 256, "pairs": i // 2 % 7, "largest": 257 - i % 3,
            "skewed": np.minimum(np.random.default_rng(1).geometric(0.4, len(i)), 257)}[kind]
    _check(torch_cuda, syms, 11)
