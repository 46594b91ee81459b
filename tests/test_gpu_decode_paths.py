"""The decoder's ways to find the group starts, each forced: jumps over whole
groups (the rule's choice for few blocks), and chains of hops by 8 or 4 warps
per block (large streams).  At their edges: group and chunk counts, codes
longer than the 8- and 12-bit tables, groups that leave the 512-bit window,
positions where no code starts, more payload than the ring of words holds,
block magics that are no block starts, malformed streams, several batches.
The oracle is libbz2 and the input."""
import bz2

import numpy as np
import pytest

import bzip2gpu_b200 as B
import bzip2gpu_b200.workloads as W
import oracle

PATHS = ["jumps", "chains8", "chains4"]


@pytest.fixture(params=PATHS)
def path(request, monkeypatch, torch_cuda):
    monkeypatch.setenv("BZ2G_DECODE_STARTS", request.param)
    return request.param


def _noise(n, k, seed):
    """n bytes over k values without 4 equal in a row (so about n symbols)."""
    a = np.random.default_rng(seed).integers(0, k, n)
    a[3::4] = (a[2::4][: a[3::4].size] + 1) % k
    return a.astype(np.uint8)


# ---- a one-block encoder with any code lengths (the format allows 1 to 20)
def _codes(lens):
    res, code, last = {}, 0, 0
    for n in range(1, 21):
        for v in [v for v, x in enumerate(lens) if x == n]:
            res[v] = format(code, f"0{n}b")
            code += 1
        code <<= 1
    return res


def _deltas(lens):
    cur, out = lens[0], format(lens[0], "05b")
    for x in lens:
        out += "10" * (x - cur) if x >= cur else "11" * (cur - x)
        out += "0"
        cur = x
    return out


def _stream(a, tables, sel):
    """a as a one-block .bz2 stream: tables(n) gives the code length lists for
    an alphabet of n symbols, sel(k) the table of group k."""
    r = oracle.rle1_cut(a, 255)
    vals, ptr, present, used = oracle.mtf(r, oracle.bwt(r))
    syms = oracle.rle2(vals, used)
    lens = tables(used + 2)
    nsel = -(-len(syms) // 50)
    choice = [sel(k) for k in range(nsel)]
    order, unary = list(range(len(lens))), ""
    for t in choice:
        j = order.index(t)
        unary += "1" * j + "0"
        order.insert(0, order.pop(j))
    rows = ["".join(str(int(x)) for x in present[16 * i:16 * i + 16]) for i in range(16)]
    bits = format(0x314159265359, "048b") + format(oracle.crc32(a), "032b") + "0"
    bits += format(ptr, "024b") + "".join("01"[int("1" in x)] for x in rows)
    bits += "".join(x for x in rows if "1" in x)
    bits += format(len(lens), "03b") + format(nsel, "015b") + unary
    bits += "".join(_deltas(x) for x in lens)
    codes = [_codes(x) for x in lens]
    bits += "".join(codes[choice[i // 50]][int(v)] for i, v in enumerate(syms))
    bits += format(0x177245385090, "048b") + format(oracle.crc32(a), "032b")
    bits += "0" * (-len(bits) % 8)
    return b"BZh9" + int(bits, 2).to_bytes(len(bits) // 8, "big")


TABLES = {
    # 50 codes take 1000 bits: the longest group, twice the window; hardly any
    # position starts a code
    "all_20": (lambda n: [[20] * n, [20] * n], lambda k: k & 1),
    # group lengths that change from one to the next, by table
    "mixed": (lambda n: [[9] * n, [20] * n, [13] * n], lambda k: (k * k + k // 7) % 3),
    # lengths on both sides of the 8- and 12-bit tables within a group
    "steps": (lambda n: [[8 + v % 12 + (v % 12 < 4) * 2 for v in range(n)],
                         [10 + (5 * v) % 11 for v in range(n)]], lambda k: (k // 3) & 1),
}


def _coded(name, n=30000):
    return _stream(_noise(n, 200, 77), *TABLES[name])


# bytes whose symbol map holds the block magic, or the end-of-stream magic
def _mapped(words, n, seed):
    vals = [16 * (i + 2) + j for i, w in enumerate(words) for j in range(16) if (w >> (15 - j)) & 1]
    rng = np.random.default_rng(seed)
    a = np.array(vals, np.uint8)[rng.integers(0, len(vals), n)]
    a[: len(vals)] = vals
    return a


MAPS = {"block": (0x3141, 0x5926, 0x5359), "end": (0x1772, 0x4538, 0x5090)}


@pytest.mark.parametrize("name", sorted(TABLES))
def test_encoder_streams_are_valid(name):
    assert bz2.decompress(_coded(name, 4000)) == _noise(4000, 200, 77).tobytes()


@pytest.mark.parametrize("which", sorted(MAPS))
def test_symbol_maps_hold_the_magic(which):
    s = bz2.compress(_mapped(MAPS[which], 5000, 3).tobytes())
    magic = {"block": 0x314159265359, "end": 0x177245385090}[which]
    assert bin(int.from_bytes(s, "big")).count(format(magic, "048b")) == 2


@pytest.mark.gpu
def test_the_path_is_the_forced_one(torch_cuda, monkeypatch):
    s, n = bz2.compress(_noise(20000, 7, 1).tobytes()), {}
    for p in PATHS:
        monkeypatch.setenv("BZ2G_DECODE_STARTS", p)
        B.decompress(s)
        before = B.launch_count()
        B.decompress(s)
        n[p] = B.launch_count() - before
    # lengths, jumps and starts come before the kernel that then has nothing to do
    assert n["jumps"] == n["chains8"] + 3 and n["chains4"] == n["chains8"], n


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 49, 50, 51, 1599, 1600, 1601, 6401, 899_981])
@pytest.mark.parametrize("k", [2, 256])
def test_symbol_counts(path, n, k):
    a = _noise(n, k, n + k).tobytes()
    assert B.decompress(bz2.compress(a, 9)) == a


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(TABLES))
def test_code_lengths(path, name):
    assert B.decompress(_coded(name)) == _noise(30000, 200, 77).tobytes()


@pytest.mark.gpu
def test_geometric_frequencies(path):
    rng = np.random.default_rng(5)
    a = np.minimum(rng.geometric(0.5, 800_000) - 1, 255).astype(np.uint8)
    a = np.concatenate([a, np.arange(256, dtype=np.uint8)])
    rng.shuffle(a)
    assert B.decompress(bz2.compress(a.tobytes(), 9)) == a.tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("which", sorted(MAPS))
@pytest.mark.parametrize("n", [300, 50_000, 2_000_000])
def test_magic_that_starts_no_block(path, which, n):
    # the tiles of the blocks end at the false candidates
    a = _mapped(MAPS[which], n, n).tobytes()
    for s in (bz2.compress(a, 1), bz2.compress(a, 9)):
        assert B.decompress(s) == a


@pytest.mark.gpu
@pytest.mark.parametrize("batch", ["1", "3", "64"])
def test_batches(path, monkeypatch, batch):
    monkeypatch.setenv("BZ2G_DECODE_BATCH", batch)
    a = W.small_markov(240_000, seed=89)
    assert B.decompress(B.compress(a, 3, 7000)) == a.tobytes()  # 35 blocks


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["all_20", "mixed", "libbz2"])
def test_malformed_streams_are_errors(path, name):
    s = _coded(name) if name in TABLES else bz2.compress(_noise(200_000, 90, 4).tobytes())
    for at in (len(s) // 3, len(s) // 2, len(s) - 40):
        bad = bytearray(s)
        bad[at] ^= 0x24
        with pytest.raises(B.Bz2gError):
            B.decompress(bytes(bad))
    with pytest.raises(B.Bz2gError):
        B.decompress(s[: len(s) * 2 // 3])
    assert len(B.decompress(s)) > 0  # and the next call is right again


@pytest.mark.gpu
def test_more_tiles_than_a_piece_of_jumps(path):
    # 240 Mbit: two pieces of jumps
    d = B.gen_uniform(30_000_000, 6, device=True)
    s = B.compress_device(d, 9)
    assert B.decompress(s) == d.cpu().numpy().tobytes()
