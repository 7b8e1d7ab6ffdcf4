"""GPU tests of single kernels at the sizes where their tiling can go wrong,
through the C ABI and against the oracle (integer work: bit-exact)."""
import numpy as np
import pytest

from golden_util import canonical_ids

pytestmark = pytest.mark.gpu


def check(orc, chars, offs, perm, lcp):
    ids, rlcp = orc.sort_ids_lcp(chars, offs)
    assert orc.check_permutation(perm)
    assert np.array_equal(canonical_ids(chars, offs, perm, rlcp), canonical_ids(chars, offs, ids, rlcp))
    if lcp is not None:
        assert np.array_equal(lcp[1:].astype(np.uint64), rlcp[1:])


def pass_loop(pkg):
    c = pkg.Context(0)
    c.set_option(c.OPT_SINGLE_LAUNCH, 0)
    return c


@pytest.mark.parametrize("at_end", [False, True])
@pytest.mark.parametrize("length", [9, 31, 32, 33, 40, 63, 65, 511, 513, 544, 545, 1056, 3000])
def test_suffix_lcp_chains(pkg, orc, length, at_end):
    """LCPs of suffixes inside copied blocks: chains of consecutive suffixes
    around a warp's 32, compares around a warp step's 512 chars, a block
    copied twice (predecessors change inside the chain), and a copy that runs
    to the text's end."""
    rng = np.random.default_rng(length)
    t = rng.choice(np.frombuffer(b"ACGT", np.uint8), 20011)
    block = t[100:100 + length].copy()
    t[7003:7003 + length] = block
    t[14001:14001 + length] = block
    text = np.concatenate([t, block] if at_end else [t]).astype(np.uint8)
    chars = np.concatenate([text, np.zeros(1, np.uint8)])
    c = pass_loop(pkg)
    try:
        perm, lcp = c.sort_host(chars, np.arange(chars.shape[0], dtype=np.uint64), lcp=True)
    finally:
        c.close()
    check(orc, chars, np.arange(chars.shape[0], dtype=np.uint64), perm, lcp)


LEAF_SIZES = [2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023,
              1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097]


def leaf_strings(kind, n, rng):
    if kind == "letters":
        return [bytes(rng.integers(97, 123, rng.integers(0, 20)).astype(np.uint8)) for _ in range(n)]
    if kind == "acgt":  # whole keys tie many times over, in runs around 32
        return [bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), rng.integers(1, 30))) for _ in range(n)]
    if kind == "ff":  # words of ones beside the padding's
        return [bytes(rng.integers(254, 256, rng.integers(6, 12)).astype(np.uint8)) for _ in range(n)]
    if kind == "eighth":  # no shared bits (an outlier at each end), keys equal in 7 chars
        s = [b"aaaaaaa" + bytes(rng.integers(97, 105, 1).astype(np.uint8)) + bytes([97 + int(rng.integers(3))])
             for _ in range(n - 2)]
        return s + [b"\x01", b"\xf0" * 9]
    if kind == "prefix":  # one group behind a long prefix
        return [b"p" * 101 + bytes(rng.integers(97, 100, rng.integers(0, 7)).astype(np.uint8)) for _ in range(n)]
    heads = [bytes(rng.integers(97, 99, 25).astype(np.uint8)) for _ in range(max(1, n // 40))]  # "runs"
    return [heads[int(rng.integers(len(heads)))] + bytes(rng.integers(97, 100, 4).astype(np.uint8)) for _ in range(n)]


@pytest.mark.parametrize("with_lcp", [True, False])
@pytest.mark.parametrize("kind", ["letters", "acgt", "ff", "eighth", "prefix", "runs"])
def test_leaf_sizes(pkg, orc, kind, with_lcp):
    """The leaf sorters at the edges of their size classes and networks, one
    instance of a batch per size: random strings, keys that tie in runs of
    about 32, chars 254 and 255, keys without a shared bit that tie in 7
    chars, one long shared prefix, and runs behind 25 shared chars."""
    rng = np.random.default_rng(len(kind))
    strings = [leaf_strings(kind, n, rng) for n in LEAF_SIZES]
    chars, offs = pkg.pack_strings([x for s in strings for x in s])
    inst = np.zeros(len(LEAF_SIZES) + 1, dtype=np.uint64)
    np.cumsum(LEAF_SIZES, out=inst[1:])
    c = pkg.Context(0)
    try:
        perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=with_lcp)
    finally:
        c.close()
    for k in range(len(LEAF_SIZES)):
        b, e = int(inst[k]), int(inst[k + 1])
        check(orc, chars, offs[b:e], perm[b:e], lcp[b:e] if with_lcp else None)


@pytest.mark.parametrize("n", [2, 31, 255, 256, 257, 1023, 1024, 1025, 2047, 4095, 4096, 4097, 4608, 16383, 16384,
                               65536, 262144])
@pytest.mark.parametrize("kind", ["letters", "acgt", "eighth", "prefix"])
def test_single_launch_sizes(pkg, orc, kind, n):
    """The one-block and single-launch sorts at the edges of their size
    rules, with and without LCPs."""
    if kind == "prefix" and n > 20000:
        pytest.skip("one segment behind a prefix: the pass loop's tests")
    rng = np.random.default_rng(n)
    chars, offs = pkg.pack_strings(leaf_strings(kind, n, rng))
    c = pkg.Context(0)
    try:
        perm, lcp = c.sort_host(chars, offs, lcp=True)
        only, _ = c.sort_host(chars, offs, lcp=False)
    finally:
        c.close()
    check(orc, chars, offs, perm, lcp)
    check(orc, chars, offs, only, None)


@pytest.mark.parametrize("with_lcp", [True, False])
@pytest.mark.parametrize("sigma", [1, 2, 3, 4, 7, 8, 15, 16, 31, 32, 63, 64, 127, 128, 255])
def test_suffix_alphabets(pkg, orc, sigma, with_lcp):
    """Suffix sets over alphabets around the powers of two (the packed keys'
    bits per char), with copies, copies of copies and a copy of all of it (the
    chains' ends part into groups of several sizes)."""
    rng = np.random.default_rng(sigma)
    symbols = np.sort(rng.choice(np.arange(1, 256, dtype=np.uint8), sigma, replace=False))
    t = rng.choice(symbols, 6000 + sigma)
    t[3000:4500] = t[100:1600]
    t[5000:5700] = t[3300:4000]
    t = np.concatenate([t, t[2500:5900], t[:40]])
    chars = np.concatenate([t, np.zeros(1, np.uint8)])
    offs = np.arange(chars.shape[0], dtype=np.uint64)
    c = pass_loop(pkg)
    try:
        perm, lcp = c.sort_host(chars, offs, lcp=with_lcp)
        assert {k["name"]: k["launches"] for k in c.kernel_stats()}["doubling"] > 0
    finally:
        c.close()
    check(orc, chars, offs, perm, lcp)


@pytest.mark.parametrize("n", [4097, 6143, 6144, 6145, 524288, 524289, 528385])
def test_pass_loop_tiles(pkg, orc, n):
    """The pass loop at the edges of its tile sizes (2048 strings up to 2^19,
    4096 above) and with a last tile of one string."""
    chars, offs, _ = pkg.workloads.random_strings(n, 0, 12, b"abcde", n)
    c = pass_loop(pkg)
    try:
        perm, lcp = c.sort_host(chars, offs, lcp=True)
    finally:
        c.close()
    check(orc, chars, offs, perm, lcp)


@pytest.mark.parametrize("ninst", [1, 31, 511, 512, 513, 1025, 310000])
def test_batch_roots(pkg, ninst):
    """Root segments of a batch, appended to the lists per block of 512
    instances and, beyond 592 blocks, by blocks in turn: every size class in
    one block, the last block part-filled."""
    rng = np.random.default_rng(ninst)
    sizes = rng.choice([1, 2, 32, 33, 300, 1500, 5000], ninst) if ninst < 2000 else rng.integers(1, 4, ninst)
    inst = np.zeros(ninst + 1, dtype=np.uint64)
    np.cumsum(sizes, out=inst[1:])
    n = int(inst[-1])
    text = np.zeros((n, 10), np.uint8)  # distinct: the string's number, shuffled, in base 16
    number = rng.permutation(n)
    for j in range(8):
        text[:, 7 - j] = 97 + ((number >> (4 * j)) & 15)
    offs = np.arange(n, dtype=np.uint64) * 10
    c = pkg.Context(0)
    try:
        perm, _ = c.sort_batch_host(text.reshape(-1), offs, inst, lcp=False)
    finally:
        c.close()
    of = np.repeat(np.arange(ninst), sizes)
    want = np.lexsort((number, of)) - inst[of].astype(np.int64)
    assert np.array_equal(perm.astype(np.int64), want)


@pytest.mark.parametrize("with_lcp", [True, False])
@pytest.mark.parametrize("length", [3, 8, 13])
def test_equal_buckets(pkg, orc, length, with_lcp):
    """Equal strings in buckets of their own, of 8 to 40 strings: around the 16
    that are copied out inline and the 32 of the smallest segments."""
    rng = np.random.default_rng(length)
    copies = np.tile(np.arange(8, 41), 50)
    values = [bytes(rng.integers(97, 123, length).astype(np.uint8)) for _ in copies]
    strings = [v for v, c in zip(values, copies) for _ in range(c)]
    chars, offs = pkg.pack_strings([strings[i] for i in rng.permutation(len(strings))])
    c = pass_loop(pkg)
    try:
        perm, lcp = c.sort_host(chars, offs, lcp=with_lcp)
    finally:
        c.close()
    check(orc, chars, offs, perm, lcp if with_lcp else None)
