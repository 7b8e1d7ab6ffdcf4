"""Root segments, whose handles each kernel makes from the offsets: both handle
formats (an id with its offset, or the id alone), ids of the whole input or of
the instance, against the oracle."""
import numpy as np
import pytest

from test_kernel_edges import LEAF_SIZES, check, leaf_strings, pass_loop

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_lcp", [True, False])
@pytest.mark.parametrize("kind", ["letters", "acgt", "eighth", "prefix", "runs"])
def test_indirect_leaf_sizes(pkg, orc, kind, with_lcp):
    """The leaf sorters at the edges of their size classes on bare ids, one
    instance of a batch per size (without LCPs: ids made local behind the
    passes)."""
    rng = np.random.default_rng(100 + len(kind))
    strings = [leaf_strings(kind, n, rng) for n in LEAF_SIZES]
    chars, offs = pkg.pack_strings([x for s in strings for x in s])
    inst = np.zeros(len(LEAF_SIZES) + 1, dtype=np.uint64)
    np.cumsum(LEAF_SIZES, out=inst[1:])
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, 1)
        perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=with_lcp)
    finally:
        c.close()
    for k in range(len(LEAF_SIZES)):
        b, e = int(inst[k]), int(inst[k + 1])
        check(orc, chars, offs[b:e], perm[b:e], lcp[b:e] if with_lcp else None)


@pytest.mark.parametrize("indirect", [0, 1])
@pytest.mark.parametrize("n", [2, 32, 33, 256, 257, 1024, 1025, 4096, 4097])
def test_single_root_sizes(pkg, orc, n, indirect):
    """One root segment in the pass loop at the edges of its kernels, with
    and without LCPs."""
    rng = np.random.default_rng(n)
    c = pass_loop(pkg)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, indirect)
        for kind in ("letters", "prefix"):
            chars, offs = pkg.pack_strings(leaf_strings(kind, n, rng))
            for lcp in (True, False):
                check(orc, chars, offs, *c.sort_host(chars, offs, lcp=lcp))
    finally:
        c.close()


@pytest.mark.parametrize("ninst", [1, 513, 310000])
def test_indirect_batch_roots(pkg, ninst):
    """Instances of every class on bare ids, without LCPs."""
    rng = np.random.default_rng(7 + ninst)
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
        c.set_option(c.OPT_INDIRECT_HANDLES, 1)
        perm, _ = c.sort_batch_host(text.reshape(-1), offs, inst, lcp=False)
    finally:
        c.close()
    of = np.repeat(np.arange(ninst), sizes)
    want = np.lexsort((number, of)) - inst[of].astype(np.int64)
    assert np.array_equal(perm.astype(np.int64), want)


@pytest.mark.parametrize("indirect", [0, 1])
def test_tiles_in_descending_sizes(pkg, orc, indirect):
    """The tile sizes' edges from the largest down on one context: a workspace
    sized for more strings serves the rules of fewer."""
    c = pass_loop(pkg)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, indirect)
        for n in (4718593, 528385, 524289, 524288, 6145, 6144, 6143, 4097):
            chars, offs, _ = pkg.workloads.random_strings(n, 0, 12, b"abcde", n)
            perm, lcp = c.sort_host(chars, offs, lcp=True)
            if n < 1 << 20:
                check(orc, chars, offs, perm, lcp)
            else:
                assert pkg.workloads.check_permutation(perm)
                assert pkg.workloads.check_sorted(chars, chars.shape[0], offs, perm) == -1
    finally:
        c.close()


@pytest.mark.parametrize("indirect", [0, 1])
@pytest.mark.parametrize("width", [7, 8, 9, 31, 32, 39, 40, 41, 100])
def test_small_segments_behind_whole_keys(pkg, orc, width, indirect):
    """Instances of 2 to 32 strings that share whole 8-char keys: all equal, in
    two halves, or apart behind `width` chars, beside instances of random
    strings (the turns of k_tiny, around their last one)."""
    rng = np.random.default_rng(width)
    strings, sizes = [], []
    for n in list(range(2, 33)) * 3:
        head = bytes(rng.integers(97, 123, width).astype(np.uint8))
        kind = int(rng.integers(4))
        if kind == 0:
            s = [head] * n
        elif kind == 1:
            s = [head] * (n // 2) + [head[:-1] + b"~"] * (n - n // 2)
        elif kind == 2:
            s = [head + bytes(rng.integers(97, 100, int(rng.integers(0, 4))).astype(np.uint8)) for _ in range(n)]
        else:
            s = [bytes(rng.integers(97, 123, int(rng.integers(0, 12))).astype(np.uint8)) for _ in range(n)]
        strings += [s[i] for i in rng.permutation(n)]
        sizes.append(n)
    chars, offs = pkg.pack_strings(strings)
    inst = np.zeros(len(sizes) + 1, dtype=np.uint64)
    np.cumsum(sizes, out=inst[1:])
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, indirect)
        for with_lcp in (True, False):
            perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=with_lcp)
            for k in range(len(sizes)):
                b, e = int(inst[k]), int(inst[k + 1])
                check(orc, chars, offs[b:e], perm[b:e], lcp[b:e] if with_lcp else None)
    finally:
        c.close()
