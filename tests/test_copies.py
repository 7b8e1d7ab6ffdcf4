"""Copies of strings in the leaf sorters: tied runs whose strings are equal,
around the 8 chars of a key and the 32 that are compared at a time."""
import numpy as np
import pytest

from test_kernel_edges import check

pytestmark = pytest.mark.gpu

SIZES = [33, 64, 200, 256, 257, 700, 1024, 1025, 3000, 4096]


def copies(kind, n, width, rng):
    """n strings, about 5 of each of n / 5 values of `width` chars."""
    values = rng.integers(97, 123, (max(1, n // 5), width)).astype(np.uint8)
    s = [bytes(v) for v in values[rng.integers(0, len(values), n)]]
    if kind == "one_longer":  # one value's copies go on
        s = [x + bytes(rng.integers(97, 99, 2).astype(np.uint8)) if x == s[0] else x for x in s]
    elif kind == "one_apart":  # they differ in the last char
        s = [x[:-1] + bytes(rng.integers(97, 99, 1).astype(np.uint8)) if x == s[0] else x for x in s]
    elif kind == "mixed_lengths":  # copies of several lengths: some end, some go on
        cut = {x: int(rng.integers(max(1, width - 40), width + 1)) for x in sorted(set(s))}
        s = [x[:cut[x]] for x in s]
    return s


@pytest.mark.parametrize("indirect", [0, 1])
@pytest.mark.parametrize("kind", ["equal", "one_longer", "one_apart", "mixed_lengths"])
@pytest.mark.parametrize("width", [8, 9, 16, 39, 40, 41, 71, 72, 73, 150])
def test_copies_by_length(pkg, orc, width, kind, indirect):
    rng = np.random.default_rng(width)
    strings = [copies(kind, n, width, rng) for n in SIZES]
    chars, offs = pkg.pack_strings([x for s in strings for x in s])
    inst = np.zeros(len(SIZES) + 1, dtype=np.uint64)
    np.cumsum(SIZES, out=inst[1:])
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, indirect)
        for with_lcp in (True, False):
            perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=with_lcp)
            for k in range(len(SIZES)):
                b, e = int(inst[k]), int(inst[k + 1])
                check(orc, chars, offs[b:e], perm[b:e], lcp[b:e] if with_lcp else None)
        for n in (700, 4096):  # the one-block sort
            k = SIZES.index(n)
            b, e = int(inst[k]), int(inst[k + 1])
            check(orc, chars, offs[b:e], *c.sort_host(chars, offs[b:e], lcp=True))
    finally:
        c.close()


@pytest.mark.parametrize("n", [60000, 1500000])
def test_copies_in_large_sorts(pkg, orc, n):
    """The single launch and the pass loop on 20 copies of each value."""
    rng = np.random.default_rng(n)
    values = rng.integers(97, 123, (n // 20, 20)).astype(np.uint8)
    text = np.zeros((n, 21), np.uint8)
    text[:, :20] = values[rng.integers(0, n // 20, n)]
    offs = np.arange(n, dtype=np.uint64) * 21
    c = pkg.Context(0)
    try:
        perm, lcp = c.sort_host(text.reshape(-1), offs, lcp=True)
    finally:
        c.close()
    check(orc, text.reshape(-1), offs, perm, lcp)


@pytest.mark.parametrize("sigma,width,n", [(2, 24, (5 << 19) - 1), (2, 24, 5 << 19), (2, 24, 3200000),
                                           (4, 20, 3000000), (2, 7, 2700000)])
def test_shared_keys_in_the_pass_loop(pkg, orc, sigma, width, n):
    """Segments of few distinct keys, around the size from which they are
    sampled again for a finer tree; keys that end are not counted."""
    rng = np.random.default_rng(sigma + width)
    text = np.zeros((n, width + 1), np.uint8)
    text[:, :width] = rng.integers(97, 97 + sigma, (n, width))
    offs = np.arange(n, dtype=np.uint64) * (width + 1)
    c = pkg.Context(0)
    try:
        perm, lcp = c.sort_host(text.reshape(-1), offs, lcp=True)
    finally:
        c.close()
    check(orc, text.reshape(-1), offs, perm, lcp)
