"""Buckets of the single-launch sort that are larger than a window: many of
them, of every kind, against the oracle."""
import numpy as np
import pytest

from test_kernel_edges import check

pytestmark = pytest.mark.gpu


def letters(n, width, sigma, rng):
    return [bytes(r) for r in rng.integers(97, 97 + sigma, (n, width)).astype(np.uint8)]


@pytest.mark.parametrize("kind", ["binary", "equal", "one_value", "over_4096", "mixed"])
@pytest.mark.parametrize("n", [5000, 40000, 300000])
def test_large_buckets(pkg, orc, kind, n):
    """Keys over 2 letters (about as many large buckets as blocks), equal
    strings that end in their key (2, 60 and all), buckets over the leaf
    sorters' 4096, and all of these with random strings between them."""
    rng = np.random.default_rng(n + len(kind))
    if kind == "binary":
        s = letters(n, 20, 2, rng)
    elif kind == "equal":
        v = letters(60, 5, 26, rng)
        s = [v[i] for i in rng.integers(0, 60, n // 2)] + [v[i] for i in rng.integers(0, 2, n - n // 2)]
    elif kind == "one_value":
        s = [b"a" * 7] * n
    elif kind == "over_4096":
        v = letters(5, 8, 26, rng)
        s = [v[i] + t for i, t in zip(rng.integers(0, 5, n), letters(n, 6, 3, rng))]
    else:
        part = n // 5
        v = letters(4, 8, 26, rng)
        s = (letters(part, 20, 2, rng) + [v[0][:6]] * part + [v[1] + t for t in letters(part, 5, 4, rng)]
             + [v[2]] * 1500 + letters(n - 3 * part - 1500, 12, 26, rng))
    s = [s[i] for i in rng.permutation(n)]
    chars, offs = pkg.pack_strings(s)
    c = pkg.Context(0)
    try:
        perm, lcp = c.sort_host(chars, offs, lcp=True)
        only, _ = c.sort_host(chars, offs, lcp=False)
    finally:
        c.close()
    check(orc, chars, offs, perm, lcp)
    check(orc, chars, offs, only, None)
