"""The tuning table covers the segments that have a splitter tree."""
import re
from pathlib import Path

import numpy as np
import pytest

from golden_util import canonical_ids

PKG = Path(__file__).resolve().parent.parent / "parallel-string-sorting_b200"


def autotune(pkg):
    from importlib import import_module
    return import_module(pkg.__name__ + ".autotune")


def test_classes_are_those_of_big_segments(pkg):
    """Segments of up to SMALL_MAX strings go to the leaf sorters, which have no
    tree: no class below it is tuned or has an entry, and the tuner's instances
    are larger."""
    at = autotune(pkg)
    leaf = int(re.search(r"SMALL_MAX = (\d+);", (PKG / "csrc" / "work.cuh").read_text()).group(1))
    assert at.LEAF_MAX == leaf
    first = leaf.bit_length() - 1
    assert list(at.CLASSES)[0] == first
    table = at.load_table()
    assert not any(table[:first]) and all(table[k] for k in at.CLASSES)
    _, offs, _, inst = at._class_batch(first, 100_000, 3)
    sizes = np.diff(inst.astype(np.int64))
    assert sizes.min() > leaf and sizes.max() < 2 << first and sizes.sum() == len(offs)


@pytest.mark.gpu
def test_every_tree_depth_keeps_the_output(pkg, orc):
    """Instances of classes 12 to 15, sorted with every depth set for all of
    them."""
    rng = np.random.default_rng(12)
    sizes = [4097, 6000, 9000, 20000, 40000]
    inst = np.zeros(len(sizes) + 1, dtype=np.uint64)
    np.cumsum(sizes, out=inst[1:])
    chars, offs, _ = pkg.workloads.random_strings(int(inst[-1]), 0, 14, b"abcd", 12)
    want = [orc.sort_ids_lcp(chars, offs[int(b):int(e)]) for b, e in zip(inst, inst[1:])]
    c = pkg.Context(0)
    try:
        for bits in range(1, 11):
            c.set_tree_bits([0] * 12 + [bits] * 4 + [0] * 17)
            perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=True)
            for (b, e), (ids, rlcp) in zip(zip(inst.astype(int), inst[1:].astype(int)), want):
                assert np.array_equal(lcp[b + 1:e].astype(np.uint64), rlcp[1:])
                assert np.array_equal(canonical_ids(chars, offs[b:e], perm[b:e], rlcp),
                                      canonical_ids(chars, offs[b:e], ids, rlcp))
    finally:
        c.close()
