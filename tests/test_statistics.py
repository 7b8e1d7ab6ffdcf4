"""What a context reports of its last sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,lcp,single,want", [
    (False, False, 1, 1),  # the one-block sort
    (False, False, 0, 3),  # roots, the leaf sorter, the end of the pass
    (False, True, 0, 4),   # and the end of the sort
    (True, False, 0, 4),   # roots, their end, the leaf sorter, the end of the pass
    (True, True, 0, 6),    # local ids and the end of the sort behind them
])
def test_kernel_launches_counts_every_kernel(pkg, batch, lcp, single, want):
    chars, offs = pkg.pack_strings([b"b", b"a", b"d", b"c"])
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_SINGLE_LAUNCH, single)
        if batch:
            c.sort_batch_host(chars, offs, np.array([0, 2, 4], np.uint64), lcp=lcp)
        else:
            c.sort_host(chars, offs, lcp=lcp)
        assert c.stats()["kernel_launches"] == want
    finally:
        c.close()


def suffix_sort_launches(pkg, orc, text):
    """The launches per kernel class of the sort of all suffixes of a text,
    whose result is checked."""
    chars = np.concatenate([text, np.zeros(1, np.uint8)])
    offs = np.arange(chars.shape[0], dtype=np.uint64)
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_SINGLE_LAUNCH, 0)
        perm, lcp = c.sort_host(chars, offs, lcp=True)
        used = {k["name"]: k["launches"] for k in c.kernel_stats()}
    finally:
        c.close()
    ids, want = orc.sort_ids_lcp(chars, offs)  # suffixes are distinct: one order
    assert np.array_equal(perm, ids)
    assert np.array_equal(lcp[1:].astype(np.uint64), want[1:])
    return used


def test_suffix_rounds_by_text(pkg, orc):
    """Which rounds finish a suffix set: none where all suffixes part within a
    key, chain rounds alone for copied blocks, rank rounds for a periodic
    text, whose groups part one member at a time."""
    rng = np.random.default_rng(5)
    letters = rng.choice(np.frombuffer(b"ACGT", np.uint8), 6000)
    used = suffix_sort_launches(pkg, orc, letters)
    assert used["doubling"] == used["chain_rounds"] == used["rank_rounds"] == 0

    copies = letters.copy()
    copies[4000:4500] = copies[100:600]
    used = suffix_sort_launches(pkg, orc, copies)
    assert used["chain_rounds"] > 0 and used["rank_rounds"] == 0
    assert used["groups32"] > 0 and used["groups1024"] == used["groups4096"] == 0

    periodic = np.tile(np.frombuffer(b"abcab", np.uint8), 2000)
    used = suffix_sort_launches(pkg, orc, periodic)
    assert used["chain_rounds"] > 0 and used["rank_rounds"] > 0 and used["groups4096"] > 0


@pytest.mark.parametrize("copies,groups", [(32, "groups32"), (33, "groups1024"), (1024, "groups1024"),
                                           (1025, "groups4096"), (4000, "groups4096")])
def test_suffix_group_classes(pkg, orc, copies, groups):
    """Groups at the edges of the three group sorts: that many copies of one
    word of 40 letters, each behind and before random ones."""
    rng = np.random.default_rng(copies)
    letters = np.frombuffer(b"ACGT", np.uint8)
    word = rng.choice(letters, 40)
    text = np.concatenate([x for _ in range(copies) for x in (word, rng.choice(letters, 25))] + [rng.choice(letters, 5000)])
    used = suffix_sort_launches(pkg, orc, text)
    assert used[groups] > 0
    if groups != "groups4096":
        assert used["groups4096"] == 0
    if groups == "groups32":
        assert used["groups1024"] == 0


@pytest.mark.parametrize("words,copies", [(100, 33), (600, 33), (1500, 40)])
def test_suffix_many_larger_groups(pkg, orc, words, copies):
    """Lists of about 2,000, 12,000 and 30,000 groups over 32 members, of which
    a warp takes one, two and eight."""
    rng = np.random.default_rng(words)
    letters = np.frombuffer(b"ACGT", np.uint8)
    word = rng.choice(letters, (words, 40))
    text = np.concatenate([np.concatenate([word, rng.choice(letters, (words, 25))], 1).reshape(-1)
                           for _ in range(copies)])
    used = suffix_sort_launches(pkg, orc, text)
    assert used["groups1024"] > 0
