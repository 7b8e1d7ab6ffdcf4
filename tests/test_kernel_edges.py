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
