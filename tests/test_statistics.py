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
