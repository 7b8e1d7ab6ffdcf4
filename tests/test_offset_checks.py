"""String offsets outside the arena: every kernel that reads a root segment
reports them (PSSGPU_EINVAL), and no address is formed from them."""
import subprocess

import numpy as np
import pytest

import __graft_entry__

SOURCE = """
#include <cstdio>
#include "device_common.cuh"
int main()
{
    unsigned long long chars, nchars, p;
    unsigned cnt;
    while (std::scanf("%llu %llu %llu %u", &chars, &nchars, &p, &cnt) == 4) {
        const pssgpu::RawRange r(chars, p, cnt);
        unsigned mask = 0;
        for (int i = 0; i < 8; ++i) mask |= (r.reads(i, nchars) ? 1u : 0u) << i;
        std::printf("%llu %u\\n", (unsigned long long)(r.at15 - 15), mask);
    }
}
"""


def test_raw_chunk_reads_stay_in_the_arena(tmp_path):
    """The address computation of the 16-byte loads, on the host: every block
    read holds a char of the arena, for any position up to 2^64 - 1; one inside
    the arena reads the blocks from its own on that its windows need, one at
    least 16 chars past the end and not just below 2^64 reads none."""
    build = __graft_entry__._load_build_module()
    src, exe = tmp_path / "raw_range.cu", tmp_path / "raw_range"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, "-std=c++17", "-I", str(build.CSRC), "-o", str(exe), str(src)], check=True)
    base = 0x7F0000000000
    cases = []
    for lead in (0, 8):
        for nchars in (1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 100, 1000, 1 << 33):
            inside = {0, 1, 7, 8, 9, 15, 16, 17, nchars // 2, nchars - 9, nchars - 2, nchars - 1}
            outside = {nchars, nchars + 1, nchars + 5, nchars + 15, nchars + 16, 1 << 62, (1 << 63) - 64,
                       (1 << 63) - 1, 1 << 63, (1 << 63) + 12345, (1 << 64) - 17, (1 << 64) - 16,
                       (1 << 64) - 9, (1 << 64) - 8, (1 << 64) - 1}
            cases += [(base + lead, nchars, p, cnt) for p in sorted(inside | outside) if p >= 0 for cnt in (1, 2, 4, 7)]
    out = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), text=True,
                         capture_output=True, check=True).stdout.split()
    assert len(out) == 2 * len(cases)
    for (chars, nchars, p, cnt), at, mask in zip(cases, map(int, out[::2]), map(int, out[1::2])):
        blocks = [(chars + at + 16 * i) % 2**64 for i in range(8) if mask >> i & 1]
        assert all(x % 16 == 0 and x + 15 >= chars and x < chars + nchars for x in blocks), (chars, nchars, p, cnt)
        if p < nchars:
            # the windows' chars and the rest of their last word
            last = (chars + p) // 8 * 8 + 8 * cnt + 7
            assert blocks == [x for x in range((chars + p) // 16 * 16, last + 1, 16) if x < chars + nchars]
        elif nchars + 16 <= p < 2**64 - 8 * (cnt + 2):
            assert not blocks


def instance(n, prefix, rng):
    return [prefix + bytes(rng.integers(97, 123, int(rng.integers(0, 12))).astype(np.uint8)) for _ in range(n)]


# strings of the instance that holds the offset, and the chars they share: a
# one-string root (k_roots), k_tiny, k_segs of 1, 4 and 16 warps, k_classify
# without and behind a common-prefix jump
ROOTS = {"one": (1, 0), "tiny": (20, 0), "segs1": (200, 0), "segs4": (700, 0), "segs16": (3000, 0),
         "classify": (6000, 0), "classify_jump": (6000, 24)}


@pytest.mark.gpu
@pytest.mark.parametrize("indirect", [0, 1])
@pytest.mark.parametrize("root", list(ROOTS))
def test_offsets_outside_the_arena(pkg, orc, root, indirect):
    """One offset of nchars or nchars + 5 among the first, middle and last
    strings of a root segment, in a batch and alone, with and without LCPs and
    with both handle formats; the context sorts the strings themselves
    afterwards."""
    n, shared = ROOTS[root]
    rng = np.random.default_rng(n + shared)
    sets = [instance(37, b"", rng), instance(n, b"p" * shared, rng), instance(5, b"", rng)]
    chars, offs = pkg.pack_strings([x for s in sets for x in s])
    inst = np.zeros(4, dtype=np.uint64)
    np.cumsum([len(s) for s in sets], out=inst[1:])
    b, e = int(inst[1]), int(inst[2])
    c = pkg.Context(0)
    try:
        c.set_option(c.OPT_INDIRECT_HANDLES, indirect)
        c.set_option(c.OPT_SINGLE_LAUNCH, 0)
        for at in sorted({b, b + n // 2, e - 1}):
            for outside in (chars.shape[0], chars.shape[0] + 5):
                bad = offs.copy()
                bad[at] = outside
                for lcp in (False, True):
                    with pytest.raises(pkg.SortError) as err:
                        c.sort_batch_host(chars, bad, inst, lcp=lcp)
                    assert err.value.status == 1
                    if n > 1:
                        with pytest.raises(pkg.SortError) as err:
                            c.sort_host(chars, bad[b:e], lcp=lcp)
                        assert err.value.status == 1
        perm, lcp = c.sort_batch_host(chars, offs, inst, lcp=True)
    finally:
        c.close()
    for k in range(3):
        lo, hi = int(inst[k]), int(inst[k + 1])
        ids, want = orc.sort_ids_lcp(chars, offs[lo:hi])
        assert orc.check_permutation(perm[lo:hi])
        assert orc.check_order(chars, offs[lo:hi], perm[lo:hi]) == -1
        assert np.array_equal(lcp[lo + 1:hi].astype(np.uint64), want[1:])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [20, 700, 4096, 4097, 60000])
def test_offsets_outside_the_arena_single_launch(pkg, n):
    """The same for the one-block and the cooperative single launch."""
    rng = np.random.default_rng(n)
    chars, offs = pkg.pack_strings(instance(n, b"", rng))
    c = pkg.Context(0)
    try:
        for outside in (chars.shape[0], chars.shape[0] + 5):
            bad = offs.copy()
            bad[n // 3] = outside
            for lcp in (False, True):
                with pytest.raises(pkg.SortError) as err:
                    c.sort_host(chars, bad, lcp=lcp)
                assert err.value.status == 1
    finally:
        c.close()
