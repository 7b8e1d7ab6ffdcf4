// kernels_suffix.cuh -- the suffix-sorting specialisation: chain rounds and
// prefix doubling on ranks for inputs that are all suffixes of one text.
//
// The reference sorts suffixes as strings (UCharSuffixSet,
// src/tools/stringset.hpp:732-804: string i is text + i up to the text's
// end), so a group of suffixes sharing a long repeat is walked 8 chars per
// step. Suffixes allow more. The string passes sort them by keys of the
// packed text (Work::ptext), 21 chars of a 4-letter text at a time, and leave
// groups that tie in a whole key: repeats. Two rules finish those:
//
// Chains. When the successors x + 1 of all members x of a group lie in one
// group B, the members share 1 + depth(B) chars and order as they do. Follow
// this from group to group to the first whose successors part, `dist` steps
// on: inside a copied block every group reaches the block's end at once,
// without a char read. A chain round sorts each group by the ranks of the
// members' suffixes dist + 1 chars further; where one of those is in no group
// (it differs from all others within a key) by the packed chars at the depth
// the chain's end is known to share. Every group parts in every round: pairs
// are done after one.
//
// Ranks. Texts whose groups part slowly (periodic ones: only the member next
// to the text's end leaves) go on by prefix doubling: two suffixes x, y that
// share d chars compare as x + d and y + d do, so each group sorts by the rank
// of x + d -- a final position, or the start of that suffix's own group. Ties
// form subgroups whose depth is d plus the depth of the tied group, so the
// depth at least doubles per round.
//
// Bound by random 4-byte accesses to isa and perm. Before, groups that tied
// in 8 chars of text (all 33.5 M suffixes of a 32 MiB text) were sorted by 6
// more and by ranks in ten rounds of doubling, each over up to 1.5 M pairs:
// 6.27 -> 3.46 ms for that sort with packed keys and chain rounds (three of
// them, 0.63 ms), 1.83 -> 1.03 ms for a 5 MB text with LCPs.
//
// Arrays (positions p, suffixes x, both in [0, n)): perm[p] = the suffix at p;
// isa[x] = the start of x's group, its final position once it has left one,
// or DBL_NONE (chain rounds: it was in none); gd[par][s] = depth of the group
// starting at s (read from one parity, written to the other, so a round reads
// a consistent snapshot); key[p] = the rank used this round; chain bits: bit
// x set when the successors of x's group lie in one group.
#pragma once

#include "kernels_small.cuh"

namespace pssgpu {

constexpr uint32_t DBL_NONE = 0xFFFFFFFFu;  // isa: in no group
// largest group of the smaller block sort (256 threads, 12 KB of shared
// memory)
constexpr uint32_t DBL_MID = 1024;
// A chain round's text key: as many packed chars as fit these bits; the key
// and a member index of up to 16 bits fill one 64-bit sort word.
constexpr uint32_t DBL_CHAR_BITS = 48;
constexpr int DBL_CHAIN_ROUNDS = 8;  // at most
constexpr uint32_t DBL_BY_RANK = 1;  // list entry's meta: keys are in key[], depth is the ranks' offset

// Group lists of a round, by size class: 0 at most 32 members (one warp
// each), 1 at most DBL_MID (a block of 256 threads), 2 at most DBL_MAX (a
// block of 512 threads); double-buffered by round parity.
constexpr int CHAIN_LEVELS = 4;
struct DblArrays {
    uint32_t* isa;
    uint32_t* gd[2];
    uint32_t* key;
    Seg* list[3][2];
    uint32_t cap[3];
    // chain bits, and per level the words of the level below that are all
    // ones (32 of them per bit word); clen: words of each level
    uint32_t* chain[CHAIN_LEVELS];
    uint32_t clen[CHAIN_LEVELS];
};

__host__ __device__ constexpr int dbl_class(uint32_t size)
{
    return size <= (uint32_t)WARP_GROUP_MAX ? 0 : size <= DBL_MID ? 1 : 2;
}

// The input is a suffix set when offs[i] == i for all i and no NUL lies
// before the last char (n == nchars is checked by the host): any other
// input sets *flag. alpha (8 words) receives the chars that occur.
__global__ void __launch_bounds__(256) k_suffix_check(const uint8_t* __restrict__ chars,
                                                      const uint64_t* __restrict__ offs, uint64_t n,
                                                      uint32_t* flag, uint32_t* alpha)
{
    __shared__ uint8_t seen[256];
    seen[threadIdx.x] = 0;
    __syncthreads();
    bool bad = false;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (__ldg(offs + i) != i) bad = true;
        const uint8_t c = __ldg(chars + i);
        if (i + 1 < n && c == 0) bad = true;
        seen[c] = 1;
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1u);
    __syncthreads();
    const uint32_t m = __ballot_sync(0xffffffffu, seen[threadIdx.x]);
    if ((threadIdx.x & 31) == 0 && m) atomicOr(alpha + (threadIdx.x >> 5), m);
}

// The packed text: char i at bits [i * kbits, (i + 1) * kbits) from the top
// of word 0 on, as its number among the chars that occur (NUL, at the end, is
// 0); words past the text are 0.
struct PackMap {
    uint8_t code[256];
};
__global__ void __launch_bounds__(256) k_pack_text(const uint8_t* __restrict__ chars, uint64_t n, uint32_t kbits,
                                                   PackMap map, uint64_t* __restrict__ out, uint64_t words)
{
    __shared__ uint8_t code[256];
    code[threadIdx.x] = map.code[threadIdx.x];
    __syncthreads();
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < words;
         j += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t i = 64 * j / kbits;  // the first char with bits in this word
        int at = (int)(64 * j - i * kbits);  // bits of it that lie in the word before
        uint64_t w = 0;
        for (int pos = -at; pos < 64 && i < n; pos += (int)kbits, ++i) {
            const uint64_t c = code[__ldg(chars + i)];
            const int sh = 64 - (int)kbits - pos;
            w |= sh >= 0 ? c << sh : c >> -sh;
        }
        out[j] = w;
    }
}

// A list append of whole warps: every lane calls, lanes with push set append
// s (one global reservation per class and warp).
__device__ __forceinline__ void dbl_push_warp(DblArrays& a, uint32_t* counters, int par, bool push,
                                              const Seg& s)
{
    const uint32_t lane = threadIdx.x & 31;
    const int cls = push ? dbl_class(s.size) : 3;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint32_t m = __ballot_sync(0xffffffffu, cls == c);
        if (!m) continue;
        const int leader = __ffs(m) - 1;
        uint32_t base = 0;
        if (lane == (uint32_t)leader) base = atomicAdd(counters + C_DBL_CNT + 3 * par + c, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (cls == c) {
            const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
            if (at < a.cap[c]) a.list[c][par][at] = s;
            else set_error(counters + C_ERR, ERR_OVERFLOW);
        }
    }
}

// A warp's share of a list: `per` consecutive entries, one per lane (at: the
// first; size 0: none).
__device__ __forceinline__ Seg dbl_entry(const Seg* __restrict__ list, uint32_t count, uint32_t per, uint32_t* at)
{
    const uint32_t lane = threadIdx.x & 31;
    *at = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per;
    const uint32_t g = *at + lane;
    return lane < per && g < count ? list[g] : Seg{0u, 0u, 0u, 0u};
}

// Entries per warp of a list that may hold groups over 32 members: its warp
// takes those one after another, so few of them get a warp each (suffixes of a
// Fibonacci word of 200,000 chars, 89 groups of 2000 on average: 3.80 ms with
// 32 per warp, 1.24 with one).
inline uint32_t dbl_per(uint32_t count)
{
    uint32_t per = 32;
    while (per > 1 && count < per * 2368u) per >>= 1;  // 8 warps on each of 2 x 148 blocks
    return per;
}
inline uint32_t dbl_blocks(uint32_t count, uint32_t per) { return (count + 8 * per - 1) / (8 * per); }

// fn(s, lane, first, step) over the members of a warp's list entries (s
// and its lane): small groups by their own lane (first 0, step 1), larger ones
// by the whole warp.
template <typename Fn>
__device__ __forceinline__ void dbl_each_group(const Seg& s, Fn fn)
{
    const uint32_t lane = threadIdx.x & 31;
    if (s.size <= (uint32_t)WARP_GROUP_MAX) fn(s, lane, 0u, 1u);
    for (uint32_t m = __ballot_sync(0xffffffffu, s.size > (uint32_t)WARP_GROUP_MAX); m; m &= m - 1) {
        const int f = __ffs(m) - 1;
        Seg g;
        g.begin = __shfl_sync(0xffffffffu, s.begin, f);
        g.size = __shfl_sync(0xffffffffu, s.size, f);
        g.depth = __shfl_sync(0xffffffffu, s.depth, f);
        g.meta = __shfl_sync(0xffffffffu, s.meta, f);
        fn(g, (uint32_t)f, lane, 32u);
    }
}

// The groups the passes handed over: their ids into perm (unless they are
// there), their members' isa, their depths, and the round lists of parity 0.
__global__ void __launch_bounds__(256) k_dbl_init(Work w, const Seg* __restrict__ list, uint32_t count,
                                                  uint32_t per, DblArrays a, unsigned long long* members)
{
    uint32_t at;
    const Seg s = dbl_entry(list, count, per, &at);
    const uint32_t m = __reduce_add_sync(0xFFFFFFFFu, s.size);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(members, (unsigned long long)m);
    dbl_each_group(s, [&](const Seg& q, uint32_t, uint32_t first, uint32_t step) {
        for (uint32_t i = first; i < q.size; i += step) {
            const uint32_t p = q.begin + i;
            uint32_t x;
            if (q.meta & META_PERM) {
                x = w.perm[p];
            } else {
                x = h_id(w, handle_at(w, q.meta, q.begin, p));
                w.perm[p] = x;
            }
            a.isa[x] = q.begin;
        }
    });
    if (s.size) a.gd[0][s.begin] = s.depth;
    dbl_push_warp(a, w.counters, 0, s.size != 0, Seg{s.begin, s.size, s.depth, 0u});
}

// Chain bits of every member: set when the successors of its group's members
// lie in one group. (Members share a char, so x + 1 is a suffix.)
__global__ void __launch_bounds__(256) k_dbl_link(const Seg* __restrict__ list, uint32_t count, uint32_t per,
                                                  const uint32_t* __restrict__ perm, DblArrays a)
{
    uint32_t at;
    const Seg s = dbl_entry(list, count, per, &at);
    dbl_each_group(s, [&](const Seg& q, uint32_t, uint32_t first, uint32_t step) {
        if (!q.size) return;
        const uint32_t b = a.isa[perm[q.begin] + 1];
        bool same = b != DBL_NONE;
        for (uint32_t i = first; i < q.size && same; i += step) same = a.isa[perm[q.begin + i] + 1] == b;
        if (step > 1) same = __all_sync(0xffffffffu, same);
        if (!same) return;
        for (uint32_t i = first; i < q.size; i += step) {
            const uint32_t x = perm[q.begin + i];
            atomicOr(a.chain[0] + (x >> 5), 1u << (x & 31));
        }
    });
}

// The next level: bit v set when word v of `in` is all ones.
__global__ void k_chain_level(const uint32_t* __restrict__ in, uint32_t words, uint32_t* __restrict__ out,
                              uint32_t out_words)
{
    for (uint32_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; v0 < 32 * out_words;
         v0 += gridDim.x * blockDim.x) {
        const uint32_t v = v0 + (threadIdx.x & 31);
        const uint32_t m = __ballot_sync(0xffffffffu, v < words && in[v] == 0xFFFFFFFFu);
        if ((threadIdx.x & 31) == 0) out[v0 >> 5] = m;
    }
}

// The first x' >= x with a clear chain bit (the text's last suffix is in no
// group, so there is one).
__device__ __forceinline__ uint32_t chain_end(const DblArrays& a, uint32_t x)
{
    uint32_t pos = x;  // in units of the current level
    int lv = 0;
    // up: the rest of the word at each level
    while (true) {
        const uint32_t wd = pos >> 5;
        if (wd >= a.clen[lv]) return x;  // not reached
        const uint32_t z = ~a.chain[lv][wd] & (0xFFFFFFFFu << (pos & 31));
        if (z) {
            pos = 32 * wd + __ffs(z) - 1;
            break;
        }
        if (lv + 1 < CHAIN_LEVELS) {
            ++lv;
            pos = wd + 1;  // the words behind this one
        } else {
            pos = 32 * (wd + 1);
        }
    }
    // down: the first clear bit of the word found
    while (lv > 0) {
        --lv;
        if (pos >= a.clen[lv]) return x;  // not reached
        const uint32_t z = ~a.chain[lv][pos];
        pos = 32 * pos + (z ? __ffs(z) - 1 : 0);
    }
    return pos;
}

// What a chain round sorts each group by, into its list entry and key[]:
// the ranks dist + 1 chars further, where all have one, else the text at the
// depth the chain's end shares. isa and gd are read as the last round left
// them.
__global__ void __launch_bounds__(256) k_dbl_chain_keys(Seg* __restrict__ list, uint32_t count, uint32_t per,
                                                        const uint32_t* __restrict__ perm, DblArrays a, int par)
{
    uint32_t at;
    const Seg s = dbl_entry(list, count, per, &at);
    dbl_each_group(s, [&](const Seg& q, uint32_t f, uint32_t first, uint32_t step) {
        if (!q.size) return;
        const uint32_t x = perm[q.begin];
        const uint32_t e = chain_end(a, x);
        const uint32_t off = e - x + 1;  // the end's members share a char: their successors exist
        bool ranks = true;
        for (uint32_t i = first; i < q.size; i += step) {
            const uint32_t r = a.isa[perm[q.begin + i] + off];
            a.key[q.begin + i] = r;
            ranks = ranks && r != DBL_NONE;
        }
        if (step > 1) ranks = __all_sync(0xffffffffu, ranks);
        if (first) return;
        const uint32_t b = a.isa[e];
        const uint32_t d = ranks || b == DBL_NONE ? q.depth : max(q.depth, e - x + a.gd[par][b]);
        list[at + f] = Seg{q.begin, q.size, ranks ? off : d, ranks ? DBL_BY_RANK : 0u};
    });
}

// Before the rank rounds: suffixes that were in no group have their position
// as rank (all: every suffix does, for the LCPs).
__global__ void k_dbl_fill(const uint32_t* __restrict__ perm, uint32_t n, uint32_t* __restrict__ isa, int all)
{
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t x = perm[p];
        if (all || isa[x] == DBL_NONE) isa[x] = p;
    }
}

// Rank round step 1: every member's key, the rank of the suffix `depth` chars
// further (members share depth chars, none of them NUL, so x + depth < n).
// k_dbl_keys_small: one thread per group of at most 32; k_dbl_keys: one warp
// per larger group.
__global__ void k_dbl_keys_small(const Seg* __restrict__ list, uint32_t count,
                                 const uint32_t* __restrict__ perm, DblArrays a,
                                 unsigned long long* members)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const Seg s = g < count ? list[g] : Seg{0u, 0u, 0u, 0u};
    const uint32_t m = __reduce_add_sync(0xFFFFFFFFu, s.size);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(members, (unsigned long long)m);
    // four members at a time: their ids, then their ranks, all in flight
    // together (stores to key would otherwise order every next load)
    for (uint32_t q = 0; q < s.size; q += 4) {
        uint32_t x[4], r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = q + j < s.size ? __ldg(perm + s.begin + q + j) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = q + j < s.size ? a.isa[x[j] + s.depth] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (q + j < s.size) a.key[s.begin + q + j] = r[j];
    }
}

__global__ void k_dbl_keys(const Seg* __restrict__ list, uint32_t count,
                           const uint32_t* __restrict__ perm, DblArrays a,
                           unsigned long long* members)
{
    const uint32_t g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g >= count) return;
    const Seg s = list[g];
    if ((threadIdx.x & 31) == 0) atomicAdd(members, (unsigned long long)s.size);
    for (uint32_t q = threadIdx.x & 31; q < s.size; q += 32)
        a.key[s.begin + q] = a.isa[perm[s.begin + q] + s.depth];
}

// The run of equal keys K that starts at offset i0 of group s and has len
// members: for len >= 2 the subgroup (with its depth recorded for the next
// round) into *out. The subgroup lies `step` chars deeper (a text key's
// chars), or, with step 0, as deep as the group ranked K. Returns whether
// *out is to be appended.
__device__ __forceinline__ bool dbl_run(DblArrays& a, int par, const Seg& s, uint32_t i0,
                                        uint32_t len, uint32_t K, Seg* out, uint32_t step)
{
    const uint32_t p = s.begin + i0;
    if (len < 2) return false;
    const uint32_t nd = s.depth + (step ? step : a.gd[par][K]);
    a.gd[par ^ 1][p] = nd;
    *out = Seg{p, len, nd, 0u};
    return true;
}

// A chain round's text key of suffix x at depth d: the packed chars at
// x + d that fit DBL_CHAR_BITS, right-aligned.
__device__ __forceinline__ uint64_t dbl_text_key(const Work& w, uint32_t x, uint32_t d)
{
    const uint32_t bits = min(w.kchars, DBL_CHAR_BITS / w.kbits) * w.kbits;
    return packed_key(w, (uint64_t)x + d) >> (64 - bits);
}
__device__ __forceinline__ uint32_t dbl_text_step(const Work& w) { return min(w.kchars, DBL_CHAR_BITS / w.kbits); }

// Round step 2 for groups of at most 32 members: each warp takes
// DBL_PER_WARP consecutive list entries and packs them into windows of 32
// lanes; a window sorts by (group, key, lane), writes perm and the new ranks,
// and splits every group into runs of equal keys.
constexpr uint32_t DBL_PER_WARP = 16;
__global__ void k_dbl_sort_small(Work w, const Seg* __restrict__ list, uint32_t count,
                                 uint32_t* __restrict__ perm, DblArrays a, uint32_t* counters, int par,
                                 int chain)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t g0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * DBL_PER_WARP;
    if (g0 >= count) return;  // whole warp
    const uint32_t ng = min(DBL_PER_WARP, count - g0);
    warp_seg_windows(list + g0, ng, [&](const Seg& s, uint32_t gq, uint32_t gs, bool real) {
        const uint32_t mem = real ? lane - gs : 0u;
        const uint32_t x = real ? perm[s.begin + mem] : 0u;
        const bool text = chain && !(s.meta & DBL_BY_RANK);
        const uint64_t key = !real ? 0ull : text ? dbl_text_key(w, x, s.depth) : a.key[s.begin + mem];
        uint64_t t = real ? ((uint64_t)gq << 58) | (key << 5) | lane : ~0ull;
#pragma unroll
        for (uint32_t kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
            for (uint32_t j = kk >> 1; j > 0; j >>= 1) {
                const uint64_t o = __shfl_xor_sync(0xffffffffu, t, j);
                const bool lower = (lane & j) == 0, asc = (lane & kk) == 0;
                if ((lower == asc) ? (o < t) : (o > t)) t = o;
            }
        }
        // groups keep their lane ranges: sorted by group first
        const uint64_t K = (t >> 5) & ((1ull << 53) - 1);  // the key (group bits dropped)
        const uint32_t mx = __shfl_sync(0xffffffffu, x, (uint32_t)t & 31u);
        const uint64_t pk = __shfl_up_sync(0xffffffffu, K, 1);
        const bool start = real && (lane == gs || pk != K);
        const uint32_t S = __ballot_sync(0xffffffffu, start);
        const uint32_t rs = 31u - __clz(S & (0xFFFFFFFFu >> (31 - lane)));
        const uint32_t above = lane == 31 ? 0u : (S & (0xFFFFFFFFu << (lane + 1)));
        const uint32_t ge = gs + (real ? s.size : 0u);
        const uint32_t re = above ? min((uint32_t)(__ffs(above) - 1), ge) : ge;
        bool push = false;
        Seg ns{};
        if (real) {
            // unchanged values are not written back: a member that kept its
            // place keeps its perm entry, a run at its group's start the
            // group's rank
            if (mx != x) perm[s.begin + mem] = mx;
            if (rs != gs) a.isa[mx] = s.begin + (rs - gs);  // final position for a single member
            if (start)
                push = dbl_run(a, par, s, rs - gs, re - rs, (uint32_t)K, &ns, text ? dbl_text_step(w) : 0u);
        }
        dbl_push_warp(a, counters, par ^ 1, push, ns);
    });
}

// Round step 2 for groups of 33..MAXM members, one block each: a bitonic
// sort of (key << 32 | member index) in shared memory (dynamic: MAXM keys,
// then MAXM member ids), padded to a power of two with keys that the network
// never moves (bitonic_sort_block_padded).
template <uint32_t MAXM>
__global__ void __launch_bounds__(MAXM <= DBL_MID ? 256 : 512) k_dbl_sort_block(
    Work w, const Seg* __restrict__ list, uint32_t* __restrict__ perm, DblArrays a, uint32_t* counters,
    int par, int chain)
{
    static_assert(MAXM <= (1u << (64 - DBL_CHAR_BITS)), "member index beside a text round's key");

    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* sk = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t* sx = reinterpret_cast<uint32_t*>(smem_raw + 8 * MAXM);
    const Seg s = list[blockIdx.x];
    const bool text = chain && !(s.meta & DBL_BY_RANK);
    const uint32_t step = text ? dbl_text_step(w) : 0u;
    const uint32_t m = s.size;
    uint32_t S = 64;
    while (S < m) S <<= 1;
    for (uint32_t q = threadIdx.x; q < S; q += blockDim.x) {
        if (q < m) {
            const uint32_t x = perm[s.begin + q];
            sx[q] = x;
            sk[q] = text ? (dbl_text_key(w, x, s.depth) << (64 - DBL_CHAR_BITS)) | q
                         : ((uint64_t)a.key[s.begin + q] << 32) | q;
        } else {
            sk[q] = ~0ull;
        }
    }
    __syncthreads();
    bitonic_sort_block_padded(sk, S, m);
    // warp-uniform trip counts, so that appends aggregate per warp
    for (uint32_t i0 = threadIdx.x & ~31u; i0 < m; i0 += blockDim.x) {
        const uint32_t i = i0 + (threadIdx.x & 31);
        bool push = false;
        Seg ns{};
        if (i < m) {
            const uint32_t ksh = text ? 64 - DBL_CHAR_BITS : 32;
            const uint64_t K = sk[i] >> ksh;
            const uint32_t src = (uint32_t)sk[i] & (MAXM - 1);
            if (src != i) perm[s.begin + i] = sx[src];  // unchanged entries are not rewritten
            if (i == 0 || (sk[i - 1] >> ksh) != K) {
                // a run starts here: its length, then every member's rank (a
                // run at the group's start keeps its own)
                uint32_t e = i + 1;
                while (e < m && (sk[e] >> ksh) == K) ++e;
                if (i)
                    for (uint32_t q = i; q < e; ++q) a.isa[sx[(uint32_t)sk[q] & (MAXM - 1)]] = s.begin + i;
                push = dbl_run(a, par, s, i, e - i, (uint32_t)K, &ns, step);
            }
        }
        dbl_push_warp(a, counters, par ^ 1, push, ns);
    }
}

// The LCP array of a suffix set, in text order, a warp per 32 suffixes (isa
// holds every suffix's position). When suffix x and its predecessor y in
// sorted order share their first char and the predecessor of x + 1 is y + 1,
// the LCP of x is one more than that of x + 1 (the Phi-array
// argument of Kasai et al.): inside a copied block a warp's suffixes form one
// chain and only its last one is compared. A chain's end takes DBL_LCP_STEPS
// steps of 8 chars by its own lane, which end nearly every compare outside
// long repeats; what is still equal is compared by the whole warp, 512 chars
// a step. Latency-bound by the longest compare: with one lane walking a
// 10 KiB repeat 8 chars a step the LCP sort of a 5 MB text with copied blocks
// took 6.38 ms (4.82 of them in that kernel), in this form 1.86 ms.
constexpr uint32_t DBL_LCP_STEPS = 4;
__global__ void k_dbl_lcp(const uint8_t* __restrict__ chars, uint64_t nchars,
                          const uint32_t* __restrict__ perm, const uint32_t* __restrict__ isa,
                          uint32_t* __restrict__ lcp, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t x0 = 32 * (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); x0 < n; x0 += 32 * nwarps) {
        const uint64_t x = x0 + lane;
        const uint32_t p = x < n ? isa[x] : 0u;
        const bool act = p != 0;  // the smallest suffix has no predecessor
        const uint32_t y = act ? perm[p - 1] : 0u;
        const uint32_t ny = __shfl_down_sync(0xFFFFFFFFu, y, 1);
        const bool nact = __shfl_down_sync(0xFFFFFFFFu, act ? 1u : 0u, 1);
        const bool tail = act && (lane == 31 || !nact || ny != y + 1 || chars[x] != chars[y]);
        uint32_t d = 0;  // depth of the compare
        uint32_t l = 0;
        bool open = tail;
        auto settle = [&](uint64_t a, uint64_t b, uint32_t dd) {  // compares 8 chars; false: all equal
            const uint64_t ka = load_key(chars, nchars, a + dd), kb = load_key(chars, nchars, b + dd);
            if (ka == kb && !key_terminated(ka)) return false;
            l = dd + (ka != kb ? lcp_key_type(ka, kb) : lcp_key_depth(ka));
            return true;
        };
        for (uint32_t s = 0; s < DBL_LCP_STEPS && open; ++s) {
            if (settle(x, y, d)) open = false;
            else d += 8;
        }
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, open); todo; todo &= todo - 1) {
            const int f = __ffs(todo) - 1;
            const uint64_t xf = x0 + f;
            const uint64_t yf = __shfl_sync(0xFFFFFFFFu, y, f);
            uint32_t df = __shfl_sync(0xFFFFFFFFu, d, f);
            while (true) {
                // lane l compares the chars from 16 l on; equal windows
                // without a NUL continue
                uint64_t ra[2], rb[2];
                load_raw_chunks<2>(chars, nchars, xf + df + 16 * lane, 2, ra);
                load_raw_chunks<2>(chars, nchars, yf + df + 16 * lane, 2, rb);
                const uint64_t z0 = (ra[0] - 0x0101010101010101ull) & ~ra[0] & 0x8080808080808080ull;
                const uint64_t z1 = (ra[1] - 0x0101010101010101ull) & ~ra[1] & 0x8080808080808080ull;
                const bool m0 = ra[0] != rb[0] || z0, m1 = ra[1] != rb[1] || z1;
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, m0 || m1);
                if (bal) {
                    const int fl = __ffs(bal) - 1;
                    df += 16 * fl + (__shfl_sync(0xFFFFFFFFu, m0 ? 1 : 0, fl) ? 0 : 8);
                    break;
                }
                df += 512;
            }
            if (lane == (uint32_t)f) settle(xf, yf, df);
        }
        const uint32_t ends = __ballot_sync(0xFFFFFFFFu, tail) & (0xFFFFFFFFu << lane);
        const uint32_t src = ends ? (uint32_t)(__ffs(ends) - 1) : lane;
        const uint32_t le = __shfl_sync(0xFFFFFFFFu, l, src);
        if (act) lcp[p] = le + (src - lane);
    }
}

}  // namespace pssgpu
