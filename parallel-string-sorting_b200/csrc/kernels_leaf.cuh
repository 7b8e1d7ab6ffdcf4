// kernels_leaf.cuh -- finishing of the segments the sample-sort passes do not
// split any further, at most SMALL_MAX strings, by sorting networks in
// registers. The device counterpart of pS5's base cases on 8-byte caches
// (sort_mkqs_cache / insertion_sort_cache, src/parallel/
// bingmann-parallel_sample_sort.hpp:805-861, 1056-1178) and its sequential
// sample sort (hpp:565-676).
//
// A string is one 64-bit word while it is sorted: its key, shifted left past
// the bits that all keys of the segment share, over the string's index in the
// segment. Words are distinct, their order is the key order, and the index
// says where the string came from, so a compare-exchange moves one register
// pair and no payload. When the shared bits leave no room for the index, the
// word holds the first 7 (or 6) chars of the key only, and ties in those
// continue at that depth.
//
//   k_tiny      2..32 strings: one thread per segment, Batcher's odd-even
//               merge network over its 8, 16 or 32 registers
//   k_segs<1>   33..256 strings: one warp per segment, 2, 4 or 8 words a lane
//   k_segs<4>   257..1024 strings: a block of 4 warps
//   k_segs<16>  1025..4096 strings: a block of 16 warps
//
// All are bound by instructions (26 warp instructions per string in k_segs<16>,
// issue slots 60% busy) and, the smaller ones, by their fetch.
// Measured in the 64 Mi prefix sort, 67 M strings: 27, 32, 32 and 62 ps per
// string. Sample-sort steps in shared memory with a warp window per 32
// strings took 30 ps (2..32 strings), 66 (33..256) and 67 (257..1024), and
// segments of 1025..4096 strings one more sample-sort pass (about 42 ps)
// before them: 9.29 -> 7.42 ms per sort; 100k-instance batch 3.86 -> 2.48 ms.
//
// Strings whose whole words tie and do not end are sorted on together by their
// next chars, end as copies of one string (equal_runs), or go to warp windows
// (kernels_small.cuh), up to 32 strings of several groups at a time, or to the
// next pass; larger tied groups are sorted again by their warps, behind their
// common prefix.
#pragma once

#include <utility>

#include "kernels_small.cuh"

namespace pssgpu {

// Order of two 64-bit words. WORD62: both are below 2^62, so that their bits
// are non-negative finite doubles in the same order, and the compare runs on
// the FP64 pipe instead of the integer ALU, which bounds the warp sorts (75%
// busy in k_segs<16>): 1.16 -> 1.07 ms for the 27.7 M strings that kernel sorts
// of the 100k-instance batch.
template <bool WORD62>
__device__ __forceinline__ bool word_less(uint64_t a, uint64_t b)
{
    if constexpr (WORD62) return __longlong_as_double((long long)a) < __longlong_as_double((long long)b);
    else return a < b;
}

template <bool WORD62>
__device__ __forceinline__ void cmp_exchange(uint64_t& a, uint64_t& b)
{
    const bool s = word_less<WORD62>(b, a);
    const uint64_t lo = s ? b : a;
    b = s ? a : b;
    a = lo;
}

// Key of the string behind handle h at depth d; SFX: a suffix set (whose keys
// are packed and whose ties go to the list dbl; the leaf kernels are built for
// each, as the one's code costs the other instruction cache: suffixes of a
// 32 MiB text 3.46 ms with both in one kernel, 3.27 with either).
template <bool SFX>
__device__ __forceinline__ uint64_t leaf_key(const Work& w, uint64_t h, uint32_t d)
{
    if constexpr (SFX) return packed_key(w, h_off(w, h) + d);
    else return load_key(w.chars, w.nchars, h_off(w, h) + d);
}

__device__ __forceinline__ void cmp_exchange(uint32_t& a, uint32_t& b)
{
    const uint32_t lo = min(a, b);
    b = max(a, b);
    a = lo;
}

// Batcher's odd-even merge sorting network for N (a power of two) inputs:
// 19 compare-exchanges for 8, 63 for 16, 191 for 32.
template <int N>
struct OddEvenNet {
    int a[N * N / 4 + N] = {};
    int b[N * N / 4 + N] = {};
    int size = 0;
    constexpr OddEvenNet()
    {
        for (int p = 1; p < N; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j + k < N; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < N; ++i)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p)) {
                            a[size] = i + j;
                            b[size] = i + j + k;
                            ++size;
                        }
    }
};

template <int N, int I>
__device__ __forceinline__ void net_step(uint32_t (&x)[N])
{
    constexpr OddEvenNet<N> net{};
    constexpr int a = net.a[I], b = net.b[I];
    cmp_exchange(x[a], x[b]);
}

template <int N, int... I>
__device__ __forceinline__ void net_run(uint32_t (&x)[N], std::integer_sequence<int, I...>)
{
    (net_step<N, I>(x), ...);
}

template <int N>
__device__ __forceinline__ void net_sort(uint32_t (&x)[N])
{
    constexpr OddEvenNet<N> net{};
    net_run<N>(x, std::make_integer_sequence<int, net.size>{});
}

// Barrier of the G warps that sort a segment together (G > 1: a whole block).
template <int G>
__device__ __forceinline__ void group_sync()
{
    if constexpr (G == 1) __syncwarp();
    else __syncthreads();
}

// Ascending bitonic sort of 32 * E * G words held by G warps (G > 1: a block
// of 32 * G threads), position t * E + e in x[e] of thread t afterwards.
// Every merge starts by comparing positions with their mirror in the merged
// block, so all compares are ascending. Partner distances below E stay
// inside a thread, those inside a warp are shuffles, longer ones go through
// xb (32 * E * G words of shared memory, G > 1 only). A merge with log2(E) or
// more of the longer ones takes that many of them, the mirror first, in one
// exchange: each thread loads the E words that meet in them, compares them in
// registers and stores them in place. That is 4 accesses per word and 3
// barriers instead of 2 and 2 per distance, and half the compares: the 27.7 M
// strings that k_segs<16> sorts of the 100k-instance batch 1.08 -> 1.04 ms, the
// batch 2.035 -> 1.994 ms. Exchanges in place of the shuffles, too, were slower
// (2.153 ms): the two shuffles of a distance cost less than shared accesses.
template <int E, int G, bool WORD62>
__device__ __forceinline__ void group_sort(uint64_t (&x)[E], uint64_t* xb)
{
    constexpr uint32_t T = 32 * G;
    constexpr int FB = E == 8 ? 3 : E == 4 ? 2 : 1;  // log2(E)
    constexpr bool FUSED = E >= 4 && G >= E;
    const uint32_t t = G == 1 ? threadIdx.x & 31 : threadIdx.x;
    auto inner = [&](int j) {  // distances j, j/2, .., 1 inside the threads
#pragma unroll
        for (int d = E / 2; d > 0; d >>= 1) {
            if (d > j) continue;
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!(e & d)) cmp_exchange<WORD62>(x[e], x[e + d]);
        }
    };
    auto publish = [&]() {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; ++e) xb[e * T + t] = x[e];
        __syncthreads();
    };
#pragma unroll
    for (int k = 2; k <= E; k <<= 1) {
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (!(e & (k >> 1))) cmp_exchange<WORD62>(x[e], x[e ^ (k - 1)]);
        inner(k / 4);
    }
    // merges of 2, 4, .. 32 * G threads
#pragma unroll 1
    for (uint32_t k = 2; k <= T; k <<= 1) {
        const bool lower = (t & (k >> 1)) == 0;
        uint32_t j = k >> 2;
        bool in_xb = false;  // xb holds x
        if (FUSED && k >= 32 * E) {
            // thread bits low .. low + FB - 1; the mirrors' order is the reverse
            const int low = __ffs(k) - 1 - FB;  // at least 5
            const uint32_t e = (t >> 5) & (E - 1), rest = t >> (5 + FB);
            const uint32_t below = rest & ((1u << (low - 5)) - 1u);
            const uint32_t r = (t & 31u) | (below << 5) | ((rest >> (low - 5)) << (low + FB));
            uint64_t lo[E / 2], hi[E / 2];
            publish();
#pragma unroll
            for (uint32_t v = 0; v < E / 2; ++v) {
                const uint32_t p = r | (v << low);
                lo[v] = xb[e * T + p];
                hi[v] = xb[(E - 1 - e) * T + (p ^ (k - 1))];
                cmp_exchange<WORD62>(lo[v], hi[v]);
            }
#pragma unroll
            for (int d = E / 4; d > 0; d >>= 1) {
#pragma unroll
                for (int v = 0; v < E / 2; ++v)
                    if (!(v & d)) {
                        cmp_exchange<WORD62>(lo[v], lo[v + d]);
                        cmp_exchange<WORD62>(hi[v + d], hi[v]);
                    }
            }
#pragma unroll
            for (uint32_t v = 0; v < E / 2; ++v) {
                const uint32_t p = r | (v << low);
                xb[e * T + p] = lo[v];
                xb[(E - 1 - e) * T + (p ^ (k - 1))] = hi[v];
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < E; ++i) x[i] = xb[i * T + t];
            j = k >> (FB + 1);
            in_xb = true;
        } else if (G == 1 || k <= 32) {
#pragma unroll
            for (int e = 0; e < E / 2; ++e) {
                const uint64_t y0 = __shfl_xor_sync(0xFFFFFFFFu, x[E - 1 - e], k - 1);
                const uint64_t y1 = __shfl_xor_sync(0xFFFFFFFFu, x[e], k - 1);
                if (word_less<WORD62>(y0, x[e]) == lower) x[e] = y0;
                if (word_less<WORD62>(y1, x[E - 1 - e]) == lower) x[E - 1 - e] = y1;
            }
        } else {
            publish();
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t y = xb[(E - 1 - e) * T + (t ^ (k - 1))];
                if (word_less<WORD62>(y, x[e]) == lower) x[e] = y;
            }
        }
        if (G > 1) {
#pragma unroll 1
            for (; j >= 32; j >>= 1) {
                const bool low = (t & j) == 0;
                if (!in_xb) publish();
                in_xb = false;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const uint64_t y = xb[e * T + (t ^ j)];
                    if (word_less<WORD62>(y, x[e]) == low) x[e] = y;
                }
            }
        }
#pragma unroll 1
        for (; j > 0; j >>= 1) {
            const bool low = (t & j) == 0;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, x[e], j);
                if (word_less<WORD62>(y, x[e]) == low) x[e] = y;
            }
        }
        inner(E / 2);
    }
}

// The words of a segment (or tied group): 62 bits (word_less), IB index bits
// below the key's chars. x is the OR of its keys' differences from key0, not
// 0.
constexpr uint64_t WORD_PAD = ~0ull >> 2;  // after every word (no padding where index bits are all ones)
template <int IB, bool SFX>
struct WordForm {
    uint64_t key0;
    int cp;          // bits all keys share
    uint32_t chars;  // chars of the key in the word: all, or those the index leaves room for
    int low;         // bits below them
    __device__ __forceinline__ WordForm(const Work& w, uint64_t k0, uint64_t x) : key0(k0)
    {
        cp = __clzll((long long)x);
        if constexpr (SFX) {
            chars = cp >= IB + 2 ? w.kchars : (62u - IB) / w.kbits;
            low = cp >= IB + 2 ? 0 : 64 - (int)(chars * w.kbits);
        } else {
            chars = cp >= IB + 2 ? 8u : IB <= 6 ? 7u : 6u;
            low = 64 - 8 * (int)chars;
        }
        static_assert(IB <= 14, "6 chars of 8 bits leave 16 bits, 2 of them on top");
    }
    __device__ __forceinline__ uint64_t make(uint64_t key, uint32_t i) const
    {
        return (((key & (~0ull << low)) << cp) >> 2) | i;
    }
    // do two words hold the same chars?
    __device__ __forceinline__ static bool same(uint64_t a, uint64_t b) { return ((a ^ b) >> IB) == 0; }
    // chars shared by two words that differ
    __device__ __forceinline__ uint32_t lcp(uint64_t a, uint64_t b) const
    {
        return (uint32_t)(cp + __clzll((long long)(a ^ b)) - 2) >> 3;
    }
    __device__ __forceinline__ uint64_t key(uint64_t word) const
    {
        return (((word & (~0ull << IB)) << 2) >> cp) |
               (cp ? key0 & (~0ull << (64 - cp)) & (~0ull << low) : 0ull);
    }
    // do strings with this key (key()'s value) end inside the word's chars?
    __device__ __forceinline__ bool ended(uint64_t k) const { return !SFX && ((k >> low) & 0xFF) == 0; }
};

// Runs of tied strings (at most 32 each) into warp windows of up to 32
// strings. Each lane brings runs one after another: next(start, len) gives
// its next one or returns false. fn(owner, start, gs) runs on every lane of a
// window: the lane whose run the slot belongs to, the run's start and the
// slot its run starts at (32: an unused slot). scratch: 32 words of the warp.
template <typename Next, typename Fn>
__device__ __forceinline__ void tie_windows(uint32_t* scratch, Next next, Fn fn)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t start = 0, len = 0;
    bool has = next(start, len);
    while (__any_sync(0xFFFFFFFFu, has)) {
        const uint32_t end = warp_incl_sum(has ? len : 0u);
        const bool take = has && end <= 32u;
        const uint32_t at = end - len;
        const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, take ? 1u << at : 0u);
        const uint32_t used = __reduce_max_sync(0xFFFFFFFFu, take ? end : 0u);
        if (take) scratch[at] = lane;
        __syncwarp();
        const bool real = lane < used;
        const uint32_t gs = 31u - __clz(starts & (0xFFFFFFFFu >> (31 - lane)));
        const uint32_t owner = scratch[gs];
        __syncwarp();
        fn(owner, __shfl_sync(0xFFFFFFFFu, start, owner), real ? gs : 32u);
        if (take) has = next(start, len);
    }
}

// ---- 2..32 strings ----------------------------------------------------------
// A block takes up to TINY_THREADS list entries, orders them by network size so
// that the threads of a warp run the same one, and each warp stages the keys
// of its segments in shared memory (rows of 32 positions across segments,
// coalesced), sorts one segment per thread, and writes perm and LCPs in rows
// again. At most TINY_ROWS rows at a time: two halves of the warp in turn
// when its segments hold more.
//
// The network runs on 32-bit words, the 27 bits behind the bits all keys of
// the segment share over a 5-bit index: a compare-exchange is a min and a
// max, and the three networks are small enough to stay in the instruction
// cache (with 64-bit words they were not, and the registers halved the
// warps: 1.8 ms instead of 0.85 ms for the 28 M strings of this class in the
// 64 Mi prefix sort at 8 strings per bucket). Neighbours that tie in 27 bits
// are put in order by their whole keys in shared memory.
constexpr int TINY_THREADS = 256;
constexpr int TINY_ROWS = 16;
constexpr uint32_t TINY_LOAD = 1u << 31;  // TinyWarp::seg's meta: keys to load
// Times that a segment whose strings share a whole key moves to its next one
// before the network, instead of a warp window per segment (4 M strings, 20
// copies of each: 1127 -> 922 us, 910 before the leaf sorters; other sorts
// unchanged).
constexpr int TINY_TURNS = 4;

struct TinyWarp {
    uint64_t key[32 * TINY_ROWS];
    uint32_t lcp[32 * TINY_ROWS];
    uint8_t idx[32 * TINY_ROWS];
    uint4 seg[32];               // base, first row entry, meta, depth (then ties) per lane
    uint32_t starts[TINY_ROWS];  // per row: positions where a segment starts
    uint32_t scratch[32];
};

// The warp's segments, one per lane (sg.size 0: none; packed from lane
// `first` on), `total` strings from row entries `off`; N the network. Sorts
// and writes them.
// Segments of equal strings (META_FINAL, 17..32 of them from k_children) need no
// case of their own: their depth is the strings' length and no key is cached,
// so every key reads the NUL, 0, all tie, and the LCPs are the depth.
template <int N, bool SFX>
__device__ __forceinline__ void tiny_warp_sort(const Work& w, TinyWarp& sm, Seg sg, uint32_t first,
                                               uint32_t off, uint32_t total)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t base = sg.begin - off;  // row entry f of the segment: position base + f
    sm.seg[lane] = make_uint4(base, off, sg.meta | TINY_LOAD, sg.depth);
    if (lane < TINY_ROWS) sm.starts[lane] = 0;
    __syncwarp();
    if (sg.size) atomicOr(&sm.starts[off >> 5], 1u << (off & 31));
    __syncwarp();
    const uint32_t mask = lane < TINY_ROWS ? sm.starts[lane] : 0u;
    const uint32_t count = __popc(mask);
    const uint32_t before = first + warp_incl_sum(count) - count;  // segments before row `lane`
    // lane of the segment that row r's entry at this lane belongs to
    auto row_seg = [&](uint32_t r) {
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, mask, r & 15);
        const uint32_t b = __shfl_sync(0xFFFFFFFFu, before, r & 15);
        return (b + __popc(m & (0xFFFFFFFFu >> (31 - lane))) - 1) & 31;
    };
    constexpr uint32_t U = 4;  // rows in flight
    const uint64_t* key = sm.key + off;
    uint8_t* idx = sm.idx + off;
    uint32_t x[N];
    uint64_t diff;
    for (int turn = 0;; ++turn) {
        for (uint32_t r0 = 0; 32 * r0 < total; r0 += U) {
            uint64_t v[U];
            uint4 q[U];
            bool stale = false;
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t f = 32 * (r0 + u) + lane;
                q[u] = sm.seg[row_seg(r0 + u)];
                if (f >= total) q[u].z = 0;
                if (!(q[u].z & TINY_LOAD)) continue;
                const bool cached = q[u].z & META_VALID;
                v[u] = cached ? w.keys[q[u].z & META_BUF][q[u].x + f]
                              : handle_at_checked(w, q[u].z, q[u].x + q[u].y, q[u].x + f);
                stale = stale || !cached;
            }
            if (stale) {
#pragma unroll
                for (uint32_t u = 0; u < U; ++u)
                    if ((q[u].z & (TINY_LOAD | META_VALID)) == TINY_LOAD) v[u] = leaf_key<SFX>(w, v[u], q[u].w);
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u)
                if (q[u].z & TINY_LOAD) sm.key[32 * (r0 + u) + lane] = v[u];
        }
        __syncwarp();
        const uint64_t key0 = key[0];  // an unused lane reads an entry and drops it
        diff = 0;
#pragma unroll
        for (int i = 1; i < N; ++i)
            if ((uint32_t)i < sg.size) diff |= key[i] ^ key0;
        if constexpr (SFX) break;
        // one group that goes on: its next keys
        const bool deeper = sg.size > 1 && !diff && !key_terminated(key0);
        if (turn == TINY_TURNS || !__any_sync(0xFFFFFFFFu, deeper)) break;
        __syncwarp();
        if (deeper) {
            sg.depth += 8;
            sm.seg[lane] = make_uint4(base, off, (sg.meta & ~META_VALID) | TINY_LOAD, sg.depth);
        } else {
            sm.seg[lane].z = sg.meta;
        }
        __syncwarp();
    }
    const int cp = __clzll((long long)(diff | 1));  // equal keys: any shift does
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = 0xFFFFFFFFu;  // a real word is smaller, or has index 31 and no unused slot beside it
        if ((uint32_t)i < sg.size) x[i] = ((uint32_t)((key[i] << cp) >> 32) & ~31u) | i;
    }
    net_sort<N>(x);
    uint32_t near = 0;  // bit i: string i ties with string i - 1 in the word
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if ((uint32_t)i < sg.size) {
            idx[i] = (uint8_t)(x[i] & 31u);
            if (i) {
                const uint32_t df = (x[i] ^ x[i - 1]) >> 5;
                if (!df) near |= 1u << i;
                else if (w.lcp) sm.lcp[off + i] = sg.depth + ((uint32_t)(cp + __clz(df) - 5) >> 3);
            }
        }
    }
    uint32_t ties = 0;  // bit i: equal keys that do not end
    if (near) {
        for (uint32_t m = near; m; m &= m - 1) {  // insert the tied strings in order
            uint32_t i = __ffs(m) - 1;
            const uint8_t me = idx[i];
            const uint64_t k = key[me];
            while ((near >> i) & 1u) {
                const uint8_t o = idx[i - 1];
                if (key[o] <= k) break;
                idx[i--] = o;
            }
            idx[i] = me;
        }
        for (uint32_t m = near; m; m &= m - 1) {
            const uint32_t i = __ffs(m) - 1;
            const uint64_t a = key[idx[i - 1]], b = key[idx[i]];
            if (a == b && (SFX || !key_terminated(b))) ties |= 1u << i;
            else if (w.lcp) sm.lcp[off + i] = sg.depth + (a != b ? lcp_key_type(a, b) : lcp_key_depth(b));
        }
    }
    sm.seg[lane].w = ties;
    __syncwarp();
    for (uint32_t r0 = 0; 32 * r0 < total; r0 += U) {
        uint64_t h[U];
        uint4 q[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t f = 32 * (r0 + u) + lane;
            q[u] = sm.seg[row_seg(r0 + u)];
            if (f < total) h[u] = handle_at(w, q[u].z, q[u].x + q[u].y, q[u].x + q[u].y + sm.idx[f]);
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t f = 32 * (r0 + u) + lane;
            if (f >= total) continue;
            w.perm[q[u].x + f] = h_id(w, h[u]);
            const uint32_t i = f - q[u].y;
            if (w.lcp && i && !((q[u].w >> i) & 1u)) w.lcp[q[u].x + f] = sm.lcp[f];
        }
    }
    if (!__any_sync(0xFFFFFFFFu, ties)) return;
    __syncwarp();
    auto next_run = [&](uint32_t& start, uint32_t& len) {
        if (!ties) return false;
        const uint32_t i = __ffs(ties) - 1;  // >= 1
        const uint32_t rest = ~(ties >> i);
        const uint32_t ones = __ffs(rest) - 1;  // at most 31: bit 0 is never set
        start = i - 1;
        len = ones + 1;
        ties &= i + ones >= 32 ? 0u : ~0u << (i + ones);
        return true;
    };
    if constexpr (SFX) {
        uint32_t start = 0, len = 0;
        bool has = next_run(start, len);
        while (__any_sync(0xFFFFFFFFu, has)) {
            push_dbl_warp(w, has, Seg{sg.begin + start, len, sg.depth + w.kchars, META_PERM});
            has = has && next_run(start, len);
        }
        return;
    }
    tie_windows(
        sm.scratch, next_run,
        [&](uint32_t owner, uint32_t start, uint32_t gs) {
            const bool real = gs < 32;
            const uint32_t o = __shfl_sync(0xFFFFFFFFu, off, owner);
            const uint32_t bo = __shfl_sync(0xFFFFFFFFu, base, owner);
            const uint32_t meta = __shfl_sync(0xFFFFFFFFu, sg.meta, owner);
            const uint32_t dep = __shfl_sync(0xFFFFFFFFu, sg.depth + 8, owner);
            const uint32_t f = o + start + (lane - gs);
            const uint32_t pos = bo + f;
            const uint64_t h = real ? handle_at(w, meta, bo + o, bo + o + sm.idx[f]) : ~0ull;
            const uint64_t r = warp_window(w, h, gs, dep, pos, false, 0ull, sm.scratch);
            if (real) w.perm[pos] = h_id(w, r);
        });
}

template <bool SFX>
__global__ void __launch_bounds__(TINY_THREADS, 3) k_tiny(Work w, const Seg* list, uint32_t count, uint32_t per)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TinyWarp* warps = reinterpret_cast<TinyWarp*>(smem_raw);
    __shared__ Seg segs[TINY_THREADS];
    __shared__ uint32_t cnt[3 * TINY_THREADS / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t here = per * (TINY_THREADS / 32);  // entries of this block
    const uint32_t g = threadIdx.x < here ? blockIdx.x * here + threadIdx.x : count;
    Seg sg{};
    if (g < count) sg = list[g];
    // stable order by network: 9..16 strings behind those up to 8, and so on;
    // unused threads last
    const uint32_t cls = g >= count ? 3 : sg.size <= 8 ? 0 : sg.size <= 16 ? 1 : 2;
    uint32_t below = 0;  // entries of this class in earlier lanes
#pragma unroll
    for (uint32_t c = 0; c < 3; ++c) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, cls == c);
        if (lane == 0) cnt[c * (TINY_THREADS / 32) + warp] = __popc(m);
        if (cls == c) below = __popc(m & ((1u << lane) - 1u));
    }
    segs[threadIdx.x] = Seg{};
    __syncthreads();
    static_assert(3 * TINY_THREADS / 32 <= 32, "one lane per class and warp");
    const uint32_t mine = lane < 3 * TINY_THREADS / 32 ? cnt[lane] : 0u;
    const uint32_t ahead = warp_incl_sum(mine) - mine;
    const uint32_t at = __shfl_sync(0xFFFFFFFFu, ahead, (cls * (TINY_THREADS / 32) + warp) & 31) + below;
    if (cls < 3) segs[at] = sg;
    __syncthreads();
    sg = lane < per ? segs[warp * per + lane] : Seg{};
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, sg.size);
    if (most == 0) return;  // whole warp
    const uint32_t all = __reduce_add_sync(0xFFFFFFFFu, sg.size);
    const uint32_t turns = all <= 32 * TINY_ROWS ? 1 : 2;
    for (uint32_t t = 0; t < turns; ++t) {
        Seg part = sg;
        if (turns == 2 && (lane >> 4) != t) part.size = 0;
        const uint32_t end = warp_incl_sum(part.size);
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, end, 31);
        if (!total) continue;
        const uint32_t off = part.size ? end - part.size : 0u;
        if (most <= 8) tiny_warp_sort<8, SFX>(w, warps[warp], part, 16 * t, off, total);
        else if (most <= 16) tiny_warp_sort<16, SFX>(w, warps[warp], part, 16 * t, off, total);
        else tiny_warp_sort<32, SFX>(w, warps[warp], part, 16 * t, off, total);
        __syncwarp();
    }
}

// Entries per warp: fewer than 32 when that leaves SMs idle (a warp takes its
// entries' loads and ties one after another).
inline uint32_t tiny_per(uint32_t count)
{
    uint32_t per = 32;
    while (per > 4 && count < per * (TINY_THREADS / 32) * 296u) per >>= 1;
    return per;
}
constexpr size_t TINY_SMEM = sizeof(TinyWarp) * (TINY_THREADS / 32);

// ---- 33..SMALL_MAX strings ------------------------------------------------------
// G warps per segment of at most 256 G strings. hnd holds the segment's
// handles as they came, idx the current order of positions; groups are sorted
// from a stack (the segment first, then tied groups of more than 32 strings).
constexpr int SEG_E = 8;  // most words a thread holds
template <int G>
struct alignas(16) SegState {
    static constexpr int N = 32 * SEG_E * G;
    static constexpr int IDX = N + N / 16;  // padded (idx_at)
    static constexpr int LCP = N + N / 32;  // padded (lcp_at)
    // G > 1: the sort's exchange buffer and the LCP staging share one array
    static constexpr int TAIL = G > 1 ? 8 * N : 4 * LCP;
    uint64_t hnd[N];
    uint64_t last[G], key0, diff;
    uint16_t idx[IDX];
    uint16_t tpos[N], trun[N];  // tied strings of a group: position and run number
    uint32_t tied[N / 32];    // bit i: the string at i ties with the one before
    uint32_t wsum[G];
    uint32_t scratch[G][32];
    uint16_t g_start[N / 32], g_len[N / 32];
    uint32_t g_dep[N / 32];
    uint32_t ng, jump, ntied;
};

// dynamic shared memory of a block that sorts `segs` segments at a time
template <int G>
constexpr size_t segs_smem(int segs, bool lcp)
{
    return (size_t)segs * (sizeof(SegState<G>) + (G > 1 || lcp ? SegState<G>::TAIL : 0));
}

// padded positions: a thread's consecutive entries start on another bank than
// its neighbours'
__device__ __forceinline__ uint32_t idx_at(uint32_t i) { return i + ((i >> 5) << 1); }
__device__ __forceinline__ uint32_t lcp_at(uint32_t i) { return i + (i >> 5); }

// Ties per warp beyond which all tied runs of a group are sorted together
// (sort_runs), up to LEAF_RESORTS times in a row: 200 k ACGT strings (3 per
// 8-char key) 186 -> 95 us, 2 M of them with LCPs 0.56 -> 0.52 ms, against warp
// windows and another pass alone.
constexpr uint32_t LEAF_RESORT_TIES = 24;
constexpr int LEAF_RESORTS = 2;
// Ties per warp beyond which a group hands its tied runs to the next pass
// instead of sorting them in warp windows, or (runs over 32 strings) by all
// its warps, one after another. Runs over LEAF_WINDOW_TIES * G stay: the
// group's warps are not too many for them.
constexpr uint32_t LEAF_WINDOW_TIES = 48;
// equal_runs in a row, where sort_runs finds that the runs share more chars. Runs
// of more than 32 strings on average (a long prefix of many strings) go on as
// they are: the jump of the pass that gets them costs less (4 Mi prefix strings
// with LCPs: 880 us, 916 with every run compared).
constexpr int LEAF_EQUAL_TURNS = 2;
constexpr uint32_t LEAF_TIED = 0xFFFFFFFFu;  // LCP staging: not known yet

// Bits that hold an index below n (a power of two).
__host__ __device__ constexpr int word_index_bits(int n)
{
    int b = 0;
    while ((1 << b) < n) ++b;
    return b;
}

// Sum over the group of the ties each thread found (G > 1: sm.ntied is 0
// before). Synchronises.
template <int G>
__device__ __forceinline__ uint32_t count_ties(SegState<G>& sm, uint32_t tied)
{
    uint32_t nt = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)__popc(tied));
    if constexpr (G > 1) {
        if ((threadIdx.x & 31) == 0 && nt) atomicAdd(&sm.ntied, nt);
        __syncthreads();
        nt = sm.ntied;
    } else {
        __syncwarp();
    }
    return nt;
}

// Sort the group of c strings (c <= 32 E G) at offset s of the segment, depth
// d; with the segment's cached keys when `cached` (then s is 0). Writes perm
// and the LCPs it finds. Returns how many strings tie with their predecessor
// (marked in sm.tied; *chars deeper than d); a group whose keys are all equal
// goes back to the stack behind its common prefix.
template <int E, int G, bool SFX>
__device__ __forceinline__ uint32_t sort_group(const Work& w, SegState<G>& sm, unsigned char* tail, uint32_t begin,
                                               int buf, uint32_t s, uint32_t c, uint32_t d, bool cached,
                                               uint32_t* chars)
{
    constexpr uint32_t T = 32 * G;
    constexpr int IB = word_index_bits(32 * E * G);
    const uint32_t lane = threadIdx.x & 31, warp = G == 1 ? 0u : threadIdx.x >> 5;
    const uint32_t t = 32 * warp + lane;
    uint32_t* slcp = reinterpret_cast<uint32_t*>(tail);
    uint64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = t + T * e;
        x[e] = 0;
        if (j < c)
            x[e] = cached ? __ldcg(w.keys[buf] + begin + j) : leaf_key<SFX>(w, sm.hnd[sm.idx[idx_at(s + j)]], d);
    }
    uint64_t key0 = __shfl_sync(0xFFFFFFFFu, x[0], 0);
    if constexpr (G > 1) {
        if (t == 0) {
            sm.key0 = key0;
            sm.diff = 0;
            sm.ntied = 0;
        }
        __syncthreads();
        key0 = sm.key0;
    }
    uint64_t diff = 0;
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (t + T * e < c) diff |= x[e] ^ key0;
    diff = ((uint64_t)__reduce_or_sync(0xFFFFFFFFu, (uint32_t)(diff >> 32)) << 32) |
           __reduce_or_sync(0xFFFFFFFFu, (uint32_t)diff);
    if constexpr (G > 1) {
        if (lane == 0 && diff) atomicOr((unsigned long long*)&sm.diff, (unsigned long long)diff);
        __syncthreads();
        diff = sm.diff;
    }
    if (diff == 0) {
        if constexpr (SFX) {
            for (uint32_t j = t; j < c; j += T) w.perm[begin + s + j] = h_id(w, sm.hnd[sm.idx[idx_at(s + j)]]);
            if (t == 0) push_dbl(w, Seg{begin + s, c, d + w.kchars, META_PERM});
            return 0;
        }
        if (key_terminated(key0)) {  // all equal: any order
            for (uint32_t j = t; j < c; j += T) {
                w.perm[begin + s + j] = h_id(w, sm.hnd[sm.idx[idx_at(s + j)]]);
                if (w.lcp && j) w.lcp[begin + s + j] = d + lcp_key_depth(key0);
            }
            return 0;
        }
        // one tied group: its common prefix in chunks of 8 chars (at least 1)
        if (t == 0) sm.jump = 0xFFFFFFFFu;
        group_sync<G>();
        const uint64_t first = sm.hnd[sm.idx[idx_at(s)]];
        for (uint32_t j = 1 + t; j < c; j += T)
            atomicMin(&sm.jump, chunks_equal(w, first, sm.hnd[sm.idx[idx_at(s + j)]], d, &sm.jump));
        group_sync<G>();
        if (t == 0) {
            const uint32_t at = sm.ng++;
            sm.g_start[at] = (uint16_t)s;
            sm.g_len[at] = (uint16_t)c;
            sm.g_dep[at] = d + 8u * sm.jump;
        }
        return 0;
    }
    const WordForm<IB, SFX> form(w, key0, diff);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = t + T * e;
        x[e] = j < c ? form.make(x[e], j) : WORD_PAD;
    }
    group_sort<E, G, true>(x, reinterpret_cast<uint64_t*>(tail));
    // LCPs and ties, from each word and the one before
    uint64_t up = __shfl_up_sync(0xFFFFFFFFu, x[E - 1], 1);
    if constexpr (G > 1) {
        if (lane == 31) sm.last[warp] = x[E - 1];
        __syncthreads();  // and the exchange buffer is free
        if (lane == 0 && warp) up = sm.last[warp - 1];
    }
    uint32_t tied = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = t * E + e;
        const uint64_t prev = e ? x[e > 0 ? e - 1 : 0] : up;
        if (i == 0 || i >= c) continue;
        uint32_t l = LEAF_TIED;
        if (!WordForm<IB, SFX>::same(prev, x[e])) {
            l = d + form.lcp(prev, x[e]);
        } else {
            const uint64_t k = form.key(x[e]);
            if (form.ended(k)) l = d + lcp_key_depth(k);
            else tied |= 1u << e;
        }
        if (w.lcp) slcp[lcp_at(i)] = l;
    }
    // the order, in terms of the handles as they came
    uint16_t o[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = (uint32_t)x[e] & ((1u << IB) - 1);
        o[e] = t * E + e < c ? sm.idx[idx_at(s + j)] : (uint16_t)0;
    }
    const uint32_t nt = count_ties<G>(sm, tied);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (t * E + e < c) sm.idx[idx_at(s + t * E + e)] = o[e];
    if (nt && t < E * G) sm.tied[t] = 0;
    group_sync<G>();
    if (tied) atomicOr(&sm.tied[(t * E) >> 5], tied << ((t * E) & 31));
#pragma unroll 4
    for (uint32_t j = t; j < c; j += T) {
        w.perm[begin + s + j] = h_id(w, sm.hnd[sm.idx[idx_at(s + j)]]);
        if (w.lcp && j) {
            const uint32_t l = slcp[lcp_at(j)];
            if (l != LEAF_TIED) w.lcp[begin + s + j] = l;
        }
    }
    *chars = form.chars;
    group_sync<G>();
    return nt;
}

// The tied strings of a group of c strings (their runs marked in sm.tied) into
// sm.tpos / sm.trun in order of their positions; returns how many, *runs the
// number of runs. A thread takes 8 positions.
template <int G>
__device__ __forceinline__ uint32_t collect_ties(SegState<G>& sm, uint32_t c, uint32_t* runs)
{
    const uint32_t lane = threadIdx.x & 31, warp = G == 1 ? 0u : threadIdx.x >> 5;
    const uint32_t p0 = 8 * (32 * warp + lane);
    const uint32_t words = (c + 31) / 32;
    uint32_t at = 0;  // ties of positions p0 .. p0 + 8
    if (p0 < c) {
        const uint32_t lo = sm.tied[p0 >> 5], hi = (p0 >> 5) + 1 < words ? sm.tied[(p0 >> 5) + 1] : 0u;
        at = __funnelshift_r(lo, hi, p0 & 31) & 0x1FFu;
    }
    const uint32_t member = (at | (at >> 1)) & 0xFFu, starts = (at >> 1) & ~at & 0xFFu;
    const uint32_t mine = __popc(member) | (__popc(starts) << 16);
    const uint32_t incl = warp_incl_sum(mine);
    uint32_t before = incl - mine, total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    if constexpr (G > 1) {
        if (lane == 31) sm.wsum[warp] = incl;
        __syncthreads();
        total = 0;
        for (int v = 0; v < G; ++v) {
            if (v < (int)warp) before += sm.wsum[v];
            total += sm.wsum[v];
        }
    }
    uint32_t j = before & 0xFFFFu, r = before >> 16;  // runs started before p0
    for (uint32_t m = member; m; m &= m - 1) {
        const uint32_t q = __ffs(m) - 1;
        r += (starts >> q) & 1u;
        sm.tpos[j] = (uint16_t)(p0 + q);
        sm.trun[j++] = (uint16_t)(r - 1);
    }
    *runs = total >> 16;
    group_sync<G>();
    return total & 0xFFFFu;
}

// Sort the runs of n tied strings (collect_ties; n <= 32 E G) of the group at
// offset s, all at once, by the chars at depth d: a word is (run, chars,
// index), as many chars as fit (4 to 6). Writes perm, the LCPs it finds and
// the new sm.tied; returns how many strings still tie (*chars deeper). Where
// most neighbours in the runs share these chars too (a long common prefix),
// nothing is done: *chars is 0.
template <int E, int G>
__device__ __forceinline__ uint32_t sort_runs(const Work& w, SegState<G>& sm, unsigned char* tail, uint32_t begin,
                                              uint32_t s, uint32_t c, uint32_t n, uint32_t runs, uint32_t ties,
                                              uint32_t d, uint32_t* chars)
{
    constexpr uint32_t T = 32 * G;
    constexpr int IB = word_index_bits(32 * E * G);
    const uint32_t lane = threadIdx.x & 31, warp = G == 1 ? 0u : threadIdx.x >> 5;
    const uint32_t t = 32 * warp + lane;
    const int rb = 32 - __clz((int)runs);  // run numbers are below 2^rb
    const int kc = (62 - IB - rb) / 8;
    const int ksh = 62 - rb - 8 * kc;      // the chars' lowest bit
    uint64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t j = t + T * e;
        x[e] = WORD_PAD;
        if (j < n) {
            const uint64_t k = leaf_key<false>(w, sm.hnd[sm.idx[idx_at(s + sm.tpos[j])]], d);
            x[e] = ((uint64_t)sm.trun[j] << (62 - rb)) | ((k >> (64 - 8 * kc)) << ksh) | j;
        }
    }
    uint32_t pairs = 0;  // neighbours of one run, and (<< 16) those equal
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint64_t df = x[e] ^ __shfl_up_sync(0xFFFFFFFFu, x[e], 1);
        if (lane && t + T * e < n && !(df >> (62 - rb))) pairs += df >> ksh ? 1u : 0x10001u;
    }
    pairs = __reduce_add_sync(0xFFFFFFFFu, pairs);
    if constexpr (G > 1) {
        if (lane == 0) sm.wsum[warp] = pairs;
        if (t == 0) sm.ntied = 0;
        __syncthreads();
        pairs = 0;
        for (int v = 0; v < G; ++v) pairs += sm.wsum[v];
    }
    *chars = 0;
    if ((pairs >> 16) * 2 > (pairs & 0xFFFFu)) return ties;
    group_sort<E, G, true>(x, reinterpret_cast<uint64_t*>(tail));
    uint64_t up = __shfl_up_sync(0xFFFFFFFFu, x[E - 1], 1);
    if constexpr (G > 1) {
        if (lane == 31) sm.last[warp] = x[E - 1];
        __syncthreads();
        if (lane == 0 && warp) up = sm.last[warp - 1];
    }
    uint32_t tied = 0;
    uint16_t o[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = t * E + e;
        const uint64_t prev = e ? x[e > 0 ? e - 1 : 0] : up;
        o[e] = 0;
        if (i >= n) continue;
        o[e] = sm.idx[idx_at(s + sm.tpos[(uint32_t)x[e] & ((1u << IB) - 1)])];
        if (i == 0) continue;
        const uint64_t df = x[e] ^ prev;
        if (df >> (62 - rb)) continue;  // another run
        uint32_t l;
        if (df >> ksh) {
            l = (uint32_t)(__clzll((long long)df) - 2 - rb) >> 3;
        } else {
            const uint64_t k = (x[e] >> ksh) << (64 - 8 * kc);  // the chars, left-aligned (run bits shifted out)
            if ((k >> (64 - 8 * kc)) & 0xFF) {
                tied |= 1u << e;
                continue;
            }
            l = lcp_key_depth(k);
        }
        if (w.lcp) w.lcp[begin + s + sm.tpos[i]] = d + l;
    }
    const uint32_t nt = count_ties<G>(sm, tied);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (t * E + e < n) {
            const uint32_t p = s + sm.tpos[t * E + e];
            sm.idx[idx_at(p)] = o[e];
            w.perm[begin + p] = h_id(w, sm.hnd[o[e]]);
        }
    for (uint32_t v = t; v < (c + 31) / 32; v += T) sm.tied[v] = 0;
    group_sync<G>();
#pragma unroll
    for (int e = 0; e < E; ++e)
        if ((tied >> e) & 1u) {
            const uint32_t p = sm.tpos[t * E + e];
            atomicOr(&sm.tied[p >> 5], 1u << (p & 31));
        }
    *chars = kc;
    group_sync<G>();
    return nt;
}

// How the strings behind handles a and b compare in the 32 chars from depth d:
// EQ_APART they differ, EQ_OPEN they share all of them, else they are equal and
// this is their length.
constexpr uint32_t EQ_APART = 0xFFFFFFFFu, EQ_OPEN = 0xFFFFFFFEu;
__device__ __forceinline__ uint32_t equal_in_32(const Work& w, uint64_t a, uint64_t b, uint32_t d)
{
    uint64_t ra[4], rb[4];
    load_raw_chunks<4>(w.chars, w.nchars, h_off(w, a) + d, 4, ra);
    load_raw_chunks<4>(w.chars, w.nchars, h_off(w, b) + d, 4, rb);
    uint32_t r = EQ_OPEN;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        const uint64_t ka = finish_key(ra[q]), kb = finish_key(rb[q]);
        if (r != EQ_OPEN) continue;
        if (ka != kb) r = EQ_APART;
        else if (key_terminated(ka)) r = d + 8 * q + lcp_key_depth(ka);
    }
    return r;
}

// The runs of n tied strings (collect_ties) of the group at offset s, when no
// two strings of one differ in the 32 chars from depth d: those that end there
// are done (LCPs written, their ties cleared). Returns whether that is so; *nt
// is how many strings still tie, 32 chars deeper. Copies of the same string
// end here instead of in the next pass (4 M strings, 5 copies of each: 1213 ->
// 757 us; of 60 chars, 20 copies: 1950 -> 907; prefixes 0 to 7% faster, random
// strings unchanged). 8 chars at a time cost the prefixes 3% at 0.5 M strings.
template <int G>
__device__ __forceinline__ bool equal_runs(const Work& w, SegState<G>& sm, uint32_t begin, uint32_t s, uint32_t n,
                                           uint32_t d, uint32_t* nt)
{
    constexpr uint32_t T = 32 * G;
    const uint32_t t = G == 1 ? threadIdx.x & 31 : threadIdx.x;
    auto handle = [&](uint32_t j) { return sm.hnd[sm.idx[idx_at(s + sm.tpos[j])]]; };
    bool apart = false;
    uint32_t done = 0, open = 0;  // bit e: of the pair t + e T, t + e T + 1
#pragma unroll 1
    for (int e = 0; e < SEG_E; ++e) {
        const uint32_t j = t + T * e + 1;
        if (j >= n || sm.trun[j] != sm.trun[j - 1]) continue;
        const uint32_t l = equal_in_32(w, handle(j - 1), handle(j), d);
        apart = apart || l == EQ_APART;
        if (l == EQ_OPEN) open |= 1u << e;
        if (l >= EQ_OPEN) continue;
        done |= 1u << e;
        if (w.lcp) w.lcp[begin + s + sm.tpos[j]] = l;  // written again when the run goes on
    }
    if constexpr (G == 1) apart = __any_sync(0xFFFFFFFFu, apart);
    else apart = __syncthreads_or(apart);
    if (apart) return false;
    if constexpr (G > 1) {
        if (t == 0) sm.ntied = 0;
        __syncthreads();
    }
    for (uint32_t m = done; m; m &= m - 1) {
        const uint32_t p = sm.tpos[t + T * (__ffs(m) - 1) + 1];
        atomicAnd(&sm.tied[p >> 5], ~(1u << (p & 31)));
    }
    *nt = count_ties<G>(sm, open);
    if constexpr (G > 1) __syncthreads();
    return true;
}

// The nt ties left in the group of c strings at offset s, whose runs share
// `dep` chars: to the list dbl (a suffix set), to the next pass when there are
// many, else runs of up to 32 strings to warp windows and longer ones to the
// stack.
template <int G, bool SFX>
__device__ __forceinline__ void finish_ties(const Work& w, SegState<G>& sm, uint32_t begin, int buf, uint32_t s,
                                            uint32_t c, uint32_t dep, uint32_t nt)
{
    constexpr uint32_t T = 32 * G;
    const uint32_t lane = threadIdx.x & 31, warp = G == 1 ? 0u : threadIdx.x >> 5;
    const uint32_t t = 32 * warp + lane;
    // lane l of a warp takes the runs that start in positions
    // [32 v, 32 v + 32), v = l G + warp
    const uint32_t words = (c + 31) / 32;
    const uint32_t v = lane * G + warp;
    uint32_t starts = 0;
    if (v < words) {
        const uint32_t m = sm.tied[v], nx = v + 1 < words ? sm.tied[v + 1] : 0u;
        starts = ((m >> 1) | (nx << 31)) & ~m;
    }
    // runs over `most` strings stay with this group's warps
    const bool pass_on = nt > LEAF_WINDOW_TIES * G;
    const uint32_t most = SFX ? c : pass_on ? LEAF_WINDOW_TIES * G : (uint32_t)WARP_GROUP_MAX;
    auto next_run = [&](uint32_t& start, uint32_t& len) {
        while (starts) {
            start = 32 * v + __ffs(starts) - 1;
            starts &= starts - 1;
            len = 1;
            for (uint32_t q = start + 1; q < c;) {  // ones from q on
                const uint32_t rest = ~(sm.tied[q >> 5] >> (q & 31));
                const uint32_t room = 32 - (q & 31);
                const uint32_t ones = rest ? min((uint32_t)(__ffs(rest) - 1), room) : 32u;
                len += ones;
                if (ones < room) break;
                q += ones;
            }
            if (len <= most) return true;
            const uint32_t at = atomicAdd(&sm.ng, 1u);
            sm.g_start[at] = (uint16_t)(s + start);
            sm.g_len[at] = (uint16_t)len;
            sm.g_dep[at] = dep;
        }
        return false;
    };
    if constexpr (SFX) {
        uint32_t start = 0, len = 0;
        bool has = next_run(start, len);
        while (__any_sync(0xFFFFFFFFu, has)) {
            push_dbl_warp(w, has, Seg{begin + s + start, len, dep, META_PERM});
            has = has && next_run(start, len);
        }
        return;
    }
    if (pass_on) {
        // the next pass sorts the runs as segments of their own size, from the
        // segment's handles in the order reached here
        for (uint32_t j = t; j < c; j += T) w.hnd[buf][begin + s + j] = sm.hnd[sm.idx[idx_at(s + j)]];
        uint32_t start = 0, len = 0;
        bool has = next_run(start, len);
        while (__any_sync(0xFFFFFFFFu, has)) {
            push_seg_warp(w, w.cur ^ 1, has, Seg{begin + s + start, len, dep, (uint32_t)buf});
            has = has && next_run(start, len);
        }
        return;
    }
    uint64_t* const defer = w.deep[w.cur ^ 1] ? w.hnd[buf] : nullptr;
    tie_windows(sm.scratch[warp], next_run, [&](uint32_t, uint32_t start, uint32_t gs) {
        const bool real = gs < 32;
        const uint32_t q = s + start + (lane - gs);
        const uint64_t h = real ? sm.hnd[sm.idx[idx_at(q)]] : ~0ull;
        const uint64_t r = warp_window(w, h, gs, dep, begin + q, false, 0ull, sm.scratch[warp], defer, (uint32_t)buf);
        if (real) w.perm[begin + q] = h_id(w, r);
    });
}

// Sort the segment of m strings at position begin by its group of G warps:
// handles in sm.hnd (idx: 0..m-1), buf the buffer they came from, depth the
// chars they share, cached whether keys[buf] holds their keys.
template <int G, bool SFX>
__device__ __forceinline__ void sort_segment(const Work& w, SegState<G>& sm, unsigned char* tail, uint32_t begin,
                                             uint32_t m, int buf, uint32_t depth, bool cached)
{
    const uint32_t t = threadIdx.x % (32 * G);
    if (t == 0) {
        sm.ng = 1;
        sm.g_start[0] = 0;
        sm.g_len[0] = (uint16_t)m;
        sm.g_dep[0] = depth;
    }
    group_sync<G>();
    while (true) {
        const uint32_t n = sm.ng;
        if (n == 0) break;
        const uint32_t s = sm.g_start[n - 1], c = sm.g_len[n - 1], d = sm.g_dep[n - 1];
        group_sync<G>();
        if (t == 0) sm.ng = n - 1;
        group_sync<G>();
        uint32_t chars = 0;
        uint32_t nt = c <= 64 * G    ? sort_group<2, G, SFX>(w, sm, tail, begin, buf, s, c, d, cached, &chars)
                      : c <= 128 * G ? sort_group<4, G, SFX>(w, sm, tail, begin, buf, s, c, d, cached, &chars)
                                     : sort_group<8, G, SFX>(w, sm, tail, begin, buf, s, c, d, cached, &chars);
        uint32_t dep = d + chars;
        for (int r = 0; !SFX && r < LEAF_RESORTS && nt > LEAF_RESORT_TIES * G; ++r) {
            uint32_t runs = 0;
            const uint32_t k = collect_ties<G>(sm, c, &runs);
            nt = k <= 64 * G    ? sort_runs<2, G>(w, sm, tail, begin, s, c, k, runs, nt, dep, &chars)
                 : k <= 128 * G ? sort_runs<4, G>(w, sm, tail, begin, s, c, k, runs, nt, dep, &chars)
                                : sort_runs<8, G>(w, sm, tail, begin, s, c, k, runs, nt, dep, &chars);
            if (!chars) {
                uint32_t k2 = k;
                const bool copies = k <= runs * (uint32_t)WARP_GROUP_MAX;
                for (int q = 0; copies && q < LEAF_EQUAL_TURNS && nt; ++q) {
                    if (!equal_runs<G>(w, sm, begin, s, k2, dep, &nt)) break;
                    dep += 32;
                    if (nt) k2 = collect_ties<G>(sm, c, &runs);
                }
                break;
            }
            dep += chars;
        }
        if (nt) finish_ties<G, SFX>(w, sm, begin, buf, s, c, dep, nt);
        cached = false;
        group_sync<G>();
    }
}

// SEGS segments per block for G == 1, one for G > 1.
template <int G, int SEGS, int BLOCKS, bool SFX>
__global__ void __launch_bounds__(32 * G * SEGS, BLOCKS) k_segs(Work w, const Seg* list, uint32_t count)
{
    static_assert(G == 1 || SEGS == 1, "a block's barriers serve one segment");
    constexpr uint32_t T = 32 * G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t t = threadIdx.x % T, sub = threadIdx.x / T;
    SegState<G>& sm = reinterpret_cast<SegState<G>*>(smem_raw)[sub];
    // behind the states: exchange buffer and LCP staging (G == 1: sorts with LCP output only)
    unsigned char* tail = smem_raw + SEGS * sizeof(SegState<G>) + sub * (size_t)SegState<G>::TAIL;
    const uint32_t g = blockIdx.x * SEGS + sub;
    if (g >= count) return;  // whole group
    const Seg sg = list[g];
    const uint32_t m = sg.size, begin = sg.begin;
    const int buf = sg.meta & META_BUF;
    if (sg.meta & META_FINAL) {
        for (uint32_t i = t; i < m; i += T) {
            w.perm[begin + i] = h_id(w, handle_at(w, sg.meta, begin, begin + i));
            if (w.lcp && i) w.lcp[begin + i] = sg.depth;
        }
        return;
    }
    const uint64_t* src = handle_src(w, sg.meta) + begin;
#pragma unroll 8
    for (uint32_t i = t; i < m; i += T) {
        sm.hnd[i] = __ldg(src + i);
        sm.idx[idx_at(i)] = (uint16_t)i;
    }
    if (sg.meta & META_ROOT) {  // the offsets become handles (short code beside the loads' loop)
        bool bad = false;
#pragma unroll 1
        for (uint32_t i = t; i < m; i += T) {
            const uint64_t x = sm.hnd[i];
            bad |= x >= w.nchars;
            sm.hnd[i] = h_make(w, w.local ? i : begin + i, x);
        }
        if (bad) set_error(w.counters + C_ERR, ERR_OFFSET);
    }
    sort_segment<G, SFX>(w, sm, tail, begin, m, buf, sg.depth, sg.meta & META_VALID);
}

// The whole sort of an input of at most 256 G strings, by one block: handles
// from the offsets, the input checks, and the counters, which go to the
// host's copy at the end (mapped memory: no memset before and no copy after
// the kernel). w.cur is 0: what is left over goes to the lists of parity 1,
// in buffer 0.
template <int G>
__global__ void __launch_bounds__(32 * G) k_one(Work w, uint32_t* host_counters)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SegState<G>& sm = *reinterpret_cast<SegState<G>*>(smem_raw);
    constexpr uint32_t T = 32 * G;
    const uint32_t t = threadIdx.x;
    for (uint32_t k = t; k < (uint32_t)C_COUNT; k += T) w.counters[k] = 0;
    uint32_t err = t == 0 && w.chars[w.nchars - 1] != 0 ? ERR_UNTERMINATED : 0u;
#pragma unroll 8
    for (uint32_t i = t; i < w.n; i += T) {
        const uint64_t off = __ldg(w.offs + i);
        if (off >= w.nchars) err |= ERR_OFFSET;
        sm.hnd[i] = h_make(w, i, off);
        sm.idx[idx_at(i)] = (uint16_t)i;
    }
    if (t == 0) sm.ntied = 0;
    __syncthreads();
    if (err) {
        set_error(w.counters + C_ERR, err);
        sm.ntied = 1;
    }
    __syncthreads();
    if (!sm.ntied) sort_segment<G, false>(w, sm, smem_raw + sizeof(SegState<G>), 0, w.n, 0, 0, false);
    __syncthreads();
    for (uint32_t k = t; k < (uint32_t)C_COUNT; k += T) host_counters[k] = __ldcg(w.counters + k);
}

constexpr int SEGS_A_WARPS = 8;
template <bool SFX>
constexpr auto k_segs_a = k_segs<1, SEGS_A_WARPS, 3, SFX>;
template <bool SFX>
constexpr auto k_segs_b = k_segs<4, 1, 6, SFX>;
template <bool SFX>
constexpr auto k_segs_c = k_segs<16, 1, 2, SFX>;

}  // namespace pssgpu
