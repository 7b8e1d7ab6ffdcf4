// kernels_wave.cuh -- the whole sort of an input that fits one wave of
// resident blocks, in one cooperative launch (no host round trip between
// the steps, no kernel boundaries).
//
// pS5 runs an input of this size as one sample-sort step over all strings
// followed by a SmallsortJob per bucket on its job queue
// (src/parallel/bingmann-parallel_sample_sort.hpp:1613-1634, 1264-1611,
// 405-676). Here the same steps are phases of one kernel, separated by grid
// barriers (all blocks are co-resident by the cooperative launch):
//   A  every block gathers the first 8 chars (get_char_uint64_simple) of its
//      tile of strings into registers, draws the same `over` * 2^L samples, sorts
//      them and builds the level-order tree (SampleSortStep::sample,
//      TreeBuilderLevelOrder)
//   B  classifies its tile (find_bkt), counts per bucket in shared memory,
//      reserves the tile's share of every bucket with one global atomic per
//      non-empty bucket (count, hpp:1414-1435)
//   C  bucket starts (count_finished), scatter keys and handles in bucket
//      order (distribute, hpp:1464-1490)
//   D  a dynamic queue of windows of `window` positions: the runs of buckets
//      of at most `window` strings that start in a window are finished by the
//      leaf sorter as one segment (sort_segment, the SmallsortJob
//      counterpart); larger buckets, which come first, are finished alone (up
//      to SMALL_MAX strings), copied out when their strings are all equal, or
//      handed to the level-synchronous passes as a segment
//      (distribute_finished, hpp:1492-1584). With LCP output a third barrier precedes the LCPs at
//      the first positions of the runs, which come from the neighbouring
//      buckets' key ranges (sample_sort_lcp, hpp:311-396).
// Latency-bound: dependent gathers, the sorts' chains and the barriers.
// Sorting the samples in every block costs less than a barrier after one
// shared sort did, and the register sorts of phase D less than sample-sort
// steps in shared memory: 487 k digit strings 150 -> 96 us, 7.8 k strings
// 65 -> 33 us of device time.
// Every barrier wait is bounded: after `limit` polls a block sets
// ERR_TIMEOUT and returns, and the blocks still waiting see the flag and
// return as well.
#pragma once

#include "kernels_leaf.cuh"

namespace pssgpu {

constexpr int WAVE_G = 16;
constexpr int WAVE_THREADS = 32 * WAVE_G;
constexpr int WAVE_PER = 8;           // strings per thread through phases A-C
constexpr int WAVE_MAX_BITS = 11;     // at most 2047 splitters, 4095 buckets
constexpr int WAVE_BKT = 2 << WAVE_MAX_BITS;   // 4096 bucket slots
constexpr uint32_t WAVE_WINDOW_MAX = 1024;     // largest window (positions)
constexpr uint32_t WAVE_TILE_MAX = (uint32_t)WAVE_THREADS * WAVE_PER;

// Global state of one wave sort (in the workspace). Everything up to the
// splitters is zeroed by the host before the launch.
struct WaveState {
    uint32_t bar;        // grid barrier arrivals
    uint32_t next_task;  // phase-D tasks taken behind the blocks' first ones
    uint32_t nruns;      // runs recorded (LCP output only)
    uint32_t done;       // blocks that have ended
    uint32_t pad[2];
    // with tracing on: the largest SM-clock cycles any block spent in phase
    // A, B, the wait behind it, C (+ its wait) and D (+ the LCPs)
    unsigned long long cycles[5];
    uint32_t gcount[WAVE_BKT];   // bucket counts
    uint64_t spl[WAVE_BKT / 2];  // sorted splitters
    // LCP output only: the first bucket of every run that phase D finished
    // or handed over, its smallest key and the largest key of its last bucket
    uint16_t run[WAVE_BKT];
    uint64_t bmin[WAVE_BKT];
    uint64_t bmax[WAVE_BKT];
};

// Dynamic shared memory of k_wave: bucket starts, then either the phase A-C
// view (samples, tree, per-bucket counts) or the leaf sorter's.
struct WaveSmemABC {
    uint64_t samp[WAVE_BKT];     // exchange buffer of the sort, then the sorted samples
    uint64_t tree[WAVE_BKT / 2]; // level order, index 1..k
    uint32_t cnt[WAVE_BKT];      // per bucket: count in the tile, then the tile's base
};
struct WaveSmemSort {
    SegState<WAVE_G> seg;
    unsigned char tail[SegState<WAVE_G>::TAIL];
};
struct WaveSmem {
    uint32_t start[WAVE_BKT + 1];  // bucket starts (exclusive scan), start[B] = n
    uint32_t pad[3];
    union {
        WaveSmemABC abc;
        WaveSmemSort sort;
    } u;
};

// Grid barrier number `round` (1, 2, ...): every block arrives once; false
// when the wait gave up (ERR_TIMEOUT set here or by another block).
__device__ __forceinline__ bool wave_barrier(WaveState* ws, uint32_t round, uint32_t* err,
                                             uint32_t limit)
{
    __shared__ uint32_t ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&ws->bar, 1u);
        const uint32_t target = round * gridDim.x;
        uint32_t polls = 0;
        ok = 1;
        while (*(volatile uint32_t*)&ws->bar < target) {
            if ((*(volatile uint32_t*)err & ERR_TIMEOUT) || ++polls > limit) {
                set_error(err, ERR_TIMEOUT);
                ok = 0;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// first b in [0, B] with start[b] >= x (start is non-decreasing, start[B] = n)
__device__ __forceinline__ uint32_t wave_lower(const uint32_t* start, uint32_t B, uint32_t x)
{
    uint32_t lo = 0, hi = B;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (start[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// LCP output: record the run of positions [P, P + m), m >= 1, which starts
// and ends with a bucket, and its key range. red: two words of shared memory.
__device__ __forceinline__ void wave_note_run(const Work& w, WaveState* ws, const uint32_t* start, uint32_t B,
                                              uint32_t P, uint32_t m, uint64_t* red)
{
    uint64_t mn = ~0ull, mx = 0;
    for (uint32_t q = threadIdx.x; q < m; q += WAVE_THREADS) {
        const uint64_t k = __ldcg(w.keys[1] + P + q);
        mn = min(mn, k);
        mx = max(mx, k);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if (threadIdx.x == 0) {
        red[0] = ~0ull;
        red[1] = 0;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        atomicMin((unsigned long long*)&red[0], (unsigned long long)mn);
        atomicMax((unsigned long long*)&red[1], (unsigned long long)mx);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t b = wave_lower(start, B, P + 1) - 1;   // the bucket that starts at P
        const uint32_t e = wave_lower(start, B, P + m) - 1;   // the bucket that ends the run
        ws->bmin[b] = red[0];
        ws->bmax[e] = red[1];
        if (P) ws->run[atomicAdd(&ws->nruns, 1u)] = (uint16_t)b;
    }
    __syncthreads();
}

// Phase D: sort the strings at positions [P, P + m) of buffer 1 (m <=
// SMALL_MAX), whole buckets, by the leaf sorter. The run is one segment at
// depth 0: its buckets are consecutive key ranges and the keys at depth 0 are
// cached.
__device__ __forceinline__ void wave_sort_run(const Work& w, WaveState* ws, WaveSmem& sm, uint32_t B,
                                              uint32_t P, uint32_t m, uint64_t* red)
{
    if (m == 0) return;
    if (w.lcp) wave_note_run(w, ws, sm.start, B, P, m, red);
    if (m == 1) {
        if (threadIdx.x == 0) w.perm[P] = h_id(w, __ldcg(w.hnd[1] + P));
        return;
    }
    SegState<WAVE_G>& seg = sm.u.sort.seg;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < m; i += WAVE_THREADS) {
        seg.hnd[i] = __ldcg(w.hnd[1] + P + i);
        seg.idx[idx_at(i)] = (uint16_t)i;
    }
    sort_segment<WAVE_G, false>(w, seg, sm.u.sort.tail, P, m, 1, 0, true);
    __syncthreads();
}

// Phase D: bucket b, of more than `window` strings.
__device__ __forceinline__ void wave_large_bucket(const Work& w, WaveState* ws, WaveSmem& sm, uint32_t B,
                                                  uint32_t b, uint64_t* red)
{
    const uint32_t P = sm.start[b], c = sm.start[b + 1] - P;
    const uint64_t s = (b & 1) ? __ldcg(ws->spl + (b >> 1)) : 0ull;
    const bool equal = (b & 1) && key_terminated(s);
    if (!equal && c <= (uint32_t)SMALL_MAX) {
        wave_sort_run(w, ws, sm, B, P, c, red);
        return;
    }
    if (w.lcp) {
        if (!(b & 1)) {
            wave_note_run(w, ws, sm.start, B, P, c, red);
        } else if (threadIdx.x == 0) {  // all of its keys are the splitter
            ws->bmin[b] = ws->bmax[b] = s;
            if (P) ws->run[atomicAdd(&ws->nruns, 1u)] = (uint16_t)b;
        }
    }
    if (equal) {
        for (uint32_t q = threadIdx.x; q < c; q += WAVE_THREADS) {
            w.perm[P + q] = h_id(w, __ldcg(w.hnd[1] + P + q));
            if (w.lcp && q) w.lcp[P + q] = lcp_key_depth(s);
        }
    } else if (threadIdx.x == 0) {
        push_seg(w, 1, (b & 1) ? Seg{P, c, 8u, 1u} : Seg{P, c, 0u, 1u | META_VALID});
    }
}

// Draw and sort S samples (at most E * WAVE_THREADS) into samp, the same ones
// in every block.
template <int E>
__device__ __forceinline__ void wave_samples(const Work& w, uint32_t S, uint64_t* samp)
{
    uint64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = threadIdx.x + e * WAVE_THREADS;
        const uint64_t h = mix64(0x7761766573616d70ull ^ i);
        const uint32_t r = (uint32_t)(((h >> 32) * w.n) >> 32);
        x[e] = i < S ? load_key(w.chars, w.nchars, __ldg(w.offs + r)) : ~0ull;
    }
    group_sort<E, WAVE_G, false>(x, samp);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) samp[threadIdx.x * E + e] = x[e];
    __syncthreads();
}

// L: levels of the splitter tree, over: samples per splitter (1 or 2).
// w.cur must be 0: the wave's leftovers (big segments, tied runs, deep
// groups) go to the lists of parity 1, with their strings in buffer 1.
__global__ void __launch_bounds__(WAVE_THREADS, 2) k_wave(Work w, WaveState* ws, uint32_t L, uint32_t over,
                                                          uint32_t window, uint32_t limit, int trace,
                                                          uint32_t* host_counters)
{
    long long cl = clock64();
    auto lap = [&](int k) {  // phase k ended here (tracing only)
        if (!trace || threadIdx.x) return;
        const long long t = clock64();
        atomicMax(ws->cycles + k, (unsigned long long)(t - cl));
        cl = t;
    };
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WaveSmem& sm = *reinterpret_cast<WaveSmem*>(smem_raw);
    __shared__ uint32_t tmp[32];
    __shared__ uint64_t red[2];
    __shared__ uint32_t task, big_at;
    __shared__ uint32_t ended;
    // every block's way out: the last one hands the counters to the host (no
    // copy after the kernel)
    auto leave = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            ended = atomicAdd(&ws->done, 1u);
            __threadfence();
        }
        __syncthreads();
        if (ended + 1 == gridDim.x)
            for (uint32_t q = threadIdx.x; q < (uint32_t)C_COUNT; q += WAVE_THREADS)
                host_counters[q] = __ldcg(w.counters + q);
    };
    uint32_t* err = w.counters + C_ERR;
    const uint32_t G = gridDim.x, n = w.n;
    const uint32_t k = (1u << L) - 1, B = 2 * k + 1;
    const uint32_t per_blk = (n + G - 1) / G;  // <= WAVE_TILE_MAX (host)
    const uint32_t t0 = min(blockIdx.x * per_blk, n), t1 = min(t0 + per_blk, n);

    // ---- A: keys of the tile; samples and tree -------------------------------
    if (blockIdx.x == 0 && threadIdx.x == 0 && w.chars[w.nchars - 1] != 0)
        set_error(err, ERR_UNTERMINATED);
    uint64_t key[WAVE_PER];
#pragma unroll
    for (int j = 0; j < WAVE_PER; ++j) {
        const uint32_t i = t0 + threadIdx.x + j * WAVE_THREADS;
        key[j] = 0;
        if (i < t1) {
            const uint64_t off = __ldg(w.offs + i);
            if (off >= w.nchars) set_error(err, ERR_OFFSET);
            key[j] = load_key(w.chars, w.nchars, off);
        }
    }
    uint64_t* samp = sm.u.abc.samp;
    const uint32_t S = over << L;
    if (S <= 2u * WAVE_THREADS) wave_samples<2>(w, S, samp);
    else if (S <= 4u * WAVE_THREADS) wave_samples<4>(w, S, samp);
    else wave_samples<8>(w, S, samp);
    uint64_t* tree = sm.u.abc.tree;
    uint32_t* cnt = sm.u.abc.cnt;
    if (blockIdx.x == 0)
        for (uint32_t j = threadIdx.x; j < k; j += WAVE_THREADS) ws->spl[j] = samp[over * (j + 1) - (over - 1)];
    for (uint32_t v = 1 + threadIdx.x; v <= k; v += WAVE_THREADS) {
        const uint32_t h = 31 - __clz((int)v);
        const uint32_t p = v - (1u << h);
        const uint32_t r = ((2 * p + 1) << (L - 1 - h)) - 1;  // in-order rank
        tree[v] = samp[over * (r + 1) - (over - 1)];
    }
    for (uint32_t b = threadIdx.x; b < B; b += WAVE_THREADS) cnt[b] = 0;
    __syncthreads();
    lap(0);

    // ---- B: classify, count, reserve ---------------------------------------------
    uint32_t pk[WAVE_PER];  // (bucket << 16) | rank inside the tile's share
#pragma unroll
    for (int j = 0; j < WAVE_PER; ++j) {
        const uint32_t i = t0 + threadIdx.x + j * WAVE_THREADS;
        pk[j] = 0xFFFFFFFFu;
        if (i < t1) {
            uint32_t v = 1;
            uint64_t cand = 0;
            for (uint32_t l = 0; l < L; ++l) {
                const uint64_t tv = tree[v];
                const bool gt = key[j] > tv;
                cand = gt ? cand : tv;
                v = 2 * v + (gt ? 1u : 0u);
            }
            const uint32_t r = v - (1u << L);
            const uint32_t b = 2 * r + ((r < k && cand == key[j]) ? 1u : 0u);
            pk[j] = (b << 16) | atomicAdd(&cnt[b], 1u);
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < B; b += WAVE_THREADS) {
        const uint32_t c = cnt[b];
        cnt[b] = c ? atomicAdd(&ws->gcount[b], c) : 0u;
    }
    lap(1);
    if (!wave_barrier(ws, 1, err, limit)) return leave();
    lap(2);
    // input errors are all flagged in phase A: every block sees the same
    // bits here and leaves together
    if (*(volatile uint32_t*)err & (ERR_OFFSET | ERR_UNTERMINATED)) return leave();

    // ---- C: bucket starts, scatter ----------------------------------------
    for (uint32_t b = threadIdx.x; b < B; b += WAVE_THREADS) sm.start[b] = __ldcg(ws->gcount + b);
    __syncthreads();
    block_scan_array<WAVE_THREADS>(sm.start, (int)B, tmp);
    if (threadIdx.x == 0) sm.start[B] = n;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < WAVE_PER; ++j) {
        if (pk[j] == 0xFFFFFFFFu) continue;
        const uint32_t i = t0 + threadIdx.x + j * WAVE_THREADS;
        const uint32_t b = pk[j] >> 16;
        const uint32_t dest = sm.start[b] + cnt[b] + (pk[j] & 0xFFFFu);
        if (dest >= n) {  // counts and starts disagree
            set_error(err, ERR_INTERNAL);
            continue;
        }
        w.keys[1][dest] = key[j];
        w.hnd[1][dest] = h_make(w, i, __ldg(w.offs + i));
    }
    if (!wave_barrier(ws, 2, err, limit)) return leave();
    lap(3);

    // ---- D: buckets over `window` strings, then the windows of small buckets ----
    // One queue, whose first G tasks are the blocks' own: the large buckets, then
    // the windows. Large buckets by b modulo G left a block with four of them
    // while others had none (700 k strings over 2 letters, 256 buckets: 530 us,
    // 236 from the queue). They are numbered by the threads that find them, in
    // every block alike.
    const uint32_t ntask = (n + window - 1) / window;
    uint32_t flags = 0;  // bit q: bucket threadIdx.x + q * WAVE_THREADS is large
    for (uint32_t b = threadIdx.x, q = 0; b < B; b += WAVE_THREADS, ++q)
        if (sm.start[b + 1] - sm.start[b] > window) flags |= 1u << q;
    uint32_t large;
    const uint32_t before = block_excl_sum<WAVE_THREADS>(__popc(flags), tmp, &large);
    if (threadIdx.x == 0) big_at = B;
    __syncthreads();
    for (uint32_t t = blockIdx.x; t < large + ntask; t = task) {
        if (t < large) {
            if (t - before < (uint32_t)__popc(flags)) {
                uint32_t m = flags;
                for (uint32_t q = t - before; q; --q) m &= m - 1;
                big_at = threadIdx.x + (__ffs(m) - 1) * WAVE_THREADS;
            }
            __syncthreads();
            wave_large_bucket(w, ws, sm, B, big_at, red);
        } else {
            const uint32_t lo = (t - large) * window, hi = min(lo + window, n);
            const uint32_t b_lo = wave_lower(sm.start, B, lo);
            const uint32_t b_hi = wave_lower(sm.start, B, hi);
            if (large)  // at most one starts in a window
                for (uint32_t b = b_lo + threadIdx.x; b < b_hi; b += WAVE_THREADS)
                    if (sm.start[b + 1] - sm.start[b] > window) atomicMin(&big_at, b);
            __syncthreads();
            const uint32_t bb = min(big_at, b_hi);
            wave_sort_run(w, ws, sm, B, sm.start[b_lo], sm.start[bb] - sm.start[b_lo], red);
            if (bb < b_hi) wave_sort_run(w, ws, sm, B, sm.start[bb + 1], sm.start[b_hi] - sm.start[bb + 1], red);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            task = G + atomicAdd(&ws->next_task, 1u);
            big_at = B;
        }
        __syncthreads();
    }
    if (!w.lcp) {
        lap(4);
        return leave();
    }

    // ---- LCPs at the first positions of the runs --------------------------------
    if (!wave_barrier(ws, 3, err, limit)) return leave();
    const uint32_t nruns = __ldcg(&ws->nruns);
    for (uint32_t q = blockIdx.x * WAVE_THREADS + threadIdx.x; q < nruns; q += G * WAVE_THREADS) {
        const uint32_t b = __ldcg(ws->run + q);
        const uint32_t P = sm.start[b];
        const uint32_t p = wave_lower(sm.start, B, P) - 1;  // previous non-empty bucket
        w.lcp[P] = lcp_key_type(__ldcg(ws->bmax + p), __ldcg(ws->bmin + b));
    }
    lap(4);
    leave();
}

}  // namespace pssgpu
