// work.cuh -- the device-side state of one sort, passed by value to kernels.
#pragma once

#include "device_common.cuh"

namespace pssgpu {

constexpr int TILE = 8192;          // most strings per classify / scatter tile (Work::tshift)
constexpr int TILE_THREADS = 512;   // 16 strings per thread
constexpr int MAX_TREE_BITS = 10;   // 1023 splitters, 2047 buckets (pS5's DefaultTreebits)
constexpr int MAX_BKT = 2056;       // bucket slots per big segment: 2047 + the two prefix buckets
constexpr int JMAX_CHUNKS = 32;     // common-prefix jump of one pass: at most 32 8-byte chunks
constexpr int SMALL_MAX = 4096;     // largest segment the leaf sorters take
constexpr int WARP_GROUP_MAX = 32;  // groups this small are finished by one warp
// equal-string buckets this small are copied out by one thread of k_children
// (1.95 M strings over 4 letters with LCPs: 480 us at 64, 472 at 16, 476 at 4);
// larger ones become META_FINAL segments, whose depth is the strings' length
constexpr int FINAL_INLINE = 16;
constexpr int CHUNK = 32;           // tiles per chunk of the destination scan
constexpr uint32_t DBL_MAX = 4096;  // largest group a suffix sort hands to the rounds of kernels_suffix.cuh

// segment list classes
// (at most 32, 256, 1024 and SMALL_MAX strings; L_BIG above)
enum : int { L_BIG = 0, L_TINY = 1, L_SMALLA = 2, L_SMALLB = 3, L_SMALLC = 4, L_NCLASS = 5 };

// counters[] layout
enum : int {
    C_PAR = 10,       // counters per parity block: [class] lengths, then tiles
    C_NTILES = 5,     // + C_PAR * parity: tiles of the big list
    C_NSTR = 5,       // + C_PAR * parity + class (1..4): strings in the small lists
    C_NBND = 20,      // boundary list length
    C_ERR = 22,       // error bits
    // per-pass statistics, reset every pass
    C_P_BIG = 24,     // strings in big sample-sort segments
    C_P_STALE = 25,   // of those, strings whose key was gathered this pass
    C_P_FINAL = 26,   // strings copied out of big all-equal segments
    C_P_SCATTER = 27, // strings moved by the scatter
    C_P_TIE = 28,     // of the big strings, those classified behind a common-prefix jump
    C_P_JCHUNKS = 29, // their prefix chunks: sum over jump segments of size * jump / 8
    C_P_FIRST = C_P_BIG,
    C_P_LAST = C_P_JCHUNKS,
    C_MULTI = 30,     // + parity: big segments of more than CHUNK tiles in the list
    C_DEEP = 32,      // + parity: length of the deep-group list
    C_SFX = 34,       // suffix-set check: nonzero when the input is not all suffixes of a text
    C_DBL = 35,       // suffix groups the passes hand to the rounds of kernels_suffix.cuh
    C_DBL_CNT = 36,   // + 3 * parity + class: lists of a suffix round
    C_DBL_MEMB = 42,  // 64-bit (42, 43): members of those groups, summed over rounds
    C_ALPHA = 44,     // suffix-set check: which of the 256 chars occur (8 words)
    C_COUNT = 52
};

struct Work {
    // input arena
    const uint8_t* chars;
    uint64_t nchars;
    const uint64_t* offs;
    uint32_t n;
    // String handles: (id << hbits) | arena offset when both fit in 64 bits
    // (packed), else the id alone and the offset is read from offs[id].
    // Carrying the offset saves the dependent offs[id] load of every gather.
    uint32_t hbits;
    uint64_t hmask;
    int packed;
    // Ids count from their root segment's begin (a batch without LCP output and
    // with packed handles: the permutation needs no pass that makes it local)
    int local;
    // handle / key ping-pong
    uint64_t* hnd[2];
    uint64_t* keys[2];
    uint16_t* bkt;
    // outputs
    uint32_t* perm;
    uint32_t* lcp;  // may be null
    // bookkeeping
    uint32_t* counters;
    uint2* bnd;  // (position, depth) of split boundaries
    uint32_t bnd_cap;
    // segment lists per class, double-buffered by pass parity
    Seg* list[L_NCLASS][2];
    uint32_t cap[L_NCLASS];
    // per big segment of the current pass
    uint32_t* tile_start;  // [cap[L_BIG] + 1]
    uint8_t* tree_bits;    // [cap[L_BIG]]; 0 = all-equal copy
    uint64_t* tree;        // [cap[L_BIG]][1024], level order, index 1..k
    uint64_t* spl;         // [cap[L_BIG]][1024], sorted splitters
    uint32_t* bcount;      // [cap[L_BIG]][MAX_BKT]
    uint32_t* bstart;      // [cap[L_BIG]][MAX_BKT]
    uint8_t* bflags;       // [cap[L_BIG]]: 1 = whole segment in one bucket
    // Common-prefix jump: when every sample shares more chars beyond the
    // segment depth, jump[s] = that many chars (a multiple of 8) and jpre holds
    // them as keys; the tree then splits at depth + jump, and strings that
    // leave the prefix earlier go to a first ('<' prefix) or last ('>' prefix)
    // bucket.
    uint32_t* jump;        // [cap[L_BIG]]
    uint64_t* jpre;        // [cap[L_BIG]][JMAX_CHUNKS]
    // Scatter destinations, pS5's count / count_finished over parts (hpp:1414-1460)
    // with tiles as parts: per tile and bucket the count, then (after the
    // bucket-major, tile-minor exclusive scan) the tile's first destination.
    // The scan runs in chunks of CHUNK tiles.
    uint32_t* chunk_start;  // [cap[L_BIG] + 1]: first chunk of each big segment
    uint32_t* tcount;       // [tile_cap][MAX_BKT]
    uint32_t* ccount;       // [tile_cap][MAX_BKT]: chunk sums, then chunk bases
    uint32_t tile_cap;
    uint32_t tshift;        // strings per tile: 2^tshift, at most TILE (tile_shift)
    int cur;               // parity of the lists read in this pass
    // Deep groups: groups of at most 32 strings that a leaf sorter's warp
    // window found stuck on a long common prefix, handed to k_deep (one warp
    // each) in the next pass; double-buffered by pass parity, null when not
    // allocated
    Seg* deep[2];
    uint32_t deep_cap;
    // splitter-tree levels for a big segment of 2^k..2^(k+1)-1 strings
    // (0: the default rule), set from a tuning table
    uint8_t tree_bits_by_size[33];
    // Suffix sets (every string is a suffix of one text: offs[i] = i, no NUL
    // before the last char): the text is packed at kbits bits per char (its
    // chars numbered from 1 in their order, 0 past the end), so a key holds
    // kchars chars, 21 of a 4-letter text where bytes hold 8, and most
    // suffixes are told apart by their first key. Groups of at most DBL_MAX
    // that share a key go to the list dbl, which is finished by the rounds of
    // kernels_suffix.cuh. No LCPs are written before that.
    // kchars is 8 and kbits 8 otherwise.
    const uint64_t* ptext;
    uint64_t kmask;  // the kchars * kbits top bits
    uint32_t kbits, kchars;
    int suffix;
    Seg* dbl;
    uint32_t dbl_cap;
};

// buckets of a classified big segment: the tree's 2^(L+1) - 1, plus the two
// prefix buckets of a jump segment
__device__ __forceinline__ uint32_t seg_buckets(const Work& w, int s)
{
    return (2u << w.tree_bits[s]) - 1 + (w.jump[s] ? 2u : 0u);
}

__host__ __device__ __forceinline__ uint32_t seg_tiles(const Work& w, uint32_t size)
{
    return (size + (1u << w.tshift) - 1) >> w.tshift;
}

// Strings per tile in a sort of n: fewer where 8192 would leave a thread 16
// strings to gather one after another while SMs idle, or one wave of tiles
// just over full (classify 53 -> 26 us for 143 tiles; 1.3 M strings 326 -> 303
// us); 8192 where tiles are plenty, as every tile pays for its buckets. With
// 8192 and with 4096, in us, of 2, 4, 6, 8 and 12 Mi strings: prefixes 702 / 678,
// 918 / 892, 1118 / 1100, 1314 / 1298, 1722 / 1736 (24 Mi: 2946 / 3067);
// letters 335 / 340, 495 / 499, 634 / 653, 773 / 799; suffixes 498 / 496, 718 /
// 727, 8 Mi 1093 / 1124, 16 Mi 1774 / 1856. The line lies where the one's gain
// is 3% and the other's loss 1%; beyond it the loss grows.
constexpr uint64_t TILE_MID_N = 9u << 19, TILE_SMALL_N = 1u << 19;
__host__ __device__ constexpr uint32_t tile_shift(uint64_t n)
{
    return n > TILE_MID_N ? 13 : n > TILE_SMALL_N ? 12 : 11;
}

// list class of a segment
__host__ __device__ __forceinline__ int seg_class(uint32_t size)
{
    if (size > (uint32_t)SMALL_MAX) return L_BIG;
    return size > 1024 ? L_SMALLC : size > 256 ? L_SMALLB : size > (uint32_t)WARP_GROUP_MAX ? L_SMALLA : L_TINY;
}

__device__ __forceinline__ uint64_t h_make(const Work& w, uint32_t id, uint64_t off)
{
    return w.packed ? (((uint64_t)id << w.hbits) | off) : (uint64_t)id;
}

__device__ __forceinline__ uint32_t h_id(const Work& w, uint64_t h)
{
    return w.packed ? (uint32_t)(h >> w.hbits) : (uint32_t)h;
}

__device__ __forceinline__ uint64_t h_off(const Work& w, uint64_t h)
{
    return w.packed ? (h & w.hmask) : __ldg(w.offs + h);
}

// Handle of the string at position p of the segment that begins at `begin`.
// Root segments have none stored: their strings are read once, in order, and
// a pass that wrote 8 bytes of handle per string for them took 0.2 ms of the
// 64 Mi sort. One load from either array, without a branch before it.
__device__ __forceinline__ const uint64_t* handle_src(const Work& w, uint32_t meta)
{
    return (meta & META_ROOT) ? w.offs : w.hnd[meta & META_BUF];
}
__device__ __forceinline__ uint64_t handle_of(const Work& w, uint32_t meta, uint32_t begin, uint32_t p, uint64_t x)
{
    return (meta & META_ROOT) ? h_make(w, w.local ? p - begin : p, x) : x;
}
__device__ __forceinline__ uint64_t handle_at(const Work& w, uint32_t meta, uint32_t begin, uint32_t p)
{
    return handle_of(w, meta, begin, p, __ldg(handle_src(w, meta) + p));
}

// handle_at for the first read of every string, which checks root offsets.
__device__ __forceinline__ uint64_t handle_at_checked(const Work& w, uint32_t meta, uint32_t begin, uint32_t p)
{
    const uint64_t x = __ldg(handle_src(w, meta) + p);
    if ((meta & META_ROOT) && x >= w.nchars) set_error(w.counters + C_ERR, ERR_OFFSET);
    return handle_of(w, meta, begin, p, x);
}

// Key of the kchars chars of a packed text at position p (0 past its end).
__device__ __forceinline__ uint64_t packed_key(const Work& w, uint64_t p)
{
    if (p >= w.nchars) return 0;
    const uint64_t bit = p * w.kbits;
    const uint64_t* q = w.ptext + (bit >> 6);
    const uint32_t s = (uint32_t)bit & 63u;
    const uint64_t hi = __ldg(q), lo = __ldg(q + 1);
    return (s ? (hi << s) | (lo >> (64 - s)) : hi) & w.kmask;
}

// key at arena position p
__device__ __forceinline__ uint64_t key_at(const Work& w, uint64_t p)
{
    return w.suffix ? packed_key(w, p) : load_key(w.chars, w.nchars, p);
}

// key of the string behind handle h at depth d
__device__ __forceinline__ uint64_t h_key(const Work& w, uint64_t h, uint32_t d)
{
    return key_at(w, h_off(w, h) + d);
}

// Do strings that share this key end inside it (and so are equal)? Suffixes
// of one text never are.
__device__ __forceinline__ bool key_ends(const Work& w, uint64_t k)
{
    return !w.suffix && key_terminated(k);
}

// A tied group of a suffix set: the strings at [pos, pos + size), which share
// depth chars, to the list dbl. META_PERM: their ids are in perm, else their
// handles in buffer meta & META_BUF.
__device__ __forceinline__ void push_dbl(const Work& w, const Seg& g)
{
    const uint32_t at = atomicAdd(w.counters + C_DBL, 1u);
    if (at < w.dbl_cap) w.dbl[at] = g;
    else set_error(w.counters + C_ERR, ERR_OVERFLOW);
}

// push_dbl for a whole warp: lanes with push set append g.
__device__ __forceinline__ void push_dbl_warp(const Work& w, bool push, const Seg& g)
{
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(0xffffffffu, push);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == (uint32_t)leader) base = atomicAdd(w.counters + C_DBL, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!push) return;
    const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
    if (at < w.dbl_cap) w.dbl[at] = g;
    else set_error(w.counters + C_ERR, ERR_OVERFLOW);
}

// Append segment c to its class's list of parity nxt.
__device__ __forceinline__ void push_seg(const Work& w, int nxt, Seg c)
{
    const int cls = seg_class(c.size);
    const uint32_t at = atomicAdd(w.counters + C_PAR * nxt + cls, 1u);
    if (at >= w.cap[cls]) {
        set_error(w.counters + C_ERR, ERR_OVERFLOW);
        return;
    }
    w.list[cls][nxt][at] = c;
    if (cls == L_BIG) {
        const uint32_t tiles = seg_tiles(w, c.size);
        atomicAdd(w.counters + C_PAR * nxt + C_NTILES, tiles);
        if (tiles > (uint32_t)CHUNK) atomicAdd(w.counters + C_MULTI + nxt, 1u);
    } else {
        atomicAdd(w.counters + C_PAR * nxt + C_NSTR + cls, c.size);
    }
}

// push_seg for a whole warp: lanes with push set append c. One reservation
// per class and warp, and the class's tile or string count added once (a
// launch that pushes many segments would otherwise serialise on these few
// counters).
__device__ __forceinline__ void push_seg_warp(const Work& w, int nxt, bool push, const Seg& c)
{
    const uint32_t lane = threadIdx.x & 31;
    const int cls = push ? seg_class(c.size) : -1;
#pragma unroll
    for (int k = 0; k < L_NCLASS; ++k) {
        const uint32_t m = __ballot_sync(0xffffffffu, cls == k);
        if (!m) continue;
        const int leader = __ffs(m) - 1;
        const uint32_t tiles = cls == k && k == L_BIG ? seg_tiles(w, c.size) : 0u;
        const uint32_t amount = __reduce_add_sync(0xffffffffu, cls != k ? 0u : k == L_BIG ? tiles : c.size);
        const uint32_t multi = __reduce_add_sync(0xffffffffu, tiles > (uint32_t)CHUNK ? 1u : 0u);
        uint32_t base = 0;
        if (lane == (uint32_t)leader) {
            base = atomicAdd(w.counters + C_PAR * nxt + k, (uint32_t)__popc(m));
            if (k == L_BIG) {
                atomicAdd(w.counters + C_PAR * nxt + C_NTILES, amount);
                if (multi) atomicAdd(w.counters + C_MULTI + nxt, multi);
            } else {
                atomicAdd(w.counters + C_PAR * nxt + C_NSTR + k, amount);
            }
        }
        base = __shfl_sync(0xffffffffu, base, leader);
        if (cls == k) {
            const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
            if (at >= w.cap[k]) set_error(w.counters + C_ERR, ERR_OVERFLOW);
            else w.list[k][nxt][at] = c;
        }
    }
}

// push_seg for a whole block (every thread calls it): one reservation per class
// and block, for launches whose warps all push to several classes. The roots
// of a 100k-instance batch: 35 us per warp, 9 per block of 512 (batch 2.005 -> 1.979 ms).
struct PushBlock {
    uint32_t count[L_NCLASS], amount[L_NCLASS], base[L_NCLASS], multi;
};
__device__ __forceinline__ void push_seg_block(const Work& w, PushBlock& sm, int nxt, bool push, const Seg& c)
{
    const uint32_t t = threadIdx.x, lane = t & 31;
    if (t < (uint32_t)L_NCLASS) sm.count[t] = sm.amount[t] = 0;
    if (t == 0) sm.multi = 0;
    __syncthreads();
    const int cls = push ? seg_class(c.size) : -1;
    const uint32_t tiles = cls == L_BIG ? seg_tiles(w, c.size) : 0u;
    uint32_t at = 0;  // in the block's share of the class
#pragma unroll
    for (int k = 0; k < L_NCLASS; ++k) {
        const uint32_t m = __ballot_sync(0xffffffffu, cls == k);
        if (!m) continue;
        const int leader = __ffs(m) - 1;
        const uint32_t amount = __reduce_add_sync(0xffffffffu, cls != k ? 0u : k == L_BIG ? tiles : c.size);
        uint32_t base = 0;
        if (lane == (uint32_t)leader) {
            base = atomicAdd(&sm.count[k], (uint32_t)__popc(m));
            atomicAdd(&sm.amount[k], amount);
        }
        base = __shfl_sync(0xffffffffu, base, leader);
        if (cls == k) at = base + __popc(m & ((1u << lane) - 1u));
    }
    if (tiles > (uint32_t)CHUNK) atomicAdd(&sm.multi, 1u);
    __syncthreads();
    if (t < (uint32_t)L_NCLASS && sm.count[t]) {
        sm.base[t] = atomicAdd(w.counters + C_PAR * nxt + t, sm.count[t]);
        atomicAdd(w.counters + C_PAR * nxt + (t == L_BIG ? C_NTILES : C_NSTR + t), sm.amount[t]);
        if (t == L_BIG && sm.multi) atomicAdd(w.counters + C_MULTI + nxt, sm.multi);
    }
    __syncthreads();
    if (push) {
        at += sm.base[cls];
        if (at >= w.cap[cls]) set_error(w.counters + C_ERR, ERR_OVERFLOW);
        else w.list[cls][nxt][at] = c;
    }
    __syncthreads();  // sm is free
}

}  // namespace pssgpu
