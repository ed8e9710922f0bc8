// Index inverse of the sparse attention pattern: from indices [s_q, topk] (kv row chosen by each slot of each
// query) to a CSR by kv row -- row_ptr [s_kv + 1] and entries [s_q * topk], where the entries of a row are the flat
// slot ids q * topk + slot of the valid slots that chose it, in ascending order.  The order is fixed (not the
// arrival order of atomics), so the result is reproducible bit for bit.
//
// Method: a stable least-significant-digit radix sort of (key = kv row, value = flat slot id).  The values start in
// ascending order, so a stable sort by key alone yields (row, flat id) order.  Unused slots get the key s_kv and end
// up behind row_ptr[s_kv] in flat order.  Per pass three kernels: digit histogram per block, exclusive scan of the
// [digit][block] matrix, stable scatter; keys are formed from the indices on the fly in the first pass, travel as 16 bits
// where s_kv fits, and are not written by the last pass.  row_ptr: the last pass takes, for every row, the smallest
// position at which a run of its key begins (integer minimum: order does not matter), and a last kernel (with two small ones
// before it for many rows) gives rows without a slot the next row's position.  Inputs of at most one block (8192 slots) are sorted by that block in shared memory.
// Where the rows' counters fit into shared memory and the slots are many enough for them, no sort: a count per row and group of queries,
// then every slot goes to its place at once (direct form, below).
// All kernels are launched behind their predecessor's start (programmatic dependent launch).
//
// The reference has no such operator; the validity rule is the one of its kernel (mla_bwd/mla_bwd.cu:765-789).
#pragma once
#include <algorithm>
#include <cstdint>
#include <climits>
#include <cuda_runtime.h>

#include "sm100_ptx.cuh"

namespace inv {

constexpr int kThreads = 512;
// Entries per thread; a block's entries are contiguous, a warp's are (32 kItems of them): (warp, step, lane) order is flat
// order.  Large inputs take fourteen (8.4 M slots: 159 us with eight, 144 with twelve, 139 with sixteen, 137 with fourteen), or sixteen
// where the last round of blocks on the 148 SMs would be nearly empty otherwise: where rounds x entries, the entries that a thread
// goes through one after the other, are fewer with sixteen.  Fourteen / sixteen measured (us; * what the rule takes): 2.1 M slots
// 38.9* / 41.4, 2.4 M 54.4 / 43.2* (two rounds against one), 3.0 M 56.3* / 62.5, 4.3 M 85.3 / 80.3* (three against two), 5.2 M 86.2* / 95.2,
// 7.1 M 117.4 / 115.5*, 8.4 M 134.5* / 135.4, 9.0 M 148.7 / 150.2* (70 entries against 64; the one range where it is wrong, by 1 %), 9.6 M
// 160.9 / 153.2*, 10.7 M 176.6 / 169.9*, 12 M 194.1 / 190.7*, 14.5 M 226.4 / 227.2*, 16.8 M 258.9* / 264.5.  Below kLargeInput they take four,
// so that there are blocks for all SMs (270,000 slots: 46 us with sixteen, 29 with eight).
constexpr int kItemsLarge = 14, kItemsFewerRounds = 16, kItemsMid = 4, kItemsSmall = 16;
constexpr int64_t kLargeInput = 1 << 20;
constexpr int kSmallInput = kThreads * kItemsSmall;     // one block sorts this many alone
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRadix = 256;
constexpr int kRowTile = 1024;                   // rows per block of the row_ptr kernel
// Up to this many blocks of rows, a block of the row_ptr kernel finds the first run behind its rows by looking at the rows
// themselves, a block at a time: one step where slots are spread, 0.28 us a step where the rows behind are unused.  With more
// of them two small kernels prepare it (see row_min_kernel): 32 K slots all in the first 1024 of 4 M rows 9.4 ms by looking.
constexpr int kMaxLook = 64;
constexpr int kResidentBlocks = 2 * 148;         // scatter blocks that a B200 runs at once

// Direct form (see there): one block per SM, the counters that fit into its shared memory, threads of the counting, threads and slots
// a thread of the placing.
constexpr int kMaxGroups = 148;
constexpr int64_t kMaxDirect = 20 << 20;         // slots
constexpr int kPlaceRows = 53248;
constexpr int kCountThreads = 1024;
constexpr int kPlaceThreads = 512, kPlaceItems = 10, kBatch = kPlaceThreads * kPlaceItems;

struct Plan {
    int passes;      // 1..4
    int digit_bits;  // <= 8
    int items;       // entries per thread
    int n_blocks;
    bool key16;      // keys fit 16 bits
    bool by_masks;   // block_rank's kMasks (large form; the others always)
    int groups;      // direct form: groups of queries, 0 where the sort is taken
    int per_group;   // queries of a group
    int rows_pad;    // s_kv + 1, padded
};

// Whether the direct form is taken: where its time, by the slots of its largest group and the rows, is not above the sort's, by the slots
// and the rounds of its blocks (units of 0.05 us, without 13.8 us that both have).  So long as `entries` stays in the L2: past that its
// stores, four bytes at a time, go to memory.  Sort / direct, us, distinct rows (* what the rule takes): 16 x 2048 slots on 8192 rows 23.8 /
// 16.7*, on 52000 24.1* / 25.6, 256 x 2048 on 16384 24.1 / 17.6*, on 36000 24.8 / 24.5*, on 44000 24.9* / 28.0, 1 x 20000 on 8192 23.7* /
// 29.5, 300 x 2048 on 32768 29.8 / 25.1*, 512 x 2048 on 52000 41.0 / 35.2*, 8192 x 128 on 4096 36.6 / 19.1*, 1024 x 2048 on 32768 42.4 / 33.8*,
// on 52000 43.4* / 42.0, 4096 x 512 on 8192 39.1 / 26.4*, 20 x 100000 on 50000 44.5* / 115, 2048 x 2048 on 32768 73.5 / 47.2*, 4096 x 2048
// 135 / 75.8*, 8192 x 2048 on 16384 255 / 143*, 10000 x 2048 on 32768 314 / 249*, 12000 x 2048 374* / 385, 16000 x 2048 488* / 818.  However
// often the queries name a row the direct form is the faster one there, too: 4096 x 2048 slots, random rows with repetitions 135 / 75.8, random
// among 64 rows 139 / 104, all the same 135 / 61.5; 1024 x 2048 on 8192 39.2 / 26.2, 44.7 / 33.7 and 49.5 / 21.2.
inline bool direct_form(int32_t s_q, int32_t topk, int32_t s_kv) {
    const int64_t n = static_cast<int64_t>(s_q) * topk;
    if (n <= kSmallInput || s_kv >= kPlaceRows - 4 || n > kMaxDirect) return false;
    const int64_t slots = static_cast<int64_t>((s_q + kMaxGroups - 1) / kMaxGroups) * topk;
    const int64_t sort = n <= kResidentBlocks * kThreads * kItemsMid ? 230
                         : n < kLargeInput                           ? 300
                                                                     : 480 + 300 * std::max<int64_t>(0, n - 2 * kLargeInput) / kLargeInput;
    return slots * 19 / 1024 + 8 * std::max(0, s_kv / 1024 - 16) <= sort;
}

inline Plan make_plan(int32_t s_q, int32_t topk, int32_t s_kv, bool may_be_direct = true) {
    const int64_t n = static_cast<int64_t>(s_q) * topk;
    int bits = 1;
    while ((static_cast<int64_t>(1) << bits) <= static_cast<int64_t>(s_kv)) ++bits;   // keys are 0..s_kv inclusive
    Plan pl;
    pl.passes = (bits + 7) / 8;
    pl.digit_bits = (bits + pl.passes - 1) / pl.passes;
    const auto blocks = [n](int items) { return (n + kThreads * items - 1) / (kThreads * items); };
    const auto steps = [&](int items) { return (blocks(items) + kResidentBlocks - 1) / kResidentBlocks * items; };
    if (n > kSmallInput && n < kLargeInput) pl.items = kItemsMid;
    else pl.items = steps(kItemsFewerRounds) < steps(kItemsLarge) ? kItemsFewerRounds : kItemsLarge;
    pl.n_blocks = static_cast<int>(blocks(pl.items));
    pl.key16 = s_kv < 65536;
    pl.by_masks = pl.n_blocks <= kResidentBlocks;
    pl.groups = pl.per_group = 0;
    pl.rows_pad = (s_kv + 1 + 3) & ~3;
    if (may_be_direct && direct_form(s_q, topk, s_kv)) {
        pl.per_group = (s_q + kMaxGroups - 1) / kMaxGroups;
        pl.groups = (s_q + pl.per_group - 1) / pl.per_group;
    }
    return pl;
}

// What turns a flat slot into its key.
struct Source {
    const int32_t* indices;
    uint32_t topk;
    int32_t s_kv, causal, q_start;
    __device__ __forceinline__ uint32_t key(uint32_t i, int idx) const {
        bool valid = idx >= 0 && idx < s_kv;
        if (causal) valid = valid && idx <= q_start + static_cast<int>(i / topk);
        return static_cast<uint32_t>(valid ? idx : s_kv);
    }
};

__device__ __forceinline__ uint32_t digit_of(uint32_t key, int shift, uint32_t mask) { return (key >> shift) & mask; }

// Digit histogram of every block's entries -> hist[digit][block].  kFirst: keys come from the indices, and row_ptr is
// set to "no run yet".  Bound by reading the keys once.
template <typename KeyT, bool kFirst, int kItems>
__global__ void __launch_bounds__(kThreads)
histogram_kernel(const KeyT* __restrict__ keys, const Source src, uint32_t* __restrict__ hist, uint32_t n, int shift, uint32_t mask,
                 int n_blocks, int32_t* __restrict__ row_ptr) {
    __shared__ uint32_t h[kMaxRadix];
    if (threadIdx.x <= mask) h[threadIdx.x] = 0;
    smla::pdl_wait();
    smla::pdl_trigger();
    __syncthreads();
    const uint32_t first = blockIdx.x * (kThreads * kItems) + threadIdx.x;
    uint32_t k[kItems];
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * kThreads;
        if (kFirst) k[t] = i < n ? static_cast<uint32_t>(__ldg(src.indices + i)) : 0u;
        else k[t] = i < n ? keys[i] : 0u;
    }
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * kThreads;
        if (i < n) atomicAdd(&h[digit_of(kFirst ? src.key(i, static_cast<int>(k[t])) : k[t], shift, mask)], 1u);
    }
    if (kFirst) {
        for (uint32_t r = blockIdx.x * kThreads + threadIdx.x; r <= static_cast<uint32_t>(src.s_kv); r += gridDim.x * kThreads) row_ptr[r] = INT_MAX;
    }
    __syncthreads();
    if (threadIdx.x <= mask) hist[static_cast<size_t>(threadIdx.x) * n_blocks + blockIdx.x] = h[threadIdx.x];
}

// Block-wide exclusive scan of one value per thread (blockDim.x a multiple of 32, at most 1024); returns the
// exclusive prefix and leaves the block total in *total_out (shared).  `warp_sums` holds 32 words.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < n_warps ? warp_sums[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += up;
        }
        warp_sums[lane] = wi - w;
        if (lane == 31) *total_out = wi;
    }
    __syncthreads();
    const uint32_t r = warp_sums[warp] + incl - v;
    __syncthreads();   // warp_sums may be reused by the caller's next call
    return r;
}

// One block per digit: hist[digit][0..n_blocks) becomes its exclusive prefix over the blocks; the digit's total goes
// to totals[digit].  The scatter kernel adds the prefix over the digits itself (at most 256 values).
__global__ void __launch_bounds__(1024)
scan_rows_kernel(uint32_t* __restrict__ hist, uint32_t* __restrict__ totals, int n_blocks) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t tile_total;
    smla::pdl_wait();
    smla::pdl_trigger();
    uint32_t* row = hist + static_cast<size_t>(blockIdx.x) * n_blocks;
    uint32_t carry = 0;
    for (int base = 0; base < n_blocks; base += 1024) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < n_blocks ? row[i] : 0u;
        const uint32_t ex = block_exclusive_scan(v, warp_sums, &tile_total);
        if (i < n_blocks) row[i] = carry + ex;
        carry += tile_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Lanes of the warp whose digit (below 256) equals this lane's, among the active lanes.  Eight ballots: the
// `match.any` instruction gives the same mask but runs on a pipe that takes a warp every ~64 cycles per SM, which
// bounded the whole sort (70 % pipe utilisation under ncu) when it was used.
__device__ __forceinline__ uint32_t same_digit_lanes(uint32_t d, bool active) {
    uint32_t peers = __ballot_sync(0xffffffffu, active);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

constexpr int kChains = 2;                       // independent ranking chains per warp, half of its entries each
constexpr int kRuns = kWarps * kChains;
struct RankShared {
    uint16_t count[kRuns][kMaxRadix];           // entries so far of (run, digit); then the position of the first of them
    uint32_t half[kMaxRadix];                   // entries of the digit in the lower half of the runs
    uint32_t local_base[kMaxRadix];             // first staged position of the digit
    uint32_t warp_sums[32];
    uint32_t total;
};

// Position of every entry of the block in digit order (stable): pos[t] of entry (warp, t, lane).  A warp ranks its
// entries 32 at a time against its own running counts, with no counting round before, as two chains with counts of their
// own (a step's read of a count waits for the step before it; two chains hide that); the counts then are
// prefixed over the runs and the digits.  Ends with all threads past a barrier.
//
// kMasks: the lanes of a step that share a digit are found by each setting its bit in the digit's word of shared memory
// (`words`, kRuns * kMaxRadix of them; the atomic-or match known from radix sorts by ranking), not by eight ballots.  That is a third of
// the instructions and the shorter chain, but more shared-memory traffic: clearly faster while every block runs at once, slower where a
// great many wait for an SM.  By ballots / by masks, us: 10 x 512 slots 17.6 / 15.0; 0.9 M slots (450 small blocks) 49.6 / 46.0; 2.1 M
// (293 blocks) 42.8 / 38.9; then, in fourteens, 3.0 M (419) 56.2 / 54.7, 5.2 M (726) 86.1 / 84.0, 8.4 M (1171) 134.5 / 134.6, 12 M (1674)
// 194.1 / 201.8, 16.8 M (2341) 258.8 / 275.2; with 32-bit keys 3.0 M 85.8 / 81.6, 9.0 M 214.8 / 202.4, 16.8 M 373.7 / 366.3.  The line lies at
// the blocks that run at once, where masks win by a tenth whatever the keys.
template <bool kMasks, int kItems>
__device__ __forceinline__ void block_rank(const uint32_t (&keys)[kItems], int shift, uint32_t mask, uint32_t first, uint32_t n,
                                           RankShared& sh, uint32_t* words, uint32_t (&pos)[kItems]) {
    static_assert(kChains == 2 && kThreads == 2 * kMaxRadix, "two threads per digit below");
    constexpr int kSteps = kItems / kChains;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lanes_below = (1u << lane) - 1u;
    uint16_t* mine = sh.count[warp * kChains];
    uint32_t* same = words + warp * kChains * kMaxRadix;
    for (int d = lane; d < kChains * kMaxRadix / 2; d += 32) reinterpret_cast<uint32_t*>(mine)[d] = 0;
    if (kMasks) {
        for (int d = lane; d < kChains * kMaxRadix; d += 32) same[d] = 0;
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < kSteps; ++t) {
        uint32_t at[kChains], peers[kChains], before[kChains];
#pragma unroll
        for (int c = 0; c < kChains; ++c) {
            const int e = c * kSteps + t;
            const uint32_t d = digit_of(keys[e], shift, mask);
            at[c] = c * kMaxRadix + d;
            if (!kMasks) peers[c] = same_digit_lanes(d, first + e * 32 < n);
            else if (first + e * 32 < n) atomicOr(&same[at[c]], 1u << lane);
        }
        if (kMasks) __syncwarp();
#pragma unroll
        for (int c = 0; c < kChains; ++c) {
            if (kMasks) peers[c] = same[at[c]];
            before[c] = mine[at[c]];
            pos[c * kSteps + t] = before[c] + __popc(peers[c] & lanes_below);
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < kChains; ++c)
            if (first + (c * kSteps + t) * 32 < n && (peers[c] & lanes_below) == 0) {     // the lowest of them
                mine[at[c]] = static_cast<uint16_t>(before[c] + __popc(peers[c]));
                if (kMasks) same[at[c]] = 0;
            }
        __syncwarp();
    }
    __syncthreads();
    // thread (h, digit): the runs [16 h, 16 h + 16)
    const int digit = threadIdx.x & (kMaxRadix - 1), h = threadIdx.x / kMaxRadix;
    uint32_t c[kRuns / 2], run = 0;
#pragma unroll
    for (int w = 0; w < kRuns / 2; ++w) {
        c[w] = sh.count[h * (kRuns / 2) + w][digit];
        run += c[w];
    }
    if (h == 0) sh.half[digit] = run;
    __syncthreads();
    const uint32_t upper = block_exclusive_scan(h == 0 ? 0u : sh.half[digit] + run, sh.warp_sums, &sh.total);   // totals sit in the upper threads
    if (h == 1) sh.local_base[digit] = upper;
    __syncthreads();
    uint32_t at = sh.local_base[digit] + (h == 0 ? 0u : sh.half[digit]);
#pragma unroll
    for (int w = 0; w < kRuns / 2; ++w) {
        sh.count[h * (kRuns / 2) + w][digit] = static_cast<uint16_t>(at);
        at += c[w];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kItems; ++e) pos[e] += mine[(e / kSteps) * kMaxRadix + digit_of(keys[e], shift, mask)];
}

// Stable scatter of one pass: rank, put the entries into a shared-memory copy of the block's output in digit order, send
// that out (entry j of digit d lands at the global base of (d, block) + j - local base of d, so consecutive threads write
// consecutive addresses inside a digit's run instead of 32 different lines per warp instruction).
// kFirst: keys from the indices, values are the flat positions themselves.  kLast: keys are not written; the head of every
// run of equal keys lowers its row's row_ptr to its position.
// In the first pass with 16-bit keys a value is its position, so key and position inside the block share a staged word (139 -> 134 us
// for the whole sort, with fourteen entries a thread).
// What bounds it: instruction issue (0.5 a cycle and scheduler), shared-memory bank conflicts of the ranked accesses and latency, about
// a third each.  8.4 M slots, 32768 rows: 76 -> 52 us per pass.
template <typename KeyT, int kItems> constexpr int scatter_smem() {
    constexpr int kEntries = kThreads * kItems * static_cast<int>(4 + sizeof(KeyT)), kWords = kRuns * kMaxRadix * 4;
    return kEntries > kWords ? kEntries : kWords;      // staged entries; before them block_rank's words
}

template <typename KeyT, bool kFirst, bool kLast, int kItems, bool kMasks>
__global__ void __launch_bounds__(kThreads, 2)
scatter_kernel(const KeyT* __restrict__ keys_in, const int32_t* __restrict__ vals_in, const Source src, KeyT* __restrict__ keys_out,
               int32_t* __restrict__ vals_out, const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals, uint32_t n,
               int shift, uint32_t mask, int n_blocks, int32_t* __restrict__ row_ptr) {
    constexpr int kBlockItems = kThreads * kItems, kWarpItems = 32 * kItems;
    // in the first pass a value is its position: key and position inside the block share a word
    constexpr bool kPacked = kFirst && sizeof(KeyT) == 2;
    static_assert(kBlockItems <= 65536, "positions inside a block in 16 bits");
    extern __shared__ __align__(16) uint32_t staged[];
    int32_t* svals = reinterpret_cast<int32_t*>(staged);
    KeyT* skeys = reinterpret_cast<KeyT*>(staged + kBlockItems);
    __shared__ RankShared sh;
    __shared__ uint32_t out_base[kMaxRadix];      // global position of staged position 0 of the digit's run
    const int radix = static_cast<int>(mask) + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t block0 = blockIdx.x * kBlockItems;
    const uint32_t first = block0 + warp * kWarpItems + lane;
    smla::pdl_wait();
    smla::pdl_trigger();
    uint32_t keys[kItems], pos[kItems];
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * 32;
        if (kFirst) keys[t] = i < n ? static_cast<uint32_t>(__ldg(src.indices + i)) : 0u;
        else keys[t] = i < n ? keys_in[i] : 0u;
    }
    const uint32_t tot = threadIdx.x < radix ? totals[threadIdx.x] : 0u;
    const uint32_t blk = threadIdx.x < radix ? hist[static_cast<size_t>(threadIdx.x) * n_blocks + blockIdx.x] : 0u;
    if (kFirst) {
#pragma unroll
        for (int t = 0; t < kItems; ++t) keys[t] = src.key(first + t * 32, static_cast<int>(keys[t]));
    }
    const uint32_t digit0 = block_exclusive_scan(tot, sh.warp_sums, &sh.total);
    block_rank<kMasks>(keys, shift, mask, first, n, sh, staged, pos);
    if (threadIdx.x < radix) out_base[threadIdx.x] = digit0 + blk - sh.local_base[threadIdx.x];
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * 32;
        if (i < n) {
            if constexpr (kPacked) {
                staged[pos[t]] = keys[t] << 16 | (i - block0);
            } else {
                skeys[pos[t]] = static_cast<KeyT>(keys[t]);
                svals[pos[t]] = kFirst ? static_cast<int32_t>(i) : __ldg(vals_in + i);
            }
        }
    }
    __syncthreads();
    const uint32_t count = min(n - block0, static_cast<uint32_t>(kBlockItems));
#pragma unroll 8
    for (uint32_t j = threadIdx.x; j < count; j += kThreads) {
        const uint32_t key = kPacked ? staged[j] >> 16 : skeys[j];
        const uint32_t at = out_base[digit_of(key, shift, mask)] + j;
        vals_out[at] = kPacked ? static_cast<int32_t>(block0 + (staged[j] & 0xffffu)) : svals[j];
        if (!kLast) keys_out[at] = static_cast<KeyT>(key);
        else if (j == 0 || (kPacked ? staged[j - 1] >> 16 : skeys[j - 1]) != key) atomicMin(row_ptr + key, static_cast<int32_t>(at));
    }
}

// Where many blocks of rows (kMaxLook) are to be filled in: the first run of each block of rows, ...
__global__ void __launch_bounds__(kRowTile)
row_min_kernel(const int32_t* __restrict__ heads, int32_t* __restrict__ first, int32_t s_kv) {
    __shared__ int warp_min[32];
    smla::pdl_wait();
    smla::pdl_trigger();
    const int64_t r = static_cast<int64_t>(blockIdx.x) * kRowTile + threadIdx.x;
    const int m = __reduce_min_sync(0xffffffffu, r <= s_kv ? heads[r] : INT_MAX);
    if ((threadIdx.x & 31) == 0) warp_min[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        const int all = __reduce_min_sync(0xffffffffu, warp_min[threadIdx.x]);
        if (threadIdx.x == 0) first[blockIdx.x] = all;
    }
}
// ... and of each block and all behind it (one block of threads, from the end).
__global__ void __launch_bounds__(1024)
suffix_min_kernel(int32_t* __restrict__ first, int32_t n_blocks) {
    __shared__ int warp_min[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    smla::pdl_wait();
    smla::pdl_trigger();
    int carry = INT_MAX;
    for (int base = (n_blocks - 1) / 1024 * 1024; base >= 0; base -= 1024) {
        const int i = base + threadIdx.x;
        int v = i < n_blocks ? first[i] : INT_MAX;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int down = __shfl_down_sync(0xffffffffu, v, o);
            if (lane + o < 32) v = min(v, down);
        }
        if (lane == 0) warp_min[warp] = v;
        __syncthreads();
        const int mine = warp_min[lane];
        const int behind = __reduce_min_sync(0xffffffffu, lane > warp ? mine : INT_MAX);
        if (i < n_blocks) first[i] = min(min(v, behind), carry);
        carry = min(carry, __reduce_min_sync(0xffffffffu, mine));
        __syncthreads();
    }
}
// Rows without a slot take the next row's position: suffix minimum of the run heads (they ascend with the row).  first: what
// suffix_min_kernel left, or null.
__global__ void __launch_bounds__(kRowTile)
row_ptr_kernel(const int32_t* __restrict__ heads, const int32_t* __restrict__ first, int32_t* __restrict__ row_ptr, int32_t n, int32_t s_kv) {
    __shared__ int warp_min[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    smla::pdl_wait();
    smla::pdl_trigger();
    const int r = blockIdx.x * kRowTile + threadIdx.x;
    int v = r <= s_kv ? heads[r] : INT_MAX;
    // the first run behind this block's rows
    int later = INT_MAX;
    if (first) {
        if (blockIdx.x + 1 < gridDim.x) later = first[blockIdx.x + 1];
    } else {
        for (int base = (blockIdx.x + 1) * kRowTile; base <= s_kv; base += kRowTile) {
            const int i = base + threadIdx.x;
            const int h = i <= s_kv ? heads[i] : INT_MAX;
            if (__syncthreads_or(h != INT_MAX)) {
                later = h;
                break;
            }
        }
    }
    later = __reduce_min_sync(0xffffffffu, later);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int down = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o < 32) v = min(v, down);
    }
    __shared__ int later_min[32];
    if (lane == 0) {
        warp_min[warp] = v;
        later_min[warp] = later;
    }
    __syncthreads();
    int m = min(later_min[lane], n);
    if (lane > warp) m = min(m, warp_min[lane]);
    m = __reduce_min_sync(0xffffffffu, m);
    if (r <= s_kv) row_ptr[r] = min(v, m);
}

// ---- direct form: a counter per kv row in shared memory, no sort ----------------------------------------------------------
// The queries are cut into groups of consecutive ones, one block each.  A row's word in shared memory holds the position in `entries` of
// the row's next slot in the group; slots without a valid row have a word of their own, behind the rows'.  place_kernel goes through its
// group's slots in batches, each warp through its piece of a batch.  The lanes of a warp that name the same row find each other by
// marks in shared memory, the first of them takes positions for all of them by adding their number to the row's word, and the warps do
// this one after the other, in the order of their pieces (a named barrier hands the turn on).  So the order holds whichever rows the
// slots name and however often, and nothing but these additions is in turn: loads, marks and stores of other warps go on meanwhile.  The
// words start at the rows' positions: group_count_kernel counts every group's slots per row, group_scan_kernel turns these [group][row]
// counts into positions.
// What bounds it: place_kernel (three quarters of 75.8 us with 8.4 M slots and 32768 rows; the sort: 135), its turns, and its stores of four bytes
// all over `entries`, a sector each: where all slots name one row and the stores are whole lines 61.5.  Pieces of 512 slots 77.1, of 384
// 74.5, of 256 76.8; where a group has 4096 slots 24.3, 23.5, 22.7 (these of 320: 75.7 and 23.2).  A bit per query in the row's word, a barrier
// between phases, and slots that repeat a row placed one after the other: 87, with random rows 151, with two rows 475.  Lanes of a row found
// by sixteen ballots 98, by match.any 98; additions under a predicate, not sent nowhere, 122: the warp waits for each.
constexpr int kPlaceWarps = kPlaceThreads / 32, kPiece = kBatch / kPlaceWarps;
static_assert(kPlaceWarps <= 16, "as many warps as named barriers");
constexpr int kMarks = 512;
constexpr int kScanThreads = 512, kScanRows = 64, kScanSegs = kScanThreads / kScanRows;      // a block of group_scan_kernel: rows x pieces of the groups

// counts[group][row] of the group's slots; row s_kv: its unused ones.  `entries` is cleared, so that its lines are in the L2, whole, when
// place_kernel stores four bytes at a time into them: on lines that are not there these stores fetch their sectors (8.4 M slots, buffers that
// change from call to call: 81.2 us without the clearing, 79.3 with it; with an L2 full of other data 109.6 and 87.0; done by
// group_scan_kernel, whose blocks are few with few rows, 1 us more on 32768 rows and 8 on 8192).  Four slots a load: 2.5 us less, with smaller
// blocks of group_scan_kernel.
__global__ void __launch_bounds__(kCountThreads, 1)
group_count_kernel(const Source src, uint32_t* __restrict__ counts, int32_t* __restrict__ entries, int s_q, int per_group, int rows_pad) {
    extern __shared__ __align__(16) uint32_t cnt[];
    for (int i = threadIdx.x; i < rows_pad / 4; i += kCountThreads) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
    smla::pdl_wait();
    smla::pdl_trigger();
    __syncthreads();
    const uint32_t q0 = blockIdx.x * per_group, q1 = min(q0 + per_group, static_cast<uint32_t>(s_q));
    const uint32_t begin = q0 * src.topk, end = q1 * src.topk;
    uint32_t none = 0;
    auto count = [&](uint32_t i, int idx) {
        const uint32_t key = src.key(i, idx);
        if (key != static_cast<uint32_t>(src.s_kv)) atomicAdd(&cnt[key], 1u);
        else ++none;
    };
    // four slots a load from the first 16-byte boundary on; what lies before and behind, one by one
    const uint32_t head = min(end - begin, static_cast<uint32_t>((16 - (reinterpret_cast<uintptr_t>(src.indices + begin) & 15)) & 15) / 4);
    const uint32_t body = begin + head, vectors = (end - body) / 4, tail = body + 4 * vectors;
    const int4* in = reinterpret_cast<const int4*>(src.indices + body);
    const bool wide = (reinterpret_cast<uintptr_t>(entries + body) & 15) == 0;
    constexpr int kLoads = 4;
    int4 next[kLoads];
    auto load = [&](uint32_t v0) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k) next[k] = v0 + k * kCountThreads < vectors ? __ldg(in + v0 + k * kCountThreads) : make_int4(-1, -1, -1, -1);
    };
    load(threadIdx.x);
    if (threadIdx.x < head) {
        entries[begin + threadIdx.x] = 0;
        count(begin + threadIdx.x, __ldg(src.indices + begin + threadIdx.x));
    }
    if (tail + threadIdx.x < end) {
        entries[tail + threadIdx.x] = 0;
        count(tail + threadIdx.x, __ldg(src.indices + tail + threadIdx.x));
    }
    for (uint32_t v0 = threadIdx.x; v0 < vectors; v0 += kLoads * kCountThreads) {
        int4 idx[kLoads];
#pragma unroll
        for (int k = 0; k < kLoads; ++k) idx[k] = next[k];
        load(v0 + kLoads * kCountThreads);
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const uint32_t v = v0 + k * kCountThreads, i = body + 4 * v;
            if (v >= vectors) continue;
            if (wide) {
                *reinterpret_cast<int4*>(entries + i) = make_int4(0, 0, 0, 0);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) entries[i + e] = 0;
            }
            count(i, idx[k].x);
            count(i + 1, idx[k].y);
            count(i + 2, idx[k].z);
            count(i + 3, idx[k].w);
        }
    }
    none = __reduce_add_sync(0xffffffffu, none);
    if ((threadIdx.x & 31) == 0 && none) atomicAdd(&cnt[src.s_kv], none);
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(counts + static_cast<size_t>(blockIdx.x) * rows_pad);
    for (int i = threadIdx.x; i < rows_pad / 4; i += kCountThreads) out[i] = reinterpret_cast<uint4*>(cnt)[i];
}

// counts[group][row] -> position of the group's first entry of the row, counted from the first entry of the block's rows; totals[block]:
// entries of the block's rows.  "Row" s_kv, the unused slots, is the last one and so lands behind all others.
__global__ void __launch_bounds__(kScanThreads, 2)
group_scan_kernel(uint32_t* __restrict__ counts, uint32_t* __restrict__ totals, int n_groups, int rows_pad) {
    constexpr int kPer = (kMaxGroups + kScanSegs - 1) / kScanSegs;
    __shared__ uint32_t seg_sum[kScanSegs][kScanRows];
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t total;
    const int r = threadIdx.x % kScanRows, seg = threadIdx.x / kScanRows, row = blockIdx.x * kScanRows + r;
    smla::pdl_wait();
    smla::pdl_trigger();
    uint32_t* mine = counts + static_cast<size_t>(seg * kPer) * rows_pad + row;
    const int n = row < rows_pad ? min(kPer, n_groups - seg * kPer) : 0;
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) c[i] = i < n ? mine[static_cast<size_t>(i) * rows_pad] : 0u;
#pragma unroll
    for (int i = 0; i < kPer; ++i) sum += c[i];
    seg_sum[seg][r] = sum;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int s = 0; s < kScanSegs; ++s) {
        const uint32_t x = seg_sum[s][r];
        if (s < seg) before += x;
        all += x;
    }
    // rows before this one: segment 0's threads hold one row each
    const uint32_t at = block_exclusive_scan(seg == 0 ? all : 0u, warp_sums, &total);
    if (seg == 0) seg_sum[0][r] = at;
    __syncthreads();
    before += seg_sum[0][r];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        if (i < n) mine[static_cast<size_t>(i) * rows_pad] = before;
        before += c[i];
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// The turn: a barrier for the warp that gives it and the one that takes it, with the taker's number.  What the giver has done in shared
// memory is there for the taker.
__device__ __forceinline__ void take_turn(int warp) { asm volatile("bar.sync %0, 64;" ::"r"(warp) : "memory"); }
__device__ __forceinline__ void give_turn(int warp) { asm volatile("bar.arrive %0, 64;" ::"r"(warp) : "memory"); }

__global__ void __launch_bounds__(kPlaceThreads, 1)
place_kernel(const Source src, const uint32_t* __restrict__ counts, const uint32_t* __restrict__ totals, int32_t* __restrict__ row_ptr,
             int32_t* __restrict__ entries, int s_q, int per_group, int rows_pad, int n_scan_blocks) {
    extern __shared__ __align__(16) uint32_t word[];
    static_assert(kPlaceRows / kScanRows + 1 <= 2 * kPlaceThreads, "two a thread");
    __shared__ uint32_t base[2 * kPlaceThreads], warp_sums[32], total, nowhere[32];
    __shared__ uint8_t marks[kPlaceWarps][kMarks];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t q0 = blockIdx.x * per_group, q1 = min(q0 + per_group, static_cast<uint32_t>(s_q));
    const uint32_t begin = q0 * src.topk, end = q1 * src.topk;
    smla::pdl_wait();
    smla::pdl_trigger();
    int next[kPlaceItems];                       // the next piece's slots
    auto load = [&](uint32_t first) {
#pragma unroll
        for (int k = 0; k < kPlaceItems; ++k) next[k] = first + 32 * k < end ? __ldg(src.indices + first + 32 * k) : -1;
    };
    uint32_t first = begin + warp * kPiece + lane;
    load(first);
    const int i0 = 2 * threadIdx.x, i1 = i0 + 1;
    const uint32_t t0 = i0 < n_scan_blocks ? totals[i0] : 0u, t1 = i1 < n_scan_blocks ? totals[i1] : 0u;
    base[i0] = block_exclusive_scan(t0 + t1, warp_sums, &total);
    base[i1] = base[i0] + t0;
    __syncthreads();
    const uint4* in = reinterpret_cast<const uint4*>(counts + static_cast<size_t>(blockIdx.x) * rows_pad);
#pragma unroll 8
    for (int i = threadIdx.x; i < rows_pad / 4; i += kPlaceThreads) {
        const uint4 v = __ldcg(in + i);
        const uint32_t b = base[i / (kScanRows / 4)];
        reinterpret_cast<uint4*>(word)[i] = make_uint4(v.x + b, v.y + b, v.z + b, v.w + b);
    }
    // row_ptr: where group 0's entries of the row begin; every block writes its share
    for (int r = blockIdx.x * kPlaceThreads + threadIdx.x; r <= src.s_kv; r += gridDim.x * kPlaceThreads)
        row_ptr[r] = static_cast<int32_t>(__ldcg(counts + r) + base[r / kScanRows]);
    __syncthreads();
    // (a warp's piece has the number of its turn)
    const uint32_t n_turns = (end - begin + kPiece - 1) / kPiece;
    for (uint32_t turn = warp; turn < n_turns; turn += kPlaceWarps, first += kBatch) {
        uint32_t who[kPlaceItems];               // its first lane, the lanes of the row before this one, all of them: 8 bits each; 0: no slot
        uint32_t* at[kPlaceItems];
#pragma unroll
        for (int k = 0; k < kPlaceItems; ++k) {
            const uint32_t i = first + 32 * k;
            const bool active = i < end;
            const uint32_t row = src.key(i, next[k]);
            // Every lane leaves its number at its row's mark.  Where it finds another's, that lane has the same row, or one of the same mark.
            uint8_t* mark = &marks[warp][row % kMarks];
            if (active) *mark = static_cast<uint8_t>(lane);
            __syncwarp();
            uint32_t peers = 1u << lane;
            for (uint32_t rest = __ballot_sync(0xffffffffu, active && *mark != lane); rest;) {
                const uint32_t lead = __shfl_sync(0xffffffffu, row, __ffs(rest) - 1);
                const uint32_t same = __ballot_sync(0xffffffffu, active && row == lead);
                if (row == lead) peers = same;
                rest &= ~same;
            }
            who[k] = !active ? 0u : (__ffs(peers) - 1) | __popc(peers & below) << 8 | __popc(peers) << 16;
            at[k] = active && (peers & below) == 0 ? &word[row] : &nowhere[lane];
            __syncwarp();
        }
        if (turn + kPlaceWarps < n_turns) load(first + kBatch);
        uint32_t pos[kPlaceItems];
        if (turn) take_turn(warp);
#pragma unroll
        for (int k = 0; k < kPlaceItems; ++k) {
            pos[k] = atomicAdd(at[k], who[k] >> 16);
            __syncwarp();                            // (in this order, too)
        }
        if (turn + 1 < n_turns) give_turn((warp + 1) % kPlaceWarps);
#pragma unroll
        for (int k = 0; k < kPlaceItems; ++k) {
            const uint32_t p = __shfl_sync(0xffffffffu, pos[k], who[k] & 31u) + (who[k] >> 8 & 31u);
            if (who[k]) entries[p] = static_cast<int32_t>(first + 32 * k);
        }
    }
}

// ---- at most one block's worth of slots: every pass in shared memory -----------------------------------------------------
template <typename KeyT>
__global__ void __launch_bounds__(kThreads, 1)
small_sort_kernel(const Source src, KeyT* __restrict__ keys_out, int32_t* __restrict__ vals_out, uint32_t n, int passes, int digit_bits) {
    constexpr int kItems = kItemsSmall, kBlockItems = kSmallInput, kWarpItems = 32 * kItems;
    extern __shared__ __align__(16) uint32_t staged[];
    int32_t* svals = reinterpret_cast<int32_t*>(staged);
    KeyT* skeys = reinterpret_cast<KeyT*>(staged + kBlockItems);
    __shared__ RankShared sh;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = warp * kWarpItems + lane;
    const uint32_t mask = (1u << digit_bits) - 1u;
    smla::pdl_wait();
    smla::pdl_trigger();
    uint32_t keys[kItems], vals[kItems], pos[kItems];
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * 32;
        keys[t] = i < n ? src.key(i, __ldg(src.indices + i)) : 0u;
        vals[t] = i;
    }
    for (int pass = 0; pass < passes; ++pass) {
        block_rank<true>(keys, pass * digit_bits, mask, first, n, sh, staged, pos);
#pragma unroll
        for (int t = 0; t < kItems; ++t)
            if (first + t * 32 < n) {
                skeys[pos[t]] = static_cast<KeyT>(keys[t]);
                svals[pos[t]] = static_cast<int32_t>(vals[t]);
            }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kItems; ++t) {
            const uint32_t i = first + t * 32;
            keys[t] = i < n ? skeys[i] : 0u;
            vals[t] = i < n ? static_cast<uint32_t>(svals[i]) : 0u;
        }
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < kItems; ++t) {
        const uint32_t i = first + t * 32;
        if (i < n) {
            keys_out[i] = static_cast<KeyT>(keys[t]);
            vals_out[i] = static_cast<int32_t>(vals[t]);
        }
    }
}
// row_ptr[r] = first position in the sorted keys whose key is >= r, for r in [0, s_kv] (a few thousand keys: they sit in L1).
template <typename KeyT>
__global__ void __launch_bounds__(256)
small_row_ptr_kernel(const KeyT* __restrict__ sorted_keys, int32_t* __restrict__ row_ptr, int32_t n, int32_t s_kv) {
    smla::pdl_wait();
    smla::pdl_trigger();
    const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r > s_kv) return;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sorted_keys[mid] < static_cast<uint32_t>(r)) lo = mid + 1;
        else hi = mid;
    }
    row_ptr[r] = lo;
}

}  // namespace inv
