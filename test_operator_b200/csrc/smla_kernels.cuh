// Device kernels of the sparse MLA backward for sm_100a.
//
// The backward of one query token is a chain of five contractions around a softmax-gradient
// step.  It is split into four kernels that hand bf16 S / dS through a scratch buffer:
//
//   prep       Delta[q,h] = sum_j O[q,h,j] * dO[q,h,j], slots in use per query   (HBM-bound)
//   recompute  P^T = K_g Q^T, dP^T = V_g dO^T  (tcgen05, keys on the M axis),
//              S = exp2(P*scale*log2e - lse), dS = S*(dP - Delta)*scale -> bf16 scratch; dKV cleared
//   dkv        dKV^T[d, key] = dO^T S + Q^T dS (tcgen05, d on the M axis), then one coalesced
//              fp32 reduction per (key, 32 consecutive d) straight from TMEM registers
//   dq         dQ[head, d] = dS^T K_g (tcgen05, heads on the M axis, d on N) accumulated over all keys
//
// The forward (o, lse for the same indices) is one kernel of its own, smla_fwd_kernel: heads on the M axis, an online
// softmax between the two contractions, nothing but o and lse written.
//
// Heads are padded to HP = 64 or 128, so h_q = 16 / 64 / 128 use the same code.  Gathered kv rows and
// Q / dO are held as 128-byte-swizzled [rows x 64 bf16] chunks (kv rows by 16-byte cp.async, Q / dO by
// TMA); S / dS tiles arrive by TMA in the no-swizzle core-matrix order.  A chunk is read K-major or
// MN-major by choosing the descriptor, never by moving data.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cstdint>

#include "sm100_ptx.cuh"

namespace smla {

constexpr unsigned kPollSleepNs = 32;   // back-off of producer / consumer warps waiting on mbarriers
constexpr int kDQK = 576;
constexpr int kDV = 512;
constexpr int kQChunks = kDQK / 64;   // 9 column chunks of 64
constexpr int kVChunks = kDV / 64;    // 8
constexpr int kDqChunks = 3;          // dq: three d-parts of three column chunks (192 columns) each

struct KParams {
    const __nv_bfloat16* kv;  // [s_kv, 576]
    const int32_t* indices;   // [s_q, topk]
    const float* lse;         // [s_q, h_q]
    const float* delta;       // [s_q, h_q]
    const int* n_used;        // [s_q] slots up to and including the query's last valid one
    __nv_bfloat16* s_scr;     // [q_chunk][HP/8 head blocks][topk_pad keys][8 heads], see scratch_offset
    __nv_bfloat16* ds_scr;    // likewise
    float* dKV;               // [s_kv, 576]
    float* staging;           // reproducible mode: [q_chunk][topk_pad slots][576] fp32, one row per slot
    __nv_bfloat16* dQ;        // [s_q, h_q, 576]
    // forward only
    float* lse_out;           // [s_q, h_q]
    float lse_out_mult;       // 1 (base 2) or ln 2 (natural log)
    float* part_o;            // partial results of queries spread over several clusters: [slot][HP][512]
    float2* part_ml;          // [slot][HP] {reference of the exponentials (log2), sum}
    int4* range_q;            // [clusters] {first query of the cluster's range, position of that query's first tile, tiles of the launch}
    __nv_bfloat16* gout;      // [s_q, h_q, 512] o (forward only)
    int* g_err;
    int q0;                   // first query (global row) of this launch
    int nq;                   // queries in this launch
    int scr0;                 // scratch row of query q0 (a launch may cover a part of the queries a scratch holds)
    int s_q, s_kv, h_q, topk, topk_pad;
    float sm_scale, scale_log2e, lse_mult;
    int q_start, causal;
    const int4* qmeta;        // optional per query {first kv row of its sequence, kv rows of its sequence,
                              // position for the causal rule, top-k slots in use}; null: one sequence
    long long wait_limit;     // cycles a bounded wait may take
    int early_start;          // dkv, dq: launched behind the trigger of the kernel before in the same call (see there)
    int every_slot;           // > 0 (topk): count every slot of every query as used and do not read n_used (slots_used)
    size_t clear_bytes;       // recompute: how much of dKV it clears (all or nothing)
    // recompute without a prep kernel in front (own_prep, only with every_slot): O, dO, and Delta for calls of single stages
    int own_prep;
    const uint4 *o_in, *do_in;
    float* delta_out;
};

// What a query may attend to: rows [kv_base, kv_base + kv_len) of kv, index values relative to kv_base.
struct QMeta {
    int kv_base, kv_len, q_pos, topk_len;
};
__device__ __forceinline__ QMeta load_qmeta(const KParams& p, int q_global) {
    if (p.qmeta) {
        const int4 m = __ldg(p.qmeta + q_global);
        return QMeta{m.x, m.y, m.z, m.w};
    }
    return QMeta{0, p.s_kv, p.q_start + q_global, p.topk};
}
__device__ __forceinline__ bool slot_valid(int idx, int key, const QMeta& m, const KParams& p) {
    return key < m.topk_len && idx >= 0 && idx < m.kv_len && m.kv_base + idx < p.s_kv && (!p.causal || idx <= m.q_pos);
}
// kv row a slot gathers from, -1 for one that takes no part (nothing is read then, zeros land).  The whole rule, not the range alone:
// the contractions over keys (forward, dQ) multiply a masked slot's row by an exact 0, and a masked slot may name a row that holds NaN or
// an infinity (one of a cache that has not been written yet).
__device__ __forceinline__ int gather_row(int idx, int key, const QMeta& m, const KParams& p) {
    return slot_valid(idx, key, m, p) ? m.kv_base + idx : -1;
}
// The same by the range alone, for the recompute kernel: there a row meets its own slot's S and dS only, which are masked bit by bit.
// (64 queries x 16 heads x top-k 64 19.57 us a call with the whole rule, 19.45 so.)
__device__ __forceinline__ int gather_row_in_range(int idx, const QMeta& m, const KParams& p) {
    const int row = m.kv_base + idx;
    return idx >= 0 && idx < m.kv_len && row < p.s_kv ? row : -1;
}
// After a bounded wait has given up: let this thread's own cp.async land and leave in-flight TMA loads (they
// depend on nothing and complete within microseconds) the time to land before the CTA gives up its shared memory.
__device__ __forceinline__ void abort_wind_down(volatile int* s_abort) {
    if (*s_abort) {
        cp_async_wait_all();
        for (int i = 0; i < 32; ++i) __nanosleep(1000);
    }
}

// S / dS scratch of one query: [HP/8 head blocks][topk_pad keys][8 heads] bf16, i.e. the UMMA core matrices
// (8 keys x 16 bytes) of the no-swizzle layouts stored one after another.  A warp of the recompute kernel holds 32
// consecutive keys, so each of its stores writes 512 consecutive bytes (four full cache lines) instead of 32
// scattered sectors; the consumers fetch [head block][keys of a tile][8 heads] with one TMA box of 512-byte rows.
__device__ __forceinline__ size_t scratch_offset(int key, int head, int topk_pad) {
    return (static_cast<size_t>(head >> 3) * topk_pad + key) * 8 + (head & 7);
}


// error codes recorded by bounded waits: 100*kernel + site
enum { kErrRecompute = 100, kErrDkv = 200, kErrDq = 300, kErrFwd = 400 };

__device__ __forceinline__ float dot8_bf16(const uint4& a, const uint4& b, float acc) {
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 x = __bfloat1622float2(pa[k]), y = __bfloat1622float2(pb[k]);
        acc = fmaf(x.x, y.x, acc);
        acc = fmaf(x.y, y.y, acc);
    }
    return acc;
}
// read once, so first out of the caches
__device__ __forceinline__ uint4 ld_stream_v4(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
    return v;
}

// =============================================================================================
// Delta = rowsum(O * dO).  One warp per (query, head) row of 512 bf16; each lane reads 2 x 16 B
// of each tensor, so a warp reads 2 x 1 KB fully coalesced.
// =============================================================================================
__global__ void __launch_bounds__(256) smla_delta_kernel(const uint4* __restrict__ O, const uint4* __restrict__ dO,
                                                         float* __restrict__ delta, int n_rows) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n_rows) return;
    const uint4* o = O + static_cast<size_t>(row) * (kDV / 8);
    const uint4* g = dO + static_cast<size_t>(row) * (kDV / 8);
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) acc = dot8_bf16(__ldg(o + lane + 32 * i), __ldg(g + lane + 32 * i), acc);
    acc = warp_sum(acc);
    if (lane == 0) delta[row] = acc;
}

// =============================================================================================
// prep: everything the three tensor-core kernels need that is not a contraction, in one launch.
//   block b < s_q   Delta of query b's rows (backward), and n_used[b]: the slots up to the query's last valid one (early tokens of a
//                   causal sequence use a fraction of their top-k, the rest are out-of-range values at the end)
// Bound by HBM: O, dO and the indices read once.
// =============================================================================================
constexpr int kSmCount = 148;           // of a B200: for splits of small grids
constexpr int kWorkTileKeys = 256;      // granularity of the work ranges: what the recompute kernel does per accumulator
constexpr int kPrepThreads = 256;

// Sum of one value per thread over the lower-numbered threads of the block; *total: over all.  warp_sums: 32 words.
__device__ __forceinline__ int block_exclusive_sum(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < n_warps; ++w) {
        const int x = warp_sums[w];
        if (w < warp) before += x;
        all += x;
    }
    __syncthreads();
    *total = all;
    return before + incl - v;
}

// Delta of `kRows` (query, head) rows, row[i] of [rows, 512] each: 4 kRows 16-byte loads of a lane in flight.  Returned in every lane.
template <int kRows>
__device__ __forceinline__ void delta_rows(const uint4* O, const uint4* dO, const size_t (&row)[kRows], float (&out)[kRows]) {
    const int lane = threadIdx.x & 31;
    uint4 a[2 * kRows], b[2 * kRows];
#pragma unroll
    for (int i = 0; i < 2 * kRows; ++i) {
        const size_t at = row[i >> 1] * (kDV / 8) + 32 * (i & 1) + lane;
        a[i] = ld_stream_v4(O + at);
        b[i] = ld_stream_v4(dO + at);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) out[i] = warp_sum(dot8_bf16(a[2 * i + 1], b[2 * i + 1], dot8_bf16(a[2 * i], b[2 * i], 0.f)));
}
__global__ void __launch_bounds__(kPrepThreads)
smla_prep_kernel(const uint4* __restrict__ O, const uint4* __restrict__ dO, float* __restrict__ delta,
                 int* __restrict__ n_used, int head_parts, const KParams p) {
    __shared__ int red[kPrepThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarps = kPrepThreads / 32;
    pdl_wait();                   // (nothing above touches memory another kernel of the stream may still use)
    pdl_trigger();
    // with few queries several blocks share one query's heads; the first of them also looks at its indices
    const int q = blockIdx.x / head_parts, hp = blockIdx.x % head_parts;
    if (q < p.s_q && hp == 0) {
        const QMeta qm = load_qmeta(p, q);
        int last = -1;
        for (int key = threadIdx.x; key < p.topk; key += kPrepThreads)
            if (slot_valid(__ldg(p.indices + static_cast<size_t>(q) * p.topk + key), key, qm, p)) last = key;
        last = __reduce_max_sync(0xffffffffu, last);
        if (lane == 0) red[warp] = last;
    }
    __syncthreads();
    if (threadIdx.x == 0 && q < p.s_q && hp == 0) {
        int m = red[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) m = max(m, red[w]);
        n_used[q] = m + 1;
    }
    if (O == nullptr) {                          // forward, or a backward that is given Delta
        if (q >= p.s_q || p.gout == nullptr) return;
        int m = -1;                              // a query without a valid slot is in nobody's range
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = max(m, red[w]);
        if (m < 0) {
            uint4* o = reinterpret_cast<uint4*>(p.gout) + static_cast<size_t>(q) * p.h_q * (kDV / 8);
            for (int i = threadIdx.x; i < p.h_q * (kDV / 8); i += kPrepThreads) o[i] = make_uint4(0, 0, 0, 0);
            for (int h = threadIdx.x; h < p.h_q; h += kPrepThreads)
                p.lse_out[static_cast<size_t>(q) * p.h_q + h] = __int_as_float(0x7f800000) * p.lse_out_mult;
        }
    } else if (q < p.s_q) {
        const size_t row0 = static_cast<size_t>(q) * p.h_q;
        const int h_end = p.h_q * (hp + 1) / head_parts;
        for (int h = p.h_q * hp / head_parts + warp; h < h_end; h += 2 * kWarps) {
            const int h2 = h + kWarps < h_end ? h + kWarps : h;
            const size_t row[2] = {row0 + h, row0 + h2};
            float d[2];
            delta_rows(O, dO, row, d);
            if (lane == 0) {
                delta[row[0]] = d[0];
                delta[row[1]] = d[1];
            }
        }
    }
}

// Per-query table for packed sequences (KParams::qmeta) from a table of sequences that travels in the kernel's parameters:
// no host-to-device copy, no synchronisation.  One launch covers kMetaSeqs sequences.
constexpr int kMetaSeqs = 128;
struct MetaTable {
    int q0[kMetaSeqs + 1];        // first query row of each sequence, then the end of the last one
    int kv0[kMetaSeqs], kv_len[kMetaSeqs];
};
__global__ void __launch_bounds__(256) smla_query_meta_kernel(int4* __restrict__ meta, const __grid_constant__ MetaTable t, int n_seq,
                                                              int pos0, int topk, const int* __restrict__ topk_length) {
    const int q = t.q0[0] + static_cast<int>(blockIdx.x) * 256 + static_cast<int>(threadIdx.x);
    if (q >= t.q0[n_seq]) return;
    int lo = 0, hi = n_seq - 1;                       // the last sequence that starts at or before q
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (t.q0[mid] <= q) lo = mid;
        else hi = mid - 1;
    }
    const int used = topk_length ? min(max(__ldg(topk_length + q), 0), topk) : topk;
    meta[q] = make_int4(t.kv0[lo], t.kv_len[lo], pos0 + q - t.q0[lo], used);
}

// ---- work ranges of the persistent kernels ---------------------------------------------------------------------------
// The 256-key tiles of a launch's queries, one after the other (a query has ceil(n_used / 256) of them), are cut into as
// many equal contiguous ranges as there are clusters: every cluster gets the same number of tiles (4096 queries of eight
// tiles over 74 clusters as whole queries would be 56 queries for some and 55 for the others), a few long queries
// spread over the whole chip, and tiles without a valid slot do not exist.  kMul: tiles of 256 / kMul keys.
//
// In a call whose queries have no more tiles than there are clusters no cluster has more than one tile (the dKV kernel, which cuts
// ranges of 128 keys, up to two of its own), and the kernels that go by these ranges take as long as one tile takes, whether or not
// some of the tiles are empty.  There the ranges are cut as if every slot
// were in use (every_slot): nothing has to look at the indices first, which saves both directions their prep kernel (own_prep in the
// backward).  From the next tile on some cluster has two, and an empty tile would cost as much as a full one.
// The dQ kernel, where a CTA goes through a query's tiles, does work on empty ones.  128 heads, with a prep kernel / so, us:
//   8 queries x top-k 2048, slots in use   2048          700           100           1
//   forward                                25.6 / 20.2   22.7 / 20.3   18.6 / 17.8   19.2 / 17.8
//   backward                               45.0 / 35.9   39.4 / 34.6   32.1 / 33.0   28.4 / 32.8
// The last two of the backward are what it costs.  A dQ kernel that looked for the last valid slot first took 32.1 and 31.8 there, and
// 36.9 with all in use (37 queries x 512 31.1 -> 31.8).
__device__ __forceinline__ int slots_used(const KParams& p, int q) { return p.every_slot ? p.every_slot : __ldcg(p.n_used + q); }
struct WorkRange {
    int begin, end;               // positions among the launch's tiles
    int q, lo;                    // the query `begin` lies in; position of its first tile
};
template <int kKeys = kWorkTileKeys> __device__ __forceinline__ int work_tiles(int n_used) { return (n_used + kKeys - 1) / kKeys; }
__device__ __forceinline__ int range_start(int n_tiles, int cluster, int n_clusters) {     // n_tiles * cluster / n_clusters in 32 bits
    const uint32_t n = n_tiles, c = cluster, m = n_clusters;
    return static_cast<int>(n / m * c + n % m * c / m);
}
// Which range is this cluster's; called by the whole block, which passes a barrier before it reads *out.  Every block adds up
// the slot counts itself (a few per thread: 8192 queries are 32 KB out of L2, all in flight at once), so that the ranges need
// no prefix sum made by a kernel before and no counter that would have to survive from launch to launch.
// scratch: one word of shared memory per warp.  Returns, in the one thread that wrote *out, the launch's tiles; -1 in the others.
template <int kThreads, int kKeys = kWorkTileKeys>
__device__ __forceinline__ int find_range(const KParams& p, int cluster, int n_clusters, int* scratch, WorkRange* out) {
    if (p.every_slot) {
        if (threadIdx.x != 0) return -1;
        const int tiles = work_tiles<kKeys>(p.every_slot), total = p.nq * tiles, begin = range_start(total, cluster, n_clusters);
        *out = WorkRange{begin, range_start(total, cluster + 1, n_clusters), p.q0 + begin / tiles, begin / tiles * tiles};
        return total;
    }
    const int* used = p.n_used + p.q0;
    const int per = (p.nq + kThreads - 1) / kThreads;          // consecutive queries of a thread
    const int i0 = min(static_cast<int>(threadIdx.x) * per, p.nq), i1 = min(i0 + per, p.nq);
    int sum = 0, total;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) sum += work_tiles<kKeys>(__ldcg(used + i));
    int lo = block_exclusive_sum(sum, scratch, &total);
    const int begin = range_start(total, cluster, n_clusters);
    if (total == 0 ? threadIdx.x != 0 : begin < lo || begin >= lo + sum) return -1;
    int q = i0;
    if (total > 0) {
        for (int n; begin >= lo + (n = work_tiles<kKeys>(__ldcg(used + q))); ++q) lo += n;
    }
    *out = WorkRange{begin, range_start(total, cluster + 1, n_clusters), p.q0 + q, lo};
    return total;
}
// Broadcast, so that the bounds of the loops around the UMMAs are warp-uniform to the compiler as well (see elect_one).
__device__ __forceinline__ WorkRange uniform_range(const WorkRange& w) {
    return WorkRange{__shfl_sync(0xffffffffu, w.begin, 0), __shfl_sync(0xffffffffu, w.end, 0), __shfl_sync(0xffffffffu, w.q, 0),
                     __shfl_sync(0xffffffffu, w.lo, 0)};
}
template <int kMul, int kKeys = kWorkTileKeys> struct TileIter {
    const int* used;
    int every_slot;               // KParams::every_slot
    int q, q_last, lo, hi, pos, end;
    int stop;                     // behind the query's last tile with a slot in use (kMul 2: hi or hi - 1)
    int n_cur, n_next;            // slots in use of queries q and q + 1 (one query ahead: the load is done when it is needed)
    __device__ __forceinline__ TileIter(const KParams& p, const WorkRange& w)
        : used(p.n_used), every_slot(p.every_slot), q(w.q), q_last(p.q0 + p.nq), lo(w.lo * kMul), pos(w.begin * kMul), end(w.end * kMul) {
        n_next = slots(q);
        open_query();
    }
    __device__ __forceinline__ int slots(int query) const { return every_slot ? every_slot : __ldcg(used + query); }
    __device__ __forceinline__ void open_query() {
        n_cur = n_next;
        hi = lo + work_tiles<kKeys>(n_cur) * kMul;
        stop = kMul > 1 ? lo + work_tiles<kKeys / kMul>(n_cur) : hi;
        n_next = slots(min(q + 1, q_last - 1));
    }
    __device__ __forceinline__ bool more() const { return pos < end; }
    __device__ __forceinline__ int tile() const { return pos - lo; }
    __device__ __forceinline__ bool last_of_query() const { return pos + 1 == stop || pos + 1 == end; }
    // to the next tile; true if that is another query's (or the range is finished)
    __device__ __forceinline__ bool advance() {
        if (++pos < stop) return pos >= end;
        pos = hi;
        while (pos < end) {
            ++q;
            lo = hi;
            open_query();
            if (hi > lo) break;
        }
        return true;
    }
};

// =============================================================================================
// recompute: persistent 2-CTA clusters, 18 warps per CTA
// The pair works on 256-key tiles with cta_group::2 UMMAs of shape M = 256 keys x N = 2*HP:
//   A  each CTA gathers ITS 128 keys of the tile (every kv row is fetched once per query, not once
//      per head group), chunk by chunk through a 5-slot ring of [128 keys x 64 col] chunks;
//   B  each CTA holds the Q and dO rows of ITS half of the heads, stored per column chunk as
//      [Q_j | dO_j] so that one UMMA of N = 2*HP yields P^T and dP^T side by side
//      (chunk 8 has no V columns: its dO half is a block of zeros);
//   D  each CTA ends up with [its 128 keys] x [P^T | dP^T of all heads] in its own TMEM, columns
//      ordered (head half 0: P, dP), (head half 1: P, dP); two buffers.
//   warps 0-7   softmax-gradient on the CTA's own keys: warp w -> TMEM lane quarter w % 4, head half w / 4
//   warps 8-15  gather producers (cp.async 16 B, swizzled); completion arrives on the slot's mbarrier
//   warp 16     even CTA: the UMMA issuer for the pair, one elected thread (behind elect_one its UMMAs enter at the
//               pipe's rate; two threads taking alternate chunks were needed only while a lane comparison guarded them:
//               4096 queries x 128 heads x 2048 keys 2.02 -> 1.93 ms, 64 heads 1.40 -> 1.08 ms)
//               odd CTA: forwards "my slot is full" to the even CTA (cp.async cannot signal remotely)
//   warp 17     TMA of the CTA's Q / dO chunks, one barrier per column chunk; clears dKV by bulk copies
// Slot-free, chunk-free and accumulator-ready signals are tcgen05.commit arrivals delivered to both CTAs.
// A cluster works through its range of (query, key tile) pairs (WorkRange); nothing is drained between queries: the ring,
// the two accumulator buffers and the counters behind their
// barrier phases run on, the Q / dO chunk j of the next query is fetched as soon as the last tile's UMMAs
// on chunk j have finished, and the softmax of a query's last tile overlaps the next query's first UMMAs.
// =============================================================================================
namespace rp {
constexpr int kThreads = 576;
constexpr int kProducerThreads = 256;
constexpr int kTileKeys = 256;             // per pair; 128 per CTA
constexpr int kChunkA = 128 * 128;         // 16 KB gathered chunk
template <int HP> struct Cfg {
    static constexpr int NH = HP / 2;                  // heads whose Q / dO rows this CTA holds
    static constexpr int kStages = HP == 128 ? 5 : 9;  // what the stacked Q / dO leaves of the shared memory
    static constexpr int kBHalf = NH * 128;            // one [NH heads x 64 col] chunk
    static constexpr int kBChunk = 2 * kBHalf;         // stacked [Q_j | dO_j]
    static constexpr int kOffB = 0;
    static constexpr int kOffRing = kQChunks * kBChunk;
    static constexpr int kOffMisc = kOffRing + kStages * kChunkA;
    static constexpr int kSmemBytes = kOffMisc + 1024 + 512 + 1024;   // lse/delta + barriers + alignment slack
    static constexpr int kAccCols = 2 * HP;                        // one accumulator buffer: [S | dP]
    static constexpr int kTmemCols = 2 * kAccCols;                 // two buffers
};
}  // namespace rp

template <int HP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(rp::kThreads, 1)
smla_recompute_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                           const KParams p) {
    using namespace rp;
    using C = Cfg<HP>;
    constexpr int NH = C::NH;
    constexpr int kStages = C::kStages;
    const uint32_t rank = cluster_ctarank();
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform to the compiler
    const int lane = threadIdx.x & 31;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s_base = smem_u32(smem);
    uint8_t* misc = smem + C::kOffMisc;
    float* lse_s = reinterpret_cast<float*>(misc);          // [HP] base-2 lse, +inf for padded heads
    float* delta_s = lse_s + HP;                            // [HP] Delta * sm_scale
    uint64_t* bars = reinterpret_cast<uint64_t*>(misc + 1024);
    const uint32_t bar_full = smem_u32(bars);               // [kStages] gathered chunk landed (even CTA: in both CTAs)
    const uint32_t bar_empty = bar_full + 8 * kStages;      // [kStages] pair UMMAs reading the slot finished
    const uint32_t bar_bfull = bar_empty + 8 * kStages;     // [9] Q / dO column chunk of the current query landed
    const uint32_t bar_bfree = bar_bfull + 8 * kQChunks;    // [9] the query's last UMMAs on the chunk finished
    const uint32_t bar_tfull = bar_bfree + 8 * kQChunks;    // [2] accumulator buffer complete
    const uint32_t bar_tempty = bar_tfull + 16;             // [2] (even CTA) both CTAs have read the buffer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(misc + 1024 + 8 * (2 * kStages + 2 * kQChunks + 4));
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar_drain = smem_u32(tmem_slot + 2);     // used only while winding down after an abort
    const uint32_t bar_delta = smem_u32(tmem_slot + 4);     // (own_prep) the other CTA's heads' Delta has arrived
    WorkRange* range_s = reinterpret_cast<WorkRange*>(tmem_slot + 6);
    static_assert(8 * (2 * kStages + 2 * kQChunks + 4) + 24 + sizeof(WorkRange) <= 512, "barrier area");
    const WaitCtx wc{p.g_err, s_abort, p.wait_limit, map_to_cta(smem_u32(tmem_slot + 1), rank ^ 1)};

    if (threadIdx.x == 0) {
        *s_abort = 0;
        for (int i = 0; i < kStages; ++i) {
            // the even CTA's "full" also counts one arrival forwarded from the odd CTA
            mbar_init(bar_full + 8 * i, kProducerThreads + (rank == 0 ? 1 : 0));
            mbar_init(bar_empty + 8 * i, 1);
        }
        for (int i = 0; i < kQChunks; ++i) {
            mbar_init(bar_bfull + 8 * i, 1);
            mbar_init(bar_bfree + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, 16);   // 8 softmax warps in each CTA
        }
        mbar_init(bar_drain, 1);
        mbar_init(bar_delta, 1);
        fence_mbar_init();
        if (p.own_prep) mbar_arrive_expect_tx(bar_delta, 4 * max(0, min(NH, p.h_q - NH * static_cast<int>(rank ^ 1))));
    }
    {   // zero block standing in for the dO half of column chunk 8 (never overwritten)
        uint4* z = reinterpret_cast<uint4*>(smem + C::kOffB + 8 * C::kBChunk + C::kBHalf);
        for (int i = threadIdx.x; i < C::kBHalf / 16; i += kThreads) z[i] = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
    }
    if (warp == 16) {
        tmem_alloc_2cta(smem_u32(tmem_slot), C::kTmemCols);
        tmem_relinquish_2cta();
    }
    if (!p.own_prep) pdl_wait();     // slot counts and Delta of the prep kernel; the scratch's previous readers are done
    find_range<kThreads>(p, blockIdx.x >> 1, gridDim.x >> 1, reinterpret_cast<int*>(lse_s), range_s);   // (lse_s: not in use yet)
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // barriers of both CTAs are initialised before anyone signals across
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const WorkRange range = uniform_range(*range_s);
    static_assert(kTileKeys == kWorkTileKeys, "one work tile per accumulator");
    if (p.own_prep) pdl_wait();      // nothing of the caller's has been touched so far
    pdl_trigger();                   // (the tensor memory is this CTA's: see the dq kernel)

    if (warp >= 8 && warp < 16) {
        // ------------------------------------------------------------------ gather producers
        const int pt = threadIdx.x - 256;   // 0..255
        const int u = pt & 7;               // 16-byte unit inside a 128-byte chunk row
        const int r0 = pt >> 3;             // rows r0, r0+32, r0+64, r0+96 of this CTA's 128 keys
        const uint32_t dst0 = s_base + C::kOffRing + r0 * 128 + ((u ^ (r0 & 7)) << 4);
        const char* kvb = reinterpret_cast<const char*>(p.kv) + u * 16;
        const uint64_t pol_keep = l2_policy_evict_last();
        // Indices are loaded one tile ahead, so that their latency never stalls the ring (raw values: nothing may depend
        // on a load here, or the wait for it would sit in front of the copies; they are turned into kv rows one tile
        // later, when they are used).  -1 past the top-k.
        TileIter<1> it(p, range);
        QMeta qm_next = load_qmeta(p, range.q);
        auto load_idx = [&](int (&idx)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = it.tile() * kTileKeys + static_cast<int>(rank) * 128 + r0 + 32 * i;
                idx[i] = it.more() && key < p.topk ? __ldg(p.indices + static_cast<size_t>(it.q) * p.topk + key) : -1;
            }
        };
        int idx_next[4];
        load_idx(idx_next);
        int s = 0;
        uint32_t ph = 1;                    // parity that means "slot free" for the current pass over the ring
        while (it.more()) {
            // A slot whose index is out of range reads nothing and lands as zeros (its S, dS are forced to 0
            // anyway).  Sending all of them to one stand-in row instead would make that row's cache lines a
            // hot spot that every SM queues on.
            const char* src[4];
            uint32_t nb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = gather_row_in_range(idx_next[i], qm_next, p);
                nb[i] = row >= 0 ? 16u : 0u;
                src[i] = kvb + static_cast<size_t>(row >= 0 ? row : 0) * (kDQK * 2);
            }
            if (it.advance() && it.more()) qm_next = load_qmeta(p, it.q);
            load_idx(idx_next);
            for (int j = 0; j < kQChunks; ++j) {
                mbar_wait(bar_empty + 8 * s, ph, wc, kErrRecompute + 11, kPollSleepNs);
                const uint32_t d = dst0 + s * kChunkA;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    cp_async16_zfill_hint(d + i * 32 * 128, src[i] + j * 128, nb[i], pol_keep);
                cp_async_mbar_arrive_noinc(bar_full + 8 * s);
                if (++s == kStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 17) {
        // ------------------------------------------------------------------ Q / dO chunks of this CTA's heads
        if (lane == 0) {
            tma_prefetch_desc(&tm_q);
            tma_prefetch_desc(&tm_do);
            const uint64_t pol_stream = l2_policy_evict_first();
            uint32_t qpar = 1;              // parity of "chunk free" left by the previous query
            bool first = true;
            // dKV is cleared here, for the kernel behind this one: bulk copies of the zero block, this CTA's share in step with its
            // tiles and behind their operands.  They pass by the load/store pipe that the gathers and the scratch stores fill.
            // A kernel in front of this one that stored the zeros had this one's first gathers wait behind its write-backs: 27 queries x 64
            // heads x top-k 2048 on 48000 rows 91.7 -> 87.3 us a call, 2 x 128 heads x 512 on 60000 rows 51.6 -> 46.1, 300 x 128 heads x
            // 512 on 30000 rows 216.6 -> 210.7, 4096 queries alike.
            char *clear = nullptr, *clear_end = nullptr;
            auto clear_part = [&](int done, int of) {           // this CTA's share up to tile `done` of `of`
                if (!clear) {                                   // (64-bit divisions: behind the first query's loads)
                    const size_t n = p.clear_bytes / 16;
                    clear = reinterpret_cast<char*>(p.dKV) + n * blockIdx.x / gridDim.x * 16;
                    clear_end = reinterpret_cast<char*>(p.dKV) + n * (blockIdx.x + 1) / gridDim.x * 16;
                }
                const size_t left = clear_end - clear;
                char* const to = done == of ? clear_end : clear + left / (of - done + 1);
                while (clear < to) {                            // (to <= clear_end; a piece may reach beyond `to`, never beyond the end)
                    const uint32_t bytes = static_cast<uint32_t>(min(static_cast<size_t>(C::kBHalf), static_cast<size_t>(clear_end - clear)));
                    bulk_store(clear, s_base + C::kOffB + 8 * C::kBChunk + C::kBHalf, bytes);
                    clear += bytes;
                }
            };
            for (TileIter<1> it(p, range); it.more(); first = false, qpar ^= 1) {
                const int row0 = it.q * p.h_q + NH * static_cast<int>(rank);
                for (int j = 0; j < kQChunks; ++j) {
                    if (!first) mbar_wait(bar_bfree + 8 * j, qpar, wc, kErrRecompute + 16, kPollSleepNs);
                    const bool with_do = j < kVChunks;
                    mbar_arrive_expect_tx(bar_bfull + 8 * j, (with_do ? 2 : 1) * C::kBHalf);
                    tma_load_2d_hint(s_base + C::kOffB + j * C::kBChunk, &tm_q, 64 * j, row0, bar_bfull + 8 * j, pol_stream);
                    if (with_do)
                        tma_load_2d_hint(s_base + C::kOffB + j * C::kBChunk + C::kBHalf, &tm_do, 64 * j, row0,
                                         bar_bfull + 8 * j, pol_stream);
                }
                if (p.clear_bytes) clear_part(min(it.hi, it.end), it.end);
                while (!it.advance()) {}
            }
            if (p.clear_bytes) {
                clear_part(0, 0);           // (a cluster without a tile)
                bulk_commit();
                bulk_wait_all();
            }
        }
    } else if (warp == 16) {
        if (elect_one()) {
            if (rank == 1) {
                // -------------------------------------------------------------- forward slot-full to the even CTA
                RingReader<kStages> ring(bar_full);
                const uint32_t full_even = map_to_cta(bar_full, 0);
                uint32_t qpar = 0;
                bool new_query = true;
                for (TileIter<1> it(p, range); it.more();) {
                    for (int j = 0; j < kQChunks; ++j) {
                        // this CTA's half of Q / dO is part of what "full" promises
                        if (new_query) mbar_wait(bar_bfull + 8 * j, qpar, wc, kErrRecompute + 15);
                        ring.wait(wc, kErrRecompute + 17);
                        const uint32_t s = ring.slot;
                        ring.next();
                        // The copies have landed in this CTA's shared memory (the wait above saw them complete);
                        // make them visible to the tensor core's proxy here, then signal without a cluster-scope
                        // release, which would cost this thread about a thousand cycles per chunk.
                        fence_proxy_async_smem();
                        mbar_arrive_cluster_relaxed(full_even + 8 * s);
                    }
                    new_query = it.advance();
                    if (new_query) qpar ^= 1;
                }
            } else {
                // -------------------------------------------------------------- UMMA issuer for the pair
                // One thread issues everything, so the UMMAs of an accumulator enter the pipe in chunk order and the
                // results are reproducible bit for bit.
                constexpr uint32_t idesc = make_idesc_bf16(256, C::kAccCols, 0, 0);
                const uint64_t desc_hi = make_smem_desc(0, 16, 1024, kSwizzle128) & 0xFFFFFFFF00000000ull;
                const uint32_t desc_lo = static_cast<uint32_t>(make_smem_desc(0, 16, 1024, kSwizzle128));
                const uint32_t a_lo0 = desc_lo + desc_addr(s_base + C::kOffRing);
                const uint32_t b_lo0 = desc_lo + desc_addr(s_base + C::kOffB);
                RingReader<kStages> ring(bar_full);
                int gt = 0;                     // tiles so far
                uint32_t qpar = 0;
                bool new_query = true;
                TileIter<1> it(p, range);
                const int n_tiles = range.end - range.begin;
                for (; gt < n_tiles; ++gt) {
                    const int b = gt & 1;
                    const bool last = it.last_of_query();
                    mbar_spin(bar_tempty + 8 * b, ((gt >> 1) & 1) ^ 1, wc, kErrRecompute + 13);
                    const uint32_t d = tmem + b * C::kAccCols;
#pragma unroll
                    for (int j = 0; j < kQChunks; ++j) {
                        if (new_query) mbar_wait(bar_bfull + 8 * j, qpar, wc, kErrRecompute + 12);
                        ring.wait(wc, kErrRecompute + 14);
                        const uint32_t s = ring.slot;
                        ring.next();
                        tc_fence_after_sync();
                        const uint32_t a_lo = a_lo0 + s * (kChunkA >> 4);
                        const uint32_t b_lo = b_lo0 + j * (C::kBChunk >> 4);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)   // 32 bytes further along K = +2 in the address field
                            umma_ss_2cta(d, desc_hi | (a_lo + 2 * kk), desc_hi | (b_lo + 2 * kk), idesc, (j | kk) != 0);
                        umma_commit_2cta_mask(bar_empty + 8 * s, 3);
                        if (last) umma_commit_2cta_mask(bar_bfree + 8 * j, 3);   // the next query's chunk may come in
                    }
                    umma_commit_2cta_mask(bar_tfull + 8 * b, 3);
                    new_query = it.advance();
                    if (new_query) qpar ^= 1;
                }
                if (*s_abort) {   // winding down: nothing of this thread's may still be in the tensor pipe at dealloc
                    umma_commit_2cta_mask(bar_drain, 1);
                    mbar_wait_drain(bar_drain, 0, p.wait_limit);
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax gradient (own 128 keys)
        const int quarter = warp & 3;
        const int g = warp >> 2;            // head half
        const int row = quarter * 32 + lane;
        const uint32_t tempty0 = map_to_cta(bar_tempty, 0);
        const uint64_t pol_stream = l2_policy_evict_first();
        // lse (threads 0..HP-1) and Delta (threads HP..2HP-1) of a query go through shared memory; the value for
        // the next query is fetched one query ahead
        const int t = threadIdx.x;
        auto load_stat = [&](int qg) -> float {
            if (qg >= p.q0 + p.nq) return 0.f;
            const int h = t < HP ? t : t - HP;
            if (t >= 2 * HP) return 0.f;
            if (h >= p.h_q) return t < HP ? __int_as_float(0x7f800000) : 0.f;
            const size_t o = static_cast<size_t>(qg) * p.h_q + h;
            if (t >= HP && p.own_prep) return delta_s[h];
            return t < HP ? p.lse[o] * p.lse_mult : p.delta[o] * p.sm_scale;
        };
        if (p.own_prep) {
            // Delta of the one query this cluster works on: each CTA its half of the heads, four rows a warp at a time, written to both
            // CTAs; it is done before the tile's logits are.  One launch less in a chain of four, host and GPU: 64 queries x 16 heads
            // x top-k 64 21.2 -> 20.6 us with this kernel behind the prep kernel's trigger before; on its own 24.9 -> 20.6.
            if (range.begin < range.end) {
                const uint32_t peer_delta = map_to_cta(smem_u32(delta_s), rank ^ 1), peer_bar = map_to_cta(bar_delta, rank ^ 1);
                const int h0 = NH * static_cast<int>(rank), h1 = min(p.h_q, h0 + NH);
                for (int h = h0 + warp; h < h1; h += 32) {
                    size_t at[4];
                    float d[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) at[i] = static_cast<size_t>(range.q) * p.h_q + (h + 8 * i < h1 ? h + 8 * i : h);
                    delta_rows(p.o_in, p.do_in, at, d);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (lane == i && h + 8 * i < h1) {
                            delta_s[h + 8 * i] = d[i] * p.sm_scale;
                            st_async_f32(peer_delta + 4 * (h + 8 * i), d[i] * p.sm_scale, peer_bar);
                            p.delta_out[at[i]] = d[i];
                        }
                    }
                }
            }
            if (range.begin < range.end) mbar_wait(bar_delta, 0, wc, kErrRecompute + 19, kPollSleepNs);
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        int stat_q = range.q;               // the query stat_next belongs to
        float stat_next = load_stat(stat_q);
        int gt = 0;
        int n_used = 0;
        QMeta qm{};
        bool new_query = true;
        for (TileIter<1> it(p, range); it.more(); new_query = it.advance(), ++gt) {
            const int qg = it.q, tile = it.tile();
            if (new_query) {
                n_used = slots_used(p, qg);
                qm = load_qmeta(p, qg);
                if (stat_q != qg) stat_next = load_stat(qg);       // queries without a valid slot lay in between
                asm volatile("bar.sync 1, 256;" ::: "memory");      // every softmax warp is done with the previous query
                if (t < 2 * HP) lse_s[t] = stat_next;              // delta_s follows lse_s
                asm volatile("bar.sync 1, 256;" ::: "memory");
                stat_q = qg + 1;
                stat_next = load_stat(stat_q);
            }
            {
                const int key = tile * kTileKeys + static_cast<int>(rank) * 128 + row;
                const int idx = key < p.topk ? __ldg(p.indices + static_cast<size_t>(qg) * p.topk + key) : -1;
                const bool valid = slot_valid(idx, key, qm, p);
                const int b = gt & 1;
                mbar_wait(bar_tfull + 8 * b, (gt >> 1) & 1, wc, kErrRecompute + 18, kPollSleepNs);
                tc_fence_after_sync();
                // this CTA's 128 keys are all behind the last slot in use: neither the dKV nor the dQ kernel reads them
                if (tile * kTileKeys + static_cast<int>(rank) * 128 < n_used) {
                    const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + b * C::kAccCols + g * 2 * NH;
                    // the 32 lanes hold consecutive keys: 32 x 16 bytes of consecutive addresses per store
                    const size_t off = static_cast<size_t>(p.scr0 + qg - p.q0) * p.topk_pad * HP + scratch_offset(key, g * NH, p.topk_pad);
                    __nv_bfloat16* s_out = p.s_scr + off;
                    __nv_bfloat16* ds_out = p.ds_scr + off;
                    const uint32_t vmask = valid ? 0xFFFFFFFFu : 0u;
                    // 16 heads at a time (loading the next 16 columns under the work on these was measured: no change)
                    auto work = [&](int c0, const uint32_t (&pv)[16], const uint32_t (&dpv)[16]) {
                        uint32_t so[8], dso[8];
                        const float4* l4 = reinterpret_cast<const float4*>(lse_s + g * NH + c0);     // 16 heads: 4 + 4 vector loads
                        const float4* d4 = reinterpret_cast<const float4*>(delta_s + g * NH + c0);
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            const float4 l = l4[v], dl = d4[v];
                            const float lv[4] = {l.x, l.y, l.z, l.w}, dv[4] = {dl.x, dl.y, dl.z, dl.w};
                            float sv[4], dsv[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int c = 4 * v + e;
                                // dv holds Delta * sm_scale: dS = S * (dP - Delta) * sm_scale in two instructions
                                const float sx = ex2_approx(fmaf(__uint_as_float(pv[c]), p.scale_log2e, -lv[e]));
                                sv[e] = sx;
                                dsv[e] = sx * fmaf(__uint_as_float(dpv[c]), p.sm_scale, -dv[e]);
                            }
                            // an unused slot is masked after packing (one AND per two values; also wipes the
                            // NaN / inf its never-gathered operand row may have produced)
                            so[2 * v] = pack_bf16x2(sv[0], sv[1]) & vmask;
                            so[2 * v + 1] = pack_bf16x2(sv[2], sv[3]) & vmask;
                            dso[2 * v] = pack_bf16x2(dsv[0], dsv[1]) & vmask;
                            dso[2 * v + 1] = pack_bf16x2(dsv[2], dsv[3]) & vmask;
                        }
                        // 16 heads = two blocks of 8; a block is topk_pad * 8 elements further
                        __nv_bfloat16* s0 = s_out + static_cast<size_t>(c0) * p.topk_pad;
                        __nv_bfloat16* d0 = ds_out + static_cast<size_t>(c0) * p.topk_pad;
                        const size_t blk = static_cast<size_t>(p.topk_pad) * 8;
                        st_global_v4_hint(s0, so[0], so[1], so[2], so[3], pol_stream);
                        st_global_v4_hint(s0 + blk, so[4], so[5], so[6], so[7], pol_stream);
                        st_global_v4_hint(d0, dso[0], dso[1], dso[2], dso[3], pol_stream);
                        st_global_v4_hint(d0 + blk, dso[4], dso[5], dso[6], dso[7], pol_stream);
                    };
#pragma unroll 1
                    for (int c0 = 0; c0 < NH; c0 += 16) {
                        uint32_t pv[16], dpv[16];
                        tmem_ld_32x16(taddr + c0, pv);
                        tmem_ld_32x16(taddr + NH + c0, dpv);
                        tmem_ld_wait();
                        work(c0, pv, dpv);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                // The accumulator reads have completed (tcgen05.wait::ld above), which is all the issuer needs to know;
                // the stores to the scratch are ordered by the kernel boundary.  A cluster-scope release here would hold
                // the warp for about a thousand cycles per tile.
                if (lane == 0) mbar_arrive_cluster_relaxed(tempty0 + 8 * b);
            }
        }
    }
    abort_wind_down(s_abort);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 16) tmem_dealloc_2cta(tmem, C::kTmemCols);
}

// =============================================================================================
// forward: o = softmax(scale q K_g^T) V_g and lse in one pass over the keys, as persistent 2-CTA clusters.
//
// Heads are the M side of both contractions (cta_group::2 UMMAs of M = 128: 64 head rows per CTA, which run at the full
// rate of the pair: a 128 x 256 x 16 UMMA takes 64 cycles), so a head's logits, probabilities and outputs all sit in the
// same tensor-memory lanes of the same CTA: no exchange of probabilities between the CTAs and row statistics that are
// local to four threads.
//   S  [64 heads per CTA x 256 keys] = Q . K_g^T    A = this CTA's Q rows (resident, 72 KB), B = this CTA's 128 gathered
//      keys; lanes 0-63 hold keys 0-127 of the tile, lanes 64-127 the same heads with keys 128-255; two buffers
//   O  [64 heads per CTA x 512 d] += P . V_g        A = P (bf16, written to shared memory by the softmax warps), B = for two
//      d-blocks of 256 this CTA's 128 columns of all 256 keys, gathered a second time in that form
//   tensor memory: O 2 x 128 columns, S 2 x 128 columns
// Both gathers go through one ring of 16 KB slots in the order the UMMAs consume them: K of tile n + 1 (nine slots of
// [128 keys x 64 columns]), then V of tile n (eight slots of [64 keys x 128 columns]); a slot feeds four UMMAs of 64
// cycles either way, and the softmax of tile n runs under the UMMAs of S n + 1.
//   warps 0-15  softmax: warp w reads lane quarter w % 4, columns [32 (w / 4), + 32) of S: one head, 32 keys per thread
//   warps 16-19 gather producers (cp.async 16 B, swizzled)
//   warp 20     even CTA: the UMMA issuer (one elected thread); odd CTA: forwards "my slot is full"
//   warp 21     TMA of the CTA's Q chunks; odd CTA: forwards "my P is written"
// The exponentials of a tile are taken against the maximum of the row so far; where a tile raises it, O and the sum are
// rescaled.  A reference that lags behind the maximum (moved only when exceeded by 2^8) makes most of the rescaling
// unnecessary and is 3 % faster (128 heads, 2.34 against 2.42 ms), but the heaviest probabilities then lose in their rounding
// to bf16: against the maximum the heaviest is 1 exactly and the ones next to it lie where bf16 is finest.  Error of o against
// 64 bits, lagging / in this form / two passes with the final maximum: 1.974 / 1.940 / 1.956e-3 for inputs of N(0, 1),
// 1.930 / 1.665 / 1.695e-3 with logits eight times as large (2048 slots, 128 heads).  Nothing depends on timing, o and lse
// repeat bit for bit.
// What bounds it: per tile and CTA 17 slots x 4 UMMAs x 64 cycles = 4352 cycles of tensor pipe; 275 KB of gathered rows
// written and 408 KB of operands read in shared memory, 5350 cycles at 128 B/clk.  Eight softmax warps of 64 keys a thread were
// busy 95 % of a launch, the issuer waiting 1900 cycles a tile for P (8330 cycles a tile, 128 heads).  Sixteen warps of 32 keys
// hide each other's latency, P is announced by a local arrival that a thread of the odd CTA forwards (a cluster-scope release by
// every warp held it for hundreds of cycles): what is left are waits for gathered slots.  4096 queries x 128 heads x top-k 2048
// back to back, where the power cap holds the clock down: 2568 us with eight warps, 2458 with sixteen and a forwarded arrival that
// released nothing, 2 % above that as it is (see warp 21).  Five, six and seven ring slots were compared with eight warps only (2.48 /
// 2.47 / 2.48 ms), when the ring was not what the issuer waited for.
// A query whose tiles lie in several clusters' ranges leaves unnormalised partial results, which
// smla_fwd_combine_kernel adds up.
// =============================================================================================
namespace ff {
constexpr int kSoftmaxWarps = 16;
constexpr int kProducerThreads = 128;
constexpr int kThreads = kSoftmaxWarps * 32 + kProducerThreads + 64;
constexpr int kIssueWarp = kThreads / 32 - 2, kLoadWarp = kThreads / 32 - 1;
constexpr int kParts = 8;                  // a head's 256 keys of a tile over eight warps
constexpr int kTileKeys = 256;             // per pair; 128 per CTA
constexpr int kSlotBytes = 16384;
constexpr int kStages = 7;
constexpr int kQChunk = 64 * 128;          // [64 head rows x 64 columns]
constexpr int kPChunk = 64 * 128;          // [64 head rows x 64 keys]
constexpr int kOffQ = 0;
constexpr int kOffP = kQChunks * kQChunk;
constexpr int kOffRing = kOffP + 4 * kPChunk;
constexpr int kOffRows = kOffRing + kStages * kSlotBytes;     // [3 tiles][256] kv rows
constexpr int kOffStat = kOffRows + 3 * kTileKeys * 4;        // [2 tile parities][8 key parts][64 heads] row maxima / sums
constexpr int kOffMisc = kOffStat + 2 * kParts * 64 * 4;
constexpr int kSmemBytes = kOffMisc + 512 + 1024;             // barriers + alignment slack
constexpr int kTmemO = 0, kTmemS = 256;
static_assert(kSmemBytes <= 232448, "shared memory of one SM");
// Groups of 64 keys (two slots each) up to the last slot in use of the iterator's tile: what lies behind takes no part in P V.  4096
// queries x 128 heads x top-k 100 418 -> 370 us, 3000 x 64 heads x 330 428 -> 388, 4000 x 128 heads of a causal prefix 2268 -> 2079; full
// tiles alike (128 heads) or 2.5 % faster (64).  It takes loops with variable ends, and with eight producer warps (72 registers a
// thread) those spilled: full tiles 2 - 13 % slower.  Four producer warps leave 80 registers.
__device__ __forceinline__ int v_groups(const TileIter<1>& it) { return (min(kTileKeys, it.n_cur - it.tile() * kTileKeys) + 63) >> 6; }
}  // namespace ff

// lse of a row that has a valid slot (the prep kernel writes the rows of a query that has none) from the reference of its
// exponentials and their sum; o is O / sum.  What is not a number stays none, as in plain torch: a NaN logit makes the sum and
// with it o and lse NaN; a logit of +inf gives o NaN, lse +inf; logits that are all -inf (sum 0) give o NaN, lse -inf.
__device__ __forceinline__ float row_lse(float ref, float sum) {
    const float inf = __int_as_float(0x7f800000);
    return ref == inf ? inf : ref + __log2f(sum);
}

// lse of a query without a valid slot, and the row sum that marks partial results without one (a sum is never negative).
__device__ __forceinline__ float no_slot_lse(const KParams& p) { return __int_as_float(0x7f800000) * p.lse_out_mult; }
constexpr float kNoSlot = -1.f;

template <int HP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ff::kThreads, 1)
smla_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const KParams p) {
    using namespace ff;
    constexpr int NH = HP / 2;               // heads of this CTA (of the 64 rows the UMMAs compute)
    constexpr int kBusyWarps = NH / 4;       // with 64 heads a CTA's rows 32-63 do not exist: the warps of those lane quarters idle
    const uint32_t rank = cluster_ctarank();
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s_base = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kOffMisc);
    const uint32_t bar_full = smem_u32(bars);               // [kStages] slot landed (even CTA: in both CTAs)
    const uint32_t bar_empty = bar_full + 8 * kStages;      // [kStages] the UMMAs reading the slot finished
    const uint32_t bar_qfull = bar_empty + 8 * kStages;     // [9] Q column chunk of the current query landed
    const uint32_t bar_qfree = bar_qfull + 8 * kQChunks;    // [9] the query's last UMMAs on the chunk finished
    const uint32_t bar_tfull = bar_qfree + 8 * kQChunks;    // [2] S buffer complete
    const uint32_t bar_tempty = bar_tfull + 16;             // [2] (even CTA) both CTAs have read the S buffer
    const uint32_t bar_pfull = bar_tempty + 16;             // P of the tile written (even CTA: in both CTAs)
    const uint32_t bar_pv = bar_pfull + 8;                  // O += P V of the tile finished
    const uint32_t bar_drain = bar_pv + 8;                  // used only while winding down after an abort
    constexpr int kBars = 2 * kStages + 2 * kQChunks + 7;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffMisc + 8 * kBars);
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    WorkRange* range_s = reinterpret_cast<WorkRange*>(tmem_slot + 2);
    static_assert(8 * kBars + 8 + sizeof(WorkRange) <= 512, "barrier area");
    const WaitCtx wc{p.g_err, s_abort, p.wait_limit, map_to_cta(smem_u32(tmem_slot + 1), rank ^ 1)};

    if (threadIdx.x == 0) {
        *s_abort = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(bar_full + 8 * i, kProducerThreads + (rank == 0 ? 1 : 0));   // + the odd CTA's forwarded arrival
            mbar_init(bar_empty + 8 * i, 1);
        }
        for (int i = 0; i < kQChunks; ++i) {
            mbar_init(bar_qfull + 8 * i, 1);
            mbar_init(bar_qfree + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, 2 * kBusyWarps);
        }
        mbar_init(bar_pfull, kBusyWarps + (rank == 0 ? 1 : 0));      // + the odd CTA's forwarded arrival
        mbar_init(bar_pv, 1);
        mbar_init(bar_drain, 1);
        fence_mbar_init();
    }
    if constexpr (NH < 64) {     // head rows that do not exist: computed from zeros, never read
        for (int i = threadIdx.x; i < kQChunks * (64 - NH) * 8; i += kThreads) {
            const int j = i / ((64 - NH) * 8), r = i % ((64 - NH) * 8);
            *reinterpret_cast<uint4*>(smem + kOffQ + j * kQChunk + NH * 128 + r * 16) = make_uint4(0, 0, 0, 0);
        }
        fence_proxy_async_smem();
    }
    if (warp == kIssueWarp) {
        tmem_alloc_2cta(smem_u32(tmem_slot), 512);
        tmem_relinquish_2cta();
    }
    if (warp == kLoadWarp && lane == 0) tma_prefetch_desc(&tm_q);
    if (!p.every_slot) pdl_wait();   // the prep kernel's slot counts
    const int total = find_range<kThreads>(p, blockIdx.x >> 1, gridDim.x >> 1, reinterpret_cast<int*>(smem + kOffStat), range_s);
    if (total >= 0 && rank == 0 && !p.every_slot) p.range_q[blockIdx.x >> 1] = make_int4(range_s->q, range_s->lo, total, 0);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // barriers of both CTAs are initialised before anyone signals across
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const WorkRange range = uniform_range(*range_s);
    const int n_tiles = range.end - range.begin;
    if (p.every_slot) pdl_wait();    // nothing of the caller's has been touched so far
    pdl_trigger();                   // (the tensor memory is this CTA's: see the dq kernel)

    if (warp >= kSoftmaxWarps && warp < kIssueWarp) {
        // ------------------------------------------------------------------ gather producers
        const int pt = threadIdx.x - kSoftmaxWarps * 32;   
        constexpr int kRowsK = kProducerThreads / 8, kRowsV = kProducerThreads / 16;     // rows that the producers copy side by side
        const char* kvb = reinterpret_cast<const char*>(p.kv);
        const uint64_t pol_keep = l2_policy_evict_last();
        int* rows = reinterpret_cast<int*>(smem + kOffRows);
        // K: thread copies 16-byte unit uk of rows rk + 32 i of this CTA's 128 keys
        const int uk = pt & 7, rk = pt >> 3;
        const uint32_t dst_k = s_base + kOffRing + rk * 128 + ((uk ^ (rk & 7)) << 4);
        // V: unit uv of the 256 bytes (two swizzled 64-column halves of 8 KB) of rows rv + 16 i of 64 keys
        const int uv = pt & 15, rv = pt >> 4;
        const uint32_t dst_v = s_base + kOffRing + (uv >> 3) * 8192 + rv * 128 + (((uv & 7) ^ (rv & 7)) << 4);
        const char* src_v = kvb + rank * 256 + uv * 16;      // columns [256 block + 128 rank, + 128)
        int s = 0;
        uint32_t ph = 1;                    // parity that means "slot free" for the current pass over the ring
        // key pt of every tile: raw index loaded one tile ahead, turned into a kv row when it is published
        TileIter<1> it(p, range);
        QMeta qm = load_qmeta(p, range.q);
        constexpr int kKeys = kTileKeys / kProducerThreads;
        int idx_next[kKeys];
        auto load_idx = [&]() {
#pragma unroll
            for (int i = 0; i < kKeys; ++i) {
                const int key = it.tile() * kTileKeys + pt + i * kProducerThreads;
                idx_next[i] = it.more() && key < p.topk ? __ldg(p.indices + static_cast<size_t>(it.q) * p.topk + key) : -1;
            }
        };
        load_idx();
        auto next_slot = [&]() {
            cp_async_mbar_arrive_noinc(bar_full + 8 * s);
            if (++s == kStages) {
                s = 0;
                ph ^= 1;
            }
        };
        int groups = 0, groups_next = 0;                // V's groups of 64 keys: of tile n, of tile n + 1
        for (int n = -1; n < n_tiles; ++n, groups = groups_next) {            // K of tile n + 1, then V of tile n
            if (n + 1 < n_tiles) {
                // three buffers: the one written now was last read two steps ago, before the previous step's barrier
                int* mine = rows + (n + 1) % 3 * kTileKeys;
#pragma unroll
                for (int i = 0; i < kKeys; ++i) {
                    const int at = pt + i * kProducerThreads;
                    mine[at] = gather_row(idx_next[i], it.tile() * kTileKeys + at, qm, p);
                }
                groups_next = v_groups(it);
                if (it.advance() && it.more()) qm = load_qmeta(p, it.q);
                load_idx();
                asm volatile("bar.sync 3, %0;" ::"n"(kProducerThreads) : "memory");
                const char* src[128 / kRowsK];
                uint32_t nb[128 / kRowsK];  // 0: the slot takes no part, read nothing and land zeros
#pragma unroll
                for (int i = 0; i < 128 / kRowsK; ++i) {
                    const int row = mine[rank * 128 + rk + kRowsK * i];
                    nb[i] = row >= 0 ? 16u : 0u;
                    src[i] = kvb + static_cast<size_t>(row >= 0 ? row : 0) * (kDQK * 2) + uk * 16;
                }
                for (int j = 0; j < kQChunks; ++j) {
                    mbar_wait(bar_empty + 8 * s, ph, wc, kErrFwd + 11, kPollSleepNs);
                    const uint32_t d = dst_k + s * kSlotBytes;
#pragma unroll
                    for (int i = 0; i < 128 / kRowsK; ++i) cp_async16_zfill_hint(d + i * kRowsK * 128, src[i] + j * 128, nb[i], pol_keep);
                    next_slot();
                }
            }
            if (n >= 0) {
                const int* mine = rows + n % 3 * kTileKeys;
#pragma unroll 1
                for (int g = 0; g < groups; ++g) {
                    const char* src[64 / kRowsV];
                    uint32_t nb[64 / kRowsV];
#pragma unroll
                    for (int i = 0; i < 64 / kRowsV; ++i) {
                        const int row = mine[g * 64 + rv + kRowsV * i];
                        nb[i] = row >= 0 ? 16u : 0u;
                        src[i] = src_v + static_cast<size_t>(row >= 0 ? row : 0) * (kDQK * 2);
                    }
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        mbar_wait(bar_empty + 8 * s, ph, wc, kErrFwd + 11, kPollSleepNs);
                        const uint32_t d = dst_v + s * kSlotBytes;
#pragma unroll
                        for (int i = 0; i < 64 / kRowsV; ++i) cp_async16_zfill_hint(d + i * kRowsV * 128, src[i] + b * 512, nb[i], pol_keep);
                        next_slot();
                    }
                }
            }
        }
    } else if (warp == kLoadWarp) {
        // ------------------------------------------------------------------ Q chunks of this CTA's heads; odd CTA: "my P is written"
        if (lane == 0) {
            const uint64_t pol_stream = l2_policy_evict_first();
            const uint32_t pfull_even = map_to_cta(bar_pfull, 0);
            uint32_t qpar = 1;              // parity of "chunk free" left by the previous query
            TileIter<1> it(p, range);
            bool new_query = true;
            for (int n = -1; n < n_tiles; ++n) {
                if (new_query && it.more()) {                 // of tile n + 1: free once the logits of tile n are done
                    const int row0 = it.q * p.h_q + NH * static_cast<int>(rank);
                    for (int j = 0; j < kQChunks; ++j) {
                        if (n >= 0) mbar_wait(bar_qfree + 8 * j, qpar, wc, kErrFwd + 16, kPollSleepNs);
                        mbar_arrive_expect_tx(bar_qfull + 8 * j, NH * 128);
                        tma_load_2d_hint(s_base + kOffQ + j * kQChunk, &tm_q, 64 * j, row0, bar_qfull + 8 * j, pol_stream);
                    }
                    qpar ^= 1;
                }
                if (it.more()) new_query = it.advance();
                // P is plain stores of this CTA's softmax warps, and they have rescaled its O and read it out: none of that is a case
                // for a relaxed arrival, so it is released for the issuer at cluster scope, once a tile.
                // That adds a tile's latency where a cluster has one tile and 1 - 2 % where it has many (without the release / with it):
                // 8 tokens x 128 heads x 2048 19.4 / 19.9 us, 74 x 256 12.3 / 12.9, 4096 x 256 408 / 416, x 2048 2383 / 2407.  By the thread
                // that forwards the slots, whose next slot waits for it: 20.1, -, 448, 2429; a wait at cluster scope in the issuer on
                // top of that: 20.2, -, 451, 2482.  By a warp of its own the block leaves no room for one of the combine kernel beside
                // it: 20.0, 13.1, 417, 2423, and one query x 18944 slots 52.6 us against 39.1.
                if (rank == 1 && n >= 0) {
                    mbar_wait(bar_pfull, n & 1, wc, kErrFwd + 22);
                    tc_fence_after_sync();
                    fence_proxy_async_smem();
                    tc_fence_before_sync();
                    mbar_arrive_cluster_release(pfull_even);
                }
            }
        }
    } else if (warp == kIssueWarp) {
        if (elect_one()) {
            if (rank == 1) {
                // -------------------------------------------------------------- forward slot-full to the even CTA
                RingReader<kStages> ring(bar_full);
                const uint32_t full_even = map_to_cta(bar_full, 0);
                uint32_t qpar = 0;
                TileIter<1> it(p, range);
                bool new_query = true;
                int groups = 0, groups_next = 0;
                for (int n = -1; n < n_tiles; ++n, groups = groups_next) {
                    const int k_slots = n + 1 < n_tiles ? kQChunks : 0;
                    const int slots = k_slots + 2 * groups;
                    for (int j = 0; j < slots; ++j) {
                        // this CTA's half of Q is part of what "full" promises
                        if (j < k_slots && new_query) mbar_wait(bar_qfull + 8 * j, qpar, wc, kErrFwd + 15);
                        ring.wait(wc, kErrFwd + 17);
                        const uint32_t s = ring.slot;
                        ring.next();
                        // The copies have landed in this CTA's shared memory (the wait above saw them complete); make them
                        // visible to the tensor core's proxy here, then signal without a cluster-scope release
                        // (hundreds of cycles per call).
                        fence_proxy_async_smem();
                        mbar_arrive_cluster_relaxed(full_even + 8 * s);
                    }
                    if (k_slots) {
                        groups_next = v_groups(it);
                        new_query = it.advance();
                        if (new_query) qpar ^= 1;
                    }
                }
            } else {
                // -------------------------------------------------------------- UMMA issuer for the pair
                constexpr uint32_t idesc_s = make_idesc_bf16(128, 256, 0, 0);
                constexpr uint32_t idesc_o = make_idesc_bf16(128, 256, 0, 1);      // V: d contiguous (MN-major)
                const uint64_t k_hi = make_smem_desc(0, 16, 1024, kSwizzle128) & 0xFFFFFFFF00000000ull;
                const uint32_t k_lo = static_cast<uint32_t>(make_smem_desc(0, 16, 1024, kSwizzle128));
                const uint64_t v_hi = make_smem_desc(0, 8192, 1024, kSwizzle128) & 0xFFFFFFFF00000000ull;
                const uint32_t v_lo = static_cast<uint32_t>(make_smem_desc(0, 8192, 1024, kSwizzle128)) + desc_addr(s_base + kOffRing);
                const uint32_t q_lo = k_lo + desc_addr(s_base + kOffQ), p_lo = k_lo + desc_addr(s_base + kOffP);
                const uint32_t kr_lo = k_lo + desc_addr(s_base + kOffRing);
                RingReader<kStages> ring(bar_full);
                uint32_t qpar = 0;
                TileIter<1> it(p, range);
                bool new_query = true;
                uint32_t first_bits = 0;      // bit n & 1: tile n is its query's first in this range
                int groups = 0, groups_next = 0;
                for (int n = -1; n < n_tiles; ++n, groups = groups_next) {
                    if (n + 1 < n_tiles) {
                        // S of tile n + 1
                        const int t = n + 1, b = t & 1;
                        const bool last = it.last_of_query();
                        mbar_wait(bar_tempty + 8 * b, ((t >> 1) & 1) ^ 1, wc, kErrFwd + 13);
                        const uint32_t d = tmem + kTmemS + b * 128;
#pragma unroll 1
                        for (int j = 0; j < kQChunks; ++j) {
                            if (new_query) mbar_wait(bar_qfull + 8 * j, qpar, wc, kErrFwd + 12);
                            ring.wait(wc, kErrFwd + 14);
                            const uint32_t s = ring.slot;
                            ring.next();
                            fence_proxy_async_smem();        // the slot was written by cp.async, the tensor core reads it
                            tc_fence_after_sync();
                            const uint32_t a = q_lo + j * (kQChunk >> 4), bb = kr_lo + s * (kSlotBytes >> 4);
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)   // 32 bytes further along K = +2 in the address field
                                umma_ss_2cta(d, k_hi | (a + 2 * kk), k_hi | (bb + 2 * kk), idesc_s, (j | kk) != 0);
                            umma_commit_2cta_mask(bar_empty + 8 * s, 3);
                            if (last) umma_commit_2cta_mask(bar_qfree + 8 * j, 3);   // the next query's chunk may come in
                        }
                        umma_commit_2cta_mask(bar_tfull + 8 * b, 3);
                        groups_next = v_groups(it);
                        first_bits = (first_bits & ~(1u << b)) | (static_cast<uint32_t>(new_query) << b);
                        new_query = it.advance();
                        if (new_query) qpar ^= 1;
                    }
                    if (n >= 0) {
                        // O += P V of tile n
                        const uint32_t acc0 = ((first_bits >> (n & 1)) & 1u) ^ 1u;
                        mbar_wait(bar_pfull, n & 1, wc, kErrFwd + 19);
#pragma unroll 1
                        for (int g = 0; g < groups; ++g) {
#pragma unroll
                            for (int b = 0; b < 2; ++b) {
                                ring.wait(wc, kErrFwd + 14);
                                const uint32_t s = ring.slot;
                                ring.next();
                                fence_proxy_async_smem();        // the slot was written by cp.async, the tensor core reads it
                                tc_fence_after_sync();
                                const uint32_t a = p_lo + g * (kPChunk >> 4), bb = v_lo + s * (kSlotBytes >> 4);
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)   // 16 keys: 32 bytes along P's rows, 16 rows (2 KB) of V
                                    umma_ss_2cta(tmem + kTmemO + b * 128, k_hi | (a + 2 * kk), v_hi | (bb + kk * (2048 >> 4)), idesc_o,
                                                 (g | kk) != 0 ? 1u : acc0);
                                umma_commit_2cta_mask(bar_empty + 8 * s, 3);
                            }
                        }
                        umma_commit_2cta_mask(bar_pv, 3);
                    }
                }
                if (*s_abort) {   // winding down: nothing of this thread's may still be in the tensor pipe at dealloc
                    umma_commit_2cta_mask(bar_drain, 1);
                    mbar_wait_drain(bar_drain, 0, p.wait_limit);
                }
            }
        }
    } else if ((warp & 1) * 32 < NH) {
        // ------------------------------------------------------------------ softmax (one head, 32 keys of the tile per thread)
        const int quarter = warp & 3, cg = warp >> 2;
        const int part = (quarter >> 1) * 4 + cg;                // which 32 keys of the tile
        const int row = (quarter & 1) * 32 + lane;               // head row of this CTA
        const int head = static_cast<int>(rank) * NH + row;
        const bool real = head < p.h_q;
        const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
        const uint32_t tempty0 = map_to_cta(bar_tempty, 0);
        const uint32_t p_row = s_base + kOffP + (part >> 1) * kPChunk + row * 128;
        const int bar_id = 1 + (quarter & 1);                    // the eight warps that share 32 rows
        float* stat = reinterpret_cast<float*>(smem + kOffStat) + row;
        const float ninf = __int_as_float(0xff800000);
        TileIter<1> it(p, range);
        QMeta qm = load_qmeta(p, range.q);
        int idx = -1;                        // of the lane's key, loaded a tile ahead
        auto load_idx = [&]() {
            const int key = it.tile() * kTileKeys + part * 32 + lane;
            idx = it.more() && key < p.topk ? __ldg(p.indices + static_cast<size_t>(it.q) * p.topk + key) : -1;
        };
        load_idx();
        bool new_query = true;
        float ref = ninf, sum = 0.f;         // reference of the row's exponentials (log2 units), sum over this thread's keys
        bool any_valid = false;              // the query has had a valid slot (only every_slot gives tiles to one that has none)
        // A query's O leaves when the next tile's exponentials are done: waiting for the last P V right behind its P held
        // up the next query's softmax, and the tensor pipe with it, by about 4000 cycles a query.
        bool pending = false, pend_whole = false;
        float pend_inv = 0.f;
        size_t pend_row = 0;                 // row of o, or slot of the partial results
        // o may start at any multiple of 16 bytes; where it is one of 32 it leaves in 32-byte stores (4096 queries x 128 heads x
        // top-k 256: 488 us, 565 us in 16-byte stores)
        const bool wide_o = (reinterpret_cast<uintptr_t>(p.gout) & 31) == 0;
        const uint32_t o_cols = tmem + lanes + kTmemO + cg * 32;         // this warp's 32 columns of either d-block
        auto write_out = [&]() {
            pending = false;
            // lanes 0-63: columns [256 block, + 128), lanes 64-127: [256 block + 128, + 128)
#pragma unroll 1
            for (int blk = 0; blk < 2; ++blk) {
                uint32_t o[32];
                tmem_ld_32x32(o_cols + blk * 128, o);
                tmem_ld_wait();
                const int col = blk * 256 + (quarter >> 1) * 128 + cg * 32;
                const size_t at = pend_row * kDV + col;
                if (real && pend_whole) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        uint32_t w[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            w[i] = pack_bf16x2(__uint_as_float(o[16 * e + 2 * i]) * pend_inv, __uint_as_float(o[16 * e + 2 * i + 1]) * pend_inv);
                        if (wide_o) {
                            st_global_v8(p.gout + at + 16 * e, w);
                        } else {
#pragma unroll
                            for (int v = 0; v < 2; ++v)
                                *reinterpret_cast<uint4*>(p.gout + at + 16 * e + 8 * v) = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
                        }
                    }
                } else if (real) {
#pragma unroll
                    for (int v = 0; v < 4; ++v)      // [slot][8 columns][heads]: a warp's store is 1 KB in one piece
                        st_global_v8(p.part_o + ((pend_row * (kDV / 8) + (col >> 3) + v) * HP + head) * 8, *reinterpret_cast<const uint32_t(*)[8]>(o + 8 * v));
                }
            }
        };
        int seg_begin = 0;
        for (int n = 0; n < n_tiles; ++n) {
            const uint32_t mask = __ballot_sync(0xffffffffu, slot_valid(idx, it.tile() * kTileKeys + part * 32 + lane, qm, p));
            if (new_query) {
                ref = ninf;
                sum = 0.f;
                any_valid = false;
                seg_begin = it.pos;
            }
            const int qg = it.q, q_lo = it.lo, q_hi = it.hi;
            const bool last = it.last_of_query();
            const int seg_end = it.pos + 1;
            const bool next_query = it.advance();
            if (next_query && it.more()) qm = load_qmeta(p, it.q);
            load_idx();

            const int b = n & 1;
            mbar_wait(bar_tfull + 8 * b, (n >> 1) & 1, wc, kErrFwd + 18, kPollSleepNs);
            tc_fence_after_sync();
            uint32_t sv[32];
            tmem_ld_32x32(tmem + lanes + kTmemS + b * 128 + cg * 32, sv);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            // the S buffer has been read (tcgen05.wait::ld), which is all the issuer needs to know
            if (lane == 0) mbar_arrive_cluster_relaxed(tempty0 + 8 * b);
            if (mask != 0xffffffffu) {                       // warp-uniform
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (!((mask >> i) & 1u)) sv[i] = 0xff800000u;
            }
            float m[4] = {ninf, ninf, ninf, ninf};
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k) m[k] = fmaxf(m[k], __uint_as_float(sv[i + k]));
            }
            stat[(b * kParts + part) * 64] = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
            any_valid = bar_or(bar_id, 256, mask != 0u) || any_valid;
            float scale_o = 1.f;
            bool rescale = false;
            float top = ninf;
#pragma unroll
            for (int i = 0; i < kParts; ++i) top = fmaxf(top, stat[(b * kParts + i) * 64]);
            top *= p.scale_log2e;
            if (top > ref) {             // (first valid tile: O and the sum are still empty)
                rescale = ref > ninf;
                if (rescale) scale_o = ex2_approx(ref - top);
                ref = top;
            }
            const float neg = ref == ninf ? 0.f : -ref;
            sum *= scale_o;
            float add[2] = {0.f, 0.f};
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float x = ex2_approx(fmaf(__uint_as_float(sv[2 * i]), p.scale_log2e, neg));
                const float y = ex2_approx(fmaf(__uint_as_float(sv[2 * i + 1]), p.scale_log2e, neg));
                add[0] += x;
                add[1] += y;
                pk[i] = pack_bf16x2(x, y);
            }
            sum += add[0] + add[1];
            // P of the previous tile has been consumed and O is at rest
            if (n > 0) mbar_wait(bar_pv, (n - 1) & 1, wc, kErrFwd + 20, kPollSleepNs);
            tc_fence_after_sync();
#pragma unroll
            for (int u = 0; u < 4; ++u)
                st_shared_v4(p_row + ((((part & 1) * 4 + u) ^ (row & 7)) << 4), pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
            fence_proxy_async_smem();
            if (pending) write_out();
            if (__any_sync(0xffffffffu, rescale)) {          // this warp's quarter of the columns of both d-blocks
#pragma unroll 1
                for (int blk = 0; blk < 2; ++blk) {
                    uint32_t o[32];
                    tmem_ld_32x32(o_cols + blk * 128, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * scale_o);
                    tmem_st_32x32(o_cols + blk * 128, o);
                }
                tmem_st_wait();
            }
            tc_fence_before_sync();
            __syncwarp();
            // Local arrival, forwarded by warp 21 of the odd CTA: a cluster-scope release would hold this warp for hundreds of cycles.
            if (lane == 0) mbar_arrive(bar_pfull);

            if (last) {
                // ---- the query's (or the range's) last tile: lse now, o once its P V is done - or an unnormalised part of them
                const bool whole = seg_begin == q_lo && seg_end == q_hi;
                float* sums = stat + kParts * ((n + 1) & 1) * 64;
                sums[part * 64] = sum;
                asm volatile("bar.sync %0, 256;" ::"r"(bar_id) : "memory");
                float total = 0.f;
#pragma unroll
                for (int i = 0; i < kParts; ++i) total += sums[i * 64];
                asm volatile("bar.sync %0, 256;" ::"r"(bar_id) : "memory");      // the next tile's maxima go to the same place
                const size_t orow = static_cast<size_t>(qg) * p.h_q + head;
                // partial results: slot 2 c for a range that starts inside the query, 2 c + 1 for one that starts at or before it
                const size_t slot = (blockIdx.x >> 1) * 2 + (seg_begin == q_lo ? 1 : 0);
                if (real && part == 0) {
                    if (whole) p.lse_out[orow] = any_valid ? row_lse(ref, total) * p.lse_out_mult : no_slot_lse(p);
                    else p.part_ml[slot * HP + head] = make_float2(ref, any_valid ? total : kNoSlot);
                }
                pending = true;
                pend_whole = whole;
                pend_inv = any_valid ? 1.f / total : 0.f;        // no valid slot: O is 0
                pend_row = whole ? orow : slot;
            }
            new_query = next_query;
        }
        if (pending) {
            mbar_wait(bar_pv, (n_tiles - 1) & 1, wc, kErrFwd + 21, kPollSleepNs);
            tc_fence_after_sync();
            write_out();
        }
    }
    abort_wind_down(s_abort);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // neither CTA leaves while the other may still signal it or read its operands
    if (warp == kIssueWarp) tmem_dealloc_2cta(tmem, 512);
}

// Queries whose tiles were spread over several clusters: o = sum of 2^(ref_i - ref) O_i over the parts, divided by the sum
// of their weighted row sums.  The items are the queries where there are at most as many as boundaries between ranges, else
// the boundaries (the one that is its query's first does the work; the forward kernel has noted each range's first
// query).  A lane takes one head and sixteen columns: the parts lie as [8 columns][heads][8], so a warp loads a part in pieces of
// 1 KB, and a lane's weights need no other lane.  The first parts' O is on its way while the others' references and sums are read.
// Parts are added in their order.  Bound by the latency of its dependent loads; eight queries of eight parts: 5.5 us of a call,
// 7.6 us with a warp per head and half of the columns, whose weights took two rounds of loads before the first row.
// Blocks are small, so that many of them are in place beside the forward kernel's last blocks when it ends.  kFly: parts in flight, two
// where no query has more (80 registers a thread instead of 110).  30 queries x 128 heads x top-k 512 18.2 us a call with blocks of
// 256 and four parts, 17.4 so; 90 queries x 600 41.6 / 39.4; one query x 2048 (eight parts) 15.4 / 14.9; eight x 2048 alike, and
// 19.4 -> 22.9 with two parts in flight.  112 registers at most: a block then fits beside one of the forward kernel, by the register file's
// four parts (16384 each; six warps of 80 x 32 there and one of these).  With 118 all blocks come up on the first SMs that are free, and
// one query x 18944 slots takes 49.5 us, 31.9 so.
constexpr int kCombineThreads = 64;
template <int kFly>
__global__ void __maxnreg__(112) smla_fwd_combine_kernel(const KParams p, int n_clusters, int h_pad) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    constexpr int kCols = kCombineThreads / 32, kBlocks = 32 / kCols;      // column groups of a block, blocks of 32 heads
    const int per_item = (p.h_q + 31) / 32 * kBlocks;
    const int item = static_cast<int>(blockIdx.x) / per_item, in_item = static_cast<int>(blockIdx.x) % per_item;
    const int head = in_item / kBlocks * 32 + lane, col = (in_item % kBlocks * kCols + static_cast<int>(threadIdx.x >> 5)) * 16;
    int q, n_tiles, q_begin, q_end;
    if (p.every_slot) {
        const int tiles = work_tiles(p.every_slot);
        q = p.q0 + item;
        n_tiles = p.nq * tiles;
        q_begin = item * tiles;
        q_end = q_begin + tiles;
    } else {
        const bool by_query = p.nq < n_clusters;
        const int4 boundary = __ldcg(p.range_q + (by_query ? 0 : item + 1));
        q = by_query ? p.q0 + item : boundary.x;
        n_tiles = boundary.z;
        q_begin = boundary.y;
        if (by_query) {                          // (fewer queries than clusters: at most three of them per lane)
            q_begin = 0;
            for (int i = lane; i < item; i += 32) q_begin += work_tiles(__ldcg(p.n_used + p.q0 + i));
            q_begin = __reduce_add_sync(0xffffffffu, q_begin);
        }
        q_end = q_begin + work_tiles(__ldcg(p.n_used + q));
        if (q_begin >= q_end) return;            // no valid slot: the prep kernel has written o and lse
    }
    // the clusters whose ranges hold a tile t: the largest k with range_start(k) <= t
    const int first = static_cast<int>((static_cast<long long>(q_begin + 1) * n_clusters - 1) / n_tiles);
    const int last = static_cast<int>((static_cast<long long>(q_end) * n_clusters - 1) / n_tiles);
    if (first == last || (!p.every_slot && p.nq >= n_clusters && first != item)) return;
    const float ninf = __int_as_float(0xff800000);
    // Lane i: the slot of part k0 + i, -1 where its range is empty or there is no such part.  (Once for all: the two divisions a
    // part took a good part of the kernel's time.)  All lanes stay to the end, those of heads beyond h_q with rows of the padding.
    auto slots_from = [&](int k0) {
        const int k = k0 + lane;
        if (k > last) return -1;
        const int begin = range_start(n_tiles, k, n_clusters);
        return begin == range_start(n_tiles, k + 1, n_clusters) ? -1 : 2 * k + (begin <= q_begin ? 1 : 0);
    };
    auto load_ml = [&](int slot) { return __ldcg(p.part_ml + static_cast<size_t>(slot) * h_pad + head); };
    uint32_t v[kFly][2][8];
    float2 ml[kFly];
    auto load_part = [&](int u, int slot) {
        const float* o = p.part_o + ((static_cast<size_t>(slot) * (kDV / 8) + (col >> 3)) * h_pad + head) * 8;
        ml[u] = load_ml(slot);
        ld_global_v8(o, v[u][0]);
        ld_global_v8(o + h_pad * 8, v[u][1]);
    };
    auto no_part = [&](int u) {
        ml[u] = make_float2(ninf, kNoSlot);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[u][i / 8][i % 8] = 0u;
    };
    int slots = slots_from(first);
#pragma unroll
    for (int u = 0; u < kFly; ++u) {
        const int slot = __shfl_sync(0xffffffffu, slots, u);
        no_part(u);
        if (slot >= 0) load_part(u, slot);
    }
    float ref = ninf, sum = 0.f, acc[16];
    bool any = false;
    // The other parts: their references first.  Those without a valid slot (every_slot counts their tiles as used) hold zeros and are
    // passed over:
    // one query x 128 heads x 18944 slots of which 300 are in use 38.7 -> 17.2 us, 8 x 2048 with 100 20.1 -> 17.8; all in use 38.8 -> 31.9
    // (the divisions of slots_from), 20.2 and 20.2.
    uint32_t live = 0;                           // lane w: bit i says that part first + kFly + 32 w + i has a valid slot (of all heads or of none)
#pragma unroll 1
    for (int w = 0, k0 = first + kFly; k0 <= last; ++w, k0 += 32) {
        slots = slots_from(k0);
        const uint32_t word = __ballot_sync(0xffffffffu, slots >= 0 && __ldcg(&p.part_ml[static_cast<size_t>(slots) * h_pad].y) != kNoSlot);
        if (lane == w) live = word;
        any = any || word;
        constexpr int kBatch = 8;
        for (uint32_t todo = word; todo;) {
            float x[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {   // (the first again where there are no more)
                const int slot = __shfl_sync(0xffffffffu, slots, __ffs(todo ? todo : word) - 1);
                x[u] = load_ml(slot).x;
                todo &= todo - 1;
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) ref = fmaxf(ref, x[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < kFly; ++u) {
        ref = fmaxf(ref, ml[u].x);               // -inf: no valid slot in this part, or none above -inf
        any = any || ml[u].y != kNoSlot;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    auto add_parts = [&]() {
#pragma unroll
        for (int u = 0; u < kFly; ++u) {
            const float w = ml[u].x > ninf ? ex2_approx(ml[u].x - ref) : 0.f;
            sum = fmaf(w, ml[u].y, sum);
            // (a part of weight 0 counts too: its O may hold a NaN)
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = fmaf(__uint_as_float(v[u][i / 8][i % 8]), w, acc[i]);
        }
    };
    add_parts();
#pragma unroll 1
    for (int w = 0, k0 = first + kFly; k0 <= last; ++w, k0 += 32) {
        uint32_t todo = __shfl_sync(0xffffffffu, live, w);
        if (todo == 0) continue;
        if (last - first - kFly >= 32) slots = slots_from(k0);       // (else they are the ones from before)
        while (__popc(todo) >= kFly) {
#pragma unroll
            for (int u = 0; u < kFly; ++u) {
                load_part(u, __shfl_sync(0xffffffffu, slots, __ffs(todo) - 1));
                todo &= todo - 1;
            }
            add_parts();
        }
        if (todo) {
#pragma unroll
            for (int u = 0; u < kFly; ++u) {
                const int slot = __shfl_sync(0xffffffffu, slots, todo ? __ffs(todo) - 1 : 0);
                no_part(u);
                if (todo) load_part(u, slot);
                todo &= todo - 1;
            }
            add_parts();
        }
    }
    if (head >= p.h_q) return;
    const size_t orow = static_cast<size_t>(q) * p.h_q + head;
    if (col == 0) p.lse_out[orow] = any ? row_lse(ref, sum) * p.lse_out_mult : no_slot_lse(p);
    const float inv = any ? 1.f / sum : 0.f;
    uint4* out = reinterpret_cast<uint4*>(p.gout + orow * kDV + col);
#pragma unroll
    for (int i = 0; i < 2; ++i)
        out[i] = make_uint4(pack_bf16x2(acc[8 * i] * inv, acc[8 * i + 1] * inv), pack_bf16x2(acc[8 * i + 2] * inv, acc[8 * i + 3] * inv),
                            pack_bf16x2(acc[8 * i + 4] * inv, acc[8 * i + 5] * inv), pack_bf16x2(acc[8 * i + 6] * inv, acc[8 * i + 7] * inv));
}

// =============================================================================================
// dkv as persistent 2-CTA clusters: a pair works through its range of (query, key tile) pairs, all 576 columns of d.
//
//   dKV^T[d, key] = dO^T . S + Q^T . dS with cta_group::2 UMMAs of M = 256 rows of d (128 per CTA) x N = 128 keys
//   (64 supplied by each CTA): a CTA reads 4 KB of A and 2 KB of B per 64 cycles of math, where the single-CTA
//   128x128x16 form reads 8 KB, which is all the shared-memory bandwidth there is.  The S / dS scratch of a query is
//   read once (half a tile per CTA) instead of once per d-part.
//
//   blocks of d   0: [0,256)   1: [256,512)   2: [512,576) (Q^T . dS only: V has 512 columns)
//   CTA r holds rows [128 r, 128 r + 128) of blocks 0 and 1 as resident Q^T / dO^T chunk pairs.  Block 2 is M = 128 (slot 4 holds
//   chunk 8 in both CTAs, so both compute the same 64 rows): lanes 0-63 end up with the first 64 keys of the tile, lanes 64-127 with the
//   others, and each CTA drains one half, in turn.  As one half of an M = 256 UMMA, drained by the CTAs in turn and always from lanes 64-127,
//   it took twice the tensor work and left two of the four sub-partitions a quarter more reductions than the others: 4096 queries x
//   top-k 2048 back to back, at the power cap, 4578 -> 4507 us (128 heads), 3720 -> 3677 (64).
//   warp 0      producer: resident chunks per query; per 128-key tile this CTA's 64 keys of S and dS, two or four stages
//   warp 1      even CTA: UMMA issuer for the pair; odd CTA: relays "my half landed" to the even CTA's barriers
//   warps 2-17  drain, two groups of eight on alternate accumulator units (ring of four 128-column units per CTA):
//               lane = d row, one predicated fp32 reduction per key = 128 contiguous bytes of dKV
// =============================================================================================
namespace dp {
constexpr int kThreads = 576;
constexpr int kTileKeys = 128;
constexpr int kUnits = 4;
template <int HP> struct Cfg {
    static constexpr int kChunk = HP * 128;                 // resident chunk [HP heads x 64 d] bytes
    static constexpr int kHalfMat = HP * 128;               // S (or dS) of 64 keys: [HP/8][64 keys][8 heads]
    static constexpr int kStage = 2 * kHalfMat;             // S then dS
    // What the resident chunks leave; 64 heads, 4096 queries of 16 tiles: 6.56 M cycles with two or three, 6.45 with four, 6.46
    // with six or eight.  (A second set of resident chunks beside four stages: 6.50.)
    static constexpr int kTileStages = HP == 64 ? 4 : 2;
    static constexpr int kOffQ = 0;                         // 5 slots
    static constexpr int kOffDO = 5 * kChunk;               // 4 slots
    static constexpr int kOffStage = 9 * kChunk;
    static constexpr int kOffMisc = kOffStage + kTileStages * kStage;
    static constexpr int kOffIdx = kOffMisc + 256;          // [2 groups][2 tile parities][2 key halves][64] int
    static constexpr int kSmemBytes = kOffMisc + 256 + 2048 + 1024;
};
}  // namespace dp

// kStaged: instead of adding a slot's [576] contribution into dKV with fp32 reductions (whose order, and therefore
// rounding, changes from run to run), write it to the slot's own row of a staging buffer; smla_dkv_segment_sum_kernel
// then adds the rows that belong to one kv row in a fixed order.
// kFine: ranges of 128-key tiles, what a cluster takes its time for, instead of 256-key ones, of which a query's last may be half empty: in
// six documents of 99 - 357 tokens some clusters took 157000 cycles and some 300000 (the kernel 203 -> 160 us; not so the call, whose dQ
// CTAs had filled the SMs that became free), and few queries go to twice as many clusters: one query x 128 heads x top-k 2048 36.5 -> 34.1
// us a call, 3 x 64 x 1000 27.3 -> 25.7.  Queries of one 128-key tile at most keep the other form: 64 queries x 16 heads x 64 19.4, 19.6 so.
template <int HP, bool kStaged = false, bool kFine = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(dp::kThreads, 1)
smla_dkv_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                     const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_ds, const KParams p) {
    using namespace dp;
    using C = Cfg<HP>;
    constexpr int kTileStages = C::kTileStages;
    const uint32_t rank = cluster_ctarank();
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform to the compiler
    const int lane = threadIdx.x & 31;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s_base = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffMisc);
    const uint32_t bar_tfull = smem_u32(bars);                        // [kTileStages] tile stage landed (even CTA: in both CTAs)
    const uint32_t bar_tempty = bar_tfull + 8 * kTileStages;          // [kTileStages] the tile's UMMAs finished
    const uint32_t bar_res = bar_tempty + 8 * kTileStages;            // [2] resident chunks of block 0 / of blocks 1 and 2 landed (even CTA: in both CTAs)
    const uint32_t bar_resfree = bar_res + 16;                        // [2] the query's last UMMAs on them finished
    const uint32_t bar_ufull = bar_resfree + 16;                      // [kUnits] accumulator unit complete
    const uint32_t bar_uempty = bar_ufull + 8 * kUnits;               // [kUnits] (even CTA) both CTAs have drained the unit
    const uint32_t bar_drain = bar_uempty + 8 * kUnits;               // 1  used only while winding down after an abort
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::kOffMisc + 8 * (2 * kTileStages + 5 + 2 * kUnits));
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    WorkRange* range_s = reinterpret_cast<WorkRange*>(tmem_slot + 2);
    static_assert(8 * (2 * kTileStages + 5 + 2 * kUnits) + 8 + sizeof(WorkRange) <= 256, "barrier area");
    const WaitCtx wc{p.g_err, s_abort, p.wait_limit, map_to_cta(smem_u32(tmem_slot + 1), rank ^ 1)};

    if (threadIdx.x == 0) {
        *s_abort = 0;
        for (int i = 0; i < kTileStages; ++i) {
            mbar_init(bar_tfull + 8 * i, rank == 0 ? 2 : 1);   // own expect_tx arrival (+ the odd CTA's relayed one)
            mbar_init(bar_tempty + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_res + 8 * i, rank == 0 ? 2 : 1);
            mbar_init(bar_resfree + 8 * i, 1);
        }
        mbar_init(bar_drain, 1);
        for (int i = 0; i < kUnits; ++i) {
            mbar_init(bar_ufull + 8 * i, 1);
            mbar_init(bar_uempty + 8 * i, 16);                 // eight drain warps of the unit's group in each CTA
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_2cta(smem_u32(tmem_slot), 512);
        tmem_relinquish_2cta();
    }
    // Behind the recompute kernel's trigger (it triggers after it has waited for what was before it) slot counts, indices, Q and dO
    // are in place.  S, dS and a cleared dKV are not, before that kernel has ended: the first S / dS load waits for that, and no
    // reduction can be issued before UMMAs on what it has loaded.
    if (!p.early_start) pdl_wait();
    constexpr int kRangeKeys = kFine ? kTileKeys : kWorkTileKeys;
    find_range<kThreads, kRangeKeys>(p, blockIdx.x >> 1, gridDim.x >> 1, reinterpret_cast<int*>(smem + C::kOffIdx), range_s);    // (index buffers: not in use yet)
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // barriers of both CTAs are initialised before anyone signals across
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const WorkRange range = uniform_range(*range_s);
    using Iter = TileIter<kRangeKeys / kTileKeys, kRangeKeys>;

    if (warp == 0) {
        // ------------------------------------------------------------------ producer
        if (lane == 0) {
            tma_prefetch_desc(&tm_q);
            tma_prefetch_desc(&tm_do);
            tma_prefetch_desc(&tm_s);
            tma_prefetch_desc(&tm_ds);
            const uint64_t pol_stream = l2_policy_evict_first();
            bool waited = false;
            int s = 0;
            uint32_t ph = 1, k = 0;        // ph: parity that means "stage free" in the current pass over the ring
            bool new_query = true;
            // The resident operands are replaced in two parts, each as soon as the previous query's last UMMAs on it are done
            // and behind the new query's first S / dS tile; the drain warps meanwhile still work through the accumulator ring.
            // (All nine chunks at once, in front of the tile: 265 against 225 us for 1531 queries of at most three key tiles, 6.54 against
            // 6.37 M cycles for 4096 queries of 16 tiles, 128 heads.)
            auto load_resident = [&](int q) {
                const int row0 = q * p.h_q;
                for (int i = 0; i < 2; ++i) {              // slots 0 .. 3: chunks {2r, 2r+1} of block 0, of block 1
                    if (k) mbar_wait(bar_resfree + 8 * i, (k - 1) & 1, wc, kErrDkv + 6 + i, kPollSleepNs);
                    mbar_arrive_expect_tx(bar_res + 8 * i, (4 + i) * C::kChunk);
                    for (int j = 2 * i; j < 2 * i + 2; ++j) {
                        const int chunk = i * 4 + 2 * static_cast<int>(rank) + (j & 1);
                        tma_load_2d_hint(s_base + C::kOffQ + j * C::kChunk, &tm_q, 64 * chunk, row0, bar_res + 8 * i, pol_stream);
                        tma_load_2d_hint(s_base + C::kOffDO + j * C::kChunk, &tm_do, 64 * chunk, row0, bar_res + 8 * i, pol_stream);
                    }
                    if (i) tma_load_2d_hint(s_base + C::kOffQ + 4 * C::kChunk, &tm_q, 64 * 8, row0, bar_res + 8 * i, pol_stream);
                }
                ++k;
            };
            for (Iter it(p, range); it.more(); new_query = it.advance()) {
                if (!waited) {                 // the first query's Q and dO do not wait for the kernel before this one
                    waited = true;
                    load_resident(it.q);
                    new_query = false;
                    pdl_wait();
                    pdl_trigger();
                }
                mbar_wait(bar_tempty + 8 * s, ph, wc, kErrDkv + 1, kPollSleepNs);
                mbar_arrive_expect_tx(bar_tfull + 8 * s, C::kStage);
                const uint32_t dst = s_base + C::kOffStage + s * C::kStage;
                // box = this CTA's 64 keys of every head block -> [HP/8][64 keys][8 heads]
                const int kb = it.tile() * (kTileKeys / 32) + 2 * static_cast<int>(rank);
                const int sq = p.scr0 + it.q - p.q0;
                tma_load_4d_hint(dst, &tm_s, 0, kb, 0, sq, bar_tfull + 8 * s, pol_stream);
                tma_load_4d_hint(dst + C::kHalfMat, &tm_ds, 0, kb, 0, sq, bar_tfull + 8 * s, pol_stream);
                if (new_query) load_resident(it.q);
                if (++s == kTileStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
            if (!waited) {                 // nothing to do: the kernel behind this one still relies on the wait
                pdl_wait();
                pdl_trigger();
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            if (rank == 1) {
                // -------------------------------------------------------------- relay "landed" to the even CTA
                // TMA wrote the data (async proxy) and the tensor core reads it (async proxy): no proxy fence; the
                // relaxed arrive costs a few cycles where a cluster-scope release costs hundreds.
                int s = 0;
                uint32_t ph = 0, k = 0;
                bool new_query = true;
                for (Iter it(p, range); it.more(); new_query = it.advance()) {
                    mbar_spin(bar_tfull + 8 * s, ph, wc, kErrDkv + 11);
                    mbar_arrive_cluster_relaxed(map_to_cta(bar_tfull + 8 * s, 0));
                    if (new_query) {
                        for (int i = 0; i < 2; ++i) {
                            mbar_wait(bar_res + 8 * i, k & 1, wc, kErrDkv + 10);
                            mbar_arrive_cluster_relaxed(map_to_cta(bar_res + 8 * i, 0));
                        }
                        ++k;
                    }
                    if (++s == kTileStages) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            } else {
                // -------------------------------------------------------------- UMMA issuer for the pair
                constexpr uint32_t idesc = make_idesc_bf16(256, 128, 1, 0);   // A MN-major (d contiguous), B K-major
                constexpr uint32_t idesc2 = make_idesc_bf16(128, 128, 1, 0);  // block 2: 64 rows per CTA
                int s = 0;
                uint32_t ph = 0, k = 0, unit = 0;
                bool new_query = true;
                for (Iter it(p, range); it.more();) {
                    k += new_query;
                    const bool last = it.last_of_query();
                    mbar_wait(bar_tfull + 8 * s, ph, wc, kErrDkv + 4);
                    const uint32_t st_s = s_base + C::kOffStage + s * C::kStage;
                    const uint32_t st_ds = st_s + C::kHalfMat;
                    for (int blk = 0; blk < 3; ++blk, ++unit) {
                        const int us = unit % kUnits;
                        if (new_query && blk < 2) mbar_wait(bar_res + 8 * blk, (k - 1) & 1, wc, kErrDkv + 2);
                        mbar_wait(bar_uempty + 8 * us, ((unit / kUnits) & 1) ^ 1, wc, kErrDkv + 3);
                        tc_fence_after_sync();
                        const uint32_t d = tmem + us * 128;
                        // each CTA's 128 rows: slot pair (0,1) or (2,3); for block 2 the 64 rows of slot 4, the same in both
                        const int slot = blk == 2 ? 4 : 2 * blk;
                        if (blk < 2) {
                            const uint32_t a_do = s_base + C::kOffDO + slot * C::kChunk;
#pragma unroll
                            for (int ks = 0; ks < HP / 16; ++ks)
                                umma_ss_2cta(d, make_smem_desc(a_do + ks * 2048, C::kChunk, 1024, kSwizzle128),
                                             make_smem_desc(st_s + ks * 2048, 1024, 128, kSwizzleNone), idesc, ks != 0);
                        }
                        const uint32_t a_q = s_base + C::kOffQ + slot * C::kChunk;
#pragma unroll
                        for (int ks = 0; ks < HP / 16; ++ks)
                            umma_ss_2cta(d, make_smem_desc(a_q + ks * 2048, C::kChunk, 1024, kSwizzle128),
                                         make_smem_desc(st_ds + ks * 2048, 1024, 128, kSwizzleNone), blk < 2 ? idesc : idesc2,
                                         blk < 2 || ks != 0);
                        umma_commit_2cta_mask(bar_ufull + 8 * us, 3);
                        if (last && blk != 1) umma_commit_2cta_mask(bar_resfree + 8 * (blk >> 1), 3);
                    }
                    umma_commit_2cta_mask(bar_tempty + 8 * s, 3);
                    if (++s == kTileStages) {
                        s = 0;
                        ph ^= 1;
                    }
                    new_query = it.advance();
                }
                if (*s_abort) {   // winding down: nothing of this thread's may still be in the tensor pipe at dealloc
                    umma_commit_2cta_mask(bar_drain, 1);
                    mbar_wait_drain(bar_drain, 0, p.wait_limit);
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ drain (this CTA's 128 rows of every unit)
        // Two groups of eight warps take alternate units: one group's fixed cost per unit (wait, accumulator load,
        // indices) runs under the other group's reductions.
        const int dw = warp - 2;                // 0..15
        const int grp = dw >> 3;
        const int quarter = warp & 3;           // the TMEM lane quarter a warp may read is warp % 4
        const int e = (dw >> 2) & 1;            // which 64 keys of the 128-key tile this warp scatters
        const int member = dw & 3;              // the four warps of a (group, key half) share one index buffer
        // index buffers [group][tile parity][key half][64]: filled by member 0 from registers it loaded one tile ahead,
        // published with a named barrier of the four warps.  Every tile shows up in both groups' unit sequences and
        // the barrier keeps the four within one tile of each other, so two buffers per (group, key half) suffice.
        int* idx_base = reinterpret_cast<int*>(smem + C::kOffIdx) + (grp * 4 + e) * 64;
        const int bar_id = 1 + grp * 2 + e;
        const uint32_t uempty0 = map_to_cta(bar_uempty, 0);
        int pf[2] = {-1, -1};
        // (the dKV row a valid slot adds to, -1 for an unused slot)
        auto fetch_idx = [&](int qg, int tile) {
            const QMeta qm = load_qmeta(p, qg);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int key = tile * kTileKeys + 64 * e + 32 * i + lane;
                const int idx = key < p.topk ? __ldg(p.indices + static_cast<size_t>(qg) * p.topk + key) : -1;
                pf[i] = slot_valid(idx, key, qm, p) ? qm.kv_base + idx : -1;
            }
        };
        // dKV stays in the L2 as far as it fits, ahead of the S / dS and Q / dO that stream by: 1024 queries x 128 heads x top-k 2048 on 32768
        // rows write 0.27 GB to HBM instead of 1.13.  Back to back, calls: 4096 x 128 heads x 2048 on 32768 rows 8167 -> 8071 us, on 65536
        // rows 9950 -> 9310, 2048 x 64 x 1024 on 65536 2123 -> 1933, 1000 x 64 x 300 on 50000 389 -> 362; on 8192 and 16384 rows alike.
        const uint64_t pol_keep = l2_policy_evict_last();
        Iter it(p, range);
        if (member == 0 && it.more()) fetch_idx(it.q, it.tile());
        for (uint32_t n = 0; it.more(); ++n) {      // n: tiles so far; unit 3 n + blk of the range belongs to group (n + blk) % 2
            const int tile = it.tile(), sq = p.scr0 + it.q - p.q0;
            const int left = it.n_cur - tile * kTileKeys - 64 * e;      // slots in use from this warp's 64 keys on
            int* idx_s = idx_base + (n & 1) * 128;
            if (member == 0) {
                idx_s[lane] = pf[0];
                idx_s[32 + lane] = pf[1];
            }
            asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
            it.advance();
            if (member == 0 && it.more()) fetch_idx(it.q, it.tile());
            for (int blk = (n ^ grp) & 1; blk < 3; blk += 2) {
                const uint32_t unit = 3 * n + blk;
                const int us = unit % kUnits;
                mbar_wait(bar_ufull + 8 * us, (unit / kUnits) & 1, wc, kErrDkv + 5, kPollSleepNs);
                tc_fence_after_sync();
                // Blocks 0, 1: every row is real (d = 256 blk + 128 rank + row).  Block 2: 64 rows, d 512..575 in both CTAs; lanes 0-63 hold
                // them for the first 64 keys of the tile, lanes 64-127 for the others.  Each CTA drains one half, the warps that have
                // that half's indices; which one changes from tile to tile, so that the four sub-partitions have the same to do.
                const int half = (static_cast<int>(n) ^ static_cast<int>(rank)) & 1;
                const bool mine = blk < 2 || (e == half && (quarter >> 1) == half);
                if (mine) {
                    const int d = blk < 2 ? 256 * blk + 128 * static_cast<int>(rank) + quarter * 32 + lane : 512 + (quarter & 1) * 32 + lane;
                    float* out = p.dKV + d;
                    // staged form: the row of slot (query, first key of this warp's 64) in the staging buffer
                    float* sout = nullptr;
                    if constexpr (kStaged)
                        sout = p.staging + (static_cast<size_t>(sq) * p.topk_pad + tile * kTileKeys + 64 * e) * kDQK + d;
                    const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + us * 128 + (blk < 2 ? 64 * e : 0);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (left <= 32 * i) break;      // behind the last slot in use: a predicated-off reduction costs its issue
                        uint32_t r[32];
                        tmem_ld_32x32(taddr + 32 * i, r);
                        int ix[32];
#pragma unroll
                        for (int v = 0; v < 8; ++v) {
                            const int4 t = reinterpret_cast<const int4*>(idx_s)[8 * i + v];
                            ix[4 * v] = t.x; ix[4 * v + 1] = t.y; ix[4 * v + 2] = t.z; ix[4 * v + 3] = t.w;
                        }
                        tmem_ld_wait();
                        if constexpr (kStaged) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                st_global_f32_if_row(sout + static_cast<size_t>(32 * i + j) * kDQK, __uint_as_float(r[j]), ix[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                red_add_f32_if_row(out + static_cast<size_t>(static_cast<unsigned>(ix[j])) * kDQK,
                                                   __uint_as_float(r[j]), ix[j], pol_keep);
                        }
                    }
                }
                // the accumulator reads have completed (tcgen05.wait::ld), which is all the issuer needs to know
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_relaxed(uempty0 + 8 * us);
            }
        }
    }
    abort_wind_down(s_abort);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();          // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 1) tmem_dealloc_2cta(tmem, 512);
}


// =============================================================================================
// Reproducible dKV, second half: one warp per kv row walks the row's slots in the index inverse (CSR by kv row, flat
// slot ids ascending) and adds their staged [576] contributions in that order, so a row's sum is rounded the same way
// in every run.  A pass covers the queries [q_lo, q_hi); a row's slots of that range are a contiguous piece of its
// CSR segment (found by binary search), and passes follow one another in a fixed order.  Bound by reading the staging
// rows once: four rows of 2304 bytes in flight per warp (with two, in 4-byte loads: 4.3 TB/s; now 5.7).
// =============================================================================================
// Two blocks an SM go through the rows: all of them are there from the start, so the dQ kernel behind this one, which needs nothing of it,
// comes up beside the last rows.  1024 queries x 64 heads x top-k 2048 2677 -> 2590 us, 300 x 128 x 1000 572 -> 548, 40 x 128 x 512 84.8 ->
// 73.4, 1000 x 64 x 128 on 60000 rows 428 -> 380.  With one block, and dQ CTAs beside it throughout, too little is in flight (3147).
constexpr int kFlight = 4;
constexpr int kSegThreads = 256;
__global__ void __launch_bounds__(kSegThreads) smla_dkv_segment_sum_kernel(const int* __restrict__ row_ptr,
                                                                           const int* __restrict__ entries,
                                                                           const float* __restrict__ staging, float* __restrict__ dKV,
                                                                           int s_kv, int topk, int topk_pad, int q_lo, int q_hi) {
    const int lane = threadIdx.x & 31;
    pdl_wait();                   // the staging rows
    pdl_trigger();
    for (int row = blockIdx.x * (kSegThreads / 32) + (threadIdx.x >> 5); row < s_kv; row += gridDim.x * (kSegThreads / 32)) {
        const int b = __ldg(row_ptr + row), e = __ldg(row_ptr + row + 1);
        auto lower = [&](long long flat) {      // first position in [b, e) whose flat slot id is >= flat
            int lo = b, hi = e;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(entries + mid) < flat) lo = mid + 1;
                else hi = mid;
            }
            return lo;
        };
        const int i0 = lower(static_cast<long long>(q_lo) * topk), i1 = lower(static_cast<long long>(q_hi) * topk);
        if (i1 <= i0) continue;
        constexpr int kPer = kDQK / 64;          // nine pairs of elements per lane
        float2 acc[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) acc[k] = make_float2(0.f, 0.f);
        for (int c = i0; c < i1; c += 32) {      // a lane locates one of the next 32 slots, the warp adds them in order
            const int n = min(32, i1 - c);
            unsigned long long mine = 0;
            if (lane < n) {
                const int flat = __ldg(entries + c + lane);
                const int q = flat / topk;
                mine = reinterpret_cast<unsigned long long>(staging + (static_cast<size_t>(q - q_lo) * topk_pad + (flat - q * topk)) * kDQK);
            }
            for (int j = 0; j < n; j += kFlight) {
                float2 v[kFlight][kPer];
#pragma unroll
                for (int u = 0; u < kFlight; ++u) {
                    const unsigned long long src = __shfl_sync(0xffffffffu, mine, min(j + u, 31));
                    if (j + u < n) {
#pragma unroll
                        for (int k = 0; k < kPer; ++k) v[u][k] = __ldcs(reinterpret_cast<const float2*>(src) + lane + 32 * k);
                    }
                }
#pragma unroll
                for (int u = 0; u < kFlight; ++u)
                    if (j + u < n) {
#pragma unroll
                        for (int k = 0; k < kPer; ++k) {
                            acc[k].x += v[u][k].x;
                            acc[k].y += v[u][k].y;
                        }
                    }
            }
        }
        float2* out = reinterpret_cast<float2*>(dKV + static_cast<size_t>(row) * kDQK) + lane;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            float2 x = out[32 * k];
            x.x += acc[k].x;
            x.y += acc[k].y;
            out[32 * k] = x;
        }
    }
}

// =============================================================================================
// dq: one CTA per (query, d-part of three column chunks); 14 warps; two CTAs per SM, so that one's start-up (TMEM,
// first gathers) and epilogue run under the other's tiles.
//   warps 0-3   epilogue: TMEM -> bf16 -> dQ[q, head, d]; lane = head (64 heads: sixteen in the lower lanes of every warp), so a
//               thread stores whole 64-byte pieces of its head's row
//   warps 4-11  producers: per 64-key tile the part's columns of the kv rows picked by index (16-byte
//               cp.async into the swizzled layout)
//   warp 13     TMA: the dS scratch tile
//   warp 12     UMMA issuer: acc[128 heads, d of the part] += dS^T . Kg  (both operands MN-major: the key index is
//               the contraction and runs along shared-memory rows).  Heads are the M side so that N can be the 192
//               columns of the part.  64 heads use M = 64: as fast in cycles as M = 128 with 64 rows to spare, but these
//               cost power, and long calls run at the power cap: 4096 queries x 64 heads x top-k 2048 back to back 1207 ->
//               1048 us for the kernel, 6064 -> 5917 for the call; 777 x 64 x 600 402 -> 388.
// With few queries a cluster of up to eight CTAs splits the keys of one (query, d-part) and adds up in rank order.
// =============================================================================================
namespace dq {
constexpr int kThreads = 448;
constexpr int kProducerWarps = 8;
constexpr int kTileKeys = 64;
constexpr int kParts = kQChunks / kDqChunks;
// kDeep: one CTA per SM with as many stages as its shared memory holds, for launches that do not give every SM two CTAs: with
// two stages a CTA alone on its SM waits for its gathers, 1300 cycles a tile against 625 of shared-memory traffic.  Calls of 37 queries
// x 128 heads x top-k 2048 117.4 -> 104.9 us, 27 x 64 heads 96.0 -> 91.8, 12 x 128 heads 58.1 -> 54.9, 3 x 128 40.2 -> 38.8.
template <int HP, bool kDeep> struct Cfg {
    static constexpr int kStages = kDeep ? (HP == 64 ? 6 : 5) : HP == 64 ? 3 : 2;      // (not deep: what fits twice into an SM's shared memory)
    static constexpr int kKgBytes = kDqChunks * 8192;
    static constexpr int kDsBytes = (HP / 64) * 8192;
    static constexpr int kStage = kKgBytes + kDsBytes;     // dS right after Kg
    static constexpr int kOffMisc = kStages * kStage;
    static constexpr int kSmemBytes = kOffMisc + 256 + 1024;
    static_assert((kDeep ? 1 : 2) * (kSmemBytes + 1024) <= 233472, "one or two CTAs per SM");
    static constexpr int kTmemCols = 256;                  // up to 256 columns of d; two CTAs share the SM's 512
    static constexpr int kRowBytes = kDqChunks * 128 + 16;    // epilogue staging of one head's row
    static_assert(128 * kRowBytes <= kOffMisc, "the epilogue stages its rows in the pipeline's memory");
    // keys of a query split over a cluster: every CTA leaves its fp32 accumulator [heads][columns] in the pipeline's memory for
    // the others to read (rows 16 bytes apart modulo 128: conflict-free 16-byte accesses)
    static constexpr int kPartPitch = kDqChunks * 64 + 4;
    static_assert(!kDeep || HP * kPartPitch * 4 <= kOffMisc, "the accumulator of a split query");
};
}  // namespace dq

template <int HP, bool kDeep>
__global__ void __launch_bounds__(dq::kThreads, kDeep ? 1 : 2)
smla_dq_kernel(const __grid_constant__ CUtensorMap tm_ds, const KParams p) {
    using namespace dq;
    using C = Cfg<HP, kDeep>;
    constexpr int kStages = C::kStages;
    // the CTAs of a cluster (usually one) share a (query, d-part) and split its keys
    const int nz = static_cast<int>(cluster_nctas()), z = static_cast<int>(cluster_ctarank());
    const int unit = static_cast<int>(blockIdx.x) / nz;
    const int part = unit % kParts;
    const int ql = unit / kParts;
    const int qg = p.q0 + ql;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform to the compiler
    const int lane = threadIdx.x & 31;
    const int chunk0 = part * kDqChunks;      // first kv column chunk of the d-part

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t s_base = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffMisc);
    const uint32_t bar_full = smem_u32(bars);             // [kStages]
    const uint32_t bar_empty = bar_full + 8 * kStages;    // [kStages]
    const uint32_t bar_acc = bar_empty + 8 * kStages;     // 1
    const uint32_t bar_drain = bar_acc + 8;               // 1  used only while winding down after an abort
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::kOffMisc + 8 * (2 * kStages + 2));
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const WaitCtx wc{p.g_err, s_abort, p.wait_limit, 0u};

    if (threadIdx.x == 0) {
        *s_abort = 0;
        for (int i = 0; i < kStages; ++i) {
            mbar_init(bar_full + 8 * i, kProducerWarps * 32 + 1);   // cp.async threads + the TMA expect_tx arrival
            mbar_init(bar_empty + 8 * i, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_drain, 1);
        fence_mbar_init();
    }
    if (warp == 12) {
        tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    // A chain of small kernels ends here: the next one of the stream may come up to its own wait (64 queries x 16 heads x top-k 64:
    // 20.6 -> 19.6 us).  Large grids keep their SMs to themselves: 37 queries x 128 heads x 2048 116 -> 119 us with it.
    // Not before this CTA has its tensor memory: a block of the next kernel that fits beside it could take all of it and then wait for
    // this grid to end, which waits for its share.
    if (p.every_slot) pdl_trigger();
    // Behind the dKV kernel's trigger everything this kernel reads is in place already (that kernel triggers after it has
    // waited for the recompute kernel), so its CTAs fill whatever SMs the dKV kernel leaves; the last CTA then holds the
    // grid open until the dKV kernel is done, so that "dq done" still means "all done" to whatever follows.
    if (!p.early_start) pdl_wait();
    const int n_all = __shfl_sync(0xffffffffu, (slots_used(p, qg) + kTileKeys - 1) / kTileKeys, 0);
    const int tile0 = n_all * z / nz, n_tiles = n_all * (z + 1) / nz - tile0;

    if (warp >= 4 && warp < 12) {
        const int pt = threadIdx.x - 128;   // 0..255
        const int u = pt & 7;
        const int r0 = pt >> 3;             // rows r0 and r0+32 of the tile
        const uint32_t dst0 = s_base + r0 * 128 + ((u ^ (r0 & 7)) << 4);
        const char* kvb = reinterpret_cast<const char*>(p.kv) + chunk0 * 128 + u * 16;
        const uint64_t pol_keep = l2_policy_evict_last();
        // the indices of a tile are loaded one tile ahead, so that their latency is never in front of the copies
        // (raw values, turned into kv rows when they are used: nothing may depend on a load here)
        int idx_next[2];
        const QMeta qm = load_qmeta(p, qg);
        auto load_idx = [&](int tile) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int key = (tile0 + tile) * kTileKeys + r0 + 32 * i;
                idx_next[i] = (tile < n_tiles && key < p.topk) ? __ldg(p.indices + static_cast<size_t>(qg) * p.topk + key) : -1;
            }
        };
        load_idx(0);
        int s = 0;
        uint32_t ph = 1;                    // parity that means "stage free" for the current pass over the ring
        for (int tile = 0; tile < n_tiles; ++tile) {
            const char* src[2];
            uint32_t nb[2];   // 0: the slot takes no part, read nothing and land zeros (no shared stand-in row: it would be a hot spot)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = gather_row(idx_next[i], (tile0 + tile) * kTileKeys + r0 + 32 * i, qm, p);
                nb[i] = row >= 0 ? 16u : 0u;
                src[i] = kvb + static_cast<size_t>(row >= 0 ? row : 0) * (kDQK * 2);
            }
            load_idx(tile + 1);
            mbar_wait(bar_empty + 8 * s, ph, wc, kErrDq + 1, kPollSleepNs);
            const uint32_t d = dst0 + s * C::kStage;
#pragma unroll
            for (int c = 0; c < kDqChunks; ++c) {
                cp_async16_zfill_hint(d + c * 8192, src[0] + c * 128, nb[0], pol_keep);
                cp_async16_zfill_hint(d + c * 8192 + 32 * 128, src[1] + c * 128, nb[1], pol_keep);
            }
            cp_async_mbar_arrive_noinc(bar_full + 8 * s);
            if (++s == kStages) {
                s = 0;
                ph ^= 1;
            }
        }
    } else if (warp == 13) {
        if (lane == 0) tma_prefetch_desc(&tm_ds);
        const uint64_t pol_stream = l2_policy_evict_first();
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 1;
            for (int tile = 0; tile < n_tiles; ++tile) {
                mbar_wait(bar_empty + 8 * s, ph, wc, kErrDq + 4, kPollSleepNs);
                const uint32_t dst = s_base + s * C::kStage;
                mbar_arrive_expect_tx(bar_full + 8 * s, C::kDsBytes);
                // box = 64 keys of every head block -> [HP/8][64 keys][8 heads]
                tma_load_4d_hint(dst + C::kKgBytes, &tm_ds, 0, (tile0 + tile) * (kTileKeys / 32), 0, p.scr0 + ql, bar_full + 8 * s, pol_stream);
                if (++s == kStages) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 12) {
        if (elect_one()) {
            constexpr uint32_t idesc1 = make_idesc_bf16(HP, kDqChunks * 64, 1, 1);     // N = the part's columns in one UMMA
            // A = dS^T: [HP/8 head blocks][64 keys][8 heads], 8-key groups 128 B apart, head blocks 1 KB apart.
            // Descriptors: the fixed fields once, the address (16-byte units, the low 14 bits) added per UMMA.
            const uint64_t a_hi = make_smem_desc(0, 128, 1024, kSwizzleNone) & 0xFFFFFFFF00000000ull;
            const uint32_t a_lo0 = static_cast<uint32_t>(make_smem_desc(0, 128, 1024, kSwizzleNone)) + desc_addr(s_base + C::kKgBytes);
            const uint64_t b_hi = make_smem_desc(0, 8192, 1024, kSwizzle128) & 0xFFFFFFFF00000000ull;
            const uint32_t b_lo0 = static_cast<uint32_t>(make_smem_desc(0, 8192, 1024, kSwizzle128)) + desc_addr(s_base);
            RingReader<kStages> ring(bar_full);
            for (int tile = 0; tile < n_tiles; ++tile) {
                ring.wait(wc, kErrDq + 2);
                const uint32_t s = ring.slot;
                ring.next();
                fence_proxy_async_smem();
                tc_fence_after_sync();
                const uint32_t a_lo = a_lo0 + s * (C::kStage >> 4), b_lo = b_lo0 + s * (C::kStage >> 4);
#pragma unroll
                for (int ks = 0; ks < kTileKeys / 16; ++ks) {
                    const uint64_t a = a_hi | (a_lo + ks * (256 >> 4));
                    umma_ss(tmem, a, b_hi | (b_lo + ks * (2048 >> 4)), idesc1, (tile | ks) != 0);
                }
                umma_commit(bar_empty + 8 * s);
            }
            umma_commit(bar_acc);
            if (*s_abort) {   // winding down: nothing of this thread's may still be in the tensor pipe at dealloc
                umma_commit(bar_drain);
                mbar_wait_drain(bar_drain, 0, p.wait_limit);
            }
        }
    } else {
        const int quarter = warp;
        mbar_wait(bar_acc, 0, wc, kErrDq + 3, kPollSleepNs);
        tc_fence_after_sync();
        const uint32_t zero_mask = n_tiles > 0 ? 0xFFFFFFFFu : 0u;      // no tile at all: the accumulator was never written
        // lane = head, columns = d of the part.  Each thread converts its head's row to bf16 in shared memory (the
        // pipeline stages are idle by now; rows 16 bytes apart modulo 128 so that the 16-byte stores of a warp
        // spread over all banks) and sends it off as one bulk copy: whole cache lines instead of 32 scattered
        // 16-byte pieces per store instruction.
        constexpr int kRowBytes = C::kRowBytes;
        // 128 heads: one per lane; 64 (UMMAs of M = 64): sixteen in the lower lanes of every quarter
        constexpr int kQuarterHeads = HP / 4;
        const int head = quarter * kQuarterHeads + (lane & (kQuarterHeads - 1));
        const bool real = lane < kQuarterHeads && head < p.h_q;
        const uint32_t row_s = s_base + head * kRowBytes;
        const uint32_t taddr = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
        if (kDeep && nz > 1) {
            if (quarter * kQuarterHeads < p.h_q) {
                const uint32_t part_s = s_base + head * (C::kPartPitch * 4);
#pragma unroll 1
                for (int cg = 0; cg < kDqChunks * 4; ++cg) {
                    uint32_t r[16];
                    tmem_ld_32x16(taddr + cg * 16, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        if (lane < kQuarterHeads)
                            st_shared_v4(part_s + cg * 64 + v * 16, r[4 * v] & zero_mask, r[4 * v + 1] & zero_mask, r[4 * v + 2] & zero_mask,
                                         r[4 * v + 3] & zero_mask);
                }
            }
        } else if (quarter * kQuarterHeads < p.h_q) {        // warp-uniform: heads are padded to a multiple of 8 only
#pragma unroll 1
            // 32 columns at a time: two CTAs per SM leave 64 registers a thread (16 at a time: 64 queries x 16 heads x top-k 64
            // 19.64 against 19.43 us, larger calls alike)
            for (int cg = 0; cg < kDqChunks * 2; ++cg) {
                uint32_t r[32];
                tmem_ld_32x32(taddr + cg * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] &= zero_mask;
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (lane < kQuarterHeads) st_shared_v4(row_s + cg * 64 + v * 16,
                                 pack_bf16x2(__uint_as_float(r[8 * v]), __uint_as_float(r[8 * v + 1])),
                                 pack_bf16x2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3])),
                                 pack_bf16x2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5])),
                                 pack_bf16x2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7])));
            }
            if (real) {
                fence_proxy_async_smem();         // this thread's row only: no one else touches it
                // (first out of the L2: dQ streams by kv rows and dS that are read again.  100 x 128 heads x 600 82.6 -> 81.9 us a call, 1531 x 128
                // x 141 477 -> 472, 4096 x 128 x 2048 8262 -> 8225)
                bulk_store_hint(p.dQ + (static_cast<size_t>(qg) * p.h_q + head) * kDQK + chunk0 * 64, row_s, kDqChunks * 128, l2_policy_evict_first());
                bulk_commit();
                bulk_wait_read();
            }
        }
    }
    abort_wind_down(s_abort);
    if (p.early_start && blockIdx.x == gridDim.x - 1) pdl_wait();
    tc_fence_before_sync();
    __syncthreads();
    if (kDeep && nz > 1) {
        // every CTA adds up its share of the heads, always in rank order
        cluster_sync_all();
        constexpr int kGroups = kDqChunks * 8;   // 8 columns at a time
        const int h0 = p.h_q * z / nz, h1 = p.h_q * (z + 1) / nz;
        for (int i = threadIdx.x; i < (h1 - h0) * kGroups; i += kThreads) {
            const int h = h0 + i / kGroups, c = (i % kGroups) * 8;
            const uint32_t at = s_base + (h * C::kPartPitch + c) * 4;
            float acc[8] = {};
            for (int r = 0; r < nz; ++r) {
                const uint32_t a = map_to_cta(at, r);
                const float4 lo = ld_cluster_v4(a), hi = ld_cluster_v4(a + 16);
                acc[0] += lo.x; acc[1] += lo.y; acc[2] += lo.z; acc[3] += lo.w;
                acc[4] += hi.x; acc[5] += hi.y; acc[6] += hi.z; acc[7] += hi.w;
            }
            *reinterpret_cast<uint4*>(p.dQ + (static_cast<size_t>(qg) * p.h_q + h) * kDQK + chunk0 * 64 + c) =
                make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                           pack_bf16x2(acc[6], acc[7]));
        }
        cluster_sync_all();                      // nobody leaves while another still reads its part
    }
    if (warp == 12) tmem_dealloc(tmem, C::kTmemCols);
}

// =============================================================================================
// Self-test of the bounded waits: one CTA waits on a barrier (or a counter) that nothing ever signals, with a
// short limit.  The wait must give up, record `code`, raise the abort flag, and the kernel must return
// normally; a second wait must then return at once.  out[0] = what the first wait returned, out[1] = what
// the second returned, out[2] = cycles the first wait took.
// =============================================================================================
__global__ void __launch_bounds__(32) smla_selftest_wait_kernel(int* g_err, long long* out, int which, long long limit,
                                                                int code) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    __shared__ uint32_t counter;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        counter = 0;
        mbar_init(smem_u32(&bar), 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const WaitCtx wc{g_err, &abort_flag, limit, 0u};
        const long long t0 = clock64();
        bool a;
        if (which == 0) a = mbar_wait(smem_u32(&bar), 0, wc, code, kPollSleepNs);
        else if (which == 1) a = mbar_spin(smem_u32(&bar), 0, wc, code);
        else a = flag_wait(smem_u32(&counter), 1u, wc, code);
        const long long t1 = clock64();
        const bool b = mbar_wait(smem_u32(&bar), 0, wc, code + 1);
        out[0] = a ? 1 : 0;
        out[1] = b ? 1 : 0;
        out[2] = t1 - t0;
    }
}

}  // namespace smla
