// Batched execution of many light queries: one persistent launch per plan
// step over a packed multi-query history, replayed as a CUDA graph.
//
// The batch holds up to max_queries queries of up to max_steps patterns each,
// every query starting from a constant (Engine::const_to_unknown,
// core/engine.hpp:96-122) and continuing with known_to_unknown /
// known_to_known / known_to_const steps (core/engine.hpp:126-225).  A query
// with fewer patterns passes its table through the remaining steps.
//
// Packed layout (device, per step, ping-pong A/B):
//   row_off[q]  first row of query q in the step's global row order (Q+1)
//   int_off[q]  first int32 of query q's table in the packed buffer
//   cols[q]     column count of query q's table
// Step kernels:
//   batch_count : per (query,row): probe with the query's own predicate
//                 (lanes of one warp may probe different segments), output
//                 row count (degree, or 0/1 for a filter, 1 for a pass),
//                 per-tile sums and per-query sums (warp-aggregated atomics)
//   batch_scan  : two blocks: exclusive scans of tile sums and of per-query
//                 output rows / ints -> next step's layout; capacity check
//   batch_write : per tile: warp scan of the counts, then every output row
//                 written at out_int_off[q] + pos_in_q * width; rows whose
//                 output exceeds `split` ints are written warp-cooperatively,
//                 the rest thread-per-row
//
// A tile is the rows one warp takes: total / warps of the grid, from one row
// up (rows_per_tile).  Light steps are bound by latency, not by bytes: 4096
// start rows with lists of 100 are 128 warps of 32 rows, or 4 blocks of 1024,
// that walk their lists one after another, but 4096 warps that walk one list
// each.  A batch of 4096 light requests (packed, run, results on the host)
// took 559 us with tiles of 1024 rows a block, 208 so.
// The three phases run either as three kernels per step or as one
// cooperative persistent kernel per step (batch_step_kernel) whose blocks
// meet at two grid barriers -- after the count and after the scan, which
// the first and last block run -- each wait bounded; the autotuner picks the faster.  Every
// size lives in device memory and every grid is persistent, so the launch
// sequence of a batch never depends on its data: it is captured once into a
// CUDA graph and replayed for each new batch.  Each query's rows come out in
// exactly the order the query produces alone.
#include <algorithm>
#include <cstring>
#include <unordered_map>
#include <vector>

#include "wk_probe.cuh"
#include "wk_runtime.h"

namespace wk {
namespace dev {

#define FULL 0xffffffffu

enum { BK_K2U = 0, BK_K2K = 1, BK_K2C = 2, BK_C2U = 3, BK_NOP = 4 };

struct StepDesc {
    int32_t kind, pid, dir, scol, ecol, cst;   // cst: constant start (c2u) or constant end (k2c)
};

struct BatchTune {
    int blocks_per_sm;   // persistent grid = SMs x blocks_per_sm
    int rounds;          // rows per warp per tile = 32 * rounds
    int split;           // output ints above which a row is written by a whole warp
    int fused;           // 1: one cooperative kernel per step; 0: count, scan and write kernels
    int bt;              // threads per block of the step kernels: 128 or 256
};

constexpr int kErrBarrier = 1 << 4;         // flags[0]: a grid-barrier wait ran out
constexpr long kBarrierIters = 1l << 24;    // polls of a grid-barrier wait (about 1 s with the back-off)

constexpr int kBTMax = 256;                 // the larger of the two block sizes (128, 256 threads)
constexpr int kMaxBlocksPerSm = 16;
constexpr int kMaxQ = 4096;                 // queries per batch

// largest q with off[q] <= g (off: the step's input row offsets, Q + 1 of
// them, read through L1)
__device__ __forceinline__ int find_query(const int64_t *off, int Q, int64_t g) {
    int lo = 0, hi = Q - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ld_prior(off + mid) <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// As find_query for one row by a whole warp: each round asks 32 pivots with
// one load, so 4096 queries take three dependent loads instead of twelve (the
// step kernels are chains of such loads, each starting with a cold L1).
__device__ __forceinline__ int find_query_warp(const int64_t *off, int Q, int64_t g, int lane) {
    int lo = 0, n = Q;
    while (n > 1) {
        const int step = (n + 31) >> 5, i = lane * step;
        const unsigned m = __ballot_sync(FULL, i < n && ld_prior(off + lo + i) <= g);
        const int k = 31 - __clz((int)m);   // off is ascending: the pivots at or below g come first
        lo += k * step;
        n = n - k * step < step ? n - k * step : step;
    }
    return lo;
}

// The queries of 32 consecutive rows g0 + lane, whose first belongs to q0: the
// boundaries of the next 32 queries, one per lane, searched by shuffles; rows
// past them (behind that many empty queries) search on their own.
__device__ __forceinline__ int find_queries(const int64_t *off, int Q, int64_t g0, int q0, int lane) {
    const int64_t rel = q0 + 1 + lane < Q ? ld_prior(off + q0 + 1 + lane) - g0 : 64;
    const int p = rel < 64 ? (int)rel : 64;   // > 0: q0 is the last query that begins at or before g0
    int k = 0;                                // boundaries at or before row g0 + lane
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(FULL, p, k + s - 1) <= lane) k += s;
    if (__shfl_sync(FULL, p, k) <= lane) ++k;
    if (k == 32) return find_query(off, Q, g0 + lane);
    return q0 + k;
}

// Rows per tile of a step of `total` rows on a grid of `warps` warps: as many
// as give every warp a tile (a power of two below 32, then a multiple of 32),
// at most 32 x rounds.
__host__ __device__ __forceinline__ int rows_per_tile(int64_t total, int64_t warps, int rounds) {
    const int64_t need = (total + warps - 1) / warps;
    if (need >= 32) {
        const int64_t r = (need + 31) / 32;
        return 32 * (int)(r < rounds ? r : rounds);
    }
    int rho = 1;
    while (rho < need) rho *= 2;
    return rho;
}

__device__ __forceinline__ bool b_contains(const int32_t *e, uint32_t n, int32_t v) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(e + mid) < v) lo = mid + 1;
        else hi = mid;
    }
    return lo < n && __ldg(e + lo) == v;
}

struct StepIO {
    const int32_t *hist;
    int32_t *out;
    const int64_t *in_row_off, *in_int_off;
    const int32_t *in_cols;
    int64_t *out_row_off, *out_int_off;
    int32_t *out_cols;
    const StepDesc *desc;     // [Q]
    const PredView *pvs;      // [num_ids + 1]
    uint32_t *cnt, *off;      // per input row
    unsigned long long *tile_sum;   // per tile
    unsigned long long *q_rows;     // per query output rows (zeroed by the scan)
    int *flags;               // [0] error bits, [1] overflow
    int32_t *pub;             // last step: pinned words for the flags and the layout behind them, or null
    int64_t cap_ints, cap_rows;
    int Q;
    int64_t warps;            // of the count and write grids
};

// tiles of a step and this warp's: warp w of block b takes tiles b + w G,
// + G BT / 32, ... (G blocks), so few tiles spread over the blocks
__device__ __forceinline__ int64_t first_tile() {
    return (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}

__device__ __forceinline__ unsigned long long warp_scan(unsigned long long v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long x = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += x;
    }
    return v;
}

// count: per (query, row) output counts, per-tile and per-query sums
template <int BT>
__device__ __forceinline__ void count_phase(const StepIO &io, int rounds) {
    const int lane = threadIdx.x & 31;
    const int64_t total = ld_prior(io.in_row_off + io.Q);
    const int rho = rows_per_tile(total, io.warps, rounds);
    const int64_t ntiles = (total + rho - 1) / rho;
    for (int64_t tile = first_tile(); tile < ntiles; tile += (int64_t)gridDim.x * (BT / 32)) {
        unsigned long long my = 0ull;
        int q0 = find_query_warp(io.in_row_off, io.Q, tile * rho, lane);
        for (int r0 = 0; r0 < rho && tile * rho + r0 < total; r0 += 32) {
            const int64_t g = tile * rho + r0 + lane;
            const bool valid = r0 + lane < rho && g < total;
            const int q = find_queries(io.in_row_off, io.Q, g - lane, q0, lane);
            q0 = __shfl_sync(FULL, q, 31);   // the next window's row may begin a later query: found from here
            StepDesc d{BK_NOP, 0, 0, 0, 0, 0};
            if (valid) d = io.desc[q];
            PredView pv{};
            int32_t vid = -1;
            bool probe = valid && d.kind != BK_NOP;
            int32_t target = 0;
            if (probe) {
                pv = io.pvs[d.pid];
                if (d.kind == BK_C2U) {
                    vid = d.cst;
                } else {
                    const int64_t r = g - ld_prior(io.in_row_off + q);
                    const int32_t *row = io.hist + io.in_int_off[q] + r * io.in_cols[q];
                    vid = ld_prior(row + d.scol);
                    target = d.kind == BK_K2K ? ld_prior(row + d.ecol) : d.cst;
                }
            }
            uint32_t o = 0u, deg = 0u;
            if (__any_sync(FULL, probe))
                probe_warp_multi(pv, (uint32_t)d.pid, probe, vid, (uint32_t)d.dir, o, deg, io.flags);
            uint32_t c = 0u;
            if (valid) {
                if (d.kind == BK_NOP) c = 1u;
                else if (d.kind == BK_K2U || d.kind == BK_C2U) c = deg;
                else c = (deg > 0u && b_contains(pv.edges + o, deg, target)) ? 1u : 0u;
                io.cnt[g] = c;
                io.off[g] = o;
            }
            // per-query sums, one atomic per distinct query in the warp
            const unsigned grp = __match_any_sync(FULL, valid ? q : -1);
            unsigned long long qs = c;
            // sum within the group: lanes of a group are contiguous (rows of one query)
            for (int sh = 16; sh > 0; sh >>= 1) {
                const unsigned long long v = __shfl_down_sync(FULL, qs, sh);
                if (lane + sh < 32 && ((grp >> (lane + sh)) & 1u)) qs += v;
            }
            // after the down-sweep the lowest lane of each contiguous group holds its total
            if (valid && (__ffs(grp) - 1) == lane && qs) atomicAdd(&io.q_rows[q], qs);
            my += c;
        }
        for (int o2 = 16; o2 > 0; o2 >>= 1) my += __shfl_xor_sync(FULL, my, o2);
        if (lane == 0) io.tile_sum[tile] = my;
    }
}

// Programmatic dependent launch: the step kernels are placed while the kernel
// before them ends, and each waits for it before reading anything.
__device__ __forceinline__ void after_prior_kernel() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

template <int BT>
__global__ void __launch_bounds__(BT)
batch_count_kernel(StepIO io, int rounds) {
    after_prior_kernel();
    if (io.flags[1]) return;
    count_phase<BT>(io, rounds);
}

// Exclusive scan of the threads' values over the block (any multiple of 32
// threads up to 1024), and their sum.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long v, unsigned long long *ws,
                                                         unsigned long long &all) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const unsigned long long in = warp_scan(v, lane);
    if (lane == 31) ws[wid] = in;
    __syncthreads();
    const unsigned long long x = warp_scan(lane < nw ? ws[lane] : 0ull, lane);   // in every warp
    all = __shfl_sync(FULL, x, 31);
    const unsigned long long before = __shfl_sync(FULL, x, wid > 0 ? wid - 1 : 0);
    __syncthreads();   // ws is free again
    return in - v + (wid > 0 ? before : 0ull);
}

// The scan's two parts, each one block's work: the tiles' prefix sums, and the
// queries' output layout with the capacity check.  One SM's memory
// transactions and the chain of its loads bound them, so they run on two SMs, a
// thread takes neighbouring entries of its neighbours (pairs of tiles, single
// queries: whole sectors), and a pass's loads are issued together.  (Both on
// one SM, four consecutive queries a thread and 8 B stores 32 B apart: 14.5 us
// for 4096 queries; on one SM 11.5; this 9.)  The one-kernel step reads here
// and in the write phase what other blocks wrote in the same launch: past L1.
constexpr int kScanPer = 4;   // loads in flight
__device__ __forceinline__ void scan_tiles(const StepIO &io, int rounds, unsigned long long *ws) {
    const int nt = blockDim.x, t = threadIdx.x;
    const int64_t total = ld_prior(io.in_row_off + io.Q);
    const int rho = rows_per_tile(total, io.warps, rounds);
    const int64_t n = (total + rho - 1) / rho;
    unsigned long long carry = 0ull;
    for (int64_t i0 = 0; i0 < n; i0 += 2 * kScanPer * (int64_t)nt) {
        ulonglong2 p[kScanPer];
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int64_t i = i0 + 2 * ((int64_t)k * nt + t);   // the buffer holds an even number of tiles
            p[k] = i < n ? ld_l2(reinterpret_cast<const ulonglong2 *>(io.tile_sum + i)) : make_ulonglong2(0ull, 0ull);
            if (i + 1 >= n) p[k].y = 0ull;
        }
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int64_t i = i0 + 2 * ((int64_t)k * nt + t);
            if (i0 + 2 * (int64_t)k * nt >= n) break;   // the same in every thread
            unsigned long long all;
            const unsigned long long e = carry + block_scan(p[k].x + p[k].y, ws, all);
            if (i < n) *reinterpret_cast<ulonglong2 *>(io.tile_sum + i) = make_ulonglong2(e, e + p[k].x);
            carry += all;
        }
    }
}

__device__ __forceinline__ void scan_queries(const StepIO &io, unsigned long long *ws) {
    const int nt = blockDim.x, t = threadIdx.x;
    const int Q = io.Q;
    unsigned long long row_at = 0ull, int_at = 0ull;
    for (int q0 = 0; q0 < Q; q0 += kScanPer * nt) {
        unsigned long long r[kScanPer];
        int w[kScanPer];
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int q = q0 + k * nt + t;
            r[k] = 0ull;
            w[k] = 0;
            if (q < Q) {
                const int kind = io.desc[q].kind, cols = io.in_cols[q];
                r[k] = ld_l2(io.q_rows + q);
                w[k] = kind == BK_K2U ? cols + 1 : (kind == BK_C2U ? 1 : cols);
            }
        }
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int q = q0 + k * nt + t;
            if (q0 + k * nt >= Q) break;   // the same in every thread
            unsigned long long ar, ai;
            const unsigned long long er = block_scan(r[k], ws, ar), ei = block_scan(r[k] * (unsigned long long)w[k], ws, ai);
            if (q < Q) {
                io.out_row_off[q] = (int64_t)(row_at + er);
                io.out_int_off[q] = (int64_t)(int_at + ei);
                io.out_cols[q] = w[k];
                io.q_rows[q] = 0ull;   // the next step's count kernel accumulates afresh
            }
            row_at += ar;
            int_at += ai;
        }
    }
    if (t == 0) {
        io.out_row_off[Q] = (int64_t)row_at;
        if ((int64_t)row_at > io.cap_rows || (int64_t)int_at > io.cap_ints) io.flags[1] = 1;
    }
}

constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads)
batch_scan_kernel(StepIO io, int rounds) {
    __shared__ unsigned long long ws[32];
    after_prior_kernel();
    // Over capacity: nothing of this step is used.  The other block may be finding
    // that out just now, so the block's threads, which meet at barriers below, go by
    // one vote on what they read.
    if (__syncthreads_or(*(volatile int *)(io.flags + 1))) return;
    if (blockIdx.x == 0) scan_tiles(io, rounds, ws);
    else scan_queries(io, ws);
}

// One row's output of nw = c x w ints, by the whole warp: four ints a lane in
// flight, the row and column of each kept by steps of 32 (no division).
__device__ __forceinline__ void write_row_warp(int kind, const int32_t *row, const int32_t *e, int32_t *dst, int cin,
                                               int w, uint32_t c, int lane) {
    const int64_t nw = (int64_t)c * w;
    const uint32_t dr = 32u / (uint32_t)w;
    const int dc = 32 % w;
    uint32_t r = (uint32_t)lane / (uint32_t)w;
    int cc = lane % w;
    for (int64_t x = lane; x < nw; x += 128) {
        int32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (x + 32 * k < nw) {
                if (kind == BK_K2U) v[k] = cc < cin ? __ldg(row + cc) : __ldg(e + r);
                else if (kind == BK_C2U) v[k] = __ldg(e + r);
                else v[k] = __ldg(row + cc);
            }
            r += dr;
            cc += dc;
            if (cc >= w) { cc -= w; ++r; }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (x + 32 * k < nw) dst[x + 32 * k] = v[k];
    }
}

// Per tile: warp scan of the counts, then write.  A row with more than
// `split` output ints -- fewer in tiles below 32 rows, whose other lanes are
// idle -- is written by the whole warp.
template <int BT>
__device__ __forceinline__ void write_phase(const StepIO &io, int rounds, int split) {
    const int lane = threadIdx.x & 31;
    const int64_t total = ld_prior(io.in_row_off + io.Q);
    const int rho = rows_per_tile(total, io.warps, rounds);
    const int64_t ntiles = (total + rho - 1) / rho;
    const int64_t most = rho < 32 ? ((int64_t)split * rho + 31) / 32 : split;
    for (int64_t tile = first_tile(); tile < ntiles; tile += (int64_t)gridDim.x * (BT / 32)) {
        unsigned long long base = ld_l2(io.tile_sum + tile);
        int q0 = find_query_warp(io.in_row_off, io.Q, tile * rho, lane);
        for (int r0 = 0; r0 < rho && tile * rho + r0 < total; r0 += 32) {
            const int64_t g = tile * rho + r0 + lane;
            const int q = find_queries(io.in_row_off, io.Q, g - lane, q0, lane);
            q0 = __shfl_sync(FULL, q, 31);
            const uint32_t c = r0 + lane < rho && g < total ? ld_l2(io.cnt + g) : 0u;
            const unsigned long long inc = warp_scan(c, lane);
            const unsigned long long pos = base + inc - c;
            base += __shfl_sync(FULL, inc, 31);
            int kind = BK_NOP, cin = 0, w = 0;
            const int32_t *row = nullptr, *e = nullptr;
            int32_t *dst = nullptr;
            if (c) {
                const StepDesc d = io.desc[q];
                kind = d.kind;
                cin = io.in_cols[q];
                w = (kind == BK_K2U) ? cin + 1 : (kind == BK_C2U ? 1 : cin);
                row = io.hist + io.in_int_off[q] + (g - ld_prior(io.in_row_off + q)) * cin;
                dst = io.out + ld_l2(io.out_int_off + q) + ((int64_t)pos - ld_l2(io.out_row_off + q)) * w;
                if (kind == BK_K2U || kind == BK_C2U) e = io.pvs[d.pid].edges + ld_l2(io.off + g);
            }
            const bool big = c != 0u && (int64_t)c * w > most;
            if (c != 0u && !big) {
                if (kind == BK_K2U || kind == BK_C2U) {
                    for (uint32_t x = 0; x < c; ++x) {
                        if (kind == BK_K2U) for (int cc = 0; cc < cin; ++cc) dst[cc] = __ldg(row + cc);
                        dst[w - 1] = __ldg(e + x);
                        dst += w;
                    }
                } else {
                    for (int cc = 0; cc < cin; ++cc) dst[cc] = __ldg(row + cc);
                }
            }
            for (unsigned left = __ballot_sync(FULL, big); left; left &= left - 1u) {
                const int src = __ffs(left) - 1;
                write_row_warp(__shfl_sync(FULL, kind, src),
                               reinterpret_cast<const int32_t *>(__shfl_sync(FULL, (unsigned long long)row, src)),
                               reinterpret_cast<const int32_t *>(__shfl_sync(FULL, (unsigned long long)e, src)),
                               reinterpret_cast<int32_t *>(__shfl_sync(FULL, (unsigned long long)dst, src)),
                               __shfl_sync(FULL, cin, src), __shfl_sync(FULL, w, src), __shfl_sync(FULL, c, src), lane);
            }
        }
    }
}

template <int BT>
__global__ void __launch_bounds__(BT)
batch_write_kernel(StepIO io, int rounds, int split) {
    after_prior_kernel();
    // the flags and the final tables' layout, complete since the scan: on their way
    // to the host while the rows are written (by a copy behind the batch, 41 queries
    // took 93 us, 4096 200; this way 84 and 192)
    if (io.pub != nullptr) {
        const int n = 2 * (2 * io.Q + 2) + io.Q;
        for (int i = blockIdx.x * BT + threadIdx.x; i < n; i += gridDim.x * BT) io.pub[i] = ld_l2(io.flags + i);
    }
    if (io.flags[1]) return;
    write_phase<BT>(io, rounds, split);
}

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(unsigned int *p, unsigned int v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid barrier of a cooperative launch: bar[0] counts arrivals, bar[1] is the
// generation.  The block arriving last resets the count and advances the
// generation; the others poll the generation with a back-off,
// at most kBarrierIters times -- a wait that runs out sets kErrBarrier and
// returns false in every thread of the block (the caller then leaves; every
// other block's wait ends the same way, so the launch ends).
__device__ __forceinline__ bool grid_barrier(unsigned int *bar, int *flags) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int gen = ld_acquire(bar + 1);
        __threadfence();   // this block's writes before its arrival
        int ok = 1;
        if (atomicAdd(bar, 1u) + 1u == gridDim.x) {
            atomicExch(bar, 0u);
            __threadfence();
            st_release(bar + 1, gen + 1u);
        } else {
            long it = 0;
            while (ld_acquire(bar + 1) == gen) {
                if (++it > kBarrierIters) {
                    ok = 0;
                    atomicOr(flags, kErrBarrier);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// One step in one cooperative launch: count, barrier, scan (the first and last block),
// barrier, write.  Launched with at most as many blocks as fit on the device
// at once (the cooperative launch refuses more).
template <int BT>
__global__ void __launch_bounds__(BT)
batch_step_kernel(StepIO io, int rounds, int split, unsigned int *bar) {
    if (io.flags[1]) return;             // set before the launch: the same in every block
    count_phase<BT>(io, rounds);
    if (!grid_barrier(bar, io.flags)) return;
    __shared__ unsigned long long ws[32];
    if (blockIdx.x == 0) scan_tiles(io, rounds, ws);
    if (blockIdx.x == gridDim.x - 1) scan_queries(io, ws);   // another block where there are two
    if (!grid_barrier(bar, io.flags)) return;
    if (*(volatile int *)(io.flags + 1)) return;   // this step's scan found the batch over capacity
    write_phase<BT>(io, rounds, split);
}

// The step descriptors from pinned host memory (Q of each of `steps` rows of
// `pitch` 8 B words), and the step-0 layout: every query has one virtual row and
// no columns.  Reading them here takes as long as a copy ahead of this kernel
// (786 KB in 4 us), but a kernel behind a copy starts late: a batch of 4096
// queries took 206 us so, 200 this way.
__global__ void batch_init_kernel(int Q, int64_t *row_off, int64_t *int_off, int32_t *cols,
                                  unsigned long long *q_rows, int *flags, const uint64_t *__restrict__ h_desc,
                                  uint64_t *__restrict__ desc, int64_t pitch, int steps) {
    constexpr int kWords = sizeof(StepDesc) / 8;
    const int64_t row = (int64_t)Q * kWords, n = row * steps;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t at = i / row * pitch + i % row;
        desc[at] = h_desc[at];
    }
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q <= Q; q += gridDim.x * blockDim.x) {
        row_off[q] = q;
        if (q < Q) { int_off[q] = 0; cols[q] = 0; q_rows[q] = 0ull; }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { flags[0] = 0; flags[1] = 0; }
}

}  // namespace dev
}  // namespace wk

using namespace wk;
using namespace wk::dev;

struct wk_batch {
    wk_ctx *ctx = nullptr;
    cudaStream_t stream = nullptr;          // the batch's own stream (batches overlap)
    cudaEvent_t done = nullptr;
    int32_t max_q = 0, max_steps = 0;
    int64_t cap_ints = 0, cap_rows = 0;
    int sms = 0;
    BatchTune tune{4, 4, 64, 0, 256};
    // device
    PredView *d_pvs = nullptr;
    StepDesc *d_desc = nullptr;             // [max_steps][max_q]
    int64_t *d_row_off[2] = {}, *d_int_off[2] = {};
    int32_t *d_cols[2] = {};
    int32_t *d_hist[2] = {};
    uint32_t *d_cnt = nullptr, *d_off = nullptr;
    unsigned long long *d_tile = nullptr, *d_qrows = nullptr;
    int *d_flags = nullptr;                 // d_block
    unsigned int *d_bar = nullptr;          // grid barrier of the one-kernel steps (count, generation)
    // host (pinned), read by the first kernel of a batch
    StepDesc *h_desc = nullptr, *h_desc_dev = nullptr;
    // the flags (one word) and the final tables' layout -- row_off (Q+1), int_off
    // (Q), cols as int32 (Q) -- on the device, and their pinned copy
    int64_t *d_block = nullptr, *h_block = nullptr;
    int32_t *h_block_dev = nullptr;         // the copy's device address
    int64_t *h_layout = nullptr;            // h_block + 1
    int *h_flags = nullptr;                 // h_block
    // graph
    // executable graphs by batch size (a serving loop's batch sizes vary from
    // batch to batch; each size is captured once), all for graph_tune
    std::unordered_map<int, cudaGraphExec_t> graphs;
    BatchTune graph_tune{0, 0, 0, 0, 0};
    cudaGraphExec_t gexec = nullptr;   // the last one launched
    int32_t last_q = 0;
    int final_buf = 0;
    double form_best_ms[2] = {-1.0, -1.0};   // the last autotune's best per step form (-1: none ran)
    int64_t kernels = 0;
};

namespace {

// A batch's stream has the device's highest priority: batches are short runs
// of small persistent kernels, and when they share the GPU with a large query
// (a serving loop's heavy requests) the block scheduler then places their
// blocks ahead of the large kernels' remaining blocks.
cudaError_t create_priority_stream(cudaStream_t *st) {
    int least = 0, greatest = 0;
    cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
    if (e != cudaSuccess) return e;
    return cudaStreamCreateWithPriority(st, cudaStreamNonBlocking, greatest);
}

// most tiles of any tuning: one per warp of the widest grid, or of 32 rows
int64_t max_tiles(const wk_batch *b) {
    return std::max((int64_t)b->sms * kMaxBlocksPerSm * (kBTMax / 32), (b->cap_rows + 31) / 32) + 2;   // read in pairs
}

void free_batch(wk_batch *b) {
    cudaSetDevice(b->ctx->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    for (auto &kv : b->graphs) cudaGraphExecDestroy(kv.second);
    b->graphs.clear();
    if (b->done) cudaEventDestroy(b->done);
    if (b->stream) cudaStreamDestroy(b->stream);
    cudaFree(b->d_pvs); cudaFree(b->d_desc);
    for (int i = 0; i < 2; ++i) { cudaFree(b->d_row_off[i]); cudaFree(b->d_int_off[i]); cudaFree(b->d_cols[i]); cudaFree(b->d_hist[i]); }
    cudaFree(b->d_cnt); cudaFree(b->d_off); cudaFree(b->d_tile); cudaFree(b->d_qrows); cudaFree(b->d_block);
    cudaFree(b->d_bar);
    if (b->h_desc) cudaFreeHost(b->h_desc);
    if (b->h_block) cudaFreeHost(b->h_block);
    delete b;
}

StepIO make_io(wk_batch *b, int s, int Q, int64_t warps) {
    StepIO io;
    const int in = s & 1, out = in ^ 1;
    io.hist = b->d_hist[in];
    io.out = b->d_hist[out];
    io.in_row_off = b->d_row_off[in];
    io.in_int_off = b->d_int_off[in];
    io.in_cols = b->d_cols[in];
    io.out_row_off = b->d_row_off[out];
    io.out_int_off = b->d_int_off[out];
    io.out_cols = b->d_cols[out];
    io.desc = b->d_desc + (size_t)s * b->max_q;
    io.pvs = b->d_pvs;
    io.cnt = b->d_cnt;
    io.off = b->d_off;
    io.tile_sum = b->d_tile;
    io.q_rows = b->d_qrows;
    io.flags = b->d_flags;
    io.pub = nullptr;
    io.cap_ints = b->cap_ints;
    io.cap_rows = b->cap_rows;
    io.Q = Q;
    io.warps = warps;
    if (s == b->max_steps - 1) {   // the final tables' layout, in one range for one copy to the host
        io.out_row_off = b->d_block + 1;
        io.out_int_off = b->d_block + Q + 2;
        io.out_cols = reinterpret_cast<int32_t *>(b->d_block + 2 * Q + 2);
    }
    return io;
}

// the max_steps steps of a batch with BT-thread blocks: three kernels per
// step, or one cooperative kernel
template <int BT>
int enqueue_steps(wk_batch *b, int Q, const BatchTune &t, unsigned grid, cudaStream_t st) {
    if (t.fused) {
        // every block of a cooperative launch must be resident at once
        int occ = 0;
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_step_kernel<BT>, BT, 0);
        if (e != cudaSuccess) return cuda_fail(e, "batch step occupancy");
        if (occ < 1) return set_error(WK_EDEVICE, "batch step kernel: no block fits on an SM");
        const unsigned gf = (unsigned)std::min<int64_t>(grid, (int64_t)occ * b->sms);
        // the barrier words start at zero in every batch (a wait that ran out leaves them unbalanced)
        if ((e = cudaMemsetAsync(b->d_bar, 0, 2 * sizeof(unsigned int), st)) != cudaSuccess)
            return cuda_fail(e, "batch barrier reset");
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(gf);
        cfg.blockDim = dim3(BT);
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        for (int s = 0; s < b->max_steps; ++s) {
            StepIO io = make_io(b, s, Q, (int64_t)gf * (BT / 32));
            if ((e = cudaLaunchKernelEx(&cfg, batch_step_kernel<BT>, io, t.rounds, t.split, b->d_bar)) != cudaSuccess)
                return cuda_fail(e, "batch step launch");
        }
    } else {
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        for (int s = 0; s < b->max_steps; ++s) {
            StepIO io = make_io(b, s, Q, (int64_t)grid * (BT / 32));
            if (s == b->max_steps - 1) io.pub = b->h_block_dev;
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(BT);
            cudaError_t e = cudaLaunchKernelEx(&cfg, batch_count_kernel<BT>, io, t.rounds);
            cfg.gridDim = dim3(2);
            cfg.blockDim = dim3(kScanThreads);
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, batch_scan_kernel, io, t.rounds);
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(BT);
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, batch_write_kernel<BT>, io, t.rounds, t.split);
            if (e != cudaSuccess) return cuda_fail(e, "batch step launch");
        }
    }
    return WK_OK;
}

// kernels of one batch: the layout init, then per step three kernels or one
int64_t batch_kernels(const wk_batch *b, const BatchTune &t) {
    return 1 + (t.fused ? 1 : 3) * (int64_t)b->max_steps;
}

// the whole batch: descriptors and layout init, max_steps x (count, scan,
// write) as three kernels or as one cooperative kernel
int enqueue(wk_batch *b, int Q, const BatchTune &t, cudaStream_t st) {
    static_assert(sizeof(StepDesc) % 8 == 0, "descriptors are copied as 8 B words");
    const int64_t words = (int64_t)(sizeof(StepDesc) / 8) * Q * b->max_steps;
    const unsigned gi = (unsigned)std::min<int64_t>((words + 511) / 512, 2 * (int64_t)b->sms);   // two words a thread
    batch_init_kernel<<<std::max(gi, 1u), 256, 0, st>>>(
        Q, b->d_row_off[0], b->d_int_off[0], b->d_cols[0], b->d_qrows, b->d_flags,
        reinterpret_cast<const uint64_t *>(b->h_desc_dev), reinterpret_cast<uint64_t *>(b->d_desc),
        (int64_t)(sizeof(StepDesc) / 8) * b->max_q, b->max_steps);
    // The step kernels loop over tiles, so any grid gives the same rows.  A
    // small batch gets a grid in proportion to its queries (at least a
    // quarter of the SMs): beside a large query on another stream, a few
    // light queries then hold a few SMs, not all of them.
    const int64_t full = (int64_t)b->sms * t.blocks_per_sm;
    const unsigned grid = (unsigned)std::min<int64_t>(full, std::max<int64_t>(b->sms / 4, 2 * (int64_t)Q));
    const int st2 = t.bt == 128 ? enqueue_steps<128>(b, Q, t, grid, st) : enqueue_steps<256>(b, Q, t, grid, st);
    if (st2) return st2;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "batch launch");
    b->kernels += batch_kernels(b, t);
    return WK_OK;
}

}  // namespace

extern "C" int wk_batch_create(wk_ctx *ctx, int32_t max_queries, int32_t max_steps, int64_t capacity_ints,
                               wk_batch **out) {
    if (!ctx || !out || max_queries < 1 || max_queries > kMaxQ || max_steps < 1 || max_steps > 16 ||
        capacity_ints < 1)
        return set_error(WK_EINVAL, "wk_batch_create: bad arguments (1..%d queries, 1..16 steps)", kMaxQ);
    if (!ctx->store) return set_error(WK_ENOSTORE, "wk_batch_create: no store built");
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_batch_create: host-only context");
    if (ctx->store->pool) return set_error(WK_EINVAL, "wk_batch_create: batches need a resident store");
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    wk_batch *b = new wk_batch();
    b->ctx = ctx;
    b->max_q = max_queries;
    b->max_steps = max_steps;
    b->cap_ints = capacity_ints;
    b->cap_rows = capacity_ints;   // every row holds at least one int
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const size_t npv = ctx->store->views.size();
    const int64_t tiles = max_tiles(b);
    // a step's input rows: what the step before may leave, or one for each query
    const size_t rows = (size_t)std::max<int64_t>(b->cap_rows, max_queries);
    bool ok = cudaMalloc(&b->d_pvs, sizeof(PredView) * npv) == cudaSuccess &&
              cudaMalloc(&b->d_desc, sizeof(StepDesc) * (size_t)max_queries * max_steps) == cudaSuccess &&
              cudaMalloc(&b->d_cnt, 4 * rows) == cudaSuccess &&
              cudaMalloc(&b->d_off, 4 * rows) == cudaSuccess &&
              cudaMalloc(&b->d_tile, 8 * (size_t)tiles) == cudaSuccess &&
              cudaMalloc(&b->d_qrows, 8 * (size_t)max_queries) == cudaSuccess &&
              cudaMalloc(&b->d_block, 8 * (size_t)(3 * max_queries + 2)) == cudaSuccess &&
              cudaMalloc(&b->d_bar, 2 * sizeof(unsigned int)) == cudaSuccess &&
              cudaHostAlloc((void **)&b->h_desc, sizeof(StepDesc) * (size_t)max_queries * max_steps, cudaHostAllocMapped) ==
                  cudaSuccess &&
              cudaHostGetDevicePointer((void **)&b->h_desc_dev, b->h_desc, 0) == cudaSuccess &&
              cudaHostAlloc((void **)&b->h_block, 8 * (size_t)(3 * max_queries + 2), cudaHostAllocMapped) == cudaSuccess &&
              cudaHostGetDevicePointer((void **)&b->h_block_dev, b->h_block, 0) == cudaSuccess &&
              create_priority_stream(&b->stream) == cudaSuccess &&
              cudaEventCreateWithFlags(&b->done, cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; ok && i < 2; ++i)
        ok = cudaMalloc(&b->d_row_off[i], 8 * (size_t)(max_queries + 1)) == cudaSuccess &&
             cudaMalloc(&b->d_int_off[i], 8 * (size_t)max_queries) == cudaSuccess &&
             cudaMalloc(&b->d_cols[i], 4 * (size_t)max_queries) == cudaSuccess &&
             cudaMalloc(&b->d_hist[i], 4 * (size_t)capacity_ints) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        free_batch(b);
        return set_error(WK_ENOMEM, "wk_batch_create: allocation failed (capacity %lld ints)", (long long)capacity_ints);
    }
    b->d_flags = reinterpret_cast<int *>(b->d_block);
    b->h_flags = reinterpret_cast<int *>(b->h_block);
    b->h_layout = b->h_block + 1;
    e = cudaMemcpy(b->d_pvs, ctx->store->views.data(), sizeof(PredView) * npv, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(b->d_flags, 0, 8);
    if (e == cudaSuccess) e = cudaMemset(b->d_bar, 0, 2 * sizeof(unsigned int));
    if (e != cudaSuccess) { int r = cuda_fail(e, "wk_batch_create"); free_batch(b); return r; }
    *out = b;
    return WK_OK;
}

extern "C" int wk_batch_destroy(wk_batch *b) {
    if (b) free_batch(b);
    return WK_OK;
}

extern "C" int wk_batch_set_tuning(wk_batch *b, int32_t blocks_per_sm, int32_t rows_per_warp, int32_t split_ints) {
    if (!b || blocks_per_sm < 1 || blocks_per_sm > kMaxBlocksPerSm || rows_per_warp < 32 || rows_per_warp > 256 ||
        rows_per_warp % 32 || split_ints < 1)
        return set_error(WK_EINVAL, "wk_batch_set_tuning: blocks/SM 1..16, rows/warp 32..256 (x32), split >= 1");
    b->tune = BatchTune{blocks_per_sm, rows_per_warp / 32, split_ints, b->tune.fused, b->tune.bt};
    return WK_OK;
}

extern "C" int wk_batch_set_fused(wk_batch *b, int32_t fused) {
    if (!b || (fused != 0 && fused != 1)) return set_error(WK_EINVAL, "wk_batch_set_fused: 0 or 1");
    b->tune.fused = fused;
    return WK_OK;
}

extern "C" int wk_batch_get_fused(wk_batch *b) { return b ? b->tune.fused : 0; }

extern "C" int wk_batch_set_block_threads(wk_batch *b, int32_t threads) {
    if (!b || (threads != 128 && threads != 256)) return set_error(WK_EINVAL, "wk_batch_set_block_threads: 128 or 256");
    b->tune.bt = threads;
    return WK_OK;
}

extern "C" int wk_batch_get_block_threads(wk_batch *b) { return b ? b->tune.bt : 0; }

extern "C" int wk_batch_get_tuning(wk_batch *b, int32_t *blocks_per_sm, int32_t *rows_per_warp, int32_t *split_ints) {
    if (!b || !blocks_per_sm || !rows_per_warp || !split_ints) return set_error(WK_EINVAL, "wk_batch_get_tuning: null");
    *blocks_per_sm = b->tune.blocks_per_sm;
    *rows_per_warp = b->tune.rounds * 32;
    *split_ints = b->tune.split;
    return WK_OK;
}

// Fill the step descriptors from the queries.  A query starts from a
// constant vertex or from an index: a type index [c, type, IN, -1] is the list
// of key [0|c|IN] and a predicate index [p, 0, d, -1] the list of key [0|p|d]
// (core/gstore.hpp:546-560), so both run as a constant start at vertex 0.
static int fill_desc(wk_batch *b, const int64_t *cmd, const int32_t *npat, int32_t Q) {
    int64_t at = 0;
    const int num_ids = b->ctx->store->hs->num_ids;
    for (int q = 0; q < Q; ++q) {
        const int n = npat[q];
        if (n < 1 || n > b->max_steps) return set_error(WK_EINVAL, "wk_batch_run: query %d has %d patterns (1..%d)", q, n, b->max_steps);
        int col = 0;
        for (int s = 0; s < b->max_steps; ++s) {
            StepDesc &d = b->h_desc[(size_t)s * b->max_q + q];
            if (s >= n) { d = StepDesc{BK_NOP, 1, 0, 0, 0, 0}; continue; }
            const int64_t st = cmd[at + 4 * s], pid = cmd[at + 4 * s + 1], dir = cmd[at + 4 * s + 2], en = cmd[at + 4 * s + 3];
            if (s == 0 && st > 1 && st < WK_VID_BASE) {   // index start
                const bool ok = en == -1 && st <= num_ids &&
                                ((pid == WK_TYPE_ID && dir == WK_DIR_IN) || (pid == WK_PREDICATE_ID && (dir == 0 || dir == 1)));
                if (!ok) return set_error(WK_EINVAL, "wk_batch_run: query %d: bad index start", q);
                d = StepDesc{BK_C2U, (int32_t)st, (int32_t)dir, 0, 0, 0};
                col = 1;
                continue;
            }
            if (pid < 1 || pid > num_ids || (dir != 0 && dir != 1))
                return set_error(WK_EINVAL, "wk_batch_run: query %d step %d: predicate %lld / direction %lld", q, s,
                                 (long long)pid, (long long)dir);
            const bool start_known = st < 0 && -st <= col, end_unknown = en < 0 && -en > col, end_known = en < 0 && -en <= col;
            if (s == 0) {
                if (st < WK_VID_BASE || st > 0x7fffffffll || en != -1)
                    return set_error(WK_EINVAL, "wk_batch_run: query %d must start from a constant vertex or an index, binding -1", q);
                d = StepDesc{BK_C2U, (int32_t)pid, (int32_t)dir, 0, 0, (int32_t)st};
                col = 1;
            } else if (start_known && end_unknown) {
                if (-en - 1 != col) return set_error(WK_EINVAL, "wk_batch_run: query %d step %d skips a column", q, s);
                d = StepDesc{BK_K2U, (int32_t)pid, (int32_t)dir, (int32_t)(-st - 1), 0, 0};
                ++col;
            } else if (start_known && end_known) {
                d = StepDesc{BK_K2K, (int32_t)pid, (int32_t)dir, (int32_t)(-st - 1), (int32_t)(-en - 1), 0};
            } else if (start_known && en >= 0 && en <= 0x7fffffffll) {
                d = StepDesc{BK_K2C, (int32_t)pid, (int32_t)dir, (int32_t)(-st - 1), 0, (int32_t)en};
            } else {
                return set_error(WK_EINVAL, "wk_batch_run: query %d step %d: unsupported pattern shape", q, s);
            }
        }
        at += 4 * n;
    }
    return WK_OK;
}

extern "C" int wk_batch_launch(wk_batch *b, const int64_t *cmd_chains, const int32_t *n_patterns, int32_t nq,
                               int32_t use_graph) {
    if (!b || !cmd_chains || !n_patterns || nq < 1 || nq > b->max_q)
        return set_error(WK_EINVAL, "wk_batch_launch: bad arguments (1..%d queries)", b ? b->max_q : 0);
    wk_ctx *ctx = b->ctx;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    // the pinned descriptors may still be read by a previous launch
    if ((e = cudaEventSynchronize(b->done)) != cudaSuccess) return cuda_fail(e, "batch previous launch");
    int st = fill_desc(b, cmd_chains, n_patterns, nq);
    if (st) return st;
    cudaStream_t s = b->stream;
    if (use_graph) {
        if (std::memcmp(&b->graph_tune, &b->tune, sizeof(BatchTune)) != 0 || b->graphs.size() >= 512) {
            for (auto &kv : b->graphs) cudaGraphExecDestroy(kv.second);
            b->graphs.clear();
            b->graph_tune = b->tune;
        }
        auto it = b->graphs.find(nq);
        if (it == b->graphs.end()) {
            cudaGraph_t g;
            if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
                return cuda_fail(e, "batch capture");
            st = enqueue(b, nq, b->tune, s);
            e = cudaStreamEndCapture(s, &g);
            if (st) { if (e == cudaSuccess) cudaGraphDestroy(g); return st; }
            if (e != cudaSuccess) return cuda_fail(e, "batch capture end");
            cudaGraphExec_t ge = nullptr;
            e = cudaGraphInstantiate(&ge, g, 0);
            cudaGraphDestroy(g);
            if (e != cudaSuccess) return cuda_fail(e, "batch graph instantiate");
            it = b->graphs.emplace(nq, ge).first;
            b->kernels -= batch_kernels(b, b->tune);   // capture does not launch
        }
        b->gexec = it->second;
        if ((e = cudaGraphLaunch(b->gexec, s)) != cudaSuccess) return cuda_fail(e, "batch graph launch");
        b->kernels += batch_kernels(b, b->tune);
    } else {
        if ((st = enqueue(b, nq, b->tune, s))) return st;
    }
    ctx->launches += batch_kernels(b, b->tune);
    b->last_q = nq;
    b->final_buf = b->max_steps & 1;
    // the flags and the layout of the final tables (the last write kernel has sent
    // them where there is one), then the completion event
    if ((b->tune.fused && (e = cudaMemcpyAsync(b->h_block, b->d_block, 8 * (2 * (size_t)nq + 2) + 4 * (size_t)nq,
                                               cudaMemcpyDeviceToHost, s)) != cudaSuccess) ||
        (e = cudaEventRecord(b->done, s)) != cudaSuccess)
        return cuda_fail(e, "batch layout readback");
    return WK_OK;
}

// 1 when the last launch has finished, 0 while it runs
extern "C" int wk_batch_ready(wk_batch *b) {
    if (!b) return 1;
    return cudaEventQuery(b->done) == cudaSuccess ? 1 : 0;
}

extern "C" int wk_batch_wait(wk_batch *b) {
    if (!b) return set_error(WK_EINVAL, "wk_batch_wait: null");
    cudaError_t e = cudaEventSynchronize(b->done);
    if (e != cudaSuccess) return cuda_fail(e, "batch wait");
    if (b->h_flags[1]) return set_error(WK_EOVERFLOW, "wk_batch: a step exceeded the batch capacity of %lld ints",
                                        (long long)b->cap_ints);
    if (b->h_flags[0] & kErrBarrier)
        return set_error(WK_ETIMEDOUT, "wk_batch: a grid-barrier wait of the one-kernel step ran out");
    if (b->h_flags[0]) return set_error(WK_EDEVICE, "wk_batch: corrupt overflow chain in the store");
    return WK_OK;
}

extern "C" int wk_batch_run(wk_batch *b, const int64_t *cmd_chains, const int32_t *n_patterns, int32_t nq,
                            int32_t use_graph) {
    int st = wk_batch_launch(b, cmd_chains, n_patterns, nq, use_graph);
    return st ? st : wk_batch_wait(b);
}

extern "C" int wk_batch_result(wk_batch *b, int32_t q, int64_t *rows, int32_t *cols, int64_t *int_offset) {
    if (!b || q < 0 || q >= b->last_q || !rows || !cols || !int_offset) return set_error(WK_EINVAL, "wk_batch_result");
    const int nq = b->last_q;
    const int32_t *c = reinterpret_cast<const int32_t *>(b->h_layout + 2 * nq + 1);
    *rows = b->h_layout[q + 1] - b->h_layout[q];
    *cols = c[q];
    *int_offset = b->h_layout[nq + 1 + q];
    return WK_OK;
}

extern "C" int wk_batch_layouts(wk_batch *b, int32_t nq, int64_t *rows, int32_t *cols, int64_t *int_offsets) {
    if (!b || nq != b->last_q || (nq > 0 && (!rows || !cols || !int_offsets)))
        return set_error(WK_EINVAL, "wk_batch_layouts: bad arguments (the last run had %d queries)", b ? b->last_q : 0);
    const int32_t *c = reinterpret_cast<const int32_t *>(b->h_layout + 2 * nq + 1);
    for (int q = 0; q < nq; ++q) {
        rows[q] = b->h_layout[q + 1] - b->h_layout[q];
        cols[q] = c[q];
        int_offsets[q] = b->h_layout[nq + 1 + q];
    }
    return WK_OK;
}

extern "C" int wk_batch_download(wk_batch *b, int32_t *host, int64_t cap, int64_t *total_ints) {
    if (!b || !total_ints) return set_error(WK_EINVAL, "wk_batch_download: null");
    const int nq = b->last_q;
    const int32_t *c = reinterpret_cast<const int32_t *>(b->h_layout + 2 * nq + 1);
    const int64_t tot = nq ? b->h_layout[nq + 1 + nq - 1] + (b->h_layout[nq] - b->h_layout[nq - 1]) * c[nq - 1] : 0;
    *total_ints = tot;
    if (!host) return WK_OK;
    if (cap < tot) return set_error(WK_EOVERFLOW, "wk_batch_download: %lld ints, room for %lld", (long long)tot, (long long)cap);
    cudaError_t e;
    if (tot && (e = cudaMemcpyAsync(host, b->d_hist[b->final_buf], 4 * (size_t)tot, cudaMemcpyDeviceToHost,
                                    b->stream)) != cudaSuccess)
        return cuda_fail(e, "wk_batch_download");
    if ((e = cudaStreamSynchronize(b->stream)) != cudaSuccess) return cuda_fail(e, "wk_batch_download sync");
    return WK_OK;
}

// Autotuner: time the batch with every candidate (three kernels or one per
// step, 128 or 256 threads a block, blocks/SM, rows/warp, split) on the given
// queries (CUDA events, best of `reps` after a warm run) and keep the fastest.  A one-kernel candidate
// the device refuses (its cooperative launch, or its capture into a graph) is
// skipped.  Writes the chosen candidate's time.
extern "C" int wk_batch_autotune(wk_batch *b, const int64_t *cmd_chains, const int32_t *n_patterns, int32_t nq,
                                 int32_t reps, double *best_ms) {
    if (!b || reps < 1) return set_error(WK_EINVAL, "wk_batch_autotune: bad arguments");
    static const int kBlocks[] = {2, 4, 8};
    static const int kRows[] = {32, 64, 128};
    static const int kSplit[] = {16, 64, 256};
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
        return set_error(WK_EDEVICE, "wk_batch_autotune: events");
    double best = 1e30;
    BatchTune keep = b->tune;
    b->form_best_ms[0] = b->form_best_ms[1] = -1.0;
    for (int fu = 0; fu < 2; ++fu)
    for (int bt : {256, 128})
    for (int bl : kBlocks)
        for (int rw : kRows)
            for (int sp : kSplit) {
                b->tune = BatchTune{bl, rw / 32, sp, fu, bt};
                int st = wk_batch_run(b, cmd_chains, n_patterns, nq, 1);   // builds the graph
                if (st && fu && st != WK_EOVERFLOW && st != WK_ETIMEDOUT) {
                    cudaGetLastError();
                    continue;
                }
                if (st) { cudaEventDestroy(e0); cudaEventDestroy(e1); b->tune = keep; return st; }
                double tbest = 1e30;
                for (int r = 0; r < reps; ++r) {
                    cudaEventRecord(e0, b->stream);
                    cudaGraphLaunch(b->gexec, b->stream);
                    cudaEventRecord(e1, b->stream);
                    cudaEventSynchronize(e1);
                    float ms = 0.f;
                    cudaEventElapsedTime(&ms, e0, e1);
                    tbest = std::min(tbest, (double)ms);
                }
                if (tbest < best) { best = tbest; keep = b->tune; }
                if (b->form_best_ms[fu] < 0.0 || tbest < b->form_best_ms[fu]) b->form_best_ms[fu] = tbest;
            }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->tune = keep;
    if (best_ms) *best_ms = best;
    return wk_batch_run(b, cmd_chains, n_patterns, nq, 1);
}

extern "C" int64_t wk_batch_kernel_launches(wk_batch *b) { return b ? b->kernels : 0; }

extern "C" int wk_batch_autotune_forms(wk_batch *b, double *three_kernel_ms, double *one_kernel_ms) {
    if (!b || !three_kernel_ms || !one_kernel_ms) return set_error(WK_EINVAL, "wk_batch_autotune_forms: null");
    *three_kernel_ms = b->form_best_ms[0];
    *one_kernel_ms = b->form_best_ms[1];
    return WK_OK;
}
