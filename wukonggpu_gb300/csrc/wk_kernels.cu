// Expansion kernels of the per-pattern operator (sm_103a).
//
// Every op is integer work bounded by HBM: random 64 B bucket reads for the
// probe, then streaming reads of history/adjacency and streaming writes of the
// new table.  No tensor cores are involved.
//
//   k2u     : count (probe; per block of rows, those with a list: their first
//             output row, list offset and row; per-block output count;
//             per-group sums of output rows and of slices, a slice being at
//             most kSliceRows output rows of one block) -> publish (the group
//             sums to the host, which adds them up and sizes the output; one
//             record per slice for the expansion) -> expand (one CTA per
//             slice: its record, its block's entries, its rows written)
//   k2k/k2c : probe + membership (per-row ballot masks; per-block counts;
//             per-group sums) -> filtered copy (per input block: output prefix
//             from the group sums and its group's counts, selected rows copied)
//             -> publish (the sums to the host)
//
// A dense functional direction takes one launch for either (wk_fused.cu).
//
// Result order equals the reference CPU engine's (core/engine.hpp:126-225):
// output rows follow input row order, and for k2u each input row's block of
// output rows follows adjacency order.
#include "wk_kernels.h"
#include "wk_probe.cuh"

namespace wk {
namespace dev {

#define FULL 0xffffffffu

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

// block-wide sum of (u64, u32) pairs; result valid in thread 0
__device__ __forceinline__ void block_sum2(unsigned long long &a, unsigned int &b) {
    __shared__ unsigned long long sa[32];
    __shared__ unsigned int sb[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) { sa[wid] = a; sb[wid] = b; }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        a = lane < nw ? sa[lane] : 0ull;
        b = lane < nw ? sb[lane] : 0u;
        a = warp_sum(a);
        b = warp_sum(b);
    }
}

// --------------------------------------------------------------- k2u count
// A block's output rows are written by slices_of(count) expansion CTAs (none
// for an empty block), so a block that holds hub rows is spread over many
// CTAs and an op with few input blocks but a large fan-out still fills the
// GPU.  The + 3 covers the 16 B alignment lead of the block's first row.
__device__ __forceinline__ unsigned long long slices_of(unsigned long long t) {
    return t == 0ull ? 0ull : (t + 3ull + kSliceRows - 1) / kSliceRows;
}

// Programmatic dependent launch: a count kernel is launched so that its CTAs
// may be placed while the previous op's expansion finishes its last wave, and
// the publish kernel so that its CTA is in place when the count finishes.
// Each CTA of such a kernel first waits (in hardware) until the previous grid
// has completed and its writes are visible; expansion and count CTAs allow
// the dependent launch as soon as they run.
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependent_grid() { asm volatile("griddepcontrol.launch_dependents;"); }

// A warp owns kRounds * 32 consecutive rows.  Their start vertices are loaded
// first (kRounds independent coalesced loads), then each round of 32 rows is
// probed, so the history read does not sit in front of every bucket read.
constexpr int kRounds = kRowsPerBlock / (kThreads / 32) / 32;

// Which of a lane's NR start vertices a direction can hold at all: a bit per
// round.  A hashed direction with a presence bitmap answers with one 4 B read a
// row, all rounds' reads in flight together and equal neighbours' reads merged
// by the load unit; the run search and bucket reads of probe_warp are then only
// for rounds that hold one (a sparse predicate's rounds rarely do).  Going
// through probe_warp for every round took 116 instructions a round of 32 rows
// and one read's latency after another: the count of 9M rows of 5 columns 49
// us, 39 so.
template <int NR>
__device__ __forceinline__ unsigned may_hold(const PredView &pv, uint32_t dir, const int32_t (&v)[NR]) {
    unsigned present = 0u;
    const uint32_t *bm = dir ? pv.bm[1] : pv.bm[0];
    if (bm != nullptr) {
        const uint32_t bvmin = dir ? pv.bvmin[1] : pv.bvmin[0], bn = dir ? pv.bn[1] : pv.bn[0];
        uint32_t w[NR];
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) {
            const uint32_t x = (uint32_t)v[rd] - bvmin;   // wraps above bn below bvmin
            w[rd] = (v[rd] > 0 && x < bn) ? __ldg(bm + (x >> 5)) : 0u;
        }
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) {
            const uint32_t x = (uint32_t)v[rd] - bvmin;
            present |= (v[rd] == 0 ? 1u : (w[rd] >> (x & 31u)) & 1u) << rd;   // an index key: always hashed
        }
    } else {
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) present |= (v[rd] >= 0 ? 1u : 0u) << rd;
    }
    return present;
}

// a first pass's CTA asks L2 for the rows of the CTA this many on: 3 an SM of 152,
// half of those in flight (912 gave 121.8 us where this gave 120.4, 1824 127.9)
constexpr int64_t kPrefetch = 456;

// where a block's number of entries sits in its blk_sum word
constexpr int kEntryShift = 48;
constexpr unsigned long long kSumMask = (1ull << kEntryShift) - 1;

// blk_sum[b] = the block's output rows, added into its group's sums, and from
// bit 48 on its rows with a list.  Err bit 1 when a block's output count
// reaches 2^31 (block-local positions are 32 bits).
//
// A block's rows with a list are its entries, written in order from the
// block's first row on: pos = the entry's first output row within the block
// (and the block's total behind the last), rel = its list offset minus pos
// (modulo 2^32: rel + j is the list entry of output row j), row = its row in
// the block.  The expansion's CTAs, several of them for a block with a large
// fan-out, then copy what they need instead of scanning 1024 degrees each
// (half of their instructions on a step of low fan-out), and rows without a
// list -- 99% of them for a sparse predicate -- cost no traffic.
//
// FUNC (a direction whose lists hold at most one vertex, hashed): pos receives
// the neighbour of every row as an int32, or -1 for no match; no entries.
// DENSE (the direction is an offsets array): a warp issues the lookups of all
// its rounds phase by phase -- every round's start vertex, then every round's
// offsets -- and a lane looks up its own key (no shuffles).  BPC blocks per
// CTA: 2 for a large dense op, so each warp keeps eight rounds of loads in
// flight and a CTA's fixed costs (reduction, exit) are shared by 2048 rows; 1
// otherwise, so a small op still spreads over many CTAs.
template <bool FUNC, bool DENSE, int BPC>
__global__ void __launch_bounds__(kThreads, 6)
k2u_count_kernel(const int32_t *__restrict__ hist, int64_t R, int C, int scol, uint32_t dir, PredView pv, Entries en,
                 unsigned long long *__restrict__ blk_sum, unsigned long long *__restrict__ group_sums, int *err,
                 unsigned long long *__restrict__ clear, int64_t nclear) {
    constexpr int NR = kRounds * BPC;   // rounds of 32 rows per warp
    wait_prior_grid();   // before anything is read or cleared
    allow_dependent_grid();   // the publish kernel behind it
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b0 = (int64_t)blockIdx.x * BPC;
    // the other sums buffer, read by the previous op's expansion, is cleared
    // for the next op (a few hundred words at most)
    for (int64_t w = (int64_t)blockIdx.x * kThreads + threadIdx.x; w < nclear; w += (int64_t)gridDim.x * kThreads)
        clear[w] = 0ull;
    if (threadIdx.x == 0)
        prefetch_rows(hist, R, C, (b0 + kPrefetch * BPC) * kRowsPerBlock, (b0 + (kPrefetch + 1) * BPC) * kRowsPerBlock);
    const int64_t nblk = (R + kRowsPerBlock - 1) / kRowsPerBlock;
    // round rd: block b0 + rd / kRounds, the warp's rows 32 (rd % kRounds) + lane
    auto row_at = [&](int rd) -> int64_t {
        return (b0 + rd / kRounds) * kRowsPerBlock + (int64_t)warp * (kRounds * 32) + (rd % kRounds) * 32 + lane;
    };
    int32_t v[NR];
#pragma unroll
    for (int rd = 0; rd < NR; ++rd) {
        const int64_t r = row_at(rd);
        v[rd] = r < R ? ld_prior(hist + r * C + scol) : -1;
    }
    unsigned long long my_sum[BPC];
    unsigned int nent[BPC], run[BPC];   // the warp's entries and output rows so far
#pragma unroll
    for (int j = 0; j < BPC; ++j) { my_sum[j] = 0ull; nent[j] = run[j] = 0u; }
    uint32_t o[NR], d[NR];   // a row's list offset; its degree, then its first output row within the warp's
    unsigned has = 0u;       // rounds in which the lane's row has a list
    if constexpr (DENSE) {
        const uint32_t vmin = dir ? pv.vmin[1] : pv.vmin[0], dn = dir ? pv.dn[1] : pv.dn[0];
        const uint32_t *rp = dir ? pv.rp[1] : pv.rp[0];
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) {
            const int32_t vid = v[rd];
            o[rd] = d[rd] = 0u;
            const uint32_t x = (uint32_t)vid - vmin;   // wraps above dn below vmin
            if (vid > 0 && x < dn) {
                o[rd] = __ldg(rp + x);
                d[rd] = __ldg(rp + x + 1);
            } else if (vid == 0) {   // index key: the hash table
                d[rd] = probe_seg(pv.buckets, pv.nmain, pv.nover, seg_key(0u, dir), &o[rd], err);
                d[rd] += o[rd];
            }
        }
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) d[rd] -= o[rd];   // v is -1 past the table: no list
    } else {
        // hashed: runs of equal keys probed once (probe_warp), a round at a time
        const unsigned present = may_hold(pv, dir, v);
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) {
            const int64_t r = row_at(rd);
            o[rd] = d[rd] = 0u;
            const bool here = (present >> rd) & 1u;
            if (__any_sync(FULL, here)) probe_warp(pv, here ? v[rd] : -1, dir, o[rd], d[rd], err);
            if constexpr (FUNC) {
                if (r < R) reinterpret_cast<int32_t *>(en.pos)[r] = d[rd] ? __ldg(pv.edges + o[rd]) : -1;
                if (d[rd] > 1u) atomicOr(err, 8);   // an index list: the op reruns unspecialised
                // at most one output row per input row, so a block's output never
                // exceeds its rows even before the rerun
                my_sum[rd / kRounds] += d[rd] ? 1u : 0u;
            }
        }
    }
    if constexpr (!FUNC) {
#pragma unroll
        for (int rd = 0; rd < NR; ++rd) {
            const int j = rd / kRounds;
            const unsigned m = __ballot_sync(FULL, d[rd] != 0u);
            if (d[rd] != 0u) has |= 1u << rd;
            my_sum[j] += d[rd];
            nent[j] += (unsigned)__popc(m);
            if (m) {   // the same in every lane
                uint32_t in = d[rd];
#pragma unroll
                for (int sh = 1; sh < 32; sh <<= 1) {
                    const uint32_t x = __shfl_up_sync(FULL, in, sh);
                    if (lane >= sh) in += x;
                }
                d[rd] = run[j] + in - d[rd];
                run[j] += __shfl_sync(FULL, in, 31);
            }
        }
    }
    // each block's output rows: a warp reduction (one REDUX instruction while the
    // partial sums are small, as every valid block's are) and one barrier
    __shared__ unsigned long long s_part[BPC][kThreads / 32];
    __shared__ unsigned int s_ent[BPC][kThreads / 32];
#pragma unroll
    for (int j = 0; j < BPC; ++j) {
        unsigned long long ws;
        if (!__any_sync(FULL, my_sum[j] >= (1ull << 26))) ws = __reduce_add_sync(FULL, (unsigned int)my_sum[j]);
        else ws = warp_sum(my_sum[j]);
        if (lane == 0) { s_part[j][warp] = ws; s_ent[j][warp] = nent[j]; }
    }
    __syncthreads();
    if constexpr (!FUNC) {
#pragma unroll
        for (int j = 0; j < BPC; ++j) {
            if (nent[j] == 0u) continue;   // the same in every lane
            unsigned int at = 0u, base = 0u;
            for (int w = 0; w < warp; ++w) {
                at += s_ent[j][w];
                base += (unsigned int)s_part[j][w];
            }
            const int64_t first = (b0 + j) * kRowsPerBlock;
#pragma unroll
            for (int q = 0; q < kRounds; ++q) {
                const int rd = j * kRounds + q;
                const bool mine = (has >> rd) & 1u;
                const unsigned m = __ballot_sync(FULL, mine);
                if (mine) {
                    const int64_t k = first + at + (unsigned)__popc(m & ((1u << lane) - 1u));
                    en.pos[k] = base + d[rd];
                    en.rel[k] = o[rd] - (base + d[rd]);
                    en.row[k] = (uint16_t)(warp * (kRounds * 32) + q * 32 + lane);
                }
                at += (unsigned)__popc(m);
            }
        }
    }
    if (threadIdx.x < BPC) {
        const int j = threadIdx.x;
        const int64_t b = b0 + j;
        unsigned long long sum = 0ull;
        unsigned int n = 0u;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) { sum += s_part[j][w]; n += s_ent[j][w]; }
        if (b < nblk) {
            if (!FUNC && n < kRowsPerBlock) en.pos[b * kRowsPerBlock + n] = (uint32_t)sum;
            blk_sum[b] = sum | (unsigned long long)n << kEntryShift;   // a sum past 2^31 is an error
            // group sums spread the atomics over many addresses (256 blocks each);
            // the host adds them up for the op totals, so no address takes one per block
            if (sum) {
                unsigned long long *gs = group_sums + 2 * (b >> kGroupShift);
                atomicAdd(gs, sum);
                atomicAdd(gs + 1, slices_of(sum));
            }
            if (sum >> 31) atomicOr(err, 2);
        }
    }
}

// ------------------------------------------------- publish, slice records
static_assert(kThreads == (1 << kGroupShift), "one thread per block of a group");

// inclusive scan of (x, y) pairs over the CTA's threads
__device__ __forceinline__ void cta_scan2(unsigned long long &x, unsigned long long &y,
                                          unsigned long long (&sw)[2][kThreads / 32]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int sh = 1; sh < 32; sh <<= 1) {
        const unsigned long long ax = __shfl_up_sync(FULL, x, sh), ay = __shfl_up_sync(FULL, y, sh);
        if (lane >= sh) { x += ax; y += ay; }
    }
    if (lane == 31) { sw[0][wid] = x; sw[1][wid] = y; }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kThreads / 32 - 1; ++w)
        if (w < wid) { x += sw[0][w]; y += sw[1][w]; }
}

// The records of the slices of group g, of those in [first, first + cap): the
// slices are numbered in block order over the op, a block of count output rows
// having slices_of(count) of them.
__device__ __forceinline__ void plan_group(const SlicePlan &a, int64_t g) {
    __shared__ unsigned long long sw[2][kThreads / 32], s_before[2][kThreads / 32];
    __shared__ unsigned long long s_x[kThreads], s_word[kThreads];
    __shared__ uint32_t s_y[kThreads + 1];   // a group has fewer than 2^32 slices
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    // output rows and slices of the groups before
    unsigned long long op = 0ull, sp = 0ull;
    for (int64_t i = t; i < g; i += kThreads) {
        op += ld_prior(a.group_sums + 2 * i);
        sp += ld_prior(a.group_sums + 2 * i + 1);
    }
    op = warp_sum(op);
    sp = warp_sum(sp);
    if (lane == 0) { s_before[0][wid] = op; s_before[1][wid] = sp; }
    const int64_t bi = (g << kGroupShift) + t;
    const unsigned long long word = bi < a.nblk ? ld_prior(a.blk_sum + bi) : 0ull;
    unsigned long long x = word & kSumMask, y = slices_of(word & kSumMask);
    const unsigned long long x0 = x, y0 = y;
    cta_scan2(x, y, sw);
    s_x[t] = x - x0;
    s_y[t] = (uint32_t)(y - y0);
    s_word[t] = word;
    if (t == kThreads - 1) s_y[kThreads] = (uint32_t)y;
    __syncthreads();
    op = sp = 0ull;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) { op += s_before[0][w]; sp += s_before[1][w]; }
    if (t == 0 && a.head != nullptr && (g + 1) << kGroupShift >= a.nblk) {   // the last group
        const unsigned long long rows = op + s_x[kThreads - 1] + (s_word[kThreads - 1] & kSumMask);
        const unsigned long long n = sp + s_y[kThreads];
        *a.head = ld_prior(a.err) == 0 && n <= a.max_slices && rows <= a.max_rows ? (uint32_t)n : 0u;
    }
    const unsigned long long last = a.first + a.cap;   // the group's slices of the window
    const uint32_t i0 = a.first > sp ? (uint32_t)min(a.first - sp, (unsigned long long)s_y[kThreads]) : 0u;
    const uint32_t i1 = last > sp ? (uint32_t)min(last - sp, (unsigned long long)s_y[kThreads]) : 0u;
    for (uint32_t i = i0 + t; i < i1; i += kThreads) {
        const unsigned long long k = sp + i;
        int lo = 0, hi = kThreads - 1;   // the last block whose slices begin at or before i
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_y[mid] <= i) lo = mid;
            else hi = mid - 1;
        }
        SliceRec r;
        r.P = op + s_x[lo];
        r.block = (uint32_t)((g << kGroupShift) + lo);
        r.T = (uint32_t)(s_word[lo] & kSumMask);   // below 2^31 (the count kernel flags larger blocks)
        r.slice = i - s_y[lo];
        r.n = (uint32_t)(s_word[lo] >> kEntryShift);
        r.pad[0] = r.pad[1] = 0u;
        uint4 *dst = reinterpret_cast<uint4 *>(a.slices + (k - a.first));
        const uint4 *src = reinterpret_cast<const uint4 *>(&r);
        dst[0] = src[0];
        dst[1] = src[1];
    }
}

// Stream-ordered behind a count kernel.  CTA 0 copies the op's error word and
// group sums into pinned host memory, fences them system-wide, then writes the
// sequence number the host waits for; CTA 1 + g writes the slice records of
// group g, while the host adds up the sums and launches the expansion.
__global__ void __launch_bounds__(kThreads) publish_kernel(const Publish pub, const SlicePlan plan) {
    wait_prior_grid();   // the count kernel's sums are complete
    // no early start for an expansion behind: its CTAs would keep to the small
    // shared memory that these leave an SM, and few at a time, for all of its run
    if (blockIdx.x > 0) {
        plan_group(plan, (int64_t)blockIdx.x - 1);
        return;
    }
    if (pub.dst == nullptr) return;
    for (long long w = threadIdx.x; w < pub.n; w += blockDim.x) pub.dst[2 + w] = ld_prior(pub.src + w);
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *(volatile unsigned long long *)pub.dst = pub.seq;
}

// -------------------------------------------------------------- k2u expand
// last entry k in [0, n) with pos[k] <= j; pos is non-decreasing with pos[0] =
// 0 (n >= 1), so for j below the block's total that entry's list covers j
__device__ __forceinline__ int row_of(const uint32_t *pos, int n, uint32_t j) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pos[mid] <= j) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The block's entries as the count kernel left them: entry k is block row
// row[k], its first output row pos[k] (block-local), its list offset minus
// pos[k] in erel[k] (modulo 2^32: erel + j is the entry index of output row
// j), and pos[n] = the block's total.
struct ExpandRows {
    alignas(16) uint32_t pos[kRowsPerBlock + 4];
    alignas(16) uint32_t erel[kRowsPerBlock];
    alignas(16) uint16_t row[kRowsPerBlock];
};

// The entry of each of 32 consecutive output rows, one per lane: k0 covers the
// window's first row j.  A list that begins inside the window sets its row's
// bit, so a lane's entry is k0 plus the bits at or below it: one shared read
// and one REDUX a window, where a search per row took ten dependent reads.
// k0 moves on to the entry of row j + 32.  j may be "negative" (modulo 2^32)
// by up to 3 rows, before the block's first row.
__device__ __forceinline__ int window_entries(const ExpandRows &xr, int n, uint32_t j, int lane, int &k0) {
    const int i = k0 + 1 + lane;
    const uint32_t p = xr.pos[i < n ? i : n] - j;   // > 0; entry n holds the block's total
    const unsigned heads = __reduce_or_sync(FULL, p < 32u && i < n ? 1u << p : 0u);
    const int k = k0 + __popc(heads & (0xffffffffu >> (31 - lane)));
    k0 += __popc(__ballot_sync(FULL, p <= 32u && i < n));
    return k;
}

// A window's output row as the lane holds it, stored to shared memory in the
// widest words that the row's width keeps aligned.
template <int W>
__device__ __forceinline__ void stage_row(int32_t *dst, const int32_t (&v)[W]) {
    if constexpr (W % 4 == 0) {
#pragma unroll
        for (int c = 0; c < W; c += 4)
            *reinterpret_cast<int4 *>(dst + c) = make_int4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    } else if constexpr (W % 2 == 0) {
#pragma unroll
        for (int c = 0; c < W; c += 2) *reinterpret_cast<int2 *>(dst + c) = make_int2(v[c], v[c + 1]);
    } else {
#pragma unroll
        for (int c = 0; c < W; ++c) dst[c] = v[c];
    }
}

// Shared memory to global by the copy engine (both 16 B aligned, bytes a
// multiple of 16), in a group of the calling thread's own; and the wait until
// its copies have read their source.
__device__ __forceinline__ void bulk_store(int32_t *dst, const int32_t *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n\tcp.async.bulk.commit_group;" ::"l"(dst),
                 "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// 16 B from global to shared memory without registers
__device__ __forceinline__ void copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

constexpr int kChunk = 64;   // output rows a warp stages at a time: two windows

// Output rows [u, u + kChunk) of a warp, W = 2..8 columns.  Rows are counted
// locally from P - lead, the 16 B-aligned row at or before the block's first
// output row P (lead = P mod 4); local row u is block row u - lead, valid for
// lo <= u < hi.  A lane gathers the row it owns in each window (its input row
// through L1, lanes of one list reading one row; its list entry, consecutive
// lanes reading consecutive entries), the warp stages the rows packed in
// shared memory and writes them as consecutive 16 B vectors.
//
// The stores bound this kernel before DRAM does: with each thread storing its
// own four rows, 4 W words apart in a warp's instruction, every 16 B store was
// a half-filled sector of its own.  Consecutive vectors took the k2u op (count
// and expansion) on 120k -> 12M rows of 4 columns from 65.6 to 47.0 us (3.7 to
// 5.1 TB/s of its input, list entries and output) and on 9M -> 18.6M rows of
// 6 columns from 185.9 to 159.0 us (4.0 to 4.6 TB/s).
template <int W>
__device__ __forceinline__ void write_chunk(uint32_t u, uint32_t lead, uint32_t lo, uint32_t hi, const ExpandRows &xr,
                                            int n, int &k0, const int32_t *__restrict__ rows,
                                            const int32_t *__restrict__ edges, int32_t *__restrict__ obase,
                                            int32_t *stg, int lane) {
    constexpr int C = W - 1, kWin = kChunk / 32;
    const bool whole = u >= lo && u + kChunk <= hi;   // the same in every lane
    int32_t v[kWin][W];
    auto gather = [&](int q, int k) {
        const int32_t *src = rows + (int)xr.row[k] * C;
#pragma unroll
        for (int c = 0; c < C; ++c) v[q][c] = __ldg(src + c);
        v[q][C] = __ldg(edges + (xr.erel[k] + (u + 32u * q - lead) + (uint32_t)lane));
    };
    if (whole) {
#pragma unroll
        for (int q = 0; q < kWin; ++q) gather(q, window_entries(xr, n, u + 32u * q - lead, lane, k0));
    } else {
#pragma unroll
        for (int q = 0; q < kWin; ++q) {
            const uint32_t uq = u + 32u * q + (uint32_t)lane;
            const int k = window_entries(xr, n, u + 32u * q - lead, lane, k0);
            if (uq >= lo && uq < hi) gather(q, k);
        }
    }
    // the chunk before has left the staging area (lane 0 issued its copy); the
    // wait comes after this chunk's loads
    if (lane == 0) bulk_read_done();
    __syncwarp();
#pragma unroll
    for (int q = 0; q < kWin; ++q) stage_row<W>(stg + (q * 32 + lane) * W, v[q]);
    int32_t *g = obase + (size_t)u * W;
    if (whole) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) bulk_store(g, stg, kChunk * W * 4);
    } else {
        __syncwarp();
        const int w0 = lo > u ? (int)(lo - u) * W : 0;
        const int w1 = (hi > u ? (hi - u < (uint32_t)kChunk ? (int)(hi - u) : kChunk) : 0) * W;
        for (int i = w0 + lane; i < w1; i += 32) g[i] = stg[i];
        __syncwarp();   // the staging area is written again by the next chunk
    }
}

// As write_chunk for one window of 32 output rows of any width, without
// staging: lane l takes the window's vectors l, l + 32, ... of four words and
// fetches each word from the input row, or the list entry, that the lane
// holding the word's output row knows.  A table of 10 columns (800k -> 1.66M
// rows of 11) took 72.3 us with one output row per thread and scalar stores,
// 45.7 so.
__device__ __forceinline__ void write_window_any(uint32_t u, uint32_t lead, uint32_t lo, uint32_t hi, int C,
                                                 const ExpandRows &xr, int n, int &k0,
                                                 const int32_t *__restrict__ rows, const int32_t *__restrict__ edges,
                                                 int32_t *__restrict__ obase, int lane) {
    const int W = C + 1;
    const uint32_t uq = u + (uint32_t)lane;
    const int k = window_entries(xr, n, u - lead, lane, k0);
    int src = 0;
    int32_t nb = 0;
    if (uq >= lo && uq < hi) {
        src = (int)xr.row[k] * C;
        nb = __ldg(edges + (xr.erel[k] + (uq - lead)));
    }
    int32_t *g = obase + (size_t)u * W;
    const int words = 32 * W;
    const int w0 = lo > u ? (int)(lo - u) * W : 0;
    const int w1 = (hi > u ? (hi - u < 32u ? (int)(hi - u) : 32) : 0) * W;
    int r = 4 * lane / W, c = 4 * lane % W;                 // row and column of the lane's first word
    const int dr = 124 / W, dc = 124 % W;                   // from a vector's last word + 1 to the next's first
    for (int i = 0; i < words; i += 128) {                  // the same trips in every lane
        const int at = i + 4 * lane;
        int32_t v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int rr = r & 31;
            const int s = __shfl_sync(FULL, src, rr);
            const int32_t e = __shfl_sync(FULL, nb, rr);
            v[q] = e;
            if (c < C && at + q >= w0 && at + q < w1) v[q] = __ldg(rows + s + c);
            if (++c == W) { c = 0; ++r; }
        }
        if (at >= w0 && at + 4 <= w1) {
            *reinterpret_cast<int4 *>(g + at) = make_int4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (at + q >= w0 && at + q < w1) g[at + q] = v[q];
        }
        r += dr;
        c += dc;
        if (c >= W) { c -= W; ++r; }
    }
}

// As write_chunk for one window of 32 output rows of C + 1 columns, 9 to
// kMaxStaged: the lane's row goes to shared memory word by word, starting at
// column lane of an even pitch (an odd pitch needs no turn), so that the 32
// lanes' words fall in different banks.  The expansion of 800k -> 1.66M rows of 11
// columns took 41.4 us with write_window_any (ten instructions a word), 26.8 us
// so; both with cold caches.
__device__ __forceinline__ void write_window_staged(uint32_t u, uint32_t lead, uint32_t lo, uint32_t hi, int C,
                                                    const ExpandRows &xr, int n, int &k0,
                                                    const int32_t *__restrict__ rows,
                                                    const int32_t *__restrict__ edges, int32_t *__restrict__ obase,
                                                    int32_t *stg, int lane) {
    const int W = C + 1;
    const uint32_t uq = u + (uint32_t)lane;
    const bool whole = u >= lo && u + 32u <= hi;   // the same in every lane
    const int k = window_entries(xr, n, u - lead, lane, k0);
    if (lane == 0) bulk_read_done();   // the window before has left the staging area
    __syncwarp();
    if (uq >= lo && uq < hi) {
        const int32_t *src = rows + (int)xr.row[k] * C;
        int32_t *dst = stg + lane * W;
        const int32_t nb = __ldg(edges + (xr.erel[k] + (uq - lead)));
        int c = W % 2 == 0 ? lane % C : 0;
        int i = 0;
        for (; i + 4 <= C; i += 4) {
            int32_t v[4];
            int at[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                at[q] = c;
                v[q] = __ldg(src + c);
                c = c + 1 < C ? c + 1 : 0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[at[q]] = v[q];
        }
        for (; i < C; ++i) {
            dst[c] = __ldg(src + c);
            c = c + 1 < C ? c + 1 : 0;
        }
        dst[C] = nb;
    }
    int32_t *g = obase + (size_t)u * W;
    if (whole) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) bulk_store(g, stg, 32u * (uint32_t)W * 4u);
    } else {
        __syncwarp();
        const int w0 = lo > u ? (int)(lo - u) * W : 0;
        const int w1 = (hi > u ? (hi - u < 32u ? (int)(hi - u) : 32) : 0) * W;
        for (int i = w0 + lane; i < w1; i += 32) g[i] = stg[i];
        __syncwarp();
    }
}

// One CTA per slice: CTA k of the launch takes slice record k and writes local
// rows [slice kSliceRows, (slice + 1) kSliceRows) of its block.  W = C + 1
// output columns for 2 <= W <= 8; kStaged for 9 to kMaxStaged (32 W words of
// dynamic shared memory a warp); 0 for any width.  The CTA's chain before
// its first row is the record, the block's entries (copied asynchronously) and
// one barrier; finding the block by a scan of its group's counts and scanning
// the block's degrees there was two thirds of its instructions on steps of low
// fan-out.  Each warp takes a contiguous run of the slice's chunks, so it
// searches for its first entry once and walks on from there.  History rows are
// read through L1 (consecutive output rows of one input row reuse it).
//
// On 9M -> 18.6M rows of 6 columns the expansion took 112 us with the scans,
// 86 us from records (627 MB in and out: 7.3 TB/s), which bounds it by memory;
// the whole op 159 us before, 129 us after (124.5 launched ahead of the totals).
//
// NT = 128 when the slices are many and mostly full (wide_slices): more and
// smaller CTAs even out the last wave.  Those CTAs, 15 an SM, take nearly all
// of an SM's shared memory, and a grid that starts on an SM before they have
// left it would keep their small L1 for all of its run (a functional step
// behind one took 165 us more): they don't let it start early.
//
// CTAs per SM the register budget is set for: the widest instantiations need
// more registers to avoid spills
constexpr int kStaged = 1, kMaxStaged = 32;
template <int W, int NT>
constexpr int expand_min_ctas() { return (W <= 6 ? 8 : 6) * (kThreads / NT); }

template <int W, int NT>
__global__ void __launch_bounds__(NT, expand_min_ctas<W, NT>())
k2u_expand_kernel(const int32_t *__restrict__ hist, int C_rt, const int32_t *__restrict__ edges, const Entries en,
                  const SliceRec *__restrict__ slices, const uint32_t *__restrict__ head, int32_t *__restrict__ out) {
    constexpr int kWarps = NT / 32;
    __shared__ ExpandRows xr;
    __shared__ __align__(16) int32_t stage[W >= 2 ? kWarps * kChunk * W : 4];
    extern __shared__ __align__(16) int32_t stage_any[];   // kStaged
    const int C = W >= 2 ? W - 1 : C_rt;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    wait_prior_grid();   // the records are complete
    if constexpr (NT == kThreads) allow_dependent_grid();   // see above

    if (head != nullptr && blockIdx.x >= ld_prior(head)) return;

    // 1. the slice
    const uint4 *rec = reinterpret_cast<const uint4 *>(slices + blockIdx.x);
    const uint4 ra = ld_prior(rec), rb = ld_prior(rec + 1);
    const unsigned long long P = (unsigned long long)ra.y << 32 | ra.x;   // SliceRec: P, block, T | slice, n
    const uint32_t T = ra.w, slice = rb.x;
    const int n = (int)rb.y;
    const int64_t r0 = (int64_t)ra.z * kRowsPerBlock;

    // 2. its block's entries, with the total behind the last
    for (int i = t; i < min(n / 4 + 1, kRowsPerBlock / 4); i += NT) {
        copy16(xr.pos + 4 * i, en.pos + r0 + 4 * i);
        if (4 * i < n) copy16(xr.erel + 4 * i, en.rel + r0 + 4 * i);
        if (i % 2 == 0 && 4 * i < n) copy16(xr.row + 4 * i, en.row + r0 + 4 * i);
    }
    if (t == 0 && n == kRowsPerBlock) xr.pos[n] = T;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int32_t *hblk = hist + r0 * C;

    // 3. the slice's share of output rows [P, P + T): a run of chunks per warp
    constexpr int kStep = W >= 2 ? kChunk : 32;
    const uint32_t lead = (uint32_t)(P & 3ull), span = T + lead;
    const uint32_t u0 = slice * (uint32_t)kSliceRows;
    const uint32_t u1 = u0 >= span ? u0 : (span - u0 < (uint32_t)kSliceRows ? span : u0 + (uint32_t)kSliceRows);
    const uint32_t lo = u0 > lead ? u0 : lead;
    const uint32_t per = ((u1 - u0 + kStep - 1) / kStep + kWarps - 1) / kWarps * kStep;
    uint32_t u = u0 + (uint32_t)wid * per;
    const uint32_t ue = u < u1 ? (u1 - u < per ? u1 : u + per) : u;
    if (u >= ue) return;   // the same in every lane
    int32_t *obase = out + ((int64_t)P - lead) * (C + 1);
    int k0 = row_of(xr.pos, n, u >= lead ? u - lead : 0u);
    for (; u < ue; u += kStep) {
        if constexpr (W >= 2)
            write_chunk<W>(u, lead, lo, u1, xr, n, k0, hblk, edges, obase, stage + wid * (kChunk * W), lane);
        else if constexpr (W == kStaged)
            write_window_staged(u, lead, lo, u1, C, xr, n, k0, hblk, edges, obase, stage_any + wid * 32 * (C + 1), lane);
        else
            write_window_any(u, lead, lo, u1, C, xr, n, k0, hblk, edges, obase, lane);
    }
    if (W != 0 && lane == 0) bulk_read_done();   // the staging area goes with the CTA
}

// ------------------------------------------------- k2u expand, functional
// A hashed direction whose lists hold at most one vertex (a dense one takes
// wk_fused.cu): the expansion is a compaction of the matched rows with their neighbour appended.  One CTA per
// non-empty input block (its only slice).  Warp w takes rows 128 w .. 128 w +
// 127 in four passes of 32 consecutive rows, finds each matched row's output
// position by ballots, copies the row and its neighbour into shared memory
// (rows kPitch words apart, an odd pitch so the 32 lanes' rows fall in 32
// banks), and the CTA then streams the block's output words to HBM as
// aligned int4 stores.
template <int W>
__global__ void __launch_bounds__(kThreads)
k2u_expand_func_kernel(const int32_t *__restrict__ hist, int64_t R, const int32_t *__restrict__ nbr,
                       const SliceRec *__restrict__ slices, int32_t *__restrict__ out) {
    constexpr int C = W - 1;
    constexpr int kPitch = W | 1;
    __shared__ int32_t rows[kRowsPerBlock * kPitch];
    __shared__ uint32_t s_w[kThreads / 32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    allow_dependent_grid();

    // the block (every non-empty block has one slice)
    const SliceRec loc = slices[blockIdx.x];
    const int64_t r0 = (int64_t)loc.block * kRowsPerBlock;
    const int n = (int)((R - r0) < kRowsPerBlock ? (R - r0) : kRowsPerBlock);

    // matched rows and their block-local output positions
    int32_t x[4];
    unsigned bm[4];
    unsigned wtot = 0;
#pragma unroll
    for (int ps = 0; ps < 4; ++ps) {
        const int r = wid * 128 + ps * 32 + lane;
        x[ps] = r < n ? __ldg(nbr + r0 + r) : -1;
        bm[ps] = __ballot_sync(FULL, x[ps] >= 0);
        wtot += __popc(bm[ps]);
    }
    if (lane == 0) s_w[wid] = wtot;
    __syncthreads();
    unsigned base = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w)
        if (w < wid) base += s_w[w];
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int ps = 0; ps < 4; ++ps) {
        if (x[ps] >= 0) {
            const int r = wid * 128 + ps * 32 + lane;
            const unsigned q = base + __popc(bm[ps] & below);
            const int32_t *src = hist + (r0 + r) * C;
            int32_t *dst = rows + q * kPitch;
#pragma unroll
            for (int c = 0; c < C; ++c) dst[c] = __ldg(src + c);
            dst[C] = x[ps];
        }
        base += __popc(bm[ps]);
    }
    __syncthreads();

    // output words [P W, (P + T) W): int4 stores aligned to 16 B of out
    const unsigned long long P = loc.P;
    const uint32_t T = loc.T;
    const uint32_t lead = (uint32_t)((P * W) & 3ull), words = T * W;
    int32_t *g = out + (P * W - lead);
    for (uint32_t i = (uint32_t)t; 4u * i < lead + words; i += kThreads) {
        int32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t kk = 4u * i + j - lead;   // wraps above `words` before the lead
            v[j] = kk < words ? rows[(kk / W) * kPitch + kk % W] : 0;
        }
        if (4u * i >= lead && 4u * i + 4u <= lead + words) {
            reinterpret_cast<int4 *>(g)[i] = make_int4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t kk = 4u * i + j - lead;
                if (kk < words) g[4u * i + j] = v[j];
            }
        }
    }
}

// ------------------------------------------------------- k2k / k2c probe
// One CTA per block of input rows (two blocks per CTA, with eight rounds of
// loads in flight per lane, took 48 registers and ran slower).  Membership is
// the lower bound of the end value in the row's ascending list.  Lists hold
// distinct ids, so that is also the position where the reference's linear scan
// (core/engine.hpp:172-179) stops: group_sums[2 g + 1] += the entries that scan
// touches (position + 1 on a match, the whole list otherwise), group_sums[2 g]
// += rows kept.
//
// The searches are chains of dependent reads, so a lane's rounds are searched two
// at a time.  One after another they take longer (422k rows of 8 columns in runs of
// 40, half kept, 51.7 us a step, 35.3 so; 2.8k rows 46.8 and 31.8), four at a time a
// short search pays for the longest of four (9M rows of 3 columns, half kept, 275
// us, 257 so and 266 one after another; nearly all kept 460, 441 and 427).
template <bool DENSE>
__global__ void __launch_bounds__(kThreads, 6)
filter_probe_kernel(const int32_t *__restrict__ hist, int64_t R, int C, int scol, int ecol,
                    int32_t end_const, uint32_t dir, PredView pv,
                    uint32_t *__restrict__ mask, unsigned int *__restrict__ blk_nz,
                    unsigned long long *__restrict__ group_sums, unsigned long long *__restrict__ clear,
                    int64_t nclear, int *err) {
    wait_prior_grid();   // before anything is read or cleared
    // the copy behind it does not start early: its CTAs would keep to the small
    // shared memory of this kernel's SMs, few at a time (51 -> 75 us a step on 422k
    // rows of 8 columns)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the other sums buffer, read by the previous op's write or expansion, is
    // cleared for the next op (a few hundred words at most)
    for (int64_t w = (int64_t)blockIdx.x * kThreads + threadIdx.x; w < nclear; w += (int64_t)gridDim.x * kThreads)
        clear[w] = 0ull;
    const int64_t b = blockIdx.x;
    const int64_t wrow0 = b * kRowsPerBlock + (int64_t)warp * (kRounds * 32);
    if (threadIdx.x == 0) prefetch_rows(hist, R, C, (b + kPrefetch) * kRowsPerBlock, (b + kPrefetch + 1) * kRowsPerBlock);
    int32_t v[kRounds], tg[kRounds];
#pragma unroll
    for (int rd = 0; rd < kRounds; ++rd) {
        const int64_t r = wrow0 + rd * 32 + lane;
        v[rd] = r < R ? ld_prior(hist + r * C + scol) : -1;
        tg[rd] = (r < R && ecol >= 0) ? ld_prior(hist + r * C + ecol) : end_const;
    }
    // every round's list: offset and entries (none past the table)
    uint32_t o[kRounds], d[kRounds];
    if constexpr (DENSE) {
        const uint32_t vmin = dir ? pv.vmin[1] : pv.vmin[0], dn = dir ? pv.dn[1] : pv.dn[0];
        const uint32_t *rp = dir ? pv.rp[1] : pv.rp[0];
#pragma unroll
        for (int rd = 0; rd < kRounds; ++rd) {
            o[rd] = d[rd] = 0u;
            const uint32_t x = (uint32_t)v[rd] - vmin;   // wraps above dn below vmin
            if (v[rd] > 0 && x < dn) {
                o[rd] = __ldg(rp + x);
                d[rd] = __ldg(rp + x + 1);
            } else if (v[rd] == 0) {   // index key: the hash table
                d[rd] = probe_seg(pv.buckets, pv.nmain, pv.nover, seg_key(0u, dir), &o[rd], err);
                d[rd] += o[rd];
            }
        }
#pragma unroll
        for (int rd = 0; rd < kRounds; ++rd) d[rd] -= o[rd];
    } else {
        const unsigned present = may_hold(pv, dir, v);
#pragma unroll
        for (int rd = 0; rd < kRounds; ++rd) {
            o[rd] = d[rd] = 0u;
            const bool here = (present >> rd) & 1u;
            if (__any_sync(FULL, here)) probe_warp(pv, here ? v[rd] : -1, dir, o[rd], d[rd], err);
        }
    }
    // lo[rd]: the first entry not below tg[rd], two rounds' searches at a time
    static_assert(kRounds % 2 == 0, "rounds come in pairs");
    uint32_t lo[kRounds], hi[kRounds];
#pragma unroll
    for (int rd = 0; rd < kRounds; ++rd) {
        lo[rd] = 0u;
        hi[rd] = d[rd];
    }
#pragma unroll
    for (int q = 0; q < kRounds; q += 2) {
        while (lo[q] < hi[q] || lo[q + 1] < hi[q + 1]) {
            int32_t x[2];
#pragma unroll
            for (int k = q; k < q + 2; ++k)
                x[k - q] = lo[k] < hi[k] ? __ldg(pv.edges + o[k] + ((lo[k] + hi[k]) >> 1)) : 0;
#pragma unroll
            for (int k = q; k < q + 2; ++k) {
                if (lo[k] < hi[k]) {
                    const uint32_t mid = (lo[k] + hi[k]) >> 1;
                    if (x[k - q] < tg[k]) lo[k] = mid + 1;
                    else hi[k] = mid;
                }
            }
        }
    }
    int32_t e[kRounds];
#pragma unroll
    for (int rd = 0; rd < kRounds; ++rd) e[rd] = lo[rd] < d[rd] ? __ldg(pv.edges + o[rd] + lo[rd]) : 0;
    unsigned int my_nz = 0u;   // kept rows (lane 0)
    unsigned long long my_scan = 0ull;
#pragma unroll
    for (int rd = 0; rd < kRounds; ++rd) {
        const bool found = lo[rd] < d[rd] && e[rd] == tg[rd];
        my_scan += found ? lo[rd] + 1u : d[rd];
        const uint32_t m = __ballot_sync(FULL, found);
        const int64_t row0 = wrow0 + rd * 32;
        if (lane == 0 && row0 < R) {
            mask[row0 >> 5] = m;
            my_nz += __popc(m);
        }
    }
    block_sum2(my_scan, my_nz);
    if (threadIdx.x == 0) {
        blk_nz[b] = my_nz;
        unsigned long long *gs = group_sums + 2 * (b >> kGroupShift);
        if (my_nz) atomicAdd(gs, (unsigned long long)my_nz);
        if (my_scan) atomicAdd(gs + 1, my_scan);
    }
}

// ----------------------------------------------------------- filter write
// A write CTA takes kWriteBlocks consecutive blocks of input rows, one per
// warp (or one block, filter_per_block), all in one group of 2^kGroupShift blocks.  Their output prefixes need
// no look-back and no wait: the probe kernel added every block's kept-row
// count into its group's sum, so the prefix of the CTA's first block is the
// sum of the group sums before its group and of the block counts before it in
// the group -- one CTA reduction -- and warp w adds the counts of the CTA's
// blocks before its own.  Each warp then writes its block alone: the kept
// rows' positions from the block's 32 mask words (one per lane, a warp scan
// of their popcounts), then the block's output words [P C, (P + nb) C) as
// aligned 16 B stores where whole, each word gathered from its kept row (the
// block's rows stay in L1 and L2 while the warp copies them).
constexpr int kWriteBlocks = kThreads / 32;
static_assert(((1 << kGroupShift) % kWriteBlocks) == 0, "a write CTA's blocks share a group");

template <int CT, bool PB>   // CT: the columns, or 0 for any (C_rt); PB: a block per CTA
__global__ void __launch_bounds__(kThreads)
filter_write_kernel(const int32_t *__restrict__ hist, int64_t R, int C_rt, const uint32_t *__restrict__ mask,
                    const unsigned int *__restrict__ blk_nz, const unsigned long long *__restrict__ group_sums,
                    int32_t *__restrict__ out) {
    __shared__ uint16_t sel[PB ? 1 : kWriteBlocks][kRowsPerBlock];   // each block's kept rows, in order
    __shared__ unsigned long long s_part[kThreads / 32];
    __shared__ unsigned int s_nz[kWriteBlocks];
    const int C = CT > 0 ? CT : C_rt;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int64_t nblk = (R + kRowsPerBlock - 1) / kRowsPerBlock;
    const int64_t b0 = (int64_t)blockIdx.x * (PB ? 1 : kWriteBlocks);
    const int64_t g = b0 >> kGroupShift;
    wait_prior_grid();

    // 1. the prefix of block b0, and the CTA's blocks' counts
    unsigned long long x = 0ull;
    for (int64_t i = t; i < g; i += kThreads) x += ld_prior(group_sums + 2 * i);
    for (int64_t i = (g << kGroupShift) + t; i < b0; i += kThreads) x += ld_prior(blk_nz + i);
    if (t < kWriteBlocks) s_nz[t] = b0 + t < nblk ? ld_prior(blk_nz + b0 + t) : 0u;
    x = warp_sum(x);
    if (lane == 0) s_part[w] = x;
    __syncthreads();
    unsigned long long P = 0ull;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) P += s_part[i];
    if constexpr (!PB)
        for (int i = 0; i < w; ++i) P += s_nz[i];
    const unsigned int nb = s_nz[PB ? 0 : w];
    if (nb == 0u) return;   // the block keeps nothing (or lies past the table)

    // 2. the block's kept rows, in order
    const int64_t b = PB ? b0 : b0 + w, r0 = b * kRowsPerBlock;
    const int64_t wi = (r0 >> 5) + lane, nwords = (R + 31) >> 5;
    uint32_t m = wi < nwords ? ld_prior(mask + wi) : 0u;   // bits past R are 0
    const unsigned int c = __popc(m);
    unsigned int pos = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(FULL, pos, o);
        if (lane >= o) pos += v;
    }
    pos -= c;
    uint16_t *ws = sel[PB ? 0 : w];
    if (PB && lane / (32 / (kThreads / 32)) != w) m = 0u;   // each warp lists its four words' rows
    while (m) {
        ws[pos++] = (uint16_t)(lane * 32 + __ffs(m) - 1);
        m &= m - 1u;
    }
    if constexpr (PB) __syncthreads();
    else __syncwarp();

    // 3. output words [P C, (P + nb) C) as int4 stores aligned to 16 B of out
    const int32_t *hb = hist + r0 * C;
    const uint32_t words = nb * (uint32_t)C;
    const uint32_t lead = (uint32_t)((P * (unsigned long long)C) & 3ull);
    int32_t *gout = out + (P * (unsigned long long)C - lead);
    for (uint32_t u = (uint32_t)(PB ? t : lane); 4u * u < lead + words; u += PB ? kThreads : 32u) {
        int32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t kk = 4u * u + (uint32_t)j - lead;   // wraps above `words` before the lead
            v[j] = kk < words ? __ldg(hb + (int)ws[kk / (uint32_t)C] * C + (int)(kk % (uint32_t)C)) : 0;
        }
        if (4u * u >= lead && 4u * u + 4u <= lead + words) {
            reinterpret_cast<int4 *>(gout)[u] = make_int4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t kk = 4u * u + (uint32_t)j - lead;
                if (kk < words) gout[4u * u + j] = v[j];
            }
        }
    }
}

// ------------------------------------------------------------- list copy
__global__ void copy_list_kernel(const int32_t *__restrict__ src, int64_t n, int32_t *__restrict__ dst) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = __ldg(src + i);
}

// ============================================================== launchers
static inline unsigned int nblocks_rows(int64_t R) {
    return (unsigned int)((R + kRowsPerBlock - 1) / kRowsPerBlock);
}

static cudaLaunchConfig_t dependent_launch(cudaLaunchAttribute *attr, unsigned int grid, cudaStream_t st) {
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

void launch_k2u_count(const int32_t *hist, int64_t R, int C, int scol, uint32_t dir, PredView pv, const Entries &en,
                      unsigned long long *blk_sum, unsigned long long *group_sums, int *err, bool func,
                      unsigned long long *clear, int64_t nclear, int sms, cudaStream_t st) {
    const bool dense = (dir ? pv.rp[1] : pv.rp[0]) != nullptr;
    const unsigned int nb = nblocks_rows(R);
    // two blocks per CTA once the op has enough blocks to fill the GPU with half as many CTAs
    if (sms < 1) sms = 1;
    const bool pair = dense && nb >= 16u * (unsigned int)sms;
    cudaLaunchAttribute attr[1];
#define WK_COUNT(F, D, B)                                                                                       \
    do {                                                                                                       \
        const cudaLaunchConfig_t cfg = dependent_launch(attr, (nb + B - 1) / B, st);                           \
        cudaLaunchKernelEx(&cfg, k2u_count_kernel<F, D, B>, hist, R, C, scol, dir, pv, en, blk_sum, group_sums, \
                           err, clear, nclear);                                                                \
    } while (0)
    if (func) WK_COUNT(true, false, 1);   // hashed: a dense one takes wk_fused.cu
    else if (dense && pair) WK_COUNT(false, true, 2);
    else if (dense) WK_COUNT(false, true, 1);
    else WK_COUNT(false, false, 1);
#undef WK_COUNT
}

// launched so that its CTAs are in place when the kernel before it finishes
void launch_publish(const Publish &pub, const SlicePlan &plan, cudaStream_t st) {
    cudaLaunchAttribute attr[1];
    const int64_t ng = plan.slices ? (plan.nblk + (1 << kGroupShift) - 1) >> kGroupShift : 0;
    const cudaLaunchConfig_t cfg = dependent_launch(attr, (unsigned int)(1 + ng), st);
    cudaLaunchKernelEx(&cfg, publish_kernel, pub, plan);
}

void launch_k2u_expand_func(const int32_t *hist, int64_t R, int C, const int32_t *nbr, const SliceRec *slices,
                            unsigned int n, int32_t *out, cudaStream_t st) {
    if (n == 0u) return;
#define WK_EXPAND_F(WC) k2u_expand_func_kernel<WC><<<n, kThreads, 0, st>>>(hist, R, nbr, slices, out)
    switch (C + 1) {
        case 2: WK_EXPAND_F(2); break;
        case 3: WK_EXPAND_F(3); break;
        case 4: WK_EXPAND_F(4); break;
        case 5: WK_EXPAND_F(5); break;
        case 6: WK_EXPAND_F(6); break;
        case 7: WK_EXPAND_F(7); break;
        default: WK_EXPAND_F(8); break;
    }
#undef WK_EXPAND_F
}

// More slices than CTAs of 256 threads fit at once, half full on average or
// more: 120k rows of fan-out 100 (1524 slices, 1.25 waves of such CTAs) take
// 43.2 us with 128 threads a CTA and 47.7 us with 256.  On steps of low fan-out,
// a slice per block of rows, each CTA copies more than it writes: 9M -> 18.6M
// rows take 144 us with 128 threads and 129 us with 256.
bool wide_slices(unsigned long long slices, unsigned long long rows_out, int sms) {
    return slices > 8ull * (unsigned long long)(sms < 1 ? 1 : sms) && rows_out / slices >= kSliceRows / 2;
}

void launch_k2u_expand(const int32_t *hist, int C, const int32_t *edges, const Entries &en, const SliceRec *slices,
                       unsigned int n, const uint32_t *head, bool wide, int32_t *out, cudaStream_t st) {
    if (n == 0u) return;
    const int W = C + 1;
    const size_t any = W > 8 && W <= kMaxStaged ? (size_t)32 * W * 4 : 0;   // per warp
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = dependent_launch(attr, n, st);
    if (head == nullptr) cfg.numAttrs = 0;
#define WK_EXPAND_T(WC, NT)                                                                                \
    do {                                                                                                   \
        cfg.blockDim = dim3(NT);                                                                           \
        cfg.dynamicSmemBytes = any * (NT / 32);                                                            \
        cudaLaunchKernelEx(&cfg, k2u_expand_kernel<WC, NT>, hist, C, edges, en, slices, head, out);        \
    } while (0)
#define WK_EXPAND(WC)                                      \
    do {                                                   \
        if (wide) WK_EXPAND_T(WC, 128);                    \
        else WK_EXPAND_T(WC, 256);                         \
    } while (0)
    switch (W) {
        case 2: WK_EXPAND(2); break;
        case 3: WK_EXPAND(3); break;
        case 4: WK_EXPAND(4); break;
        case 5: WK_EXPAND(5); break;
        case 6: WK_EXPAND(6); break;
        case 7: WK_EXPAND(7); break;
        case 8: WK_EXPAND(8); break;
        default:
            if (any) WK_EXPAND(kStaged);
            else WK_EXPAND_T(0, 256);
            break;
    }
#undef WK_EXPAND
#undef WK_EXPAND_T
}

// Load every k2u count and expansion kernel now (with lazy module loading a
// kernel's code is otherwise loaded, and device memory taken for it, at its
// first launch).
int preload_k2u_kernels() {
    cudaFuncAttributes a;
    cudaError_t e = cudaSuccess;
    auto get = [&](const void *f) {
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, f);
    };
    get((const void *)k2u_count_kernel<false, false, 1>);
    get((const void *)k2u_count_kernel<false, true, 1>);
    get((const void *)k2u_count_kernel<false, true, 2>);
    get((const void *)k2u_count_kernel<true, false, 1>);
    get((const void *)publish_kernel);
    get((const void *)k2u_expand_kernel<0, 256>);
    get((const void *)k2u_expand_kernel<kStaged, 128>);
    get((const void *)k2u_expand_kernel<kStaged, 256>);
    get((const void *)k2u_expand_kernel<2, 128>);
    get((const void *)k2u_expand_kernel<2, 256>);
    get((const void *)k2u_expand_kernel<3, 128>);
    get((const void *)k2u_expand_kernel<3, 256>);
    get((const void *)k2u_expand_kernel<4, 128>);
    get((const void *)k2u_expand_kernel<4, 256>);
    get((const void *)k2u_expand_kernel<5, 128>);
    get((const void *)k2u_expand_kernel<5, 256>);
    get((const void *)k2u_expand_kernel<6, 128>);
    get((const void *)k2u_expand_kernel<6, 256>);
    get((const void *)k2u_expand_kernel<7, 128>);
    get((const void *)k2u_expand_kernel<7, 256>);
    get((const void *)k2u_expand_kernel<8, 128>);
    get((const void *)k2u_expand_kernel<8, 256>);
    return (int)e;
}

void launch_filter_probe(const int32_t *hist, int64_t R, int C, int scol, int ecol, int32_t end_const,
                         uint32_t dir, PredView pv, uint32_t *mask, unsigned int *blk_nz,
                         unsigned long long *group_sums, unsigned long long *clear, int64_t nclear,
                         int *err, cudaStream_t st) {
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = dependent_launch(attr, nblocks_rows(R), st);
    auto *k = (dir ? pv.rp[1] : pv.rp[0]) != nullptr ? filter_probe_kernel<true> : filter_probe_kernel<false>;
    cudaLaunchKernelEx(&cfg, k, hist, R, C, scol, ecol, end_const, dir, pv, mask, blk_nz, group_sums, clear, nclear, err);
}

void launch_filter_write(const int32_t *hist, int64_t R, int C, const uint32_t *mask, const unsigned int *blk_nz,
                         const unsigned long long *group_sums, int32_t *out, int sms, cudaStream_t st) {
    const unsigned int nb = nblocks_rows(R);
    const bool pb = filter_per_block(nb, sms);
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = dependent_launch(attr, pb ? nb : (nb + kWriteBlocks - 1) / kWriteBlocks, st);
#define WK_FWRITE(CC)                                                                                             \
    do {                                                                                                          \
        if (pb) cudaLaunchKernelEx(&cfg, filter_write_kernel<CC, true>, hist, R, C, mask, blk_nz, group_sums, out); \
        else cudaLaunchKernelEx(&cfg, filter_write_kernel<CC, false>, hist, R, C, mask, blk_nz, group_sums, out);   \
    } while (0)
    switch (C) {
        case 1: WK_FWRITE(1); break;
        case 2: WK_FWRITE(2); break;
        case 3: WK_FWRITE(3); break;
        case 4: WK_FWRITE(4); break;
        case 5: WK_FWRITE(5); break;
        case 6: WK_FWRITE(6); break;
        case 7: WK_FWRITE(7); break;
        case 8: WK_FWRITE(8); break;
        default: WK_FWRITE(0); break;
    }
#undef WK_FWRITE
}

void launch_copy_list(const int32_t *src, int64_t n, int32_t *dst, cudaStream_t st) {
    int64_t nb = (n + 255) / 256;
    if (nb > 152 * 16) nb = 152 * 16;
    if (nb < 1) nb = 1;
    copy_list_kernel<<<(unsigned int)nb, 256, 0, st>>>(src, n, dst);
}

}  // namespace dev
}  // namespace wk
