// k2u, k2k and k2c over a dense functional direction in one launch (sm_103a).
//
// A direction that keeps one neighbour per id (PredView::nb) answers a row
// with one 4 B read and gives at most one output row per input row, so nothing
// has to reach the host between counting and writing where the output buffer
// holds the rows there are (the device leaves out what it does not hold, and the
// host, which learns the rows from the same launch, has the blocks written again):
//
//   k2u     : the rows that have a neighbour, with it appended
//   k2k/k2c : the rows whose neighbour is the end value
//
// What bounds it.  Counting is bound by the look-ups: a random 4 B read is one
// L1 tag look-up per lane and a 32 B sector from L2, at most 245 G/s on this
// chip however the load is written (12M of them take 49 us), while DRAM is
// half idle.  Writing streams: the table in, the output out.  As two kernels
// in a row each leaves the other's resource idle, and the second reads the
// table from DRAM again.  Here both kinds of CTA run at once: CTAs are ordered
// so that the count of block b + lag and the writing of block b are neighbours,
// with a lag of some 1200 blocks of 1024 rows.  What a write CTA needs has then
// been counted before (1216 CTAs are in flight at most), and most of the rows
// it reads are still in L2.  The op is left bound by L2 bandwidth (1.1 GB
// through it in 130 us on 12M rows of 4 columns, a third of it look-ups).
//
// Two kernels and a host round trip before, this launch after, us a call:
// k2u on 12M rows of 4 columns 163 -> 131, k2k on 10M rows of 3 105 -> 95, k2c on 3M
// rows of 6 50 -> 48; k2u on 50k rows of 6 about 49 -> 22.  A
// single pass with a decoupled look-back was slower (177 / 139 / 65): every tile
// waited for the slowest load among the 300 tiles in flight before it.
//
// A write CTA checks that the groups of 256 blocks up to its own have been
// counted, and waits if not.  It depends only on CTAs before it in the grid,
// which the device starts in order, so the wait ends; it is bounded all the
// same, and an op whose wait ran out runs again as the general kernels.
//
// Per-block counts and per-group sums are those of the two-kernel ops: a
// group's word holds its counted blocks (low 16 bits) and kept rows.  One CTA
// placed behind the last count waits for every group and writes the op's
// totals into pinned host memory, so that the host goes on while a k2u op's last
// blocks are still written.  A filter's host waits for every kept row too: a
// caller may reuse the input of a k2k or k2c op as soon as it returns.
#include "wk_kernels.h"
#include "wk_probe.cuh"

namespace wk {
namespace dev {

#define FULL 0xffffffffu

constexpr int kOct = 8;   // blocks per step of the CTA order

__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long warp_add(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

struct Fused {
    const int32_t *hist;
    int64_t R, nblk;
    int C, scol, ecol;            // k2k: the end column; k2c: ecol < 0 and end_const
    int32_t end_const;
    uint32_t dir;
    const int32_t *nb;            // the direction's neighbour array, ids [vmin, vmin + dn)
    uint32_t vmin, dn;
    int32_t *nbr;                 // k2u: per row, the neighbour or -1
    uint32_t *mask;               // filter: a bit per row
    unsigned int *blk_nz;         // kept rows per block
    unsigned long long *gs;       // two words per group, zero at launch
    int *err;
    unsigned long long *written;  // filter: write CTAs done
    unsigned long long *clear;    // the other sums buffer, cleared for the next op
    int64_t nclear;
    int32_t *out;
    unsigned long long max_rows;  // k2u: rows that out has room for
    unsigned long long *pub;      // pinned host words: [0] seq, [2] error bits, [3] rows, [4] second count
    unsigned long long seq;
    int steps, lag;               // octets of blocks, and how many the writing trails by
    int first;                    // the launch's first CTA in that order
    int pub_polls, write_polls;   // the waits' bounds (FusedOp)
};

// What CTA `i` does: role 0 counts unit `unit` of octet `oct`, 1 writes it, 2
// publishes.  nc count and nw write CTAs per octet; the first `lag` octets'
// counts, then per octet its counts and an earlier one's writes, the
// publisher, and the last `lag` octets' writes.
struct Role {
    int kind, oct, unit;
};
__device__ __forceinline__ Role role_of(int i, int steps, int lag, int nc, int nw) {
    const int head = lag * nc, mid = (steps - lag) * (nc + nw);
    Role r;
    if (i < head) {
        r.kind = 0;
        r.oct = i / nc;
        r.unit = i % nc;
    } else if (i < head + mid) {
        const int j = i - head, s = j / (nc + nw), u = j % (nc + nw);
        r.kind = u < nc ? 0 : 1;
        r.oct = u < nc ? s + lag : s;
        r.unit = u < nc ? u : u - nc;
    } else if (i == head + mid) {
        r.kind = 2;
        r.oct = r.unit = 0;
    } else {
        const int j = i - head - mid - 1;
        r.kind = 1;
        r.oct = steps - lag + j / nw;
        r.unit = j % nw;
    }
    return r;
}

// Wait until groups 0 .. g are counted; the sum of the kept rows of groups
// before g, the same in every thread (and of all of them when g is past the
// last group).  False when the wait ran out, which the error word says by then.
//
// A write CTA's wait may run out at the moment the groups are complete.  So the CTA
// sets the error first and then looks once more: if the groups are not there now,
// either, the publisher, which reads the word after it has seen them all, finds
// the error in it and does not report an op whose block is missing.
struct WaitShared {
    unsigned long long sum[2][kThreads / 32];
    int there[2][kThreads / 32];
};
__device__ __forceinline__ bool groups_before(const Fused &a, int64_t g, int polls, WaitShared &sh,
                                              unsigned long long &sum) {
    const int64_t ng = (a.nblk + (1 << kGroupShift) - 1) >> kGroupShift;
    const int64_t last = g < ng ? g : ng - 1;
    const int t = threadIdx.x;
    for (int poll = 0;; ++poll) {
        bool there = true;
        unsigned long long x = 0ull;
        for (int64_t i = t; i <= last; i += kThreads) {
            const int64_t left = a.nblk - (i << kGroupShift);
            const unsigned long long w = ld_acquire64(a.gs + 2 * i);
            there = there && (w & 0xffffull) == (unsigned long long)(left < (1 << kGroupShift) ? left : (1 << kGroupShift));
            if (i < g) x += w >> 16;
        }
        // a group's sum is at most 2^18: a warp's fits 32 bits for up to 2^16 groups
        x = ng <= (1 << 16) ? (unsigned long long)__reduce_add_sync(FULL, (unsigned int)x) : warp_add(x);
        there = __all_sync(FULL, there);
        if ((t & 31) == 0) {
            sh.sum[poll & 1][t >> 5] = x;
            sh.there[poll & 1][t >> 5] = there;
        }
        __syncthreads();   // one a poll: the polls alternate between two sets of words
        int all = 1;
        sum = 0ull;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) {
            all &= sh.there[poll & 1][w];
            sum += sh.sum[poll & 1][w];
        }
        if (all) return true;
        if (poll > polls) return false;
        if (poll == polls) {
            if (t == 0) atomicOr(a.err, kErrWait);
            __threadfence();
            __syncthreads();
        } else {
            __nanosleep(100);
        }
    }
}

// A row whose start is an index key (a value of 0), looked up in the hash
// table: whether its list holds v, and the entries a linear scan touches.
__device__ __forceinline__ bool index_key_holds(const PredView &pv, uint32_t dir, int32_t v, unsigned int *scanned,
                                             int *err) {
    uint32_t off;
    const uint32_t deg = probe_seg(pv.buckets, pv.nmain, pv.nover, seg_key(0u, dir), &off, err);
    const int32_t *e = pv.edges + off;
    uint32_t lo = 0, hi = deg;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(e + mid) < v) lo = mid + 1;
        else hi = mid;
    }
    const bool f = lo < deg && __ldg(e + lo) == v;
    *scanned = f ? lo + 1 : deg;
    return f;
}

// Count BPC blocks from block b0: every start vertex, then every neighbour, in
// flight together (4 BPC rounds of 32 rows a warp).
template <int CT, bool FILTER, int BPC>
__device__ __forceinline__ void count_blocks(const Fused &a, const PredView &pv, int64_t b0, unsigned int (*s_n)[kThreads / 32],
                                             unsigned long long *s_x) {
    constexpr int kRounds = kRowsPerBlock / kThreads, NR = kRounds * BPC;
    const int C = CT > 0 ? CT : a.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto row_at = [&](int rd) -> int64_t {
        return (b0 + rd / kRounds) * kRowsPerBlock + warp * (kRounds * 32) + (rd % kRounds) * 32 + lane;
    };
    int32_t v[NR], tg[FILTER ? NR : 1];
#pragma unroll
    for (int rd = 0; rd < NR; ++rd) {
        const int64_t r = row_at(rd);
        v[rd] = r < a.R ? ld_prior(a.hist + r * C + a.scol) : -1;
        if constexpr (FILTER) tg[rd] = r < a.R && a.ecol >= 0 ? ld_prior(a.hist + r * C + a.ecol) : a.end_const;
    }
    unsigned zeros = 0u;   // rounds in which this lane's row starts at an index key
    int32_t g[NR];
#pragma unroll
    for (int rd = 0; rd < NR; ++rd) {
        const uint32_t x = (uint32_t)v[rd] - a.vmin;   // wraps above dn below vmin
        g[rd] = (v[rd] > 0 && x < a.dn) ? __ldg(a.nb + x) : -1;
        if (v[rd] == 0) zeros |= 1u << rd;
    }
    unsigned int n[BPC];
    unsigned long long extra = 0ull;   // in lane 0 unless a row started at an index key
    bool keyed = false;
#pragma unroll
    for (int j = 0; j < BPC; ++j) n[j] = 0u;
#pragma unroll
    for (int rd = 0; rd < NR; ++rd) {
        const int64_t r = row_at(rd);
        bool keep = g[rd] >= 0;
        if constexpr (FILTER) {
            const unsigned had = __ballot_sync(FULL, keep);
            extra += lane == 0 ? (unsigned long long)__popc(had) : 0ull;   // entries a linear scan touches
            keep = keep && g[rd] == tg[rd];
            if (__any_sync(FULL, (zeros >> rd) & 1u)) {
                unsigned int sc = 0u;
                if ((zeros >> rd) & 1u) keep = index_key_holds(pv, a.dir, tg[rd], &sc, a.err);
                extra += sc;   // of every lane: summed over the warp below
                keyed = true;
            }
            const unsigned m = __ballot_sync(FULL, keep);
            if (lane == 0 && r < a.R) a.mask[r >> 5] = m;
            n[rd / kRounds] += (unsigned)__popc(m);
        } else {
            if (r < a.R) a.nbr[r] = g[rd];
            n[rd / kRounds] += (unsigned)__popc(__ballot_sync(FULL, keep));
        }
    }
    if constexpr (!FILTER) extra = __any_sync(FULL, zeros != 0u) ? 1ull : 0ull;   // the op reruns unspecialised
    if (keyed) extra = warp_add(extra);   // the same in every lane
    if (lane == 0) {
#pragma unroll
        for (int j = 0; j < BPC; ++j) s_n[j][warp] = n[j];
        s_x[warp] = extra;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sum = 0ull, x = 0ull;
        unsigned int done = 0u;
#pragma unroll
        for (int j = 0; j < BPC; ++j) {
            unsigned int c = 0u;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) c += s_n[j][w];
            if (b0 + j < a.nblk) {
                a.blk_nz[b0 + j] = c;
                sum += c;
                ++done;
            }
        }
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) x += s_x[w];
        unsigned long long *gw = a.gs + 2 * (b0 >> kGroupShift);
        if (x) atomicAdd(gw + 1, x);
        __threadfence();   // the CTA's rows and counts, before the group's word says so
        if (done) atomicAdd(gw, (sum << 16) | done);
    }
}

// One row of C words, in the widest loads that C (and the table's alignment) allows.
template <int C>
__device__ __forceinline__ void copy_row_regs(const int32_t *src, int32_t *v, bool aligned) {
    if (C % 4 == 0 && aligned) {
#pragma unroll
        for (int c = 0; c + 3 < C; c += 4) {
            const int4 x = ld_prior(reinterpret_cast<const int4 *>(src + c));
            v[c] = x.x; v[c + 1] = x.y; v[c + 2] = x.z; v[c + 3] = x.w;
        }
    } else if (C % 2 == 0 && aligned) {
#pragma unroll
        for (int c = 0; c + 1 < C; c += 2) {
            const int2 x = ld_prior(reinterpret_cast<const int2 *>(src + c));
            v[c] = x.x; v[c + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = ld_prior(src + c);
    }
}

// The kept rows of this thread's block of group g before block b, by warps
// (at most 2^18).
__device__ __forceinline__ unsigned int blocks_before(const Fused &a, int64_t b) {
    static_assert(kThreads == (1 << kGroupShift), "one thread per block of a group");
    const int64_t i = ((b >> kGroupShift) << kGroupShift) + threadIdx.x;
    return __reduce_add_sync(FULL, i < b ? ld_l2(a.blk_nz + i) : 0u);
}

// Write block b of a k2u op: its matched rows with the neighbour appended,
// packed in shared memory at the output's 16 B phase; its whole vectors leave
// by the copy engine, which spares the load-store unit the look-ups need (some 3
// of 138 us a step on 12M rows of 4 columns).
// The rows are loaded before the wait for the groups (they are in L2), unless the
// block's count says that few of them are kept: then only those are read, behind it.
// The count is there already for nearly every block where the writing trails the
// counting; read too early it is some earlier op's, and costs time only.  12M rows of
// 4 columns take 119 / 92 / 80 / 67 us a step with all / half / one in eight / none of the rows
// kept; with every block's rows loaded ahead 125 / 97 / 81 / 67; as two kernels,
// whose second is not launched for none, 169 / 131 / 102 / 48.  Rows of one or two
// columns, and tables short enough to be counted before the first block is written,
// are loaded ahead always (4M rows of one column 41.1 us, 44 by the count; 600k 18
// and 23).  The ballots are taken twice: held in registers they made the kernel spill.
// Nothing is written when the wait ran out.
template <int C>
__device__ __forceinline__ void write_k2u(const Fused &a, int64_t b, WaitShared &s_wait, int32_t *buf,
                                          unsigned int *s_w, unsigned int *s_b) {
    constexpr int W = C + 1, kPasses = kRowsPerBlock / kThreads;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int64_t r0 = b * kRowsPerBlock;
    const int n = (int)((a.R - r0) < kRowsPerBlock ? (a.R - r0) : kRowsPerBlock);
    const bool aligned = ((uintptr_t)a.hist & 15u) == 0;
    int32_t x[kPasses], v[kPasses][W];
    unsigned kept = 0u;
    const bool most = C <= 2 || a.lag >= a.steps || ld_l2(a.blk_nz + b) >= (unsigned)kRowsPerBlock / 4;
    if (most) {
#pragma unroll
        for (int q = 0; q < kPasses; ++q) {
            const int r = wid * (32 * kPasses) + q * 32 + lane;
            if (r < n) copy_row_regs<C>(a.hist + (r0 + r) * C, v[q], aligned);
        }
    }
    unsigned long long P;
    if (!groups_before(a, b >> kGroupShift, a.write_polls, s_wait, P)) return;
    const bool any = most || ld_l2(a.blk_nz + b) != 0u;
#pragma unroll
    for (int q = 0; q < kPasses; ++q) {
        const int r = wid * (32 * kPasses) + q * 32 + lane;
        x[q] = any && r < n ? ld_l2(a.nbr + r0 + r) : -1;
    }
    if (!most) {
#pragma unroll
        for (int q = 0; q < kPasses; ++q) {
            const int r = wid * (32 * kPasses) + q * 32 + lane;
            if (x[q] >= 0) copy_row_regs<C>(a.hist + (r0 + r) * C, v[q], aligned);
        }
    }
    const unsigned int before = blocks_before(a, b);
#pragma unroll
    for (int q = 0; q < kPasses; ++q) kept += (unsigned)__popc(__ballot_sync(FULL, x[q] >= 0));
    if (lane == 0) { s_w[wid] = kept; s_b[wid] = before; }
    __syncthreads();
    unsigned at = 0u, T = 0u;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        if (w == wid) at = T;
        T += s_w[w];
        P += s_b[w];
    }
    if (T == 0u || P + T > a.max_rows) return;
    const int lead = (int)((P * W) & 3ull), end = lead + (int)T * W;
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int q = 0; q < kPasses; ++q) {
        const unsigned m = __ballot_sync(FULL, x[q] >= 0);
        if (x[q] >= 0) {
            v[q][C] = x[q];
            int32_t *d = buf + lead + (at + (unsigned)__popc(m & below)) * W;
            if constexpr (W % 4 == 0) {          // lead is 0
#pragma unroll
                for (int c = 0; c < W; c += 4)
                    *reinterpret_cast<int4 *>(d + c) = make_int4(v[q][c], v[q][c + 1], v[q][c + 2], v[q][c + 3]);
            } else if constexpr (W % 2 == 0) {   // lead is 0 or 2
#pragma unroll
                for (int c = 0; c < W; c += 2) *reinterpret_cast<int2 *>(d + c) = make_int2(v[q][c], v[q][c + 1]);
            } else {
#pragma unroll
                for (int c = 0; c < W; ++c) d[c] = v[q][c];
            }
        }
        at += (unsigned)__popc(m);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    int32_t *o = a.out + (P * W - (unsigned)lead);
    const int i0 = (lead + 3) & ~3, i1 = end & ~3;   // whole vectors: the copy engine's
    if (t == 0 && i1 > i0) {
        uint64_t first;
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;\n\t"
                     "cp.async.bulk.commit_group;" ::"l"(o + i0), "r"((uint32_t)__cvta_generic_to_shared(buf + i0)),
                     "r"((uint32_t)(i1 - i0) * 4u), "l"(first)
                     : "memory");
    }
    // the words before and behind them, at most three each
    if (t < 4 && lead + t < i0 && lead + t < end) o[lead + t] = buf[lead + t];
    if (t >= 4 && t < 8 && i1 + t - 4 < end && i1 >= i0) o[i1 + t - 4] = buf[i1 + t - 4];
    if (t == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the buffer goes with the CTA
}

// Write a filter's blocks: the block's kept rows from its mask words, its
// output words as vectors, each gathered from its row.  An octet of blocks a
// CTA, one per warp; or, PB, one block by the whole CTA (filter_per_block).
template <int CT, bool PB>
__device__ __forceinline__ void write_filter(const Fused &a, int64_t b0, unsigned long long P, uint16_t *sel,
                                             unsigned int *s_nz, unsigned int *s_b) {
    const int C = CT > 0 ? CT : a.C;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned int before = blocks_before(a, b0);
    if (lane == 0) s_b[w] = before;
    if (t < kOct) s_nz[t] = b0 + t < a.nblk ? ld_l2(a.blk_nz + b0 + t) : 0u;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) P += s_b[i];
    if constexpr (!PB)
        for (int i = 0; i < w; ++i) P += s_nz[i];
    const unsigned int nb = s_nz[PB ? 0 : w];
    if (nb == 0u) return;   // the block keeps nothing (or lies past the table)
    const int64_t r0 = (PB ? b0 : b0 + w) * kRowsPerBlock;
    const int64_t wi = (r0 >> 5) + lane, nwords = (a.R + 31) >> 5;
    uint32_t m = wi < nwords ? ld_l2(a.mask + wi) : 0u;   // bits past R are 0
    const unsigned int c = __popc(m);
    unsigned int pos = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int v = __shfl_up_sync(FULL, pos, o);
        if (lane >= o) pos += v;
    }
    pos -= c;
    uint16_t *ws = PB ? sel : sel + w * kRowsPerBlock;
    if (PB && lane / (32 / (kThreads / 32)) != w) m = 0u;   // each warp lists its four words' rows
    while (m) {
        ws[pos++] = (uint16_t)(lane * 32 + __ffs(m) - 1);
        m &= m - 1u;
    }
    if constexpr (PB) __syncthreads();
    else __syncwarp();
    const int32_t *hb = a.hist + r0 * C;
    const uint32_t words = nb * (uint32_t)C;
    const uint32_t lead = (uint32_t)((P * (unsigned long long)C) & 3ull);
    int32_t *gout = a.out + (P * (unsigned long long)C - lead);
    // The kept row and column of the vector's first word.  CT 0: moved on by steps (a
    // row of -1 before the lead), not found by a division, which took a warp most of its
    // time: 2.6M / 4M rows of 12 columns, nine in ten kept, 173 / 188 us a step with it,
    // 118 / 138 so (the block by a CTA 90 / 123, but 67 where nothing of the 4M is kept
    // and this takes 56)
    constexpr int kStep = 4 * (PB ? kThreads : 32);
    int q = 0, c0 = 0, dq = 0, dc = 0;
    if constexpr (CT == 0) {
        const int k = 4 * (PB ? t : lane) - (int)lead;
        q = k < 0 ? -1 : k / C;
        c0 = k - q * C;
        dq = kStep / C;
        dc = kStep % C;
    }
    for (uint32_t u = (uint32_t)(PB ? t : lane); 4u * u < lead + words; u += kStep / 4) {
        int32_t v[4];
        int row = q, col = c0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t kk = 4u * u + (uint32_t)j - lead;   // wraps above `words` before the lead
            if constexpr (CT > 0) {
                row = (int)(kk / (uint32_t)C);
                col = (int)(kk % (uint32_t)C);
            }
            v[j] = kk < words ? ld_prior(hb + (int)ws[row] * C + col) : 0;
            if constexpr (CT == 0) {
                if (++col == C) { col = 0; ++row; }
            }
        }
        if constexpr (CT == 0) {
            q += dq;
            c0 += dc;
            if (c0 >= C) { c0 -= C; ++q; }
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

// CT columns (0: any, filters only).  BPC: blocks per count CTA.  PB (filters): a
// block per write CTA, as k2u always.
template <int CT, bool FILTER, int BPC, bool PB>
__global__ void __launch_bounds__(kThreads, FILTER ? (BPC == 2 ? 5 : 6) : (CT <= 4 ? 6 : (CT <= 6 ? 5 : 4)))
fused_kernel(const __grid_constant__ Fused a, const __grid_constant__ PredView pv) {
    constexpr int NC = kOct / BPC, NW = PB ? kOct : 1;
    __shared__ __align__(16) int32_t buf[FILTER ? (PB ? 1 : kOct) * kRowsPerBlock / 2 : kRowsPerBlock * (CT + 1) + 4];
    __shared__ unsigned long long s_part[kThreads / 32];
    __shared__ unsigned int s_n[BPC][kThreads / 32], s_b[kThreads / 32];
    __shared__ WaitShared s_wait;
    asm volatile("griddepcontrol.wait;" ::: "memory");   // the previous op's table and sums are complete
    asm volatile("griddepcontrol.launch_dependents;");
    const Role role = role_of(a.first + (int)blockIdx.x, a.steps, a.lag, NC, NW);
    if (role.kind == 0) {
        // the other sums buffer, read by the previous op, is cleared for the next
        for (int64_t w = ((int64_t)role.oct * NC + role.unit) * kThreads + threadIdx.x; w < a.nclear;
             w += (int64_t)a.steps * NC * kThreads)
            a.clear[w] = 0ull;
        const int64_t b0 = (int64_t)role.oct * kOct + role.unit * BPC;
        if (b0 < a.nblk) count_blocks<CT, FILTER, BPC>(a, pv, b0, s_n, s_part);
        return;
    }
    unsigned long long P = 0ull;
    if (role.kind == 2) {
        // every group counted: the op's totals for the host
        const int64_t ng = (a.nblk + (1 << kGroupShift) - 1) >> kGroupShift;
        bool ok = groups_before(a, ng, a.pub_polls, s_wait, P);
        if (FILTER && ok) {   // and every write CTA done
            const unsigned long long want = PB ? (unsigned long long)a.nblk : (unsigned long long)a.steps;
            bool all = false;
            for (int poll = 0; poll < a.pub_polls && !all; ++poll) {
                all = ld_acquire64(a.written) == want;
                if (!all) __nanosleep(100);
            }
            ok = __syncthreads_and(all) != 0;
        }
        // the groups were read before the error word will be (groups_before): a fence of a
        // thread whose warp has no sums to load, beside the others' loads
        if (threadIdx.x == kThreads - 1) __threadfence();
        unsigned long long x = 0ull;
        for (int64_t i = threadIdx.x; ok && i < ng; i += kThreads) x += ld_l2(a.gs + 2 * i + 1);
        x = warp_add(x);
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            x = 0ull;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) x += s_part[w];
            a.pub[2] = (unsigned long long)(unsigned int)atomicOr(a.err, 0) | (ok ? 0ull : (unsigned long long)kErrWait);
            a.pub[3] = P;
            a.pub[4] = x;
            __threadfence_system();
            *(volatile unsigned long long *)a.pub = a.seq;
        }
        return;
    }
    const int64_t b = (int64_t)role.oct * kOct + role.unit;
    if (b >= a.nblk) return;   // the same in every thread
    if constexpr (FILTER) {
        if (groups_before(a, b >> kGroupShift, a.write_polls, s_wait, P)) {
            write_filter<CT, PB>(a, b, P, reinterpret_cast<uint16_t *>(buf), s_n[0], s_b);
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(a.written, 1ull);
            }
        }
    } else {
        write_k2u<CT>(a, b, s_wait, buf, s_n[0], s_b);
    }
}

bool fused_takes(int C, bool filter) { return filter || C + 1 <= kFusedCols; }

template <int CT, bool FILTER, int BPC, bool PB>
static int run_fused(Fused a, const PredView &pv, int part, cudaStream_t st) {
    constexpr int NC = kOct / BPC, NW = PB ? kOct : 1;
    // with every octet counted before the first is written, the order is the
    // counts, the publisher, the writes
    if (part != kFusedAll) a.lag = a.steps;
    const int counts = a.steps * NC + 1, all = counts + a.steps * NW;
    a.first = part == kFusedWrite ? counts : 0;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned int)((part == kFusedCount ? counts : all) - a.first));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, fused_kernel<CT, FILTER, BPC, PB>, a, pv);
}

int launch_fused(const FusedOp &op, cudaStream_t st) {
    Fused a;
    a.hist = op.hist;
    a.R = op.R;
    a.nblk = (op.R + kRowsPerBlock - 1) / kRowsPerBlock;
    a.C = op.C;
    a.scol = op.scol;
    a.ecol = op.ecol;
    a.end_const = op.end_const;
    a.dir = op.dir;
    a.nb = op.dir ? op.pv.nb[1] : op.pv.nb[0];
    a.vmin = op.dir ? op.pv.vmin[1] : op.pv.vmin[0];
    a.dn = op.dir ? op.pv.dn[1] : op.pv.dn[0];
    a.nbr = op.nbr;
    a.mask = op.mask;
    a.blk_nz = op.blk_nz;
    a.gs = op.group_sums;
    a.err = op.err;
    a.written = op.written;
    a.clear = op.clear;
    a.nclear = op.nclear;
    a.out = op.out;
    a.max_rows = op.max_rows;
    a.pub = op.pub;
    a.seq = op.seq;
    a.pub_polls = op.pub_polls;
    a.write_polls = op.write_polls;
    a.steps = (int)((a.nblk + kOct - 1) / kOct);
    // The writing trails by what the CTAs in flight reach over (6 to 8 a SM, 9 to
    // 16 an octet) and a group's 256 blocks, no more: the rows should still be in
    // L2 when they are read again.  222 octets instead of 146 made a k2u op on
    // 12M rows of 4 columns read 392 instead of 278 MB from DRAM (192 MB is the
    // table) and took it from 144 to 153 us; 184 octets (an SM's share of 1 instead
    // of 3/4) take 120.4 where these take 118.7.
    const int lag = op.sms * 3 / 4 + (1 << kGroupShift) / kOct;
    a.lag = a.steps < lag ? a.steps : lag;
    // two blocks per count CTA (eight look-ups in flight a lane) once there are
    // enough of them to fill the GPU.  A filter of 12M rows of 4 columns takes 92 us
    // with one block a CTA and 84.5 with two when nothing is kept (two kernels: 79),
    // 100 and 95 (103) at one row in eight, 156 and 156 (169) when all are; of 4M rows
    // of 8 columns 50, 58.5, 114 and 48, 55, 109
    const bool pair = a.nblk >= 16 * (int64_t)op.sms;
#define WK_FUSED(CC)                                                      \
    case CC: return pair ? run_fused<CC, false, 2, true>(a, op.pv, op.part, st) : run_fused<CC, false, 1, true>(a, op.pv, op.part, st)
    if (!op.filter) {
        switch (op.C) {
            WK_FUSED(1); WK_FUSED(2); WK_FUSED(3); WK_FUSED(4); WK_FUSED(5);
            WK_FUSED(6); WK_FUSED(7); WK_FUSED(8); WK_FUSED(9); WK_FUSED(10);
        }
        return (int)cudaErrorInvalidValue;   // not reached: fused_takes
    }
#undef WK_FUSED
    // a filter that is not written block by block has blocks enough for pairs
    const bool pb = filter_per_block(a.nblk, op.sms);
#define WK_FUSED(CC) \
    return pb ? run_fused<CC, true, 1, true>(a, op.pv, kFusedAll, st) : run_fused<CC, true, 2, false>(a, op.pv, kFusedAll, st)
    switch (op.C) {
        case 1: WK_FUSED(1);
        case 2: WK_FUSED(2);
        case 3: WK_FUSED(3);
        case 4: WK_FUSED(4);
        case 5: WK_FUSED(5);
        case 6: WK_FUSED(6);
        case 7: WK_FUSED(7);
        case 8: WK_FUSED(8);
        default: WK_FUSED(0);
    }
#undef WK_FUSED
}

}  // namespace dev
}  // namespace wk
