// Fork-join across ranks: the device-side split of a history table by the
// rank that owns each row's start vertex, and device-to-device transfers of
// tables in and out of a context (for a collective's buffers).
//
//   wk_history_partition <-> RCache::generate_sub_query (core/rcache.hpp:964-1030)
//                            with calc_dispatched_position / history_dispatch
//                            (core/gpu_hash.cu:698-790), as GPU_Engine::
//                            generate_sub_query calls it (core/gpu_engine.hpp:293-370)
//
// The owner of a row is its start column's value modulo the number of parts,
// the rule of mymath::hash_mod (utils/mymath.hpp:55-59) applied by
// d_hash_dispatched_server_id and Engine::generate_sub_requests
// (core/engine.hpp:355-358).  The reference places rows within a part by an
// atomicAdd per row, so their order there depends on scheduling; here the
// split is stable (a part keeps the rows in their input order), which gives
// every part the same multiset of rows and a fixed order besides.
//
// Steps on the op stream, a stable counting split in two passes over the
// table:
//   1. part_count: per tile of rows, the rows of each owner;
//   2. part_scan: one exclusive scan of those counts laid out owner by owner,
//      tile by tile: the global start of every (owner, tile) slot, so a part
//      keeps its tiles, and the rows within a tile, in input order; and the
//      parts' bounds, into pinned host memory;
//   3. part_move: each tile again, brought into shared memory whole; a row's
//      place in the tile's owner order is found by ranks (warps in order,
//      chunks of 32 rows in order, lanes in order), and the rows leave in that
//      order, so that consecutive threads write consecutive words of a part.
//
// What bounds it: DRAM and L2, once the stores are consecutive.  With each lane
// copying its own row to its place, a warp's store touched a sector per row;
// owners were found by a division, lanes of one owner by match_any, and the
// bounds came back through pageable memory.  6M rows of 3 columns over 8 owners
// took 148 us so, 85 now; the moves are left bound by their issue slots.
#include "wk_runtime.h"
#include "wk_loads.cuh"

#include <algorithm>

namespace wk {
int scan_u32_device(uint32_t *x, int64_t m, DevBuf &scratch, cudaStream_t st, int64_t *launches);
}

using namespace wk;

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxParts = 256;
constexpr int kTileWords = 6144;            // a staged tile: up to 24 KB
constexpr int kMaxRounds = 8;               // rows per thread of a tile
#define FULL 0xffffffffu

// n % d for 32-bit n: the quotient from a product with m = floor(2^32 / d)
// (2^32 - 1 for d = 1) is the true one or one less, so the remainder is below 2 d
struct Mod {
    uint32_t d, m;
};
__device__ __forceinline__ uint32_t mod(uint32_t n, const Mod &by) {
    const uint32_t r = n - __umulhi(n, by.m) * by.d;
    return r >= by.d ? r - by.d : r;
}

// the lanes whose owner is this lane's, of the lanes in `there`: one ballot a
// bit of the owner (bits above the owners' are 0 in every lane)
template <int BITS>
__device__ __forceinline__ unsigned same_owner(uint32_t o, unsigned there) {
    unsigned m = there;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        const bool one = (o >> b) & 1u;
        const unsigned v = __ballot_sync(FULL, one);
        m &= one ? v : ~v;
    }
    return m;
}

struct Split {
    const int32_t *hist;
    int64_t R;
    int C, col;
    Mod by;
    int rounds;              // rows per thread of a tile: kThreads x rounds rows
    int64_t ntiles;
};

// Programmatic dependent launch: the scan's block is placed while the count
// ends, and the move's blocks while the scan runs: they bring their tiles in
// and find the owners before they wait for it.  (The count starts after
// everything before it, so the table is complete by then.)
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// row i of round c of warp w within a tile (warps, rounds and lanes in input order)
__device__ __forceinline__ int tile_row(int w, int c, int lane, int rounds) { return (w * rounds + c) * 32 + lane; }

// cnt[p * ntiles + t] = rows of owner p in tile t.  FEW: up to 8 owners, counted
// by each thread in the bytes of one word (8 rows at most); else by one shared
// add per owner and round of 32 rows.  The issue slots bound it: a match_any, a
// 64-bit remainder and a shared add for every round were 86 instructions.
template <bool FEW>
__global__ void __launch_bounds__(kThreads, 8)
part_count_kernel(const Split a, uint32_t *__restrict__ cnt) {
    __shared__ uint32_t h[kMaxParts];
    allow_dependents();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t nparts = a.by.d;
    for (uint32_t p = threadIdx.x; p < nparts; p += kThreads) h[p] = 0u;
    __syncthreads();
    const int64_t t = blockIdx.x, r0 = t * kThreads * a.rounds;
    const int n = (int)(a.R - r0 < kThreads * a.rounds ? a.R - r0 : kThreads * a.rounds);
    const int32_t *key = a.hist + r0 * a.C + a.col;
    uint32_t v[kMaxRounds];   // every load in flight before the first is used
#pragma unroll
    for (int c = 0; c < kMaxRounds; ++c) {
        const int r = tile_row(w, c, lane, a.rounds);
        v[c] = c < a.rounds && r < n ? (uint32_t)__ldg(key + (int64_t)r * a.C) : 0u;
    }
    if constexpr (FEW) {
        unsigned long long bytes = 0ull;
#pragma unroll
        for (int c = 0; c < kMaxRounds; ++c)
            if (c < a.rounds && tile_row(w, c, lane, a.rounds) < n) bytes += 1ull << (8u * mod(v[c], a.by));
        // bytes 0 and 2, 1 and 3, ... as 16-bit halves: the warp's sums are at most 256
        const uint32_t lo = (uint32_t)bytes, hi = (uint32_t)(bytes >> 32);
        const uint32_t s[4] = {__reduce_add_sync(FULL, lo & 0xff00ffu), __reduce_add_sync(FULL, (lo >> 8) & 0xff00ffu),
                               __reduce_add_sync(FULL, hi & 0xff00ffu), __reduce_add_sync(FULL, (hi >> 8) & 0xff00ffu)};
        if (lane < (int)nparts) {
            const uint32_t x = lane < 4 ? (lane & 1 ? s[1] : s[0]) : (lane & 1 ? s[3] : s[2]);
            const uint32_t k = (x >> (lane & 2 ? 16 : 0)) & 0xffffu;
            if (k) atomicAdd(&h[lane], k);
        }
    } else {
#pragma unroll
        for (int c = 0; c < kMaxRounds; ++c) {
            if (c >= a.rounds) break;
            const unsigned there = __ballot_sync(FULL, tile_row(w, c, lane, a.rounds) < n);
            const uint32_t o = mod(v[c], a.by);
            const unsigned m = same_owner<8>(o, there);
            if (lane == __ffs(m) - 1) atomicAdd(&h[o], (uint32_t)__popc(m));   // not a lane past the table: m has none
        }
    }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < nparts; p += kThreads) cnt[(int64_t)p * a.ntiles + t] = h[p];
}

// One block: exclusive scan of the m = nparts x ntiles counts in place, and
// bound[p] = the first row of part p, bound[nparts] = R.
constexpr int kScanThreads = 1024, kScanPer = 8;   // uint4 per thread and pass: 32768 counts
constexpr int64_t kScanMost = 4 * 4 * kScanPer * kScanThreads;
__global__ void __launch_bounds__(kScanThreads)
part_scan_kernel(uint32_t *__restrict__ cnt, int64_t m, int64_t ntiles, int64_t R, uint32_t nparts,
                 unsigned long long *__restrict__ bound) {
    __shared__ uint32_t sw[32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    allow_dependents();
    wait_prior();
    uint32_t carry = 0u;
    for (int64_t i0 = 0; i0 < m; i0 += 4 * kScanPer * kScanThreads) {
        uint4 v[kScanPer];
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int64_t i = i0 + 4 * ((int64_t)k * kScanThreads + t);   // the buffer ends on a multiple of 4
            v[k] = i < m ? *reinterpret_cast<const uint4 *>(cnt + i) : make_uint4(0u, 0u, 0u, 0u);
            if (i + 1 >= m) v[k].y = 0u;
            if (i + 2 >= m) v[k].z = 0u;
            if (i + 3 >= m) v[k].w = 0u;
        }
#pragma unroll
        for (int k = 0; k < kScanPer; ++k) {
            const int64_t i = i0 + 4 * ((int64_t)k * kScanThreads + t);
            if (i0 + 4 * (int64_t)k * kScanThreads >= m) break;   // the same in every thread
            const uint32_t s = v[k].x + v[k].y + v[k].z + v[k].w;
            uint32_t in = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(FULL, in, o);
                if (lane >= o) in += x;
            }
            if (lane == 31) sw[wid] = in;
            __syncthreads();
            uint32_t x = sw[lane];   // 32 warps
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            const uint32_t all = __shfl_sync(FULL, x, 31), before = __shfl_sync(FULL, x, wid > 0 ? wid - 1 : 0);
            const uint32_t e = carry + in - s + (wid > 0 ? before : 0u);
            if (i < m)
                *reinterpret_cast<uint4 *>(cnt + i) =
                    make_uint4(e, e + v[k].x, e + v[k].x + v[k].y, e + v[k].x + v[k].y + v[k].z);
            carry += all;
            __syncthreads();   // sw is written again
        }
    }
    __syncthreads();
    for (uint32_t p = t; p <= nparts; p += kScanThreads)
        bound[p] = p < nparts ? (unsigned long long)cnt[(int64_t)p * ntiles] : (unsigned long long)R;
}

// the bounds alone, after a scan by scan_u32_device
__global__ void part_bounds_kernel(const uint32_t *__restrict__ start, int64_t ntiles, int64_t R, uint32_t nparts,
                                   unsigned long long *__restrict__ bound) {
    for (uint32_t p = threadIdx.x; p <= nparts; p += blockDim.x)
        bound[p] = p < nparts ? (unsigned long long)start[(int64_t)p * ntiles] : (unsigned long long)R;
}

// The rows of tile t to their places: start[p * ntiles + t] is where owner p's
// rows of the tile begin.  V: the vector a row is moved in (the widest that its
// bytes and both tables' alignment allow), PER of them a row (0: any); STAGED:
// the tile goes through shared memory (up to kTileWords words), else each lane
// copies its row.  BITS: of the largest owner, or more.
template <typename V, int PER, int BITS, bool STAGED>
__global__ void __launch_bounds__(kThreads, 6)
part_move_kernel(const Split a, const uint32_t *start, int32_t *__restrict__ out) {
    __shared__ uint32_t wc[kWarps][kMaxParts];   // per warp: its rows per owner, then its next place per owner
    __shared__ uint32_t s_at[kMaxParts];         // STAGED: an owner's start in `out` minus its place in the tile
    __shared__ uint32_t s_w[kWarps];
    extern __shared__ __align__(16) unsigned char smem[];   // STAGED: the tile, then per place its row and its output row
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t nparts = a.by.d;
    const int rows = kThreads * a.rounds;
    const int64_t t = blockIdx.x, r0 = t * rows;
    const int n = (int)((a.R - r0) < rows ? (a.R - r0) : rows);
    const int per = PER > 0 ? PER : a.C / (int)(sizeof(V) / 4);   // vectors a row
    V *tile = reinterpret_cast<V *>(smem);
    uint32_t *s_out = reinterpret_cast<uint32_t *>(tile + (STAGED ? rows * per : 0));
    uint16_t *s_src = reinterpret_cast<uint16_t *>(s_out + (STAGED ? rows : 0));
    for (uint32_t p = threadIdx.x; p < nparts; p += kThreads)
#pragma unroll
        for (int x = 0; x < kWarps; ++x) wc[x][p] = 0u;
    const V *src = reinterpret_cast<const V *>(a.hist + r0 * a.C);
    if constexpr (STAGED) {
        // every copy in flight at once: 16 B each, but for what is left of the
        // last tile, or all of a table that is not 16 B aligned
        const int32_t *g = a.hist + r0 * a.C;
        const int words = n * a.C, whole = ((uintptr_t)a.hist & 15u) == 0 ? words & ~3 : 0;
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
        for (int i = 4 * threadIdx.x; i < whole; i += 4 * kThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + 4u * i), "l"(g + i) : "memory");
        for (int i = whole + threadIdx.x; i < words; i += kThreads)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(base + 4u * i), "l"(g + i) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    const int32_t *key = STAGED ? reinterpret_cast<const int32_t *>(tile) : a.hist + r0 * a.C;
    uint32_t own[kMaxRounds];
    unsigned same[kMaxRounds];
#pragma unroll
    for (int c = 0; c < kMaxRounds; ++c) {
        const int r = tile_row(w, c, lane, a.rounds);
        own[c] = c < a.rounds && r < n ? (uint32_t)key[(STAGED ? r * a.C : (int64_t)r * a.C) + a.col] : 0u;
    }
#pragma unroll
    for (int c = 0; c < kMaxRounds; ++c) {
        same[c] = 0u;
        if (c >= a.rounds) break;
        const unsigned there = __ballot_sync(FULL, tile_row(w, c, lane, a.rounds) < n);
        own[c] = mod(own[c], a.by);
        const unsigned m = same_owner<BITS>(own[c], there);   // by every lane
        same[c] = (there >> lane) & 1u ? m : 0u;
        if (same[c] && lane == __ffs(same[c]) - 1) wc[w][own[c]] += (uint32_t)__popc(same[c]);   // this warp's row of wc only
        __syncwarp();
    }
    __syncthreads();
    // per owner: its place (STAGED: in the tile, else in `out`), then the warps in order
    wait_prior();
    uint32_t total = 0u, first = 0u;
    const uint32_t p = threadIdx.x;   // kThreads == kMaxParts
    if (p < nparts) {
        first = dev::ld_prior(start + (int64_t)p * a.ntiles + t);
#pragma unroll
        for (int x = 0; x < kWarps; ++x) total += wc[x][p];
    }
    uint32_t acc = first;
    if constexpr (STAGED) {
        uint32_t in = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(FULL, in, o);
            if (lane >= o) in += x;
        }
        if (lane == 31) s_w[w] = in;
        __syncthreads();
        acc = in - total;
#pragma unroll
        for (int x = 0; x < kWarps; ++x)
            if (x < w) acc += s_w[x];
        if (p < nparts) s_at[p] = first - acc;   // modulo 2^32
    }
    if (p < nparts) {
#pragma unroll
        for (int x = 0; x < kWarps; ++x) {
            const uint32_t k = wc[x][p];
            wc[x][p] = acc;
            acc += k;
        }
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int c = 0; c < kMaxRounds; ++c) {
        if (c >= a.rounds) break;
        const int r = tile_row(w, c, lane, a.rounds);
        if (same[c]) {
            const uint32_t at = wc[w][own[c]] + (uint32_t)__popc(same[c] & below);
            if constexpr (STAGED) {
                s_src[at] = (uint16_t)r;
                s_out[at] = s_at[own[c]] + at;
            } else {
                V *dst = reinterpret_cast<V *>(out + (int64_t)at * a.C);
                for (int k = 0; k < per; ++k) dst[k] = __ldg(src + (int64_t)r * per + k);
            }
        }
        __syncwarp();
        if (same[c] && lane == __ffs(same[c]) - 1) wc[w][own[c]] += (uint32_t)__popc(same[c]);
        __syncwarp();
    }
    if constexpr (STAGED) {
        __syncthreads();
        // vectors in owner order.  A warp takes 32 rows at a time, lane l their
        // vectors l, l + 32, ..., whose row and place in it are the same for
        // every 32 rows
        V *dst = reinterpret_cast<V *>(out);
        if constexpr (PER > 0) {
            int row[PER], col[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                row[k] = (lane + 32 * k) / PER;
                col[k] = (lane + 32 * k) % PER;
            }
            for (int i0 = w * 32; i0 < n; i0 += kThreads) {
#pragma unroll
                for (int k = 0; k < PER; ++k) {
                    const int i = i0 + row[k];
                    if (i < n) dst[(int64_t)s_out[i] * PER + col[k]] = tile[(int)s_src[i] * PER + col[k]];
                }
            }
        } else {
            const int dr = kThreads / per, dc = kThreads % per;
            int i = threadIdx.x / per, c = threadIdx.x % per;
            while (i < n) {
                dst[(int64_t)s_out[i] * per + c] = tile[(int)s_src[i] * per + c];
                i += dr;
                c += dc;
                if (c >= per) { c -= per; ++i; }
            }
        }
    }
}

}  // namespace

extern "C" int wk_history_partition(wk_ctx *ctx, const wk_history *in, int64_t start, int32_t nparts,
                                    int64_t *part_rows, wk_history *out) {
    if (!ctx || !in || !out || !part_rows) return set_error(WK_EINVAL, "wk_history_partition: null argument");
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_history_partition: host-only context");
    if (nparts < 1 || nparts > kMaxParts)
        return set_error(WK_EINVAL, "wk_history_partition: %d parts (1..%d)", nparts, kMaxParts);
    const int C = in->col_num;
    if (start >= 0 || C <= 0 || -start - 1 >= C)
        return set_error(WK_EINVAL, "wk_history_partition: start %lld is not a bound variable of a %d-column table",
                         (long long)start, C);
    if (in->size < 0 || in->size % C != 0 || (in->size > 0 && !in->data))
        return set_error(WK_EINVAL, "wk_history_partition: bad table (size %lld, %d columns)", (long long)in->size, C);
    const int64_t R = in->size / C;
    if (R >= (int64_t)UINT32_MAX) return set_error(WK_EINVAL, "wk_history_partition: %lld rows (< 2^32 - 1)", (long long)R);
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    const int32_t *src = in->data;
    const int32_t step = in->step;
    DevBuf &ob = (src == static_cast<const int32_t *>(ctx->hbuf[0].ptr)) ? ctx->hbuf[1] : ctx->hbuf[0];
    int st = ob.reserve((size_t)in->size * 4 + 16);
    if (st) return st;
    cudaStream_t s = ctx->stream;
    DevBuf &cb = ctx->part_cnt, &sb = ctx->part_scan;
    if ((st = wk::reserve_published(ctx, kMaxParts + 1))) return st;
    const unsigned long long *bound = ctx->h_gs + 2;
    if (R > 0) {
        Split a;
        a.hist = src;
        a.R = R;
        a.C = C;
        a.col = (int)(-start - 1);
        a.by.d = (uint32_t)nparts;
        a.by.m = nparts == 1 ? 0xffffffffu : (uint32_t)((1ull << 32) / (unsigned)nparts);
        // a tile of up to 2048 rows: as many as fit 24 KB; rows of more than
        // kTileWords / kThreads columns are copied lane by lane
        const bool staged = C <= kTileWords / kThreads;
        a.rounds = staged ? std::min(kMaxRounds, kTileWords / (C * kThreads)) : kMaxRounds;
        const int rows = kThreads * a.rounds;
        a.ntiles = (R + rows - 1) / rows;
        const int64_t m = a.ntiles * nparts;
        if ((st = cb.reserve(((size_t)m * 4 + 15) & ~(size_t)15))) return st;
        uint32_t *cnt = cb.as<uint32_t>();
        const bool few = nparts <= 8;
        if (few) part_count_kernel<true><<<(unsigned)a.ntiles, kThreads, 0, s>>>(a, cnt);
        else part_count_kernel<false><<<(unsigned)a.ntiles, kThreads, 0, s>>>(a, cnt);
        ++ctx->launches;
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "partition count");
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        // one block scans up to 131072 counts (three launches cost more than its
        // passes up to there)
        if (m <= kScanMost) {
            cfg.gridDim = dim3(1);
            cfg.blockDim = dim3(kScanThreads);
            cudaLaunchKernelEx(&cfg, part_scan_kernel, cnt, m, a.ntiles, R, (uint32_t)nparts, ctx->h_gs_dev + 2);
        } else {
            if ((st = scan_u32_device(cnt, m, sb, s, &ctx->launches))) return st;
            part_bounds_kernel<<<1, kThreads, 0, s>>>(cnt, a.ntiles, R, (uint32_t)nparts, ctx->h_gs_dev + 2);
        }
        // vectors need their alignment in both tables (the history buffers are
        // 256 B aligned; a caller's table may not be)
        const uintptr_t al = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(ob.ptr);
        const size_t shared = staged ? (size_t)rows * ((size_t)C * 4 + 4 + 2) : 0;
        int32_t *dst = ob.as<int32_t>();
        cfg.gridDim = dim3((unsigned)a.ntiles);
        cfg.blockDim = dim3(kThreads);
#define WK_MOVE(V, PER, ST, SMEM)                                                                                    \
    do {                                                                                                             \
        cfg.dynamicSmemBytes = SMEM;                                                                                 \
        if (few) cudaLaunchKernelEx(&cfg, part_move_kernel<V, PER, 3, ST>, a, (const uint32_t *)cnt, dst);           \
        else cudaLaunchKernelEx(&cfg, part_move_kernel<V, PER, 8, ST>, a, (const uint32_t *)cnt, dst);               \
    } while (0)
        // the odd widths up to 3 and their doubles and quadruples know their
        // vectors at compile time
        if (C % 4 == 0 && !(al & 15u)) {
            if (!staged) WK_MOVE(int4, 0, false, 0);
            else if (C == 4) WK_MOVE(int4, 1, true, shared);
            else if (C == 8) WK_MOVE(int4, 2, true, shared);
            else WK_MOVE(int4, 0, true, shared);
        } else if (C % 2 == 0 && !(al & 7u)) {
            if (!staged) WK_MOVE(int2, 0, false, 0);
            else if (C == 2) WK_MOVE(int2, 1, true, shared);
            else if (C == 6) WK_MOVE(int2, 3, true, shared);
            else WK_MOVE(int2, 0, true, shared);
        } else {
            if (!staged) WK_MOVE(int, 0, false, 0);
            else if (C == 1) WK_MOVE(int, 1, true, shared);
            else if (C == 3) WK_MOVE(int, 3, true, shared);
            else WK_MOVE(int, 0, true, shared);
        }
#undef WK_MOVE
        ctx->launches += 2;
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "partition move");
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(e, "partition sync");
    }
    for (int p = 0; p < nparts; ++p) part_rows[p] = R > 0 ? (int64_t)(bound[p + 1] - bound[p]) : 0;
    out->data = ob.as<int32_t>();
    out->size = in->size;
    out->col_num = C;
    out->step = step;
    return WK_OK;
}

extern "C" int wk_history_to_device(wk_ctx *ctx, const wk_history *h, int32_t *dst, int64_t cap) {
    if (!ctx || !h || (h->size > 0 && (!dst || cap < h->size)))
        return set_error(WK_EINVAL, "wk_history_to_device: bad arguments (cap %lld < size %lld)", (long long)cap,
                         h ? (long long)h->size : 0ll);
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_history_to_device: host-only context");
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    if (h->size > 0 &&
        (e = cudaMemcpyAsync(dst, h->data, (size_t)h->size * 4, cudaMemcpyDeviceToDevice, ctx->stream)) != cudaSuccess)
        return cuda_fail(e, "wk_history_to_device");
    if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_fail(e, "wk_history_to_device sync");
    return WK_OK;
}

extern "C" int wk_history_from_device(wk_ctx *ctx, wk_history *h, const int32_t *src, int64_t size, int32_t col_num) {
    if (!ctx || !h || size < 0 || (size > 0 && !src) || col_num < 0 || (col_num == 0 && size != 0) ||
        (col_num > 0 && size % col_num != 0))
        return set_error(WK_EINVAL, "wk_history_from_device: bad arguments");
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_history_from_device: host-only context");
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    DevBuf &b = ctx->hbuf[0];
    int st = b.reserve((size_t)size * 4 + 16);
    if (st) return st;
    if (size > 0 && (e = cudaMemcpyAsync(b.ptr, src, (size_t)size * 4, cudaMemcpyDeviceToDevice, ctx->stream)) != cudaSuccess)
        return cuda_fail(e, "wk_history_from_device");
    if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_fail(e, "wk_history_from_device sync");
    h->data = static_cast<int32_t *>(b.ptr);
    h->size = size;
    h->col_num = col_num;
    return WK_OK;
}
