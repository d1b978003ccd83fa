// A light query in one launch: one CTA takes the request's start list through
// every step while the tables stay small (sm_103a).
//
// What bounds a light request is latency: each step is a few dependent reads
// (row, look-up, list entry) on a few hundred rows, 2 us of work, while as
// steps of their own each costs a launch, its start on the device and a host
// round trip for its totals, 5 to 12 us.  Here a step costs its reads and two
// or three barriers, and the host waits once.  A request of four patterns on
// 100 rows, its table brought to the host, takes 36 us this way, 57 by the steps'
// kernels.
//
// One CTA of 1024 threads, kLightRows rows at most: the prefix of a step's rows
// stays in shared memory, and a step's cost grows with its rows, from 2 us at 64 to
// 7 at 2048, where the steps' kernels take 11 whatever the rows are.  Lists of 64 /
// 1024 / 2048 rows and 1 step 17.9 / 17.8 / 19.1 us (steps' kernels 20 / 19.5 /
// 19.6), 3 steps 21.5 / 23 / 27 (42), 8 steps 32 / 46 / 67 (99).  A step whose output
// is larger (or passes the row limit) is not started: the host goes on from there
// with the steps' own kernels.
#include "wk_kernels.h"
#include "wk_probe.cuh"

namespace wk {
namespace dev {

#define FULL 0xffffffffu

constexpr int kLightThreads = 1024, kLightWarps = kLightThreads / 32;
constexpr int kLightRounds = kLightRows / kLightThreads;
// a list longer than this is never written here; clamped, 2048 of them add up in 32 bits
constexpr uint32_t kDegreeCap = 1u << 16;

// the first entry of e[0 .. n) not below v (e ascending): *scanned as a linear scan to it
__device__ __forceinline__ bool light_contains(const int32_t *e, uint32_t n, int32_t v, uint32_t *scanned) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(e + mid) < v) lo = mid + 1;
        else hi = mid;
    }
    const bool f = lo < n && __ldg(e + lo) == v;
    *scanned = f ? lo + 1 : n;
    return f;
}

__global__ void __launch_bounds__(kLightThreads, 1) light_kernel(const __grid_constant__ LightOp a) {
    __shared__ uint32_t s_pos[kLightRows + 1];
    __shared__ unsigned long long s_list[kLightRows];   // the list's offset, or bit 63 and the one neighbour
    __shared__ uint32_t s_w[2][kLightRounds][kLightWarps];   // two sets, so that a step needs no barrier to reuse one
    __shared__ unsigned long long s_scan;
    __shared__ int s_err;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    for (int i = t; i < a.deg; i += kLightThreads) a.buf[0][i] = __ldg(a.src + i);
    if (t == 0) s_err = 0;
    int R = a.deg, cur = 0, done = 0;
    for (; done < a.n; ++done) {
        const LightStep &st = a.s[done];
        const int32_t *T = a.buf[cur];
        int32_t *O = a.buf[cur ^ 1];
        const int C = st.C;
        const bool k2u = st.kind == kLightK2U;
        const int32_t *nb = st.dir ? st.pv.nb[1] : st.pv.nb[0];
        const uint32_t vmin = st.dir ? st.pv.vmin[1] : st.pv.vmin[0], dn = st.dir ? st.pv.dn[1] : st.pv.dn[0];
        if (t == 0) s_scan = 0ull;
        __syncthreads();   // the table is complete, shared memory free
        uint32_t d[kLightRounds], pos[kLightRounds];
        unsigned long long l[kLightRounds], scanned = 0ull;
#pragma unroll
        for (int q = 0; q < kLightRounds; ++q) {
            const int r = q * kLightThreads + t;
            d[q] = 0u;
            l[q] = 0ull;
            if (r < R) {
                const int32_t v = T[r * C + st.scol];
                const uint32_t x = (uint32_t)v - vmin;   // wraps above dn below vmin
                if (nb != nullptr && v > 0) {
                    const int32_t g = x < dn ? __ldg(nb + x) : -1;
                    d[q] = g >= 0 ? 1u : 0u;
                    l[q] = 1ull << 63 | (uint32_t)g;
                } else if (v >= 0) {
                    uint32_t o;
                    d[q] = probe_view(st.pv, (uint32_t)v, st.dir, &o, &s_err);
                    l[q] = o;
                }
                if (!k2u && d[q] > 0u) {
                    const int32_t tg = st.ecol >= 0 ? T[r * C + st.ecol] : st.end_const;
                    uint32_t sc = 1u;
                    const bool keep = l[q] >> 63 ? (int32_t)l[q] == tg : light_contains(st.pv.edges + l[q], d[q], tg, &sc);
                    d[q] = keep ? 1u : 0u;
                    scanned += sc;
                }
                if (d[q] > kDegreeCap) d[q] = kDegreeCap;
            }
        }
        // each row's first output row: rows are in order of (round, thread)
#pragma unroll
        for (int q = 0; q < kLightRounds; ++q) {
            uint32_t x = d[q];
#pragma unroll
            for (int sh = 1; sh < 32; sh <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, sh);
                if (lane >= sh) x += y;
            }
            pos[q] = x - d[q];
            if (lane == 31) s_w[done & 1][q][wid] = x;
        }
        if (scanned) atomicAdd(&s_scan, scanned);
        __syncthreads();
        uint32_t total = 0u;
#pragma unroll
        for (int q = 0; q < kLightRounds; ++q) {
            const uint32_t w = s_w[done & 1][q][lane];
            pos[q] += total + __reduce_add_sync(FULL, lane < wid ? w : 0u);
            total += __reduce_add_sync(FULL, w);
        }
        if (s_err != 0 || total > (uint32_t)kLightRows || (k2u && (long long)total > a.row_limit)) break;   // in every thread
        if (k2u) {
#pragma unroll
            for (int q = 0; q < kLightRounds; ++q) {
                const int r = q * kLightThreads + t;
                s_pos[r] = r < R ? pos[q] : total;
                s_list[r] = l[q];
            }
            __syncthreads();
            for (uint32_t j = t; j < total; j += kLightThreads) {
                int lo = 0, hi = R - 1;   // the last row whose output begins at or before j
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_pos[mid] <= j) lo = mid;
                    else hi = mid - 1;
                }
                const unsigned long long e = s_list[lo];
                const int32_t g = e >> 63 ? (int32_t)e : __ldg(st.pv.edges + (e + (j - s_pos[lo])));
                const int32_t *src = T + lo * C;
                int32_t *dst = O + (int)j * (C + 1);
                for (int c = 0; c < C; ++c) dst[c] = src[c];
                dst[C] = g;
            }
        } else {
#pragma unroll
            for (int q = 0; q < kLightRounds; ++q) {
                if (d[q] == 0u) continue;
                const int32_t *src = T + (q * kLightThreads + t) * C;
                int32_t *dst = O + (int)pos[q] * C;
                for (int c = 0; c < C; ++c) dst[c] = src[c];
            }
        }
        R = (int)total;
        cur ^= 1;
        if (t == 0) {
            a.pub[kLightWords + done] = (unsigned long long)R;
            a.pub[4] = s_scan;
        }
    }
    __syncthreads();
    if (t == 0) {
        a.pub[2] = (unsigned long long)(unsigned int)s_err;
        a.pub[3] = (unsigned long long)done;
        __threadfence_system();
        *(volatile unsigned long long *)a.pub = a.seq;
    }
}

void launch_light(const LightOp &op, cudaStream_t st) { light_kernel<<<1, kLightThreads, 0, st>>>(op); }

}  // namespace dev
}  // namespace wk
