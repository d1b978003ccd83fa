// The estimator's GEMM on the 5th-generation tensor cores (sm_100 family):
// C[M x N] fp32 = A[M x K] . B[N x K]^T (+ bias[n]), A and B bf16 row-major
// (K contiguous), FP32 accumulation in tensor memory (TMEM).
//
// One CTA of 4 warps computes a 128 x BN tile (BN = 32, 64, 128 or 256: one
// MMA shape); the grid is M tiles x N / BN.  K is walked in slabs of 64 bf16 -- one
// 128-byte row of the 128 B swizzle -- through kStages shared-memory stages:
//   - thread 0 (the producer) loads each slab's A box (64 x 128) and B box
//     (64 x BN) with TMA (cp.async.bulk.tensor.2d, 128 B swizzle; rows past M
//     and columns past K read as zero), completing on the stage's "full"
//     mbarrier, once the stage's "empty" mbarrier says its last products ran;
//   - thread 32 (the MMA issuer) waits for "full", issues the slab's
//     tcgen05.mma (kind::f16, 128 x BN x 16 each) from shared-memory
//     descriptors and commits them to the stage's "empty" mbarrier;
//   - after the last commit, warp w reads TMEM lanes 32w..32w+31 (rows) in
//     32-column chunks with tcgen05.ld and runs the epilogue the template
//     names (EpiArgs):
//       kEpiGeluFwd: C = Z = acc + bias (the pre-activation), staged in shared
//                    memory (the pipeline stages are free by then) and written
//                    as whole rows of float4, so a store instruction covers 4
//                    rows x 128 B, and H = GELU(Z) in bf16, row-major and
//                    transposed (zero for rows >= m_real);
//       kEpiGeluBwd: dZ = acc * GELU'(Z) in bf16, row-major and transposed
//                    (zero for rows >= m_real), and the column sums of the
//                    rounded dZ added into colsum[] -- C is not written;
//       kEpiHead:    the end of the forward pass and the start of the backward
//                    one, 16 rows a CTA (head_rows);
//       kEpiGroup:   C = acc for columns below n_real, or the tile's 32 columns added to
//                    the rows' embedding gradients (demb).
// The products of a training step are small and follow one another, so their
// kernels are launched ahead of their turn (programmatic dependent launch): a
// CTA sets up its barriers and TMEM and reads its tensor maps, then waits for
// the kernel before.  It lets the next one start only once it holds its TMEM,
// so no CTA waits for columns that one behind it has taken.
// Every mbarrier wait is bounded.  A wait that runs out sets bit 2 of *err and
// stops the pipeline: the producer waits (bounded) for the copies it issued
// and the issuer for the last commit of the products it issued.  If those
// drain waits also run out, work may still be in flight, so the CTA sets bit
// 3 as well and exits without freeing its TMEM columns -- a unit still
// writing them must not find them given to another CTA.  The host then
// refuses every later call on the estimator (the TMEM and the device state
// are no longer trusted); nothing is reused.
#pragma once

#include <cstdint>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "wk_loads.cuh"

namespace wk {
namespace tc {

constexpr int kTM = 128;            // tile rows = MMA M
constexpr int kSlab = 64;           // K elements per stage (128 B rows)
constexpr int kStages = 4;          // kDeepStages where K is the batch and the tiles are few
constexpr int kDeepStages = 8;
constexpr int kThreads = 128;
constexpr int kEpiPitch = 36;       // floats per staged output row: rows 16 B apart modulo 128 B
constexpr long kWaitIters = 1l << 22;

enum { kEpiGeluFwd, kEpiGeluBwd, kEpiHead, kEpiGroup };

// The epilogue's extra operands.  Rows below m_store get
// h / ht written (row-major with ld ldh, transposed with ld ldt); rows below
// m_real carry values, the rest zeros.
struct EpiArgs {
    int m_real = 0, m_store = 0;
    __nv_bfloat16 *h = nullptr;
    int ldh = 0;
    __nv_bfloat16 *ht = nullptr;
    int ldt = 0;
    const float *z = nullptr;   // kEpiGeluBwd: the layer's pre-activation (ld ldz)
    int ldz = 0;
    float *colsum = nullptr;    // kEpiGeluBwd, kEpiHead: column sums of dZ are added here
    int n_real = 1 << 30;       // kEpiGroup: columns of C
    // kEpiGroup, demb not null: column c of row r is added to demb[32 pids[r] + c]
    float *demb = nullptr;
    const int32_t *pids = nullptr;
    int n_ids = 0;
    // kEpiHead: the output layer's weights and bias, the targets; dY in bf16; each
    // CTA's sums of (y - t)^2 and dY
    const __nv_bfloat16 *w = nullptr;
    const float *b = nullptr, *tgt = nullptr;
    __nv_bfloat16 *dy = nullptr;
    float2 *part = nullptr;
};

// The estimator's activation, exact GELU: x Phi(x), and its derivative
// Phi(x) + x phi(x) (Phi, phi the standard normal CDF and density).
__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, 128 B swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);   // start address / 16
    d |= (uint64_t)1 << 16;                   // leading byte offset (not used by swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset: the next group of 8 rows
    d |= (uint64_t)1 << 46;                   // descriptor version
    d |= (uint64_t)2 << 61;                   // 128 B swizzle
    return d;
}

// instruction descriptor of kind::f16: BF16 A and B, FP32 D, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    uint32_t done = 0;
    for (long it = 0; it < kWaitIters && !done; ++it)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    return done != 0;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(mbar) : "memory");
}

// 32 consecutive fp32 columns of the warp's 32 TMEM lanes: lane i gets row i
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The step's output layer, loss and first backward layer for the CTA's 16 rows,
// a warp four of them: y = acc + b, loss mean((y - t)^2), dY = 2 (y - t) / M in
// bf16 (rows >= m_real: zero), and of the hidden layer below dZ = dY w GELU'(Z) in
// bf16, row-major and transposed, with its column sums.  The layer has one output,
// so these are row-wise: as products padded to tiles of 64 with kernels of their
// own for bias, loss and sums they were seven launches and 30 us of a step of 1024
// rows; this takes 9, with cold caches 11.5.  (The weights' gradient dY^T H is a product of
// gemm_group_kernel: added up here by atomics it took whichever order the CTAs
// came in.)  y: the CTA's 16 accumulators.  sm: 14 KB, free.
__device__ __forceinline__ void head_rows(const EpiArgs &ea, const float *y, int row0, unsigned char *sm) {
    constexpr int kCols = 256, kPitch = 18;   // an odd number of words: the 32 lanes' columns fall in 32 banks
    __nv_bfloat16 *st = reinterpret_cast<__nv_bfloat16 *>(sm);                    // dZ^T: [256][16]
    float *s_cs = reinterpret_cast<float *>(sm + kCols * kPitch * 2);             // per warp: column sums of dZ
    __shared__ float2 s_sum[kThreads / 32];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // every row's words in flight at once
    constexpr int kRows = 16 / (kThreads / 32);
    float w[8], z[kRows][8], cs[8] = {}, tg[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int row = row0 + warp * kRows + i;
#pragma unroll
        for (int j = 0; j < 8; ++j) z[i][j] = ea.z[(size_t)row * ea.ldz + lane + 32 * j];
        tg[i] = row < ea.m_real ? ea.tgt[row] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = __bfloat162float(ea.w[lane + 32 * j]);
    const float b = *ea.b;
    float sq = 0.f, sdy = 0.f;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int r = warp * kRows + i, row = row0 + r;
        float dy = 0.f;
        if (row < ea.m_real) {   // the same in every lane
            const float d = (y[r] + b) - tg[i];
            sq += d * d;
            dy = __bfloat162float(__float2bfloat16(2.f * d / (float)ea.m_real));
            sdy += dy;
        }
        if (lane == 0) ea.dy[row] = __float2bfloat16(dy);   // its own bf16 value
        __nv_bfloat16 *out = ea.h + (size_t)row * ea.ldh + lane;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const __nv_bfloat16 v = __float2bfloat16(row < ea.m_real ? __fmul_rn(dy, w[j]) * gelu_grad(z[i][j]) : 0.f);
            out[32 * j] = v;
            st[(lane + 32 * j) * kPitch + r] = v;
            cs[j] += __bfloat162float(v);
        }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s_cs[warp * kCols + lane + 32 * j] = cs[j];
    if (lane == 0) s_sum[warp] = make_float2(sq, sdy);
    __syncthreads();
    for (int c = t; c < kCols; c += kThreads) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(st + c * kPitch);
        uint4 *dst = reinterpret_cast<uint4 *>(ea.ht + (size_t)c * ea.ldt + row0);
        dst[0] = make_uint4(src[0], src[1], src[2], src[3]);
        dst[1] = make_uint4(src[4], src[5], src[6], src[7]);
        float a = s_cs[c];
        for (int i = 1; i < kThreads / 32; ++i) a += s_cs[i * kCols + c];
        if (a != 0.f) atomicAdd(ea.colsum + c, a);
    }
    if (t == 0) {   // added up over the CTAs by sum_rows, in a later kernel: nothing waits for it
        float2 v = s_sum[0];
        for (int i = 1; i < kThreads / 32; ++i) { v.x += s_sum[i].x; v.y += s_sum[i].y; }
        ea.part[blockIdx.x] = v;
    }
}

// The loss (the mean over m rows, also added into loss[1]) and the output
// bias's gradient from the n CTAs' sums.  One CTA.
__device__ __forceinline__ void sum_rows(const float2 *part, int n, int m, float *loss, float *db) {
    __shared__ float2 s_sum[kThreads / 32];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    float sq = 0.f, sdy = 0.f;
    for (int i = t; i < n; i += kThreads) {
        const float2 v = dev::ld_prior(part + i);
        sq += v.x;
        sdy += v.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        sdy += __shfl_xor_sync(0xffffffffu, sdy, o);
    }
    if (lane == 0) s_sum[warp] = make_float2(sq, sdy);
    __syncthreads();
    if (t == 0) {
        float2 v = s_sum[0];
        for (int i = 1; i < kThreads / 32; ++i) { v.x += s_sum[i].x; v.y += s_sum[i].y; }
        const float l = v.x / (float)(m > 0 ? m : 1);
        loss[0] = l;
        loss[1] += l;
        *db = v.y;
    }
}

// One tile: rows m0.. and columns n0.. of C.  C must be 16 B aligned with ldc a
// multiple of 4, and bias (if any) 16 B aligned; h (and z) 16 B aligned with
// ldh (ldz) a multiple of 8 (4).
template <int BN, int EPI, int STAGES>
__device__ __forceinline__ void gemm_tile(const CUtensorMap *tmA, const CUtensorMap *tmB, int m0, int n0,
                                          float *__restrict__ C, int ldc, int M, int K,
                                          const float *__restrict__ bias, int *err, const EpiArgs &ea) {
    static_assert(BN == 32 || BN == 64 || BN == 128 || BN == 256, "tile width: an MMA N and a TMEM allocation");
    constexpr uint32_t kABytes = kTM * 128, kBBytes = BN * 128, kStage = kABytes + kBBytes;
    static_assert(4 * 32 * kEpiPitch * 4 <= kStage, "the output staging fits in stage 0");
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_full[STAGES], s_empty[STAGES];
    __shared__ float s_y[16];             // kEpiHead
    __shared__ volatile int s_fail;
    __shared__ volatile int s_inflight;   // a drain wait ran out: copies or products may be in flight
    // 128 B swizzle: stage bases 1024 B aligned
    unsigned char *sm = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int nslab = (K + kSlab - 1) / kSlab;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&s_tmem)), "r"((uint32_t)BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (t == 0) {
        s_fail = 0;
        s_inflight = 0;
        for (int i = 0; i < STAGES; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_full[i])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_empty[i])));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(tmA) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(tmB) : "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");   // nothing of the kernels before is read or written until here
    // slab j lives in stage j % STAGES as that stage's use u = j / STAGES; each
    // barrier completes once per use, so the wait for use u is parity u % 2
    if (t == 0) {
        int issued = 0;
        for (int j = 0; j < nslab; ++j) {
            const int s = j % STAGES, u = j / STAGES;
            if (u > 0 && !mbar_wait(smem_u32(&s_empty[s]), (uint32_t)((u - 1) & 1))) {
                s_fail = 1;
                break;
            }
            const uint32_t a = smem_u32(sm + s * kStage), b = a + kABytes, fb = smem_u32(&s_full[s]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(kStage) : "memory");
            tma_load_2d(a, tmA, j * kSlab, m0, fb);
            tma_load_2d(b, tmB, j * kSlab, n0, fb);
            issued = j + 1;
        }
        // every copy in flight lands before the CTA can leave (immediate when all were consumed)
        for (int j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)
            if (!mbar_wait(smem_u32(&s_full[j % STAGES]), (uint32_t)((j / STAGES) & 1))) {
                s_fail = 1;
                s_inflight = 1;
                break;
            }
    } else if (t == 32) {
        int committed = 0;
        for (int sl = 0; sl < nslab; ++sl) {
            const int s = sl % STAGES;
            if (!mbar_wait(smem_u32(&s_full[s]), (uint32_t)((sl / STAGES) & 1))) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ad = smem_u32(sm + s * kStage), bd = ad + kABytes;
            const int ksteps = (K - sl * kSlab) >= kSlab ? kSlab / 16 : (K - sl * kSlab + 15) / 16;
            for (int kk = 0; kk < ksteps; ++kk) {
                const uint32_t acc = (sl > 0 || kk > 0) ? 1u : 0u;
                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                             " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                             ::"r"(tmem), "l"(sw128_desc(ad + kk * 32)), "l"(sw128_desc(bd + kk * 32)),
                               "r"(idesc_bf16(kTM, BN)), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(&s_empty[s])) : "memory");
            committed = sl + 1;
        }
        // the last commit covers every product issued: they complete before TMEM is read or freed
        if (committed > 0) {
            const int c = committed - 1;
            if (!mbar_wait(smem_u32(&s_empty[c % STAGES]), (uint32_t)((c / STAGES) & 1))) {
                s_fail = 1;
                s_inflight = 1;
            }
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!s_fail && nslab > 0) {
        // every copy landed and every product ran: stage 0 is free for the output rows
        float *stg = reinterpret_cast<float *>(sm) + warp * 32 * kEpiPitch;
        const int q = lane & 7;
        const int myrow = m0 + warp * 32 + lane;   // the row of this lane's TMEM lane
        if constexpr (EPI == kEpiHead) {
            const int row0 = blockIdx.x * 16;
            uint32_t r[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), r);   // column 0: the layer's one output
            if (myrow >= row0 && myrow < row0 + 16) s_y[myrow - row0] = __uint_as_float(r[0]);
            __syncthreads();
            head_rows(ea, s_y, row0, sm);
        }
        for (int c0 = 0; EPI != kEpiHead && c0 < BN; c0 += 32) {
            uint32_t r[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
            const int cb = n0 + c0;   // the chunk's first column
            float4 *mine = reinterpret_cast<float4 *>(stg + lane * kEpiPitch);
            if (EPI == kEpiGroup && ea.demb != nullptr) {
                // one row's 32 columns at a time, a lane each: rows of one vertex meet in 32 addresses
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    mine[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                          __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                int p = myrow < ea.m_real ? ea.pids[myrow] : 0;
                p = p < 0 ? 0 : (p > ea.n_ids ? ea.n_ids : p);
                __syncwarp();
                const int rows = min(32, ea.m_real - (m0 + warp * 32));
                for (int rr = 0; rr < rows; ++rr)
                    atomicAdd(ea.demb + (size_t)__shfl_sync(0xffffffffu, p, rr) * 32 + lane, stg[rr * kEpiPitch + lane]);
                __syncwarp();
            } else if constexpr (EPI != kEpiGeluBwd) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    mine[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                          __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                __syncwarp();
                const int col = cb + q * 4;
                const float4 bv = bias ? *reinterpret_cast<const float4 *>(bias + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int rr = i * 4 + (lane >> 3);
                    const int row = m0 + warp * 32 + rr;
                    float4 v = *reinterpret_cast<const float4 *>(stg + rr * kEpiPitch + q * 4);
                    v.x += bv.x; v.y += bv.y; v.z += bv.z; v.w += bv.w;
                    if (row < M && (EPI != kEpiGroup || col < ea.n_real))
                        *reinterpret_cast<float4 *>(C + (size_t)row * ldc + col) = v;
                }
                __syncwarp();
            }
            if constexpr (EPI == kEpiGeluFwd || EPI == kEpiGeluBwd) {
                // this lane's row of the chunk: 32 values in bf16
                __nv_bfloat16 hv[32];
                if constexpr (EPI == kEpiGeluFwd) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float zv = __uint_as_float(r[i]) + (bias ? bias[cb + i] : 0.f);
                        hv[i] = __float2bfloat16(myrow < ea.m_real ? gelu(zv) : 0.f);
                    }
                } else {
                    float zr[32] = {};
                    if (myrow < ea.m_real) {
                        const float4 *zp = reinterpret_cast<const float4 *>(ea.z + (size_t)myrow * ea.ldz + cb);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 z4 = zp[i];
                            zr[4 * i] = z4.x; zr[4 * i + 1] = z4.y; zr[4 * i + 2] = z4.z; zr[4 * i + 3] = z4.w;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        hv[i] = __float2bfloat16(myrow < ea.m_real ? __uint_as_float(r[i]) * gelu_grad(zr[i]) : 0.f);
                    // column sums of the rounded values: rows staged in shared memory, lane i sums column i
                    float *mrow = stg + lane * kEpiPitch;
#pragma unroll
                    for (int i = 0; i < 32; ++i) mrow[i] = __bfloat162float(hv[i]);
                    __syncwarp();
                    float cs = 0.f;
#pragma unroll 8
                    for (int rr = 0; rr < 32; ++rr) cs += stg[rr * kEpiPitch + lane];
                    if (cs != 0.f) atomicAdd(ea.colsum + cb + lane, cs);
                    __syncwarp();
                }
                if (myrow < ea.m_store) {
                    // element 2k at the lower address: the low half of word k
                    uint32_t w[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        w[k] = (uint32_t)__bfloat16_as_ushort(hv[2 * k]) |
                               ((uint32_t)__bfloat16_as_ushort(hv[2 * k + 1]) << 16);
                    uint4 *hp = reinterpret_cast<uint4 *>(ea.h + (size_t)myrow * ea.ldh + cb);
#pragma unroll
                    for (int i = 0; i < 4; ++i) hp[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
#pragma unroll
                    for (int i = 0; i < 32; ++i) ea.ht[(size_t)(cb + i) * ea.ldt + myrow] = hv[i];
                }
            }
        }
    } else if (s_fail && t == 0) {
        atomicOr(err, s_inflight ? (4 | 8) : 4);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // products still in flight may write these columns: they stay allocated
    if (warp == 0 && !s_inflight) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN));
    }
}

template <int BN, int EPI>
__global__ void __launch_bounds__(kThreads)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               float *__restrict__ C, int ldc, int M, int K, const float *__restrict__ bias, int *err,
               const EpiArgs ea) {
    // kEpiHead: a CTA for each 16 rows, all of a tile's CTAs taking its product
    const int m0 = EPI == kEpiHead ? (int)(blockIdx.x * 16 / kTM) * kTM : (int)blockIdx.x * kTM;
    gemm_tile<BN, EPI, kStages>(&tmA, &tmB, m0, blockIdx.y * BN, C, ldc, M, K, bias, err, ea);
}

// Up to kGroup products of one launch, tiles of 128 x 32 numbered product by product
constexpr int kGroup = 5;
struct GroupArgs {
    CUtensorMap a[kGroup], b[kGroup];
    int first[kGroup + 1];        // first tile of each product; the number of tiles
    int mt[kGroup], n0[kGroup];   // tiles along M; the first column
    float *C[kGroup];
    int ldc[kGroup], M[kGroup], K[kGroup], n_real[kGroup];
    // the last product's columns go to the embedding gradients
    float *demb;
    const int32_t *pids;
    int n_ids, m_real, n;
    int *err;
    // sum_rows, by a CTA behind the tiles
    const float2 *part;
    int nparts;
    float *loss, *db;
};
__global__ void __launch_bounds__(kThreads) gemm_group_kernel(const __grid_constant__ GroupArgs g) {
    if ((int)blockIdx.x == g.first[g.n]) {
        asm volatile("griddepcontrol.launch_dependents;");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        sum_rows(g.part, g.nparts, g.m_real, g.loss, g.db);
        return;
    }
    int p = 0;
    while (p + 1 < g.n && (int)blockIdx.x >= g.first[p + 1]) ++p;
    const int i = (int)blockIdx.x - g.first[p];
    EpiArgs ea;
    ea.n_real = g.n_real[p];
    ea.m_real = g.m_real;
    ea.demb = p == g.n - 1 ? g.demb : nullptr;
    ea.pids = g.pids;
    ea.n_ids = g.n_ids;
    gemm_tile<32, kEpiGroup, kDeepStages>(&g.a[p], &g.b[p], i % g.mt[p] * kTM, g.n0[p] + i / g.mt[p] * 32, g.C[p],
                                          g.ldc[p], g.M[p], g.K[p], nullptr, g.err, ea);
}

inline size_t smem_bytes(int BN, int stages = kStages) {
    return stages * ((size_t)kTM * 128 + (size_t)BN * 128) + 1024;
}

// 2-D tensor map of a row-major bf16 matrix (rows x cols, row pitch ld elements,
// 16 B aligned): boxes of 64 columns x box_rows rows, 128 B swizzle, zero outside.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        // the entry point as CUDA 12.0 introduced it (its signature has not changed since)
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

inline bool make_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint64_t ld,
                     uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn || ((uintptr_t)base & 15u) || ((ld * 2) & 15u)) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kSlab, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tc
}  // namespace wk
