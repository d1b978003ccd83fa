// The estimator's prediction as one kernel on the 5th-generation tensor cores:
// input (48 features | 32-d embedding) -> 3 hidden layers of 256 with GELU ->
// one output, 128 samples a tile, nothing between the layers leaving the SM.
//
// What bounds it: the activation.  A tile's 3 x 128 x 256 exact GELUs (erff) are
// 98k warp instructions, 13 us of an SM's issue slots; its matrix products are
// 3 us of tensor pipe and its 320 KB of weights 4 us of L2 reads.  As separate
// kernels (input, three GEMMs with GELU, output GEMM, bias) every layer's
// values went through L2 in fp32 and bf16, row-major and transposed, the
// products ran on 16 to 64 CTAs, and each batch of 4096 samples cost six
// launches, 45 us.  100k samples from host memory to host memory took 2130 us
// so, 249 with this kernel and copies that overlap it.
//
// A CTA (one per SM) works on two tiles at once, eight warps each, so that one
// tile's products and their latency are behind the other's activation: with
// one tile a CTA issued in half of the cycles and took 26 us a tile, with two
// 20.  Warp w of a tile takes TMEM lanes 32 (w % 4) .. and columns 128 (w / 4)
// ..; one thread loads weights, slabs of 64 input columns x 256 outputs (TMA,
// 128 B swizzle) through two stages, ahead of the products across layers and
// tiles; one thread issues the products, the two tiles' layers in turn.  A
// tile's activations are one buffer of four 128 x 64 bf16 slabs in the same
// swizzle: a layer's products have read it (acc_ready) before the epilogue
// overwrites it with the next layer's input (act_ready).  Values are rounded to
// bf16 and accumulated in fp32 exactly where the training path's kernels
// (wk_tc_gemm.cuh) do.
//
// Every wait is bounded, as there: one that runs out sets bit 2 of *err and
// ends the CTA; if the CTA's copies or products cannot be drained either, bit 3
// and its TMEM columns stay allocated.
#pragma once

#include "wk_tc_gemm.cuh"

namespace wk {
namespace mlpf {

using tc::mbar_wait;
using tc::smem_u32;

constexpr int kTile = 128, kHid = 256, kStages = 2;
constexpr int kEpi = 256, kThreads = 2 * kEpi + 64;   // a tile's threads; two tiles, the loads, the products
constexpr int kInCols = 48, kEmbCols = 32;
constexpr uint32_t kActSlab = kTile * 128, kWSlab = kHid * 128, kOutSlab = 32 * 128;   // 64 bf16 columns each
constexpr uint32_t kSmem = 2 * 4 * kActSlab + kStages * kWSlab + 4 * kOutSlab + 1024;

struct Args {
    const float *feats;     // [n x 48], 16 B aligned
    const int32_t *pids;
    const float *bias[4];   // three of 256 (16 B aligned) and the output's
    const float *emb;       // [(n_ids + 1) x 32], 16 B aligned
    float *out;
    int *err;
    int n_ids;
    long long n;
};

__device__ __forceinline__ void arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mma(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                 "l"(tc::sw128_desc(a)), "l"(tc::sw128_desc(b)), "r"(idesc), "r"(acc));
}
// eight consecutive columns (a 16 B chunk) of a row of a swizzled slab
__device__ __forceinline__ uint32_t chunk_at(int row, int chunk) {
    return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {   // lo at the lower address
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16(lo)) |
           ((uint32_t)__bfloat16_as_ushort(__float2bfloat16(hi)) << 16);
}

__global__ void __launch_bounds__(kThreads, 1)
forward_kernel(const __grid_constant__ CUtensorMap w0, const __grid_constant__ CUtensorMap w1,
               const __grid_constant__ CUtensorMap w2, const __grid_constant__ CUtensorMap w3,
               const __grid_constant__ Args a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t w_full[kStages], w_empty[kStages], out_full, act_ready[2], acc_ready[2], drained;
    __shared__ __align__(16) float s_bias[3][kHid];
    __shared__ volatile int s_fail, s_inflight;
    unsigned char *sm = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *acts = sm, *wst = sm + 2 * 4 * kActSlab, *wout = wst + kStages * kWSlab;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const long long ntiles = (a.n + kTile - 1) / kTile;
    // tile g of round k; the first of a CTA's two is there when the second is
    auto tile_at = [&](long long k, int g) { return (2 * k + g) * (long long)gridDim.x + blockIdx.x; };
    if (warp == 2 * kEpi / 32 + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(2u * kHid));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (t == 0) {
        s_fail = 0;
        s_inflight = 0;
        auto init = [](uint64_t *b, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
        };
        for (int i = 0; i < kStages; ++i) { init(&w_full[i], 1); init(&w_empty[i], 1); }
        init(&out_full, 1);
        for (int g = 0; g < 2; ++g) { init(&act_ready[g], kEpi); init(&acc_ready[g], 1); }
        init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = t; i < 3 * kHid; i += kThreads) (&s_bias[0][0])[i] = a.bias[i / kHid][i % kHid];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;

    if (t == 2 * kEpi) {
        // ---- weights, in the order of the products
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&out_full)),
                     "r"(4 * kOutSlab)
                     : "memory");
        for (int s = 0; s < 4; ++s)
            tc::tma_load_2d(smem_u32(wout + s * kOutSlab), &w3, s * 64, 0, smem_u32(&out_full));
        long long issued = 0;
        bool ok = true;
        for (long long k = 0; ok && tile_at(k, 0) < ntiles && !s_fail; ++k) {
            for (int i = 0; ok && i < 6; ++i) {
                const int layer = i >> 1, g = i & 1;
                if (tile_at(k, g) >= ntiles) continue;
                const CUtensorMap *map = layer == 0 ? &w0 : (layer == 1 ? &w1 : &w2);
                for (int j = 0; j < (layer == 0 ? 2 : 4); ++j, ++issued) {
                    const int s = (int)(issued % kStages);
                    const long long u = issued / kStages;
                    if (u > 0 && !mbar_wait(smem_u32(&w_empty[s]), (uint32_t)((u - 1) & 1))) {
                        ok = false;
                        break;
                    }
                    const uint32_t full = smem_u32(&w_full[s]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(kWSlab)
                                 : "memory");
                    tc::tma_load_2d(smem_u32(wst + s * kWSlab), map, j * 64, 0, full);
                }
            }
        }
        if (!ok) s_fail = 1;
        // every copy lands before the CTA can leave
        bool landed = mbar_wait(smem_u32(&out_full), 0u);
        for (long long i = issued > kStages ? issued - kStages : 0; i < issued; ++i)
            landed = mbar_wait(smem_u32(&w_full[i % kStages]), (uint32_t)((i / kStages) & 1)) && landed;
        if (!landed) {
            s_fail = 1;
            s_inflight = 1;
        }
    } else if (t == 2 * kEpi + 32) {
        // ---- products: layers 0..2 and the output (3), the two tiles in turn
        long long used = 0;
        uint32_t act_parity[2] = {0u, 0u};
        bool ok = mbar_wait(smem_u32(&out_full), 0u);
        for (long long k = 0; ok && tile_at(k, 0) < ntiles && !s_fail; ++k) {
            for (int i = 0; ok && i < 8; ++i) {
                const int layer = i >> 1, g = i & 1;
                if (tile_at(k, g) >= ntiles) continue;
                const uint32_t d = tmem + (uint32_t)(g * kHid), act = smem_u32(acts + g * 4 * kActSlab);
                ok = mbar_wait(smem_u32(&act_ready[g]), act_parity[g]);
                act_parity[g] ^= 1u;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (layer == 3) {
                    for (int kk = 0; kk < 16; ++kk)
                        mma(d, act + (kk >> 2) * kActSlab + (kk & 3) * 32,
                            smem_u32(wout + (kk >> 2) * kOutSlab) + (kk & 3) * 32, tc::idesc_bf16(kTile, 32),
                            kk > 0 ? 1u : 0u);
                } else {
                    for (int j = 0; j < (layer == 0 ? 2 : 4); ++j, ++used) {
                        const int s = (int)(used % kStages);
                        ok = mbar_wait(smem_u32(&w_full[s]), (uint32_t)((used / kStages) & 1));
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t ad = act + j * kActSlab, bd = smem_u32(wst + s * kWSlab);
                        const int ksteps = layer == 0 && j == 1 ? 1 : 4;   // 80 input columns
                        for (int kk = 0; kk < ksteps; ++kk)
                            mma(d, ad + kk * 32, bd + kk * 32, tc::idesc_bf16(kTile, kHid), j > 0 || kk > 0 ? 1u : 0u);
                        commit(smem_u32(&w_empty[s]));
                    }
                }
                if (ok) commit(smem_u32(&acc_ready[g]));
            }
        }
        if (!ok) s_fail = 1;
        // every product issued completes before TMEM is freed
        commit(smem_u32(&drained));
        if (!mbar_wait(smem_u32(&drained), 0u)) {
            s_fail = 1;
            s_inflight = 1;
        }
    } else if (t < 2 * kEpi) {
        // ---- input and epilogues
        const int g = t / kEpi, row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1;
        const uint32_t tm = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * kHid);
        const uint32_t act_done = smem_u32(&act_ready[g]), acc_done = smem_u32(&acc_ready[g]);
        unsigned char *act = acts + g * 4 * kActSlab;
        uint32_t acc_parity = 0u;
        bool ok = true;
        // tcgen05.ld takes a whole warp: its lanes go on or leave together
        auto all = [](bool x) { return __all_sync(0xffffffffu, x) != 0; };
        for (long long k = 0; ok && tile_at(k, g) < ntiles && all(!s_fail); ++k) {
            const long long r = tile_at(k, g) * kTile + row;
            {
                int p = 0;
                if (r < a.n) {
                    p = a.pids[r];
                    p = p < 0 ? 0 : (p > a.n_ids ? a.n_ids : p);
                }
                const float4 *f4 = reinterpret_cast<const float4 *>(a.feats + r * kInCols);
                const float4 *e4 = reinterpret_cast<const float4 *>(a.emb + (size_t)p * kEmbCols);
#pragma unroll
                for (int i = 0; i < 5; ++i) {   // chunks of 8 columns: 0..5 features, 6..9 embedding
                    const int c = half * 5 + i;
                    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
                    if (r < a.n) {
                        const float4 *src = c < kInCols / 8 ? f4 + 2 * c : e4 + 2 * (c - kInCols / 8);
                        x = __ldg(src);
                        y = __ldg(src + 1);
                    }
                    *reinterpret_cast<uint4 *>(act + (c >> 3) * kActSlab + chunk_at(row, c & 7)) =
                        make_uint4(pack2(x.x, x.y), pack2(x.z, x.w), pack2(y.x, y.y), pack2(y.z, y.w));
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            arrive(act_done);
            for (int layer = 0; ok && layer < 3; ++layer) {
                ok = all(mbar_wait(acc_done, acc_parity));
                acc_parity ^= 1u;
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = half * 128; c0 < half * 128 + 128; c0 += 32) {
                    uint32_t v[32];
                    tc::tmem_ld32(tm + (uint32_t)c0, v);
                    uint32_t w[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float2 b = *reinterpret_cast<const float2 *>(&s_bias[layer][c0 + 2 * i]);
                        w[i] = pack2(tc::gelu(__uint_as_float(v[2 * i]) + b.x),
                                     tc::gelu(__uint_as_float(v[2 * i + 1]) + b.y));
                    }
                    unsigned char *slab = act + (c0 >> 6) * kActSlab;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        *reinterpret_cast<uint4 *>(slab + chunk_at(row, ((c0 & 63) >> 3) + i)) =
                            make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                arrive(act_done);
            }
            if (!ok) break;
            ok = all(mbar_wait(acc_done, acc_parity));
            acc_parity ^= 1u;
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (half == 0) {
                uint32_t y;
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(y) : "r"(tm));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (r < a.n) a.out[r] = __uint_as_float(y) + __ldg(a.bias[3]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        if (!ok) s_fail = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (t == 0 && s_fail) atomicOr(a.err, s_inflight ? (4 | 8) : 4);
    // products still in flight may write these columns: they stay allocated
    if (warp == 2 * kEpi / 32 + 1 && !s_inflight) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kHid));
    }
}

}  // namespace mlpf
}  // namespace wk
