// The learned cardinality estimator: an MLP trained and evaluated by
// hand-written BF16 tensor-core kernels.
//
// Model: x = [48 pattern features | 32-d embedding of the predicate] (80)
//        -> 256 -> 256 -> 256 (GELU after each) -> 1
// It predicts log(1 + rows) of the table after a pattern is applied.  Weights
// and activations are BF16, every product accumulates in FP32 in tensor
// memory on the 5th-generation tensor cores (tcgen05.mma with TMA-staged
// operands, wk_tc_gemm.cuh), and the optimiser is FP32 Adam over FP32 master
// weights whose BF16 copies are refreshed after each step.
//
// One GEMM kernel does all products: C[M x N] = A[M x K] . B[N x K]^T with A
// and B row-major (K contiguous), which is the natural form for the forward
// product (X . W^T), for the input gradient (dZ . W, with W^T kept as a BF16
// copy) and for the weight gradient (dZ^T . X, with the transposed
// activations written by the forward pass).  Dimensions are padded: M and N
// to multiples of 64, K to multiples of 16; padding is zero.  The hidden
// layers' activation runs in the GEMM's epilogue: the forward product writes
// GELU(Z) in bf16 (row-major and transposed) beside Z, and the input-gradient
// product of the layer above writes dZ = dH * GELU'(Z) with the bias
// gradient (its column sums), so dH itself is never stored.  Prediction, which
// keeps nothing for a backward pass, is one kernel (wk_mlp_forward.cuh).
//
// A forward and backward pass is eight kernels, each launched ahead of its
// turn: the input, three layers, the output layer with the loss and the first
// backward layer, two layers back, and every weight gradient with the
// embedding's in one.  What bounds a step of 1024 rows is the chain of those
// launches and a product's latency (5 to 8 us, 64 CTAs).  As 16 kernels and 4
// copies, each weight gradient in the chain, the step kept the GPU for 155 us,
// so for 61 us.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_bf16.h>

#include "wk_runtime.h"
#include "wk_tc_gemm.cuh"
#include "wk_mlp_forward.cuh"

namespace wk {
namespace mlp {

constexpr int kIn = 48;       // pattern features
constexpr int kEmb = 32;      // predicate embedding
constexpr int kX = kIn + kEmb;   // 80
constexpr int kH = 256;
constexpr int kOutPad = 64;   // output layer padded to one GEMM tile
constexpr int kXPadN = 128;   // W1^T rows padded (dX GEMM has N = 80 -> 128)
constexpr float kB1 = 0.9f, kB2 = 0.999f;   // Adam moment decay rates

// ------------------------------------------------------------ elementwise
// X0 [Mp x 80] bf16 = [feats | emb[pid]] for real rows, 0 for padding, and its
// transpose, 32 rows a CTA; the ids and targets, which may lie in host memory,
// brought to the device (pids_to and tgt_to, or in place); and the words that
// the step adds into, cleared.
__global__ void __launch_bounds__(256)
build_input_kernel(const float *feats, const int32_t *pids, const float *tgt,
                   int32_t *pids_to, float *tgt_to, int M, int Mp,
                   const float *__restrict__ emb, int n_ids, __nv_bfloat16 *__restrict__ X0,
                   __nv_bfloat16 *__restrict__ X0t, float *__restrict__ zero, int64_t nzero) {
    __shared__ __nv_bfloat16 tile[kX][34];   // 17 words a column: the transposing reads and writes spread over the banks
    __shared__ int s_pid[32];
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r0 = blockIdx.x * 32, t = threadIdx.x;
    if (t < 32 && r0 + t < M) {
        const int p = pids[r0 + t];
        s_pid[t] = p < 0 ? 0 : (p > n_ids ? n_ids : p);
        pids_to[r0 + t] = p;
        tgt_to[r0 + t] = tgt[r0 + t];
    }
    float fv[32 * kIn / 256];   // the features, in flight with the ids
#pragma unroll
    for (int q = 0; q < 32 * kIn / 256; ++q) {
        const int i = q * 256 + t;
        fv[q] = r0 + i / kIn < M ? feats[(size_t)r0 * kIn + i] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 32 * kIn / 256; ++q) tile[(q * 256 + t) % kIn][(q * 256 + t) / kIn] = __float2bfloat16(fv[q]);
    for (int i = t; i < 32 * kEmb; i += 256) {
        const int r = i / kEmb, c = i % kEmb;
        tile[kIn + c][r] = __float2bfloat16(r0 + r < M ? emb[(size_t)s_pid[r] * kEmb + c] : 0.f);
    }
    __syncthreads();
    for (int i = t; i < 32 * kX; i += 256) X0[(size_t)r0 * kX + i] = tile[i % kX][i / kX];
    for (int i = t; i < 32 * kX; i += 256) X0t[(size_t)(i / 32) * Mp + r0 + i % 32] = tile[i / 32][i % 32];
    for (int64_t i = (int64_t)blockIdx.x * 256 + t; i < nzero; i += (int64_t)gridDim.x * 256) zero[i] = 0.f;
}

// Adam over fp32 master weights; g, m, v, w all of length n.  The bias
// corrections (1 - b1^t, 1 - b2^t) of this step are cbias[*bidx], so that a
// captured step reads the current ones when it is replayed.
__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, int64_t n, float lr, float b1, float b2, float eps,
                            const float2 *__restrict__ cbias, const int *__restrict__ bidx) {
    const float2 c = cbias[*bidx];
    const float c1 = c.x, c2 = c.y;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// Batch *bidx of an epoch: rows order[*bidx * batch + i], i < M, of the
// device-resident samples into the step's input buffers.
__global__ void gather_batch_kernel(const float *__restrict__ all_feats, const int32_t *__restrict__ all_pids,
                                    const float *__restrict__ all_tgt, const int64_t *__restrict__ order,
                                    const int *__restrict__ bidx, int batch, int M, float *__restrict__ feats,
                                    int32_t *__restrict__ pids, float *__restrict__ tgt) {
    const int64_t b0 = (int64_t)(*bidx) * batch;
    const int64_t n = (int64_t)M * kIn;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / kIn), c = (int)(i % kIn);
        const int64_t j = order[b0 + r];
        feats[i] = all_feats[j * kIn + c];
        if (c == 0) {
            pids[r] = all_pids[j];
            tgt[r] = all_tgt[j];
        }
    }
}

// the next batch of the epoch
__global__ void bump_kernel(int *bidx) { ++*bidx; }

// bf16 copies of a weight matrix W [rows x cols] (fp32): row-major into Wb
// (ld = ldb, zero padded) and transposed into Wt (ld = ldt)
__global__ void weight_copy_kernel(const float *__restrict__ W, int rows, int cols, __nv_bfloat16 *__restrict__ Wb,
                                   int ldb, int rows_pad, __nv_bfloat16 *__restrict__ Wt, int ldt, int cols_pad) {
    const int64_t n = (int64_t)rows_pad * ldb;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / ldb), c = (int)(i % ldb);
        const float v = (r < rows && c < cols) ? W[(size_t)r * cols + c] : 0.f;
        Wb[i] = __float2bfloat16(v);
        if (c < cols_pad && r < ldt) Wt[(size_t)c * ldt + r] = __float2bfloat16(v);
    }
}

}  // namespace mlp
}  // namespace wk

using namespace wk;
using namespace wk::mlp;

struct wk_mlp {
    wk_ctx *ctx = nullptr;
    int n_ids = 0;
    int trusted = 1;             // cleared by wk_mlp_validate when held-out q-error exceeds its bound
    int cap_m = 0;               // padded batch capacity
    // fp32 master parameters, gradients, Adam moments (one contiguous block)
    float *params = nullptr, *grads = nullptr, *m1 = nullptr, *m2 = nullptr;
    int64_t n_params = 0;
    // views into params/grads
    int64_t off_w[4] = {}, off_b[4] = {}, off_emb = 0;
    // bf16 weights (row-major, padded) and transposes
    __nv_bfloat16 *wb[4] = {}, *wt[4] = {};
    // activations (capacity cap_m)
    __nv_bfloat16 *x0 = nullptr, *x0t = nullptr, *h[3] = {}, *ht[3] = {}, *dz[3] = {}, *dzt[3] = {},
                  *dy = nullptr;
    float *z[3] = {}, *feats = nullptr, *tgt = nullptr;
    float *loss = nullptr;       // the step's, the epoch's sum; then d_err, an int
    float2 *part = nullptr;      // the output layer's sums per CTA
    int32_t *pids = nullptr;
    int *bidx = nullptr;         // the batch of the epoch a training step takes
    float2 *cbias = nullptr;     // Adam bias corrections of an epoch's steps
    int64_t cbias_cap = 0;
    int64_t step = 0;
    int64_t kernels = 0;
    int *d_err = nullptr;        // device flag of the tensor-core GEMM (bit 2: a wait ran out,
                                 // bit 3: work left in flight, TMEM kept)
    float *h_loss = nullptr;     // pinned mirror of loss and what follows it
    int status = 0;              // a host-side GEMM failure since the last check
    int sms = 152;               // multiprocessors of the device (GEMM tile width choice)
    bool broken = false;         // a GEMM left work in flight: no further GEMM is launched
    // prediction: two buffers of features in flight, the outputs and ids, a stream for the copies in, and a pinned block for small calls
    DevBuf stage[2], pred;
    cudaStream_t copy = nullptr;
    cudaEvent_t copied[2] = {}, used[2] = {};
    unsigned char *h_small = nullptr, *h_small_dev = nullptr;
};

namespace {

const int kRows[4] = {kH, kH, kH, 1};        // output dim of each layer
const int kCols[4] = {kX, kH, kH, kH};       // input dim of each layer
const int kRowsPad[4] = {kH, kH, kH, kOutPad};

inline int pad64(int x) { return (x + 63) / 64 * 64; }
unsigned int nblk(int64_t n) { int64_t b = (n + 255) / 256; return (unsigned int)(b > 2048 ? 2048 : (b < 1 ? 1 : b)); }

void refresh_bf16(wk_mlp *m, cudaStream_t s) {
    for (int l = 0; l < 4; ++l) {
        // W^T of layer l is [cols x rows_pad]: the dX product takes it as B
        // with N = cols (layer 0 pads 80 -> 128; the extra rows stay zero)
        // (the output layer's is not needed: its dX is row-wise)
        const int tcols = (l == 0) ? kXPadN : (l == 3 ? 0 : kH);
        weight_copy_kernel<<<nblk((int64_t)kRowsPad[l] * kCols[l]), 256, 0, s>>>(
            m->params + m->off_w[l], kRows[l], kCols[l], m->wb[l], kCols[l], kRowsPad[l], m->wt[l], kRowsPad[l], tcols);
    }
    m->kernels += 4;
}

// A launch that may take its place before the kernels ahead of it are done
// (its kernel waits for them before it touches memory).
template <class... P, class... A>
void launch_ahead(void (*k)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, const A &...args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, args...);
}

bool refused(wk_mlp *m) {
    if (m->broken && !m->status)
        m->status = set_error(WK_EDEVICE, "estimator: an earlier tensor-core GEMM left work in flight; "
                                          "destroy the estimator");
    return m->broken;
}

// C = A . B^T (+ bias) on the tensor cores (wk_tc_gemm.cuh), with the
// epilogue EPI; N is a multiple of 64.  The tile width is the widest that still
// gives a full wave of CTAs, else 32: these products are small, and more CTAs
// means more copies and products in flight and more warps for the epilogue.
template <int EPI>
void gemm(wk_mlp *m, const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, float *C, int ldc, int M, int N,
          int K, const float *bias, cudaStream_t s, const tc::EpiArgs &ea) {
    if (refused(m)) return;
    if (M <= 0 || K <= 0 || N <= 0 || N % 64 || ldc % 4 || ((uintptr_t)C & 15u) || ((uintptr_t)bias & 15u) ||
        ((uintptr_t)ea.h & 15u) || ea.ldh % 8 || !ea.ht || ea.m_store > M ||
        (EPI == tc::kEpiGeluBwd && (((uintptr_t)ea.z & 15u) || ea.ldz % 4 || !ea.colsum))) {
        if (!m->status) m->status = set_error(WK_EINVAL, "estimator GEMM: shape or alignment (M %d, N %d, K %d)", M, N, K);
        return;
    }
    const int mt = (M + tc::kTM - 1) / tc::kTM;
    const int bn = (N % 256 == 0 && mt * (N / 256) >= m->sms)   ? 256
                   : (N % 128 == 0 && mt * (N / 128) >= m->sms) ? 128
                   : (mt * (N / 64) >= m->sms)                  ? 64
                                                                : 32;
    CUtensorMap ta, tb;
    if (!tc::make_map(&ta, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda, tc::kTM) ||
        !tc::make_map(&tb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, (uint32_t)bn)) {
        if (!m->status) m->status = set_error(WK_EDEVICE, "estimator GEMM: tensor map (M %d, N %d, K %d)", M, N, K);
        return;
    }
    auto *k = bn == 32    ? tc::gemm_tc_kernel<32, EPI>
              : bn == 64  ? tc::gemm_tc_kernel<64, EPI>
              : bn == 128 ? tc::gemm_tc_kernel<128, EPI>
                          : tc::gemm_tc_kernel<256, EPI>;
    launch_ahead(k, dim3((unsigned)mt, (unsigned)(N / bn)), tc::kThreads, tc::smem_bytes(bn), s, ta, tb, C, ldc, M, K,
                 bias, m->d_err, ea);
    m->kernels++;
}

// the epilogue operands of a hidden layer's activation: h / ht written for
// rows below Mp, values for rows below M
tc::EpiArgs act_args(int M, int Mp, __nv_bfloat16 *h, __nv_bfloat16 *ht, const float *z = nullptr,
                     float *colsum = nullptr) {
    tc::EpiArgs ea;
    ea.m_real = M;
    ea.m_store = Mp;
    ea.h = h;
    ea.ldh = kH;
    ea.ht = ht;
    ea.ldt = Mp;
    ea.z = z;
    ea.ldz = kH;
    ea.colsum = colsum;
    return ea;
}

template <int BN, int EPI>
bool set_gemm_smem() {
    return cudaFuncSetAttribute(tc::gemm_tc_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tc::smem_bytes(BN)) == cudaSuccess;
}

template <int EPI>
bool set_gemm_smem_all() {
    return set_gemm_smem<32, EPI>() && set_gemm_smem<64, EPI>() && set_gemm_smem<128, EPI>() &&
           set_gemm_smem<256, EPI>();
}

// the loss, the epoch's sum and the device flag to their pinned mirror
cudaError_t copy_status(wk_mlp *m, cudaStream_t s) {
    return cudaMemcpyAsync(m->h_loss, m->loss, 16, cudaMemcpyDeviceToHost, s);
}

// An error return once copies or kernels of the call are queued: nothing of them
// still reads or writes the caller's arrays or the pinned block when it returns.
int settled(wk_mlp *m, cudaStream_t s, int st) {
    cudaStreamSynchronize(m->copy);
    cudaStreamSynchronize(s);
    m->status = WK_OK;   // reported with this call
    return st;
}

// the status of the work queued since the last check: a host-side failure, a
// launch error, or a tensor-core wait that ran out (bit 2 of the device flag)
int check_status(wk_mlp *m, cudaStream_t s, const char *what, bool copied = false) {
    int st = m->status;
    m->status = WK_OK;
    if (st) return settled(m, s, st);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && !copied) e = copy_status(m, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return settled(m, s, cuda_fail(e, what));
    int f;
    std::memcpy(&f, m->h_loss + 2, sizeof(f));
    if (f) {
        cudaMemsetAsync(m->d_err, 0, sizeof(int), s);
        if (f & 8) {
            // copies or products may still be in flight and their CTA kept its
            // TMEM: the estimator launches no further GEMM
            m->broken = true;
            return set_error(WK_EDEVICE, "%s: a tensor-core GEMM wait ran out with work in flight; "
                                         "destroy the estimator", what);
        }
        return set_error(WK_ETIMEDOUT, "%s: a tensor-core GEMM wait ran out", what);
    }
    return WK_OK;
}

// The pinned block of small calls, which the kernels read and write in place: a
// copy to or from the caller's memory holds the host for some 14 us whatever its
// size.  The features of up to kSmallRows samples go through it (100 KB in 6 us
// on the host), ids, targets and predictions of up to kMidRows.
constexpr int kSmallRows = 1024, kMidRows = 16384;
constexpr size_t kSmallPids = sizeof(float) * kIn * kSmallRows, kSmallOut = kSmallPids + sizeof(int32_t) * kMidRows;
constexpr size_t kSmallBytes = kSmallOut + sizeof(float) * kMidRows;

// predictions for n samples in device-readable memory (wk_mlp_forward.cuh)
void predict(wk_mlp *m, const float *feats, const int32_t *pids, int64_t n, float *out, cudaStream_t s) {
    if (refused(m)) return;
    mlpf::Args a;
    a.feats = feats;
    a.pids = pids;
    for (int l = 0; l < 4; ++l) a.bias[l] = m->params + m->off_b[l];
    a.emb = m->params + m->off_emb;
    a.out = out;
    a.err = m->d_err;
    a.n_ids = m->n_ids;
    a.n = n;
    CUtensorMap w[4];
    bool ok = (((uintptr_t)feats | (uintptr_t)a.emb) & 15u) == 0;
    for (int l = 0; ok && l < 4; ++l)
        ok = tc::make_map(&w[l], m->wb[l], (uint64_t)kRowsPad[l], (uint64_t)kCols[l], (uint64_t)kCols[l],
                          l < 3 ? (uint32_t)kH : 32u);
    if (!ok) {
        if (!m->status) m->status = set_error(WK_EDEVICE, "estimator: tensor map or alignment of the prediction");
        return;
    }
    const int64_t tiles = (n + mlpf::kTile - 1) / mlpf::kTile;
    mlpf::forward_kernel<<<(unsigned)std::min<int64_t>(tiles, m->sms), mlpf::kThreads, mlpf::kSmem, s>>>(w[0], w[1], w[2],
                                                                                                       w[3], a);
    m->kernels++;
}

// The weight gradients dW_l = dZ_l^T . X_l (the layer's input), K the batch (of the
// output layer one row, dY^T . H_2), the embedding's from dX = dZ_0 . W_0, and the loss, in one launch: nothing waits for
// any of them, and each alone is 1 to 16 CTAs.
void gradient_group(wk_mlp *m, int M, int Mp, cudaStream_t s) {
    if (refused(m)) return;
    tc::GroupArgs g;
    bool ok = true;
    int at = 0;
    for (int i = 0; i < 3; ++i) {   // layers 2, 1, 0
        const int l = 2 - i, kin = kCols[l];
        ok = ok && tc::make_map(&g.a[i], m->dzt[l], kH, (uint64_t)Mp, (uint64_t)Mp, tc::kTM) &&
             tc::make_map(&g.b[i], l ? m->ht[l - 1] : m->x0t, (uint64_t)kin, (uint64_t)Mp, (uint64_t)Mp, 32);
        g.first[i] = at;
        g.mt[i] = kH / tc::kTM;
        g.n0[i] = 0;
        g.C[i] = m->grads + m->off_w[l];
        g.ldc[i] = g.n_real[i] = kin;
        g.M[i] = kH;
        g.K[i] = Mp;
        at += g.mt[i] * ((kin + 31) / 32);
    }
    ok = ok && tc::make_map(&g.a[3], m->dy, 1, (uint64_t)Mp, (uint64_t)Mp, tc::kTM) &&
         tc::make_map(&g.b[3], m->ht[2], kH, (uint64_t)Mp, (uint64_t)Mp, 32);
    g.first[3] = at;
    g.mt[3] = 1;
    g.n0[3] = 0;
    g.C[3] = m->grads + m->off_w[3];
    g.ldc[3] = g.n_real[3] = kH;
    g.M[3] = 1;
    g.K[3] = Mp;
    at += kH / 32;
    // columns 48..79 of dX: a tile of 32 from row 48 of W_0^T
    ok = ok && tc::make_map(&g.a[4], m->dz[0], (uint64_t)Mp, kH, kH, tc::kTM) &&
         tc::make_map(&g.b[4], m->wt[0], kXPadN, kH, kH, 32);
    g.first[4] = at;
    g.mt[4] = (Mp + tc::kTM - 1) / tc::kTM;
    g.n0[4] = kIn;
    g.C[4] = nullptr;
    g.ldc[4] = 0;
    g.n_real[4] = 0;
    g.M[4] = Mp;
    g.K[4] = kH;
    at += g.mt[4];
    g.first[5] = at;
    g.n = 5;
    g.demb = m->grads + m->off_emb;
    g.pids = m->pids;
    g.n_ids = m->n_ids;
    g.m_real = M;
    g.err = m->d_err;
    if (!ok) {
        if (!m->status) m->status = set_error(WK_EDEVICE, "estimator: tensor map of the weight gradients (M %d)", M);
        return;
    }
    g.part = m->part;
    g.nparts = Mp / 16;
    g.loss = m->loss;
    g.db = m->grads + m->off_b[3];
    launch_ahead(tc::gemm_group_kernel, dim3((unsigned)at + 1u), tc::kThreads, tc::smem_bytes(32, tc::kDeepStages), s, g);
    m->kernels++;
}

// The loss and every gradient for M rows of device-readable feats, pids and tgt
// (the latter two brought to m->pids and m->tgt).
void gradient_step(wk_mlp *m, const float *feats, const int32_t *pids, const float *tgt, int M, cudaStream_t s) {
    const int Mp = pad64(M);
    float *g = m->grads;
    // the biases' gradients and the embedding's are added into; they lie together
    launch_ahead(build_input_kernel, dim3((unsigned)(Mp / 32)), 256, 0, s, feats, pids, tgt, m->pids, m->tgt, M, Mp, (const float *)(m->params + m->off_emb), m->n_ids, m->x0, m->x0t,
                 g + m->off_b[0], m->n_params - m->off_b[0]);
    m->kernels++;
    const __nv_bfloat16 *in = m->x0;
    int kin = kX;
    for (int l = 0; l < 3; ++l) {
        // Z_l = X W_l^T + b_l, and H_l = GELU(Z_l) from the epilogue
        gemm<tc::kEpiGeluFwd>(m, in, kin, m->wb[l], kin, m->z[l], kH, Mp, kH, kin, m->params + m->off_b[l], s,
                              act_args(M, Mp, m->h[l], m->ht[l]));
        in = m->h[l];
        kin = kH;
    }
    // the output layer, the loss, dY, dZ_2 and the gradients of b4, b3
    if (!refused(m)) {
        tc::EpiArgs ea = act_args(M, Mp, m->dz[2], m->dzt[2], m->z[2], g + m->off_b[2]);
        ea.w = m->wb[3];
        ea.b = m->params + m->off_b[3];
        ea.tgt = m->tgt;
        ea.dy = m->dy;
        ea.part = m->part;
        CUtensorMap ta, tb;
        if (tc::make_map(&ta, m->h[2], (uint64_t)Mp, kH, kH, tc::kTM) && tc::make_map(&tb, m->wb[3], kOutPad, kH, kH, 32)) {
            launch_ahead(tc::gemm_tc_kernel<32, tc::kEpiHead>, dim3((unsigned)(Mp / 16)), tc::kThreads, tc::smem_bytes(32),
                         s, ta, tb, (float *)nullptr, 0, Mp, kH, (const float *)nullptr, m->d_err, ea);
            m->kernels++;
        } else if (!m->status) {
            m->status = set_error(WK_EDEVICE, "estimator: tensor map of the output layer (M %d)", M);
        }
    }
    // dZ_{l-1} = (dZ_l . W_l) * GELU'(Z_{l-1}) (B = W_l^T [256 x 256]), with db_{l-1}
    for (int l = 2; l > 0; --l)
        gemm<tc::kEpiGeluBwd>(m, m->dz[l], kH, m->wt[l], kH, nullptr, kH, Mp, kH, kH, nullptr, s,
                              act_args(M, Mp, m->dz[l - 1], m->dzt[l - 1], m->z[l - 1], g + m->off_b[l - 1]));
    gradient_group(m, M, Mp, s);
}

// an Adam update from the gradients
void update(wk_mlp *m, float lr, cudaStream_t s) {
    adam_kernel<<<nblk(m->n_params), 256, 0, s>>>(m->params, m->grads, m->m1, m->m2, m->n_params, lr, kB1, kB2, 1e-8f,
                                                  m->cbias, m->bidx);
    m->kernels++;
    refresh_bf16(m, s);
}

void free_mlp(wk_mlp *m) {
    if (m->ctx && m->ctx->device >= 0) cudaSetDevice(m->ctx->device);
    cudaFree(m->params);
    cudaFree(m->grads);
    cudaFree(m->m1);
    cudaFree(m->m2);
    for (int l = 0; l < 4; ++l) { cudaFree(m->wb[l]); cudaFree(m->wt[l]); }
    for (int l = 0; l < 3; ++l) {
        cudaFree(m->h[l]); cudaFree(m->ht[l]); cudaFree(m->z[l]); cudaFree(m->dz[l]); cudaFree(m->dzt[l]);
    }
    cudaFree(m->x0); cudaFree(m->x0t); cudaFree(m->dy);
    cudaFree(m->feats); cudaFree(m->tgt); cudaFree(m->loss); cudaFree(m->part); cudaFree(m->pids);
    cudaFree(m->bidx);
    cudaFree(m->cbias);
    if (m->h_loss) cudaFreeHost(m->h_loss);
    if (m->h_small) cudaFreeHost(m->h_small);
    for (int i = 0; i < 2; ++i) {
        if (m->copied[i]) cudaEventDestroy(m->copied[i]);
        if (m->used[i]) cudaEventDestroy(m->used[i]);
    }
    if (m->copy) cudaStreamDestroy(m->copy);
    delete m;
}

}  // namespace

extern "C" int wk_mlp_create(wk_ctx *ctx, int32_t n_ids, int32_t max_batch, uint64_t seed, wk_mlp **out) {
    if (!ctx || !out || n_ids < 1 || max_batch < 1 || max_batch > (1 << 20))
        return set_error(WK_EINVAL, "wk_mlp_create: bad arguments");
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_mlp_create: host-only context");
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    wk_mlp *m = new wk_mlp();
    m->ctx = ctx;
    m->n_ids = n_ids;
    m->cap_m = pad64(max_batch);
    cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, ctx->device);
    int64_t at = 0;
    for (int l = 0; l < 4; ++l) { m->off_w[l] = at; at += (int64_t)kRows[l] * kCols[l]; }
    for (int l = 0; l < 4; ++l) { m->off_b[l] = at; at += kRowsPad[l]; }
    m->off_emb = at;
    at += (int64_t)(n_ids + 1) * kEmb;
    m->n_params = at;
    const size_t P = sizeof(float) * (size_t)at, Mp = (size_t)m->cap_m;
    bool ok = cudaMalloc(&m->params, P) == cudaSuccess && cudaMalloc(&m->grads, P) == cudaSuccess &&
              cudaMalloc(&m->m1, P) == cudaSuccess && cudaMalloc(&m->m2, P) == cudaSuccess;
    for (int l = 0; ok && l < 4; ++l) {
        const int tcols = (l == 0) ? kXPadN : kH;
        ok = cudaMalloc(&m->wb[l], 2 * (size_t)kRowsPad[l] * kCols[l]) == cudaSuccess &&
             (l == 3 || cudaMalloc(&m->wt[l], 2 * (size_t)tcols * kRowsPad[l]) == cudaSuccess);
    }
    for (int l = 0; ok && l < 3; ++l)
        ok = cudaMalloc(&m->h[l], 2 * Mp * kH) == cudaSuccess && cudaMalloc(&m->ht[l], 2 * Mp * kH) == cudaSuccess &&
             cudaMalloc(&m->z[l], 4 * Mp * kH) == cudaSuccess && cudaMalloc(&m->dz[l], 2 * Mp * kH) == cudaSuccess &&
             cudaMalloc(&m->dzt[l], 2 * Mp * kH) == cudaSuccess;
    ok = ok && cudaMalloc(&m->x0, 2 * Mp * kX) == cudaSuccess && cudaMalloc(&m->x0t, 2 * Mp * kX) == cudaSuccess &&
         cudaMalloc(&m->dy, 2 * Mp) == cudaSuccess &&
         cudaMalloc(&m->part, sizeof(float2) * Mp / 16) == cudaSuccess &&
         cudaMalloc(&m->feats, 4 * Mp * kIn) == cudaSuccess && cudaMalloc(&m->tgt, 4 * Mp) == cudaSuccess &&
         cudaMalloc(&m->loss, 16) == cudaSuccess && cudaMalloc(&m->pids, 4 * Mp) == cudaSuccess &&
         cudaMalloc(&m->bidx, sizeof(int)) == cudaSuccess &&
         cudaHostAlloc((void **)&m->h_loss, 16, 0) == cudaSuccess &&
         cudaHostAlloc((void **)&m->h_small, kSmallBytes, cudaHostAllocMapped) == cudaSuccess &&
         cudaHostGetDevicePointer((void **)&m->h_small_dev, m->h_small, 0) == cudaSuccess &&
         cudaStreamCreateWithFlags(&m->copy, cudaStreamNonBlocking) == cudaSuccess &&
         cudaEventCreateWithFlags(&m->copied[0], cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&m->copied[1], cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&m->used[0], cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&m->used[1], cudaEventDisableTiming) == cudaSuccess &&
         cudaFuncSetAttribute(mlpf::forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlpf::kSmem) ==
             cudaSuccess &&
         set_gemm_smem_all<tc::kEpiGeluFwd>() && set_gemm_smem_all<tc::kEpiGeluBwd>() &&
         set_gemm_smem<32, tc::kEpiHead>() &&
         cudaFuncSetAttribute(tc::gemm_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)tc::smem_bytes(32, tc::kDeepStages)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        free_mlp(m);
        return set_error(WK_ENOMEM, "wk_mlp_create: allocation failed");
    }
    m->d_err = reinterpret_cast<int *>(m->loss + 2);
    // He-style initialisation (uniform with the fan-in bound), zero biases, small embeddings
    std::vector<float> h((size_t)at, 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < 4; ++l) {
        const float bound = std::sqrt(6.f / (float)kCols[l]) * (l == 3 ? 0.5f : 1.f);
        std::uniform_real_distribution<float> U(-bound, bound);
        for (int64_t i = 0; i < (int64_t)kRows[l] * kCols[l]; ++i) h[(size_t)(m->off_w[l] + i)] = U(rng);
    }
    std::normal_distribution<float> Nrm(0.f, 0.1f);
    for (int64_t i = 0; i < (int64_t)(n_ids + 1) * kEmb; ++i) h[(size_t)(m->off_emb + i)] = Nrm(rng);
    cudaStream_t s = ctx->stream;
    e = cudaMemcpyAsync(m->params, h.data(), P, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m1, 0, P, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->m2, 0, P, s);
    for (int l = 0; e == cudaSuccess && l < 3; ++l) {
        const int tcols = (l == 0) ? kXPadN : kH;
        e = cudaMemsetAsync(m->wt[l], 0, 2 * (size_t)tcols * kRowsPad[l], s);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(m->grads, 0, P, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->bidx, 0, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->loss, 0, 16, s);
    if (e != cudaSuccess) { int r = cuda_fail(e, "wk_mlp_create init"); free_mlp(m); return r; }
    refresh_bf16(m, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) { int r = cuda_fail(e, "wk_mlp_create sync"); free_mlp(m); return r; }
    *out = m;
    return WK_OK;
}

extern "C" int wk_mlp_destroy(wk_mlp *m) {
    if (m) free_mlp(m);
    return WK_OK;
}

extern "C" int64_t wk_mlp_num_params(wk_mlp *m) { return m ? m->n_params : 0; }

// parameter block layout: W1 [256x80], W2, W3 [256x256], W4 [1x256], b1, b2, b3 [256], b4 [64, first used], emb [(n_ids+1) x 32]
extern "C" int wk_mlp_get_params(wk_mlp *m, float *host, int64_t n) {
    if (!m || !host || n < m->n_params) return set_error(WK_EINVAL, "wk_mlp_get_params");
    cudaError_t e = cudaMemcpy(host, m->params, sizeof(float) * (size_t)m->n_params, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? WK_OK : cuda_fail(e, "wk_mlp_get_params");
}

extern "C" int wk_mlp_set_params(wk_mlp *m, const float *host, int64_t n) {
    if (!m || !host || n < m->n_params) return set_error(WK_EINVAL, "wk_mlp_set_params");
    cudaSetDevice(m->ctx->device);
    cudaError_t e = cudaMemcpy(m->params, host, sizeof(float) * (size_t)m->n_params, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "wk_mlp_set_params");
    refresh_bf16(m, m->ctx->stream);
    e = cudaStreamSynchronize(m->ctx->stream);
    return e == cudaSuccess ? WK_OK : cuda_fail(e, "wk_mlp_set_params sync");
}

// One forward + backward on rows 0..M-1 without an update: loss and the
// gradients of every parameter (same layout as the parameters).
extern "C" int wk_mlp_gradients(wk_mlp *m, const float *feats, const int32_t *pids, const float *tgt, int32_t M,
                                float *grads_host, float *loss_host) {
    if (!m || !feats || !pids || !tgt || M < 1 || M > m->cap_m) return set_error(WK_EINVAL, "wk_mlp_gradients");
    cudaSetDevice(m->ctx->device);
    cudaStream_t s = m->ctx->stream;
    int st;
    cudaError_t e = cudaSuccess;
    const float *f = m->feats, *t = m->tgt;
    const int32_t *p = m->pids;
    if (M <= kSmallRows) {
        std::memcpy(m->h_small, feats, sizeof(float) * (size_t)M * kIn);
        f = reinterpret_cast<const float *>(m->h_small_dev);
    } else {
        e = cudaMemcpyAsync(m->feats, feats, sizeof(float) * (size_t)M * kIn, cudaMemcpyHostToDevice, s);
    }
    if (M <= kMidRows) {
        std::memcpy(m->h_small + kSmallPids, pids, sizeof(int32_t) * (size_t)M);
        std::memcpy(m->h_small + kSmallOut, tgt, sizeof(float) * (size_t)M);
        p = reinterpret_cast<const int32_t *>(m->h_small_dev + kSmallPids);
        t = reinterpret_cast<const float *>(m->h_small_dev + kSmallOut);
    } else {
        if (e == cudaSuccess) e = cudaMemcpyAsync(m->pids, pids, sizeof(int32_t) * (size_t)M, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(m->tgt, tgt, sizeof(float) * (size_t)M, cudaMemcpyHostToDevice, s);
    }
    if (e != cudaSuccess) return settled(m, s, cuda_fail(e, "mlp upload"));
    gradient_step(m, f, p, t, M, s);
    e = cudaGetLastError();
    // the status first: the copy to the caller's memory holds the host until it is done
    if (e == cudaSuccess) e = copy_status(m, s);
    if (e == cudaSuccess && grads_host)
        e = cudaMemcpyAsync(grads_host, m->grads, sizeof(float) * (size_t)m->n_params, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return settled(m, s, cuda_fail(e, "wk_mlp_gradients"));
    if ((st = check_status(m, s, "wk_mlp_gradients", true))) return st;
    if (loss_host) *loss_host = m->h_loss[0];
    return WK_OK;
}

// Mini-batch training: `epochs` passes over n samples in batches of `batch`
// (sample order shuffled with `seed`), Adam with learning rate lr.  Returns
// the mean loss of the last epoch.
//
// The samples are uploaded once and stay on the device; every step gathers
// its batch there by the epoch's order.  A step of a full batch is the same
// launch sequence every time (its batch index and Adam bias corrections are
// read from device memory), so the second full batch is captured as a CUDA
// graph and every later one replays it: one launch instead of fifteen.
// A shorter last batch runs as plain launches.  The host reads the device
// once per epoch (the loss sum and the GEMM status).
extern "C" int wk_mlp_train(wk_mlp *m, const float *feats, const int32_t *pids, const float *tgt, int64_t n,
                            int32_t epochs, int32_t batch, float lr, uint64_t seed, float *last_loss) {
    if (!m || !feats || !pids || !tgt || n < 1 || epochs < 1 || batch < 1 || batch > m->cap_m)
        return set_error(WK_EINVAL, "wk_mlp_train: bad arguments");
    cudaError_t e = cudaSetDevice(m->ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    cudaStream_t s = m->ctx->stream;
    const int64_t nb = (n + batch - 1) / batch, nfull = n / batch;
    const int tail = (int)(n - nfull * batch);
    DevBuf d_feats, d_pids, d_tgt, d_order;
    int st;
    if ((st = d_feats.reserve(sizeof(float) * (size_t)n * kIn)) || (st = d_pids.reserve(sizeof(int32_t) * (size_t)n)) ||
        (st = d_tgt.reserve(sizeof(float) * (size_t)n)) || (st = d_order.reserve(sizeof(int64_t) * (size_t)n)))
        return st;
    if (nb > m->cbias_cap) {
        cudaFree(m->cbias);
        m->cbias = nullptr;
        m->cbias_cap = 0;
        if ((e = cudaMalloc(&m->cbias, sizeof(float2) * (size_t)nb)) != cudaSuccess) {
            cudaGetLastError();
            return set_error(WK_ENOMEM, "wk_mlp_train: bias-correction table");
        }
        m->cbias_cap = nb;
    }
    if ((e = cudaMemcpyAsync(d_feats.ptr, feats, sizeof(float) * (size_t)n * kIn, cudaMemcpyHostToDevice, s)) ||
        (e = cudaMemcpyAsync(d_pids.ptr, pids, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, s)) ||
        (e = cudaMemcpyAsync(d_tgt.ptr, tgt, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, s)))
        return cuda_fail(e, "wk_mlp_train upload");
    std::vector<int64_t> order((size_t)n);
    for (int64_t i = 0; i < n; ++i) order[(size_t)i] = i;
    std::vector<float2> cb((size_t)nb);
    std::mt19937_64 rng(seed);
    float *h_loss = nullptr;
    if (cudaHostAlloc((void **)&h_loss, 8, 0) != cudaSuccess) return set_error(WK_ENOMEM, "wk_mlp_train: pinned");
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int64_t graph_kernels = 0;
    auto one_step = [&](int M) {
        gather_batch_kernel<<<nblk((int64_t)M * kIn), 256, 0, s>>>(d_feats.as<float>(), d_pids.as<int32_t>(),
                                                                   d_tgt.as<float>(), d_order.as<int64_t>(), m->bidx,
                                                                   batch, M, m->feats, m->pids, m->tgt);
        gradient_step(m, m->feats, m->pids, m->tgt, M, s);
        update(m, lr, s);
        bump_kernel<<<1, 1, 0, s>>>(m->bidx);
        m->kernels += 2;   // gather, bump
    };
    auto finish = [&](int rc) {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        cudaStreamSynchronize(s);   // the pinned loss and the device samples may still be in use
        cudaFreeHost(h_loss);
        m->ctx->launches += m->kernels;
        m->kernels = 0;
        return rc;
    };
    double ep_loss = 0.0;
    for (int ep = 0; ep < epochs; ++ep) {
        std::shuffle(order.begin(), order.end(), rng);
        // Adam step t = step + k + 1 for batch k of this epoch
        for (int64_t k = 0; k < nb; ++k) {
            const float t = (float)(m->step + k + 1);
            cb[(size_t)k] = make_float2(1.f - std::pow(kB1, t), 1.f - std::pow(kB2, t));
        }
        if ((e = cudaMemcpyAsync(d_order.ptr, order.data(), sizeof(int64_t) * (size_t)n, cudaMemcpyHostToDevice, s)) ||
            (e = cudaMemcpyAsync(m->cbias, cb.data(), sizeof(float2) * (size_t)nb, cudaMemcpyHostToDevice, s)) ||
            (e = cudaMemsetAsync(m->bidx, 0, sizeof(int), s)) || (e = cudaMemsetAsync(m->loss + 1, 0, sizeof(float), s)))
            return finish(cuda_fail(e, "wk_mlp_train epoch"));
        for (int64_t k = 0; k < nfull; ++k) {
            if (exec) {
                if ((e = cudaGraphLaunch(exec, s)) != cudaSuccess) return finish(cuda_fail(e, "wk_mlp_train replay"));
                m->kernels += graph_kernels;
            } else if (k == 0 && ep == 0) {
                one_step(batch);
            } else {
                const int64_t k0 = m->kernels;
                if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
                    return finish(cuda_fail(e, "wk_mlp_train capture"));
                one_step(batch);
                e = cudaStreamEndCapture(s, &graph);
                graph_kernels = m->kernels - k0;
                m->kernels = k0;
                if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
                if (e != cudaSuccess) return finish(cuda_fail(e, "wk_mlp_train graph"));
                if ((e = cudaGraphLaunch(exec, s)) != cudaSuccess) return finish(cuda_fail(e, "wk_mlp_train replay"));
                m->kernels += graph_kernels;
            }
        }
        if (tail) one_step(tail);
        m->step += nb;
        if ((e = cudaMemcpyAsync(h_loss, m->loss, 8, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
            return finish(cuda_fail(e, "wk_mlp_train loss"));
        if ((st = check_status(m, s, "wk_mlp_train"))) return finish(st);
        ep_loss = (double)h_loss[1] / (double)nb;
    }
    if (last_loss) *last_loss = (float)ep_loss;
    return finish(WK_OK);
}

// Predictions (log(1 + rows)) for n samples: a small call through the pinned
// block, up to kMidRows samples with their features copied, more in chunks of two tiles per SM, whose copies in run on
// their own stream while the chunk before is computed.
extern "C" int wk_mlp_predict(wk_mlp *m, const float *feats, const int32_t *pids, int64_t n, float *out) {
    if (!m || (n > 0 && (!feats || !pids || !out)) || n < 0) return set_error(WK_EINVAL, "wk_mlp_predict");
    cudaSetDevice(m->ctx->device);
    cudaStream_t s = m->ctx->stream;
    int st = WK_OK;
    if (n > 0 && n <= kMidRows) {
        const float *f = reinterpret_cast<const float *>(m->h_small_dev);
        if (n <= kSmallRows) {
            std::memcpy(m->h_small, feats, sizeof(float) * (size_t)n * kIn);
        } else {
            if ((st = m->stage[0].reserve(sizeof(float) * (size_t)n * kIn))) return st;
            const cudaError_t e = cudaMemcpyAsync(m->stage[0].ptr, feats, sizeof(float) * (size_t)n * kIn, cudaMemcpyHostToDevice, s);
            if (e != cudaSuccess) return cuda_fail(e, "wk_mlp_predict");
            f = m->stage[0].as<float>();
        }
        std::memcpy(m->h_small + kSmallPids, pids, sizeof(int32_t) * (size_t)n);
        predict(m, f, reinterpret_cast<const int32_t *>(m->h_small_dev + kSmallPids), n,
                reinterpret_cast<float *>(m->h_small_dev + kSmallOut), s);
        if ((st = check_status(m, s, "wk_mlp_predict"))) return st;
        std::memcpy(out, m->h_small + kSmallOut, sizeof(float) * (size_t)n);
    } else if (n > 0) {
        const int64_t chunk = std::min<int64_t>(n, 2 * (int64_t)mlpf::kTile * m->sms);
        for (int i = 0; i < (n > chunk ? 2 : 1); ++i)
            if ((st = m->stage[i].reserve(sizeof(float) * (size_t)chunk * kIn))) return st;
        if ((st = m->pred.reserve(2 * sizeof(float) * (size_t)n))) return st;   // the outputs, then the ids
        cudaStream_t in = n > chunk ? m->copy : s;
        int32_t *p = m->pred.as<int32_t>() + n;
        cudaError_t e = cudaMemcpyAsync(p, pids, sizeof(int32_t) * (size_t)n, cudaMemcpyHostToDevice, in);
        for (int64_t b0 = 0, k = 0; b0 < n && e == cudaSuccess; b0 += chunk, ++k) {
            const int64_t rows = std::min<int64_t>(chunk, n - b0);
            const int b = (int)(k & 1);
            float *f = m->stage[b].as<float>();
            if (k >= 2) e = cudaStreamWaitEvent(in, m->used[b], 0);   // the chunk two before has read the buffer
            if (e == cudaSuccess) e = cudaMemcpyAsync(f, feats + b0 * kIn, sizeof(float) * (size_t)rows * kIn, cudaMemcpyHostToDevice, in);
            if (in != s) {
                if (e == cudaSuccess) e = cudaEventRecord(m->copied[b], in);
                if (e == cudaSuccess) e = cudaStreamWaitEvent(s, m->copied[b], 0);
            }
            if (e != cudaSuccess) break;
            predict(m, f, p + b0, rows, m->pred.as<float>() + b0, s);
            if (in != s) e = cudaEventRecord(m->used[b], s);
        }
        // the status first: the copy to the caller's memory holds the host until it is done
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e == cudaSuccess) e = copy_status(m, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(out, m->pred.ptr, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) return settled(m, s, cuda_fail(e, "wk_mlp_predict"));
        if ((st = check_status(m, s, "wk_mlp_predict", true))) return st;
    }
    m->ctx->launches += m->kernels;
    m->kernels = 0;
    return WK_OK;
}

// Held-out check of the model: q-error of each sample is exp(|predicted -
// true|) in log(1 + rows) (the ratio of the larger to the smaller of rows + 1;
// a negative prediction counts as 0, as the planners clamp it).  The model is
// trusted while the 95th percentile stays within qerror_bound; an untrusted
// model makes the learned planners return the statistics plan.
extern "C" int wk_mlp_validate(wk_mlp *m, const float *feats, const int32_t *pids, const float *target, int64_t n,
                               double qerror_bound, double *p95_qerror, int32_t *trusted) {
    if (!m || n < 1 || !feats || !pids || !target || !(qerror_bound >= 1.0))
        return set_error(WK_EINVAL, "wk_mlp_validate: bad arguments");
    std::vector<float> pred((size_t)n);
    int st = wk_mlp_predict(m, feats, pids, n, pred.data());
    if (st) return st;
    std::vector<double> q((size_t)n);
    for (int64_t i = 0; i < n; ++i)
        q[(size_t)i] = std::exp(std::fabs((double)std::max(0.f, pred[(size_t)i]) - (double)target[(size_t)i]));
    const size_t k = (size_t)std::ceil(0.95 * (double)n) - 1;
    std::nth_element(q.begin(), q.begin() + (ptrdiff_t)k, q.end());
    const double p95 = q[k];
    m->trusted = p95 <= qerror_bound ? 1 : 0;
    if (p95_qerror) *p95_qerror = p95;
    if (trusted) *trusted = m->trusted;
    return WK_OK;
}

extern "C" int wk_mlp_is_trusted(wk_mlp *m) { return m ? m->trusted : 0; }
