// The per-pattern ops and the step dispatcher.
//
//   wk_known_to_unknown  <-> RCache::known_to_unknown  (core/rcache.hpp:232-414)
//   wk_known_to_known    <-> RCache::known_to_known    (core/rcache.hpp:417-612)
//   wk_known_to_const    <-> RCache::known_to_const    (core/rcache.hpp:614-809)
//   wk_index_to_unknown  <-> RCache::index_to_unknown  (core/rcache.hpp:811-962)
//   wk_const_to_unknown  <-> Engine::const_to_unknown  (core/engine.hpp:96-122)
//   wk_execute           <-> GPU_Engine::execute_one_step / execute_request
//                            (core/gpu_engine.hpp:395-526)
//
// Differences from the reference, none of which changes a result row:
// each op needs at most one host synchronisation (to size the k2u output);
// k2k/k2c need none before their last kernel; a missing key yields an empty
// adjacency instead of the reference GPU's out-of-bounds read of slot -1
// (core/gpu_hash.cu:276-277); tables are not limited to 20 columns or to
// GPU_MAX_ELEM elements; errors are returned, never asserted.
#include "wk_runtime.h"

#include <algorithm>
#include <cstring>

using namespace wk;

namespace {

enum { KIND_K2U = 0, KIND_K2K = 1, KIND_K2C = 2, KIND_I2U = 3, KIND_C2U = 4 };

inline bool is_tpid(int64_t id) { return id > 1 && id < WK_VID_BASE; }   // core/gstore.hpp:111

int check_ctx(wk_ctx *ctx, wk_history *h, const char *what) {
    if (!ctx || !h) return set_error(WK_EINVAL, "%s: null argument", what);
    if (!ctx->store) return set_error(WK_ENOSTORE, "%s: no store built", what);
    if (ctx->device < 0) return set_error(WK_EDEVICE, "%s: host-only context", what);
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    return WK_OK;
}

int check_pid(wk_ctx *ctx, int64_t pid, int32_t dir, const char *what) {
    if (pid < 1 || pid > ctx->store->hs->num_ids)
        return set_error(WK_EINVAL, "%s: predicate %lld outside [1,%d]", what, (long long)pid, ctx->store->hs->num_ids);
    if (dir != WK_DIR_IN && dir != WK_DIR_OUT) return set_error(WK_EINVAL, "%s: direction %d", what, dir);
    return WK_OK;
}

// ---- per-op timing: a begin/end CUDA event pair around every kernel on the
// op stream, so host gaps between kernels are never counted
struct OpClock {
    wk_ctx *ctx;
    explicit OpClock(wk_ctx *c) : ctx(c) {
        ctx->tn = 0;
        ctx->tmain.clear();
        ctx->last = wk_op_stats{};
    }
    int record() {
        if (!ctx->timing) return WK_OK;
        if ((int)ctx->tev.size() <= ctx->tn) {
            cudaEvent_t ev;
            cudaError_t e = cudaEventCreate(&ev);
            if (e != cudaSuccess) return cuda_fail(e, "timing event");
            ctx->tev.push_back(ev);
        }
        cudaError_t e = cudaEventRecord(ctx->tev[(size_t)ctx->tn++], ctx->stream);
        return e == cudaSuccess ? WK_OK : cuda_fail(e, "timing record");
    }
    int begin() { return record(); }
    int end(bool is_main) {   // after the kernel's launch
        ++ctx->launches;
        ++ctx->last.kernels;
        if (!ctx->timing) return WK_OK;
        if (is_main) ctx->tmain.push_back(ctx->tn - 1);   // begin event of this pair
        return record();
    }
    // call after the stream has been synchronised
    void finish() {
        if (!ctx->timing) return;
        double tot = 0.0, main = 0.0;
        size_t m = 0;   // tmain is ascending
        for (int i = 0; i + 1 < ctx->tn; i += 2) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ctx->tev[(size_t)i], ctx->tev[(size_t)i + 1]);
            tot += ms;
            if (m < ctx->tmain.size() && ctx->tmain[m] == i) {
                main += ms;
                ++m;
            }
        }
        ctx->last.ms = tot;
        ctx->last.ms_main = main;
        float span = 0.f;
        if (ctx->tn >= 2) cudaEventElapsedTime(&span, ctx->tev[0], ctx->tev[(size_t)ctx->tn - 1]);
        ctx->last.span_ms = span;
    }
};

int launch_check(const char *what) {
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? WK_OK : cuda_fail(e, what);
}

// output buffer: the ping-pong partner of the input
wk::DevBuf &out_buf(wk_ctx *ctx, const wk_history *h) {
    return (h->data == ctx->hbuf[0].ptr) ? ctx->hbuf[1] : ctx->hbuf[0];
}

int ensure_seg(wk_ctx *ctx, int id, PredView *pv) {
    DeviceStore &ds = *ctx->store;
    if (ds.pool) {
        std::vector<int> prot = ctx->protect;
        prot.push_back(id);
        int st = ds.ensure(id, prot, ctx->query_rest, ctx->stream, ctx->stream, nullptr);
        if (st) return st;
    }
    *pv = ds.views[(size_t)id];
    return WK_OK;
}

// Wait until the publish kernel of sequence number seq has written its copy
// into ctx->h_gs.  The wait ends with the stream's work: the stream is polled
// every 4096 reads of the word (a few microseconds; no clock is read, as a
// clock read can enter the kernel and cost the thread its core), and a stream
// that has finished (or failed) without the number there is an error.
int wait_published(wk_ctx *ctx, unsigned long long seq) {
    for (unsigned int i = 1;; ++i) {
        if (__atomic_load_n(ctx->h_gs, __ATOMIC_ACQUIRE) == seq) return WK_OK;
        if ((i & 4095u) != 0u) continue;
        const cudaError_t e = cudaStreamQuery(ctx->stream);
        if (e == cudaErrorNotReady) continue;
        if (e != cudaSuccess) return cuda_fail(e, "op sync");
        if (__atomic_load_n(ctx->h_gs, __ATOMIC_ACQUIRE) == seq) return WK_OK;
        return set_error(WK_EDEVICE, "op finished without publishing its totals");
    }
}

int fail_corrupt() {
    return set_error(WK_EDEVICE, "probe found an overflow chain longer than the segment's overflow area (corrupt store)");
}

}  // namespace

namespace {
// The k2u sums buffers for ops of up to `groups` groups: zero when allocated
// (both), then each count kernel clears the buffer it does not add into.
int reserve_gsum(wk_ctx *ctx, int64_t groups) {
    if (groups <= ctx->gs_groups) return WK_OK;
    const int64_t want = std::max(groups, ctx->gs_groups + ctx->gs_groups / 2);
    const size_t buf_bytes = 16 + (size_t)want * 16;
    ctx->gs_groups = 0;   // until both are there: a failed reservation has given the old ones back
    int st = ctx->gsum.reserve(2 * buf_bytes);
    if (st) return st;
    cudaError_t e = cudaMemsetAsync(ctx->gsum.ptr, 0, ctx->gsum.cap, ctx->stream);
    if (e != cudaSuccess) return cuda_fail(e, "k2u: clear group sums");
    // every publish into the old copy has been waited for
    if (ctx->h_gs) cudaFreeHost(ctx->h_gs);
    ctx->h_gs = ctx->h_gs_dev = nullptr;
    ctx->h_gs_bytes = 0;
    e = cudaHostAlloc((void **)&ctx->h_gs, 16 + buf_bytes, cudaHostAllocMapped);
    if (e == cudaSuccess) {
        std::memset(ctx->h_gs, 0, 16 + buf_bytes);   // no sequence number yet
        e = cudaHostGetDevicePointer((void **)&ctx->h_gs_dev, ctx->h_gs, 0);
    }
    if (e != cudaSuccess) {
        if (ctx->h_gs) cudaFreeHost(ctx->h_gs);
        ctx->h_gs = ctx->h_gs_dev = nullptr;
        return cuda_fail(e, "k2u: pinned group sums");
    }
    ctx->h_gs_bytes = 16 + buf_bytes;
    ctx->gs_groups = want;
    ctx->gs_par = 0;
    ctx->gs_used[0] = ctx->gs_used[1] = 0;
    return WK_OK;
}

unsigned long long *gsum_buffer(wk_ctx *ctx, int par) {
    return ctx->gsum.as<unsigned long long>() + (size_t)par * (size_t)(2 + 2 * ctx->gs_groups);
}
}  // namespace

// Slice records kept for an op of nblk blocks: enough for a mean fan-out of 128;
// an op with more slices expands in rounds of that many (33M output rows at
// least).
namespace {
inline int64_t slice_records(int64_t nblk) { return 16 * nblk + 4096; }

// The scratch of a k2u op of nblk blocks, in the context's `deg` buffer: per row
// pos, rel and row (Entries), per block its sum, the slice records, the head.  In
// one buffer, and with few records for a small op, because a new context's first
// step pays for each allocation, some 60 us where it takes a new piece of device
// memory.
struct K2uScratch {
    dev::Entries en;
    unsigned long long *blk_sum;
    dev::SliceRec *recs;
    uint32_t *head;
    static size_t bytes(int64_t nblk) {
        return (size_t)nblk * dev::kRowsPerBlock * 10 + (size_t)(nblk + (nblk & 1)) * 8 +
               (size_t)(slice_records(nblk) + 1) * sizeof(dev::SliceRec);
    }
    K2uScratch(const DevBuf &b, int64_t nblk) {
        const size_t whole = (size_t)nblk * dev::kRowsPerBlock;   // entries come by whole blocks
        unsigned char *p = b.as<unsigned char>();
        en = dev::Entries{reinterpret_cast<uint32_t *>(p), reinterpret_cast<uint32_t *>(p + whole * 4),
                          reinterpret_cast<uint16_t *>(p + whole * 8)};
        blk_sum = reinterpret_cast<unsigned long long *>(p + whole * 10);
        recs = reinterpret_cast<dev::SliceRec *>(blk_sum + nblk + (nblk & 1));
        head = reinterpret_cast<uint32_t *>(recs + slice_records(nblk));
    }
};
}

int wk::reserve_published(wk_ctx *ctx, int64_t words) { return reserve_gsum(ctx, (words + 1) / 2); }

int wk::reserve_op_scratch(wk_ctx *ctx, int64_t rows) {
    if (!ctx || rows < 0) return set_error(WK_EINVAL, "reserve_op_scratch: bad arguments");
    if (ctx->device < 0) return WK_OK;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    const int64_t nblk = (rows + dev::kRowsPerBlock - 1) / dev::kRowsPerBlock + 1;
    int st;
    if ((st = ctx->deg.reserve(K2uScratch::bytes(nblk))) ||
        (st = ctx->mask.reserve((size_t)((rows + 31) / 32) * 4)) ||
        (st = ctx->blk_nz.reserve((size_t)nblk * 4)) ||
        (st = reserve_gsum(ctx, (nblk + (1 << dev::kGroupShift) - 1) >> dev::kGroupShift)))
        return st;
    return WK_OK;
}

namespace {

// An op's device-buffer reservation.  A context given injected allocation
// failures (wk_ctx_inject_alloc_failure) fails its next ones with WK_ENOMEM
// here, as a failed cudaMalloc inside DevBuf::reserve would.
int take(wk_ctx *ctx, DevBuf &b, size_t bytes) {
    if (ctx->inject_alloc_fail.load(std::memory_order_relaxed) > 0 &&
        ctx->inject_alloc_fail.fetch_sub(1, std::memory_order_relaxed) > 0)
        return set_error(WK_ENOMEM, "cudaMalloc: out of memory (injected allocation failure)");
    return b.reserve(bytes);
}

bool alloc_failure_pending(wk_ctx *ctx) { return ctx->inject_alloc_fail.load(std::memory_order_relaxed) > 0; }

// A k2u or filter op over a dense functional direction (wk_fused.cu), at most
// one row out per row in: one launch.  A k2u op writes as it counts, as long as the
// output buffer has room; when the buffer turns out too small it is grown to the
// rows there are and the rows are written by a second launch.  An op whose row
// limit is below its input's rows is counted, held to the limit and only then
// written; so is one whose buffer has room for less than half of the rows to expect,
// as it will have to be grown: those of the direction's share of ids with a
// neighbour, or of the context's last such step if that kept fewer.  The first step of
// a new context on 12M rows that all match, from room for 3.4M, takes 494 us when it
// writes first, 442 so; a step one in ten of whose 8M rows match, with room for 3.4M,
// 77 us when it is counted first, 59 so.
// *done is false when the op has to run as the general kernels instead: more
// columns than the launch takes, a start that is an index key (k2u), or a device
// wait that ran out.
int op_fused(wk_ctx *ctx, wk_history *h, int scol, int ecol, int32_t end_const, uint32_t pid, uint32_t dir, bool filter,
             const PredView &pv, OpClock &clk, bool *done) {
    *done = false;
    const int C = h->col_num;
    const int64_t R = h->size / C;
    const int width = filter ? C : C + 1;
    if (pv.nb[dir] == nullptr || !dev::fused_takes(C, filter)) return WK_OK;
    DevBuf &ob = out_buf(ctx, h);
    const int64_t nblk = (R + dev::kRowsPerBlock - 1) / dev::kRowsPerBlock;
    const int64_t groups = (nblk + (1 << dev::kGroupShift) - 1) >> dev::kGroupShift;
    int st;
    if ((st = filter ? take(ctx, ctx->mask, (size_t)((R + 31) / 32) * 4) : take(ctx, ctx->deg, (size_t)R * 4)) ||
        (st = take(ctx, ctx->blk_nz, (size_t)nblk * 4)) || (st = reserve_gsum(ctx, groups)) ||
        (filter && (st = take(ctx, ob, (size_t)R * C * 4))))
        return st;
    const int64_t room = (int64_t)(ob.cap / ((size_t)width * 4));
    const PredSeg &sg = ctx->store->hs->segs[pid];
    const double share = (double)(dir == WK_DIR_OUT ? sg.subjects : sg.objects) / (double)std::max(sg.dn[dir], 1u);
    const bool count_first = !filter && (R > ctx->row_limit || (double)room < 0.5 * std::min(share, ctx->func_share) * (double)R);
    if ((st = clk.begin())) return st;
    const int par = ctx->gs_par;
    unsigned long long *gs = gsum_buffer(ctx, par);
    dev::FusedOp op;
    if (const int polls = ctx->wait_polls.load(std::memory_order_relaxed); polls >= 0) op.pub_polls = op.write_polls = polls;
    op.part = count_first ? dev::kFusedCount : dev::kFusedAll;
    op.hist = h->data;
    op.R = R;
    op.C = C;
    op.scol = scol;
    op.ecol = ecol;
    op.end_const = end_const;
    op.dir = dir;
    op.filter = filter;
    op.pv = pv;
    op.nbr = ctx->deg.as<int32_t>();
    op.mask = ctx->mask.as<uint32_t>();
    op.blk_nz = ctx->blk_nz.as<unsigned int>();
    op.group_sums = gs + 2;
    op.err = reinterpret_cast<int *>(gs);
    op.written = gs + 1;
    op.clear = gsum_buffer(ctx, par ^ 1);
    op.nclear = 2 + 2 * ctx->gs_used[par ^ 1];
    op.out = ob.as<int32_t>();
    op.max_rows = (unsigned long long)room;
    op.pub = ctx->h_gs_dev;
    op.seq = ++ctx->pub_seq;
    op.sms = ctx->sms;
    cudaError_t le = (cudaError_t)dev::launch_fused(op, ctx->stream);
    if (le != cudaSuccess) return cuda_fail(le, "one-launch op");
    if ((st = launch_check("one-launch op")) || (st = clk.end(!count_first))) return st;
    ctx->gs_par = par ^ 1;
    ctx->gs_used[par ^ 1] = 0;
    ctx->gs_used[par] = groups;
    if ((st = wait_published(ctx, op.seq))) return st;
    const unsigned long long err = ctx->h_gs[2];
    const int64_t R_out = (int64_t)ctx->h_gs[3], extra = (int64_t)ctx->h_gs[4];
    if (err & 1ull)
        return fail_corrupt();
    if ((err & (unsigned long long)dev::kErrWait) || (!filter && extra)) return WK_OK;
    if (!filter && R_out > ctx->row_limit)   // nothing was written
        return set_error(WK_EOVERFLOW, "k2u: %lld output rows exceed the context's row limit %lld", (long long)R_out,
                         (long long)ctx->row_limit);
    if (!filter) ctx->func_share = (double)R_out / (double)R;
    if (!ob.ptr && (st = take(ctx, ob, 16))) return st;
    if (!filter && (R_out > room || (count_first && R_out > 0))) {
        if ((st = take(ctx, ob, (size_t)R_out * width * 4))) return st;
        op.part = dev::kFusedWrite;
        op.out = ob.as<int32_t>();
        op.max_rows = (unsigned long long)R_out;
        if ((st = clk.begin())) return st;
        if ((le = (cudaError_t)dev::launch_fused(op, ctx->stream)) != cudaSuccess) return cuda_fail(le, "functional write");
        if ((st = launch_check("functional write")) || (st = clk.end(true))) return st;
    }
    ctx->last.rows_out = R_out;
    ctx->last.alg_bytes = filter ? 4 * R * C + 16 * R + 4 * extra + 4 * R_out * C
                                 : 4 * R * C + 16 * R + 4 * R_out + 4 * R_out * (C + 1);
    if (ctx->timing) {
        cudaError_t e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) return cuda_fail(e, "one-launch op sync");
    }
    clk.finish();
    h->data = ob.as<int32_t>();
    h->size = R_out * width;
    h->col_num = width;
    h->step++;
    *done = true;
    return WK_OK;
}

// two-pass k2u (count -> host adds up the group sums -> expand)
int op_k2u(wk_ctx *ctx, wk_history *h, int scol, uint32_t pid, uint32_t dir) {
    const int C = h->col_num;
    const int64_t R = h->size / C;
    OpClock clk(ctx);
    ctx->last.kind = KIND_K2U;
    ctx->last.rows_in = R;
    ctx->last.cols_in = C;
    PredView pv;
    int st = ensure_seg(ctx, (int)pid, &pv);
    if (st) return st;
    DevBuf &ob = out_buf(ctx, h);
    if (R == 0) {
        if ((st = take(ctx, ob, 16))) return st;
        h->data = ob.as<int32_t>();
        h->size = 0;
        h->col_num = C + 1;
        h->step++;
        return WK_OK;
    }
    bool done = false;
    if ((st = op_fused(ctx, h, scol, -1, 0, pid, dir, false, pv, clk, &done)) || done) return st;
    const int64_t nblk = (R + dev::kRowsPerBlock - 1) / dev::kRowsPerBlock;
    const int64_t groups = (nblk + (1 << dev::kGroupShift) - 1) >> dev::kGroupShift;
    if ((st = take(ctx, ctx->deg, K2uScratch::bytes(nblk))) || (st = reserve_gsum(ctx, groups))) return st;
    const K2uScratch sc(ctx->deg, nblk);
    const dev::Entries &en = sc.en;
    dev::SliceRec *recs = sc.recs;
    uint32_t *head = sc.head;
    dev::SlicePlan plan{sc.blk_sum, nullptr, nblk, recs, 0ull, (unsigned long long)slice_records(nblk), nullptr, nullptr,
                        0ull, 0ull};
    // a hashed functional direction (at most one neighbour per vertex) expands as a
    // compaction; if a row hits an index list (vertex 0) the op reruns unspecialised
    bool func = pv.func[dir] != 0u && pv.nb[dir] == nullptr && C + 1 <= 8;
    // The output buffer an earlier op grew often holds this op's rows too, which
    // the device can tell as well as the host: the expansion then goes in behind
    // the publish kernel, and the GPU does not wait while the host adds up the
    // totals and launches it.  Back to back, 800k -> 1.66M rows of 11 columns took
    // 47.0 us a step so, 41.4 us this way, 120k -> 12M rows of 4 columns 43.1 and
    // 41.3.  The device runs it only if the op is in order and its rows and slices
    // fit; else the host sees to it as for an op without a buffer.  The launch has
    // a CTA for each slice that the buffer has room for, up to four times what the
    // direction's mean list gives and at least half a wave: a CTA that finds no
    // slice is gone in half a microsecond, but a buffer that a large step has grown
    // has room for thousands (the steps of a query of 61M rows: 761 us with up to
    // two waves of them, 751 so).
    unsigned int ncta = 0;
    bool ahead_wide = false;
    if (!func && !ctx->timing && !alloc_failure_pending(ctx)) {
        const unsigned long long b = (unsigned long long)nblk, wave = 8ull * (unsigned long long)std::max(ctx->sms, 1);
        plan.max_rows = std::min<unsigned long long>(ob.cap / ((size_t)(C + 1) * 4),
                                                     (unsigned long long)std::max<int64_t>(ctx->row_limit, 0));
        const PredSeg &sg = ctx->store->hs->segs[pid];
        const int64_t keys = std::max<int64_t>(dir == WK_DIR_OUT ? sg.subjects : sg.objects, 1);
        const double expect = (double)R * (double)std::max<int64_t>(sg.triples, 0) / (double)keys / dev::kSliceRows;
        const unsigned long long room = plan.max_rows / dev::kSliceRows;
        const unsigned long long likely = std::min(room, (unsigned long long)std::min(expect, 1e9));
        plan.max_slices = std::min(plan.cap, b + std::min(room, std::max(wave / 2, 4 * likely)));
        ahead_wide = b < wave && likely >= wave;
        if (plan.max_rows) ncta = (unsigned int)plan.max_slices;
    }
    int errf = 0;
    unsigned long long *gs = nullptr;
    for (;;) {
        const int par = ctx->gs_par;
        gs = gsum_buffer(ctx, par);
        if ((st = clk.begin())) return st;
        // the op's error flags and group sums come to the host through pinned
        // memory (the publish kernel behind the count, which also writes the
        // expansion's slice records); the host adds up the totals
        const dev::Publish pub{gs, ctx->h_gs_dev, 2 + 2 * groups, ++ctx->pub_seq};
        dev::launch_k2u_count(h->data, R, C, scol, dir, pv, en, sc.blk_sum, gs + 2,
                              reinterpret_cast<int *>(gs), func, gsum_buffer(ctx, par ^ 1),
                              2 + 2 * ctx->gs_used[par ^ 1], ctx->sms, ctx->stream);
        if ((st = launch_check("k2u count")) || (st = clk.end(false))) return st;
        // outside the count's timing events: the op's device span counts it,
        // the count kernel's time does not
        plan.group_sums = gs + 2;
        if (ncta) plan.head = head;
        plan.err = reinterpret_cast<int *>(gs);
        dev::launch_publish(pub, plan, ctx->stream);
        if ((st = launch_check("k2u publish"))) return st;
        ++ctx->launches;
        ++ctx->last.kernels;
        if (ncta) {
            dev::launch_k2u_expand(h->data, C, pv.edges, en, recs, ncta, head, ahead_wide, ob.as<int32_t>(), ctx->stream);
            if ((st = launch_check("k2u expand"))) return st;
            ++ctx->launches;
        }
        ctx->gs_par = par ^ 1;
        ctx->gs_used[par ^ 1] = 0;
        ctx->gs_used[par] = groups;
        if ((st = wait_published(ctx, pub.seq))) return st;
        errf = (int)(ctx->h_gs[2] & 0xffffffffull);
        if (!(func && (errf & 8))) break;
        func = false;   // the next count adds into the other, cleared buffer
    }
    if (errf & 1)
        return fail_corrupt();
    if (errf & 2) return set_error(WK_EOVERFLOW, "k2u: 1024 consecutive input rows expand to 2^31 rows or more");
    unsigned long long rows_out = 0ull, slices = 0ull;
    for (int64_t g = 0; g < groups; ++g) {
        rows_out += ctx->h_gs[4 + 2 * g];
        slices += ctx->h_gs[5 + 2 * g];
    }
    const int64_t R_out = (int64_t)rows_out;
    if (R_out > ctx->row_limit)
        return set_error(WK_EOVERFLOW, "k2u: %lld output rows exceed the context's row limit %lld", (long long)R_out,
                         (long long)ctx->row_limit);
    ctx->last.rows_out = R_out;
    ctx->last.alg_bytes = 4 * R * C + 16 * R + 4 * R_out + 4 * R_out * (C + 1);
    if (R_out == 0) {
        if ((st = take(ctx, ob, 16))) return st;
    } else if (ncta && slices <= plan.max_slices && rows_out <= plan.max_rows) {
        ++ctx->last.kernels;   // the expansion behind the publish kernel did it
    } else {
        if ((st = take(ctx, ob, (size_t)R_out * (C + 1) * 4))) return st;
        if ((st = clk.begin())) return st;
        const bool wide = dev::wide_slices(slices, rows_out, ctx->sms);
        for (unsigned long long s0 = 0ull;;) {
            const unsigned int n = (unsigned int)std::min<unsigned long long>(slices - s0, plan.cap);
            if (func)
                dev::launch_k2u_expand_func(h->data, R, C, ctx->deg.as<int32_t>(), recs, n, ob.as<int32_t>(), ctx->stream);
            else
                dev::launch_k2u_expand(h->data, C, pv.edges, en, recs, n, nullptr, wide, ob.as<int32_t>(), ctx->stream);
            if ((s0 += n) >= slices) break;
            plan.head = nullptr;
            plan.first = s0;   // the next records, behind the expansion that reads these
            dev::launch_publish(dev::Publish{nullptr, nullptr, 0, 0ull}, plan, ctx->stream);
            ctx->launches += 2;
            ctx->last.kernels += 2;
        }
        if ((st = launch_check("k2u expand")) || (st = clk.end(true))) return st;
        if (ctx->timing) {
            cudaError_t e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) return cuda_fail(e, "k2u sync");
        }
    }
    clk.finish();
    h->data = ob.as<int32_t>();
    h->size = R_out * (C + 1);
    h->col_num = C + 1;
    h->step++;
    return WK_OK;
}

// two-pass k2k / k2c (probe + membership -> filtered copy); the output is
// sized by the input, so the host reads the totals only at the end
int op_filter(wk_ctx *ctx, wk_history *h, int scol, int ecol, int32_t end_const, uint32_t pid, uint32_t dir) {
    const int C = h->col_num;
    const int64_t R = h->size / C;
    OpClock clk(ctx);
    ctx->last.kind = ecol >= 0 ? KIND_K2K : KIND_K2C;
    ctx->last.rows_in = R;
    ctx->last.cols_in = C;
    PredView pv;
    int st = ensure_seg(ctx, (int)pid, &pv);
    if (st) return st;
    DevBuf &ob = out_buf(ctx, h);
    if (R == 0) {
        if ((st = take(ctx, ob, 16))) return st;
        h->data = ob.as<int32_t>();
        h->size = 0;
        h->step++;
        return WK_OK;
    }
    bool done = false;
    if ((st = op_fused(ctx, h, scol, ecol, end_const, pid, dir, true, pv, clk, &done)) || done) return st;
    const int64_t nblk = (R + dev::kRowsPerBlock - 1) / dev::kRowsPerBlock;
    const int64_t groups = (nblk + (1 << dev::kGroupShift) - 1) >> dev::kGroupShift;
    if ((st = take(ctx, ctx->mask, (size_t)((R + 31) / 32) * 4)) || (st = take(ctx, ctx->blk_nz, (size_t)nblk * 4)) ||
        (st = reserve_gsum(ctx, groups)) || (st = take(ctx, ob, (size_t)R * C * 4)))
        return st;
    // as in a k2u op: the error word and the group sums in one of two buffers,
    // the other cleared for the next op, and the sums to the host through pinned
    // memory, here behind the copy of the kept rows: the op has finished with its
    // input when it returns
    const int par = ctx->gs_par;
    unsigned long long *gs = gsum_buffer(ctx, par);
    if ((st = clk.begin())) return st;
    dev::launch_filter_probe(h->data, R, C, scol, ecol, end_const, dir, pv, ctx->mask.as<uint32_t>(),
                             ctx->blk_nz.as<unsigned int>(), gs + 2, gsum_buffer(ctx, par ^ 1),
                             2 + 2 * ctx->gs_used[par ^ 1], reinterpret_cast<int *>(gs), ctx->stream);
    if ((st = launch_check("filter probe"))) return st;
    ctx->gs_par = par ^ 1;
    ctx->gs_used[par ^ 1] = 0;
    ctx->gs_used[par] = groups;
    if ((st = clk.end(true)) || (st = clk.begin())) return st;
    dev::launch_filter_write(h->data, R, C, ctx->mask.as<uint32_t>(), ctx->blk_nz.as<unsigned int>(), gs + 2,
                             ob.as<int32_t>(), ctx->sms, ctx->stream);
    if ((st = launch_check("filter write")) || (st = clk.end(false))) return st;
    const dev::Publish pub{gs, ctx->h_gs_dev, 2 + 2 * groups, ++ctx->pub_seq};
    dev::launch_publish(pub, dev::SlicePlan{}, ctx->stream);
    if ((st = launch_check("filter publish"))) return st;
    ++ctx->launches;
    ++ctx->last.kernels;
    if ((st = wait_published(ctx, pub.seq))) return st;
    if (ctx->h_gs[2] & 0xffffffffull) return fail_corrupt();
    int64_t nz = 0, E = 0;
    for (int64_t g = 0; g < groups; ++g) {
        nz += (int64_t)ctx->h_gs[4 + 2 * g];
        E += (int64_t)ctx->h_gs[5 + 2 * g];
    }
    clk.finish();
    ctx->last.rows_out = nz;
    ctx->last.alg_bytes = 4 * R * C + 16 * R + 4 * E + 4 * nz * C;
    h->data = ob.as<int32_t>();
    h->size = nz * C;
    h->step++;
    return WK_OK;
}

// one adjacency list -> one-column table (index or constant start)
int op_list(wk_ctx *ctx, wk_history *h, uint64_t vid, uint32_t pid, uint32_t dir, int kind) {
    OpClock clk(ctx);
    ctx->last.kind = kind;
    ctx->last.rows_in = 1;
    const HostStore &hs = *ctx->store->hs;
    const int32_t *e = nullptr;
    const uint64_t deg = hs.lookup(vid, pid, dir, &e);
    DevBuf &ob = out_buf(ctx, h);
    int st;
    if ((st = take(ctx, ob, (size_t)deg * 4 + 16))) return st;
    if (deg) {
        PredView pv;
        if ((st = ensure_seg(ctx, (int)pid, &pv))) return st;
        const uint64_t off = (uint64_t)(e - (hs.edges + hs.segs[pid].edge_off));
        if ((st = clk.begin())) return st;
        dev::launch_copy_list(pv.edges + off, (int64_t)deg, ob.as<int32_t>(), ctx->stream);
        if ((st = launch_check("list copy")) || (st = clk.end(true))) return st;
        if (ctx->timing) {
            cudaError_t ce = cudaStreamSynchronize(ctx->stream);
            if (ce != cudaSuccess) return cuda_fail(ce, "list sync");
        }
    }
    clk.finish();
    ctx->last.rows_out = (int64_t)deg;
    ctx->last.alg_bytes = 16 + 8 * (int64_t)deg;
    h->data = ob.as<int32_t>();
    h->size = (int64_t)deg;
    h->col_num = 1;
    h->step++;
    return WK_OK;
}

int known_col(const wk_history *h, int64_t v, const char *what, int *col) {
    if (v >= 0 || -v > h->col_num)
        return set_error(WK_EINVAL, "%s: %lld is not a bound variable (col_num %d)", what, (long long)v, h->col_num);
    *col = (int)(-v - 1);
    return WK_OK;
}

int check_table(const wk_history *h, const char *what) {
    if (h->col_num <= 0 || h->size < 0 || h->size % h->col_num != 0 || (h->size > 0 && !h->data))
        return set_error(WK_EINVAL, "%s: malformed history (size %lld, col_num %d)", what, (long long)h->size,
                         h->col_num);
    return WK_OK;
}

}  // namespace

extern "C" int wk_known_to_unknown(wk_ctx *ctx, wk_history *h, int64_t start, int32_t direction, int32_t predict) {
    int st, scol;
    if ((st = check_ctx(ctx, h, "known_to_unknown")) || (st = check_table(h, "known_to_unknown")) ||
        (st = check_pid(ctx, predict, direction, "known_to_unknown")) ||
        (st = known_col(h, start, "known_to_unknown start", &scol)))
        return st;
    return op_k2u(ctx, h, scol, (uint32_t)predict, (uint32_t)direction);
}

extern "C" int wk_known_to_known(wk_ctx *ctx, wk_history *h, int64_t start, int32_t direction, int32_t predict,
                                 int64_t end) {
    int st, scol, ecol;
    if ((st = check_ctx(ctx, h, "known_to_known")) || (st = check_table(h, "known_to_known")) ||
        (st = check_pid(ctx, predict, direction, "known_to_known")) ||
        (st = known_col(h, start, "known_to_known start", &scol)) ||
        (st = known_col(h, end, "known_to_known end", &ecol)))
        return st;
    return op_filter(ctx, h, scol, ecol, 0, (uint32_t)predict, (uint32_t)direction);
}

extern "C" int wk_known_to_const(wk_ctx *ctx, wk_history *h, int64_t start, int32_t direction, int32_t predict,
                                 int64_t end) {
    int st, scol;
    if ((st = check_ctx(ctx, h, "known_to_const")) || (st = check_table(h, "known_to_const")) ||
        (st = check_pid(ctx, predict, direction, "known_to_const")) ||
        (st = known_col(h, start, "known_to_const start", &scol)))
        return st;
    if (end < 0 || end > 0x7fffffffll) return set_error(WK_EINVAL, "known_to_const: end %lld is not a constant", (long long)end);
    return op_filter(ctx, h, scol, -1, (int32_t)end, (uint32_t)predict, (uint32_t)direction);
}

extern "C" int wk_index_to_unknown(wk_ctx *ctx, wk_history *h, int32_t index_vertex, int32_t direction) {
    int st;
    if ((st = check_ctx(ctx, h, "index_to_unknown")) || (st = check_pid(ctx, index_vertex, direction, "index_to_unknown")))
        return st;
    if (h->col_num != 0) return set_error(WK_EINVAL, "index_to_unknown: history already has %d columns", h->col_num);
    return op_list(ctx, h, 0, (uint32_t)index_vertex, (uint32_t)direction, KIND_I2U);
}

extern "C" int wk_const_to_unknown(wk_ctx *ctx, wk_history *h, int64_t start, int32_t direction, int32_t predict) {
    int st;
    if ((st = check_ctx(ctx, h, "const_to_unknown")) || (st = check_pid(ctx, predict, direction, "const_to_unknown")))
        return st;
    if (h->col_num != 0) return set_error(WK_EINVAL, "const_to_unknown: history already has %d columns", h->col_num);
    if (start < WK_VID_BASE || start > 0xffffffffll)
        return set_error(WK_EINVAL, "const_to_unknown: start %lld is not a vertex id", (long long)start);
    return op_list(ctx, h, (uint64_t)start, (uint32_t)predict, (uint32_t)direction, KIND_C2U);
}

// GPU_Engine::execute_one_step dispatch (core/gpu_engine.hpp:395-467) with the
// variable typing of request_or_reply::variable_type (core/query.hpp:141-149).
static int vtype(int64_t v, int col_num) {   // 0 known, 1 unknown, 2 const
    if (v >= 0) return 2;
    return (-v > col_num) ? 1 : 0;
}

// Run a request's first steps as a light query (wk_light.cu) when it starts from
// a short list: *done receives the patterns done, the start among them, and h the
// table after them (0: nothing was run).  Not taken: a paged store, which loads
// segments step by step; timing, which times each step; anything the steps' own
// checks would refuse, which is left for them to refuse.
static int execute_light(wk_ctx *ctx, const int64_t *cmd, int32_t n, wk_history *h, int64_t *step_rows, int *done) {
    *done = 0;
    DeviceStore &ds = *ctx->store;
    if (ds.pool || ctx->timing || alloc_failure_pending(ctx) || n < 2 || n > dev::kLightSteps + 1) return WK_OK;
    const auto pid_ok = [&](int64_t pid, int64_t d) {
        return pid >= 1 && pid <= ds.hs->num_ids && (d == WK_DIR_IN || d == WK_DIR_OUT);
    };
    const int64_t start = cmd[0];
    const bool index = is_tpid(start);
    const int64_t lpid = index ? start : cmd[1];
    if (cmd[3] != -1 || start < 0 || start > 0xffffffffll || !pid_ok(lpid, cmd[2]) || (!index && start < WK_VID_BASE)) return WK_OK;
    const int32_t *e = nullptr;
    const uint64_t deg = ds.hs->lookup(index ? 0ull : (uint64_t)start, (uint32_t)lpid, (uint32_t)cmd[2], &e);
    if (deg == 0 || deg > (uint64_t)dev::kLightRows) return WK_OK;
    dev::LightOp op;
    op.n = n - 1;
    op.deg = (int)deg;
    int cols = 1;
    for (int i = 1; i < n; ++i) {
        const int64_t *c = cmd + 4 * i;
        if (!pid_ok(c[1], c[2]) || vtype(c[0], cols) != 0) return WK_OK;
        dev::LightStep &s = op.s[i - 1];
        s.pv = ds.views[(size_t)c[1]];
        s.C = cols;
        s.scol = (int)(-c[0] - 1);
        s.ecol = -1;
        s.end_const = 0;
        s.dir = (uint32_t)c[2];
        const int te = vtype(c[3], cols);
        s.kind = te == 1 ? dev::kLightK2U : dev::kLightFilter;
        if (te == 1) {
            if (-c[3] - 1 != cols) return WK_OK;
            ++cols;
        } else if (te == 0) {
            s.ecol = (int)(-c[3] - 1);
        } else {
            if (c[3] > 0x7fffffffll) return WK_OK;
            s.end_const = (int32_t)c[3];
        }
    }
    int st;
    const size_t bytes = (size_t)dev::kLightRows * (size_t)cols * 4;
    if ((st = take(ctx, ctx->hbuf[0], bytes)) || (st = take(ctx, ctx->hbuf[1], bytes)) ||
        (st = wk::reserve_published(ctx, dev::kLightWords + dev::kLightSteps)))
        return st;
    op.src = ds.views[(size_t)lpid].edges + (e - (ds.hs->edges + ds.hs->segs[lpid].edge_off));
    op.buf[0] = ctx->hbuf[0].as<int32_t>();
    op.buf[1] = ctx->hbuf[1].as<int32_t>();
    op.row_limit = ctx->row_limit;
    op.pub = ctx->h_gs_dev;
    op.seq = ++ctx->pub_seq;
    dev::launch_light(op, ctx->stream);
    if ((st = launch_check("light query"))) return st;
    ++ctx->launches;
    if ((st = wait_published(ctx, op.seq))) return st;
    if (ctx->h_gs[2] & 1ull) return fail_corrupt();
    const int k = (int)ctx->h_gs[3];   // steps behind the start
    h->data = op.buf[k & 1];
    h->col_num = k == 0 ? 1 : op.s[k - 1].C + (op.s[k - 1].kind == dev::kLightK2U ? 1 : 0);
    h->step = k + 1;
    int64_t rows = (int64_t)deg, rows_in = 1;
    if (step_rows) step_rows[0] = rows;
    for (int i = 0; i < k; ++i) {
        rows_in = rows;
        rows = (int64_t)ctx->h_gs[dev::kLightWords + i];
        if (step_rows) step_rows[i + 1] = rows;
    }
    h->size = rows * h->col_num;
    ctx->last = wk_op_stats{};
    ctx->last.rows_in = rows_in;
    ctx->last.rows_out = rows;
    ctx->last.kernels = 1;
    if (k == 0) {
        ctx->last.kind = index ? KIND_I2U : KIND_C2U;
        ctx->last.alg_bytes = 16 + 8 * rows;
    } else {
        const dev::LightStep &s = op.s[k - 1];
        ctx->last.cols_in = s.C;
        ctx->last.kind = s.kind == dev::kLightK2U ? KIND_K2U : (s.ecol >= 0 ? KIND_K2K : KIND_K2C);
        ctx->last.alg_bytes = 4 * rows_in * s.C + 16 * rows_in +
                              (s.kind == dev::kLightK2U ? 4 * rows + 4 * rows * (s.C + 1)
                                                        : 4 * (int64_t)ctx->h_gs[4] + 4 * rows * s.C);
    }
    *done = k + 1;
    return WK_OK;
}

extern "C" int wk_execute(wk_ctx *ctx, const int64_t *cmd, int32_t n, wk_history *h, int64_t *step_rows) {
    if (!ctx || !cmd || !h || n <= 0) return set_error(WK_EINVAL, "wk_execute: bad arguments");
    if (!ctx->store) return set_error(WK_ENOSTORE, "wk_execute: no store");
    if (ctx->device < 0) return set_error(WK_EDEVICE, "wk_execute: host-only context");
    // a light query and a prefetch use the device before any step's op makes it current
    if (const cudaError_t e = cudaSetDevice(ctx->device)) return cuda_fail(e, "cudaSetDevice");
    wk_history_init(h);
    ctx->protect.clear();
    ctx->query_rest.clear();
    ctx->qstats.clear();
    DeviceStore &ds = *ctx->store;
    int first = 0;
    int st = execute_light(ctx, cmd, n, h, step_rows, &first);
    for (int i = first; i < n && st == WK_OK; ++i) {
        const int64_t start = cmd[i * 4], pid = cmd[i * 4 + 1], d = cmd[i * 4 + 2], end = cmd[i * 4 + 3];
        if (ds.pool) {
            // the segments of steps i.. (an index start's segment is its index id)
            ctx->query_rest.clear();
            for (int k = i; k < n; ++k) {
                const int64_t sid = (k == 0 && is_tpid(cmd[0])) ? cmd[0] : cmd[k * 4 + 1];
                if (sid >= 1 && sid <= ds.hs->num_ids) ctx->query_rest.push_back((int)sid);
            }
        }
        if (ds.pool && ctx->cfg.enable_prefetch && i + 1 < n) {
            const int64_t np = cmd[(i + 1) * 4 + 1];
            const int64_t cp = (i == 0 && is_tpid(cmd[0])) ? cmd[0] : pid;
            if (np >= 1 && np <= ds.hs->num_ids && cp >= 1 && cp <= ds.hs->num_ids) {
                std::vector<int> prot{(int)cp, (int)np};
                ds.ensure((int)np, prot, ctx->query_rest, ctx->side, ctx->stream, ctx->use_ready, false);
                ctx->protect = prot;
            }
        }
        if (i == 0 && is_tpid(start)) {
            if (end != -1) return set_error(WK_EINVAL, "wk_execute: index pattern must bind variable -1");
            st = wk_index_to_unknown(ctx, h, (int32_t)start, (int32_t)d);
        } else {
            if (pid < 0) return set_error(WK_EINVAL, "wk_execute: variable predicates are not supported");
            const int ts = vtype(start, h->col_num), te = vtype(end, h->col_num);
            if (ts == 2 && te == 1) {
                if (h->col_num != 0 || end != -1)
                    return set_error(WK_EINVAL, "wk_execute: constant start must be the first pattern and bind -1");
                st = wk_const_to_unknown(ctx, h, start, (int32_t)d, (int32_t)pid);
            } else if (ts == 0 && te == 1) {
                if (-end - 1 != h->col_num)
                    return set_error(WK_EINVAL, "wk_execute: pattern %d binds %lld but the next column is %d", i,
                                     (long long)end, h->col_num);
                st = wk_known_to_unknown(ctx, h, start, (int32_t)d, (int32_t)pid);
            } else if (ts == 0 && te == 0) {
                st = wk_known_to_known(ctx, h, start, (int32_t)d, (int32_t)pid, end);
            } else if (ts == 0 && te == 2) {
                st = wk_known_to_const(ctx, h, start, (int32_t)d, (int32_t)pid, end);
            } else {
                return set_error(WK_EINVAL, "wk_execute: unsupported pattern shape at step %d (start %lld, end %lld)",
                                 i, (long long)start, (long long)end);
            }
        }
        if (st == WK_OK && step_rows) step_rows[i] = h->col_num ? h->size / h->col_num : 0;
        if (st == WK_OK && ctx->timing) ctx->qstats.push_back(ctx->last);
    }
    ctx->protect.clear();
    ctx->query_rest.clear();
    return st;
}

extern "C" int wk_ctx_inject_alloc_failure(wk_ctx *ctx, int32_t n) {
    if (!ctx || n < 0) return set_error(WK_EINVAL, "wk_ctx_inject_alloc_failure: bad arguments");
    ctx->inject_alloc_fail.store(n);
    return WK_OK;
}

extern "C" int wk_ctx_set_wait_polls(wk_ctx *ctx, int32_t n) {
    if (!ctx || n < -1) return set_error(WK_EINVAL, "wk_ctx_set_wait_polls: bad arguments");
    ctx->wait_polls.store(n);
    return WK_OK;
}

extern "C" int wk_set_row_limit(wk_ctx *ctx, int64_t max_rows) {
    if (!ctx || max_rows < 0) return set_error(WK_EINVAL, "wk_set_row_limit: bad arguments");
    ctx->row_limit = max_rows ? max_rows : INT64_MAX;
    return WK_OK;
}
