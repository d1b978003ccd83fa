// Kernel launchers (defined in wk_kernels.cu, called by the host runtime).
#pragma once

#include <cuda_runtime.h>

#include "wk_internal.h"

namespace wk {
namespace dev {

constexpr int kRowsPerBlock = 1024;   // input rows per CTA of every op kernel
constexpr int kThreads = 256;

constexpr int kSliceRows = 8192;      // k2u output rows per expansion CTA (a multiple of 4)
constexpr int kGroupShift = 8;        // input blocks per k2u group sum: 256

// What the k2u count kernel leaves of each block's rows with a list (its
// entries), from the block's first row on: the entry's first output row within
// the block (the block's total behind the last entry, when there is room), its
// list offset minus that, and its row in the block.  The arrays hold a whole
// number of blocks of rows and are 16 B aligned.
struct Entries {
    uint32_t *pos, *rel;
    uint16_t *row;
};

// One slice of the expansion: block `block` has T output rows after the first
// P of the op, in slices of kSliceRows of which this is number `slice`, and n
// entries.
struct alignas(16) SliceRec {
    unsigned long long P;
    uint32_t block, T, slice, n, pad[2];
};

// k2u pass 1: probe hist[r][scol]; the entries of every block; blk_sum[b] =
// the block's output rows (low 48 bits) and entries (above); group_sums[2g] +=
// output rows and group_sums[2g + 1] += slices of the blocks of group g (256
// blocks; zero at launch), so the op's totals are the sums over its groups.
// clear[0 .. nclear) is set to zero (the other of two alternating sums
// buffers, for the next op).  err bit 0: overflow chain longer than the
// segment's overflow area, bit 1: a block's count reached 2^31.
// func (the direction is functional and hashed): en.pos receives each row's
// neighbour as int32 (-1 when there is none) for launch_k2u_expand_func; err
// bit 3 when a row's list had more than one entry (an index key), which the
// functional expansion cannot write.
// sms: the device's SM count (two input blocks per CTA once an op has 16 per SM).
void launch_k2u_count(const int32_t *hist, int64_t R, int C, int scol, uint32_t dir, PredView pv, const Entries &en,
                      unsigned long long *blk_sum, unsigned long long *group_sums, int *err, bool func,
                      unsigned long long *clear, int64_t nclear, int sms, cudaStream_t st);

// The op's error word and group sums (n words from src) for the host: a CTA,
// stream-ordered behind the count, copies them into dst[2 .. 2 + n) of pinned,
// device-mapped host memory and then writes seq into dst[0], so a host that
// sees seq there reads the op's totals without a device-to-host copy or a
// stream synchronisation.  dst null: nothing to publish.
struct Publish {
    const unsigned long long *src;
    unsigned long long *dst;
    long long n;
    unsigned long long seq;
};
// In the same launch, the records of the op's slices [first, first + cap) (a
// CTA per group); slices null: none.  head (a device word, or null) receives
// the number of slices when an expansion launched behind may write them: the
// count set no error, they are at most max_slices, and the output has at most
// max_rows rows; else 0.
struct SlicePlan {
    const unsigned long long *blk_sum, *group_sums;
    int64_t nblk;
    SliceRec *slices;
    unsigned long long first, cap;
    uint32_t *head;
    const int *err;
    unsigned long long max_rows, max_slices;
};
void launch_publish(const Publish &pub, const SlicePlan &plan, cudaStream_t st);

// Load every k2u count and expansion kernel on the current device (they load
// lazily, at first launch, otherwise); returns a cudaError_t.
int preload_k2u_kernels();

// k2u pass 2 of a hashed functional direction (2 <= C + 1 <= 8): the matched
// rows with their neighbour appended, compacted in order; one CTA per
// non-empty block (n slice records).
void launch_k2u_expand_func(const int32_t *hist, int64_t R, int C, const int32_t *nbr, const SliceRec *slices,
                            unsigned int n, int32_t *out, cudaStream_t st);
// k2u pass 2: the rows (row || neighbour) of n slice records, a CTA each; out
// holds the op's output rows of C + 1 columns and is 16 B aligned; wide: what
// wide_slices says of the op.  head (a device word) not null: the number of
// slices, at most n, is read from there.
bool wide_slices(unsigned long long slices, unsigned long long rows_out, int sms);
void launch_k2u_expand(const int32_t *hist, int C, const int32_t *edges, const Entries &en, const SliceRec *slices,
                       unsigned int n, const uint32_t *head, bool wide, int32_t *out, cudaStream_t st);

// k2k/k2c pass 1: probe + membership of the end value; per-row ballot masks,
// per-block kept-row counts; group_sums[2 g] += kept rows and
// group_sums[2 g + 1] += adjacency entries a linear scan touches, of the
// 2^kGroupShift blocks of group g (zero on entry).  The nclear words at `clear`
// (the other sums buffer) are zeroed.  err bit 0: corrupt overflow chain.
// ecol >= 0: end is column ecol (k2k); ecol < 0: end is the constant `end_const` (k2c).
void launch_filter_probe(const int32_t *hist, int64_t R, int C, int scol, int ecol, int32_t end_const,
                         uint32_t dir, PredView pv, uint32_t *mask, unsigned int *blk_nz,
                         unsigned long long *group_sums, unsigned long long *clear, int64_t nclear,
                         int *err, cudaStream_t st);

// k2k/k2c pass 2: copy the kept rows in order (out holds up to R rows of C columns).
void launch_filter_write(const int32_t *hist, int64_t R, int C, const uint32_t *mask, const unsigned int *blk_nz,
                         const unsigned long long *group_sums, int32_t *out, int sms, cudaStream_t st);

// Whether a filter of nblk blocks copies its kept rows with a CTA per block;
// else with a warp per block.  A warp copies a block of 1024 rows in some 70
// dependent steps, 35 us of them on 11 columns however few blocks there are:
// 12k rows of 11 columns take 65.9 us with a warp per block and 30.9 with a CTA,
// 422k rows of 8 51.9 and 36.0.  From about 16 blocks an SM on there are warps
// enough, and the CTAs' prefixes and barriers cost more.  Around the line, over a
// functional direction, 0.4 kept: 2.0M rows of 3 columns 35.2 and 35.6, 2.4M 35.9 and
// 39.1, 3M 41.7 and 44.1; of 8 columns 2.0M 51.2 and 43.0, 3M 64.2 and 61.0, 4M 76.1
// and 74.2.
inline bool filter_per_block(int64_t nblk, int sms) { return nblk <= 16 * (int64_t)(sms < 1 ? 1 : sms); }

// k2u, k2k and k2c over a dense functional direction (pv.nb[dir] set) in one
// launch; k2u for up to kFusedCols output columns (fused_takes).  out holds
// max_rows rows of C + 1 (k2u) or R rows of C columns and is 16 B aligned; nbr (k2u) holds R
// words, mask (filters) a bit per row, blk_nz a word per block, group_sums two
// zero words per group; written (filters) is a zero word.  clear[0 .. nclear) is set to zero.  The op's totals go
// to pinned host memory: pub[2] = the error word (bit 0: corrupt overflow
// chain, kErrWait: a wait ran out and the op has to run as two kernels),
// pub[3] = output rows, pub[4] = k2u: not 0 when a row's start is an index key
// (the op has to run unspecialised), filter: entries a linear scan touches;
// then seq into pub[0], once every row is counted (k2u) or every kept row
// copied (filters: the launch has finished with its input).  k2u: out holds
// max_rows rows, and blocks whose rows end past them are not written; kFusedWrite,
// a launch behind one of the others with the same scratch, writes out (all
// pub[3] rows of it) and nothing else.  kFusedCount counts and publishes and leaves
// out alone.  Returns a cudaError_t.
constexpr int kFusedCols = 11;
constexpr int kErrWait = 16;
enum { kFusedAll, kFusedCount, kFusedWrite };
struct FusedOp {
    // polls of 100 ns and more after which the publisher and a write CTA give up;
    // the publisher first: it reports the op
    int pub_polls = 1 << 20, write_polls = 1 << 22;
    int part = kFusedAll;
    const int32_t *hist;
    int64_t R;
    int C, scol, ecol;
    int32_t end_const;
    uint32_t dir;
    bool filter;
    PredView pv;
    int32_t *nbr;
    uint32_t *mask;
    unsigned int *blk_nz;
    unsigned long long *group_sums;
    int *err;
    unsigned long long *written;
    unsigned long long *clear;
    int64_t nclear;
    int32_t *out;
    unsigned long long max_rows;
    unsigned long long *pub;
    unsigned long long seq;
    int sms;
};
bool fused_takes(int C, bool filter);
int launch_fused(const FusedOp &op, cudaStream_t st);

// A request of up to kLightSteps steps from a list of at most kLightRows rows in
// one launch of one CTA (wk_light.cu).  The list's table goes to buf[0], step i's
// to buf[(i + 1) & 1]; each holds kLightRows rows of the widest table.  The host
// gets pub[2] = the error word (bit 0: corrupt overflow chain), pub[3] = steps
// done (the next one's output has more than kLightRows rows, or than row_limit),
// pub[4] = entries a linear scan touches in the last filter done, pub[kLightWords
// + i] = rows after step i; then seq in pub[0].
constexpr int kLightRows = 2048, kLightSteps = 8, kLightWords = 6;
enum { kLightK2U, kLightFilter };
struct LightStep {
    PredView pv;
    int kind, C, scol, ecol;   // C: input columns; filters: ecol < 0 for end_const
    int32_t end_const;
    uint32_t dir;
};
struct LightOp {
    int n, deg;
    const int32_t *src;
    int32_t *buf[2];
    long long row_limit;
    unsigned long long *pub;
    unsigned long long seq;
    LightStep s[kLightSteps];
};
void launch_light(const LightOp &op, cudaStream_t st);

// Copy an adjacency list (index or constant start) into a one-column table.
void launch_copy_list(const int32_t *src, int64_t n, int32_t *dst, cudaStream_t st);

}  // namespace dev
}  // namespace wk
