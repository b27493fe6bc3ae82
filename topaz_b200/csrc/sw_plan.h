// sw_plan.h -- which form of the batch Smith-Waterman kernels a pair takes
// (plain C++: the binning kernels and the host share it, tests compile it).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define TPZ_HD __host__ __device__ __forceinline__
#else
#define TPZ_HD inline
#endif

namespace tpz {
namespace sw {

constexpr int kMaxR = 32;                   // rows per lane
constexpr int kStripeRows = 32 * kMaxR;     // longest query of one stripe
constexpr int kPadScore = -64;              // score of pad rows, pad columns and bytes outside the alphabet

// Row bins.  Throughput form: queries above 32 residues with G = 32 lanes
// and R = 9..32 in bins R - 9, with G = 16, 8, 4 and R = 9..16 in bins 24,
// 32, 40 + R - 9, shorter ones with G = 4 and R = 4, 8 in bins 48, 49; with
// twice the lanes and up to 8 rows, queries up to 32, 64, 128 and 256
// residues in bins 55..58.
// Stripe form: 50..52 for queries up to 2048, 4096 and 8192, and 53, 54 for
// shorter ones, up to 512 and 1024.
constexpr int kRBins = 60;
constexpr int kTinyBin = 48;
constexpr int kLongBin = 50;
constexpr int kSmallBin = 53;
constexpr int kWideBin = 55;

// What the size of a batch decides.  The stripe form gives every pair warps
// of its own, so a small batch takes as long as its longest pair; stripe form
// against by-pair, pairs of the microbench: 128 pairs 0.28 / 0.41 ms, 1,024
// 0.32 / 0.54, 2,048 0.45 / 0.55, 4,096 0.51 / 0.63, 8,192 0.80 / 0.81.
// Short queries leave most of a warp's 256 rows to padding, and take lane
// groups from 65 pairs on; of twice the lanes, since few pairs per warp is
// what fills the GPU: 1,024 pairs of 30 x 5000 1.24 ms (stripe form), 0.85 (8
// rows, 4 lanes), 0.61 (4 rows, 8 lanes); 8,192 of 30 x 400 0.17 / 0.14 (8 /
// 4 rows), but 65,536 1.00 / 1.14.  Queries of 65-256 follow where there are
// more pairs than the kernel has warps, if their subjects are so long that
// the batch is not one that ends with a few of them: 3,000 of 180 x 5000 1.63
// / 1.10 ms.
struct Forms {
    int stripe;              // queries above it take the stripe form
    int wide;                // those up to it lane groups of twice the lanes
    int long_slen;           // queries of 65..256 too, from this subject length on
};
inline Forms forms_of(int64_t pairs) {
    const int none = INT32_MAX;
    return pairs <= 64 ? Forms{0, 0, none} : pairs <= 1536 ? Forms{64, 64, none}
           : pairs <= 4096 ? Forms{64, 64, 3072} : pairs <= 8192 ? Forms{kStripeRows, 64, none}
           : Forms{kStripeRows, 0, none};
}

// lanes of a group for a query of one stripe: the fewest that keep 16 rows
// per lane, 32 from 257 residues on
TPZ_HD int group_lanes(int ql) {
    return ql <= 64 ? 4 : ql <= 128 ? 8 : ql <= 256 ? 16 : 32;
}

// Words of 16 bits hold an alignment of up to this many diagonal steps, from
// `floor` (the zero of a score) on in steps of up to `entry`.  A pair that
// may have more of them is not laid beside another pair (see Arithmetic in
// sw_core.cuh).
TPZ_HD int shared_steps(int floor, int entry) {
    return entry > 0 ? (65535 - floor) / entry : INT32_MAX;
}

// The bin of a pair.
TPZ_HD int row_bin(int ql, int sl, Forms f, int steps) {
    if (ql > kStripeRows) return kLongBin + (ql <= 2048 ? 0 : ql <= 4096 ? 1 : 2);
    const bool wide = ql > 16 && (ql <= f.wide || (ql > 64 && ql <= 256 && sl >= f.long_slen));
    if ((ql > f.stripe && !wide) || (ql < sl ? ql : sl) > steps) return kSmallBin + (ql <= 512 ? 0 : 1);
    if (wide) return kWideBin + (ql <= 32 ? 0 : ql <= 64 ? 1 : ql <= 128 ? 2 : 3);
    if (ql <= 32) return kTinyBin + (ql - 1) / 16;
    const int G = group_lanes(ql);
    return (G == 32 ? 0 : G == 16 ? 24 : G == 8 ? 32 : 40) + (ql + G - 1) / G - 9;
}

// Blocks of a launch: no more than pairs, nor than `fit`.
inline unsigned grid_blocks(int64_t sms, int64_t blocks_per_sm, int64_t pairs, int64_t fit) {
    int64_t b = sms * blocks_per_sm;
    b = b < pairs ? b : pairs;
    b = b < fit ? b : fit;
    return (unsigned)(b > 1 ? b : 1);
}

// Query-major stripes keep a boundary row of 8 bytes per subject column for
// each of a block's warps.  `want` blocks of one of `classes` stripe counts,
// on a GPU of `sms` multiprocessors, may take this many with subjects of
// `cols`; 0 where the classes' share of kBoundaryBytes holds fewer than half
// of what would run (those pairs go by pair, whose boundaries are rings in
// shared memory).
constexpr int64_t kBoundaryBytes = (int64_t)512 << 20;
constexpr int kQmWarps = 8;                 // warps of a query-major block
inline int64_t boundary_blocks(int64_t want, int classes, int64_t cols, int sms) {
    const int64_t fit = kBoundaryBytes / classes / (8 * kQmWarps * (cols > 1 ? cols : 1));
    const int64_t need = want < sms ? want : sms;
    return fit >= want ? want : 2 * fit >= need ? fit : 0;
}

}  // namespace sw
}  // namespace tpz
