// sw_kernel.cu -- batched Smith-Waterman (scores + end coordinates) for sm_100a.
//
// The recurrence, its arithmetic and why one pass gives the results of SSW's
// u8 and i16 passes stand in sw_core.cuh.  Here: how alignments are laid on
// warps, binned and launched.
//
// Throughput form (queries of one stripe, <= 1024 residues).  One warp per
// task; a group of G = 4, 8, 16 or 32 lanes holds two pairs in the halves of
// its u16x2 words, lane t owning query rows [t*R, t*R + R) of both.  Subject
// columns stream through a group's lanes as a wavefront, lane t working on
// column k - t at step k, with H and F of a lane's last row handed to lane
// t + 1 by __shfl_up_sync.  G is the smallest group that keeps R <= 16 (32
// above 512 residues; batches of up to 8,192 pairs take more lanes for short
// queries, see sw_plan.h): the wavefront's fill (G - 1 steps) and the per-step
// work outside the rows (shuffles, letters, maximum test) shrink against the
// rows, more rows would leave fewer warps, and a query pads to G*R rows, at
// most G - 1 more than it has.  Groups of a warp take pairs of neighbouring
// subject lengths.
//
// Query-major form (the hits of one search query): the same, with a block of
// 8 warps sharing one profile.  Queries above 1024 residues take the pairs
// through stripes of 32*R rows, the last row of a stripe going to the next
// through memory, two words per column.
//
// Stripe form (queries longer than 1024, and batches too small to fill the
// GPU with warps): W warps per pair; the halves of a warp's words are two row
// ranges of one alignment, so a warp covers 64*R rows, and the warps of a
// pair follow each other three blocks of 32 columns apart, passing the last
// row of one to the first of the next through a ring in shared memory.
//
// The int8 query profile sits in shared memory, one column per lane, so the
// 32 loads of a step never share a bank; PRMT with the sign-replicate
// selector widens two profile bytes into one operand.  Subject letters sit
// in rings of 128 columns as profile offsets, refilled 32 columns at a time.
//
// Pairs are binned on the device by query length class and subject length
// (counting sort), longest subjects first, and drained by persistent kernels
// from atomic task counters, one kernel for all R with the same shared
// memory (4 values of R).

#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

#include "search_internal.cuh"
#include "sw_core.cuh"
#include "tpz_common.cuh"

namespace tpz {
namespace sw {

// scores of tpz_sw_align_one and the allocation-free call stay below this
constexpr int kBig = 32512;

constexpr int kSBins = 256;                 // subject-length buckets (32 residues each)
constexpr int kBins = kRBins * kSBins;
static_assert(kBins % 1024 == 0, "the scan gives each of 1024 threads an equal share");

// ---------------------------------------------------------- one warp's task

// bytes of a group's letter rings, low and high half
constexpr int kPairRing = 2 * kRingCols * 2;

// columns of a stripe's boundary kept in shared memory, [H, F] each
constexpr int kBndCols = 64;

// A stripe of a query above kStripeRows: which one, of how many, and the
// boundary rows -- the warp's ring, and one [H, F] per column in memory,
// read from the stripe above and written for the one below (the same words:
// lane 0 is past a column when lane 31 ends it).
struct Stripe {
    int index, count;
    uint2 *ring, *rows;
};

// f(R as a constant) for a run-time R in [R0, R1]
template <int R0, int R1, class F>
__device__ __forceinline__ void with_rows(int R, F &&f) {
    if constexpr (R0 == R1) f(std::integral_constant<int, R0>());
    else if (R == R0) f(std::integral_constant<int, R0>());
    else with_rows<R0 + 1, R1>(R, f);
}

// Up to 64 / G pairs, two per group of G lanes: pair_at(first), ..., below
// `count`.  prof: this warp's two profiles (BUILD), or the block's one
// profile of the query they share; rings: 32 / G pairs of letter rings.
// STRIPED (G = 32): one stripe of the pairs; keyA / keyB carry their best
// keys from stripe to stripe.
template <int R, bool ENDS, bool BUILD, bool STRIPED, class PairAt>
__device__ __forceinline__ void pair_task(const Args &a, PairAt pair_at, int first, int count, int G,
                                          const uint8_t *matT, uint8_t *prof, uint8_t *rings,
                                          uint4 *snap, const Stripe &sp, uint64_t &keyA, uint64_t &keyB) {
    const int lane = threadIdx.x & 31;
    const int lg = 31 - __clz(G), grp = lane >> lg, gl = lane & (G - 1);
    const int iA = first + 2 * grp, iB = iA + 1;
    const int pA = iA < count ? pair_at(iA) : -1, pB = iB < count ? pair_at(iB) : -1;
    const int slA = pA >= 0 ? a.slen[pA] : 0, slB = pB >= 0 ? a.slen[pB] : 0;
    const int8_t *sA = a.s + (pA >= 0 ? a.soff[pA] : 0), *sB = a.s + (pB >= 0 ? a.soff[pB] : 0);
    const int N = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)max(slA, slB));
    const int i0 = STRIPED ? (sp.index * 32 + lane) * R : gl * R;
    uint16_t *ringA = reinterpret_cast<uint16_t *>(rings + grp * kPairRing), *ringB = ringA + kRingCols;
    Flow f;
    f.profA = prof + lane * 4;
    f.profB = f.profA + (BUILD ? profile_bytes(R) : 0);
    if (BUILD) {
        build_profile<R>(a, a.q + (pA >= 0 ? a.qoff[pA] : 0), pA >= 0 ? a.qlen[pA] : 0, gl * R, matT,
                         prof + lane * 4);
        build_profile<R>(a, a.q + (pB >= 0 ? a.qoff[pB] : 0), pB >= 0 ? a.qlen[pB] : 0, gl * R, matT,
                         prof + profile_bytes(R) + lane * 4);
    }
    const bool above = STRIPED && sp.index > 0, below = STRIPED && sp.index + 1 < sp.count;
    f.ringA = ringA; f.ringB = ringB;
    f.lag = gl; f.lagB = 0; f.width = G;
    f.mul = gl == 0 ? 0u : 1u;
    f.add = gl == 0 ? both((uint32_t)a.floor) : 0u;
    f.bnd = nullptr;
    f.bnd2 = above && lane == 0 ? sp.ring : nullptr;
    f.bnd_end = N;
    f.snap = ENDS ? snap + lane : nullptr;
    // columns 0..63, and pad letters where the columns before 0 are read
#pragma unroll 4
    for (int c = gl; c < 64; c += G) {
        ringA[c] = letter_offset<R>(a, sA, slA, c);
        ringB[c] = letter_offset<R>(a, sB, slB, c);
        ringA[64 + c] = ringB[64 + c] = kPadLetter * words_for(R) * 128;
    }
    uint2 next = make_uint2(0, 0);              // boundary column k0 + lane of the next block
    if (above && lane < N) next = __ldcg(sp.rows + lane);
    __syncwarp();
    Lane<R> L;
    L.start(a, f);
    // the last lane ends its last column at step N + G - 2
    const int nsteps = (N + G) & ~1;
    // a read of the letters that the next refill wants, so that it finds them
    // in L1
    int touched = 0;
    for (int k0 = 0; k0 < nsteps; k0 += 32) {
        if (k0 > 0) {
            asm volatile("" ::"r"(touched));
            for (int i = 0; i < 32; i += G) {
                const int c = k0 + 32 + i + gl;
                ringA[c & (kRingCols - 1)] = letter_offset<R>(a, sA, slA, c);
                ringB[c & (kRingCols - 1)] = letter_offset<R>(a, sB, slB, c);
            }
        }
        {
            const int c = k0 + 64 + (gl << (5 - lg));
            touched = (c < slA ? sA[c] : 0) + (c < slB ? sB[c] : 0);
        }
        if (above) {
            sp.ring[(k0 + lane) & (kBndCols - 1)] = next;
            if (k0 + 32 + lane < N) next = __ldcg(sp.rows + k0 + 32 + lane);
        }
        if (ENDS) refresh<R, false>(L, G, 0u);
        __syncwarp();
        steps<R, ENDS, false, STRIPED>(L, a, f, k0, min(k0 + 32, nsteps), nullptr,
                                       below && lane == 31 ? sp.rows : nullptr);
    }
    uint64_t kA = lane_key<R, ENDS>(L, a, f, false, i0), kB = lane_key<R, ENDS>(L, a, f, true, i0);
    for (int o = G >> 1; o > 0; o >>= 1) {
        kA = max(kA, __shfl_xor_sync(0xFFFFFFFFu, kA, o));
        kB = max(kB, __shfl_xor_sync(0xFFFFFFFFu, kB, o));
    }
    if (STRIPED) {
        kA = keyA = max(keyA, kA);
        kB = keyB = max(keyB, kB);
    }
    if (!below) {
        if (gl == 0 && pA >= 0) write_result(a, pA, kA, ENDS);
        if (gl == 1 && pB >= 0) write_result(a, pB, kB, ENDS);
    }
    __syncwarp();
}

// The bins of one launch, with rows per lane and lanes per group of each;
// their tasks are taken in this order from the first bin's counter.
constexpr int kSetBins = 16;
struct BinSet {
    int n;
    int bin[kSetBins], rows[kSetBins], lanes[kSetBins];
};

// letter rings: one group above 16 rows, up to 8 below
template <int R1>
__host__ __device__ constexpr int bin_smem() {
    return kMatBytes + 2 * profile_bytes(R1) + (R1 > 16 ? 1 : 8) * kPairRing;
}

// A block is one warp: tasks differ in length, and nothing is shared but the
// matrix.  Shared memory (two profiles, 26 bytes per row and pair) holds the
// warps per SM down to 4 (R = 32) .. 8 (R = 9).  The R of a launch (R0..R1)
// take the same profile words per lane; with a launch per R (26) instead of
// one per word count (7) a kernel's last tasks had only 8 streams of others
// beside them.
template <int R0, int R1, bool ENDS>
__global__ void __launch_bounds__(32) sw_bin_kernel(const __grid_constant__ Args a,
                                                    const __grid_constant__ BinSet b) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t *prof = smem + kMatBytes, *rings = prof + 2 * profile_bytes(R1);
    int total = 0;
    for (int i = 0; i < b.n; ++i) {
        const int per = 64 / b.lanes[i];
        total += (a.rinfo[2 * b.bin[i] + 1] + per - 1) / per;
    }
    if (total == 0) return;
    load_matrix(a, smem);
    __syncwarp();
    const Stripe none{0, 1, nullptr, nullptr};
    uint4 *snap = a.snap + (size_t)blockIdx.x * snap_words(R1);
    uint64_t kA = 0, kB = 0;
    for (;;) {
        int t = 0;
        if (threadIdx.x == 0) t = atomicAdd(&a.next_task[b.bin[0]], 1);
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t >= total) break;
        int i = 0, per = 64 / b.lanes[0], count = a.rinfo[2 * b.bin[0] + 1];
        while (t >= (count + per - 1) / per) {
            t -= (count + per - 1) / per;
            ++i;
            per = 64 / b.lanes[i];
            count = a.rinfo[2 * b.bin[i] + 1];
        }
        const int32_t *ids = a.sorted + a.rinfo[2 * b.bin[i]];
        auto id = [&](int x) { return ids[x]; };
        if constexpr (R1 == 8) {
            if (b.rows[i] == 4)
                pair_task<4, ENDS, true, false>(a, id, t * per, count, b.lanes[i], smem, prof, rings, snap,
                                                 none, kA, kB);
            else
                pair_task<8, ENDS, true, false>(a, id, t * per, count, b.lanes[i], smem, prof, rings, snap,
                                                 none, kA, kB);
        } else {
            with_rows<R0, R1>(b.rows[i], [&](auto r) {
                pair_task<decltype(r)::value, ENDS, true, false>(a, id, t * per, count, b.lanes[i], smem, prof,
                                                                 rings, snap, none, kA, kB);
            });
        }
    }
}

// ------------------------------------------------------------- query-major

// Pairs that share their query (the hits of one search query): a block of
// kQmWarps warps keeps ONE profile of the query in shared memory for all of
// them, so registers, not shared memory, bound the warps per SM.  The block
// sorts the chunk's pairs by subject length, longest first.
constexpr int kQmMaxPairs = 256;      // pairs per chunk: longer pair lists of a query are cut
constexpr int kQmMinPairs = 2 * kQmWarps;

struct Chunk {
    int64_t first;            // pairs [first, first + pairs) of one query
    int32_t pairs, rows, lanes, stripes;
};

struct QmArgs {
    const Chunk *chunks;
    int count;
    int32_t *next;            // chunk counter
    int profile, ring;        // bytes of the profile, and of one warp's letter rings
    uint2 *bnd;               // stripe boundary rows, bnd_cols per warp
    int64_t bnd_cols;
};

__host__ __device__ constexpr int qm_smem_bytes(int profile, int ring, bool striped) {
    return kMatBytes + profile + kQmWarps * (ring + (striped ? kBndCols * 8 : 0)) + 4 * kQmMaxPairs;
}

// profile words of a query for the lanes of every group, one word column of
// one stripe per warp at a time; the stripes' profiles follow each other
template <int R>
__device__ __forceinline__ void qm_build_profile(const Args &a, int64_t p, int G, int stripes,
                                                 const uint8_t *matT, uint8_t *prof) {
    constexpr int W = words_for(R);
    const int lane = threadIdx.x & 31;
    const int ql = a.qlen[p];
    const int8_t *q = a.q + a.qoff[p];
    for (int i = threadIdx.x >> 5; i < W * stripes; i += kQmWarps) {
        const int w = i % W, st = i / W, i0 = (st * 32 + (lane & (G - 1))) * R;
        int x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = 4 * w + k;
            x[k] = query_letter(a, (r < R && i0 + r < ql) ? (int)q[i0 + r] : -1);
        }
        build_word<W>(matT, x[0], x[1], x[2], x[3], prof + st * profile_bytes(R) + w * 128 + lane * 4);
    }
}

// pair i of a chunk in the order of its sorted keys
struct ChunkPair {
    const uint32_t *keys;
    int first;
    __device__ __forceinline__ int operator()(int i) const { return first + 255 - (int)(keys[i] & 255u); }
};

// One chunk with R rows per lane: the profile, the keys sorted, the tasks.
template <int R, bool ENDS, bool STRIPED>
__device__ __forceinline__ void run_chunk(const Args &a, const Chunk &ch, const uint8_t *matT, uint8_t *prof,
                                          uint8_t *rings, uint32_t *keys, uint4 *snap, uint2 *ring,
                                          uint2 *rows, int *next) {
    const int lane = threadIdx.x & 31;
    const int n = ch.pairs, G = STRIPED ? 32 : ch.lanes, stripes = STRIPED ? ch.stripes : 1;
    int np = 1;
    while (np < n) np <<= 1;
    // keys: subject length (descending; < 2^24), place in the chunk
    for (int i = threadIdx.x; i < np; i += blockDim.x)
        keys[i] = i < n ? ((uint32_t)a.slen[ch.first + i] << 8) | (uint32_t)(255 - i) : 0u;
    qm_build_profile<R>(a, ch.first, G, stripes, matT, prof);
    __syncthreads();
    for (int k = 2; k <= np; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < np; i += blockDim.x) {
                const int l = i ^ j;
                if (l > i) {
                    const uint32_t x = keys[i], y = keys[l];
                    if (((i & k) == 0) ? (x < y) : (x > y)) { keys[i] = y; keys[l] = x; }
                }
            }
            __syncthreads();
        }
    }
    const int per = 64 / G;
    const ChunkPair id{keys, (int)ch.first};
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(next, 1);
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t * per >= n) break;
        uint64_t kA = 0, kB = 0;
        for (int st = 0; st < stripes; ++st) {
            const Stripe sp{st, stripes, ring, rows};
            pair_task<R, ENDS, false, STRIPED>(a, id, t * per, n, G, nullptr, prof + st * profile_bytes(R), rings,
                                               snap, sp, kA, kB);
        }
    }
}

template <int R, bool ENDS, bool STRIPED>
__device__ __forceinline__ void run_chunk_rows(const Args &a, const Chunk &ch, const uint8_t *matT, uint8_t *prof,
                                               uint8_t *rings, uint32_t *keys, uint4 *snap, uint2 *ring,
                                               uint2 *rows, int *next) {
    if constexpr (R == kMaxR) {
        run_chunk<R, ENDS, STRIPED>(a, ch, matT, prof, rings, keys, snap, ring, rows, next);
    } else {
        if (ch.rows <= R) run_chunk<R, ENDS, STRIPED>(a, ch, matT, prof, rings, keys, snap, ring, rows, next);
        else run_chunk_rows<R < 8 ? 8 : R + 1, ENDS, STRIPED>(a, ch, matT, prof, rings, keys, snap, ring, rows, next);
    }
}

// One launch for the chunks of all row counts (the longest chunks first):
// two blocks per SM share the registers (128 a thread: with scores alone the
// largest R spill nothing, 24 bytes in stripes, with ends 20 and 228), so a
// chunk's end is filled by whatever chunk comes next.  (A launch per R over 8
// streams left the SMs of a 1000-query batch half empty at each launch's end.)
template <bool ENDS, bool STRIPED>
__global__ void __launch_bounds__(kQmWarps * 32, 2) sw_query_kernel(const __grid_constant__ Args a,
                                                                    const QmArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5;
    uint8_t *prof = smem + kMatBytes;
    uint8_t *rings = prof + g.profile + warp * g.ring;
    uint2 *bnd = reinterpret_cast<uint2 *>(prof + g.profile + kQmWarps * g.ring) + warp * kBndCols;
    uint32_t *keys = reinterpret_cast<uint32_t *>(prof + g.profile + kQmWarps * g.ring +
                                                  (STRIPED ? kQmWarps * kBndCols * 8 : 0));
    uint2 *rows = g.bnd + (int64_t)(blockIdx.x * kQmWarps + warp) * g.bnd_cols;
    uint4 *snap = a.snap + (size_t)(blockIdx.x * kQmWarps + warp) * snap_words(kMaxR);
    __shared__ int s_chunk, s_next;
    load_matrix(a, smem);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_chunk = atomicAdd(g.next, 1);
            s_next = 0;
        }
        __syncthreads();
        if (s_chunk >= g.count) break;
        const Chunk ch = g.chunks[s_chunk];
        run_chunk_rows<STRIPED ? 17 : 4, ENDS, STRIPED>(a, ch, smem, prof, rings, keys, snap, bnd, rows, &s_next);
    }
}

// ------------------------------------------------------------ stripe form

constexpr int kLongWarps = 4;
constexpr int kStripeLag = 3;      // blocks of 32 columns between two warps of a pair

// W warps of one pair: a block's barrier 1 + group
__device__ __forceinline__ void group_sync(int group, int W) {
    if (W == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * W) : "memory");
}

// Warp `wg` of the W warps of one pair: rows [wg*64*R, (wg+1)*64*R), the low
// halves the first 32*R of them.  prof: this warp's two profiles; ring: its
// letters; above / below: the boundary rings of kRingCols words to the
// neighbouring warps (null: none).  Lane 31's high half ends column k - 63
// at step k, so a block of 32 columns is complete in the ring two blocks
// later, and the warp below takes it in the block after that.  Returns the
// warp's best key in every lane.
template <int R, bool ENDS>
__device__ __forceinline__ uint64_t stripe_task(const Args &a, const int8_t *q, int ql, const int8_t *s,
                                                int sl, int group, int W, int wg, const uint8_t *matT,
                                                uint8_t *prof, uint16_t *ring, const uint32_t *above,
                                                uint32_t *below, uint4 *snap) {
    const int lane = threadIdx.x & 31;
    const int i0 = (wg * 64 + lane) * R, i1 = i0 + 32 * R;
    build_profile<R>(a, q, ql, i0, matT, prof + lane * 4);
    build_profile<R>(a, q, ql, i1, matT, prof + profile_bytes(R) + lane * 4);
    Flow f;
    f.profA = prof + lane * 4;
    f.profB = f.profA + profile_bytes(R);
    f.ringA = f.ringB = ring;
    f.lag = lane; f.lagB = 32; f.width = 32;
    f.mul = lane == 0 ? 65536u : 1u;
    f.add = lane == 0 ? (uint32_t)a.floor : 0u;
    f.bnd = lane == 0 ? above : nullptr;
    f.bnd2 = nullptr;
    f.bnd_end = sl;
    f.snap = ENDS ? snap + lane : nullptr;
#pragma unroll
    for (int c = lane; c < 64; c += 32) {
        ring[c] = letter_offset<R>(a, s, sl, c);
        ring[64 + c] = kPadLetter * words_for(R) * 128;
    }
    __syncwarp();
    Lane<R> L;
    L.start(a, f);
    const int nblk = (sl + 63 + 31) >> 5;
    int touched = 0;
    for (int p = 0; p < nblk + kStripeLag * (W - 1); ++p) {
        const int b = p - kStripeLag * wg, k0 = 32 * b;
        if (b >= 0 && b < nblk) {
            if (b > 0) {
                asm volatile("" ::"r"(touched));
                ring[(k0 + 32 + lane) & (kRingCols - 1)] = letter_offset<R>(a, s, sl, k0 + 32 + lane);
            }
            touched = k0 + 64 + lane < sl ? s[k0 + 64 + lane] : 0;
            uint32_t in = 0;
            if (above && k0 + lane < sl) in = lo16(above[(k0 + lane) & (kRingCols - 1)]);
            if (ENDS) refresh<R, true>(L, 32, in);
            __syncwarp();
            steps<R, ENDS, true, false>(L, a, f, k0, k0 + 32, lane == 31 ? below : nullptr, nullptr);
        }
        group_sync(group, W);
    }
    uint64_t key = max(lane_key<R, ENDS>(L, a, f, false, i0), lane_key<R, ENDS>(L, a, f, true, i1));
    for (int o = 16; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(0xFFFFFFFFu, key, o));
    return key;
}

template <bool ENDS, int RMAX>
__device__ __forceinline__ uint64_t stripe_rows(int R, const Args &a, const int8_t *q, int ql,
                                                const int8_t *s, int sl, int group, int W, int wg,
                                                const uint8_t *matT, uint8_t *prof, uint16_t *ring,
                                                const uint32_t *above, uint32_t *below, uint4 *snap) {
#define TPZ_STRIPE(r) \
    stripe_task<r, ENDS>(a, q, ql, s, sl, group, W, wg, matT, prof, ring, above, below, snap)
    if (R <= 4) return TPZ_STRIPE(4);
    if (RMAX == 8 || R <= 8) return TPZ_STRIPE(8);
    if constexpr (RMAX > 8) {
        if (R <= 16) return TPZ_STRIPE(16);
        if (R <= 20) return TPZ_STRIPE(20);
        if (R <= 24) return TPZ_STRIPE(24);
        if (R <= 28) return TPZ_STRIPE(28);
        return TPZ_STRIPE(32);
    }
#undef TPZ_STRIPE
}

// one warp's shared memory: two profiles, the letter ring, the boundary ring,
// and (up to 8 rows: what one pair per launch has) the stored columns
__host__ __device__ constexpr int stripe_warp_bytes(int RMAX) {
    return 2 * profile_bytes(RMAX) + 2 * kRingCols + 4 * kRingCols + (RMAX <= 8 ? 16 * snap_words(RMAX) : 0);
}
__host__ __device__ constexpr int stripe_smem(int RMAX, int warps) {
    return kMatBytes + warps * stripe_warp_bytes(RMAX);
}

// Bins of the stripe form in one launch, and the fewest and most warps that
// may share a pair of each (64 pairs: 0.20 ms with up to 4 warps for queries
// above 512 residues, 0.21 ms with 2).
struct StripeSet {
    int n;
    int bin[3], wmin[3], wmax[3];
};

// Blocks of 4 warps; a pair takes wmin warps, more of them while the bin has
// fewer pairs than would fill the grid's warps.
template <bool ENDS, int RMAX>
__global__ void __launch_bounds__(32 * kLongWarps) sw_stripe_kernel(const __grid_constant__ Args a,
                                                                    const __grid_constant__ StripeSet b) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t s_key[kLongWarps];
    __shared__ int s_task[kLongWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t *prof = smem + kMatBytes + warp * stripe_warp_bytes(RMAX);
    uint16_t *ring = reinterpret_cast<uint16_t *>(prof + 2 * profile_bytes(RMAX));
    uint32_t *below = reinterpret_cast<uint32_t *>(ring + kRingCols);
    const uint32_t *above = reinterpret_cast<const uint32_t *>(
        reinterpret_cast<const uint8_t *>(below) - stripe_warp_bytes(RMAX));
    uint4 *snap = RMAX <= 8 ? reinterpret_cast<uint4 *>(below + kRingCols)
                            : a.snap + (size_t)(blockIdx.x * kLongWarps + warp) * snap_words(RMAX);
    bool ready = false;
    for (int i = 0; i < b.n; ++i) {
        const int start = a.rinfo[2 * b.bin[i]], count = a.rinfo[2 * b.bin[i] + 1];
        if (count == 0) continue;
        if (!ready) load_matrix(a, smem);
        ready = true;
        __syncthreads();
        int W = b.wmin[i];
        while (W < b.wmax[i] && (int64_t)count * W < (int64_t)gridDim.x * kLongWarps) W *= 2;
        const int group = warp / W, wg = warp % W;
        for (;;) {
            if (wg == 0 && lane == 0) s_task[group] = atomicAdd(&a.next_task[b.bin[i]], 1);
            group_sync(group, W);
            const int t = s_task[group];
            if (t >= count) break;
            const int p = a.sorted[start + t];
            const int ql = a.qlen[p];
            const uint64_t key = stripe_rows<ENDS, RMAX>(
                (ql + 64 * W - 1) / (64 * W), a, a.q + a.qoff[p], ql, a.s + a.soff[p], a.slen[p], group,
                W, wg, smem, prof, ring, wg > 0 ? above : nullptr, wg + 1 < W ? below : nullptr, snap);
            if (lane == 0) s_key[warp] = key;
            group_sync(group, W);
            if (wg == 0 && lane == 0) {
                uint64_t best = key;
                for (int w = 1; w < W; ++w) best = max(best, s_key[warp + w]);
                write_result(a, p, best, ENDS);
            }
        }
    }
}

// One pair per launch (the per-pair form of ssw_init + ssw_align): `W` warps
// of the stripe form with at most 8 rows per lane, lengths from the host.
constexpr int kOneMaxQlen = kStripeRows;
__global__ void __launch_bounds__(64) sw_one_kernel(const __grid_constant__ Args a, int qlen, int slen) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t s_key[2];
    const int warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    uint8_t *prof = smem + kMatBytes + warp * stripe_warp_bytes(8);
    uint16_t *ring = reinterpret_cast<uint16_t *>(prof + 2 * profile_bytes(8));
    uint32_t *below = reinterpret_cast<uint32_t *>(ring + kRingCols);
    const uint32_t *above = reinterpret_cast<const uint32_t *>(
        reinterpret_cast<const uint8_t *>(below) - stripe_warp_bytes(8));
    load_matrix(a, smem);
    __syncthreads();
    const uint64_t key = stripe_rows<true, 8>((qlen + 64 * W - 1) / (64 * W), a, a.q, qlen, a.s, slen, 0, W,
                                              warp, smem, prof, ring, warp > 0 ? above : nullptr,
                                              warp + 1 < W ? below : nullptr,
                                              reinterpret_cast<uint4 *>(below + kRingCols));
    if ((threadIdx.x & 31) == 0) s_key[warp] = key;
    __syncthreads();
    if (threadIdx.x == 0) write_result(a, 0, W > 1 ? max(s_key[0], s_key[1]) : s_key[0], true);
}

// ---------------------------------------------------------------- binning

struct BinArgs {
    int64_t n;               // pairs 0..n-1, or list[0..n)
    const int32_t *list;
    const int32_t *qlen, *slen;
    int max_qlen;
    Forms forms;             // of the batch's size
    int steps;               // shared_steps of the scoring
};

__device__ __forceinline__ int pair_bin(const BinArgs &b, int ql, int sl) {
    const int sb = min(sl >> 5, kSBins - 1);
    return row_bin(ql, sl, b.forms, b.steps) * kSBins + (kSBins - 1 - sb);      // long subjects first
}

__global__ void bin_count_kernel(BinArgs b, int32_t *counts, int32_t *status) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < b.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int p = b.list ? b.list[i] : (int)i;
        const int ql = b.qlen[p], sl = b.slen[p];
        if (ql < 1 || ql > b.max_qlen || sl < 0 || sl >= TPZ_SW_MAX_SLEN) {
            status[p] = TPZ_SW_INVALID;
            continue;
        }
        atomicAdd(&counts[pair_bin(b, ql, sl)], 1);
    }
}

// one block of 1024 threads: exclusive scan of kBins counts -> cursor; the
// per-row-bin [start, count] pairs -> rinfo; task counters cleared.
__global__ void bin_scan_kernel(const int32_t *counts, int32_t *cursor, int32_t *rinfo,
                                int32_t *next_task) {
    constexpr int PER = kBins / 1024;
    __shared__ int32_t part[1024];
    const int t = threadIdx.x;
    int32_t loc[PER];
    int32_t sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) { loc[i] = counts[t * PER + i]; sum += loc[i]; }
    part[t] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const int32_t v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    int32_t run = part[t] - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) { cursor[t * PER + i] = run; run += loc[i]; }
    __syncthreads();
    if (t < kRBins) {
        const int b0 = t * kSBins, b1 = b0 + kSBins;
        const int32_t s0 = cursor[b0];
        const int32_t e1 = cursor[b1 - 1] + counts[b1 - 1];
        rinfo[2 * t] = s0;
        rinfo[2 * t + 1] = e1 - s0;
        next_task[t] = 0;
    }
}

__global__ void bin_scatter_kernel(BinArgs b, int32_t *cursor, int32_t *sorted) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < b.n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int p = b.list ? b.list[i] : (int)i;
        const int ql = b.qlen[p], sl = b.slen[p];
        if (ql < 1 || ql > b.max_qlen || sl < 0 || sl >= TPZ_SW_MAX_SLEN) continue;
        sorted[atomicAdd(&cursor[pair_bin(b, ql, sl)], 1)] = p;
    }
}

// ------------------------------------------------------------ roofline probe

// Independent chains of __viaddmax_s16x2 per thread: measures the DPX issue
// rate the SW kernel is bounded by.  kChains chains per thread, iters steps.
constexpr int kProbeChains = 8;

__global__ void __launch_bounds__(256) dpx_probe_kernel(int iters, uint32_t inc, uint32_t floor_v,
                                                        uint32_t *out) {
    uint32_t acc[kProbeChains];
#pragma unroll
    for (int c = 0; c < kProbeChains; ++c) acc[c] = (threadIdx.x + 131u * c) * 0x00010001u;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int c = 0; c < kProbeChains; ++c) acc[c] = __viaddmax_s16x2(acc[c], inc, floor_v);
    }
    uint32_t x = 0;
#pragma unroll
    for (int c = 0; c < kProbeChains; ++c) x ^= acc[c];
    out[blockIdx.x * blockDim.x + threadIdx.x] = x;
}

// ------------------------------------------------------------ host driver

constexpr int kMaxSmem = 225 * 1024;  // dynamic shared memory of a block, at most

// Kernels of one device with their launch attributes, set once.
constexpr int kBinKernels = 7;
struct Kernels {
    typedef void (*BinFn)(const Args, const BinSet);
    typedef void (*QmFn)(const Args, const QmArgs);
    typedef void (*StripeFn)(const Args, const StripeSet);
    BinFn bin[2][kBinKernels];               // [ends][most rows first]
    QmFn qm[2][2];                           // [ends][striped]
    StripeFn stripe8[2], stripe32[2];        // [ends]
    BinSet set[kBinKernels];
    int bin_smem[kBinKernels], bin_blocks[2][kBinKernels];   // blocks per SM
    int stripe8_blocks[2], stripe32_blocks[2];
};

template <int I, int R0, int R1>
static void fill_bin(Kernels &k) {
    k.bin[0][I] = sw_bin_kernel<R0, R1, false>;
    k.bin[1][I] = sw_bin_kernel<R0, R1, true>;
    k.bin_smem[I] = bin_smem<R1>();
    BinSet &s = k.set[I];
    s.n = 0;
    auto add = [&](int bin, int rows, int lanes) {
        s.bin[s.n] = bin; s.rows[s.n] = rows; s.lanes[s.n++] = lanes;
    };
    if (R1 == 8) {
        for (int w = 3; w >= 0; --w) add(kWideBin + w, w ? 8 : 4, w ? 4 << w : 8);
        add(kTinyBin + 1, 8, 4);
        add(kTinyBin, 4, 4);
        return;
    }
    for (int R = R1; R >= R0; --R) add(R - 9, R, 32);
    for (int g = 0; g < 3 && R1 <= 16; ++g)
        for (int R = R1; R >= R0; --R) add(24 + 8 * g + R - 9, R, 16 >> g);
}

// dynamic shared memory of a kernel, the whole carveout (so blocks of
// kernels running side by side share an SM), and its blocks per SM
static int set_up(const void *f, int smem, int threads, int *blocks) {
    TPZ_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    TPZ_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  (int)cudaSharedmemCarveoutMaxShared));
    if (blocks) {
        int nb = 0;
        TPZ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, threads, smem));
        *blocks = std::max(1, nb);
    }
    return TPZ_OK;
}

static int kernels(const Kernels **out) {
    static std::mutex mu;
    static std::vector<Kernels *> per_dev;
    int dev = 0;
    TPZ_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if ((int)per_dev.size() <= dev) per_dev.resize(dev + 1, nullptr);
    if (!per_dev[dev]) {
        Kernels *k = new Kernels();
        fill_bin<0, 29, 32>(*k);
        fill_bin<1, 25, 28>(*k);
        fill_bin<2, 21, 24>(*k);
        fill_bin<3, 17, 20>(*k);
        fill_bin<4, 13, 16>(*k);
        fill_bin<5, 9, 12>(*k);
        fill_bin<6, 4, 8>(*k);
        int rc = TPZ_OK;
        k->qm[0][0] = sw_query_kernel<false, false>;
        k->qm[0][1] = sw_query_kernel<false, true>;
        k->qm[1][0] = sw_query_kernel<true, false>;
        k->qm[1][1] = sw_query_kernel<true, true>;
        k->stripe8[0] = sw_stripe_kernel<false, 8>;
        k->stripe8[1] = sw_stripe_kernel<true, 8>;
        k->stripe32[0] = sw_stripe_kernel<false, 32>;
        k->stripe32[1] = sw_stripe_kernel<true, 32>;
        for (int e = 0; rc == TPZ_OK && e < 2; ++e) {
            for (int i = 0; rc == TPZ_OK && i < kBinKernels; ++i)
                rc = set_up((const void *)k->bin[e][i], k->bin_smem[i], 32, &k->bin_blocks[e][i]);
            for (int x = 0; rc == TPZ_OK && x < 2; ++x)
                rc = set_up((const void *)k->qm[e][x], kMaxSmem, kQmWarps * 32, nullptr);
            if (rc == TPZ_OK)
                rc = set_up((const void *)k->stripe8[e], stripe_smem(8, kLongWarps), 32 * kLongWarps,
                            &k->stripe8_blocks[e]);
            if (rc == TPZ_OK)
                rc = set_up((const void *)k->stripe32[e], stripe_smem(32, kLongWarps), 32 * kLongWarps,
                            &k->stripe32_blocks[e]);
        }
        if (rc == TPZ_OK) rc = set_up((const void *)sw_one_kernel, stripe_smem(8, 2), 64, nullptr);
        if (rc) { delete k; return rc; }
        per_dev[dev] = k;
    }
    *out = per_dev[dev];
    return TPZ_OK;
}

constexpr int kAuxStreams = 8;           // a kernel of a batch each

// Per host thread and device: the auxiliary streams and fork/join events of
// one call must not be shared with a call running in another thread.
struct Streams {
    cudaStream_t aux[kAuxStreams];       // bin kernels overlap their tails here
    cudaEvent_t fork, join[kAuxStreams];
};

struct StreamSets {
    std::vector<Streams *> per_dev;
    ~StreamSets() {
        for (Streams *c : per_dev) {
            if (!c) continue;
            for (int i = 0; i < kAuxStreams; ++i) {
                cudaStreamDestroy(c->aux[i]);
                cudaEventDestroy(c->join[i]);
            }
            cudaEventDestroy(c->fork);
            delete c;
        }
    }
};

// lane: calls of one thread that run at the same time (the chunks of the
// host entry point; a search's query-major kernels beside its other pairs)
// take different lanes, so they get separate streams
static int streams(Streams **out, int lane) {
    static thread_local StreamSets sets;
    int dev = 0;
    TPZ_CUDA(cudaGetDevice(&dev));
    const size_t at = 3 * (size_t)dev + lane;
    if (sets.per_dev.size() <= at) sets.per_dev.resize(at + 1, nullptr);
    if (!sets.per_dev[at]) {
        Streams *c = new Streams();
        for (int i = 0; i < kAuxStreams; ++i) {
            TPZ_CUDA(cudaStreamCreateWithFlags(&c->aux[i], cudaStreamNonBlocking));
            TPZ_CUDA(cudaEventCreateWithFlags(&c->join[i], cudaEventDisableTiming));
        }
        TPZ_CUDA(cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming));
        sets.per_dev[at] = c;
    }
    *out = sets.per_dev[at];
    return TPZ_OK;
}

static int fork(Streams *x, cudaStream_t st) {
    TPZ_CUDA(cudaEventRecord(x->fork, st));
    for (int i = 0; i < kAuxStreams; ++i) TPZ_CUDA(cudaStreamWaitEvent(x->aux[i], x->fork, 0));
    return TPZ_OK;
}

static int join(Streams *x, cudaStream_t st) {
    for (int i = 0; i < kAuxStreams; ++i) {
        TPZ_CUDA(cudaEventRecord(x->join[i], x->aux[i]));
        TPZ_CUDA(cudaStreamWaitEvent(st, x->join[i], 0));
    }
    return TPZ_OK;
}

static thread_local int64_t g_last_launches = 0;

int64_t &last_launches() { return g_last_launches; }

// scratch words of one call: counts and cursor per bin, [start, count] and a
// task counter per row bin, then the sorted pair ids
constexpr size_t kBinWords = 2 * (size_t)kBins + 3 * kRBins;

// Blocks per SM of by-pair kernel i, 0 where a batch of these forms has no
// pairs for it: small batches only for the one of up to 8 rows, and that with
// 8 blocks, so that some hundred tasks do not end up on a few SMs (3,000
// pairs of 10 x 5000: 0.70 ms, 0.84 with 12).
static int bin_blocks(const Kernels *k, int e, int i, Forms f) {
    if (f.stripe >= kStripeRows) return k->bin_blocks[e][i];
    return f.wide > 0 && i == kBinKernels - 1 ? std::min(8, k->bin_blocks[e][i]) : 0;
}

static unsigned grid_of(int blocks_per_sm, int64_t n) {
    return grid_blocks(sm_count(), blocks_per_sm, n, INT64_MAX);
}

// uint4 words for the columns that launch_batch's kernels store
static size_t batch_snap_words(const Kernels *k, int64_t n, int max_qlen) {
    size_t sum = 0;
    if (max_qlen > kStripeRows) sum += (size_t)grid_of(k->stripe32_blocks[1], n) * kLongWarps * snap_words(kMaxR);
    for (int i = 0; i < kBinKernels; ++i)
        if (const int per_sm = bin_blocks(k, 1, i, forms_of(n)))
            sum += (size_t)grid_of(per_sm, n) * snap_words(k->set[i].rows[0]);
    return sum;
}

// blocks of one SM that shared memory allows (228 KB, 1 KB of it per block)
constexpr int blocks_by_smem(int smem) { return 228 * 1024 / (smem + 1024); }
template <int R1>
constexpr size_t bin_snaps() { return (size_t)blocks_by_smem(bin_smem<R1>()) * snap_words(R1); }

int64_t search_scratch_bytes(int max_qlen, bool ends) {
    // by pair: the hits that report mode aligns again, or the rest of a batch
    size_t words = bin_snaps<32>() + bin_snaps<28>() + bin_snaps<24>() + bin_snaps<20>() + bin_snaps<16>() +
                   bin_snaps<12>() + bin_snaps<8>() + (size_t)kLongWarps * snap_words(kMaxR);
    // query-major, two blocks of an SM in each class
    if (ends) words += (max_qlen > kStripeRows ? 5 : 1) * (size_t)(2 * kQmWarps) * snap_words(kMaxR);
    return (int64_t)(16 * words * sm_count() + 4 * kBinWords) + (max_qlen > kStripeRows ? kBoundaryBytes : 0);
}

// Bins the pairs (all of them, or the n ids of `list`) in ws and launches the
// kernels that align them, over the auxiliary streams x so that each
// kernel's tail overlaps the next one.  x null: all on st, so that the kernels
// share the snap_cap words of stored columns, with no more blocks than those
// are for (x: batch_snap_words of them).
static int launch_batch(const Kernels *k, Streams *x, Args &a, int64_t n, const int32_t *list,
                        int32_t *ws, uint4 *snap, int64_t snap_cap, int max_qlen, bool ends, cudaStream_t st,
                        int64_t &launches) {
    const int nsm = sm_count();
    int32_t *counts = ws, *cursor = counts + kBins, *rinfo = cursor + kBins;
    int32_t *next_task = rinfo + 2 * kRBins, *sorted = ws + kBinWords;
    a.sorted = sorted; a.rinfo = rinfo; a.next_task = next_task;
    const Forms f = forms_of(n);
    BinArgs b{n, list, a.qlen, a.slen, max_qlen, f, a.steps};
    TPZ_CUDA(cudaMemsetAsync(counts, 0, sizeof(int32_t) * kBins, st));
    const int gb = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)nsm * 8));
    bin_count_kernel<<<gb, 256, 0, st>>>(b, counts, a.status);
    bin_scan_kernel<<<1, 1024, 0, st>>>(counts, cursor, rinfo, next_task);
    bin_scatter_kernel<<<gb, 256, 0, st>>>(b, cursor, sorted);
    launches += 4;
    const int e = ends ? 1 : 0;
    if (x) {
        const int rc = fork(x, st);
        if (rc) return rc;
    }
    int at = 0;
    auto next_stream = [&]() { return x ? x->aux[at++ % kAuxStreams] : st; };
    auto grid = [&](int blocks, int words) { return grid_blocks(nsm, blocks, n, x ? INT64_MAX : snap_cap / words); };
    a.snap = ends ? snap : nullptr;
    if (max_qlen > kStripeRows) {
        const StripeSet s{3, {kLongBin + 2, kLongBin + 1, kLongBin}, {4, 2, 1}, {4, 4, 4}};
        const int words = kLongWarps * snap_words(kMaxR);
        const unsigned blocks = grid(k->stripe32_blocks[e], words);
        k->stripe32[e]<<<blocks, 32 * kLongWarps, stripe_smem(32, kLongWarps), next_stream()>>>(a, s);
        ++launches;
        if (ends && x) a.snap += (size_t)blocks * words;
    }
    // (in a large batch: the pairs that have to have their words to themselves)
    if (f.stripe < kStripeRows || std::min(max_qlen, kStripeRows) > a.steps) {
        const StripeSet s{2, {kSmallBin + 1, kSmallBin, 0}, {2, 1, 0}, {4, 2, 0}};
        k->stripe8[e]<<<grid_of(k->stripe8_blocks[e], n), 32 * kLongWarps, stripe_smem(8, kLongWarps),
                        next_stream()>>>(a, s);
        ++launches;
    }
    for (int i = 0; i < kBinKernels; ++i) {
        const int per_sm = bin_blocks(k, e, i, f);
        if (per_sm == 0) continue;
        const int words = snap_words(k->set[i].rows[0]);
        const unsigned blocks = grid(per_sm, words);
        k->bin[e][i]<<<blocks, 32, k->bin_smem[i], next_stream()>>>(a, k->set[i]);
        ++launches;
        if (ends && x) a.snap += (size_t)blocks * words;
    }
    // the join comes after every launch, also on an error, so that the
    // caller's stream waits for all kernels before it frees their buffers
    const cudaError_t err = cudaGetLastError();
    if (x) {
        const int rc = join(x, st);
        if (rc) return rc;
    }
    return err == cudaSuccess ? TPZ_OK : cuda_fail(err, "Smith-Waterman launches");
}

static void pair_args(Args &a, const int8_t *q, const int64_t *qoff, const int32_t *qlen,
                      const int8_t *s, const int64_t *soff, const int32_t *slen, int32_t *score,
                      int32_t *ref_end, int32_t *read_end, int32_t *status) {
    memset(&a, 0, sizeof a);
    a.q = q; a.qoff = qoff; a.qlen = qlen; a.s = s; a.soff = soff; a.slen = slen;
    a.score = score; a.ref_end = ref_end; a.read_end = read_end; a.status = status;
}

int batch_device_x(int64_t n, const int8_t *q, const int64_t *qoff, const int32_t *qlen,
                   const int8_t *s, const int64_t *soff, const int32_t *slen, const int8_t *mat,
                   int go, int ge, int32_t *score, int32_t *ref_end, int32_t *read_end,
                   int32_t *status, cudaStream_t st, const int8_t *xq, const int8_t *xs,
                   int score_only, const int32_t *subset, int64_t nsub, int lane) {
    g_last_launches = 0;
    if (subset && nsub == 0) return TPZ_OK;
    if (n < 0 || n > INT32_MAX / 3 || !mat) { set_error("tpz_sw_batch: bad n or matrix"); return TPZ_E_ARG; }
    if (!(go > ge && ge >= 0 && go <= 255)) {
        set_error("tpz_sw_batch: requires 255 >= gap_open > gap_extend >= 0");
        return TPZ_E_ARG;
    }
    if (n == 0) return TPZ_OK;
    if (!q || !qoff || !qlen || !s || !soff || !slen || !score || !ref_end || !read_end || !status) {
        set_error("tpz_sw_batch: NULL buffer");
        return TPZ_E_ARG;
    }
    const Kernels *k = nullptr;
    Streams *x = nullptr;
    int rc = kernels(&k);
    if (rc || (rc = streams(&x, lane))) return rc;
    keep_pool_memory();
    if (subset) n = nsub;
    // workspace: the stored columns, then the bins and the sorted ids
    const size_t snaps = score_only ? 0 : batch_snap_words(k, n, TPZ_SW_MAX_QLEN);
    uint4 *ws = nullptr;
    TPZ_CUDA(cudaMallocAsync((void **)&ws, sizeof(uint4) * snaps + sizeof(int32_t) * (kBinWords + (size_t)n), st));
    Args a;
    pair_args(a, q, qoff, qlen, s, soff, slen, score, ref_end, read_end, status);
    set_scoring(a, mat, go, ge);
    a.translate = (xq && xs) ? 1 : 0;
    if (a.translate) {
        memcpy(a.xq, xq, 128);
        memcpy(a.xs, xs, 128);
    }
    int64_t launches = 0;
    rc = launch_batch(k, x, a, n, subset, (int32_t *)(ws + snaps), ws, (int64_t)snaps, TPZ_SW_MAX_QLEN, !score_only, st, launches);
    TPZ_CUDA(cudaFreeAsync(ws, st));
    if (rc) return rc;
    g_last_launches = launches;
    return TPZ_OK;
}

int batch_device_grouped(int64_t n, const int8_t *q, const int64_t *qoff, const int32_t *qlen,
                         const int8_t *s, const int64_t *soff, const int32_t *slen,
                         const int8_t *mat, int go, int ge, int32_t *score, int32_t *ref_end,
                         int32_t *read_end, int32_t *status, cudaStream_t st, const int8_t *xq,
                         const int8_t *xs, int score_only, int64_t ngroups,
                         const int64_t *gstart_host, const int32_t *gqlen_host, int long_slen) {
    if (n <= 0) return TPZ_OK;
    if (!(go > ge && ge >= 0 && go <= 255) || !mat) {
        set_error("tpz_sw_batch: requires 255 >= gap_open > gap_extend >= 0");
        return TPZ_E_ARG;
    }
    const Kernels *k = nullptr;
    Streams *x = nullptr;
    int rc = kernels(&k);
    if (rc || (rc = streams(&x, 2))) return rc;
    const int nsm = sm_count();
    const int e = score_only ? 0 : 1;
    Args a;
    pair_args(a, q, qoff, qlen, s, soff, slen, score, ref_end, read_end, status);
    set_scoring(a, mat, go, ge);
    a.translate = (xq && xs) ? 1 : 0;
    if (a.translate) { memcpy(a.xq, xq, 128); memcpy(a.xs, xs, 128); }
    // Chunks of pairs of one query for the query-major kernels (queries with
    // enough pairs, none of which has to have its words to itself); every
    // other pair goes by pair.  A chunk holds at most
    // kQmMaxPairs, and fewer while the blocks of the GPU would not get four
    // each, down to four tasks per warp.
    int64_t cells = 0;                  // pairs * rows, the measure of a chunk's time
    for (int64_t g = 0; g < ngroups; ++g)
        cells += (gstart_host[g + 1] - gstart_host[g]) * gqlen_host[g];
    const int64_t share = cells / (8 * nsm) + 1;
    std::vector<Chunk> chunks[5];       // one stripe, and 2, up to 4, 6, 8 of them
    int min_lanes = 32, max_rows = 1;
    int striped_profile[5] = {0, 0, 0, 0, 0};
    // shared memory of a class's blocks: profile, a warp's letter rings, all
    auto profile = [&](int cls) { return cls ? striped_profile[cls] : profile_bytes(max_rows <= 8 ? 8 : max_rows); };
    auto ring = [&](int cls) { return cls ? kPairRing : (32 / min_lanes) * kPairRing; };
    auto qm_bytes = [&](int cls) { return qm_smem_bytes(profile(cls), ring(cls), cls > 0); };
    std::vector<int32_t> rest;
    for (int64_t g = 0; g < ngroups; ++g) {
        const int64_t c = gstart_host[g + 1] - gstart_host[g];
        if (c <= 0) continue;
        const int ql = gqlen_host[g];
        if (ql < 1 || c < kQmMinPairs || (ql <= kStripeRows ? ql : std::min(ql, long_slen)) > a.steps) {
            for (int64_t k = gstart_host[g]; k < gstart_host[g + 1]; ++k) rest.push_back((int32_t)k);
            continue;
        }
        const int stripes = (ql + kStripeRows - 1) / kStripeRows;
        const int64_t most = std::min<int64_t>(kQmMaxPairs, std::max<int64_t>(8 * kQmWarps, share / ql));
        const int64_t nch = (c + most - 1) / most;
        // more lanes per pair (fewer rows each) while a chunk would leave
        // warps of its block without a task
        int G = stripes > 1 ? 32 : group_lanes(ql);
        while (G < 32 && c / nch < kQmWarps * (64 / G)) G *= 2;
        const int rows = (ql + G * stripes - 1) / (G * stripes);
        const int cls = stripes == 1 ? 0 : stripes == 2 ? 1 : (stripes + 1) / 2;
        for (int64_t i = 0; i < nch; ++i) {
            // equal cuts so that no chunk is much smaller than the others
            const int64_t b0 = gstart_host[g] + c * i / nch, b1 = gstart_host[g] + c * (i + 1) / nch;
            chunks[cls].push_back(Chunk{b0, (int32_t)(b1 - b0), rows, G, stripes});
        }
        if (cls == 0) {
            min_lanes = std::min(min_lanes, G);
            max_rows = std::max(max_rows, rows);
        } else {
            striped_profile[cls] = std::max(striped_profile[cls], stripes * profile_bytes(rows));
        }
    }
    // blocks of each class, and by pair where the boundary rows of its
    // subjects would take too much
    int64_t grids[5] = {};
    int striped = 0;
    for (int cls = 1; cls < 5; ++cls) striped += !chunks[cls].empty();
    for (int cls = 0; cls < 5; ++cls) {
        std::vector<Chunk> &c = chunks[cls];
        if (c.empty()) continue;
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, (const void *)k->qm[e][cls > 0], kQmWarps * 32,
                                                          qm_bytes(cls)) != cudaSuccess || nb < 1)
            nb = 1;
        grids[cls] = std::min<int64_t>((int64_t)nsm * nb, (int64_t)c.size());
        if (cls == 0) continue;
        grids[cls] = boundary_blocks(grids[cls], striped, long_slen, nsm);
        if (grids[cls] > 0) continue;
        for (const Chunk &x : c)
            for (int32_t i = 0; i < x.pairs; ++i) rest.push_back((int32_t)(x.first + i));
        c.clear();
    }
    // one upload: a zero counter per class, the other pairs, the chunks
    // (longest first)
    std::vector<int32_t> head(8, 0);
    head.insert(head.end(), rest.begin(), rest.end());
    if (head.size() & 1) head.push_back(0);
    size_t nchunks = 0;
    for (std::vector<Chunk> &c : chunks) {
        std::sort(c.begin(), c.end(), [](const Chunk &x, const Chunk &y) {
            return (int64_t)x.pairs * x.rows * x.stripes * x.lanes > (int64_t)y.pairs * y.rows * y.stripes * y.lanes;
        });
        nchunks += c.size();
    }
    const size_t hbytes = 4 * head.size();
    std::vector<char> up(hbytes + sizeof(Chunk) * nchunks);
    memcpy(up.data(), head.data(), hbytes);
    size_t at = hbytes;
    for (const std::vector<Chunk> &c : chunks) {
        if (!c.empty()) memcpy(up.data() + at, c.data(), sizeof(Chunk) * c.size());
        at += sizeof(Chunk) * c.size();
    }
    char *dup = nullptr;
    uint2 *dbnd = nullptr;
    auto drop = [&]() {
        if (dup) cudaFreeAsync(dup, st);
        if (dbnd) cudaFreeAsync(dbnd, st);
    };
    TPZ_CUDA(cudaMallocAsync((void **)&dup, up.size(), st));
    if (cudaMemcpyAsync(dup, up.data(), up.size(), cudaMemcpyHostToDevice, st)) {
        drop();
        return cuda_fail(cudaGetLastError(), "batch_device_grouped copies");
    }
    int32_t *dhead = (int32_t *)dup;
    int64_t launches = 0;
    struct Launch { QmArgs g; unsigned grid; int smem, striped; };
    std::vector<Launch> todo;
    int64_t bnd_words = 0, snaps = 0;   // uint2 of boundary rows, uint4 of stored columns
    at = hbytes;
    for (int cls = 0; cls < 5; ++cls) {
        const std::vector<Chunk> &c = chunks[cls];
        if (c.empty()) continue;
        Launch l;
        l.striped = cls > 0;
        l.g.chunks = (const Chunk *)(dup + at);
        at += sizeof(Chunk) * c.size();
        l.g.count = (int)c.size();
        l.g.next = dhead + cls;
        l.g.profile = profile(cls);
        l.g.ring = ring(cls);
        l.smem = qm_bytes(cls);
        l.grid = (unsigned)grids[cls];
        l.g.bnd = nullptr;
        l.g.bnd_cols = 0;
        if (cls) {
            l.g.bnd_cols = std::max(long_slen, 1);
            bnd_words += (kQmWarps * l.g.bnd_cols * l.grid + 1) & ~(int64_t)1;
        }
        if (e) snaps += (int64_t)l.grid * kQmWarps * snap_words(kMaxR);
        todo.push_back(l);
    }
    uint4 *dsnap = nullptr;
    if (bnd_words + snaps > 0) {
        if (cudaMallocAsync((void **)&dbnd, sizeof(uint2) * (size_t)bnd_words + sizeof(uint4) * (size_t)snaps, st)) {
            drop();
            return cuda_fail(cudaGetLastError(), "batch_device_grouped boundary rows");
        }
        dsnap = reinterpret_cast<uint4 *>(dbnd + bnd_words);
        bnd_words = 0;
        for (Launch &l : todo) {
            if (!l.striped) continue;
            l.g.bnd = dbnd + bnd_words;
            bnd_words += (kQmWarps * l.g.bnd_cols * l.grid + 1) & ~(int64_t)1;
        }
    }
    if (!todo.empty()) {
        // the classes with most stripes first: their chunks take longest
        if ((rc = fork(x, st))) { drop(); return rc; }
        int stream = 0;
        for (size_t i = todo.size(); i-- > 0;) {
            const Launch &l = todo[i];
            a.snap = dsnap;
            if (e) dsnap += (size_t)l.grid * kQmWarps * snap_words(kMaxR);
            k->qm[e][l.striped]<<<l.grid, kQmWarps * 32, l.smem, x->aux[stream++ % kAuxStreams]>>>(a, l.g);
            ++launches;
        }
    }
    rc = batch_device_x(n, q, qoff, qlen, s, soff, slen, mat, go, ge, score, ref_end, read_end,
                        status, st, xq, xs, score_only, dhead + 8, (int64_t)rest.size());
    launches += g_last_launches;
    if (!todo.empty()) {
        const int rj = join(x, st);
        if (rc == TPZ_OK) rc = rj;
    }
    drop();
    if (rc) return rc;
    TPZ_CUDA(cudaGetLastError());
    g_last_launches = launches;
    return TPZ_OK;
}

}  // namespace sw
}  // namespace tpz

// ------------------------------------------------------------------ C ABI

namespace {

// Grow-only device buffers reused by the host entry point, and its streams:
// two for the kernels (one per chunk), one for host-to-device and one for
// device-to-host copies, so that a chunk's copies run beside another
// chunk's kernels.
struct HostBatchBuffers {
    void *p = nullptr;
    size_t cap = 0;
    int dev = -1;
    cudaStream_t compute = nullptr, compute2 = nullptr, h2d = nullptr, d2h = nullptr;
    cudaEvent_t ev[8] = {};
};
thread_local HostBatchBuffers g_hb;

int ensure(size_t bytes) {
    int dev = 0;
    TPZ_CUDA(cudaGetDevice(&dev));
    if (g_hb.compute && g_hb.dev != dev) {
        // streams and events belong to the device they were made on
        cudaStreamDestroy(g_hb.compute);
        cudaStreamDestroy(g_hb.compute2);
        cudaStreamDestroy(g_hb.h2d);
        cudaStreamDestroy(g_hb.d2h);
        for (cudaEvent_t &e : g_hb.ev) { cudaEventDestroy(e); e = nullptr; }
        g_hb.compute = g_hb.compute2 = g_hb.h2d = g_hb.d2h = nullptr;
    }
    if (!g_hb.compute) {
        TPZ_CUDA(cudaStreamCreateWithFlags(&g_hb.compute, cudaStreamNonBlocking));
        TPZ_CUDA(cudaStreamCreateWithFlags(&g_hb.compute2, cudaStreamNonBlocking));
        TPZ_CUDA(cudaStreamCreateWithFlags(&g_hb.h2d, cudaStreamNonBlocking));
        TPZ_CUDA(cudaStreamCreateWithFlags(&g_hb.d2h, cudaStreamNonBlocking));
        for (cudaEvent_t &e : g_hb.ev) TPZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (g_hb.p && (g_hb.cap >= bytes) && g_hb.dev == dev) return TPZ_OK;
    if (g_hb.p) cudaFree(g_hb.p);
    g_hb.p = nullptr;
    g_hb.cap = 0;
    TPZ_CUDA(cudaMalloc(&g_hb.p, bytes));
    g_hb.cap = bytes;
    g_hb.dev = dev;
    return TPZ_OK;
}

// Residue byte ranges [lo, hi) of q and s that the pairs [i0, i1) read, and
// the first pair outside the limits (-1: none).
struct Span {
    int64_t qlo, qhi, slo, shi, bad;
};

Span scan_pairs(int64_t i0, int64_t i1, const int64_t *qoff, const int32_t *qlen,
                const int64_t *soff, const int32_t *slen) {
    Span r{INT64_MAX, 0, INT64_MAX, 0, -1};
    for (int64_t i = i0; i < i1; ++i) {
        if (qlen[i] < 1 || qlen[i] > TPZ_SW_MAX_QLEN || slen[i] < 0 || slen[i] >= TPZ_SW_MAX_SLEN ||
            qoff[i] < 0 || soff[i] < 0) {
            r.bad = i;
            return r;
        }
        r.qlo = std::min(r.qlo, qoff[i]);
        r.qhi = std::max(r.qhi, qoff[i] + qlen[i]);
        if (slen[i] > 0) {
            r.slo = std::min(r.slo, soff[i]);
            r.shi = std::max(r.shi, soff[i] + slen[i]);
        }
    }
    if (r.slo > r.shi) r.slo = r.shi;
    return r;
}

}  // namespace

extern "C" {

int tpz_sw_batch_device(int64_t n, const int8_t *q, const int64_t *qoff, const int32_t *qlen,
                        const int8_t *s, const int64_t *soff, const int32_t *slen,
                        const int8_t *mat625_host, int gap_open, int gap_extend,
                        int32_t *score, int32_t *ref_end, int32_t *read_end, int32_t *status,
                        void *stream) {
    return tpz::sw::batch_device_x(n, q, qoff, qlen, s, soff, slen, mat625_host, gap_open,
                                   gap_extend, score, ref_end, read_end, status,
                                   (cudaStream_t)stream, nullptr, nullptr, 0);
}

int tpz_sw_batch_host(int64_t n, const int8_t *q, const int64_t *qoff, const int32_t *qlen,
                      const int8_t *s, const int64_t *soff, const int32_t *slen,
                      const int8_t *mat625, int gap_open, int gap_extend,
                      int32_t *score, int32_t *ref_end, int32_t *read_end, int32_t *status) {
    if (n < 0 || !mat625) { tpz::set_error("tpz_sw_batch_host: n < 0 or NULL matrix"); return TPZ_E_ARG; }
    if (!(gap_open > gap_extend && gap_extend >= 0 && gap_open <= 255)) {
        tpz::set_error("tpz_sw_batch_host: requires 255 >= gap_open > gap_extend >= 0");
        return TPZ_E_ARG;
    }
    if (n == 0) return TPZ_OK;
    // Pairs go in chunks of growing size: the copy in of the inputs runs
    // several times faster than the kernels, so each chunk's inputs arrive
    // while the chunk before it computes and the GPU waits only for the first
    // one's.  Consecutive chunks run on alternating streams (lanes), so a
    // chunk's kernels fill the GPU while the previous chunk's last tasks
    // finish; each chunk's results are copied out as soon as they are done.
    // A chunk also pays its longest task: 1/8 and 7/8 took 6.3 ms at 70,000
    // pairs against 7.2 ms for 1/16, 3/16 and 12/16, 12.5 against 12.8 ms at
    // 150,000, and 23.3 against 22.5 ms at 300,000.
    constexpr int kMaxChunks = 4;
    int64_t cut[kMaxChunks + 1] = {0, n};
    int nch = 1;
    if (n >= 200000) {
        cut[1] = n / 16; cut[2] = 4 * (n / 16); cut[3] = n;
        nch = 3;
    } else if (n >= 65536) {
        cut[1] = n / 8; cut[2] = n;
        nch = 2;
    }
    // host-side validation and the byte ranges each chunk reads: the chunks
    // cut into pieces in proportion to their size, scanned on up to 16 host
    // threads, and merged per chunk
    Span sp[kMaxChunks];
    {
        const int nt = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
        struct Piece { int c; int64_t i0, i1; Span r; };
        std::vector<Piece> pieces;
        for (int c = 0; c < nch; ++c) {
            const int64_t m = cut[c + 1] - cut[c];
            // at least 32,768 pairs per piece: a thread costs more than that
            const int64_t k = std::max<int64_t>(1, std::min((nt * m + n - 1) / n, m / 32768));
            for (int64_t p = 0; p < k; ++p)
                pieces.push_back({c, cut[c] + m * p / k, cut[c] + m * (p + 1) / k, Span{}});
        }
        std::vector<std::thread> th;
        for (size_t p = 1; p < pieces.size(); ++p)
            th.emplace_back([&, p]() {
                pieces[p].r = scan_pairs(pieces[p].i0, pieces[p].i1, qoff, qlen, soff, slen);
            });
        pieces[0].r = scan_pairs(pieces[0].i0, pieces[0].i1, qoff, qlen, soff, slen);
        for (auto &t : th) t.join();
        for (int c = 0; c < nch; ++c) sp[c] = Span{INT64_MAX, 0, INT64_MAX, 0, -1};
        for (const Piece &p : pieces) {
            Span &d = sp[p.c];
            const Span &r = p.r;
            if (r.bad >= 0 && (d.bad < 0 || r.bad < d.bad)) d.bad = r.bad;
            if (p.i1 > p.i0) {
                d.qlo = std::min(d.qlo, r.qlo);
                d.qhi = std::max(d.qhi, r.qhi);
                if (r.shi > r.slo || r.shi > 0) {
                    d.slo = std::min(d.slo, r.slo);
                    d.shi = std::max(d.shi, r.shi);
                }
            }
        }
        for (int c = 0; c < nch; ++c)
            if (sp[c].slo > sp[c].shi) sp[c].slo = sp[c].shi;
    }
    int64_t qbytes = 0, sbytes = 0;
    for (int c = 0; c < nch; ++c) {
        if (sp[c].bad >= 0) {
            const int64_t i = sp[c].bad;
            char buf[160];
            snprintf(buf, sizeof buf, "tpz_sw_batch_host: pair %lld outside the limits (qlen %d, slen %d)",
                     (long long)i, qlen[i], slen[i]);
            tpz::set_error(buf);
            return TPZ_E_RANGE;
        }
        qbytes = std::max(qbytes, sp[c].qhi);
        sbytes = std::max(sbytes, sp[c].shi);
    }
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t bq = al(qbytes), bs = al(sbytes), b8 = al(8 * (size_t)n), b4 = al(4 * (size_t)n);
    const size_t total = bq + bs + 2 * b8 + 6 * b4;
    int rc = ensure(total);
    if (rc) return rc;
    char *d = (char *)g_hb.p;
    int8_t *dq = (int8_t *)d; d += bq;
    int8_t *ds = (int8_t *)d; d += bs;
    int64_t *dqoff = (int64_t *)d; d += b8;
    int64_t *dsoff = (int64_t *)d; d += b8;
    int32_t *dqlen = (int32_t *)d; d += b4;
    int32_t *dslen = (int32_t *)d; d += b4;
    int32_t *dsc = (int32_t *)d; d += b4;
    int32_t *dre = (int32_t *)d; d += b4;
    int32_t *drd = (int32_t *)d; d += b4;
    int32_t *dst = (int32_t *)d; d += b4;
    cudaStream_t cst[2] = {g_hb.compute, g_hb.compute2}, hs = g_hb.h2d, os = g_hb.d2h;
    // The device copies of q and s keep the host offsets.  Each chunk copies
    // the part of its byte range not copied yet: the copied part is kept as
    // one interval [lo, hi) that grows to cover every range seen (a gap
    // between ranges is copied too, which is harmless).
    int64_t qc_lo = 0, qc_hi = 0, sc_lo = 0, sc_hi = 0;
    auto copy_new = [&](const int8_t *src, int8_t *dst, int64_t lo, int64_t hi, int64_t &c_lo,
                        int64_t &c_hi) -> cudaError_t {
        if (hi <= lo) return cudaSuccess;
        if (c_hi <= c_lo) {
            c_lo = lo; c_hi = hi;
            return cudaMemcpyAsync(dst + lo, src + lo, hi - lo, cudaMemcpyHostToDevice, hs);
        }
        cudaError_t e = cudaSuccess;
        if (lo < c_lo) {
            e = cudaMemcpyAsync(dst + lo, src + lo, c_lo - lo, cudaMemcpyHostToDevice, hs);
            c_lo = lo;
        }
        if (e == cudaSuccess && hi > c_hi) {
            e = cudaMemcpyAsync(dst + c_hi, src + c_hi, hi - c_hi, cudaMemcpyHostToDevice, hs);
            c_hi = hi;
        }
        return e;
    };
    static_assert(2 * kMaxChunks <= (int)(sizeof g_hb.ev / sizeof g_hb.ev[0]), "events per chunk");
    cudaEvent_t *in_ready = g_hb.ev, *done = g_hb.ev + kMaxChunks;
    for (int c = 0; c < nch; ++c) {
        const int64_t a = cut[c], m = cut[c + 1] - cut[c];
        TPZ_CUDA(copy_new(q, dq, sp[c].qlo, sp[c].qhi, qc_lo, qc_hi));
        TPZ_CUDA(copy_new(s, ds, sp[c].slo, sp[c].shi, sc_lo, sc_hi));
        TPZ_CUDA(cudaMemcpyAsync(dqoff + a, qoff + a, 8 * m, cudaMemcpyHostToDevice, hs));
        TPZ_CUDA(cudaMemcpyAsync(dsoff + a, soff + a, 8 * m, cudaMemcpyHostToDevice, hs));
        TPZ_CUDA(cudaMemcpyAsync(dqlen + a, qlen + a, 4 * m, cudaMemcpyHostToDevice, hs));
        TPZ_CUDA(cudaMemcpyAsync(dslen + a, slen + a, 4 * m, cudaMemcpyHostToDevice, hs));
        TPZ_CUDA(cudaEventRecord(in_ready[c], hs));
    }
    for (int c = 0; c < nch; ++c) {
        const int64_t a = cut[c], m = cut[c + 1] - cut[c];
        cudaStream_t cs = cst[c & 1];
        TPZ_CUDA(cudaStreamWaitEvent(cs, in_ready[c], 0));
        rc = tpz::sw::batch_device_x(m, dq, dqoff + a, dqlen + a, ds, dsoff + a, dslen + a,
                                     mat625, gap_open, gap_extend, dsc + a, dre + a, drd + a,
                                     dst + a, cs, nullptr, nullptr, 0, nullptr, 0, c & 1);
        if (rc) {
            cudaStreamSynchronize(hs);
            cudaStreamSynchronize(cst[0]);
            cudaStreamSynchronize(cst[1]);
            return rc;
        }
        TPZ_CUDA(cudaEventRecord(done[c], cs));
        TPZ_CUDA(cudaStreamWaitEvent(os, done[c], 0));
        TPZ_CUDA(cudaMemcpyAsync(score + a, dsc + a, 4 * m, cudaMemcpyDeviceToHost, os));
        TPZ_CUDA(cudaMemcpyAsync(ref_end + a, dre + a, 4 * m, cudaMemcpyDeviceToHost, os));
        TPZ_CUDA(cudaMemcpyAsync(read_end + a, drd + a, 4 * m, cudaMemcpyDeviceToHost, os));
        TPZ_CUDA(cudaMemcpyAsync(status + a, dst + a, 4 * m, cudaMemcpyDeviceToHost, os));
    }
    TPZ_CUDA(cudaStreamSynchronize(os));
    TPZ_CUDA(cudaStreamSynchronize(cst[0]));
    TPZ_CUDA(cudaStreamSynchronize(cst[1]));
    return TPZ_OK;
}

int64_t tpz_sw_last_launches(void) { return tpz::sw::g_last_launches; }

int tpz_sw_align_one(const int8_t *q, int32_t qlen, const int8_t *s, int32_t slen,
                     const int8_t *mat625_host, int gap_open, int gap_extend, int32_t *out4,
                     void *stream) {
    using namespace tpz::sw;
    if (!q || !s || !out4 || !mat625_host || qlen < 1 || qlen > kOneMaxQlen || slen < 0 ||
        slen >= TPZ_SW_MAX_SLEN) {
        tpz::set_error("tpz_sw_align_one: need 1 <= qlen <= 1024, 0 <= slen < 2^24, non-NULL buffers");
        return TPZ_E_ARG;
    }
    if (!(gap_open > gap_extend && gap_extend >= 0 && gap_open <= 255)) {
        tpz::set_error("tpz_sw_align_one: requires 255 >= gap_open > gap_extend >= 0");
        return TPZ_E_ARG;
    }
    const Kernels *k = nullptr;
    int rc = kernels(&k);
    if (rc) return rc;
    int mx = 0;
    for (int i = 0; i < 625; ++i) mx = std::max<int>(mx, mat625_host[i]);
    if ((int64_t)qlen * mx >= kBig) {
        tpz::set_error("tpz_sw_align_one: matrix entries too large for 16-bit scores at this length");
        return TPZ_E_ARG;
    }
    Args a;
    pair_args(a, q, nullptr, nullptr, s, nullptr, nullptr, out4, out4 + 1, out4 + 2, out4 + 3);
    set_scoring(a, mat625_host, gap_open, gap_extend);
    const int W = qlen <= 512 ? 1 : 2;
    sw_one_kernel<<<1, 32 * W, stripe_smem(8, W), (cudaStream_t)stream>>>(a, qlen, slen);
    TPZ_CUDA(cudaGetLastError());
    return TPZ_OK;
}

int tpz_dpx_probe(int64_t blocks, int iters, uint32_t *out, void *stream, int64_t *ops) {
    if (blocks < 1 || iters < 1 || !out || !ops) { tpz::set_error("tpz_dpx_probe: bad argument"); return TPZ_E_ARG; }
    tpz::sw::dpx_probe_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
        iters, 0x00010001u, 0x80008000u, out);
    TPZ_CUDA(cudaGetLastError());
    *ops = blocks * 256 * (int64_t)iters * tpz::sw::kProbeChains;
    return TPZ_OK;
}

}  // extern "C"

// ------------------------------------------------- allocation-free variant
//
// Some callers cannot let a library allocate device memory on their request
// path: a search server that has planned its HBM around a resident index and
// a fixed set of in-flight batches (an allocation there can fail under
// memory pressure halfway through a request), or a host loop that must not
// stall on the allocator -- cudaMalloc/cudaFree synchronize the device and
// would serialize every concurrent stream.  For them the batched SW below
// keeps its scratch (bin counts, bin cursors, the sorted pair list and the
// stored columns) in one statically sized device array instead of a per-call
// allocation, and enqueues everything on the caller's stream only.

namespace tpz {
namespace sw {

constexpr int64_t kNoAllocMaxPairs = TPZ_SW_NOALLOC_MAX_PAIRS;
constexpr int kNoAllocMaxQlen = TPZ_SW_NOALLOC_MAX_QLEN;   // one stripe
// the stated entry limit keeps every score below kBig
static_assert((int64_t)kNoAllocMaxQlen * TPZ_SW_NOALLOC_MAX_ENTRY < kBig &&
                  (int64_t)kNoAllocMaxQlen * (TPZ_SW_NOALLOC_MAX_ENTRY + 1) >= kBig,
              "TPZ_SW_NOALLOC_MAX_ENTRY");

// One copy per device that loads the library, kept until the process exits.
// Behind the bins: the columns stored by the largest by-pair kernel on 148
// SMs (a kernel launches no more blocks than there is room for).
constexpr size_t kNoAllocBins = (kBinWords + (size_t)kNoAllocMaxPairs + 3) & ~(size_t)3;
constexpr size_t kNoAllocSnaps = 148 * 4 * (size_t)snap_words(kMaxR);
static __device__ __align__(256) int32_t g_noalloc_scratch[kNoAllocBins + 4 * kNoAllocSnaps];

// Device address of the static scratch array of the current device (host
// code cannot use the array's name as a device pointer).
static int noalloc_scratch(int32_t **out) {
    static std::mutex mu;
    static std::vector<int32_t *> per_dev;
    int dev = 0;
    TPZ_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if ((int)per_dev.size() <= dev) per_dev.resize(dev + 1, nullptr);
    if (!per_dev[dev]) TPZ_CUDA(cudaGetSymbolAddress((void **)&per_dev[dev], g_noalloc_scratch));
    *out = per_dev[dev];
    return TPZ_OK;
}

}  // namespace sw
}  // namespace tpz

extern "C" int tpz_sw_batch_device_noalloc(int64_t n, const int8_t *q, const int64_t *qoff,
                                           const int32_t *qlen, const int8_t *s,
                                           const int64_t *soff, const int32_t *slen,
                                           const int8_t *mat625_host, int gap_open,
                                           int gap_extend, int32_t *score, int32_t *ref_end,
                                           int32_t *read_end, int32_t *status, void *stream) {
    using namespace tpz::sw;
    if (n < 0 || !mat625_host) {
        tpz::set_error("tpz_sw_batch_device_noalloc: n < 0 or NULL matrix");
        return TPZ_E_ARG;
    }
    if (n > kNoAllocMaxPairs) {
        char buf[200];
        snprintf(buf, sizeof buf,
                 "tpz_sw_batch_device_noalloc: %lld pairs exceed the fixed scratch of %lld pairs; "
                 "split the batch or use tpz_sw_batch_device",
                 (long long)n, (long long)kNoAllocMaxPairs);
        tpz::set_error(buf);
        return TPZ_E_RANGE;
    }
    if (!(gap_open > gap_extend && gap_extend >= 0 && gap_open <= 255)) {
        tpz::set_error("tpz_sw_batch_device_noalloc: requires 255 >= gap_open > gap_extend >= 0");
        return TPZ_E_ARG;
    }
    if (n == 0) return TPZ_OK;
    if (!q || !qoff || !qlen || !s || !soff || !slen || !score || !ref_end || !read_end || !status) {
        tpz::set_error("tpz_sw_batch_device_noalloc: NULL buffer");
        return TPZ_E_ARG;
    }
    // the stated matrix limit of this call
    int mx = 0;
    for (int i = 0; i < 625; ++i) mx = std::max<int>(mx, mat625_host[i]);
    if ((int64_t)kNoAllocMaxQlen * mx >= kBig) {
        char buf[200];
        snprintf(buf, sizeof buf,
                 "tpz_sw_batch_device_noalloc: largest matrix entry %d is too large for exact "
                 "16-bit scores of %d-residue queries (limit %d); use tpz_sw_batch_device",
                 mx, kNoAllocMaxQlen, TPZ_SW_NOALLOC_MAX_ENTRY);
        tpz::set_error(buf);
        return TPZ_E_ARG;
    }
    const Kernels *k = nullptr;
    int32_t *ws = nullptr;
    int rc = kernels(&k);
    if (rc || (rc = noalloc_scratch(&ws))) return rc;
    Args a;
    pair_args(a, q, qoff, qlen, s, soff, slen, score, ref_end, read_end, status);
    set_scoring(a, mat625_host, gap_open, gap_extend);
    int64_t launches = 0;
    return launch_batch(k, nullptr, a, n, nullptr, ws, (uint4 *)(ws + kNoAllocBins), (int64_t)kNoAllocSnaps,
                        kNoAllocMaxQlen, true, (cudaStream_t)stream, launches);
}
