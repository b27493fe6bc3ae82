// sw_core.cuh -- the Smith-Waterman step shared by the batch kernels.
//
// Result semantics: exactly those of TOPAZ's striped SSW calls
//   ssw_init(q, qlen, mat, 25, 2); ssw_align(prof, s, slen, go, ge, 0, 0, 0, 15)
// (src/ssw.c:799-897): the u8 pass, the i16 pass when the u8 pass saturates
// (max + bias >= 255), and the drop when the i16 pass reaches 32767.
//
// One pass gives all of it.  The striped passes split the query into 16 (u8)
// or 8 (i16) lanes of consecutive rows and feed E from a main-loop H that
// holds only the vertical gaps opened inside a lane, so on paper the lane
// length is part of the recurrence:
//   Hp(r,c) = max(0, H(r-1,c-1) + M, E(r,c), Fm(r,c)),  H = max(Hp, F)
//   E(r,c+1) = max(E(r,c) - ge, Hp(r,c) - go),  Fm cleared at lane starts
// But H does not depend on which vertical gaps E sees.  Feed E from
// X = max(0, D + M, E) alone (the least), or from the full H (textbook
// Gotoh, the most); with go >= ge both give the same H and F in every cell:
// the only paths the first one lacks leave a vertical gap of k rows straight
// into a horizontal gap of l columns, and the same cells are joined at the
// same cost by the horizontal gap first and the vertical one second, which
// it has (E(r-k, c+l) feeds X, and X feeds F).  Every in-lane Fm lies between
// the two, and all operations are monotone, so the u8 pass, the i16 pass and
// the recurrence below agree on every H: the saturated pairs need no second
// pass and Fm is gone.  (Checked against the lane-length oracle in
// tests/test_sw_recurrence.py, over matrices and gaps chosen to be hostile.)
//   X = max(D + M, E);  Xg = X - go
//   H = max(X, F, 0);  E' = max(E - ge, Xg);  F' = max(F - ge, Xg)
// ref_end is the first column holding the maximum H, read_end the smallest
// row holding it there (src/ssw.c:264-297).
//
// Arithmetic: two alignments (or two row ranges of one) ride in the halves
// of u16x2 words, every value raised by `floor` (= the zero of a score).
// floor >= go + ge - min(M), so X - go does not borrow while no value passes
// 65,535: it is one 32-bit addition, which the compiler may put beside the
// ALU pipe -- the bound: its packed min/max/add and PRMT issue at 16 lanes a
// clock and scheduler -- and leaves that with 5.5 operations per cell pair:
// PRMT (profile bytes), X, H, E, F and half a column maximum.  (With Fm, the
// lane starts and X - go on the same pipe it was 8.5, and 1.3 times the cells
// because saturated pairs ran twice.)  A score that reaches 32767 is final
// (the pair is dropped) however far its own 16 bits run on, so nothing is
// recomputed in wider arithmetic.  But a half that wraps can leave a cell
// below go, whose subtraction borrows from the other half: a pair that may
// score past 65,535 - floor (shared_steps in sw_plan.h) takes the stripe
// form, where both halves are its own.
//
// End coordinates: each lane keeps its running maximum of X (the alignment's
// maximum is an X: F and E only hold less than an X before them).  A rise is
// looked at only when it reaches the group maximum of the last refresh (every
// 32 steps; less cannot be the alignment's maximum); then the lane stores its
// column of H, and the row is looked up once, in the last column stored.  A
// rise so costs R / 4 stores that nothing waits for.  (Of the steps of the
// 200,000-pair case 31 % have one in some lane of the warp.  Looking the row
// up at once took 1.5 ALU operations per row and their latency: 11.1 ms
// against 9.0 ms without ends.  Carrying it in the low bits of the maximum,
// one more FMA-pipe operation per cell pair, took 12.5 against 11.6 cycles
// per row with four warps per scheduler and 16.3 against 12.8 with one.)
#pragma once

#include "sw_plan.h"
#include "tpz_common.cuh"

namespace tpz {
namespace sw {

constexpr int kLetters = 26;        // 25 matrix columns + the pad letter
constexpr int kPadLetter = 25;      // subject column past a pair's end
// transposed matrix in shared memory: 26 query letters x 26 subject letters,
// rows of 9 words (an odd stride keeps the lanes' rows on different banks)
constexpr int kMatWords = 9;
constexpr int kMatBytes = 960;
static_assert(kLetters * kMatWords * 4 <= kMatBytes, "matrix table");
constexpr int kRingCols = 128;      // subject columns kept per ring

// profile words (4 rows each) per lane, and bytes of one warp's profile
__host__ __device__ constexpr int words_for(int R) { return (R + 3) / 4; }
__host__ __device__ constexpr int profile_bytes(int R) { return kLetters * words_for(R) * 128; }

struct Args {
    const int8_t *q;
    const int64_t *qoff;
    const int32_t *qlen;
    const int8_t *s;
    const int64_t *soff;
    const int32_t *slen;
    int32_t *score, *ref_end, *read_end, *status;
    const int32_t *sorted;   // pair ids sorted by bin
    const int32_t *rinfo;    // per row bin: [start, count]
    int32_t *next_task;      // per row bin: task counter
    int gap_open, gap_extend;
    int floor;               // the zero of every stored value
    int steps;               // diagonal steps that 16 bits hold (shared_steps)
    uint4 *snap;             // columns stored at a rise: snap_words() per warp
    int translate;           // 1: q/s bytes go through xq/xs first
    int8_t mat[625];
    int8_t xq[128], xs[128]; // byte -> matrix index (internal alphabet inputs)
};

// gap costs, floor and matrix of a launch
inline void set_scoring(Args &a, const int8_t *mat, int go, int ge) {
    int mn = kPadScore, mx = 0;
    for (int i = 0; i < 625; ++i) {
        mn = mat[i] < mn ? mat[i] : mn;
        mx = mat[i] > mx ? mat[i] : mx;
        a.mat[i] = mat[i];
    }
    a.gap_open = go;
    a.gap_extend = ge;
    a.floor = go + ge - mn;                 // <= 255 + 254 + 128
    a.steps = shared_steps(a.floor, mx);
}

__device__ __forceinline__ uint32_t both(uint32_t x) { return x | (x << 16); }
__device__ __forceinline__ uint32_t lo16(uint32_t x) { return x & 0xFFFFu; }
__device__ __forceinline__ uint32_t hi16(uint32_t x) { return x >> 16; }

__device__ __forceinline__ uint32_t max2u(uint32_t a, uint32_t b) { return __vimax3_u16x2(a, b, b); }

// x * m + c on the FMA pipe
__device__ __forceinline__ uint32_t mad(uint32_t x, uint32_t m, uint32_t c) {
    uint32_t d;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(m), "r"(c));
    return d;
}

__device__ __forceinline__ uint64_t best_key(int v, int col, int row) {
    return v > 0 ? ((uint64_t)v << 40) | ((uint64_t)(0xFFFFFF - col) << 16) |
                       (uint64_t)(0xFFFF - row)
                 : 0ull;
}

// transposed matrix with pad row and pad column (every thread of the block;
// the caller synchronizes)
__device__ __forceinline__ void load_matrix(const Args &a, uint8_t *matT) {
    for (int i = threadIdx.x; i < kLetters * kMatWords * 4; i += blockDim.x) {
        const int ql = i / (kMatWords * 4), sl = i % (kMatWords * 4);
        matT[i] = (uint8_t)((ql < 25 && sl < 25) ? a.mat[sl * 25 + ql] : (int8_t)kPadScore);
    }
}

// matrix index of a query residue; pad rows and bytes outside the alphabet
// take the pad row
__device__ __forceinline__ int query_letter(const Args &a, int x) {
    if (a.translate && x >= 0) x = a.xq[x & 127];
    return (unsigned)x >= 25u ? kPadLetter : x;
}

// Profile word w (rows with matrix indices x0..x3) of every letter, at
// prof[l * W * 128]: the rows' matrix rows are read as words and transposed
// 4x4 with PRMT, 2.5 operations per profile word against a byte load, a
// select and a shift for each byte.
template <int W>
__device__ __forceinline__ void build_word(const uint8_t *matT, int x0, int x1, int x2, int x3,
                                           uint8_t *p) {
    const uint32_t *m = reinterpret_cast<const uint32_t *>(matT);
    const uint32_t *m0 = m + x0 * kMatWords, *m1 = m + x1 * kMatWords;
    const uint32_t *m2 = m + x2 * kMatWords, *m3 = m + x3 * kMatWords;
#pragma unroll 1
    for (int l = 0; l < 28; l += 4) {
        const uint32_t r0 = m0[l >> 2], r1 = m1[l >> 2], r2 = m2[l >> 2], r3 = m3[l >> 2];
        const uint32_t t0 = prmt(r0, r1, 0x5140), t1 = prmt(r2, r3, 0x5140);
        const uint32_t t2 = prmt(r0, r1, 0x7362), t3 = prmt(r2, r3, 0x7362);
        *reinterpret_cast<uint32_t *>(p) = prmt(t0, t1, 0x5410);
        *reinterpret_cast<uint32_t *>(p + W * 128) = prmt(t0, t1, 0x7632);
        if (l < 24) {
            *reinterpret_cast<uint32_t *>(p + 2 * W * 128) = prmt(t2, t3, 0x5410);
            *reinterpret_cast<uint32_t *>(p + 3 * W * 128) = prmt(t2, t3, 0x7632);
        }
        p += 4 * W * 128;
    }
}

// The profile of rows [i0, i0 + R) of a query, int8, word w of letter l at
// prof[(l * W + w) * 128] (prof points at this lane's column of the warp's
// profile, so the 32 loads of a step never share a bank).
template <int R>
__device__ __forceinline__ void build_profile(const Args &a, const int8_t *q, int ql, int i0,
                                              const uint8_t *matT, uint8_t *prof) {
    constexpr int W = words_for(R);
    int x[4 * W];
#pragma unroll
    for (int r = 0; r < 4 * W; ++r) x[r] = (r < R && i0 + r < ql) ? (int)q[i0 + r] : -1;
#pragma unroll
    for (int w = 0; w < W; ++w)
        build_word<W>(matT, query_letter(a, x[4 * w]), query_letter(a, x[4 * w + 1]),
                      query_letter(a, x[4 * w + 2]), query_letter(a, x[4 * w + 3]), prof + w * 128);
}

// profile offset (bytes) of the letter of subject column c
template <int R>
__device__ __forceinline__ uint16_t letter_offset(const Args &a, const int8_t *s, int sl, int c) {
    int l = kPadLetter;
    if (c < sl) {
        l = s[c];
        if (a.translate) l = a.xs[l & 127];
        if ((unsigned)l >= 25u) l = kPadLetter;
    }
    return (uint16_t)(l * (words_for(R) * 128));
}

// Where a warp's wavefront finds its inputs.
struct Flow {
    const uint8_t *profA, *profB;     // this lane's profile columns (low, high half)
    const uint16_t *ringA, *ringB;    // letter offsets by column % kRingCols
    int lag;                          // step k works on column k - lag (low half)
    int lagB;                         // the high half's column is that much earlier
    int width;                        // lanes of a group (pair tasks)
    uint32_t mul, add;                // the incoming word is shuffled * mul + add
    // the row above lane 0's first, by column: null, or (one alignment) a ring
    // of H | F << 16, or (two) a ring of [H, F]
    const uint32_t *bnd;
    const uint2 *bnd2;
    int bnd_end;                      // its columns
    uint4 *snap;                      // this lane's stored columns
};

// One lane's state between steps.
template <int R>
struct Lane {
    static constexpr int W = words_for(R);
    uint32_t E[R], H[R];
    uint32_t diag, outH, outF;
    uint32_t run;                 // running maxima of X
    int colA, colB;               // the columns that reached them
    uint32_t wa[W], wb[W];        // profile words of the next step's column
    uint32_t nA, nB;              // profile offsets of the column after it

    __device__ __forceinline__ void load_words(const Flow &f, uint32_t (&a)[W], uint32_t (&b)[W]) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            a[w] = *reinterpret_cast<const uint32_t *>(f.profA + nA + 128 * w);
            b[w] = *reinterpret_cast<const uint32_t *>(f.profB + nB + 128 * w);
        }
    }
    __device__ __forceinline__ void load_offsets(const Flow &f, int j) {
        nA = f.ringA[j & (kRingCols - 1)];
        nB = f.ringB[(j - f.lagB) & (kRingCols - 1)];
    }
    // state before column 0; the ring holds the first columns
    __device__ __forceinline__ void start(const Args &a, const Flow &f) {
        const uint32_t z = both((uint32_t)a.floor);
#pragma unroll
        for (int r = 0; r < R; ++r) { E[r] = z; H[r] = z; }
        diag = outH = outF = run = z;
        colA = colB = 0;
        load_offsets(f, -f.lag);
        load_words(f, wa, wb);
        load_offsets(f, 1 - f.lag);
    }
    // this column of H
    __device__ __forceinline__ void store(uint4 *snap) const {
#pragma unroll
        for (int w = 0; w < W; ++w)
            snap[32 * w] = make_uint4(H[4 * w], 4 * w + 1 < R ? H[4 * w + 1 < R ? 4 * w + 1 : 0] : 0u,
                                      4 * w + 2 < R ? H[4 * w + 2 < R ? 4 * w + 2 : 0] : 0u,
                                      4 * w + 3 < R ? H[4 * w + 3 < R ? 4 * w + 3 : 0] : 0u);
    }
    // the first row of a stored column that holds the running maximum
    __device__ __forceinline__ int find_row(const uint4 *snap, bool high) const {
        const uint32_t v = high ? hi16(run) : lo16(run);
        int row = 0;
#pragma unroll
        for (int w = W - 1; w >= 0; --w) {
            const uint4 x = snap[32 * w];
            const uint32_t h[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 3; k >= 0; --k)
                if ((high ? hi16(h[k]) : lo16(h[k])) == v) row = 4 * w + k;
        }
        return row;
    }
};

// words of uint4 a warp stores columns in: the low half's, then the high
// half's, by word and lane
__host__ __device__ constexpr int snap_words(int R) { return 2 * 32 * words_for(R); }

// Step k of a lane: column j = k - lag.  Every lane computes every step: a
// lane before its first column sees pad letters and floor inputs, so its H
// stays at the floor; past the subject's end the pad columns only hold
// values below some real cell's, which can never be the maximum.
// LONG: the halves are rows [0, 32R) and [32R, 64R) of one stripe, the high
// half 32 columns behind; lane 0 takes the low half from the stripe above
// (f.bnd) and the high half from lane 31's low half.
// STRIPED: two alignments, lane 0 below another stripe of each (f.bnd2).
template <int R, bool ENDS, bool LONG, bool STRIPED>
__device__ __forceinline__ void step(Lane<R> &L, const Args &a, const Flow &f, int j,
                                     const uint32_t (&cwa)[Lane<R>::W],
                                     const uint32_t (&cwb)[Lane<R>::W],
                                     uint32_t (&nwa)[Lane<R>::W], uint32_t (&nwb)[Lane<R>::W]) {
    // sign-extend byte r % 4 of the A word into the low half, of the B word
    // into the high half
    constexpr uint32_t SEL[4] = {0xC480u, 0xD591u, 0xE6A2u, 0xF7B3u};
    const uint32_t Z = both((uint32_t)a.floor);
    const uint32_t NGE = both((uint32_t)(-a.gap_extend) & 0xFFFFu);
    const uint32_t NGO = 0u - both((uint32_t)a.gap_open);      // 32-bit: no borrow between halves
    uint32_t inH, inF;
    if (LONG) {
        const int src = (threadIdx.x + 31) & 31;
        const uint32_t vH = __shfl_sync(0xFFFFFFFFu, L.outH, src);
        const uint32_t vF = __shfl_sync(0xFFFFFFFFu, L.outF, src);
        uint32_t bH = f.add, bF = f.add;
        if (f.bnd && j < f.bnd_end) {                          // lane 0 below another stripe
            const uint32_t b = f.bnd[j & (kRingCols - 1)];
            bH = lo16(b);
            bF = hi16(b);
        }
        inH = mad(vH, f.mul, bH);
        inF = mad(vF, f.mul, bF);
    } else {
        uint32_t bH = f.add, bF = f.add;
        if (STRIPED && f.bnd2 && j < f.bnd_end) {
            const uint2 b = f.bnd2[j & 63];
            bH = b.x;
            bF = b.y;
        }
        inH = mad(__shfl_up_sync(0xFFFFFFFFu, L.outH, 1, f.width), f.mul, bH);
        inF = mad(__shfl_up_sync(0xFFFFFFFFu, L.outF, 1, f.width), f.mul, bF);
    }
    L.load_words(f, nwa, nwb);
    L.load_offsets(f, j + 2);
    uint32_t X[R], m = L.run;
#pragma unroll
    for (int r = 0; r < R; ++r)
        X[r] = __viaddmax_u16x2(r == 0 ? L.diag : L.H[r - 1], prmt(cwa[r >> 2], cwb[r >> 2], SEL[r & 3]),
                                L.E[r]);
#pragma unroll
    for (int r = 0; r < R; r += 2) m = __vimax3_u16x2(m, X[r], X[r + 1 < R ? r + 1 : r]);
    uint32_t F = inF;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t Xg = X[r] + NGO;
        L.H[r] = __vimax3_u16x2(X[r], F, Z);
        L.E[r] = __viaddmax_u16x2(L.E[r], NGE, Xg);
        F = __viaddmax_u16x2(F, NGE, Xg);
    }
    if constexpr (ENDS) {
        const uint32_t d = m ^ L.run;
        if (d) {
            if (lo16(d)) { L.store(f.snap); L.colA = j; }
            if (hi16(d)) { L.store(f.snap + 32 * words_for(R)); L.colB = j - f.lagB; }
        }
    }
    L.run = m;
    L.outH = L.H[R - 1];
    L.outF = F;
    L.diag = inH;
}

// steps [k0, kend), an even number of them.  bnd_out (LONG) / rows_out
// (STRIPED): where lane 31 leaves its last row, null in the others.
template <int R, bool ENDS, bool LONG, bool STRIPED>
__device__ __forceinline__ void steps(Lane<R> &L, const Args &a, const Flow &f, int k0, int kend,
                                      uint32_t *bnd_out, uint2 *rows_out) {
    constexpr int W = Lane<R>::W;
    uint32_t wa2[W], wb2[W];
    for (int k = k0; k < kend; k += 2) {
        step<R, ENDS, LONG, STRIPED>(L, a, f, k - f.lag, L.wa, L.wb, wa2, wb2);
        if (LONG && bnd_out) bnd_out[(k - 63) & (kRingCols - 1)] = prmt(L.outH, L.outF, 0x7632);
        if (STRIPED && rows_out && k >= 31 && k - 31 < f.bnd_end) rows_out[k - 31] = make_uint2(L.outH, L.outF);
        step<R, ENDS, LONG, STRIPED>(L, a, f, k + 1 - f.lag, wa2, wb2, L.wa, L.wb);
        if (LONG && bnd_out) bnd_out[(k - 62) & (kRingCols - 1)] = prmt(L.outH, L.outF, 0x7632);
        if (STRIPED && rows_out && k >= 30 && k - 30 < f.bnd_end) rows_out[k - 30] = make_uint2(L.outH, L.outF);
    }
}

// Before a block of 32 steps (all lanes of the warp): the group's maximum so
// far raises every lane's running maximum to one below it -- a rise to less
// cannot be the alignment's maximum, and a lane holding that raised value can
// never hold the final maximum.  LONG: both halves are one alignment, and
// `above` is the H that enters from the stripe above in one of the block's
// columns (0: none).
template <int R, bool LONG>
__device__ __forceinline__ void refresh(Lane<R> &L, int width, uint32_t above) {
    uint32_t m = LONG ? max2u(L.run, above) : L.run;
    for (int o = width >> 1; o > 0; o >>= 1) m = max2u(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (LONG) m = max2u(m, (m << 16) | (m >> 16));
    L.run = max2u(L.run, m - 0x00010001u);       // halves are at least the floor: no borrow
}

// the lane's best (score, column, row) of one half, rows from i0
template <int R, bool ENDS>
__device__ __forceinline__ uint64_t lane_key(const Lane<R> &L, const Args &a, const Flow &f, bool high, int i0) {
    const int v = (int)(high ? hi16(L.run) : lo16(L.run)) - a.floor;
    if (!ENDS || v <= 0) return best_key(v, 0, 0);
    return best_key(v, high ? L.colB : L.colA,
                    i0 + L.find_row(f.snap + (high ? 32 * words_for(R) : 0), high));
}

// result of pair p from its best key; the 16-bit pass of the reference drops
// a pair whose score reaches 32767 (src/ssw.c:866-870)
__device__ __forceinline__ void write_result(const Args &a, int p, uint64_t key, bool ends) {
    const int v = (int)(key >> 40);
    if (v >= 32767) {
        a.score[p] = 32767;
        a.ref_end[p] = a.read_end[p] = -1;
        a.status[p] = TPZ_SW_DROPPED;
        return;
    }
    a.score[p] = v;
    a.ref_end[p] = !ends ? -2 : key ? 0xFFFFFF - (int)((key >> 16) & 0xFFFFFF) : -1;
    a.read_end[p] = !ends ? -2 : key ? 0xFFFF - (int)(key & 0xFFFF) : 0;
    a.status[p] = TPZ_SW_OK;
}

}  // namespace sw
}  // namespace tpz
