// search_kernels.cu -- resident index, seed lookup, gapless extension and the
// best-first SA walk with its hitlist, for sm_100a.
//
// Reference path (src/query.c:94-174): for each query position a lower-bound
// search of the query suffix in the suffix array (sa_search), sa_hsp at the
// bound and the row before it, then a best-first walk over adjacent SA rows
// (pqueue_next) feeding a capped hitlist (hitlist_add) until -S counted pops
// or an empty queue.
//
// Device layout of the index (one copy in HBM, built once per DB):
//   T        the .psq bytes (internal alphabet + '\n'), padded with '\n'
//   SA       int64 rows; rows [Tsize, sa_rows) are zero -- the reference
//            mmaps .SA and its reads past the end (search.c:100, hit.c:138
//            with db_valid_index comparing rows against a byte size,
//            db.c:249-251) see the zero fill of the file's last page
//   pstart   protein start offsets (from .ind), Psize + 1 entries
//   nl       number of '\n' before each 64-byte block of T: the protein of a
//            text position is nl[pos/64] + the '\n' bytes in its block before
//            it (db_index, db.c:176-205, counts the delimiter as part of the
//            preceding protein)
//   lb       for each 5-symbol prefix code (26-ary, '\n' = 0, 'A'..'Y' =
//            1..25, symbols after a '\n' read as 0) the number of suffixes
//            whose prefix code is smaller; the rows of a code are
//            [lb[c], lb[c+1]).  Suffix order and prefix-code order agree
//            because '\n' sorts below every letter, so a lower bound needs a
//            binary search only inside one bucket, starting 5 symbols in.
//
// Walk state per query (one warp, exact sequential semantics):
//   the priority queue of suffix cursors is an array of per-score stacks:
//   among equal scores the newest insert pops first, as with rb_popmax on a
//   tree where equal keys go right (rbtree.c:70-78, :410-427);
//   the hitlist is a protein -> slot table and a log of insertions and score
//   rises, from which each score's list (oldest first, rbtree.c:429-457) is
//   read when something is evicted and at the end.

#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "search_internal.cuh"

namespace tpz {
namespace search {

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ int sym(uint8_t c) { return c == '\n' ? 0 : (int)c - 'A' + 1; }

// prefix code of the text suffix at idx (K symbols, zero after a '\n')
__device__ __forceinline__ int64_t text_code(const uint8_t *T, int64_t Tsize, int64_t idx) {
    int64_t code = 0;
    bool ended = false;
#pragma unroll
    for (int i = 0; i < kK; ++i) {
        int d = 0;
        if (!ended) {
            const int64_t p = idx + i;
            const uint8_t c = p < Tsize ? T[p] : (uint8_t)'\n';
            if (c == '\n') ended = true; else d = sym(c);
        }
        code = code * 26 + d;
    }
    return code;
}

// exact count of '\n' bytes in T[base, pos) with base = pos & ~63
__device__ __forceinline__ int newlines_in_block_before(const uint8_t *T, int64_t pos) {
    const int64_t base = pos & ~(int64_t)63;
    const int n = (int)(pos - base);
    const uint64_t *w = reinterpret_cast<const uint64_t *>(T + base);
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (8 * i >= n) break;
        const uint64_t x = __ldg(w + i) ^ 0x0A0A0A0A0A0A0A0Aull;
        uint64_t y = (x & 0x7F7F7F7F7F7F7F7Full) + 0x7F7F7F7F7F7F7F7Full;
        y = ~(y | x | 0x7F7F7F7F7F7F7F7Full);      // 0x80 in every byte that was '\n'
        const int keep = n - 8 * i;                   // bytes of this word before pos
        if (keep < 8) y &= (1ull << (8 * keep)) - 1;
        cnt += __popcll(y);
    }
    return cnt;
}

__device__ __forceinline__ int64_t protein_of(const DevIndex &ix, int64_t pos) {
    return (int64_t)ix.nl[pos >> 6] + newlines_in_block_before(ix.T, pos);
}

// 32 bytes of memory from p (any alignment) as 8 words in memory order:
// nine aligned 4-byte loads issued together, funnel-shifted into place, so
// the window stays in registers.  Reads up to 3 bytes before p and 35 after
// it: the text and query buffers keep 64 readable bytes in front of their
// first byte and behind their last.
__device__ __forceinline__ void load32(const uint8_t *p, uint32_t (&w)[8]) {
    const uintptr_t a = (uintptr_t)p & ~(uintptr_t)3;
    const uint32_t sh = (uint32_t)((uintptr_t)p - a) * 8u;
    const uint32_t *src = reinterpret_cast<const uint32_t *>(a);
    uint32_t r[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) r[k] = __ldg(src + k);
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = __funnelshift_r(r[k], r[k + 1], sh);
}

// Extension table of a block (shared memory), by query letter and text
// letter (the low 5 bits of the byte, 1..25): 256 * score + 1, and in row and
// column 0 a value that no extension makes up for.  A running sum of entries
// is 256 * score + index, so one addition and one maximum per residue keep
// the best score with the last index that reached it, and a residue past an
// end counts as the end.  Lanes that extend one query offset read one row of
// 32 words: different banks for different text letters.
constexpr int kExtWords = 32 * 32;
constexpr int kExtEnd = -(1 << 23);        // 128 entries of 127 * 256 stay below its half

__device__ __forceinline__ void load_ext(int32_t *ext, const int8_t *sub) {
    for (int i = threadIdx.x; i < kExtWords; i += blockDim.x) {
        const int q = i >> 5, t = i & 31;
        const bool in = q >= 1 && q <= 25 && t >= 1 && t <= 25;
        ext[i] = in ? 256 * sub[(t - 1) * 25 + (q - 1)] + 1 : kExtEnd;
    }
}

// bytes of a word below / from `n` (any int)
__device__ __forceinline__ uint32_t low_bytes(int n) {
    return n >= 4 ? ~0u : n <= 0 ? 0u : (1u << (8 * n)) - 1u;
}

// table byte offsets (q * 128 + t * 4) of bytes 0, 2 and 1, 3 of a text and a
// query word, two to a word; a '\n' (bit 6 clear) has text letter 0
__device__ __forceinline__ void ext_offsets(uint32_t t, uint32_t q, uint32_t &even, uint32_t &odd) {
    t &= ((t >> 6) & 0x01010101u) * 0x1Fu;
    q &= 0x1F1F1F1Fu;
    even = (q & 0x00FF00FFu) * 128u + (t & 0x00FF00FFu) * 4u;
    odd = (q >> 8 & 0x00FF00FFu) * 128u + (t >> 8 & 0x00FF00FFu) * 4u;
}

__device__ __forceinline__ int32_t ext_at(const int32_t *ext, uint32_t off) {
    return *reinterpret_cast<const int32_t *>(reinterpret_cast<const uint8_t *>(ext) + off);
}

// sa_hsp (src/search.c:99-190) at text position idx for query offset off.
// Returns the length (-1 when the first symbols differ; score untouched then).
// The windows (up to 128 bytes each side) are read 32 bytes per round trip
// into registers and walked in the reference's order; its stops -- a '\n', an
// end of query or text -- are table entries.  Bound: instruction issue.  (Byte
// compares, a matrix look-up in global memory and two selects per residue
// took 4.4 ms for the 20.8 M chain elements of a 1000-query search.)
__device__ int hsp_at(const DevIndex &ix, int64_t idx, const uint8_t *Q, int qlen, int off,
                      const int32_t *ext, int *score) {
    const uint8_t *t = ix.T + idx;
    const uint8_t *q = Q + off;
    int64_t mr = ix.Tsize - idx;
    if (mr > qlen - off) mr = qlen - off;
    if (mr > 128) mr = 128;
    uint32_t tw[8], qw[8];
    load32(t, tw);
    load32(q, qw);
    if ((tw[0] & 0xFFu) != (qw[0] & 0xFFu)) return -1;
    int sum = -1, best_r = 0;
    for (int i0 = 0; i0 < (int)mr; i0 += 32) {
        if (i0 > 0) {
            if (sum < kExtEnd / 2) break;
            load32(t + i0, tw);
            load32(q + i0, qw);
        }
        if (i0 + 32 > (int)mr) {
#pragma unroll
            for (int w = 0; w < 8; ++w) qw[w] &= low_bytes((int)mr - i0 - 4 * w);
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            uint32_t even, odd;
            ext_offsets(tw[w], qw[w], even, odd);
            sum += ext_at(ext, even & 0xFFFFu); best_r = max(best_r, sum);
            sum += ext_at(ext, odd & 0xFFFFu); best_r = max(best_r, sum);
            sum += ext_at(ext, even >> 16); best_r = max(best_r, sum);
            sum += ext_at(ext, odd >> 16); best_r = max(best_r, sum);
        }
    }
    int64_t ml = idx < off ? idx : off;
    if (ml > 128) ml = 128;
    int best_l = 0;
    sum = 0;
    // left: i = 1 .. ml-1 reads t[-i]; a round loads the 32 bytes that end at
    // t[-i0], so t[-(i0 + k)] is byte 31 - k
    for (int i0 = 1; i0 < (int)ml; i0 += 32) {
        if (sum < kExtEnd / 2) break;
        load32(t - (i0 + 31), tw);
        load32(q - (i0 + 31), qw);
        if (i0 + 32 > (int)ml) {
#pragma unroll
            for (int w = 0; w < 8; ++w) qw[w] &= ~low_bytes(32 - ((int)ml - i0) - 4 * w);
        }
#pragma unroll
        for (int w = 7; w >= 0; --w) {
            uint32_t even, odd;
            ext_offsets(tw[w], qw[w], even, odd);
            sum += ext_at(ext, odd >> 16); best_l = max(best_l, sum);
            sum += ext_at(ext, even >> 16); best_l = max(best_l, sum);
            sum += ext_at(ext, odd & 0xFFFFu); best_l = max(best_l, sum);
            sum += ext_at(ext, even & 0xFFFFu); best_l = max(best_l, sum);
        }
    }
    *score = (best_l >> 8) + (best_r >> 8);
    return (best_l & 255) + (best_r & 255);
}

// lower bound of the suffix P[0, m) (letters only) over the whole SA
__device__ int64_t lower_bound(const DevIndex &ix, const uint8_t *P, int m) {
    int64_t code = 0;
    const int kk = m < kK ? m : kK;
#pragma unroll
    for (int i = 0; i < kK; ++i) code = code * 26 + (i < kk ? sym(P[i]) : 0);
    int64_t lo = ix.lb[code];
    if (m <= kK) return lo;        // exact: every suffix with this prefix is >= P
    int64_t hi = ix.lb[code + 1];
    while (lo < hi) {
        const int64_t mid = lo + ((hi - lo) >> 1);
        const int64_t s = ix.SA[mid] + kK;
        // compare T[s..] with P[kK..]
        int r = 0;
        int64_t i = s;
        int j = kK;
        for (;;) {
            if (j == m) { r = 0; break; }                 // P is a prefix: not less
            if (i >= ix.Tsize) { r = -1; break; }          // text ended first: less
            const int d = (int)ix.T[i] - (int)P[j];
            if (d) { r = d; break; }
            ++i; ++j;
        }
        if (r < 0) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------- index build

__global__ void nl_block_count_kernel(const uint8_t *T, int64_t Tsize, int64_t nblocks,
                                      uint32_t *cnt) {
    for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nblocks;
         b += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t *w = reinterpret_cast<const uint64_t *>(T + 64 * b);
        int c = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t x = w[i] ^ 0x0A0A0A0A0A0A0A0Aull;
            uint64_t y = (x & 0x7F7F7F7F7F7F7F7Full) + 0x7F7F7F7F7F7F7F7Full;
            y = ~(y | x | 0x7F7F7F7F7F7F7F7Full);
            c += __popcll(y);
        }
        cnt[b] = c;   // includes pad bytes past Tsize; they are only counted
                      // for blocks after the last real position
    }
}

// lb[c] = number of rows whose prefix code is < c.  Row r fills the codes
// (code(r-1), code(r)]; row 0 fills [0, code(0)]; the codes past the last
// row get Tsize.
__global__ void lb_build_kernel(const uint8_t *T, int64_t Tsize, const int64_t *SA, int64_t *lb) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r <= Tsize;
         r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t cur = r < Tsize ? text_code(T, Tsize, SA[r]) : kCodes;
        const int64_t prev = r > 0 ? text_code(T, Tsize, SA[r - 1]) : -1;
        for (int64_t c = prev + 1; c <= cur && c <= kCodes; ++c) lb[c] = r;
    }
}

// --------------------------------------------------------------- seeding

// One thread per searched query position (query_find_suffixes,
// src/query.c:104-131).  Writes two cursor slots per position: slot 0 the
// bound row with direction +1, slot 1 the row before with direction -1
// (len < min_hit_length marks a slot that is not inserted).
__global__ void seed_kernel(DevIndex ix, SeedArgs a) {
    __shared__ int32_t ext[kExtWords];
    load_ext(ext, a.sub);
    __syncthreads();
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < a.npos;
         g += (int64_t)gridDim.x * blockDim.x) {
        // query of this position
        int lo = 0, hi = a.nq - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.pos_base[mid] <= g) lo = mid; else hi = mid - 1;
        }
        const int q = lo;
        const int i = (int)(g - a.pos_base[q]);
        const uint8_t *Q = a.qcat + a.qoff[q];
        const int qlen = a.qlen[q];
        Cursor c0, c1;
        c0.row = -1; c0.off = i; c0.dir = 1; c0.prot = -1; c0.score = 0; c0.len = -1;
        c1.row = -1; c1.off = i; c1.dir = -1; c1.prot = -1; c1.score = 0; c1.len = -1;
        if (Q[i] != 'V') {                     // _bad_prefix: internal 'V' = X
            const int64_t pos = lower_bound(ix, Q + i, qlen - i);
            if (a.lb_out) a.lb_out[g] = pos;
            if (pos >= ix.sa_rows) {
                atomicOr(&a.qstatus[q], TPZ_Q_SA_END);
            } else {
                int sc = 0;
                const int64_t t0 = ix.SA[pos];
                int ln = hsp_at(ix, t0, Q, qlen, i, ext, &sc);
                c0.row = pos; c0.score = sc; c0.len = ln;
                c0.prot = (int32_t)protein_of(ix, t0);
                if (pos != 0) {
                    sc = 0;
                    const int64_t t1 = ix.SA[pos - 1];
                    ln = hsp_at(ix, t1, Q, qlen, i, ext, &sc);
                    c1.row = pos - 1; c1.score = sc; c1.len = ln;
                    c1.prot = (int32_t)protein_of(ix, t1);
                }
            }
        } else if (a.lb_out) {
            a.lb_out[g] = -2;
        }
        a.cursors[2 * g] = c0;
        a.cursors[2 * g + 1] = c1;
    }
}

// Cursors that enter the queue (the chain kernel computes kChain elements
// for each): block sums, one atomic per block.
__global__ void count_queued_kernel(const Cursor *cursors, int64_t n, int min_hit_length,
                                    unsigned long long *count) {
    __shared__ unsigned int part;
    if (threadIdx.x == 0) part = 0;
    __syncthreads();
    unsigned int mine = 0;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n;
         c += (int64_t)gridDim.x * blockDim.x)
        mine += cursors[c].len >= min_hit_length;
    atomicAdd(&part, mine);
    __syncthreads();
    if (threadIdx.x == 0 && part) atomicAdd(count, (unsigned long long)part);
}

// One thread per pattern: the sa_search idx of a whole pattern.
__global__ void lower_bound_kernel(DevIndex ix, const uint8_t *pcat, const int64_t *poff,
                                   const int32_t *plen, int64_t n, int64_t *out) {
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n;
         g += (int64_t)gridDim.x * blockDim.x)
        out[g] = lower_bound(ix, pcat + poff[g], plen[g]);
}

// The per-call sa_search (src/search.c:237-362) in one thread, with all
// three of its outputs.  The lower bound and the match count have one answer
// each, whatever the search; `last_position` is the common prefix length of
// P with the last row the reference's binary search compares in its first
// loop (P's length once a row starting with P is found), so this search
// probes the rows in that same order: the window [lo, lo + size) with its
// probe at lo + half, both halves' known prefix lengths carried (a suffix
// between two rows shares at least the smaller of their common prefixes with
// P, so comparisons start past it).
__device__ int cmp_from(const DevIndex &ix, int64_t suf, const uint8_t *P, int64_t m,
                        int64_t *match) {
    int64_t i = suf + *match, j = *match;
    int r = 0;
    while (i < ix.Tsize && j < m && (r = (int)ix.T[i] - (int)P[j]) == 0) { ++i; ++j; }
    *match = j;
    return r == 0 ? -(j != m) : r;
}

__global__ void sa_search_call_kernel(DevIndex ix, const uint8_t *P, int64_t m, int64_t *out3) {
    int64_t lo = 0, size = ix.Tsize, half = size >> 1, lm = 0, rm = 0, match = 0;
    bool found = false;
    while (size > 0) {
        match = lm < rm ? lm : rm;
        const int r = cmp_from(ix, ix.SA[lo + half], P, m, &match);
        if (r < 0) {
            lo += half + 1;
            half -= (size & 1) ^ 1;
            lm = match;
        } else if (r > 0) {
            rm = match;
        } else {
            found = true;
            break;
        }
        size = half;
        half >>= 1;
    }
    int64_t first = lo, count = 0;
    if (found) {
        // rows starting with P form one run: its first row, then its end
        int64_t a = 0, b = ix.Tsize;
        while (a < b) {
            const int64_t mid = a + ((b - a) >> 1);
            int64_t k = 0;
            if (cmp_from(ix, ix.SA[mid], P, m, &k) < 0) a = mid + 1; else b = mid;
        }
        first = a;
        b = ix.Tsize;
        while (a < b) {
            const int64_t mid = a + ((b - a) >> 1);
            int64_t k = 0;
            if (cmp_from(ix, ix.SA[mid], P, m, &k) == 0) a = mid + 1; else b = mid;
        }
        count = a - first;
    }
    out3[0] = first;
    out3[1] = count;
    out3[2] = match;
}

// One thread per (row, query offset) for the stage entry point.
__global__ void hsp_batch_kernel(DevIndex ix, const uint8_t *qcat, const int64_t *qoff,
                                 const int32_t *qlen, const int32_t *query_of, const int32_t *off,
                                 const int64_t *row, int64_t n, const int8_t *sub, int32_t *score,
                                 int32_t *len) {
    __shared__ int32_t ext[kExtWords];
    load_ext(ext, sub);
    __syncthreads();
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int q = query_of[g];
        const int64_t r = row[g];
        int sc = 0, ln = -2;
        if (r >= 0 && r < ix.sa_rows) ln = hsp_at(ix, ix.SA[r], qcat + qoff[q], qlen[q], off[g], ext, &sc);
        score[g] = sc;
        len[g] = ln;
    }
}

// ------------------------------------------------------------------ walk

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
    return x;
}

// highest set bit index <= from, or -1
__device__ __forceinline__ int bits_max_le(const uint64_t *bits, int from) {
    int w = from >> 6;
    uint64_t m = bits[w] & (((from & 63) == 63) ? ~0ull : ((2ull << (from & 63)) - 1));
    for (;;) {
        if (m) return (w << 6) + 63 - __clzll(m);
        if (--w < 0) return -1;
        m = bits[w];
    }
}

// packed chain element: score in the low half, length in the high half
constexpr int kLenEnd = -1000;      // row outside [0, 8*Tsize): the cursor is freed
constexpr int kLenFault = -2000;    // row past the zero-filled SA page
__device__ __forceinline__ uint32_t pack_elem(int score, int len) {
    return (uint32_t)(uint16_t)(int16_t)score | ((uint32_t)(uint16_t)(int16_t)len << 16);
}
__device__ __forceinline__ int elem_score(uint32_t e) { return (int)(int16_t)(e & 0xFFFFu); }
__device__ __forceinline__ int elem_len(uint32_t e) { return (int)(int16_t)(e >> 16); }

// The chain element of a cursor `step` rows past `row` (step >= 1): the
// sa_hsp (src/suffix.c:47) of suffix_increment's next row, or a marker; and
// the protein of that row (db_index, the hitlist's key), -1 with a marker.
__device__ __forceinline__ uint32_t chain_elem(const DevIndex &ix, int64_t row, int dir, int step,
                                               const uint8_t *Q, int qlen, int off,
                                               const int32_t *ext, int32_t *prot) {
    const int64_t nr = row + (int64_t)dir * step;
    *prot = -1;
    if (nr < 0 || nr >= 8 * ix.Tsize) return pack_elem(0, kLenEnd);
    if (nr >= ix.sa_rows) return pack_elem(0, kLenFault);
    int sc = 0;
    const int64_t pos = ix.SA[nr];
    const int ln = hsp_at(ix, pos, Q, qlen, off, ext, &sc);
    *prot = (int32_t)protein_of(ix, pos);
    return pack_elem(sc, ln);
}

// One thread per (cursor, element): the first kChain chain elements of every
// queued cursor, so that the walk, whose pops run one after another, finds
// them ready.  Elements a cursor never reaches are computed and not used.
__global__ void chain_kernel(DevIndex ix, SeedArgs a, int min_hit_length, uint32_t *cache,
                             int32_t *cprot) {
    __shared__ int32_t ext[kExtWords];
    load_ext(ext, a.sub);
    __syncthreads();
    const int64_t total = 2 * a.npos * kChain;
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total;
         x += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = x / kChain;
        const int e = (int)(x % kChain);
        const Cursor cu = a.cursors[c];
        if (cu.len < min_hit_length) continue;          // never queued
        const int64_t g = c >> 1;
        int lo = 0, hi = a.nq - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.pos_base[mid] <= g) lo = mid; else hi = mid - 1;
        }
        int32_t pr;
        cache[c * kChainSlots + e] = chain_elem(ix, cu.row, cu.dir, e + 1, a.qcat + a.qoff[lo],
                                                a.qlen[lo], cu.off, ext, &pr);
        cprot[c * kChainSlots + e] = pr;
    }
}

// ------------------------------------------------------------------ hitlist
//
// hitlist_add (hit.c:126-193) for a warp.  A query's hits sit in slots found
// through an open-addressing protein table; every insertion and every rise
// of a hit's score is an event in a log, and a hit's place in its score's
// list (rb_reput re-inserts as newest, rbtree.c:496-505) is its last event.
// While the list is below its capacity, a batch of up to 32 pops is added at
// once, one per lane.  At capacity, pops that do not beat the worst hit are
// counted without a lookup (also many at once), and the others evict the
// oldest hit of the smallest score (rb_popmin, rbtree.c:429-457), found by
// walking the log: hits of the smallest score are never added while it is
// the smallest, so one pass over the log serves all evictions at a score.
struct HitState {
    uint64_t *table;        // protein (low half, all ones: free) and slot
    uint32_t hmask;
    int4 *slot;             // protein, score, length, query offset
    int32_t *last;          // last event of each slot
    int32_t *log;           // slot of each event
    int32_t *hist;          // hits per score, kept while the list is full
    int cap, logcap;
    int size, nev, smax;    // hits, events, largest score seen
    int used;               // table entries that are not free
    // full: smallest score, hits that hold it; how far the log has been read
    // for them, and which of the last 32 events are theirs (cslot: a lane's)
    int hmin, cmin, scan;
    unsigned cand;
    int cslot;
};

constexpr uint64_t kFree = ~0ull;
constexpr uint64_t kGone = ~0ull - 1;    // an evicted protein's entry: probes go on past it

__device__ __forceinline__ uint64_t table_entry(int32_t p, int32_t s) {
    return (uint64_t)(uint32_t)p | ((uint64_t)(uint32_t)s << 32);
}

// everything below reads mutable memory past L1 (other lanes write it)
__device__ __forceinline__ int4 load_slot(const HitState &h, int s) { return __ldcg(h.slot + s); }

// events in order, the outdated ones dropped
__device__ void compact_log(HitState &h, int lane) {
    int n = 0;
    for (int base = 0; base < h.nev; base += 32) {
        const int e = base + lane;
        const int s = e < h.nev ? __ldcg(h.log + e) : -1;
        const bool live = s >= 0 && __ldcg(h.last + s) == e;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, live);
        if (live) {
            const int i = n + __popc(m & ((1u << lane) - 1u));
            h.log[i] = s;
            h.last[s] = i;
        }
        n += __popc(m);
        __syncwarp();
    }
    h.nev = n;
    h.scan = 0;
    h.cand = 0;
}

// hits per score into hist[0 .. top]
__device__ void count_scores(HitState &h, int lane, int top) {
    for (int s = lane; s <= top; s += 32) h.hist[s] = 0;
    __syncwarp();
    for (int base = 0; base < h.nev; base += 32) {
        const int e = base + lane;
        const int s = e < h.nev ? __ldcg(h.log + e) : -1;
        if (s >= 0 && __ldcg(h.last + s) == e) atomicAdd(&h.hist[load_slot(h, s).y], 1);
    }
    __syncwarp();
}

// the smallest score >= from that a hit holds
__device__ int next_score(const HitState &h, int from, int lane) {
    for (int b = from; b <= h.smax; b += 32) {
        const unsigned m =
            __ballot_sync(0xFFFFFFFFu, b + lane <= h.smax && __ldcg(h.hist + b + lane) > 0);
        if (m) return b + __ffs(m) - 1;
    }
    return kSMax;
}

// Where protein p is in the table, 32 entries per read: its slot, or -1 and
// the free entry that ends its probe sequence.
__device__ int find(const HitState &h, int lane, int p, uint32_t *at) {
    for (uint32_t b = hash32((uint32_t)p);; b += 32) {
        const uint64_t e = __ldcg(h.table + ((b + lane) & h.hmask));
        const unsigned hit = __ballot_sync(0xFFFFFFFFu, (int32_t)(uint32_t)e == p);
        const unsigned end = __ballot_sync(0xFFFFFFFFu, e == kFree);
        if (!hit && !end) continue;
        const int l = __ffs(hit ? hit : end) - 1;
        *at = (b + l) & h.hmask;
        return hit ? (int)__shfl_sync(0xFFFFFFFFu, (uint32_t)(e >> 32), l) : -1;
    }
}

// one lane: protein p's entry (entries are p's, another's, gone or free)
__device__ __forceinline__ uint32_t probe(const HitState &h, int p, uint64_t *e) {
    uint32_t i = hash32((uint32_t)p) & h.hmask;
    while ((*e = __ldcg(h.table + i)) != kFree && (int32_t)(uint32_t)*e != p) i = (i + 1) & h.hmask;
    return i;
}

// one lane: claims an entry for protein p with slot s, beside other lanes
// that add other proteins; or the entry p already has, in *e
__device__ __forceinline__ bool claim(const HitState &h, int p, int s, uint32_t *at, uint64_t *e) {
    uint32_t i = hash32((uint32_t)p) & h.hmask;
    for (;; i = (i + 1) & h.hmask) {
        *e = __ldcg(h.table + i);
        if (*e == kFree) {
            *e = atomicCAS((unsigned long long *)h.table + i, kFree, table_entry(p, s));
            if (*e == kFree) { *at = i; return true; }
        }
        if ((int32_t)(uint32_t)*e == p) return false;
    }
}

// the table without its gone entries
__device__ void rebuild(HitState &h, int lane) {
    for (uint32_t i = lane; i <= h.hmask; i += 32) h.table[i] = kFree;
    __syncwarp();
    for (int s = lane; s < h.size; s += 32) {
        uint32_t at;
        uint64_t e;
        claim(h, load_slot(h, s).x, s, &at, &e);
    }
    h.used = h.size;
    __syncwarp();
}

// The `want` oldest hits of the smallest score (want <= h.cmin): lane i gets
// the slot of the i-th.
__device__ int oldest_of_min(HitState &h, int lane, int want) {
    int mine = -1;
    for (int got = 0; got < want;) {
        // what the last read of the log found, without those that rose since
        unsigned live = __ballot_sync(0xFFFFFFFFu, (h.cand >> lane & 1) &&
                                                       __ldcg(h.last + max(h.cslot, 0)) == h.scan - 32 + lane);
        for (; live && got < want; live &= live - 1) {
            const int s = __shfl_sync(0xFFFFFFFFu, h.cslot, __ffs(live) - 1);
            if (lane == got) mine = s;
            ++got;
        }
        h.cand = live;
        if (got == want) break;
        const int e = h.scan + lane;
        h.cslot = e < h.nev ? __ldcg(h.log + e) : -1;
        const bool hit = h.cslot >= 0 && __ldcg(h.last + h.cslot) == e && load_slot(h, h.cslot).y == h.hmin;
        h.cand = __ballot_sync(0xFFFFFFFFu, hit);
        h.scan += 32;
    }
    return mine;
}

// full list: the smallest score and how many hold it
__device__ void set_min(HitState &h, int lane, int from) {
    h.hmin = next_score(h, from, lane);
    h.cmin = h.hmin < kSMax ? __ldcg(h.hist + h.hmin) : 0;
    h.scan = 0;
    h.cand = 0;
}

__device__ void now_full(HitState &h, int lane) {
    count_scores(h, lane, kSMax - 1);
    set_min(h, lane, 0);
}

// one pop (the same in every lane), which beats the worst hit of a full
// list; true when it is counted
__device__ bool add_one(HitState &h, int lane, int p, int gs, int gl, int off) {
    uint32_t at;
    int s = find(h, lane, p, &at);
    const bool fresh = s < 0, full = h.size >= h.cap;
    int left = -1;                       // score that loses a hit
    if (fresh) {
        s = h.size;
        if (full) {
            s = __shfl_sync(0xFFFFFFFFu, oldest_of_min(h, lane, 1), 0);
            left = h.hmin;
            uint32_t gone;
            find(h, lane, load_slot(h, s).x, &gone);
            if (lane == 0) h.table[gone] = kGone;
        } else {
            h.size++;
        }
        if (lane == 0) h.table[at] = table_entry(p, s);
        h.used++;
    } else {
        const int4 x = load_slot(h, s);
        if (x.y >= gs) return false;
        left = x.y;
        off = x.w;                       // the offset stays the first one's
    }
    h.smax = max(h.smax, gs);
    if (lane == 0) {
        h.slot[s] = make_int4(p, gs, gl, off);
        h.log[h.nev] = s;
        h.last[s] = h.nev;
        if (full) {
            atomicAdd(&h.hist[gs], 1);
            atomicSub(&h.hist[left], 1);
        }
    }
    h.nev++;
    __syncwarp();
    if (full) {
        if (left == h.hmin && --h.cmin == 0) set_min(h, lane, h.hmin + 1);
    } else if (h.size >= h.cap) {
        now_full(h, lane);
    }
    return fresh;
}

// Adds the pops of lanes 0 .. n-1 in lane order; bit l of the result: pop l
// is counted.  Stops after the pop that brings the counted ones to `room`:
// *n is how many were added.
__device__ unsigned add_pops(HitState &h, int lane, int *n, int64_t room, int p, int gs, int gl, int off) {
    if (h.nev + 32 > h.logcap) compact_log(h, lane);
    // (the table has two entries per hit and 256 at least: a quarter stays free)
    if (h.used + 32 > (int)(h.hmask - h.hmask / 4)) rebuild(h, lane);
    const int cnt = *n;
    const bool valid = lane < cnt;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned same =
        __match_any_sync(0xFFFFFFFFu, valid ? (uint64_t)(uint32_t)p : kFree - (uint64_t)lane);
    if (h.size < h.cap && h.size + cnt <= h.cap && cnt < room) {
        // pops of one protein one after the other, the rest together
        unsigned todo = cnt == 32 ? 0xFFFFFFFFu : (1u << cnt) - 1u;
        unsigned fresh_all = 0, event_all = 0;
        int s = -1;
        while (todo) {
            const bool mine = (todo >> lane & 1) && !(same & todo & lt);
            uint32_t i = 0;
            bool fresh = false;
            if (mine) {
                uint64_t e;
                fresh = claim(h, p, -1, &i, &e);          // the slot number follows below
                if (!fresh) s = (int)(e >> 32);
            }
            const unsigned nf = __ballot_sync(0xFFFFFFFFu, fresh);
            bool event = fresh;
            if (fresh) {
                s = h.size + __popc(nf & lt);
                h.table[i] = table_entry(p, s);
                h.slot[s] = make_int4(p, gs, gl, off);
            } else if (mine) {
                const int4 x = load_slot(h, s);
                if (x.y < gs) {
                    h.slot[s] = make_int4(p, gs, gl, x.w);
                    event = true;
                }
            }
            h.size += __popc(nf);
            h.used += __popc(nf);
            fresh_all |= nf;
            event_all |= __ballot_sync(0xFFFFFFFFu, event);
            todo &= ~__ballot_sync(0xFFFFFFFFu, mine);
            __syncwarp();
        }
        // events in pop order; a slot keeps its last one
        if (event_all >> lane & 1) {
            const int e = h.nev + __popc(event_all & lt);
            h.log[e] = s;
            if (!(same & event_all & ~lt & ~(1u << lane))) h.last[s] = e;
        }
        h.nev += __popc(event_all);
        h.smax = max(h.smax, (int)__reduce_max_sync(0xFFFFFFFFu, valid ? (unsigned)gs : 0u));
        __syncwarp();
        if (h.size >= h.cap) now_full(h, lane);
        return fresh_all;
    }
    // At or near capacity.  Every pop that beats the worst hit looks its
    // protein up (together).
    int os = -1, own = -1;               // score and slot of the pop's protein, -1: not in the list
    int4 x = make_int4(0, 0, 0, 0);
    const bool looks = valid && (h.size < h.cap || gs > h.hmin);
    if (looks) {
        uint64_t e;
        probe(h, p, &e);
        if (e != kFree) {
            own = (int)(e >> 32);
            x = load_slot(h, own);
            os = x.y;
        }
    }
    if (h.size >= h.cap && cnt < room) {
        // Full: while the smallest score keeps hits, it and so the pops that
        // change the list are known beforehand, and if none of them is about
        // a hit of that score or a protein of another of them, they change
        // different hits: all at once, each new protein in the place of the
        // next oldest hit of the smallest score.
        const unsigned news = __ballot_sync(0xFFFFFFFFu, looks && os < 0);
        const unsigned rise = __ballot_sync(0xFFFFFFFFu, looks && os >= 0 && os < gs);
        const unsigned acts = news | rise;
        const bool clash = (acts >> lane & 1) && (os == h.hmin || (same & acts & ~(1u << lane)));
        if (!__any_sync(0xFFFFFFFFu, clash || (looks && (same & acts & ~(1u << lane)))) && __popc(news) < h.cmin) {
            if (acts) {
                const int victim = oldest_of_min(h, lane, __popc(news));
                const int s = __shfl_sync(0xFFFFFFFFu, victim, __popc(news & lt)) * (int)(news >> lane & 1) +
                              own * (int)(rise >> lane & 1);
                const int e = h.nev + __popc(acts & lt);
                __syncwarp();
                if (news >> lane & 1) {
                    uint64_t we, te;
                    uint32_t at;
                    const uint32_t gone = probe(h, load_slot(h, s).x, &we);
                    claim(h, p, s, &at, &te);
                    h.table[gone] = kGone;
                    h.slot[s] = make_int4(p, gs, gl, off);
                    atomicAdd(&h.hist[gs], 1);
                } else if (rise >> lane & 1) {
                    h.slot[s] = make_int4(p, gs, gl, x.w);
                    atomicAdd(&h.hist[gs], 1);
                    atomicSub(&h.hist[os], 1);
                }
                if (acts >> lane & 1) {
                    h.log[e] = s;
                    h.last[s] = e;
                }
                if (lane == 0 && news) atomicSub(&h.hist[h.hmin], __popc(news));
                h.cmin -= __popc(news);
                h.used += __popc(news);
                h.nev += __popc(acts);
                h.smax = max(h.smax, (int)__reduce_max_sync(0xFFFFFFFFu, (acts >> lane & 1) ? (unsigned)gs : 0u));
                __syncwarp();
            }
            return news | __ballot_sync(0xFFFFFFFFu, valid && gs <= h.hmin);
        }
    }
    // One by one: what an earlier pop of the batch may change of a lookup is
    // only a protein it added or raised itself, and a hit it evicted.
    unsigned counted = 0, stale = 0;
    for (int l = 0; l < cnt;) {
        const bool full = h.size >= h.cap;
        // the next pop that may change the list; those before it are counted
        // when they do not beat the worst hit, and otherwise hold a protein
        // with a score at least theirs -- above the worst, so not evicted
        const bool acts = valid && lane >= l && !(full && gs <= h.hmin) && (os < gs || (stale >> lane & 1));
        const unsigned below = __ballot_sync(0xFFFFFFFFu, valid && full && gs <= h.hmin);
        const unsigned next = __ballot_sync(0xFFFFFFFFu, acts);
        const int to = next ? __ffs(next) - 1 : cnt;
        unsigned run = below & ~((1u << l) - 1u) & (to == 32 ? 0xFFFFFFFFu : (1u << to) - 1u);
        if (__popc(run) >= room) {
            // the stop at -S is among them: the room-th set bit
            while (--room > 0) run &= run - 1;
            const int at = __ffs(run) - 1;
            *n = at + 1;
            return counted | (below & ~((1u << l) - 1u) & ((2u << at) - 1u));
        }
        room -= __popc(run);
        counted |= run;
        l = to;
        if (l >= cnt) break;
        const int bp = __shfl_sync(0xFFFFFFFFu, p, l), bs = __shfl_sync(0xFFFFFFFFu, gs, l);
        const int bl = __shfl_sync(0xFFFFFFFFu, gl, l), bo = __shfl_sync(0xFFFFFFFFu, off, l);
        if (add_one(h, lane, bp, bs, bl, bo)) {
            counted |= 1u << l;
            if (--room == 0) { *n = l + 1; return counted; }
        }
        stale |= __shfl_sync(0xFFFFFFFFu, same, l);
        ++l;
    }
    return counted;
}

// The hitlist in traversal order (score descending, newest first): a
// counting sort of the live events from the newest to the oldest.
__device__ void write_hits(HitState &h, int lane, Hit *out) {
    count_scores(h, lane, h.smax);
    int run = 0;
    for (int top = h.smax; top >= 0; top -= 32) {
        const int s = top - lane;
        const int c = s >= 0 ? __ldcg(h.hist + s) : 0;
        int x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (s >= 0) h.hist[s] = run + x - c;
        run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    __syncwarp();
    for (int base = h.nev - 1; base >= 0; base -= 32) {
        const int e = base - lane;
        const int s = e >= 0 ? __ldcg(h.log + e) : -1;
        const bool live = s >= 0 && __ldcg(h.last + s) == e;
        int4 x = make_int4(0, -1 - lane, 0, 0);
        if (live) x = load_slot(h, s);
        const unsigned same = __match_any_sync(0xFFFFFFFFu, x.y);
        if (live) {
            const int rank = __popc(same & ((1u << lane) - 1u));
            const int at = __ldcg(h.hist + x.y) + rank;
            Hit o;
            o.protein = x.x; o.gapless_score = x.y; o.gapless_length = x.z; o.suffix_offset = x.w;
            out[at] = o;
        }
        __syncwarp();
        if (live && !(same & ((1u << lane) - 1u))) h.hist[x.y] += __popc(same);
        __syncwarp();
    }
}

// --------------------------------------------------------------------- walk
//
// query_fetch_alignment_batch (src/query.c:151-157) over pqueue_next
// (priority_queue.c:36-56): pop the newest cursor of the highest score, move
// it one row on and push it again, add the popped row to the hitlist.  One
// warp per query.
//
// The order of pops has runs that do not depend on each other.  Let s be the
// highest score.  The top cursor of its stack pops, and while its next row
// scores s or more it pops again at once (it is then alone above s, or the
// newest at s); when it falls below s, or out of the queue, the cursor under
// it follows.  So up to 32 cursors of the stack take their runs together, a
// lane each, and their pushes below s are made in stack order.  Nothing in
// the queue depends on the hitlist, whose only way back is the stop at -S
// counted pops, so the popped rows are collected and added 32 at a time.
// All queue state is in shared memory: per cursor the rows advanced, the
// link to the next in its stack and the scores of its next rows.
// Bound: latency of dependent shared-memory and L2 reads, now per group of
// pops: about 40 cycles per cursor to read a stack's links, some 1,000 per
// group for the rest.  (One lane popping one cursor after the other through
// global memory took 1.15 us per pop; the same in shared memory 0.45 us.)

// a cursor's state: rows advanced, and the next cursor in its score's stack
struct CurState {
    uint32_t k;
    int32_t link;
};

constexpr int kBuf = 16;                // chain elements staged per cursor
constexpr int kHeadSmem = 1024;         // scores whose stack head is in shared memory
constexpr int kScoreWords = kSMax / 64;
// codes of a staged element besides a score >= 0
constexpr int16_t kNotQueued = -1;      // too short, or past the array: the cursor is not pushed
constexpr int16_t kFault = -2;          // row past the zero-filled SA page
static_assert(kChain == 32 && kChainSlots == 64, "blocks of 32 elements in two halves");
// bitmap, stack heads, pops of a batch and extension table in front of the cursors
constexpr int kPops = 128;              // ring of popped rows
constexpr int kWalkFixed = 8 * kScoreWords + 2 * kHeadSmem + kPops * (int)sizeof(CurState) + 4 * kExtWords;
static_assert(kWalkFixed % 16 == 0, "cursor state alignment");

__device__ __forceinline__ int16_t push_code(uint32_t elem, int minlen) {
    const int ln = elem_len(elem);
    if (ln == kLenFault) return kFault;
    return ln >= minlen ? (int16_t)elem_score(elem) : kNotQueued;
}

// A query's cursors in shared memory, or (SPILL: queries with too many) in
// global memory.
template <bool SPILL>
__global__ void __launch_bounds__(32) walk_kernel(DevIndex ix, const __grid_constant__ WalkArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x;
    const int q = a.order[blockIdx.x];
    const uint8_t *Q = a.qcat + a.qoff[q];
    const int qlen = a.qlen[q];
    const int minlen = a.min_hit_length;
    const int64_t cbase = a.cursor_base[q];
    const int ncur = (int)(a.cursor_base[q + 1] - cbase);
    const Cursor *cur = a.cursors + cbase;
    uint32_t *cache = a.ccache + cbase * kChainSlots;
    int32_t *cprot = a.cprot + cbase * kChainSlots;

    uint64_t *bits = reinterpret_cast<uint64_t *>(smem);
    int16_t *head_low = reinterpret_cast<int16_t *>(bits + kScoreWords);
    CurState *pops = reinterpret_cast<CurState *>(head_low + kHeadSmem);     // rows on, cursor
    int32_t *ext = reinterpret_cast<int32_t *>(pops + kPops);
    load_ext(ext, a.sub);
    int16_t *buf = reinterpret_cast<int16_t *>(SPILL ? a.spill + a.spill_off[blockIdx.x] : smem + kWalkFixed);
    CurState *state = reinterpret_cast<CurState *>(buf + kBuf * (size_t)ncur);

    HitState h;
    {
        uint8_t *base = a.scratch + (size_t)q * a.scratch_per_query;
        const size_t ns = (size_t)a.max_cap;
        h.table = a.table + (size_t)q * a.hash_size;
        h.hmask = (uint32_t)a.hash_size - 1;
        h.slot = (int4 *)base;
        h.last = (int32_t *)(h.slot + ns);
        h.log = h.last + ns;
        h.logcap = 2 * a.max_cap + 64;
        h.hist = h.log + h.logcap;
        h.cap = qlen > 3000 ? (int)(1.5 * a.num_hits) : a.alignments;   // hit.c:106-109
        h.size = h.nev = h.used = 0;
        h.smax = 0;
        h.hmin = kSMax;
        h.cmin = h.scan = h.cslot = 0;
        h.cand = 0;
    }
    // stack heads of the scores past shared memory, after this query's histogram
    int16_t *head_high = reinterpret_cast<int16_t *>(h.hist + kSMax);
    auto head = [&](int s) -> int16_t & { return s < kHeadSmem ? head_low[s] : head_high[s]; };
    auto has = [&](int s) { return (bits[s >> 6] >> (s & 63)) & 1; };
    // blocks of 32 elements take the two halves of a cursor's slots in turn,
    // so the element before a new block keeps its place
    auto chain_at = [](int c, uint32_t e) { return (size_t)c * kChainSlots + e % kChainSlots; };
    // the kBuf elements from e on into cursor c's staging
    auto stage = [&](int c, uint32_t e) {
        const uint4 *src = reinterpret_cast<const uint4 *>(cache + chain_at(c, e));
        uint4 x[kBuf / 4];
#pragma unroll
        for (int i = 0; i < kBuf / 4; ++i) x[i] = __ldcg(src + i);
        uint32_t *b = reinterpret_cast<uint32_t *>(buf + kBuf * c);
#pragma unroll
        for (int i = 0; i < kBuf / 4; ++i) {
            b[2 * i] = (uint16_t)push_code(x[i].x, minlen) | ((uint32_t)(uint16_t)push_code(x[i].y, minlen) << 16);
            b[2 * i + 1] = (uint16_t)push_code(x[i].z, minlen) | ((uint32_t)(uint16_t)push_code(x[i].w, minlen) << 16);
        }
    };

    // ---- the queue in seeding insertion order: a cursor's link is the one
    // before it with the same score, ncur (which links to itself) at the end
    for (int i = lane; i < kScoreWords; i += 32) bits[i] = 0;
    if (lane == 0) state[ncur].link = ncur;
    __syncwarp();
    int qmax = -1;
    for (int base = 0; base < ncur; base += 32) {
        const int c = base + lane;
        int sc = -1;
        if (c < ncur && cur[c].len >= minlen) {
            sc = cur[c].score;
            stage(c, 0);
            // the rest of its elements on the way to L2
            asm volatile("prefetch.global.L2 [%0];" ::"l"(cache + chain_at(c, kBuf)));
        }
        const unsigned same = __match_any_sync(0xFFFFFFFFu, sc >= 0 ? sc : -1 - lane);
        const unsigned below = same & ((1u << lane) - 1u), above = same & ~((2u << lane) - 1u);
        if (sc >= 0) {
            CurState st;
            st.k = 0;
            st.link = below ? base + 31 - __clz(below) : has(sc) ? head(sc) : ncur;
            state[c] = st;
        }
        __syncwarp();
        if (sc >= 0 && !above) {
            head(sc) = (int16_t)c;
            atomicOr((unsigned long long *)&bits[sc >> 6], 1ull << (sc & 63));
        }
        qmax = max(qmax, __reduce_max_sync(0xFFFFFFFFu, sc));
        __syncwarp();
    }

    int64_t npops = 0, counter = 0, refills = 0;
    PopRec *trace = a.trace ? a.trace + (int64_t)q * a.trace_cap : nullptr;
    // why a cursor's run stops before its score falls below the stack's
    enum { kNo, kLong, kRefill, kPastEnd };
    bool open = qmax >= 0;               // the queue goes on
    bool past_end = false;
    int first = 0, pending = 0;          // popped rows not yet in the hitlist: pops[first ..]
    int filled = -1;                     // cursor whose next block of elements has been computed
    int refill = -1;                     // cursor that waits for that
    for (;;) {
        while (open && refill < 0 && pending < 32) {
            const int s = qmax;
            // ---- the first 32 cursors of the stack
            int c = ncur, under = head(s);
            for (int i = 0; i < 32 && under != ncur; i += 4) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (lane == i + j) c = under;
                    under = state[under].link;
                }
            }
            const int held = __popc(__ballot_sync(0xFFFFFFFFu, c != ncur));
            // ---- their runs
            uint32_t k0 = 0, k = 0;
            int stop = kNo, sc = kNotQueued;
            if (c != ncur) {
                k = k0 = state[c].k;
                for (;;) {
                    if ((k & (kBuf - 1)) == 0 && k > 0) {
                        if (k >= kChain && k % 32 == 0 && (c != filled || k != k0)) { stop = kRefill; break; }
                        stage(c, k);
                    }
                    const int x = buf[kBuf * c + (k & (kBuf - 1))];
                    if (x == kFault) { stop = kPastEnd; break; }
                    ++k;
                    sc = x;
                    if (x < s) break;
                    if (k - k0 == 32) { stop = kLong; break; }
                }
            }
            // ---- those up to the first stopped run, as far as the ring has room
            const int run = (int)(k - k0);
            const unsigned stopped = __ballot_sync(0xFFFFFFFFu, stop != kNo);
            const int end = stopped ? __ffs(stopped) - 1 : 32;
            int sum = run;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xFFFFFFFFu, sum, o);
                if (lane >= o) sum += y;
            }
            const bool take = c != ncur && (lane < end || (lane == end && run > 0)) && sum <= kPops - 32;
            const int taken = __popc(__ballot_sync(0xFFFFFFFFu, take));
            if (take) {
                for (int i = 0; i < run; ++i) {
                    CurState r;
                    r.k = k0 + i;
                    r.link = c;
                    pops[(first + pending + sum - run + i) & (kPops - 1)] = r;
                }
                state[c].k = k;
            } else if (c != ncur && (k0 == 0 || (k0 & (kBuf - 1)) != 0) && (k0 ^ k) >= kBuf) {
                stage(c, k0 & ~(uint32_t)(kBuf - 1));     // its run went on to later elements
            }
            if (taken > 0) pending += __shfl_sync(0xFFFFFFFFu, sum, taken - 1);
            if (__any_sync(0xFFFFFFFFu, take && c == filled)) filled = -1;
            // ---- what is left of the stack, then the pushes in stack order
            const int top = taken < held ? __shfl_sync(0xFFFFFFFFu, c, taken & 31) : under;
            if (lane == 0) {
                if (top != ncur) head(s) = (int16_t)top;
                else bits[s >> 6] &= ~(1ull << (s & 63));
            }
            if (!take) sc = kNotQueued;
            const unsigned same = __match_any_sync(0xFFFFFFFFu, sc >= 0 ? sc : -1 - lane);
            const unsigned below = same & ((1u << lane) - 1u), above = same & ~((2u << lane) - 1u);
            __syncwarp();
            const int prev = below ? 31 - __clz(below) : lane;
            const int pc = __shfl_sync(0xFFFFFFFFu, c, prev);
            if (sc >= 0) state[c].link = below ? pc : has(sc) ? head(sc) : ncur;
            __syncwarp();
            if (sc >= 0 && !above) {
                head(sc) = (int16_t)c;
                atomicOr((unsigned long long *)&bits[sc >> 6], 1ull << (sc & 63));
            }
            const int up = __reduce_max_sync(0xFFFFFFFFu, sc);
            __syncwarp();
            if (up >= s) qmax = up;
            else if (top == ncur) qmax = s > 0 ? bits_max_le(bits, s - 1) : -1;
            open = qmax >= 0;
            // ---- the stopped run's reason, once every run before it is taken
            const int why = __shfl_sync(0xFFFFFFFFu, stop, end & 31);
            const int at_end = __shfl_sync(0xFFFFFFFFu, run, end & 31);
            if (end < 32 && taken == (at_end > 0 ? end + 1 : end)) {
                if (why == kRefill) refill = __shfl_sync(0xFFFFFFFFu, c, end);
                if (why == kPastEnd) { past_end = true; open = false; }
            }
            __syncwarp();
        }
        // ---- popped rows into the hitlist
        int n = min(pending, 32);
        if (n > 0) {
            int p = -1, gs = 0, gl = 0, off = 0;
            int64_t row = 0;
            if (lane < n) {
                const CurState r = pops[(first + lane) & (kPops - 1)];
                const Cursor x = cur[r.link];
                off = x.off;
                row = x.row + (int64_t)x.dir * r.k;
                p = x.prot; gs = x.score; gl = x.len;
                if (r.k > 0) {
                    const size_t at = chain_at(r.link, r.k - 1);
                    const uint32_t w = __ldcg(cache + at);
                    gs = elem_score(w);
                    gl = elem_len(w);
                    p = __ldcg(cprot + at);
                }
            }
            const unsigned counted = add_pops(h, lane, &n, (int64_t)a.seeds - counter, p, gs, gl, off);
            if (trace && lane < n && npops + lane < a.trace_cap) {
                PopRec r;
                r.row = row; r.off = off; r.score = gs; r.len = gl; r.counted = counted >> lane & 1;
                trace[npops + lane] = r;
            }
            npops += n;
            counter += __popc(counted);
            first += n;
            pending -= n;
            if (counter >= a.seeds) break;
            if (pending > 0) continue;
        }
        if (refill >= 0) {
            // past the computed elements: 32 more rows, a lane each, in the
            // place of older ones (whose pops are all in the hitlist by now)
            const Cursor x = cur[refill];
            int32_t pr;
            const uint32_t k = state[refill].k;
            const uint32_t w = chain_elem(ix, x.row, x.dir, (int)k + 1 + lane, Q, qlen, x.off, ext, &pr);
            cache[chain_at(refill, k + lane)] = w;
            cprot[chain_at(refill, k + lane)] = pr;
            ++refills;
            filled = refill;
            refill = -1;
            __syncwarp();
        } else if (!open) {
            break;
        }
    }
    write_hits(h, lane, a.hits + (int64_t)q * a.max_cap);
    if (lane == 0) {
        QueryOut qo;
        qo.nhits = h.size; qo.npops = npops; qo.ncounted = counter; qo.refills = refills;
        // a stop at -S comes before a later pop's end of the array
        qo.status = a.qstatus[q] | (counter < a.seeds && past_end ? TPZ_Q_SA_END : 0);
        a.qout[q] = qo;
    }
}

size_t walk_smem(int cursors) {
    return kWalkFixed + (sizeof(int16_t) * kBuf + sizeof(CurState)) * (size_t)cursors + sizeof(CurState);
}
size_t walk_state_bytes(int cursors) { return walk_smem(cursors) - kWalkFixed; }

size_t walk_scratch_bytes(int cap) {
    const size_t n = (size_t)cap;
    const size_t b = 16 * n + 4 * n + 4 * (2 * n + 64) + 4 * (size_t)kSMax + 2 * (size_t)kSMax;
    return (b + 15) & ~(size_t)15;
}

template __global__ void walk_kernel<false>(DevIndex ix, const __grid_constant__ WalkArgs a);
template __global__ void walk_kernel<true>(DevIndex ix, const __grid_constant__ WalkArgs a);

}  // namespace search
}  // namespace tpz
