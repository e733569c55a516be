// Ordered-statistics decoding for codes beyond the warp kernel (n > 256 or
// k > 128): one CTA per codeword, elimination on the parity-check matrix.
//
// The decoder is cpu_bp_osd_decode.m:187-305 (the reference's MATLAB BP-OSD)
// with the same result, candidate order and tie rule as the warp kernel; only
// the way the most reliable basis (MRB) and the re-encoding are obtained
// differs, because the k x n generator of a long code (up to 1536 x 2048 bits)
// does not fit in shared memory:
//   * the MRB -- the first k independent positions of G in decreasing
//     reliability, found by the column-pivoted elimination of
//     generator_to_systematic (MB:270-305) -- is the complement of the first
//     m independent positions of H in increasing reliability (the bases of a
//     code's matroid are the complements of the bases of its dual, and the
//     greedy scan gives the extreme basis in either order);
//   * those m columns are found by Gauss-Jordan elimination on H: the
//     accumulated row operations T (m x m bits, 128 KiB at m = 1024) live in
//     shared memory column-major, column c's reduced form is T h_c, the XOR
//     of the few columns of T that h_c selects (column weight <= 16).  Only the
//     columns of T at pivoted rows are stored, in pivot order: the others are
//     unit vectors.  The pivots are taken 8 at a time; their combined row
//     operation is linear in a column's 8 pivot-row bits (a -> a + sum_r
//     a_{p_r} U_r), so each stored column takes it in one pass from tables of
//     U, and one warp picks the next round's pivots while the others apply the
//     current round to T;
//   * with T H in reduced form on those columns, a candidate that keeps the
//     hard decisions on the MRB except a flip set F differs from the hard
//     decisions at the pivot positions selected by T s XOR (XOR over f in F of
//     T h_f), s = H * hard.  Only T s and the flip-pool columns are built.
// The metric sums |llr| over the differing positions in increasing sorted
// position (decreasing reliability) in single precision, exactly as MB:247-250.
#include "bp_kernels.h"

#include <algorithm>
#include <climits>

namespace sicc {

namespace {

// CTA size by class: with at least nine warps each worker reduces one of a round's eight candidates.
// 500 and 20,000 codewords of 15 mixed codes, narrow / wide: 288 / 512 446 us and 4.03 ms, 320 / 512
// 433 and 4.04, 320 / 384 433 and 4.11, 320 / 448 432 and 4.18, 352 / 576 450 and 4.17 (256 / 512 was
// 32 us and 0.04 ms slower than 288 / 512).
constexpr int kOsdHNarrow = 320, kOsdHWide = 512;
constexpr int kOsdHClassThreads[kOsdHClasses] = {kOsdHNarrow, kOsdHNarrow, kOsdHNarrow, kOsdHWide};
constexpr int kOsdHMaxWarps = kOsdHWide / 32;
constexpr int kOsdHMaxPool = 128;
constexpr int kRound = 8;  // columns of H per elimination round
constexpr int kTabStride = 33;  // words per table entry: lanes reading different entries hit different banks

struct OsdHLayout {
    int np;       // sort length: power of two >= the longest n
    int nmax;
    int mw;       // words per row of T for the largest m
    int ts;       // column stride of T in words (odd: a warp reading one word of 32 columns hits 32 banks)
    int poolmax;
    int mlo, mhi; // the launch decodes the items of codes with mlo < m <= mhi
};

struct OsdHSmem {
    uint32_t* T;             // [32*mw + 2*kRound][ts] column-major: the column of the row-operation matrix at the
                             // t-th pivot's row, then two buffers of kRound reduced candidate columns; after the
                             // elimination the tables and terms of the candidate tests
    unsigned long long* keys;// [np] sort keys; shares T's space
    float* rel;              // [nmax] |llr| by sorted position j
    int16_t* perm;           // [nmax] code position at sorted position j
    int16_t* row_of_col;     // [nmax] pivot rank of a code position, -1 for the MRB
    uint32_t* hard;          // [nmax/32+1] hard decisions by code position
    uint32_t* tab;           // [32][kTabStride]: entry g < 16 the XOR of U_0..3 selected by g, entry 16 + g that of
                             // U_4..7; aliases vs..relq, which are first written after the elimination
    uint32_t* wv;            // [2][kRound][32] by round parity: the round's basis U_r (0 for a dependent candidate)
    uint8_t* tidx;           // [32*mw] each stored column's bits at the pending round's pivot rows
    int16_t* rank;           // [32*mw] pivot rank of a row of H (its column's place in T), -1 while it has none
    int16_t* order;          // [32*mw] row of the t-th pivot
    uint32_t* vs;            // [poolmax+1][mw] T s and T h_f by row (before reordering)
    uint32_t* syn;           // [mw] s = H * hard by row of H
    int16_t* pivj;           // [32*mw] sorted position of the t-th pivot's column
    float* relq;             // [32*mw] |llr| of the t-th pivot's column
    int16_t* mrb;            // [nmax] dependent positions met during the scan (descending j); shares vs..relq's space
    int16_t* pool_j;         // [poolmax] flip pool (sorted positions, weakest first)
    uint32_t* avec;          // [poolmax][mw] T h_f for the pool, bit t = pivot rank t
    uint32_t* aug;           // [mw] T s, bit t = pivot rank t
};

// Floats of one warp's metric terms: m pivots, 3 flips, padding to a group of four.
__host__ __device__ inline size_t osd_h_terms(int mw) { return 32 * static_cast<size_t>(mw) + 8; }
__host__ __device__ inline size_t a16(size_t x) { return (x + 15) & ~size_t(15); }

__host__ __device__ inline size_t carve(const OsdHLayout& l, unsigned char* base, OsdHSmem* s)
{
    size_t o = 0;
    auto take = [&](size_t bytes) {
        unsigned char* p = base ? base + o : nullptr;
        o = a16(o + bytes);
        return p;
    };
    const size_t rows = 32 * static_cast<size_t>(l.mw);
    OsdHSmem t{};
    {  // the sort keys, then T (the keys are dead once the sorted order is extracted)
        const size_t bt = (rows + 2 * kRound) * l.ts * 4, bk = static_cast<size_t>(l.np) * 8;
        const size_t bc = (l.mw * 128 + kOsdHMaxWarps * osd_h_terms(l.mw)) * sizeof(float);  // nibble sums, the warps' terms
        const size_t most = bt > bk ? bt : bk;
        unsigned char* g = take(most > bc ? most : bc);
        t.T = reinterpret_cast<uint32_t*>(g);
        t.keys = reinterpret_cast<unsigned long long*>(g);
    }
    t.rel = reinterpret_cast<float*>(take(static_cast<size_t>(l.nmax) * 4));
    t.perm = reinterpret_cast<int16_t*>(take(static_cast<size_t>(l.nmax) * 2));
    t.row_of_col = reinterpret_cast<int16_t*>(take(static_cast<size_t>(l.nmax) * 2));
    t.hard = reinterpret_cast<uint32_t*>(take((static_cast<size_t>(l.nmax) / 32 + 1) * 4));
    t.wv = reinterpret_cast<uint32_t*>(take(2 * kRound * 32 * 4));
    t.rank = reinterpret_cast<int16_t*>(take(rows * 2));
    t.tidx = reinterpret_cast<uint8_t*>(take(rows));
    t.order = reinterpret_cast<int16_t*>(take(rows * 2));
    t.syn = reinterpret_cast<uint32_t*>(take(static_cast<size_t>(l.mw) * 4));
    t.pivj = reinterpret_cast<int16_t*>(take(rows * 2));
    t.pool_j = reinterpret_cast<int16_t*>(take(static_cast<size_t>(l.poolmax) * 2));
    {  // the tables and dependent positions of the elimination, then the vectors of the candidate search
        const size_t b_vs = a16((static_cast<size_t>(l.poolmax) + 1) * l.mw * 4);
        const size_t b_avec = a16(static_cast<size_t>(l.poolmax) * l.mw * 4);
        const size_t b_aug = a16(static_cast<size_t>(l.mw) * 4);
        const size_t b_relq = a16(rows * 4);
        const size_t b_vec = b_vs + b_avec + b_aug + b_relq, b_tab = a16(32 * kTabStride * 4), b_mrb = a16(static_cast<size_t>(l.nmax) * 2);
        unsigned char* g = take(b_vec > b_tab + b_mrb ? b_vec : b_tab + b_mrb);
        t.tab = reinterpret_cast<uint32_t*>(g);
        t.mrb = reinterpret_cast<int16_t*>(g ? g + b_tab : nullptr);
        t.vs = reinterpret_cast<uint32_t*>(g);
        t.avec = reinterpret_cast<uint32_t*>(g ? g + b_vs : nullptr);
        t.aug = reinterpret_cast<uint32_t*>(g ? g + b_vs + b_avec : nullptr);
        t.relq = reinterpret_cast<float*>(g ? g + b_vs + b_avec + b_aug : nullptr);
    }
    if (s) *s = t;
    return o;
}

__device__ __forceinline__ unsigned tbit(const uint32_t* row, int q) { return (row[q >> 5] >> (q & 31)) & 1u; }

// CTAs per SM the registers are bounded for (shared memory sets the same or less).
constexpr int osd_h_ctas(int threads) { return threads < 512 ? 2 : 1; }

}  // namespace

template <int kThreads>
__global__ void __launch_bounds__(kThreads, osd_h_ctas(kThreads))
osd_h_kernel(OsdHView hv0, OsdHLayout lay, OsdIO io)
{
    constexpr int kWarps = kThreads / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    OsdHSmem s;
    carve(lay, smem_raw, &s);
    __shared__ int s_rp[2][kRound];
    __shared__ int s_np[2], s_used[2], s_jstop[2];
    __shared__ unsigned s_found[2];  // the round's candidates that gave a pivot
    __shared__ unsigned long long s_best;
    __shared__ unsigned s_least;  // the least estimated metric (bits)
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int TS = lay.ts;
    const int count = io.count_ptr ? *io.count_ptr : io.count;

    auto next_item = [&](int prev) -> int {  // the CTA's next work item (all threads get it)
        if (!io.work_h) return prev < 0 ? static_cast<int>(blockIdx.x) : prev + static_cast<int>(gridDim.x);
        __syncthreads();  // every thread has read the previous one
        if (tid == 0) s_item = atomicAdd(io.work_h, 1);
        __syncthreads();
        return s_item;
    };
    for (int item = next_item(-1); item < count; item = next_item(item)) {
        const int cw = io.index ? io.index[item] : item;
        const OsdHView hv = io.hviews ? io.hviews[io.code_of[cw]] : hv0;
        if (hv.n == 0 || hv.m <= lay.mlo || hv.m > lay.mhi) continue;  // another kernel's item (uniform over the CTA)
        const int n = hv.n, m = hv.m, k = hv.k, MW = hv.mw, rows = 32 * hv.mw;
        const float* src = io.row_off   ? io.llr + io.row_off[item]
                           : io.llr_off ? io.llr + io.llr_off[cw]
                                        : io.llr + static_cast<size_t>(item) * n;
        uint8_t* info_dst = io.out_info ? (io.info_off ? io.out_info + io.info_off[cw]
                                                       : io.out_info + static_cast<size_t>(cw) * io.info_stride)
                                        : nullptr;

        // ---- 1. sort keys (descending |llr|, ties by position), hard decisions ----
        const int np = 1 << (32 - __clz(n - 1));
        for (int i = tid; i < np; i += kThreads) {
            const float x = (i < n) ? src[i] : 0.0f;
            s.keys[i] = (i < n) ? ((static_cast<unsigned long long>(0x7fffffffu - __float_as_uint(fabsf(x))) << 32) |
                                   static_cast<unsigned>(i))
                                : ~0ull;
        }
        for (int i = tid; i < ((n + 31) & ~31); i += kThreads) {
            const bool neg = (i < n) && (src[i] < 0.0f);
            const unsigned b = __ballot_sync(0xffffffffu, neg);
            if (lane == 0) s.hard[i >> 5] = b;
        }
        for (int i = tid; i < n; i += kThreads) s.row_of_col[i] = -1;
        __syncthreads();
        // bitonic sort (np >= 32): compare-exchange distances j2 >= 32 through shared memory, one
        // barrier each; the distances below 32 of each merge level on registers within a warp
        // (lane = element index mod 32), one barrier per level
        auto warp_stages = [&](int k2lo, int k2hi, int j2top) {
            for (int b0 = warp * 32; b0 < np; b0 += kThreads) {
                const int i = b0 + lane;
                unsigned long long v = s.keys[i];
                for (int k2 = k2lo; k2 <= k2hi; k2 <<= 1) {
                    const bool asc = (i & k2) == 0;
                    for (int j2 = min(k2 >> 1, j2top); j2 > 0; j2 >>= 1) {
                        const unsigned long long o =
                            (static_cast<unsigned long long>(__shfl_xor_sync(0xffffffffu, static_cast<unsigned>(v >> 32), j2)) << 32) |
                            __shfl_xor_sync(0xffffffffu, static_cast<unsigned>(v), j2);
                        const bool take_min = ((i & j2) == 0) == asc;
                        v = take_min ? (o < v ? o : v) : (o > v ? o : v);
                    }
                }
                s.keys[i] = v;
            }
            __syncthreads();
        };
        warp_stages(2, 32, 16);
        for (int k2 = 64; k2 <= np; k2 <<= 1) {
            for (int j2 = k2 >> 1; j2 >= 32; j2 >>= 1) {
                for (int pr = tid; pr < np / 2; pr += kThreads) {
                    const int i = ((pr & ~(j2 - 1)) << 1) | (pr & (j2 - 1));  // j2 is a power of two
                    const int ixj = i + j2;
                    const bool asc = (i & k2) == 0;
                    const unsigned long long a = s.keys[i], b = s.keys[ixj];
                    if ((a > b) == asc) {
                        s.keys[i] = b;
                        s.keys[ixj] = a;
                    }
                }
                __syncthreads();
            }
            warp_stages(k2, k2, 16);
        }
        for (int j = tid; j < n; j += kThreads) {
            const unsigned long long key = s.keys[j];
            s.perm[j] = static_cast<int16_t>(key & 0xffffffffull);
            s.rel[j] = __uint_as_float(0x7fffffffu - static_cast<unsigned>(key >> 32));
        }
        __syncthreads();  // T overwrites the keys
        // ---- 2. no row pivoted yet, syndrome of the hard decisions ----
        for (int r = tid; r < rows; r += kThreads) s.rank[r] = -1;
        for (int r = tid; r < rows; r += kThreads) {
            unsigned par = 0;
            if (r < m)
                for (int e = hv.row_ptr[r]; e < hv.row_ptr[r + 1]; ++e) par ^= tbit(s.hard, hv.col_ind[e]);
            const unsigned b = __ballot_sync(0xffffffffu, par);
            if (lane == 0) s.syn[r >> 5] = b;
        }
        __syncthreads();

        // ---- 3. Gauss-Jordan scan of H's columns in increasing reliability ----
        // A column c's reduced form is v = T h_c (the XOR of the columns of T that
        // h_c selects); its pivot is the lowest unpivoted row p with v_p = 1, and
        // the pivot's row operation T <- (I + W e_p^T) T, W = v + e_p, turns
        // column c into e_p and leaves earlier pivot columns alone.
        // Columns are taken kRound at a time.  Interval k of the pipeline:
        //   1. all warps tabulate round k-1's basis by index nibble, gather the stored columns' bits
        //      at its pivot rows (their indices) and apply its operation to round k's candidates (a
        //      warp each);
        //   2. warp 0 picks round k's pivots in order; each pivot's operation is applied at once to
        //      the later candidates and to the round's basis,
        //        a -> a + sum_r a_{p_r} U_r,  U_r <- U_r + U_r[p] W for a new pivot p
        //      (a_{p_r} a column's bits before the round, U_r = 0 for a dependent candidate);
        //      the other warps note round k-1's pivots, apply its operation to the stored columns
        //      (one thread per column, two table entries per word), append the columns of its pivot
        //      rows (e_p + U_p), meet on a named barrier and reduce round k+1's candidates against T,
        //      whose rows they fetched from H during round k-1.
        // Warp 0's chain takes about 2,000 cycles of a round, the step before it 700-1,000; with the
        // rows fetched at the reduction instead, staged in shared memory, 500 codewords of 15 mixed
        // codes took 533 us (500 now; 20,000 took the same 4.2 ms).  Tables and indices built by the
        // other warps in 2 instead of by all in 1: 512 us and 4.25 ms.  Windows of 16 candidates to
        // fill each round with 8 pivots: 538 us and 4.8 ms.
        // The column at position jj: first edge << 15 | weight (0: none), and its row
        // for this lane.  (A code has at most 27 m < 2^15 edges, m <= 1,024.)
        struct Column {
            int info, row;
        };
        auto column_at = [&](int jj) -> Column {
            Column c{0, 0};
            if (jj >= 0) {
                const int v = s.perm[jj], e0 = __ldg(hv.col_ptr + v);
                c.info = (e0 << 15) | (__ldg(hv.col_ptr + v + 1) - e0);
                if (lane < (c.info & 32767)) c.row = __ldg(hv.col_rows + e0 + lane);
            }
            return c;
        };
        auto reduce_column = [&](const Column& c, uint32_t* dst) {  // T h_c, word `lane`
            unsigned v = 0u;
            const int e0 = c.info >> 15, cnt = c.info & 32767;
            // lane e: row of the column's e-th one (none: a row no lane holds), and that row's
            // column's place in T (-1: a unit vector)
            const int mine = lane < cnt ? (c.row << 16) | static_cast<uint16_t>(s.rank[c.row]) : (2047 << 16) | 0xffff;
            // the word of row u >> 16's column of T: loaded whether or not it is stored (place 0
            // then), so that no branch stands between the loads of a group
            auto word = [&](int u) -> unsigned {
                const int at = static_cast<int16_t>(u & 0xffff), row = u >> 16;
                const unsigned x = s.T[max(at, 0) * TS + lane];
                return at >= 0 ? x : lane == (row >> 5) ? 1u << (row & 31) : 0u;
            };
            for (int e = 0; e < cnt && e < 32; e += 4) {
                unsigned part[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) part[x] = word(__shfl_sync(0xffffffffu, mine, (e + x) & 31));
                v ^= (part[0] ^ part[1]) ^ (part[2] ^ part[3]);
            }
            for (int e = 32; e < cnt; ++e) {  // columns heavier than 32
                const int row = __ldg(hv.col_rows + e0 + e);
                v ^= word((row << 16) | static_cast<uint16_t>(s.rank[row]));
            }
            if (lane < MW) dst[lane] = v;
        };
        auto workers_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kThreads - 32) : "memory"); };  // all but warp 0
        // candidate c of buffer b
        auto candidate = [&](int b, int c) -> uint32_t* { return s.T + (rows + b * kRound + c) * TS; };
        for (int c = warp; c < kRound; c += kWarps) reduce_column(column_at(n - 1 - c), candidate(0, c));
        // the columns this warp reduces next (round 1's), fetched a round ahead: candidates warp - 1
        // and, with fewer than 8 workers, warp - 1 + kWarps - 1, ...
        constexpr int kMine = (kRound + kWarps - 2) / (kWarps - 1);
        Column ahead[kMine];
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const int c = warp - 1 + i * (kWarps - 1);
            ahead[i] = column_at(warp > 0 && c < kRound ? n - 1 - kRound - c : -1);
        }
        __syncthreads();
        int t = 0, j = n - 1, nd = 0, jstop = -1;          // after the rounds selected so far
        int pt = 0, pj = 0, pnd = 0, pnp = 0, pused = 0;   // the round whose update is pending
        bool pending = false;
        unsigned pivw = 0u;  // warp 0: pivoted rows, word `lane`
        for (int k = 0;; ++k) {
            const bool select = j >= 0 && t < m;
            if (!select && !pending) break;
            const int cb = k & 1, pb = cb ^ 1;
            const uint32_t* Up = s.wv + pb * kRound * 32;  // the pending round's basis
            if (pending) {
                if (pnp > 0) {
                    // tables of the pending round's basis, one index nibble per warp, word `lane`
                    if (warp >= kWarps - 2 && lane < MW) {
                        const int h = warp - (kWarps - 2);
                        uint32_t* tb = s.tab + h * 16 * kTabStride + lane;
                        unsigned u[4], acc[16];
#pragma unroll
                        for (int b = 0; b < 4; ++b) u[b] = Up[(h * 4 + b) * 32 + lane];
                        acc[0] = 0u;
#pragma unroll
                        for (int e = 1; e < 16; ++e) {
                            const int low = (e & 1) ? 0 : (e & 2) ? 1 : (e & 4) ? 2 : 3;
                            acc[e] = acc[e & (e - 1)] ^ u[low];
                        }
#pragma unroll
                        for (int e = 0; e < 16; ++e) tb[e * kTabStride] = acc[e];
                    }
                    // every stored column's index into them
                    int woff[kRound];
                    unsigned wbit[kRound];
#pragma unroll
                    for (int r = 0; r < kRound; ++r) {
                        const int p = s_rp[pb][r];
                        woff[r] = p >= 0 ? p >> 5 : 0;
                        wbit[r] = p >= 0 ? 1u << (p & 31) : 0u;
                    }
                    for (int at = tid; at < pt; at += kThreads) {
                        const uint32_t* c = s.T + at * TS;
                        unsigned idx = 0u;
#pragma unroll
                        for (int r = 0; r < kRound; ++r)
                            if (c[woff[r]] & wbit[r]) idx |= 1u << r;
                        s.tidx[at] = static_cast<uint8_t>(idx);
                    }
                }
                if (select && pnp > 0)  // the pending operation on this round's candidates, not in them yet
                    for (int c = warp; c < kRound; c += kWarps) {
                        uint32_t* col = candidate(cb, c);
                        const int p = lane < kRound ? s_rp[pb][lane] : -1;
                        const unsigned idx = __ballot_sync(0xffffffffu, p >= 0 && ((col[p >> 5] >> (p & 31)) & 1u));
                        unsigned v = lane < MW ? col[lane] : 0u;
#pragma unroll
                        for (int r = 0; r < kRound; ++r) v ^= Up[r * 32 + lane] & (0u - ((idx >> r) & 1u));
                        if (lane < MW) col[lane] = v;
                    }
                __syncthreads();
            }
            if (warp == 0) {
                if (select) {
                    unsigned v[kRound], U[kRound];
#pragma unroll
                    for (int r = 0; r < kRound; ++r) {
                        v[r] = lane < MW ? candidate(cb, r)[lane] : 0u;
                        U[r] = 0u;
                    }
                    int np = 0, used = 0, js = -1;
                    unsigned found = 0u;
                    int pl[kRound];  // the pivot's row + 1 on its lane, 0 elsewhere
#pragma unroll
                    for (int r = 0; r < kRound; ++r) {
                        const bool valid = j - r >= 0 && t + np < m;  // warp-uniform
                        // each lane: its lowest unpivoted set row (as a mask); the lowest such lane
                        // holds the pivot.  The later candidates (c > r) and the basis (c < r) at
                        // each lane's row are balloted at once, before the pivot lane is known, so
                        // the chain from one candidate to the next is one ballot deep: the pivot
                        // lane's bit of each ballot is that vector's bit at the pivot row.
                        used = valid ? r + 1 : used;
                        const unsigned x = valid ? (v[r] & ~pivw) : 0u;
                        const unsigned bx = __ballot_sync(0xffffffffu, x != 0u);
                        pl[r] = 0;
                        if (bx == 0u) continue;  // dependent: a third or more of the columns scanned
                        const unsigned lb = x & (0u - x);
                        unsigned bc[kRound];
#pragma unroll
                        for (int c = 0; c < kRound; ++c)
                            bc[c] = c > r   ? __ballot_sync(0xffffffffu, (v[c] & lb) != 0u)
                                    : c < r ? __ballot_sync(0xffffffffu, (U[c] & lb) != 0u)
                                            : 0u;
                        const unsigned sel = bx & (0u - bx);  // the pivot lane's bit
                        const bool me = (sel >> lane) & 1u;
                        const unsigned W = me ? (v[r] ^ lb) : v[r];
#pragma unroll
                        for (int c = 0; c < kRound; ++c) {
                            if (c > r) v[c] ^= (bc[c] & sel) ? W : 0u;
                            if (c < r) U[c] ^= (bc[c] & sel) ? W : 0u;
                        }
                        U[r] = W;
                        pl[r] = me ? lane * 32 + __ffs(lb) : 0;
                        pivw |= me ? lb : 0u;
                        ++np;
                        found |= 1u << r;
                        js = t + np == m ? j - r : js;
                    }
#pragma unroll
                    for (int r = 0; r < kRound; ++r) s.wv[(cb * kRound + r) * 32 + lane] = U[r];
                    if (lane < kRound) s_rp[cb][lane] = -1;
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < kRound; ++r)
                        if (pl[r] > 0) s_rp[cb][r] = pl[r] - 1;
                    if (lane == 0) {
                        s_np[cb] = np;
                        s_found[cb] = found;
                        s_used[cb] = used;
                        s_jstop[cb] = js;
                    }
                }
            } else {
                if (pending && warp == 1 && lane < pused) {  // pivot ranks and dependent positions
                    const int pr = s_rp[pb][lane];
                    const unsigned found = s_found[pb], below = (1u << lane) - 1u;
                    if (pr >= 0) {
                        const int rk = pt + __popc(found & below);
                        s.order[rk] = static_cast<int16_t>(pr);
                        s.rank[pr] = static_cast<int16_t>(rk);
                        s.row_of_col[s.perm[pj - lane]] = static_cast<int16_t>(rk);
                        s.pivj[rk] = static_cast<int16_t>(pj - lane);
                    } else {
                        s.mrb[pnd + __popc(~found & below)] = static_cast<int16_t>(pj - lane);  // an MRB position
                    }
                }
                if (pending && pnp > 0) {
                    // a thread takes a whole column (three loads and a store per word).  Splitting a
                    // column's words over threads does not pay: pieces of 8 words took 4.50 ms and
                    // 499 us on the mixes above, halves from 25 words on 4.14 and 447, whole columns 4.07
                    // and 432.
                    for (int at = tid - 32; at < pt; at += kThreads - 32) {
                        uint32_t* c = s.T + at * TS;
                        const unsigned idx = s.tidx[at];
                        if (idx == 0u) continue;
                        const uint32_t* lo = s.tab + (idx & 15u) * kTabStride;
                        const uint32_t* hi = s.tab + (16u + (idx >> 4)) * kTabStride;
                        int w = 0;
                        for (; w + 4 <= MW; w += 4) {
                            const unsigned a0 = c[w] ^ lo[w] ^ hi[w];
                            const unsigned a1 = c[w + 1] ^ lo[w + 1] ^ hi[w + 1];
                            const unsigned a2 = c[w + 2] ^ lo[w + 2] ^ hi[w + 2];
                            const unsigned a3 = c[w + 3] ^ lo[w + 3] ^ hi[w + 3];
                            c[w] = a0;
                            c[w + 1] = a1;
                            c[w + 2] = a2;
                            c[w + 3] = a3;
                        }
                        for (; w < MW; ++w) c[w] ^= lo[w] ^ hi[w];
                    }
                    for (int r = warp - 1; r < kRound; r += kWarps - 1) {  // the pivot rows' columns: e_p + U_p
                        const int p = s_rp[pb][r];
                        if (p >= 0 && lane < MW)
                            s.T[(pt + __popc(s_found[pb] & ((1u << r) - 1u))) * TS + lane] =
                                Up[r * 32 + lane] ^ (lane == (p >> 5) ? 1u << (p & 31) : 0u);
                    }
                }
                workers_sync();  // T is final for the pending round before the next candidates read it
                if (select) {
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        const int c = warp - 1 + i * (kWarps - 1);
                        if (c >= kRound) break;
                        reduce_column(ahead[i], candidate(cb ^ 1, c));
                        ahead[i] = column_at(j - 2 * kRound - c);
                    }
                }
            }
            __syncthreads();
            pending = select;
            if (select) {
                pnp = s_np[cb];
                pused = s_used[cb];
                pt = t;
                pj = j;
                pnd = nd;
                t += pnp;
                if (t == m) jstop = s_jstop[cb];
                nd += pused - pnp;
                j -= pused;
            }
        }
        if (t < m) {  // H rank deficient: leave the BP decision in place
            __syncthreads();
            continue;
        }

        // ---- 4. flip pool: the weakest MRB positions, (|llr| ascending, position ascending) ----
        // The MRB positions in descending sorted position -- the dependent ones met during the
        // scan, then jstop-1 .. 0 -- come in ascending |llr|; ties come in descending position,
        // so the pool entry i is taken from the mirror image of i within its run of equal |llr|
        // (the runs found by binary search: |llr| is non-decreasing along that order).
        {
            const int total = nd + jstop, want = hv.pool;  // nd and jstop: the same in every thread
            auto mrb_at = [&](int c) -> int { return c < nd ? s.mrb[c] : jstop - 1 - (c - nd); };
            // |llr| compared as bit patterns, the order the sort used (a permutation whatever the values)
            auto relbits = [&](int c) -> unsigned { return __float_as_uint(s.rel[mrb_at(c)]); };
            for (int i = tid; i < want; i += kThreads) {
                const unsigned ri = relbits(i);
                int lo = 0, hi = i;  // first index with |llr| >= ri
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (relbits(mid) < ri) lo = mid + 1;
                    else hi = mid;
                }
                const int a = lo;
                lo = i + 1;
                hi = total;  // first index with |llr| > ri
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (relbits(mid) > ri) hi = mid;
                    else lo = mid + 1;
                }
                s.pool_j[i] = static_cast<int16_t>(mrb_at(a + lo - 1 - i));
            }
            if (tid == 0) s_best = ~0ull;
        }
        __syncthreads();

        // ---- 5. T s and the reduced pool columns, then in pivot order ----
        const int pool = hv.pool;
        for (int i = tid; i < (pool + 1) * MW; i += kThreads) s.vs[i] = 0u;
        __syncthreads();
        {
            // T s: XOR of the columns of T selected by s, spread over the warps
            unsigned acc = 0u;
            for (int q0 = warp; q0 < m; q0 += 4 * kWarps) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int q = min(q0 + x * kWarps, m - 1);
                    const unsigned on = q0 + x * kWarps < m ? tbit(s.syn, q) : 0u;
                    acc ^= s.T[s.rank[q] * TS + lane] & (0u - on);
                }
            }
            if (lane < MW && acc) atomicXor(&s.vs[lane], acc);
            // T h_f for the flip pool, one warp per column
            for (int i = warp; i < pool; i += kWarps) reduce_column(column_at(s.pool_j[i]), s.vs + (i + 1) * MW);
        }
        __syncthreads();
        // bit t of an ordered vector = bit order[t] of the row-indexed one (8 vectors' loads in flight)
        for (int r = tid; r < rows; r += kThreads) {
            const int q = r < m ? s.order[r] : -1;
            const int qw = q >= 0 ? q >> 5 : 0;
            const unsigned qb = q >= 0 ? 1u << (q & 31) : 0u;
            for (int v0 = 0; v0 <= pool; v0 += 8) {
                unsigned bits[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) bits[u] = v0 + u <= pool ? s.vs[(v0 + u) * MW + qw] & qb : 0u;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const unsigned b = __ballot_sync(0xffffffffu, bits[u] != 0u);
                    const int vi = v0 + u;
                    if (lane == 0 && vi <= pool) (vi == 0 ? s.aug : s.avec + (vi - 1) * MW)[r >> 5] = b;
                }
            }
        }
        for (int r = tid; r < rows; r += kThreads) s.relq[r] = r < m ? s.rel[s.pivj[r]] : 0.0f;
        if (tid == 0) s_least = 0x7f800000u;
        __syncthreads();
        // ---- 6. candidates ----
        // Bit t of T s (+ T h_f) marks a differing pivot position; pivot ranks in descending order
        // hold the positions in ascending order, the order of the metric's sum.  A flipped position f
        // joins the sum before the first rank t < cut(f), the number of pivots after it.
        // Every test meets an estimate of its metric first: its differing pivot positions summed
        // from tables of |llr| sums by nibble (in T's place, which is done with), plus its flips.
        // Estimate and in-order sum are both within 650 rounding units (1,027 terms, 262 additions)
        // of the exact sum, so a test whose estimate is over the least estimate seen by a factor
        // 1 + 2^-12 (4,096 units) cannot win.  The few others are summed in order, a warp each: its
        // lanes lay the terms out in order, one adds them up.
        float* nib = reinterpret_cast<float*>(s.T);                         // [8 MW][16]
        float* terms = nib + MW * 128 + warp * osd_h_terms(MW);             // this warp's terms in order
        for (int e = tid; e < MW * 128; e += kThreads) {
            const float* r4 = s.relq + (e >> 4) * 4;
            float x = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if ((e >> i) & 1) x += r4[i];
            nib[e] = x;
        }
        __syncthreads();
        struct Test {
            int f[3];          // pool indices of the flips, -1 for none
            int j[3];          // their positions, ascending (absent: INT_MAX)
        };
        auto test_at = [&](int ti) -> Test {
            Test q{{-1, -1, -1}, {INT_MAX, INT_MAX, INT_MAX}};
            if (ti > 0) {
                const uint32_t pk = hv.combos[ti - 1];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const int f = (pk >> (10 * i)) & 1023;
                    q.f[i] = f != 1023 ? f : -1;
                    q.j[i] = f != 1023 ? s.pool_j[f] : INT_MAX;
                }
            }
            auto order2 = [&](int a, int b) {
                const int lo = min(q.j[a], q.j[b]), hi = max(q.j[a], q.j[b]);
                q.j[a] = lo;
                q.j[b] = hi;
            };
            order2(0, 1);
            order2(1, 2);
            order2(0, 1);
            return q;
        };
        auto word_at = [&](const Test& q, int w) -> unsigned {
            unsigned word = s.aug[w];
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (q.f[i] >= 0) word ^= s.avec[q.f[i] * MW + w];
            return word;
        };
        auto estimate = [&](const Test& q) -> float {
            float part[2] = {0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < 3; ++i)
                if (q.j[i] != INT_MAX) part[0] += s.rel[q.j[i]];
            for (int w = 0; w < MW; ++w) {
                const unsigned word = word_at(q, w);
#pragma unroll
                for (int i = 0; i < 8; ++i) part[i & 1] += nib[(w * 8 + i) * 16 + ((word >> (4 * i)) & 15u)];
            }
            return part[0] + part[1];
        };
        auto note = [&](float est) {  // lower the least estimate by this warp's
            const unsigned least = __reduce_min_sync(0xffffffffu, __float_as_uint(est));
            if (lane == 0 && least < *reinterpret_cast<volatile unsigned*>(&s_least)) atomicMin(&s_least, least);
        };
        auto in_order = [&](int ti) {  // the whole warp: the metric of test ti, kept if the best
            const Test q = test_at(ti);
            const unsigned word = lane < MW ? word_at(q, lane) : 0u;
            int above = __popc(word);  // set bits in this word and the later ones, then in the later ones
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_down_sync(0xffffffffu, above, o);
                if (lane + o < 32) above += x;
            }
            const int total_bits = __shfl_sync(0xffffffffu, above, 0);
            above -= __popc(word);
            int cut[3], flips = 0;
#pragma unroll
            for (int i = 0; i < 3; ++i) {  // pivots at positions above the flip's (pivj decreases with rank)
                cut[i] = -1;
                if (q.j[i] == INT_MAX) continue;
                int lo = 0, hi = m;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s.pivj[mid] > q.j[i]) lo = mid + 1;
                    else hi = mid;
                }
                cut[i] = lo;
                // its place: after the differing pivots of rank >= cut and the flips before it
                const int c = lo - 32 * lane;  // bits c .. 31 of this word have rank >= cut
                const unsigned later = c <= 0 ? word : c >= 32 ? 0u : word & ~((1u << c) - 1u);
                const int at = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(__popc(later)))) + i;
                if (lane == 0) terms[at] = s.rel[q.j[i]];
                ++flips;
            }
            for (unsigned left = word; left;) {
                const int b = 31 - __clz(left), rank = 32 * lane + b;
                left &= ~(1u << b);
                terms[above + (cut[0] > rank) + (cut[1] > rank) + (cut[2] > rank)] = s.relq[rank];
                ++above;
            }
            const int total = total_bits + flips;
            if (lane < 4) terms[total + lane] = 0.0f;  // the last group of four adds zeros: no change
            __syncwarp();
            if (lane == 0) {
                float acc = 0.0f;
                for (int i = 0; i < total; i += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(terms + i);
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, x.x), x.y), x.z), x.w);
                }
                atomicMin(&s_best, (static_cast<unsigned long long>(__float_as_uint(acc)) << 32) | static_cast<unsigned>(ti));
            }
            __syncwarp();  // the terms are rewritten by the next test
        };
        {
            // a warp's first 32 tests are estimated before any is summed, so that those meet the least
            // estimate of all the first tests
            float first = INFINITY;
            const int ti0 = warp * 32 + lane;
            if (ti0 < hv.num_tests) first = estimate(test_at(ti0));
            if (warp * 32 < hv.num_tests) note(first);
            __syncthreads();
            for (int t0 = warp * 32; t0 < hv.num_tests; t0 += kThreads) {
                const int ti = t0 + lane;
                float est = first;
                if (t0 != warp * 32) {
                    est = ti < hv.num_tests ? estimate(test_at(ti)) : INFINITY;
                    note(est);
                }
                const float least = __uint_as_float(*reinterpret_cast<volatile unsigned*>(&s_least));
                unsigned pass = __ballot_sync(0xffffffffu, ti < hv.num_tests && !(est > least * (1.0f + 2.44140625e-04f)));
                for (; pass; pass &= pass - 1) in_order(t0 + __ffs(pass) - 1);
            }
        }
        __syncthreads();

        // ---- 7. the winning codeword ----
        const unsigned long long best = s_best;
        const int bt = static_cast<int>(best & 0xffffffffull);
        int fl[3], fpos[3], nf = 0;
        if (bt > 0) {
            const uint32_t pk = hv.combos[bt - 1];
            for (int q = 0; q < 3; ++q) {
                const int f = (pk >> (10 * q)) & 1023;
                if (f != 1023) {
                    fl[nf] = f;
                    fpos[nf] = s.perm[s.pool_j[f]];
                    ++nf;
                }
            }
        }
        auto bit_at = [&](int i) -> uint8_t {
            unsigned bit = tbit(s.hard, i);
            const int r = s.row_of_col[i];
            if (r >= 0) {
                unsigned word = s.aug[r >> 5];
                for (int q = 0; q < nf; ++q) word ^= s.avec[fl[q] * MW + (r >> 5)];
                bit ^= (word >> (r & 31)) & 1u;
            } else {
                for (int q = 0; q < nf; ++q) bit ^= (fpos[q] == i) ? 1u : 0u;
            }
            return static_cast<uint8_t>(bit);
        };
        if (info_dst)
            for (int i = tid; i < k; i += kThreads) info_dst[i] = bit_at(i);
        if (io.out_code)
            for (int i = tid; i < n; i += kThreads) io.out_code[static_cast<size_t>(cw) * n + i] = bit_at(i);
        if (tid == 0) {
            if (io.used_osd) io.used_osd[cw] = 1;
            if (io.out_metric) io.out_metric[cw] = __uint_as_float(static_cast<unsigned>(best >> 32));
        }
        __syncthreads();  // shared memory is rewritten by the next item
    }
}

namespace {

OsdHLayout osd_h_layout(const OsdHBounds& bd, int mlo, int mhi)
{
    OsdHLayout l{};
    l.nmax = bd.nmax;
    l.np = 1;
    while (l.np < bd.nmax) l.np <<= 1;
    l.mw = (bd.mmax + 31) / 32;
    l.ts = l.mw | 1;
    l.poolmax = std::max(bd.poolmax, 1);
    l.mlo = mlo;
    l.mhi = mhi;
    return l;
}

template <int kThreads>
void launch_osd_h_class(const OsdHBounds& bd, int mlo, int mhi, const OsdIO& io_all, int max_items, cudaStream_t st,
                        int cls)
{
    OsdIO io = io_all;  // the class's own work counter
    io.work_h = io_all.work_h ? io_all.work_h + cls : nullptr;
    OsdHLayout l = osd_h_layout(bd, mlo, mhi);
    const size_t smem = carve(l, nullptr, nullptr);
    if (smem > 227 * 1024) throw InvalidArgument("large-code OSD tables exceed shared memory (m <= 1024, n <= 4096)");
    // the narrow classes share this kernel with different sizes: the limit only grows
    check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(osd_h_kernel<kThreads>), smem),
               "cudaFuncSetAttribute(osd_h)");
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, osd_h_kernel<kThreads>, kThreads, smem) != cudaSuccess ||
        per_sm <= 0)
        per_sm = 1;
    const int ctas = std::max(1, std::min(max_items, per_sm * device_sm_count()));
    osd_h_kernel<kThreads><<<ctas, kThreads, smem, st>>>(OsdHView{}, l, io);
    check_cuda(cudaGetLastError(), "osd_h_kernel launch");
}

}  // namespace

void OsdHBounds::add(int n, int m, int pool)
{
    nmax = std::max(nmax, n);
    mmax = std::max(mmax, m);
    poolmax = std::max(poolmax, pool);
}

size_t osd_h_smem_bytes(int nmax, int mmax, int poolmax)
{
    OsdHBounds bd;
    bd.add(nmax, mmax, poolmax);
    const OsdHLayout l = osd_h_layout(bd, 0, 1024);
    return carve(l, nullptr, nullptr);
}

void launch_osd_h(const OsdHBounds* cls, const OsdIO& io, int max_items, cudaStream_t st, const cudaStream_t* side,
                  cudaEvent_t fork, const cudaEvent_t* join)
{
    if (max_items <= 0) return;
    int present = 0;
    for (int c = 0; c < kOsdHClasses; ++c) {
        if (cls[c].empty()) continue;
        ++present;
        if (cls[c].nmax > 32767 || cls[c].poolmax > kOsdHMaxPool)
            throw InvalidArgument("large-code OSD: n <= 32767, pool <= 128");
        if (cls[c].mmax > kOsdHClassMaxM[c]) throw InvalidArgument("large-code OSD: code in the wrong class (m <= 1024)");
    }
    if (present == 0) return;
    if (io.work_h && !io.work_zeroed)
        check_cuda(cudaMemsetAsync(io.work_h, 0, kOsdHClasses * sizeof(int), st), "reset OSD work counters");
    // the classes run side by side: the first present one on st, the others on side streams
    const bool fan = present > 1 && side && fork && join;
    if (fan) check_cuda(cudaEventRecord(fork, st), "cudaEventRecord(osd fork)");
    int used = 0;
    for (int c = kOsdHClasses - 1; c >= 0; --c) {
        if (cls[c].empty()) continue;
        cudaStream_t cs = st;
        if (fan && used > 0) {
            cs = side[used - 1];
            check_cuda(cudaStreamWaitEvent(cs, fork, 0), "cudaStreamWaitEvent(osd fork)");
        }
        const int mlo = c == 0 ? 0 : kOsdHClassMaxM[c - 1];
        if (kOsdHClassThreads[c] == kOsdHNarrow) launch_osd_h_class<kOsdHNarrow>(cls[c], mlo, kOsdHClassMaxM[c], io, max_items, cs, c);
        else launch_osd_h_class<kOsdHWide>(cls[c], mlo, kOsdHClassMaxM[c], io, max_items, cs, c);
        if (fan && used > 0) {
            check_cuda(cudaEventRecord(join[used - 1], cs), "cudaEventRecord(osd join)");
            check_cuda(cudaStreamWaitEvent(st, join[used - 1], 0), "cudaStreamWaitEvent(osd join)");
        }
        ++used;
    }
}

}  // namespace sicc
