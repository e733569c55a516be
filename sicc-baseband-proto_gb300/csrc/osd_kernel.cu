// Ordered-statistics decoding (OSD) for sm_103a: one warp per codeword.
//
// Restates cpu_bp_osd_decode.m:187-305 (the reference's MATLAB BP-OSD):
//   1. stable descending sort of |llr| (ties: lower index first);
//   2. systematic form of the column-permuted generator G = [I_k | P]: the
//      pivots are the first k linearly independent positions in reliability
//      order (the most reliable basis), found by a column scan over a
//      bit-packed row-reduced copy of G held in registers (64-bit XOR rows);
//   3. base candidate = hard decisions on the basis; flip candidates over the
//      weakest basis positions in the enumeration order of MATLAB nchoosek;
//   4. metric = sum of |llr| over positions where the candidate differs from
//      the hard decision, accumulated in decreasing-reliability order in
//      single precision; the first candidate with the smallest metric wins
//      (strict <, cpu_bp_osd_decode.m:222), realised as a minimum over
//      (metric bits, test index) keys.
// Candidates are tested by all 32 lanes in parallel; each candidate's
// difference vector is the base difference XOR at most three reduced rows.  A
// lower bound of the metric from nibble tables screens them; the few that pass
// are summed in order, stopping once over the best metric.  Both only drop
// candidates that cannot win.
//
// What bounds it: instruction issue and the ALU pipe.  Measured on GB300, the
// 13,000 failed codewords of 65,536 (128,64) frames at 2 dB (13,400 warp
// instructions each before): 265 us with a broadcast pivot row per column and
// every surviving candidate summed in order, 187 us now.
#include "bp_kernels.h"

#include <algorithm>

namespace sicc {

namespace {

constexpr int kOsdWarps = 8;

// Small shapes also keep the reduced rows in flip-pool order, so a candidate reads its
// flipped rows without the rank lookup (the larger shapes would lose occupancy to it).
template <int NW, int KR>
constexpr bool kFlipRows = NW * KR <= 4;

// The tail: sorted positions from 64 (NW / 2) on, the less reliable half (all of them at NW = 1),
// where nearly all parity positions lie.
template <int NW>
constexpr int kTailWord = NW / 2;
template <int NW>
constexpr int kTailNibbles = (NW - NW / 2) * 16;

template <int NW, int KR>
struct OsdSmem {
    float rel_sorted[NW * 64];
    int16_t perm[NW * 64];
    int16_t rowpiv[KR * 32];  // row id -> pivot index
    int16_t flip[KR * 32];    // weakness rank -> pivot index
    union {
        unsigned long long rows[KR * 32][NW];  // reduced rows by pivot index
        struct {  // before them, during the elimination:
            unsigned long long raw[8][NW];     // the round's pivot rows as the round found them
            unsigned long long tab[32][NW];    // XORs of raw[0..3] by 4-bit index, then of raw[4..7]
        } el;
    };
    unsigned long long frows[kFlipRows<NW, KR> ? KR * 32 : 1][NW];  // the same rows by flip-pool rank
    int16_t mrb_pos[KR * 32];
    float prel[KR * 32];      // flip-pool rank -> |llr| of its position (non-decreasing)
    float low[KR * 32];       // the same where the position lies below kTail, else 0
    float nib[kTailNibbles<NW>][16];  // sums of |llr| over the set bits of each nibble of the tail
    int16_t rstart[KR * 32];  // order-2 rows: first surviving pair of row a in the compact list
};

// Word `w` of a register array, selected without dynamic indexing (which
// would move the array to local memory).
template <int NW>
__device__ __forceinline__ unsigned long long pick(const unsigned long long (&a)[NW], int w)
{
    unsigned long long r = 0ull;
#pragma unroll
    for (int i = 0; i < NW; ++i)
        if (i == w) r = a[i];
    return r;
}

__device__ __forceinline__ unsigned long long shfl_xor_u64(unsigned long long v, int m)
{
    const unsigned lo = __shfl_xor_sync(0xffffffffu, static_cast<unsigned>(v), m);
    const unsigned hi = __shfl_xor_sync(0xffffffffu, static_cast<unsigned>(v >> 32), m);
    return (static_cast<unsigned long long>(hi) << 32) | lo;
}

}  // namespace

// kRounds: the best metric is exchanged at a given interval (a launch shape's choice), an instance of its
// own: a test of the interval in the default loop cost 1-4% of the whole (128,64) decode.  16,384 frames:
// order 2 at 2 dB 221 us with an exchange after each pass, 228 every 8, 233 every 64; order 3 at 1 dB
// 491, 536, 592.
template <int NW, int KR, bool kRounds>
__global__ void __launch_bounds__(kOsdWarps * 32)
osd_kernel(OsdView ov0, OsdIO io)
{
    constexpr int KW = (KR + 1) / 2;
    __shared__ OsdSmem<NW, KR> sm_all[kOsdWarps];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    OsdSmem<NW, KR>& s = sm_all[warp];
    const int count = io.count_ptr ? *io.count_ptr : io.count;
    const int total_warps = gridDim.x * kOsdWarps;

    auto next_item = [&](int prev) -> int {  // the warp's next work item
        if (!io.work) return prev < 0 ? static_cast<int>(blockIdx.x) * kOsdWarps + warp : prev + total_warps;
        int it = 0;
        if (lane == 0) it = atomicAdd(io.work, 1);
        return __shfl_sync(0xffffffffu, it, 0);
    };
    for (int item = next_item(-1); item < count; item = next_item(item)) {
        const int cw = io.index ? io.index[item] : item;
        const OsdView ov = io.views ? io.views[io.code_of[cw]] : ov0;
        if (ov.n == 0) continue;  // code without warp-kernel tables (uniform over the warp)
        const int n = ov.n, k = ov.k;
        const float* src = io.row_off   ? io.llr + io.row_off[item]
                           : io.llr_off ? io.llr + io.llr_off[cw]
                                        : io.llr + static_cast<size_t>(item) * n;
        uint8_t* info_dst = io.out_info ? (io.info_off ? io.out_info + io.info_off[cw]
                                                       : io.out_info + static_cast<size_t>(cw) * io.info_stride)
                                        : nullptr;
        // ---- 1. reliabilities, hard decisions, stable descending sort ----
        // Bitonic sort of 64-bit keys in registers (element lane * KPL + q in v[q]): ascending key =
        // descending |llr|, ties by ascending index (the order of MATLAB's stable sort,
        // cpu_bp_osd_decode.m:194).  The lowest bit carries the hard decision (the index above it is
        // unique, so it orders nothing).  The merge levels and the distances across lanes are
        // run-time loops: unrolled, the sort alone would be 30 KB of code and every warp would
        // wait for instructions.
        constexpr int NP = NW * 64, KPL = NP / 32;
        unsigned long long v[KPL];
        auto key = [&](int i, float x) -> unsigned long long {
            return (static_cast<unsigned long long>(0x7fffffffu - __float_as_uint(fabsf(x))) << 32) |
                   static_cast<unsigned>(2 * i + (x < 0.0f ? 1 : 0));
        };
        if (n == NP && (reinterpret_cast<uintptr_t>(src) & 15u) == 0 && KPL % 4 == 0) {
#pragma unroll
            for (int q = 0; q + 4 <= KPL; q += 4) {
                const int i = lane * KPL + q;
                const float4 x = *reinterpret_cast<const float4*>(src + i);
                v[q] = key(i, x.x);
                v[q + 1] = key(i + 1, x.y);
                v[q + 2] = key(i + 2, x.z);
                v[q + 3] = key(i + 3, x.w);
            }
        } else {
#pragma unroll
            for (int q = 0; q < KPL; ++q) {
                const int i = lane * KPL + q;
                v[q] = (i < n) ? key(i, src[i]) : ~0ull;
            }
        }
#pragma unroll 1
        for (int k2 = 2; k2 <= NP; k2 <<= 1) {
            const bool up = ((lane * KPL) & k2) == 0;  // the order of my elements, for k2 >= KPL
#pragma unroll 1
            for (int j2 = k2 >> 1; j2 >= KPL; j2 >>= 1) {  // partner in another lane
                const int m = j2 / KPL;
                const bool take_min = ((lane & m) == 0) == up;
#pragma unroll
                for (int q = 0; q < KPL; ++q) {
                    const unsigned long long o = shfl_xor_u64(v[q], m);
                    v[q] = ((o < v[q]) == take_min) ? o : v[q];
                }
            }
#pragma unroll
            for (int j2 = KPL / 2; j2 > 0; j2 >>= 1) {  // partner in this lane
                if (j2 >= k2) continue;
#pragma unroll
                for (int q = 0; q < KPL; ++q) {
                    if (q & j2) continue;
                    const bool asc = k2 >= KPL ? up : (q & k2) == 0;
                    const unsigned long long x = v[q], y = v[q | j2];
                    if ((x > y) == asc) {
                        v[q] = y;
                        v[q | j2] = x;
                    }
                }
            }
        }
        unsigned hb = 0u;  // hard decisions of my KPL sorted positions
#pragma unroll
        for (int q = 0; q < KPL; ++q) {
            const int r = lane * KPL + q;
            if (r < n) {
                s.perm[r] = static_cast<int16_t>((v[q] & 0xffffffffull) >> 1);
                s.rel_sorted[r] = __uint_as_float(0x7fffffffu - static_cast<unsigned>(v[q] >> 32));
                hb |= (static_cast<unsigned>(v[q]) & 1u) << q;
            }
        }
        // hard decisions in sorted order: 32 / KPL lanes per half-word
        unsigned long long hard_sorted[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            unsigned half[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                constexpr int per = 32 / KPL;
                const unsigned mine = lane / per == 2 * w + h ? hb << ((lane % per) * KPL) : 0u;
                half[h] = __reduce_or_sync(0xffffffffu, mine);
            }
            hard_sorted[w] = (static_cast<unsigned long long>(half[1]) << 32) | half[0];
        }
        __syncwarp();
        // ---- 2. permuted generator rows via ballots over column vectors ----
        unsigned long long rows[KR][NW];
#pragma unroll
        for (int a = 0; a < KR; ++a)
#pragma unroll
            for (int w = 0; w < NW; ++w) rows[a][w] = 0ull;
#pragma unroll
        for (int q = 0; q < NW * 2; ++q) {
            const int j = q * 32 + lane;
            unsigned long long col[KW];
#pragma unroll
            for (int x = 0; x < KW; ++x) col[x] = 0ull;
            if (j < n) {
                const int o = s.perm[j];
                if (o < k) {
                    col[o >> 6] = 1ull << (o & 63);
                } else {
#pragma unroll
                    for (int x = 0; x < KW; ++x)  // the code's own words (kw <= KW)
                        col[x] = x < ov.kw ? ov.pcols[static_cast<size_t>(o - k) * ov.kw + x] : 0ull;
                }
            }
            // 32 x 32 bit transposes (butterfly over lane ^ j): lane j's bits a*32.. of its
            // column become lane r's bits q*32.. of row a*32 + r
#pragma unroll
            for (int a = 0; a < KR; ++a) {
                unsigned x = static_cast<unsigned>(col[a >> 1] >> ((a & 1) * 32));
                unsigned msk = 0x0000FFFFu;
#pragma unroll
                for (int jj = 16; jj > 0; jj >>= 1) {
                    const unsigned y = __shfl_xor_sync(0xffffffffu, x, jj);
                    x = (lane & jj) ? ((x & ~msk) | ((y & ~msk) >> jj)) : ((x & msk) | ((y & msk) << jj));
                    msk ^= msk << (jj >> 1);
                }
                if (a * 32 + lane < k) rows[a][q >> 1] |= static_cast<unsigned long long>(x) << ((q & 1) * 32);
            }
        }
        // ---- 3. column-scan elimination: pivots = most reliable basis ----
        // Columns are taken 8 at a time (a byte of every row).  Within a round only the bytes are
        // eliminated, column by column: val[a] holds my row's byte (bits 0-7) and which of the
        // round's pivot rows it has taken (bits 8-15, over the rows as they were before the
        // round), so one shuffle and one XOR per column update both.  The rows themselves take
        // the round at once, from the XORs of the 8 pivot rows tabulated by 4-bit index: two
        // table reads per row instead of a broadcast row and a test per column.
        unsigned avail[KR];  // 0xff while my row in slot a exists (r < k) and is not yet a pivot row
#pragma unroll
        for (int a = 0; a < KR; ++a) avail[a] = (a * 32 + lane < k) ? 0xffu : 0u;
        int rank = 0;
        {
#pragma unroll 1
            for (int j0 = 0; j0 < n && rank < k; j0 += 8) {
                unsigned val[KR];
                int took[KR];  // this round: column << 8 | rank of the pivot my row became, -1 for none
#pragma unroll
                for (int a = 0; a < KR; ++a) {
                    val[a] = static_cast<unsigned>(pick<NW>(rows[a], j0 >> 6) >> (j0 & 63)) & 0xffu;
                    took[a] = -1;
                }
                const int before = rank;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    if (j0 + r >= n || rank >= k) break;
                    int ps = -1, pl = 0;
                    unsigned pv = 0u;
#pragma unroll
                    for (int a = 0; a < KR; ++a) {
                        const unsigned bal = __ballot_sync(0xffffffffu, (val[a] & avail[a] & (1u << r)) != 0u);
                        if (ps < 0 && bal) {
                            ps = a;
                            pl = __ffs(bal) - 1;
                            pv = val[a];
                        }
                    }
                    if (ps < 0) continue;  // dependent position
                    pv = __shfl_sync(0xffffffffu, pv, pl) ^ (0x100u << r);
#pragma unroll
                    for (int a = 0; a < KR; ++a) {
                        const bool is_p = lane == pl && a == ps;
                        if ((val[a] & (1u << r)) && !is_p) val[a] ^= pv;
                        if (is_p) {
                            avail[a] = 0u;
                            took[a] = (r << 8) | rank;
                        }
                    }
                    ++rank;
                }
                if (rank == before) continue;
#pragma unroll
                for (int a = 0; a < KR; ++a) {
                    if (took[a] >= 0) {  // the row as it was before the round
                        const int r = took[a] >> 8, t = took[a] & 0xff;
#pragma unroll
                        for (int w = 0; w < NW; ++w) s.el.raw[r][w] = rows[a][w];
                        s.rowpiv[a * 32 + lane] = static_cast<int16_t>(t);
                        s.mrb_pos[t] = static_cast<int16_t>(j0 + r);
                    }
                }
                __syncwarp();
                {  // entry `lane`: XOR of the rows its low 4 bits select (rows of dependent columns are never selected)
                    const int h = (lane >> 4) * 4;
#pragma unroll
                    for (int w = 0; w < NW; ++w) {
                        unsigned long long x = 0ull;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if ((lane >> i) & 1) x ^= s.el.raw[h + i][w];
                        s.el.tab[lane][w] = x;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int a = 0; a < KR; ++a) {
                    const unsigned lo = (val[a] >> 8) & 15u, hi = 16u + ((val[a] >> 12) & 15u);
#pragma unroll
                    for (int w = 0; w < NW; ++w) rows[a][w] ^= s.el.tab[lo][w] ^ s.el.tab[hi][w];
                }
                __syncwarp();  // read before the next round writes
            }
        }
        __syncwarp();
        if (rank < k) {  // generator not full rank: cannot happen for a valid code table
            if (lane == 0 && io.out_metric) io.out_metric[cw] = -1.0f;
            continue;
        }
        // ---- 4. reduced rows by pivot index; base difference vector ----
        unsigned long long acc[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) acc[w] = 0ull;
#pragma unroll
        for (int a = 0; a < KR; ++a) {
            const int r = a * 32 + lane;
            if (r < k) {
                const int t = s.rowpiv[r];
#pragma unroll
                for (int w = 0; w < NW; ++w) s.rows[t][w] = rows[a][w];
                const int pj = s.mrb_pos[t];
                if ((pick<NW>(hard_sorted, pj >> 6) >> (pj & 63)) & 1ull) {
#pragma unroll
                    for (int w = 0; w < NW; ++w) acc[w] ^= rows[a][w];
                }
            }
        }
#pragma unroll
        for (int w = 0; w < NW; ++w) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[w] ^= shfl_xor_u64(acc[w], o);
            acc[w] ^= hard_sorted[w];  // base difference from the hard decision
        }
        // ---- 5. flip pool: basis positions, weakest first (stable) ----
        // Pivots come in sorted-position order, so |llr| does not increase with the pivot
        // index t: t's rank is the count of later runs plus its place in its run of equal
        // |llr| (the run found by binary search).
        // |llr| compared as bit patterns, the order the sort used (a permutation whatever the values)
        auto relbits = [&](int t) -> unsigned { return __float_as_uint(s.rel_sorted[s.mrb_pos[t]]); };
        for (int t = lane; t < k; t += 32) {
            const unsigned bt = relbits(t);
            int lo = 0, hi = t;  // first index with |llr| <= bt
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (relbits(mid) > bt) lo = mid + 1;
                else hi = mid;
            }
            const int a = lo;
            lo = t + 1;
            hi = k;  // first index with |llr| < bt
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (relbits(mid) < bt) hi = mid;
                else lo = mid + 1;
            }
            const int r = (k - lo) + (t - a);
            if (r < ov.pool) {
                s.flip[r] = static_cast<int16_t>(t);
                s.prel[r] = s.rel_sorted[s.mrb_pos[t]];
                s.low[r] = s.mrb_pos[t] < kTailWord<NW> * 64 ? s.prel[r] : 0.0f;
                if (kFlipRows<NW, KR>)
#pragma unroll
                    for (int w = 0; w < NW; ++w) s.frows[kFlipRows<NW, KR> ? r : 0][w] = s.rows[t][w];
            }
        }
        // sums of |llr| over the set bits of every nibble of the tail
        for (int e = lane; e < kTailNibbles<NW> * 16; e += 32) {
            const float* rel = s.rel_sorted + kTailWord<NW> * 64 + (e >> 4) * 4;
            float x = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (((e >> i) & 1) && kTailWord<NW> * 64 + (e >> 4) * 4 + i < n) x += rel[i];
            (&s.nib[0][0])[e] = x;
        }
        __syncwarp();
        // ---- 6. all candidates in parallel ----
        // A candidate's metric is a sum of non-negative terms in a fixed order, so
        // its partial sums never decrease: once one exceeds the smallest metric
        // already found the candidate cannot win and its sum stops.  Ties are not
        // pruned (strict >), so the first minimum in test order still wins.
        // Before that walk a candidate meets a bound: its differing positions of the tail summed
        // from the nibble tables, plus its flips before the tail.  All terms are non-negative; the
        // metric's own sum (up to 256 terms in order) lies below the exact one by less than 255
        // rounding units and the bound above its exact value by less than 30, so a candidate whose
        // bound is over the best metric by a factor 1 + 2^-15 (512 units) cannot win.  The bound
        // takes the same 16 (or 32) steps in every lane, and few candidates pass it.
        unsigned long long best_key = ~0ull;
        float thr = INFINITY;
        auto flip_row = [&](int rank) -> const unsigned long long* {
            if constexpr (kFlipRows<NW, KR>) return s.frows[rank];
            else return s.rows[s.flip[rank]];
        };
        auto bound = [&](int f0, int f1, int f2) -> float {  // flips: pool ranks, -1 for none
            const int fl[3] = {f0, f1, f2};
            float lb = 0.0f;
            unsigned long long d[NW - kTailWord<NW>];
#pragma unroll
            for (int w = kTailWord<NW>; w < NW; ++w) d[w - kTailWord<NW>] = acc[w];
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                const int fi = fl[f];
                if (fi >= 0) {
                    lb += s.low[fi];
                    const unsigned long long* row = flip_row(fi);
#pragma unroll
                    for (int w = kTailWord<NW>; w < NW; ++w) d[w - kTailWord<NW>] ^= row[w];
                }
            }
            float part[2] = {lb, 0.0f};
#pragma unroll
            for (int i = 0; i < kTailNibbles<NW>; ++i) {
                const unsigned x = static_cast<unsigned>(d[i >> 4] >> ((i & 8) * 4));
                part[i & 1] += s.nib[i][(x >> ((i & 7) * 4)) & 15u];
            }
            return part[0] + part[1];
        };
        constexpr float kSlack = 1.0f + 3.0517578125e-05f;  // 1 + 2^-15
        // The metric of test q, whose flips are pool ranks f0, f1, f2 (-1: none), pruned against thr.
        auto evaluate = [&](int q, int f0, int f1, int f2) {
            unsigned long long d[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) d[w] = acc[w];
            const int fl[3] = {f0, f1, f2};
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                if (fl[f] < 0) continue;
                const unsigned long long* row = flip_row(fl[f]);
#pragma unroll
                for (int w = 0; w < NW; ++w) d[w] ^= row[w];
            }
            float metric = 0.0f;
            bool pruned = false;
#pragma unroll 1
            for (int h = 0; h < 2 * NW && !pruned; ++h) {
                unsigned bits = static_cast<unsigned>(pick<NW>(d, h >> 1) >> ((h & 1) * 32));
                const float* rel = s.rel_sorted + h * 32;
                while (bits && !pruned) {
                    const int b = __ffs(bits) - 1;
                    metric = __fadd_rn(metric, rel[b]);
                    bits &= bits - 1;
                    pruned = metric > thr;
                }
            }
            if (!pruned) {
                const unsigned long long key =
                    (static_cast<unsigned long long>(__float_as_uint(metric)) << 32) | static_cast<unsigned>(q);
                if (key < best_key) {
                    best_key = key;
                    thr = fminf(thr, metric);
                }
            }
        };
        auto share_best = [&]() {  // the best metric so far, to every lane
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = shfl_xor_u64(best_key, o);
                best_key = other < best_key ? other : best_key;
            }
            if (best_key != ~0ull) thr = __uint_as_float(static_cast<unsigned>(best_key >> 32));
        };
        const int P = ov.pool;
        // Complete order 2: the tests are the base, the P single flips, then every pair (a, b),
        // a < b, in lexicographic order (test 1 + P + a (2P - a - 1) / 2 + b - a - 1).  A candidate
        // differs from the hard decision at its flipped positions, and the metric, summed in
        // position order, is at least those terms summed alone (each rounded partial sum of a sum
        // of non-negative terms is at least that of any of its subsequences): a pair whose two
        // |llr| already add up above the best metric of the base and single-flip tests cannot win.
        // The pool is weakest first, so within row a the bound grows with b and each row keeps a
        // prefix (binary search); only those pairs are tested, 32 at a time from a compact list.
        const bool complete2 = P >= 2 && ov.num_tests == 1 + P + P * (P - 1) / 2;
        const int single = 1 + P;
        auto list_pairs = [&]() -> int {  // rstart of every row; the number of pairs kept
            const int R = (P - 1 + 31) / 32;  // rows a = 0 .. P-2, R consecutive rows per lane
            int mine = 0;
            for (int i = 0; i < R; ++i) {
                const int a = lane * R + i;
                int cnt = 0;
                if (a < P - 1) {
                    const float ra = s.prel[a];
                    int lo = a + 1, hi = P;  // first b with bound > thr
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (__fadd_rn(ra, s.prel[mid]) > thr) hi = mid;
                        else lo = mid + 1;
                    }
                    cnt = lo - (a + 1);
                }
                if (a < P - 1) s.rstart[a] = static_cast<int16_t>(mine);  // lane-local offset for now
                mine += cnt;
            }
            int incl = mine;  // inclusive scan of the lanes' pair counts
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const int base = incl - mine;
            for (int i = 0; i < R; ++i) {
                const int a = lane * R + i;
                if (a < P - 1) s.rstart[a] = static_cast<int16_t>(s.rstart[a] + base);
            }
            __syncwarp();
            return __shfl_sync(0xffffffffu, incl, 31);
        };
        // 32 tests per pass (one site for the bound, the sum and the exchange keeps the code small): first
        // the base test alone, then the tests from 1 on, and for complete order 2 the single flips, then
        // the pairs.  The best metric is exchanged after every pass that summed a test, or (kRounds) after
        // every io.share_rounds passes and at the end of a stage.
        int stage = 0, i0 = 0, end = 1, row = 0;
#pragma unroll 1
        while (true) {
            if (i0 >= end) {
                if (stage == 0) {
                    i0 = 1;
                    end = complete2 ? single : ov.num_tests;
                } else if (stage == 1 && complete2) {
                    i0 = 0;
                    end = list_pairs();
                } else {
                    break;
                }
                ++stage;
                continue;
            }
            const int i = i0 + lane;
            int q = i, f0 = -1, f1 = -1, f2 = -1;
            bool go = i < end;
            if (go && stage > 0) {
                if (!complete2) {
                    const uint32_t cmb = ov.combos[q - 1];
                    const uint32_t a = cmb & 0x3FFu, b = (cmb >> 10) & 0x3FFu, c = (cmb >> 20) & 0x3FFu;
                    f0 = a != 0x3FFu ? static_cast<int>(a) : -1;
                    f1 = b != 0x3FFu ? static_cast<int>(b) : -1;
                    f2 = c != 0x3FFu ? static_cast<int>(c) : -1;
                } else if (stage == 1) {
                    f0 = q - 1;
                } else {  // the last row with rstart[row] <= i (i only grows: walk forward)
                    while (row < P - 2 && s.rstart[row + 1] <= i) ++row;
                    f0 = row;
                    f1 = row + 1 + (i - s.rstart[row]);
                    q = single + f0 * (2 * P - f0 - 1) / 2 + (f1 - f0 - 1);
                }
                go = !(bound(f0, f1, f2) > thr * kSlack);
            }
            i0 += 32;
            if (!__any_sync(0xffffffffu, go) && (!kRounds || i0 < end)) continue;
            if (go) evaluate(q, f0, f1, f2);
            if (kRounds && i0 < end && (i0 >> 5) % io.share_rounds != 0) continue;
            share_best();
        }
        // ---- 7. winner -> original positions ----
        const int qbest = static_cast<int>(best_key & 0xffffffffull);
        unsigned long long d[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) d[w] = acc[w];
        if (qbest > 0) {
            const uint32_t cmb = ov.combos[qbest - 1];
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                const uint32_t fi = (cmb >> (10 * f)) & 0x3FFu;
                if (fi != 0x3FFu) {
                    const int t = s.flip[fi];
#pragma unroll
                    for (int w = 0; w < NW; ++w) d[w] ^= s.rows[t][w];
                }
            }
        }
#pragma unroll
        for (int w = 0; w < NW; ++w) d[w] ^= hard_sorted[w];  // decoded codeword in sorted order
        for (int j = lane; j < n; j += 32) {
            const int o = s.perm[j];
            const uint8_t bit = static_cast<uint8_t>((pick<NW>(d, j >> 6) >> (j & 63)) & 1ull);
            if (info_dst && o < k) info_dst[o] = bit;
            if (io.out_code) io.out_code[static_cast<size_t>(cw) * n + o] = bit;
        }
        if (lane == 0) {
            if (io.out_metric) io.out_metric[cw] = __uint_as_float(static_cast<unsigned>(best_key >> 32));
            if (io.used_osd) io.used_osd[cw] = 1;
        }
        __syncwarp();
    }
}

template <int NW, int KR, bool kRounds>
static void launch_osd_t(const OsdView& ov, const OsdIO& io, int max_items, cudaStream_t st, int ctas)
{
    if (ctas <= 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, osd_kernel<NW, KR, kRounds>, kOsdWarps * 32, 0) !=
                cudaSuccess ||
            per_sm <= 0)
            per_sm = 1;
        ctas = per_sm * device_sm_count();
        ctas = std::max(1, std::min(ctas, (max_items + kOsdWarps - 1) / kOsdWarps));
    }
    osd_kernel<NW, KR, kRounds><<<ctas, kOsdWarps * 32, 0, st>>>(ov, io);
    check_cuda(cudaGetLastError(), "osd_kernel launch");
}

void launch_osd(const OsdView& ov, const OsdIO& io, int max_items, cudaStream_t st, int warps_per_cta, int ctas)
{
    (void)warps_per_cta;
    if (max_items <= 0) return;
    if (io.work && !io.work_zeroed) check_cuda(cudaMemsetAsync(io.work, 0, sizeof(int), st), "reset OSD work counter");
    // for a mixed-code batch `ov` carries the largest n and k of its codes
    const int nw = (ov.n + 63) / 64;
    const int kr = (ov.k + 31) / 32;
    const int NW = nw <= 1 ? 1 : (nw <= 2 ? 2 : 4);
    const int KR = kr <= 1 ? 1 : (kr <= 2 ? 2 : 4);
    if (nw > 4 || kr > 4) throw InvalidArgument("OSD kernel supports n <= 256 and k <= 128");
#define SICC_OSD_CASE(A, B) \
    if (NW == A && KR == B) { \
        if (io.share_rounds > 1) launch_osd_t<A, B, true>(ov, io, max_items, st, ctas); \
        else launch_osd_t<A, B, false>(ov, io, max_items, st, ctas); \
        return; \
    }
    SICC_OSD_CASE(1, 1) SICC_OSD_CASE(1, 2) SICC_OSD_CASE(2, 1) SICC_OSD_CASE(2, 2)
    SICC_OSD_CASE(2, 4) SICC_OSD_CASE(4, 2) SICC_OSD_CASE(4, 4) SICC_OSD_CASE(4, 1) SICC_OSD_CASE(1, 4)
#undef SICC_OSD_CASE
    throw InvalidArgument("unsupported OSD shape");
}

}  // namespace sicc
