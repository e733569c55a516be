// OFDM receive kernels for sm_103a.
//
// sync_kernel (one CTA per frame and pass of 4352 candidates) restates the CPU receiver's frame search
// (uhd_ldpc_ofdm_link.cpp:5123-5329): Schmidl-Cox metric
//   P(d) = sum_{i<L} conj(x[d+i]) x[d+i+L],  E1 = sum |x[d+i]|^2,  E2 = sum |x[d+i+L]|^2,
//   metric(d) = |P|^2 / max(E1*E2, 1e-18);
// the earliest candidate over the threshold (or the global maximum), then a
// full-preamble cross-correlation refinement within +-radius, then the CFO
// arg(sum conj(x[s+i]) x[s+i+L]) * fs / (2 pi L).  Candidates are scanned in
// passes of 256 x 17 from a shared-memory copy of the samples (the odd chunk
// keeps shared-memory reads on distinct banks):
//   * the products of 17 consecutive samples are summed once, a window sum at a
//     chunk start is the sum of L / 17 such blocks and the last samples, and a
//     thread slides it over its 17 candidates (30 block sums instead of 512
//     products per chunk at L = 512);
//   * the fine metric is computed for four neighbouring positions at a time (one
//     read of the preamble and one energy sum for four), in increasing order, only
//     as far as the earliest position over the threshold decides the search, and
//     over half the preamble where the other half cannot reach the threshold.
// Every pass publishes its result to global scratch and the last pass of a
// frame to finish resolves the frame.  Measured on GB300, 256 frames of 16,888
// samples (1,024-sample preamble, 6-tap fading): 243 us with a product per
// sample and chunk and every position's fine metric, 57 us now (77 with the whole
// preamble everywhere on 256 threads); a frame's pass is one CTA, so it is bound by
// issue (57%) and by the barriers between its phases.
//
// demod_kernel (grid = frames x data-symbol groups) fuses the demodulator of
// gpu_ofdm_pipeline.cu:566-672 / uhd_ldpc_ofdm_link.cpp:5350-5521: CFO
// derotation and CP strip while loading, a shared-memory Stockham FFT
// (radix 4, plus one radix-2 stage for odd log2 N), LS pilot estimates with
// linear interpolation, MMSE equalisation and max-log LLRs.  The max-log
// search runs per constellation axis: for Gray square QAM the minimum of
// fl(dI^2) + fl(dQ^2) over a bit-constrained set splits into the two axis
// minima (single-precision addition is monotone in each argument), so the
// result equals the exhaustive 2^bps search of the reference bit for bit
// given the same equalised symbol.  Measured on GB300, 256 frames of 14 x 1,024
// (16-QAM): 52 us with a plain FFT buffer (half its shared-memory wavefronts
// were bank conflicts), one twiddle table read at strides and a sincospi per
// sample; 37 us with swizzled buffers, twiddles in reading order and one
// sincospi per four samples (taken together: 39 one after another).  The LLRs are 7.6e-7 (16-QAM) from
// double precision, 7.8e-7 with a sincospi of an unreduced angle per sample.  The transmitter shares the FFT: 256 frames,
// encoder 37 -> 17 us (parity words of the tables only), symbols 69 -> 35 us.
// Both are bound by instruction issue.
#include "ofdm_kernels.h"

#include <algorithm>
#include <cfloat>

#include <cstdint>

namespace sicc {

namespace {

constexpr int kSyncThreads = 512;
constexpr int kSyncOwners = 256;  // threads that own a chunk of coarse candidates
constexpr int kSyncChunk = 17;
constexpr int kSyncPass = kSyncOwners * kSyncChunk;
constexpr int kMaxRefine = 1024;  // 2 * radius + 1
constexpr int kMaxRadius = 511;

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                       __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

__device__ __forceinline__ float2 cmulconj(float2 a, float2 b)  // a * conj(b)
{
    return make_float2(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                       __fsub_rn(__fmul_rn(a.y, b.x), __fmul_rn(a.x, b.y)));
}

__device__ __forceinline__ float cnorm(float2 a) { return __fadd_rn(__fmul_rn(a.x, a.x), __fmul_rn(a.y, a.y)); }

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace

// One search result per pass, published to global scratch for the CTA that
// resolves the frame.
struct PassResult {
    int key;      // mode 0: earliest successful candidate (INT_MAX: none); mode 1: position of the maximum (-1: none)
    int start;    // mode 0: refined start
    float fine;   // mode 0: refined metric; mode 1: the maximum coarse metric
    float coarse; // mode 0: coarse metric at the candidate
};

// Full-preamble correlation metric of candidate dd, one warp: lane-strided
// products accumulated per lane with fused multiply-adds, then a butterfly
// sum.  Samples come from the shared window when it covers them
// (win[i] = x[wbase + i]).
__device__ __forceinline__ float fine_metric(const float2* __restrict__ x, const float2* win, int wbase, int wlen, int dd,
                                             const float2* __restrict__ preamble, int pre, float pre_energy, int lane)
{
    float cr = 0.f, ci = 0.f, eng = 0.f;
    const bool local = dd >= wbase && dd + pre <= wbase + wlen;
    for (int i = lane; i < pre; i += 32) {
        const float2 y = local ? win[dd - wbase + i] : x[dd + i];
        const float2 q = preamble[i];
        cr = fmaf(y.x, q.x, fmaf(y.y, q.y, cr));    // Re(y conj(q))
        ci = fmaf(y.y, q.x, fmaf(-y.x, q.y, ci));   // Im(y conj(q))
        eng = fmaf(y.x, y.x, fmaf(y.y, y.y, eng));  // |y|^2
    }
    cr = warp_sum(cr);
    ci = warp_sum(ci);
    eng = warp_sum(eng);
    return (cr * cr + ci * ci) / fmaxf(eng * pre_energy, 1e-18f);
}

// Samples of the preamble's first half, a multiple of a warp's 32.
__device__ __forceinline__ int fine_half(int pre) { return (pre >> 6) << 5; }

// fine_metric of the positions dd .. dd + 3, all inside the shared window (at win + at), pre >= 4,
// with one read of the preamble for the four and one energy sum: the samples common to the four,
// then each position's own ones (sums of non-negative terms only).  After the first half of the
// preamble |c| <= |c1| + sqrt(e2 E2) (e2, E2: energies of the other half of the samples and of the
// preamble), widened for the rounding of the sums: a lane adds pre / 32 times in each half, so c1, c,
// e2 and E2 together are off by less than 0.17 pre + 33 rounding units of sqrt(e E) (2^-24 each;
// pre / 4 + 64 are taken).  When that puts all four below the threshold they are reported as -1 and the
// other half is not correlated.  Preambles under 64 samples have no first half and no early stop.  Away from the preamble c1 is small and the bound about 1/4: most
// groups stop there (256 frames at threshold 0.45, search
// and demodulation: 120 us without the early stop and the shared energy, 106 with them).
__device__ __forceinline__ void fine_metric4(const float2* win, int at, const float2* __restrict__ preamble, int pre,
                                             float pre_energy, float tail_energy, float threshold, int lane,
                                             float (&out)[4])
{
    float cr[4] = {0.f, 0.f, 0.f, 0.f}, ci[4] = {0.f, 0.f, 0.f, 0.f}, e1 = 0.f, e2 = 0.f;
    const float2* y0 = win + at;
    auto correlate = [&](int i) {
        const float2 q = __ldg(preamble + i);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 y = y0[i + k];
            cr[k] = fmaf(y.x, q.x, fmaf(y.y, q.y, cr[k]));
            ci[k] = fmaf(y.y, q.x, fmaf(-y.x, q.y, ci[k]));
        }
    };
    auto energy = [&](int i, float e) { return fmaf(y0[i].x, y0[i].x, fmaf(y0[i].y, y0[i].y, e)); };
    const int half = fine_half(pre);
    int i = lane;
#pragma unroll 2
    for (; i < half; i += 32) {
        correlate(i);
        if (i > 2) e1 = energy(i, e1);
    }
#pragma unroll 4
    for (int t = i; t < pre; t += 32)
        if (t > 2) e2 = energy(t, e2);
    e2 = warp_sum(e2);
    const float common = warp_sum(e1) + e2;
    float eng[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        eng[k] = common;
#pragma unroll
        for (int j = 0; j < 3; ++j) eng[k] = energy(j >= k ? j : pre + j, eng[k]);
    }
    float over = e2;  // at least each position's energy against the preamble's other half
#pragma unroll
    for (int j = 0; j < 3; ++j) over = energy(pre + j, over);
    const float rest = sqrtf(over * tail_energy), widen = (0.25f * static_cast<float>(pre) + 64.0f) * 5.9604645e-08f;
    bool below = half > 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float r = warp_sum(cr[k]), j = warp_sum(ci[k]), full = eng[k] * pre_energy;
        const float most = sqrtf(r * r + j * j) + rest + widen * sqrtf(full);
        below = below && most * most < threshold * fmaxf(full, 1e-18f);
    }
    if (__all_sync(0xffffffffu, below)) {
#pragma unroll
        for (int k = 0; k < 4; ++k) out[k] = -1.0f;
        return;
    }
#pragma unroll 2
    for (; i < pre; i += 32) correlate(i);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float r = warp_sum(cr[k]), j = warp_sum(ci[k]);
        out[k] = (r * r + j * j) / fmaxf(eng[k] * pre_energy, 1e-18f);
    }
}

// Shared-memory working set of a frame search by one CTA.
struct SyncShared {
    float2* win;      // [kSyncPass + pre_len] the pass's samples (rounded up to an even count: the
                      // float4 block sums after the metric stay 16-byte aligned)
    float* metric;    // [kSyncPass] coarse metric
    float4* block;    // [kSyncOwners + L / kSyncChunk] sums over 17 samples: P.re, P.im, E1, E2;
                      // before the metric is complete, in memo's place
    float* memo;      // [kSyncPass + 2 * radius] fine metric around crossings
    uint16_t* list;   // [memo / 4] groups of four memo positions to evaluate, in increasing order
    float* red;       // [4][kSyncOwners / 32] reductions
    float* rmetric;   // [kMaxRefine] mode-1 refinement
    int* s_key;       // [kSyncThreads / 32 + 2]
    float* s_tail;    // energy of the preamble's other half (fine_metric4)
    PassResult* s_res;
};

__host__ __device__ inline int sync_memo(int radius) { return (kSyncPass + 2 * radius + 3) & ~3; }
__host__ __device__ inline size_t sync_memo_bytes(int pre_len, int radius)
{  // the fine metrics, or the block sums before them
    const size_t memo = static_cast<size_t>(sync_memo(radius)) * sizeof(float);
    const size_t block = static_cast<size_t>(kSyncOwners + pre_len / 2 / kSyncChunk) * sizeof(float4);
    return memo > block ? memo : block;
}
__host__ __device__ inline size_t sync_smem(int pre_len, int radius)
{
    return static_cast<size_t>((kSyncPass + pre_len + 1) & ~1) * sizeof(float2) + kSyncPass * sizeof(float) +
           sync_memo_bytes(pre_len, radius) + static_cast<size_t>(sync_memo(radius) / 4) * sizeof(uint16_t);
}

__device__ __forceinline__ SyncShared sync_shared(unsigned char* smem_raw, int pre_len, int radius, float* red,
                                                  float* rmetric, int* s_key, float* s_tail, PassResult* s_res)
{
    SyncShared sh;
    sh.win = reinterpret_cast<float2*>(smem_raw);
    sh.metric = reinterpret_cast<float*>(sh.win + ((kSyncPass + pre_len + 1) & ~1));
    sh.block = reinterpret_cast<float4*>(sh.metric + kSyncPass);
    sh.memo = sh.metric + kSyncPass;
    sh.list = reinterpret_cast<uint16_t*>(reinterpret_cast<unsigned char*>(sh.memo) + sync_memo_bytes(pre_len, radius));
    sh.red = red;
    sh.rmetric = rmetric;
    sh.s_key = s_key;
    sh.s_tail = s_tail;
    sh.s_res = s_res;
    return sh;
}

// One pass of the frame search over candidates [4352 pass, 4352 (pass + 1)) of x
// (avail samples, limit candidates), by the whole CTA.  Mode 0: *sh.s_res takes the
// pass's earliest successful crossing (key stays INT_MAX when none); mode 1: the
// pass maximum is folded into *sh.s_res.  Ends with a barrier.
__device__ void sync_scan_pass(const float2* __restrict__ x, int avail, int limit, int pass,
                               const float2* __restrict__ preamble, const SyncParams& p, const SyncShared& sh)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int L = p.half_len, pre = p.pre_len, R = p.radius;
    const int base = pass * kSyncPass;
    const int span = min(kSyncPass + pre, avail - base);
    for (int i = tid; i < kSyncPass + pre; i += kSyncThreads) sh.win[i] = (i < span) ? x[base + i] : make_float2(0.f, 0.f);
    __syncthreads();
    // chunks holding candidates below the limit (the rest only hold -1)
    const int nchunks = min(kSyncOwners, (limit - base + kSyncChunk - 1) / kSyncChunk);
    const int nb = L / kSyncChunk;
    for (int t = tid; t < nchunks + nb; t += kSyncThreads) {
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = t * kSyncChunk; i < (t + 1) * kSyncChunk; ++i) {
            const float2 u = sh.win[i], v = sh.win[i + L];
            const float2 c = cmulconj(v, u);  // conj(u) * v
            w.x += c.x;
            w.y += c.y;
            w.z += cnorm(u);
            w.w += cnorm(v);
        }
        sh.block[t] = w;
    }
    __syncthreads();
    if (tid >= kSyncOwners) {
        // the other threads share in the loads, the block sums and the fine metric
        if (warp == kSyncOwners / 32) {
            float e = 0.f;
            for (int i = fine_half(pre) + lane; i < pre; i += 32) {
                const float2 q = __ldg(preamble + i);
                e = fmaf(q.x, q.x, fmaf(q.y, q.y, e));
            }
            e = warp_sum(e);
            if (lane == 0) *sh.s_tail = e;
        }
    } else if (tid >= nchunks) {
        for (int c = 0; c < kSyncChunk; ++c) sh.metric[tid * kSyncChunk + c] = -1.0f;
    } else {
        const int d0 = tid * kSyncChunk;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = d0 + nb * kSyncChunk; i < d0 + L; ++i) {  // the window's last L mod 17 samples
            const float2 u = sh.win[i], v = sh.win[i + L];
            const float2 c = cmulconj(v, u);
            w.x += c.x;
            w.y += c.y;
            w.z += cnorm(u);
            w.w += cnorm(v);
        }
        for (int b = nb - 1; b >= 0; --b) {
            const float4 v = sh.block[tid + b];
            w.x += v.x;
            w.y += v.y;
            w.z += v.z;
            w.w += v.w;
        }
        for (int c = 0; c < kSyncChunk; ++c) {
            const int d = d0 + c;
            const float den = fmaxf(w.z * w.w, 1e-18f);
            sh.metric[d] = (base + d < limit) ? (w.x * w.x + w.y * w.y) / den : -1.0f;
            const float2 x0 = sh.win[d], x1 = sh.win[d + L], x2 = sh.win[d + pre];
            const float2 add = cmulconj(x2, x1), sub = cmulconj(x1, x0);
            w.x += add.x - sub.x;
            w.y += add.y - sub.y;
            w.z += cnorm(x1) - cnorm(x0);
            w.w += cnorm(x2) - cnorm(x1);
        }
    }
    __syncthreads();
    if (p.mode == 1) {
        // maximum of the pass, first occurrence (strict >)
        float bm = -1.0f;
        int bd = 0x7fffffff;
        for (int c = 0; c < kSyncChunk && tid < kSyncOwners; ++c) {
            const int d = tid * kSyncChunk + c;
            const float m = sh.metric[d];
            if (m > bm) { bm = m; bd = d; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, bm, o);
            const int od = __shfl_xor_sync(0xffffffffu, bd, o);
            if (om > bm || (om == bm && od < bd)) { bm = om; bd = od; }
        }
        if (lane == 0 && tid < kSyncOwners) { sh.red[warp] = bm; sh.red[8 + warp] = __int_as_float(bd); }
        __syncthreads();
        if (tid == 0) {
            for (int w = 0; w < kSyncOwners / 32; ++w) {
                const float m = sh.red[w];
                const int d = __float_as_int(sh.red[8 + w]);
                if (d == 0x7fffffff) continue;  // no valid candidate in that warp's chunks
                if (m > sh.s_res->fine || (m == sh.s_res->fine && base + d < sh.s_res->key)) {
                    sh.s_res->fine = m;
                    sh.s_res->key = base + d;
                }
            }
        }
    } else {
        // positions within +-R of a crossing of this pass: memo index i <-> sample x = base - R + i
        const int mspan = kSyncPass + 2 * R;
        {
            const int seg = (mspan + kSyncThreads - 1) / kSyncThreads;
            const int i0 = tid * seg, i1 = min(mspan, i0 + seg);
            auto crossing = [&](int y) -> int {  // memo index y holds candidate d = y - R
                const int d = y - R;
                return (d >= 0 && d < kSyncPass && sh.metric[d] >= p.threshold) ? 1 : 0;
            };
            int cnt = 0;
            if (i0 < i1)
                for (int y = i0 - R; y <= i0 + R; ++y) cnt += crossing(y);
            for (int i = i0; i < i1; ++i) {
                const int xs = base - R + i;
                sh.memo[i] = (cnt > 0 && xs >= 0 && xs <= avail - pre) ? -2.0f : -1.0f;
                cnt += crossing(i + R + 1) - crossing(i - R);
            }
        }
        // groups of four memo positions holding one to evaluate, listed in increasing order
        const int groups = (mspan + 3) / 4, per = (groups + kSyncThreads - 1) / kSyncThreads;
        if (tid < 4 * groups - mspan) sh.memo[mspan + tid] = -1.0f;
        if (tid == 0) {
            sh.s_key[kSyncThreads / 32] = 0x7fffffff;      // first memo position over the threshold
            sh.s_key[kSyncThreads / 32 + 1] = 0x7fffffff;  // the crossing that succeeds
        }
        __syncthreads();
        auto wanted = [&](int g) -> bool {
            const float4 v = reinterpret_cast<const float4*>(sh.memo)[g];
            return v.x == -2.0f || v.y == -2.0f || v.z == -2.0f || v.w == -2.0f;
        };
        int mine = 0;
        for (int g = tid * per; g < min(groups, (tid + 1) * per); ++g) mine += wanted(g) ? 1 : 0;
        int incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) sh.s_key[warp] = incl;
        __syncthreads();
        int at = incl - mine, total = 0;
        for (int w = 0; w < kSyncThreads / 32; ++w) {
            if (w < warp) at += sh.s_key[w];
            total += sh.s_key[w];
        }
        for (int g = tid * per; g < min(groups, (tid + 1) * per); ++g)
            if (wanted(g)) sh.list[at++] = static_cast<uint16_t>(g);
        __syncthreads();
        // The earliest crossing whose window (+-R) holds a fine metric over the threshold is the
        // first crossing within R of the first such position x: the windows of earlier ones end
        // before x.  So the positions are evaluated in order, until x and its 2R successors are.
        int* first_over = sh.s_key + kSyncThreads / 32;
        const bool every = !(p.threshold > 0.0f);  // any crossing succeeds then
        for (int b = 0; b < total; b += kSyncThreads / 32) {
            if (b + warp < total) {
                const int i0 = 4 * sh.list[b + warp], x0 = base - R + i0;
                float m[4];
                if (pre >= 4 && x0 >= base && x0 + 3 + pre <= base + span) {
                    fine_metric4(sh.win, x0 - base, preamble, pre, p.pre_energy, *sh.s_tail, p.threshold, lane, m);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        m[k] = sh.memo[i0 + k] == -2.0f ? fine_metric(x, sh.win, base, kSyncPass + pre, x0 + k, preamble,
                                                                       pre, p.pre_energy, lane)
                                                        : -1.0f;
                }
                __syncwarp();
                if (lane == 0) {
                    int over = 0x7fffffff;
#pragma unroll
                    for (int k = 3; k >= 0; --k) {
                        if (sh.memo[i0 + k] != -2.0f) continue;
                        sh.memo[i0 + k] = m[k];
                        if (m[k] >= p.threshold) over = i0 + k;
                    }
                    if (over != 0x7fffffff) atomicMin(first_over, over);
                }
            }
            __syncthreads();
            const int over = *first_over;
            __syncthreads();  // read by every thread before the next batch lowers it: all leave together
            if (!every && over != 0x7fffffff && 4 * sh.list[min(b + kSyncThreads / 32, total) - 1] + 3 >= over + 2 * R) break;
        }
        // the crossing: memo index x is sample base - R + x, so candidates d in [x - 2R, x]
        const int xo = *first_over;
        if (tid < kSyncOwners && (every || xo != 0x7fffffff)) {
            for (int c = 0; c < kSyncChunk; ++c) {
                const int d = tid * kSyncChunk + c;
                if (sh.metric[d] >= p.threshold && (every || (d >= xo - 2 * R && d <= xo))) {
                    atomicMin(first_over + 1, d);
                    break;
                }
            }
        }
        __syncthreads();
        const int d = first_over[1];
        if (d != 0x7fffffff && warp == 0) {  // the first maximum of its window, if above 0
            const int cand = base + d, lo = max(0, cand - R), hi = min(avail - pre, cand + R);
            float bm = 0.0f;
            int bd = 0x7fffffff;
            for (int dd = lo + lane; dd <= hi; dd += 32) {
                const float m = sh.memo[dd - base + R];
                if (m > bm) { bm = m; bd = dd; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const float om = __shfl_xor_sync(0xffffffffu, bm, o);
                const int od = __shfl_xor_sync(0xffffffffu, bd, o);
                if (om > bm || (om == bm && od < bd)) { bm = om; bd = od; }
            }
            if (lane == 0) {
                sh.s_res->key = cand;
                sh.s_res->start = bd == 0x7fffffff ? cand : bd;
                sh.s_res->fine = bm;
                sh.s_res->coarse = sh.metric[d];
            }
        }
    }
    __syncthreads();
}

// The record of a frame search from its resolved result `fin` (mode 1: refined
// first), with the CFO of the start found; valid in thread 0.  All threads call it.
__device__ SyncOut sync_finish(const float2* __restrict__ x, int avail, int limit, const PassResult fin,
                               const float2* __restrict__ preamble, const SyncParams& p, const SyncShared& sh)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int L = p.half_len, pre = p.pre_len, R = p.radius;

    SyncOut res{0, -1, 0.0f, 0.0f, 0.0f, -1};
    if (p.mode == 0) {
        if (fin.key != 0x7fffffff) {
            res.coarse_start = fin.key;
            res.coarse = fin.coarse >= 0.0f ? fin.coarse : 0.0f;
            res.start = fin.start;
            res.fine = fin.fine;
            res.found = (p.frame_len > 0 && res.start + p.frame_len > avail) ? 2 : 1;
        }
    } else if (fin.key >= 0 && fin.fine >= p.threshold) {
        const int cand = fin.key;
        const int lo = max(0, cand - R);
        const int hi = min(limit - 1, cand + R);
        for (int dd = lo + warp; dd <= hi; dd += kSyncThreads / 32) {
            const float m = fine_metric(x, sh.win, 0, 0, dd, preamble, pre, p.pre_energy, lane);
            if (lane == 0) sh.rmetric[dd - lo] = m;
        }
        __syncthreads();
        if (tid == 0) {
            float bm = 0.0f;
            int bd = cand;
            for (int dd = lo; dd <= hi; ++dd)
                if (sh.rmetric[dd - lo] > bm) { bm = sh.rmetric[dd - lo]; bd = dd; }
            sh.s_res->start = bd;
            sh.s_res->fine = bm;
        }
        __syncthreads();
        res.coarse_start = cand;
        res.coarse = fin.fine;
        res.fine = sh.s_res->fine;
        if (sh.s_res->fine >= p.threshold) {
            res.start = sh.s_res->start;
            res.found = 1;
        }
    }

    if (res.found == 1 || res.found == 2) {  // an incomplete frame also gets its CFO (for one-frame buffers)
        const int s0 = res.start;
        float ar = 0.f, ai = 0.f;
        for (int i = tid; i < L && tid < kSyncOwners; i += kSyncOwners) {
            const float2 c = cmulconj(x[s0 + i + L], x[s0 + i]);  // conj(x[s0+i]) * x[s0+i+L]
            ar += c.x;
            ai += c.y;
        }
        ar = warp_sum(ar);
        ai = warp_sum(ai);
        if (lane == 0 && tid < kSyncOwners) { sh.red[16 + warp] = ar; sh.red[24 + warp] = ai; }
        __syncthreads();
        if (tid == 0) {
            float sr = 0.f, si = 0.f;
            for (int w = 0; w < kSyncOwners / 32; ++w) { sr += sh.red[16 + w]; si += sh.red[24 + w]; }
            res.cfo_hz = atan2f(si, sr) * p.sample_rate / (2.0f * 3.14159265358979323846f * static_cast<float>(L));
        }
    }
    return res;
}

// Frame search, one CTA per (pass, frame): pass q scans candidates
// [4352 q, 4352 (q + 1)).  Within a pass the positions within +-radius of any
// threshold crossing are marked, and their fine metrics computed in increasing
// order, a warp per group of four, until the first one over the threshold and
// its 2 radius successors are known (groups that half the preamble rules out
// count as below).  The earliest crossing within +-radius of that position
// wins and takes the first maximum of its window (starting from 0, strict >)
// -- the outcome of the CPU receiver's sequential retry loop.  Mode 0 wants the earliest success, so a
// pass that starts after an earlier pass of its frame succeeded skips its
// scan (`ticket[frames + f]` holds passes - earliest successful pass, 0 for
// none).  Each pass stores its result in `pres`, and the CTA that takes the
// frame's last ticket (`ticket[f]`) takes the earliest result (mode 0) or the
// first global maximum (mode 1), refines it (mode 1), computes the CFO and
// writes the record.  `ticket` starts zeroed.
__global__ void __launch_bounds__(kSyncThreads)
sync_kernel(const float2* __restrict__ samples, long long stride, const long long* __restrict__ frame_off,
            const int* __restrict__ counts, int count, int frames, int passes, const float2* __restrict__ preamble,
            SyncParams p, PassResult* __restrict__ pres, int* __restrict__ ticket, SyncOut* __restrict__ out,
            const int* __restrict__ frames_ptr)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float red[4 * (kSyncOwners / 32)];
    __shared__ float rmetric[kMaxRefine];
    __shared__ int s_key[kSyncThreads / 32 + 2];
    __shared__ float s_tail;
    __shared__ PassResult s_res;
    __shared__ int s_flag;
    const SyncShared sh = sync_shared(smem_raw, p.pre_len, p.radius, red, rmetric, s_key, &s_tail, &s_res);

    // pass-major order: the first passes of all frames run first, so later
    // passes of a frame found early skip their scans
    const int pass = blockIdx.x / frames;
    const int f = blockIdx.x - pass * frames;
    // a grid sized for `frames` over a batch of *frames_ptr frames: the CTAs of absent frames
    // leave at once (uniform over the CTA, before any barrier)
    if (frames_ptr && f >= *frames_ptr) return;
    const int tid = threadIdx.x;
    const float2* x = samples + (frame_off ? frame_off[f] : static_cast<long long>(f) * stride);
    const int avail = counts ? counts[f] : count;
    int limit = avail - p.pre_len + 1;
    if (p.max_search > 0) limit = min(limit, p.max_search + 1);
    int* done = ticket + frames;

    if (tid == 0) {
        s_res.key = p.mode == 1 ? -1 : 0x7fffffff;
        s_res.start = -1;
        s_res.fine = -1.0f;
        s_res.coarse = 0.0f;
        s_flag = p.mode == 0 && *reinterpret_cast<volatile int*>(done + f) > passes - pass;
    }
    __syncthreads();

    const int base = pass * kSyncPass;
    if (!s_flag && base < limit) sync_scan_pass(x, avail, limit, pass, preamble, p, sh);
    __syncthreads();
    if (tid == 0 && p.mode == 0 && s_res.key != 0x7fffffff) atomicMax(done + f, passes - pass);

    // publish this pass; the frame's last pass to finish resolves it
    if (tid == 0) {
        pres[static_cast<long long>(f) * passes + pass] = s_res;
        __threadfence();
        s_flag = atomicAdd(ticket + f, 1) == passes - 1;
    }
    __syncthreads();
    if (!s_flag) return;
    __threadfence();
    if (tid == 0) {
        const PassResult* fr = pres + static_cast<long long>(f) * passes;
        PassResult best;
        best.key = __ldcg(&fr[0].key);
        best.start = __ldcg(&fr[0].start);
        best.fine = __ldcg(&fr[0].fine);
        best.coarse = __ldcg(&fr[0].coarse);
        for (int q = 1; q < passes; ++q) {
            PassResult o;
            o.key = __ldcg(&fr[q].key);
            o.start = __ldcg(&fr[q].start);
            o.fine = __ldcg(&fr[q].fine);
            o.coarse = __ldcg(&fr[q].coarse);
            if (p.mode == 1) {
                if (o.key >= 0 && (o.fine > best.fine || (o.fine == best.fine && (best.key < 0 || o.key < best.key))))
                    best = o;
            } else if (o.key < best.key) {
                best = o;
            }
        }
        s_res = best;
    }
    __syncthreads();
    const SyncOut res = sync_finish(x, avail, limit, s_res, preamble, p, sh);
    if (tid == 0) out[f] = res;
}

// Frame extraction over one window (one CTA): the receive loop's sequence of
// searches, each over [base, base + window) with the tracking or acquisition
// window, the earliest crossing found by scanning passes in order (mode 0),
// then the miss / late-peak / incomplete rules of extract_device; a found frame
// is copied into the next free pool slot and the search continues after it.
__global__ void __launch_bounds__(kSyncThreads)
ingest_extract_kernel(const float2* __restrict__ window, int n, const float2* __restrict__ preamble, SyncParams p,
                      IngestParams ip, const int* __restrict__ slots, float2* __restrict__ pool,
                      IngestRecord* __restrict__ rec, IngestState* __restrict__ state)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float red[4 * (kSyncOwners / 32)];
    __shared__ float rmetric[kMaxRefine];
    __shared__ int s_key[kSyncThreads / 32 + 2];
    __shared__ float s_tail;
    __shared__ PassResult s_res;
    __shared__ SyncOut s_out;
    __shared__ IngestState s_st;
    const SyncShared sh = sync_shared(smem_raw, p.pre_len, p.radius, red, rmetric, s_key, &s_tail, &s_res);
    const int tid = threadIdx.x;
    if (tid == 0) {
        s_st = *state;
        s_st.base = 0;
        s_st.frames = 0;
    }
    __syncthreads();
    while (s_st.frames < ip.max_frames) {
        const int base = s_st.base;
        const int available = n - base;
        if (available < p.pre_len) break;
        const int count = min(available, s_st.tracking ? ip.track_window : ip.acq_window);
        const float2* x = window + base;
        const int limit = count - p.pre_len + 1;
        if (tid == 0) {
            s_res.key = 0x7fffffff;
            s_res.start = -1;
            s_res.fine = -1.0f;
            s_res.coarse = 0.0f;
        }
        __syncthreads();
        for (int pass = 0; pass * kSyncPass < limit; ++pass) {  // the earliest success ends the search
            sync_scan_pass(x, count, limit, pass, preamble, p, sh);
            if (s_res.key != 0x7fffffff) break;
        }
        const SyncOut r = sync_finish(x, count, limit, s_res, preamble, p, sh);
        if (tid == 0) s_out = r;
        __syncthreads();
        const SyncOut res = s_out;
        const bool late = s_st.tracking && ip.late_threshold > 0.0f && res.start > ip.strict_window &&
                          res.fine < ip.late_threshold;
        int outcome = 0;  // 0 miss, 1 incomplete, 2 no pool slot, 3 found
        if (res.found == 0 || res.fine < p.threshold || late) outcome = 0;
        else if (res.start + ip.frame_len > available) outcome = 1;
        else if (s_st.frames >= ip.free_slots) outcome = 2;
        else outcome = 3;
        if (outcome == 3) {  // copy the frame into its pool slot
            float2* dst = pool + static_cast<size_t>(slots[s_st.frames]) * ip.frame_len;
            const float2* src = x + res.start;
            for (int i = tid; i < ip.frame_len; i += kSyncThreads) dst[i] = src[i];
        }
        __syncthreads();
        if (tid == 0) {
            if (outcome == 0) {
                if (s_st.tracking) {
                    ++s_st.tracking_miss;
                    s_st.tracking = 0;
                } else {
                    ++s_st.miss;
                }
            } else if (outcome == 1) {
                ++s_st.incomplete;
            } else if (outcome == 2) {
                s_st.base = base + res.start + ip.frame_len;
                ++s_st.miss;
                ++s_st.pool_exhausted;
            } else {
                IngestRecord& o = rec[s_st.frames];
                o.slot = slots[s_st.frames];
                o.start = base + res.start;
                o.peak = res.fine;
                o.cfo_hz = res.cfo_hz;
                ++s_st.found;
                s_st.skipped_samples += static_cast<unsigned long long>(res.start);
                if (static_cast<unsigned long long>(res.start) > s_st.max_start) s_st.max_start = res.start;
                s_st.tracking = 1;
                s_st.base = base + res.start + ip.frame_len;
                ++s_st.frames;
            }
        }
        __syncthreads();
        if (outcome != 3) break;
    }
    if (tid == 0) *state = s_st;
}

// The preambles accepted: those whose search would fit 200 KB with the widest refinement radius.
static size_t sync_smem_limit(int pre_len)
{
    return static_cast<size_t>((kSyncPass + pre_len + 1) & ~1) * sizeof(float2) + static_cast<size_t>(kSyncPass) * sizeof(float) +
           kSyncOwners * sizeof(float4) + static_cast<size_t>(kSyncPass + 2 * kMaxRadius) * sizeof(float);
}

static long long sync_passes(long long stride, const int* counts, int count, const SyncParams& p)
{
    // passes of the longest search: frames hold at most `stride` samples
    long long span = counts ? stride : std::min<long long>(count, stride);
    long long limit = span - p.pre_len + 1;
    if (p.max_search > 0) limit = std::min<long long>(limit, p.max_search + 1);
    return std::max<long long>(1, (limit + kSyncPass - 1) / kSyncPass);
}

SyncScratchLayout sync_scratch_layout(long long stride, const int* counts, int count, int frames, const SyncParams& p)
{
    const long long passes = sync_passes(stride, counts, count, p);
    SyncScratchLayout l;
    l.ticket_offset = (static_cast<size_t>(frames) * passes * sizeof(PassResult) + 15) & ~size_t(15);
    l.ticket_bytes = static_cast<size_t>(2) * frames * sizeof(int);
    l.bytes = l.ticket_offset + l.ticket_bytes;
    return l;
}

void launch_sync(const float2* samples, long long stride, const int* counts, int count, int frames,
                 const float2* preamble, const SyncParams& p, SyncOut* out, cudaStream_t st,
                 const long long* frame_off, const int* frames_ptr, void* caller_scratch, size_t caller_scratch_bytes)
{
    if (frames <= 0) return;
    if (sync_smem_limit(p.pre_len) > 200 * 1024) throw InvalidArgument("preamble too long for the sync kernel");
    if (p.radius > kMaxRadius || p.radius < 0) throw InvalidArgument("refinement radius must be 0..511");
    const size_t smem = sync_smem(p.pre_len, p.radius);
    const long long passes = sync_passes(stride, counts, count, p);
    if (passes * frames > 0x7fffffffLL) throw InvalidArgument("sync grid too large");
    const SyncScratchLayout l = sync_scratch_layout(stride, counts, count, frames, p);
    void* scratch = caller_scratch;
    const bool own = caller_scratch == nullptr;
    if (own) {
        int device = 0;
        check_cuda(cudaGetDevice(&device), "cudaGetDevice");
        check_cuda(cudaMallocFromPoolAsync(&scratch, l.bytes, scratch_pool(device), st), "cudaMallocFromPoolAsync(sync)");
    } else if (caller_scratch_bytes < l.bytes) {
        throw InvalidArgument("sync scratch smaller than the grid needs");
    }
    PassResult* pres = static_cast<PassResult*>(scratch);
    int* ticket = reinterpret_cast<int*>(static_cast<unsigned char*>(scratch) + l.ticket_offset);
    // caller scratch: the caller has zeroed the tickets in stream order before this launch
    cudaError_t err = own ? cudaMemsetAsync(ticket, 0, l.ticket_bytes, st) : cudaSuccess;
    if (err == cudaSuccess)
        err = grant_dynamic_smem(reinterpret_cast<const void*>(sync_kernel), smem);
    if (err == cudaSuccess) {
        sync_kernel<<<static_cast<unsigned>(passes * frames), kSyncThreads, smem, st>>>(
            samples, stride, frame_off, counts, count, frames, static_cast<int>(passes), preamble, p, pres, ticket, out,
            frames_ptr);
        err = cudaGetLastError();
    }
    const cudaError_t ferr = own ? cudaFreeAsync(scratch, st) : cudaSuccess;
    check_cuda(err, "sync_kernel launch");
    check_cuda(ferr, "cudaFreeAsync(sync)");
}

// ---------------------------------------------------------------------------
// demodulator
// ---------------------------------------------------------------------------

namespace {

constexpr int kDemodThreads = 256;

// Place of element i of an FFT buffer: bits 2-3 and 0-1 of the index XORed by bits 4-5.  The
// radix-4 stages write at strides 4, 16, ...; with this map the 16 lanes of a half-warp hit
// different banks in every stage (without it the stride-4 and stride-1 stages conflict 4-way).
// It is linear over XOR: swz(i ^ j) = swz(i) ^ swz(j).
__device__ __forceinline__ int swz(int i) { return i ^ (5 * ((i >> 4) & 3)); }

// Stockham autosort FFT of `nfft` points (a power of two) held in a (swizzled places, natural
// order in and out); returns the buffer that holds the result.  `tw`: the twiddles in the order
// the stages read them (fft_twiddles entries): for each radix-4 stage of span ns > 1 the factors
// w^k, w^2k, w^3k, k < ns, then the radix-2 stage's.
__device__ float2* fft_stockham(float2* a, float2* b, int nfft, const float2* __restrict__ tw)
{
    int ln = 0;  // log2 of the span
    const int lg = 31 - __clz(nfft), q = nfft >> 2, sq = swz(q), s2q = swz(2 * q);
    while (ln + 2 <= lg) {
        const int ns = 1 << ln, s1 = swz(ns), s2 = swz(2 * ns);
        for (int j = threadIdx.x; j < q; j += blockDim.x) {
            const int k = j & (ns - 1), ja = swz(j);
            float2 a0 = a[ja], a1 = a[ja ^ sq], a2 = a[ja ^ s2q], a3 = a[ja ^ sq ^ s2q];
            if (ln > 0) {
                a1 = cmul(a1, tw[k]);
                a2 = cmul(a2, tw[ns + k]);
                a3 = cmul(a3, tw[2 * ns + k]);
            }
            const float2 b0 = make_float2(a0.x + a2.x, a0.y + a2.y);
            const float2 b1 = make_float2(a0.x - a2.x, a0.y - a2.y);
            const float2 b2 = make_float2(a1.x + a3.x, a1.y + a3.y);
            const float2 b3 = make_float2(a1.y - a3.y, a3.x - a1.x);  // -i (a1 - a3)
            const int o = swz(((j >> ln) << (ln + 2)) + k);
            b[o] = make_float2(b0.x + b2.x, b0.y + b2.y);
            b[o ^ s1] = make_float2(b1.x + b3.x, b1.y + b3.y);
            b[o ^ s2] = make_float2(b0.x - b2.x, b0.y - b2.y);
            b[o ^ s1 ^ s2] = make_float2(b1.x - b3.x, b1.y - b3.y);
        }
        __syncthreads();
        if (ln > 0) tw += 3 * ns;
        float2* t = a;
        a = b;
        b = t;
        ln += 2;
    }
    if (ln < lg) {  // one radix-2 stage
        const int h = nfft >> 1, ns = h, sh = swz(h);
        for (int j = threadIdx.x; j < h; j += blockDim.x) {
            const int ja = swz(j);
            const float2 a0 = a[ja];
            const float2 a1 = cmul(a[ja ^ sh], tw[j]);  // span nfft / 2: one block of outputs
            b[ja] = make_float2(a0.x + a1.x, a0.y + a1.y);
            b[ja ^ swz(ns)] = make_float2(a0.x - a1.x, a0.y - a1.y);
        }
        __syncthreads();
        a = b;
    }
    return a;
}

// ---- bulk-async staging of a symbol's samples (cp.async.bulk + mbarrier) ----

__device__ unsigned int g_demod_wait_timeouts = 0;  // waits that hit their iteration limit (never expected)
constexpr int kMaxWaitSpins = 1 << 22;

__device__ __forceinline__ unsigned smem_addr(const void* p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity)
{
    unsigned ok = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the barrier's phase `parity` with an iteration limit; on the limit the
// timeout is counted, one more bounded wait lets an in-flight copy land, and false
// is returned (the caller skips the symbol's data).
__device__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity)
{
    for (int i = 0; i < kMaxWaitSpins; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    if (threadIdx.x == 0) atomicAdd(&g_demod_wait_timeouts, 1u);
    for (int i = 0; i < kMaxWaitSpins; ++i)
        if (mbar_try_wait(bar, parity)) break;
    return false;
}

// Where symbol `sym` of the frame at x lies, and how its samples are staged: the
// 16-byte-aligned middle [s, s + len) by one bulk copy into stage[0 .. len), the
// samples before s and from s + len on (at most one each: the rows are 8-byte
// complex samples) by plain loads when they are used.
struct SymbolStage {
    const float2* src;  // first sample of the symbol (CP stripped)
    int s, len;
};

__device__ __forceinline__ SymbolStage symbol_stage(const DemodView& v, const float2* x, int sym)
{
    SymbolStage g;
    g.src = x + v.pre_len + sym * (v.nfft + v.cp) + v.cp;
    g.s = (reinterpret_cast<uintptr_t>(g.src) & 15u) ? 1 : 0;
    g.len = v.nfft - 2 * g.s;  // nfft is even: len * 8 bytes is a multiple of 16
    return g;
}

// Thread 0: arms `bar` for the symbol's bytes and starts its bulk copy into `stage`.
__device__ __forceinline__ void stage_symbol(const SymbolStage& g, float2* stage, uint64_t* bar)
{
    const unsigned bytes = static_cast<unsigned>(g.len) * 8u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of `stage` come first
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(stage)),
                 "l"(g.src + g.s), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Carrier offset in turns per sample, cfo / fs as an unevaluated sum of two floats.
struct TurnRate {
    float hi, lo;
};
__device__ __forceinline__ TurnRate turn_rate(float cfo_hz, float sample_rate)
{
    const float hi = __fdiv_rn(cfo_hz, sample_rate);
    return {hi, __fdiv_rn(__fmaf_rn(-hi, sample_rate, cfo_hz), sample_rate)};
}

// exp(-j 2 pi cfo n / fs).  The angle is reduced to half a turn before it is rounded, so its error does not
// grow with n.
__device__ __forceinline__ float2 rotation(TurnRate c, int n)
{
    const float x = static_cast<float>(n), p = __fmul_rn(c.hi, x);
    const float rest = __fmaf_rn(c.lo, x, __fmaf_rn(c.hi, x, -p));  // what the product dropped
    float sn, cs;
    sincospif(-2.0f * __fadd_rn(__fsub_rn(p, rintf(p)), rest), &sn, &cs);
    return make_float2(cs, sn);
}

// CFO derotation and CP strip: work[swz(i)] = sample i of the symbol times
// exp(-j 2 pi cfo n / fs), n its index from the frame start; the samples come from
// the staged copy, the edge samples (and every sample if the copy did not land)
// from global memory.  A thread's samples lie kDemodThreads apart: every fourth gets its
// rotation from sincospi, the three after it by one turn each of it by step[k - 1] =
// rotation(k kDemodThreads).
__device__ __forceinline__ void derotate_symbol(const DemodView& v, const SymbolStage& g, const float2* stage,
                                                float2* work, TurnRate cfo, const float2 (&step)[3], int sym, bool staged)
{
    const int off = v.pre_len + sym * (v.nfft + v.cp) + v.cp;
    for (int i0 = threadIdx.x; i0 < v.nfft; i0 += 4 * kDemodThreads) {
        const float2 base = rotation(cfo, off + i0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k * kDemodThreads;
            if (i >= v.nfft) break;
            const float2 smp = (!staged || i < g.s || i >= g.s + g.len) ? g.src[i] : stage[i - g.s];
            work[swz(i)] = cmul(smp, k == 0 ? base : cmul(base, step[k > 0 ? k - 1 : 0]));
        }
    }
    __syncthreads();
}

__device__ __forceinline__ float sq_dist(float x, float c)
{
    const float d = __fsub_rn(x, c);
    return __fmul_rn(d, d);
}

}  // namespace

// kSharedTw: the FFT's twiddles copied to shared memory, else read from global memory (the largest
// grids, whose pilots leave no room for them).
template <int kBps, bool kSharedTw>
__global__ void __launch_bounds__(kDemodThreads)
demod_kernel(DemodView v, const float2* __restrict__ samples, long long stride, const SyncOut* __restrict__ sync,
             float* __restrict__ llr, long long llr_stride, int symbols_per_cta, const long long* __restrict__ frame_off,
             const long long* __restrict__ llr_off, const int* __restrict__ frames_ptr)
{
    // a grid sized for more frames than the batch holds: the CTAs of absent frames leave at once
    if (frames_ptr && static_cast<int>(blockIdx.x) >= *frames_ptr) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* work = reinterpret_cast<float2*>(smem_raw);  // derotated symbol, FFT buffer
    // stage(b) = work + (1 + b) * nfft: staged raw symbols (two buffers), FFT buffer after use
    auto stage = [&](int b) { return work + static_cast<size_t>(1 + b) * v.nfft; };
    float2* s_tw = work + 3 * v.nfft;                     // the FFT's twiddles in stage order
    float2* hp = s_tw + (kSharedTw ? fft_twiddles(v.nfft) : 0);  // [max_pilots_per_cta][active_sc]
    __shared__ __align__(8) uint64_t s_bar[2];

    const int f = blockIdx.x;
    const int ds0 = blockIdx.y * symbols_per_cta;
    const int ds1 = min(v.num_data, ds0 + symbols_per_cta);
    if (ds0 >= ds1) return;
    int start = 0;
    float cfo = 0.0f;
    if (sync) {
        const SyncOut so = sync[f];
        if (so.found != 1) {
            // no frame: zero LLRs (the caller sees found != 1 in the sync result)
            float* dst = llr + (llr_off ? llr_off[f] : static_cast<long long>(f) * llr_stride);
            const int hi = min(ds1 * v.active_sc * kBps, v.kept_bits);
            for (int i = ds0 * v.active_sc * kBps + threadIdx.x; i < hi; i += blockDim.x) dst[i] = 0.0f;
            return;
        }
        start = so.start;
        cfo = so.cfo_hz;
    }
    const float2* x = samples + (frame_off ? frame_off[f] : static_cast<long long>(f) * stride) + start;
    const TurnRate rate = turn_rate(cfo, v.sample_rate);

    // pilots referenced by this CTA's data symbols
    int pmin = 0x7fffffff, pmax = -1;
    for (int d = ds0; d < ds1; ++d) {
        pmin = min(pmin, min(v.interp_p0[d], v.interp_p1[d]));
        pmax = max(pmax, max(v.interp_p0[d], v.interp_p1[d]));
    }
    const int npil = v.use_pilot_est ? min(pmax - pmin + 1, v.max_pilots_per_cta) : 0;
    const int nsym = npil + (ds1 - ds0);
    // the CTA's symbols in processing order: its pilots, then its data symbols
    auto sym_at = [&](int i) { return i < npil ? v.pilot_symbols[pmin + i] : v.data_symbols[ds0 + i - npil]; };

    // Symbol i+1's samples are copied into stage[(i+1)&1] by the bulk-copy engine while
    // symbol i is transformed; each buffer's barrier completes once per copy.
    if (threadIdx.x == 0) {
        mbar_init(&s_bar[0], 1);
        mbar_init(&s_bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const float2* tw = v.twiddle;
    if constexpr (kSharedTw) {
        for (int i = threadIdx.x; i < fft_twiddles(v.nfft); i += blockDim.x) s_tw[i] = __ldg(v.twiddle + i);
        tw = s_tw;
    }
    constexpr int bps = kBps, abits = kBps >> 1, levels = 1 << abits;
    // the constellation's axis levels (at most 8: 64-QAM) in registers
    float lvl[levels];
#pragma unroll
    for (int g = 0; g < levels; ++g) lvl[g] = bps >= 2 ? __ldg(v.axis_levels + g) : 0.0f;
    const float2 step[3] = {rotation(rate, kDemodThreads), rotation(rate, 2 * kDemodThreads), rotation(rate, 3 * kDemodThreads)};
    __syncthreads();
    if (threadIdx.x == 0) stage_symbol(symbol_stage(v, x, sym_at(0)), stage(0), &s_bar[0]);
    unsigned phase = 0u;  // bit b: parity of buffer b's next completion

    float* out = llr + (llr_off ? llr_off[f] : static_cast<long long>(f) * llr_stride);
    // a symbol's LLRs in one store where they align (the caller's array may start at any float)
    const bool aligned = (bps == 2 || bps == 4) && (reinterpret_cast<uintptr_t>(out) & (sizeof(float) * bps - 1)) == 0;
    for (int i = 0; i < nsym; ++i) {
        const int b = i & 1;
        const int sym = sym_at(i);
        if (threadIdx.x == 0 && i + 1 < nsym)
            stage_symbol(symbol_stage(v, x, sym_at(i + 1)), stage(b ^ 1), &s_bar[b ^ 1]);
        const SymbolStage g = symbol_stage(v, x, sym);
        const bool staged = mbar_wait_bounded(b ? &s_bar[1] : &s_bar[0], (phase >> b) & 1u);
        phase ^= 1u << b;
        derotate_symbol(v, g, stage(b), work, rate, step, sym, staged);
        const float2* Y = fft_stockham(work, stage(b), v.nfft, tw);
        if (i < npil) {  // LS estimate at the pilot symbol
            const int p = pmin + i;
            for (int sc = threadIdx.x; sc < v.active_sc; sc += blockDim.x) {
                const float2 y = Y[swz(v.used_bins[sc])];
                const float2 pil = v.pilot_grid[static_cast<size_t>(p) * v.active_sc + sc];
                const float den = fmaxf(cnorm(pil), 1e-9f);
                const float2 t = cmulconj(y, pil);
                hp[i * v.active_sc + sc] = make_float2(__fdiv_rn(t.x, den), __fdiv_rn(t.y, den));
            }
            __syncthreads();
            continue;
        }
        const int d = ds0 + i - npil;
        const int q0 = v.interp_p0[d] - pmin, q1 = v.interp_p1[d] - pmin;
        const float al = v.interp_alpha[d];
        const float w0 = __fsub_rn(1.0f, al);
        const int sc_end = min(v.active_sc, v.kept_bits / bps - d * v.active_sc);  // REs of whole codewords
        for (int sc = threadIdx.x; sc < sc_end; sc += blockDim.x) {
            const float2 y = Y[swz(v.used_bins[sc])];
            float2 h = make_float2(1.0f, 0.0f);
            if (v.use_pilot_est) {
                const float2 h0 = hp[q0 * v.active_sc + sc], h1 = hp[q1 * v.active_sc + sc];
                h = make_float2(__fadd_rn(__fmul_rn(h0.x, w0), __fmul_rn(h1.x, al)),
                                __fadd_rn(__fmul_rn(h0.y, w0), __fmul_rn(h1.y, al)));
            }
            const float h2 = fmaxf(cnorm(h), 1e-9f);
            const float2 t = cmulconj(y, h);
            // eq = y conj(h) / (|h|^2 + N0) and LLR = (d1 - d0) / sigma^2 as products with the two
            // reciprocals (as the reference's GPU equaliser scales by 1 / (|h|^2 + N0))
            const float inv_den = __frcp_rn(__fadd_rn(h2, v.noise_var));
            const float ex = __fmul_rn(t.x, inv_den), ey = __fmul_rn(t.y, inv_den);
            const float inv_sig = __frcp_rn(fmaxf(__fdiv_rn(v.noise_var, h2), 1e-8f));
            float* o = out + (static_cast<long long>(d) * v.active_sc + sc) * bps;
            if constexpr (bps == 1) {
                const float dy = __fmul_rn(ey, ey);
                const float d0 = __fadd_rn(sq_dist(ex, 1.0f), dy), d1 = __fadd_rn(sq_dist(ex, -1.0f), dy);
                o[0] = __fmul_rn(__fsub_rn(d1, d0), inv_sig);
            } else {
                // per-axis squared distances and minima
                float mi_all = FLT_MAX, mq_all = FLT_MAX;
                float mi0[abits], mi1[abits], mq0[abits], mq1[abits];
#pragma unroll
                for (int bb = 0; bb < abits; ++bb) mi0[bb] = mi1[bb] = mq0[bb] = mq1[bb] = INFINITY;
#pragma unroll
                for (int gq = 0; gq < levels; ++gq) {
                    const float di = sq_dist(ex, lvl[gq]), dq = sq_dist(ey, lvl[gq]);
                    mi_all = fminf(mi_all, di);
                    mq_all = fminf(mq_all, dq);
#pragma unroll
                    for (int bb = 0; bb < abits; ++bb) {
                        if ((gq >> (abits - 1 - bb)) & 1) {
                            mi1[bb] = fminf(mi1[bb], di);
                            mq1[bb] = fminf(mq1[bb], dq);
                        } else {
                            mi0[bb] = fminf(mi0[bb], di);
                            mq0[bb] = fminf(mq0[bb], dq);
                        }
                    }
                }
                float vals[bps];
#pragma unroll
                for (int bb = 0; bb < abits; ++bb) {
                    vals[bb] = __fmul_rn(__fsub_rn(__fadd_rn(mi1[bb], mq_all), __fadd_rn(mi0[bb], mq_all)), inv_sig);
                    vals[abits + bb] =
                        __fmul_rn(__fsub_rn(__fadd_rn(mi_all, mq1[bb]), __fadd_rn(mi_all, mq0[bb])), inv_sig);
                }
                if (!aligned) {
#pragma unroll
                    for (int bb = 0; bb < bps; ++bb) o[bb] = vals[bb];
                } else if constexpr (bps == 4) {
                    *reinterpret_cast<float4*>(o) = make_float4(vals[0], vals[1], vals[2], vals[3]);
                } else if constexpr (bps == 2) {
                    *reinterpret_cast<float2*>(o) = make_float2(vals[0], vals[1]);
                }
            }
        }
        __syncthreads();
    }
}

unsigned demod_wait_timeouts()
{
    unsigned v = 0;
    check_cuda(cudaMemcpyFromSymbol(&v, g_demod_wait_timeouts, sizeof v), "read the demodulator's wait counter");
    return v;
}

void launch_demod(const DemodView& v, const float2* samples, long long stride, const SyncOut* sync, int frames,
                  float* llr, long long llr_stride, cudaStream_t st, int symbols_per_cta, const long long* frame_off,
                  const long long* llr_off, const int* frames_ptr)
{
    if (frames <= 0 || v.num_data <= 0) return;
    if (v.nfft < 4 || (v.nfft & (v.nfft - 1))) throw InvalidArgument("nfft must be a power of two >= 4");
    if (v.bits_per_symbol != 1 && v.bits_per_symbol != 2 && v.bits_per_symbol != 4 && v.bits_per_symbol != 6)
        throw InvalidArgument("bits_per_symbol must be 1, 2, 4 or 6");
    if (v.kept_bits <= 0 || v.kept_bits > v.num_data * v.active_sc * v.bits_per_symbol || v.kept_bits % v.bits_per_symbol)
        throw InvalidArgument("kept LLRs must be a positive multiple of bits_per_symbol within the frame");
    // the owner of the view sized max_pilots_per_cta for this grouping of data symbols
    int spc = symbols_per_cta;
    if (spc <= 0 || spc > v.num_data) throw InvalidArgument("symbols_per_cta must be in 1..num_data");
    if (v.max_pilots_per_cta < 0 || v.max_pilots_per_cta > kDemodMaxPilots)
        throw InvalidArgument("a demodulator CTA can hold at most 4 pilot symbols");
    // A few frames do not fill the GPU at that grouping: fewer symbols per CTA then, as long as
    // the CTAs do not outnumber the SMs (each CTA transforms its own pilots too, so more CTAs
    // only repeat that work).  The pilots of a part of a group are among the group's own when the
    // parts divide it.  One 96-symbol frame (72 data symbols): 3 per CTA 26 us,
    // 1 per CTA 16 us.
    while (spc > 1) {
        int part = spc - 1;
        while (spc % part) --part;
        if (static_cast<long long>(frames) * ((v.num_data + part - 1) / part) > device_sm_count()) break;
        spc = part;
    }
    // Accepted: grids that fit the 227 KB with 3/4 nfft further points (a plain twiddle table).  Of
    // these the largest (4,096 points with four pilots of more than 3,169 subcarriers) do not fit the
    // stage-ordered twiddles and read them from global memory.
    constexpr size_t most = 227 * 1024 / sizeof(float2);
    const size_t points = 3 * static_cast<size_t>(v.nfft) + static_cast<size_t>(v.max_pilots_per_cta) * v.active_sc;
    if (points + ((3 * static_cast<size_t>(v.nfft) / 4 + 1) & ~size_t(1)) > most)
        throw InvalidArgument("nfft and active_sc exceed the demodulator's shared memory");
    const bool shared_tw = points + fft_twiddles(v.nfft) <= most;
    const size_t smem = (points + (shared_tw ? fft_twiddles(v.nfft) : 0)) * sizeof(float2);
    const dim3 grid(frames, (v.num_data + spc - 1) / spc);
    const auto go = [&](auto kernel) {
        check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(kernel), smem), "cudaFuncSetAttribute(demod)");
        kernel<<<grid, kDemodThreads, smem, st>>>(v, samples, stride, sync, llr, llr_stride, spc, frame_off, llr_off,
                                                  frames_ptr);
        check_cuda(cudaGetLastError(), "demod_kernel launch");
    };
    switch (v.bits_per_symbol) {
        case 1: shared_tw ? go(demod_kernel<1, true>) : go(demod_kernel<1, false>); break;
        case 2: shared_tw ? go(demod_kernel<2, true>) : go(demod_kernel<2, false>); break;
        case 4: shared_tw ? go(demod_kernel<4, true>) : go(demod_kernel<4, false>); break;
        default: shared_tw ? go(demod_kernel<6, true>) : go(demod_kernel<6, false>); break;
    }
}

// ---------------------------------------------------------------------------
// transmitter
// ---------------------------------------------------------------------------

namespace {

constexpr int kTxThreads = 256;
constexpr int kEncWarps = 8;

// Gray square QAM, bits MSB-first per axis (gpu_ofdm_pipeline.cu:84-109).
template <int kBps>
__device__ __forceinline__ float2 qam_from_bits(const uint8_t* bits)
{
    if constexpr (kBps == 1) return make_float2(bits[0] ? -1.0f : 1.0f, 0.0f);
    if constexpr (kBps == 2) {
        constexpr float s = 0.7071067811865475f;
        return make_float2(bits[0] ? -s : s, bits[1] ? -s : s);
    }
    constexpr int ab = kBps / 2, levels = 1 << ab;
    int bi = 0, bq = 0, gi = 0, gq = 0;  // Gray -> binary: each bit is the XOR of the Gray bits down to it
#pragma unroll
    for (int i = 0; i < ab; ++i) {
        gi ^= bits[i] != 0;
        gq ^= bits[ab + i] != 0;
        bi = (bi << 1) | gi;
        bq = (bq << 1) | gq;
    }
    constexpr float scale = (kBps == 4) ? 0.3162277660168379f : 0.1543033499620919f;
    return make_float2(__fmul_rn(static_cast<float>((levels - 1) - 2 * bi), scale),
                       __fmul_rn(static_cast<float>((levels - 1) - 2 * bq), scale));
}

// Counter-based normal deviates for the frequency-domain noise: a 32-bit
// integer hash (xor-shift / multiply, "lowbias32") of seed ^ (index * golden
// ratio) gives a uniform in (0, 1], and Box-Muller turns two of them into a
// normal deviate (gpu_ofdm_pipeline.cu:259-280).
__device__ __forceinline__ uint32_t hash32(uint32_t x)
{
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

__device__ __forceinline__ float uniform_open0(uint32_t seed, uint32_t idx)
{
    const uint32_t h = hash32(seed ^ (idx * 0x9e3779b9u));
    return __fmul_rn(__fadd_rn(__uint2float_rn(h), 1.0f), 2.3283064365386963e-10f);
}

__device__ __forceinline__ float normal_dev(uint32_t seed, uint32_t idx)
{
    const float u1 = fmaxf(uniform_open0(seed, idx * 2u), 1.0e-7f);
    const float u2 = uniform_open0(seed, idx * 2u + 1u);
    return __fmul_rn(sqrtf(__fmul_rn(-2.0f, logf(u1))), cosf(__fmul_rn(__fmul_rn(2.0f, 3.14159265358979323846f), u2)));
}

// four bits -> four bytes (0/1)
__device__ __forceinline__ uint32_t spread4(uint32_t x)
{
    return (x & 1u) | ((x & 2u) << 7) | ((x & 4u) << 14) | ((x & 8u) << 21);
}

}  // namespace

// c = u G over GF(2): one warp per codeword, 4 words of the codeword per lane
// per pass.  With the byte tables each 8 information bits select one
// precomputed XOR of their 8 generator rows; otherwise each set bit selects
// its bit-packed row.
__global__ void __launch_bounds__(kEncWarps * 32)
tx_encode_generator_kernel(TxView v, const uint8_t* __restrict__ info, uint8_t* __restrict__ coded, int count)
{
    const int lane = threadIdx.x & 31;
    const int n = v.code_n, k = v.code_k, gw = v.gen_stride;
    for (int cw = blockIdx.x * kEncWarps + (threadIdx.x >> 5); cw < count; cw += gridDim.x * kEncWarps) {
        const uint8_t* u = info + static_cast<size_t>(cw) * k;
        uint8_t* c = coded + static_cast<size_t>(cw) * n;
        for (int w0 = 0; w0 < (n + 31) / 32; w0 += 128) {
            uint32_t acc[4] = {0u, 0u, 0u, 0u};
            for (int i0 = 0; i0 < k; i0 += 32) {
                unsigned bits = __ballot_sync(0xffffffffu, i0 + lane < k && (u[i0 + lane] & 1u));
                if (v.gen_tab) {  // one table entry per byte of information bits: independent loads
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int g = (i0 >> 3) + q;
                        if (g * 8 >= k) break;
                        const uint32_t* e = v.gen_tab + (static_cast<size_t>(g) * 256 + ((bits >> (8 * q)) & 255u)) * gw;
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const int w = w0 + r * 32 + lane;
                            if (w < gw) acc[r] ^= __ldg(e + w);
                        }
                    }
                    continue;
                }
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    const uint32_t* row = v.gen_words + static_cast<size_t>(i0 + b) * gw;
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const int w = w0 + r * 32 + lane;
                        if (w < gw) acc[r] ^= __ldg(row + w);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int w = w0 + r * 32 + lane;
                if (w * 32 >= n) continue;
                if (w * 32 + 32 <= n && (n & 3) == 0) {  // 32 bytes as 8 words
                    uint32_t* dst = reinterpret_cast<uint32_t*>(c + w * 32);
#pragma unroll
                    for (int q = 0; q < 8; ++q) dst[q] = spread4((acc[r] >> (4 * q)) & 15u);
                } else {
                    for (int b = 0; b < 32 && w * 32 + b < n; ++b) c[w * 32 + b] = static_cast<uint8_t>((acc[r] >> b) & 1u);
                }
            }
        }
    }
}

// Systematic + accumulator encoder (gpu_ofdm_pipeline.cu:152-214): c[i] = u[i]
// for i < k, then parity r = sum of u over row r's information columns, XOR the
// previous parity: a prefix XOR over the rows, 32 rows per ballot.
__global__ void __launch_bounds__(kEncWarps * 32)
tx_encode_accumulator_kernel(TxView v, const uint8_t* __restrict__ info, uint8_t* __restrict__ coded, int count)
{
    const int lane = threadIdx.x & 31;
    const int n = v.code_n, k = v.code_k, m = n - k;
    for (int cw = blockIdx.x * kEncWarps + (threadIdx.x >> 5); cw < count; cw += gridDim.x * kEncWarps) {
        const uint8_t* u = info + static_cast<size_t>(cw) * k;
        uint8_t* c = coded + static_cast<size_t>(cw) * n;
        for (int i = lane; i < k; i += 32) c[i] = u[i] & 1u;
        unsigned carry = 0u;
        for (int r0 = 0; r0 < m; r0 += 32) {
            const int r = r0 + lane;
            unsigned s = 0u;
            if (r < m)
                for (int q = v.acc_offsets[r]; q < v.acc_offsets[r + 1]; ++q) s ^= u[v.acc_cols[q]] & 1u;
            unsigned y = __ballot_sync(0xffffffffu, s != 0u);
            y ^= y << 1;
            y ^= y << 2;
            y ^= y << 4;
            y ^= y << 8;
            y ^= y << 16;
            if (r < m) c[k + r] = static_cast<uint8_t>(((y >> lane) & 1u) ^ carry);
            carry ^= (y >> 31) & 1u;
        }
    }
}

// c = [u | u P] for systematic generators: the byte tables' parity words only.  One warp per
// codeword; a lane packs 16 information bits at a time and copies them, then groups of the
// smallest power of two of lanes covering the parity words take different information bytes, so
// every lane reads table words in every step.  k and n are multiples of 32, at most 32 parity words.
__global__ void __launch_bounds__(kEncWarps * 32)
tx_encode_systematic_kernel(TxView v, const uint8_t* __restrict__ info, uint8_t* __restrict__ coded, int count)
{
    const int lane = threadIdx.x & 31;
    const int n = v.code_n, k = v.code_k, gw = v.gen_stride, kw = k >> 5, pw = gw - kw;
    int width = 1;
    while (width < pw) width <<= 1;
    const int groups = 32 / width, h = lane / width, wl = lane & (width - 1);
    const uint32_t* tab = v.gen_tab + kw + wl;
    for (int cw = blockIdx.x * kEncWarps + (threadIdx.x >> 5); cw < count; cw += gridDim.x * kEncWarps) {
        const uint8_t* u = info + static_cast<size_t>(cw) * k;
        uint8_t* c = coded + static_cast<size_t>(cw) * n;
        uint32_t acc = 0u;
        for (int k0 = 0; k0 < k; k0 += 512) {
            uint4 b = make_uint4(0u, 0u, 0u, 0u);
            if (k0 + lane * 16 < k) {
                b = __ldg(reinterpret_cast<const uint4*>(u + k0) + lane);
                b.x &= 0x01010101u;
                b.y &= 0x01010101u;
                b.z &= 0x01010101u;
                b.w &= 0x01010101u;
                reinterpret_cast<uint4*>(c + k0)[lane] = b;
            }
            auto pack = [](uint32_t x) { return (x * 0x01020408u) >> 24; };  // four 0/1 bytes -> four bits
            const uint32_t bits = pack(b.x) | (pack(b.y) << 4) | (pack(b.z) << 8) | (pack(b.w) << 12);
            const int bytes = min(512, k - k0) >> 3;
#pragma unroll 8
            for (int g0 = 0; g0 < bytes; g0 += groups) {
                const int g = g0 + h;
                const uint32_t e = __shfl_sync(0xffffffffu, bits, (g >> 1) & 31) >> ((g & 1) * 8) & 255u;
                if (g < bytes && wl < pw) acc ^= __ldg(tab + (static_cast<size_t>((k0 >> 3) + g) * 256 + e) * gw);
            }
        }
        for (int o = width; o < 32; o <<= 1) acc ^= __shfl_xor_sync(0xffffffffu, acc, o);
        if (h == 0 && wl < pw) {  // 32 bytes as two 16-byte words
            uint4* dst = reinterpret_cast<uint4*>(c + k + wl * 32);
            dst[0] = make_uint4(spread4(acc & 15u), spread4((acc >> 4) & 15u), spread4((acc >> 8) & 15u), spread4((acc >> 12) & 15u));
            dst[1] = make_uint4(spread4((acc >> 16) & 15u), spread4((acc >> 20) & 15u), spread4((acc >> 24) & 15u), spread4(acc >> 28));
        }
    }
}

// One CTA per (OFDM symbol, frame); blockIdx.x == num_symbols writes the preamble.
// The symbol's grid row is built in shared memory (gpu_ofdm_pipeline.cu:216-257,
// 282-314), inverse-transformed as conj(FFT(conj(X))) (unnormalised, as cuFFT's
// inverse) and written with its cyclic prefix, scaled by amplitude / nfft
// (gpu_ofdm_pipeline.cu:316-342), two samples per store where they align.
template <int kBps>
__global__ void __launch_bounds__(kTxThreads)
tx_symbol_kernel(TxView v, const uint8_t* __restrict__ coded, float2* __restrict__ out, float noise_var,
                 unsigned long long noise_seed)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* buf0 = reinterpret_cast<float2*>(smem_raw);
    float2* buf1 = buf0 + v.nfft;
    const int sym = blockIdx.x, f = blockIdx.y;
    float2* frame = out + static_cast<size_t>(f) * v.frame_samples;
    if (sym == v.num_symbols) {
        for (int i = threadIdx.x; i < v.pre_len; i += blockDim.x) {
            const float2 p = v.preamble[i];
            frame[i] = make_float2(__fmul_rn(p.x, v.amplitude), __fmul_rn(p.y, v.amplitude));
        }
        return;
    }
    for (int i = threadIdx.x; i < (v.nfft >> 1); i += blockDim.x)
        reinterpret_cast<float4*>(buf0)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int pidx = v.pilot_of_symbol[sym], didx = v.data_of_symbol[sym];
    const int coded_bits = v.blocks * v.code_n;
    const uint8_t* bits = coded + static_cast<size_t>(f) * coded_bits;
    const unsigned long long fs = noise_seed + static_cast<unsigned long long>(f);
    const uint32_t seed = static_cast<uint32_t>(fs ^ (fs >> 32));
    const float sigma = sqrtf(__fmul_rn(fmaxf(noise_var, 0.0f), 0.5f));
    uint8_t* sbits = reinterpret_cast<uint8_t*>(buf1);  // the symbol's coded bits (buf1 is free until the FFT)
    if (didx >= 0 && pidx < 0) {
        const int b0 = didx * v.active_sc * kBps, count = v.active_sc * kBps;
        const uint8_t* src = bits + b0;
        const int have = min(count, max(coded_bits - b0, 0));  // bits past the coded bits are filler zeros
        if ((reinterpret_cast<uintptr_t>(src) & 3u) == 0) {
            for (int i = threadIdx.x; i < (count + 3) >> 2; i += blockDim.x) {
                uint32_t w = 0u;
                if (4 * i + 4 <= have) w = reinterpret_cast<const uint32_t*>(src)[i];
                else
                    for (int x = 0; x < 4; ++x)
                        if (4 * i + x < have) w |= static_cast<uint32_t>(src[4 * i + x]) << (8 * x);
                reinterpret_cast<uint32_t*>(sbits)[i] = w;
            }
        } else {
            for (int i = threadIdx.x; i < count; i += blockDim.x) sbits[i] = i < have ? src[i] : 0;
        }
    }
    __syncthreads();
    for (int sc = threadIdx.x; sc < v.active_sc; sc += blockDim.x) {
        const int re = sym * v.active_sc + sc;
        float2 value = make_float2(0.0f, 0.0f);
        if (pidx >= 0) {
            value = v.pilot_grid[static_cast<size_t>(pidx) * v.active_sc + sc];
        } else if (didx >= 0) {
            value = qam_from_bits<kBps>(sbits + sc * kBps);
        }
        if (v.precomp_h) {
            const float2 h = v.precomp_h[re];
            const float s = __fdiv_rn(1.0f, fmaxf(cnorm(h), 1.0e-10f));
            value = cmul(value, make_float2(__fmul_rn(h.x, s), __fmul_rn(-h.y, s)));
        }
        if (v.actual_h) value = cmul(value, v.actual_h[re]);
        if (noise_var > 0.0f && didx >= 0)
            value = make_float2(__fadd_rn(value.x, __fmul_rn(sigma, normal_dev(seed, static_cast<uint32_t>(re)))),
                                __fadd_rn(value.y, __fmul_rn(sigma, normal_dev(seed ^ 0xa5a5a5a5u, static_cast<uint32_t>(re)))));
        buf0[swz(v.used_bins[sc])] = make_float2(value.x, -value.y);  // conjugated for the inverse transform
    }
    __syncthreads();  // the grid row is complete and the staged bits are read
    const float2* Y = fft_stockham(buf0, buf1, v.nfft, v.twiddle);
    const float scale = v.amplitude / static_cast<float>(v.nfft);
    const int sym_len = v.nfft + v.cp;
    float2* dst = frame + v.pre_len + static_cast<size_t>(sym) * sym_len;
    auto sample = [&](int pos) -> float2 {
        const float2 y = Y[swz((pos - v.cp) & (v.nfft - 1))];  // cp <= nfft: the prefix wraps round
        return make_float2(__fmul_rn(y.x, scale), __fmul_rn(-y.y, scale));
    };
    if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0 && (sym_len & 1) == 0) {
        for (int p = threadIdx.x; p < (sym_len >> 1); p += blockDim.x) {
            const float2 s0 = sample(2 * p), s1 = sample(2 * p + 1);
            reinterpret_cast<float4*>(dst)[p] = make_float4(s0.x, s0.y, s1.x, s1.y);
        }
    } else {
        for (int pos = threadIdx.x; pos < sym_len; pos += blockDim.x) dst[pos] = sample(pos);
    }
}

void launch_tx(const TxView& v, const uint8_t* info_bits, int frames, float2* frames_out, float noise_var,
               unsigned long long noise_seed, cudaStream_t st)
{
    if (frames <= 0) return;
    const size_t smem = 2 * static_cast<size_t>(v.nfft) * sizeof(float2);
    if (smem > 200 * 1024) throw InvalidArgument("nfft too large for the TX kernel");
    const int codewords = frames * v.blocks;
    int device = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    void* coded = nullptr;
    check_cuda(cudaMallocFromPoolAsync(&coded, static_cast<size_t>(codewords) * v.code_n, scratch_pool(device), st),
               "cudaMallocFromPoolAsync(tx)");
    uint8_t* cb = static_cast<uint8_t*>(coded);
    const int ctas = std::max(1, std::min((codewords + kEncWarps - 1) / kEncWarps, 8 * device_sm_count()));
    // systematic generators of 32-bit multiples read half the table (the parity words) and pack their
    // information bits 16 to a load; the information rows have to be 16-byte aligned
    const int parity_words = v.gen_stride - (v.code_k >> 5);
    const bool systematic = v.systematic && v.gen_tab && v.code_k % 32 == 0 && v.code_n % 32 == 0 && parity_words <= 32 &&
                            (reinterpret_cast<uintptr_t>(info_bits) & 15u) == 0;
    if (v.acc_offsets)
        tx_encode_accumulator_kernel<<<ctas, kEncWarps * 32, 0, st>>>(v, info_bits, cb, codewords);
    else if (systematic)
        tx_encode_systematic_kernel<<<ctas, kEncWarps * 32, 0, st>>>(v, info_bits, cb, codewords);
    else
        tx_encode_generator_kernel<<<ctas, kEncWarps * 32, 0, st>>>(v, info_bits, cb, codewords);
    cudaError_t err = cudaGetLastError();
    const auto go = [&](auto kernel) {
        if (err == cudaSuccess) err = grant_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
        if (err != cudaSuccess) return;
        kernel<<<dim3(v.num_symbols + 1, frames), kTxThreads, smem, st>>>(v, cb, frames_out, noise_var, noise_seed);
        err = cudaGetLastError();
    };
    switch (v.bits_per_symbol) {
        case 1: go(tx_symbol_kernel<1>); break;
        case 2: go(tx_symbol_kernel<2>); break;
        case 4: go(tx_symbol_kernel<4>); break;
        default: go(tx_symbol_kernel<6>); break;
    }
    const cudaError_t ferr = cudaFreeAsync(coded, st);
    check_cuda(err, "tx launch");
    check_cuda(ferr, "cudaFreeAsync(tx)");
}

void launch_ingest_extract(const float2* window, int n, const float2* preamble, const SyncParams& sp,
                           const IngestParams& ip, const int* slots, float2* pool, IngestRecord* rec,
                           IngestState* state, cudaStream_t st)
{
    if (sync_smem_limit(sp.pre_len) > 200 * 1024) throw InvalidArgument("preamble too long for the sync kernel");
    if (sp.radius > kMaxRadius || sp.radius < 0) throw InvalidArgument("refinement radius must be 0..511");
    const size_t smem = sync_smem(sp.pre_len, sp.radius);
    check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(ingest_extract_kernel), smem),
               "cudaFuncSetAttribute(ingest)");
    ingest_extract_kernel<<<1, kSyncThreads, smem, st>>>(window, n, preamble, sp, ip, slots, pool, rec, state);
    check_cuda(cudaGetLastError(), "ingest_extract_kernel launch");
}

}  // namespace sicc
