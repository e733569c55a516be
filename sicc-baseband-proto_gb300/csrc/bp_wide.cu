// Belief propagation for long codes (DVB-S2 N16200 / N64800 class) whose
// decoder state does not fit one CTA's shared memory.
//
// One CTA decodes one codeword at a time and takes the next from a global
// counter when it stops.  The posteriors live in shared memory when they fit
// (n <= ~50k); for longer codes the layered kernel keeps the first 56,320 in
// shared memory and the rest in the CTA's slice of a global scratch block (the
// flooding kernel keeps them all there); the row messages live in that slice
// too.  A slice is touched by one CTA only, so it stays in L2 when the grid's
// slices fit there (the launcher sizes the grid for that).
//
//   layered (schedules 2, 3): the rows of a layer touch disjoint variables,
//     so the CTA's threads update them in parallel, one barrier per layer;
//     the row arithmetic gives the shared-memory layered kernel's values
//     (bp_kernels.cu).
//   flooding (schedules 0, 1): check phase over all rows, variable phase
//     over all columns (the reference CPU decoder, uhd_ldpc_ofdm_link.cpp:
//     3013-3094, with the MB damping of cpu_bp_osd_decode.m:180-183).
//
// Results, stopping rule (zero syndrome or the iteration cap), best-syndrome
// tracking and the OSD hand-off are those of the shared-memory kernels, so
// both give the same bits for a code that fits either.
#include "bp_device.cuh"
#include "bp_kernels.h"
#include "bp_reg.cuh"

#include <algorithm>
#include <cfloat>

namespace sicc {

namespace {

// CTA-wide sum; every thread gets the total.  `red` holds one int per warp.
template <int kThreads>
__device__ __forceinline__ int cta_sum(int v, int* red)
{
    v = static_cast<int>(__reduce_add_sync(0xffffffffu, static_cast<unsigned>(v)));
    __syncthreads();  // the previous reduction's reads are done
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) t += red[i];
    return t;
}

template <int kThreads>
__device__ __forceinline__ unsigned cta_min(unsigned v, int* red)
{
    v = __reduce_min_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = static_cast<int>(v);
    __syncthreads();
    unsigned t = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) t = min(t, static_cast<unsigned>(red[i]));
    return t;
}

// Outputs of a finished codeword (the shared-memory kernels' finalize step).
template <int kThreads, class App>
__device__ void wide_finish(const BpParams& p, const BpIO& io, int c, int n, int w, int iter, const App& app,
                            const float* best, bool track_best, int* red, int* s_slot)
{
    const int tid = threadIdx.x;
    bool accept = (w == 0);
    if (accept && p.min_abs_accept > 0.0f) {
        unsigned mn = 0x7f800000u;
        for (int i = tid; i < n; i += kThreads) mn = min(mn, __float_as_uint(fabsf(app.ld(i))));
        accept = __uint_as_float(cta_min<kThreads>(mn, red)) >= p.min_abs_accept;
    }
    const bool route = !accept && p.route_failures_to_osd && io.osd_llr != nullptr;
    if (tid == 0) {
        if (io.success) io.success[c] = accept ? 1 : 0;
        if (io.iterations) io.iterations[c] = static_cast<uint8_t>(iter);
        if (io.used_osd) io.used_osd[c] = 0;
        if (route) *s_slot = atomicAdd(io.osd_count, 1);
    }
    if (io.out_bits) {
        uint8_t* dst = io.out_bits + static_cast<size_t>(c) * io.out_stride;
        for (int i = tid; i < io.out_len; i += kThreads) dst[i] = app.ld(i) < 0.0f ? 1 : 0;
    }
    if (io.app_out) {
        float* dst = io.app_out + static_cast<size_t>(c) * n;
        for (int i = tid; i < n; i += kThreads) dst[i] = app.ld(i);
    }
    __syncthreads();  // s_slot
    if (route) {
        const int s = *s_slot;
        float* dst = io.osd_llr + static_cast<size_t>(s) * n;
        for (int i = tid; i < n; i += kThreads) dst[i] = track_best ? best[i] : app.ld(i);
        if (tid == 0) io.osd_index[s] = c;
    }
}

// Next codeword of this CTA (all threads get it).
__device__ __forceinline__ int wide_next(const BpIO& io, int* s_next)
{
    __syncthreads();  // every thread is done with the current codeword's state
    if (threadIdx.x == 0) *s_next = static_cast<int>(gridDim.x) + atomicAdd(io.work_counter, 1);
    __syncthreads();
    return *s_next;
}

// Posteriors of the layered wide kernel by byte offset (4 x variable): those below `split` in
// shared memory, the rest in the CTA's global slice (L2), so a code a little too long for
// shared memory keeps most of its posterior gathers on chip.
struct SplitApp {
    unsigned char* s;
    unsigned char* g;  // same offsets; the bytes below `split` are unused
    unsigned split;
    __device__ __forceinline__ float at(unsigned off) const
    {
        return off < split ? *reinterpret_cast<const float*>(s + off) : *reinterpret_cast<const float*>(g + off);
    }
    __device__ __forceinline__ void put(unsigned off, float x) const
    {
        if (off < split) *reinterpret_cast<float*>(s + off) = x;
        else *reinterpret_cast<float*>(g + off) = x;
    }
    __device__ __forceinline__ float ld(int v) const { return at(4u * static_cast<unsigned>(v)); }
};

// What a row update reads besides posteriors: the row's posterior offsets (16-byte loads) and
// its compressed messages.
template <int D>
struct WideRow {
    static constexpr int kQuads = (D + 3) / 4;
    uint4 o[kQuads];
    uint4 state;  // min1, min2 (scaled), signs and argmin; the messages themselves where D <= 4

    __device__ __forceinline__ static unsigned word(const uint4& x, int j)
    {
        return (j & 3) == 0 ? x.x : (j & 3) == 1 ? x.y : (j & 3) == 2 ? x.z : x.w;
    }

    __device__ __forceinline__ unsigned off(int j) const
    {
        return word(o[j >> 2], j);
    }
    __device__ __forceinline__ void load_offsets(const uint4* __restrict__ table, int row)
    {
#pragma unroll
        for (int i = 0; i < kQuads; ++i) o[i] = __ldg(table + static_cast<size_t>(row) * kQuads + i);
    }
    __device__ __forceinline__ void load(const uint4* __restrict__ table, int row, bool fresh, const uint4* states)
    {
        load_offsets(table, row);
        state = make_uint4(0u, 0u, 0u, 0u);  // a codeword's first iteration: no messages yet
        if (!fresh) state = states[row];
    }
};

// Threads: as many as the rows' registers allow without spills in the row loop (they hide the L2
// latency of tables and messages).  608 codewords of (64800,32400), D = 7: 768 threads 5.28 ms, 896
// 5.09, 1,024 5.15; 600 of (16200,13320), D = 18: 512 threads 0.38 ms, 576 (spilling) 0.41.
template <int D>
constexpr int wide_threads() { return D <= 4 ? 1024 : D <= 7 ? 896 : D <= 10 ? 768 : 512; }

}  // namespace

// The next row's offsets and messages are loaded while the current one is updated, across the
// layer barriers too: they do not depend on posteriors.  Slots below D - kFar hold shared-memory
// posteriors in every row (columns ascend within a row, so for the accumulator codes only the
// two parity slots can lie beyond the split): only the last kFar (0, 2 or D) test.  A run-time
// bound put a branch before every access and cost 6.42 against 5.28 ms on the code below.
// Up to 4 slots a row keeps its messages as they are, in the 16 bytes that the compressed form
// takes ((16200,3240): 1.99 against 1.76 ms); for 7 slots that form outgrows L2 (7.4 ms).  Without
// best-syndrome tracking only "zero syndrome or not" matters, so the check stops at the first
// layer with an unsatisfied row.
//
// Measured on GB300, 608 codewords of (64800,32400) at 2 dB: 12.1 ms before (512 threads, a
// branch per posterior access, variable indices slot by slot, (min1, min2, argmin) row
// arithmetic, full syndrome: 78 instructions per edge and iteration), 5.10 ms now (31); the last
// SM runs 76 iterations, the average one 55.
template <int D, int kFar>
__global__ void __launch_bounds__(wide_threads<D>(), 1)
bp_layered_wide_kernel(LayeredView cv, BpParams p, BpIO io, float* scratch, long long slice, int split, int track_best)
{
    constexpr int kThreads = wide_threads<D>();
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_red[kThreads / 32];
    __shared__ int s_next, s_slot;
    const int tid = threadIdx.x;
    const int n = cv.n, n_pad = (n + 3) & ~3;
    const int mp = cv.m;  // messages of the rows in layer order, packed
    float* g = scratch + static_cast<size_t>(blockIdx.x) * static_cast<size_t>(slice);
    // posteriors [0, split) in shared memory.  The dummy posterior (index n_pad, +inf) takes the
    // empty edge slots of short rows: with split > n_pad it and every posterior are in shared
    // memory, else the slice starts with n_pad posteriors and the dummy (4 floats).
    const bool all_smem = split > n_pad;
    const SplitApp app{s_raw, reinterpret_cast<unsigned char*>(g), 4u * static_cast<unsigned>(split)};
    float* best = all_smem ? g : g + n_pad + 4;
    uint4* states = reinterpret_cast<uint4*>(best + (track_best ? n_pad : 0));
    const uint4* table = reinterpret_cast<const uint4*>(cv.wide_rows);
    constexpr int js = D - kFar;  // slots below it are in shared memory in every row

    using Row = WideRow<D>;
    auto value = [&](const Row& row, int j) -> float {
        return j < js ? reg::lds(s_raw, row.off(j)) : app.at(row.off(j));
    };
    auto put = [&](const Row& row, int j, float x) {
        if (j < js) reg::sts(s_raw, row.off(j), x);
        else app.put(row.off(j), x);
    };
    auto update = [&](const Row& in, int row) {
        float q[D], m[D];
        if constexpr (D <= 4) {
#pragma unroll
            for (int j = 0; j < D; ++j) q[j] = __fsub_rn(value(in, j), __uint_as_float(Row::word(in.state, j)));
            reg::row_messages<D>(q, p.alpha, p.beta, m);
#pragma unroll
            for (int j = 0; j < D; ++j) put(in, j, __fadd_rn(q[j], m[j]));
            auto word = [&](int j) { return j < D ? __float_as_uint(m[j < D ? j : 0]) : 0u; };
            states[row] = make_uint4(word(0), word(1), word(2), word(3));
            return;
        }
        const float o1 = __uint_as_float(in.state.x), o2 = __uint_as_float(in.state.y);
#pragma unroll
        for (int j = 0; j < D; ++j) q[j] = __fsub_rn(value(in, j), rebuild(o1, o2, in.state.z, j));
        reg::exclusive_min<D>(q, m);
        // the compressed row: all magnitudes but at most one equal the smallest input's
        const float least = fminf(fabsf(m[0]), fabsf(m[1]));
        float most = least;
        unsigned signs = 0u;
        int idx = 0;
#pragma unroll
        for (int j = 0; j < D; j += 2) most = reg::max3(most, m[j], m[j + 1 < D ? j + 1 : 0]);
#pragma unroll
        for (int j = D - 1; j >= 0; --j) {
            signs = __funnelshift_l(__float_as_uint(m[j]), signs, 1);
            idx = fabsf(m[j]) == most ? j : idx;
        }
        const float n1 = nms_mag(p.alpha, p.beta, least), n2 = nms_mag(p.alpha, p.beta, most);
#pragma unroll
        for (int j = 0; j < D; ++j) {
            // the message, signed: the scaled magnitude with the sign of m
            const float mag = fabsf(m[j]) == most ? n2 : n1;
            put(in, j, __fadd_rn(q[j], __uint_as_float(__float_as_uint(mag) ^ (__float_as_uint(m[j]) & 0x80000000u))));
        }
        states[row] = make_uint4(__float_as_uint(n1), __float_as_uint(n2), signs | (static_cast<unsigned>(idx) << 27), 0u);
    };
    auto parity_of = [&](int row) -> unsigned {
        Row r;
        r.load_offsets(table, row);
        unsigned par = 0u;
#pragma unroll
        for (int j = 0; j < D; ++j) par ^= __float_as_uint(value(r, j));
        return par >> 31;
    };
    // Syndrome weight; without tracking, any nonzero value when it is not zero.
    auto syndrome = [&]() -> int {
        int cnt = 0;
        if (track_best) {
            for (int r = tid; r < mp; r += kThreads) cnt += static_cast<int>(parity_of(r));
            return cta_sum<kThreads>(cnt, s_red);
        }
        for (int L = 0; L < cv.num_layers; ++L) {
            const int end = __ldg(cv.layer_start + L + 1);
            for (int r = __ldg(cv.layer_start + L) + tid; r < end && cnt == 0; r += kThreads)
                cnt += static_cast<int>(parity_of(r));
            if (__syncthreads_or(cnt)) return 1;
        }
        return 0;
    };

    if (tid == 0) app.put(4u * static_cast<unsigned>(n_pad), __int_as_float(0x7f800000));  // +inf, before the first __syncthreads
    for (int c = blockIdx.x; c < io.count; c = wide_next(io, &s_next)) {
        const float* src = io.llr + static_cast<size_t>(c) * n;
        for (int i = tid; i < n; i += kThreads) {
            const float v = __ldcs(src + i);
            app.put(4u * static_cast<unsigned>(i), reg::canonical(v));
            if (track_best) best[i] = v;
        }
        __syncthreads();
        int best_w = track_best ? syndrome() : 1;
        int iter = 0, w = 0;
        Row next;
        if (tid < __ldg(cv.layer_start + 1)) next.load(table, tid, true, states);
        for (;;) {
            int first = 0, rows = __ldg(cv.layer_start + 1);
            for (int L = 0; L < cv.num_layers; ++L) {
                const bool last = L + 1 == cv.num_layers;
                const int after = last ? 0 : first + rows;  // first row of the layer that comes next
                const int after_rows = __ldg(cv.layer_start + (last ? 1 : L + 2)) - after;
                const bool fresh = iter == 0, after_fresh = fresh && !last;
                for (int rs = tid;; rs += kThreads) {
                    const Row row = next;
                    if (rs + kThreads < rows) next.load(table, first + rs + kThreads, fresh, states);
                    else if (tid < after_rows) next.load(table, after + tid, after_fresh, states);
                    if (rs < rows) update(row, first + rs);
                    if (rs + kThreads >= rows) break;
                }
                __syncthreads();
                // a single layer: its rows' messages have only just been written
                if (cv.num_layers == 1 && tid < rows) next.load(table, tid, false, states);
                first = after;
                rows = after_rows;
            }
            w = syndrome();
            ++iter;
            if (track_best && (w < best_w || (w == 0 && best_w == 0))) {
                for (int i = tid; i < n; i += kThreads) best[i] = app.ld(i);
                __syncthreads();  // copied before the next layer rewrites the posteriors
            }
            if (w < best_w) best_w = w;
            if (w == 0 || iter >= p.max_iter) break;
        }
        wide_finish<kThreads>(p, io, c, n, w, iter, app, best, track_best != 0, s_red, &s_slot);
    }
}

// Plain posterior array for the flooding kernel's finish step.
struct PlainApp {
    const float* a;
    __device__ __forceinline__ float ld(int v) const { return a[v]; }
};

// Flooding threads: one row (or column) per thread and pass.
template <int D>
constexpr int flood_threads() { return D <= 18 ? 1024 : 512; }

// What the flooding kernel keeps in shared memory: nothing, the hard decisions, the messages too.
enum class Place { kSlice, kHardSmem, kAllSmem };

// One float per edge, input and message of the edge in turn: the check phase replaces a row's
// inputs by its messages, the variable phase a column's messages by its next inputs.  Edge j of
// row r sits at cv.wide_stride * j + (r with its low 5 bits XORed by the next 5): rows are read
// conflict-free and the strided rows of a quasi-cyclic column spread over the banks.  The array
// lives in shared memory when it fits (the N16200 codes), else in the CTA's slice.  The syndrome reads
// the hard decisions packed 32 to a word, in shared memory too (in the slice for codes of more than
// 1.8 million bits); without best-syndrome tracking it stops at the first unsatisfied rows.  kDamp:
// the inputs are kept beside, in the slice.
//
// Measured on GB300, 333 codewords of (16200,13320) at 4 dB: 2.8 ms before (per edge of each of
// two column passes an edge, row and row-pointer lookup and a message rebuild, all from L2),
// 0.38 ms now.
template <int D, bool kDamp, Place kPlace>
__global__ void __launch_bounds__(flood_threads<D>(), 1)
bp_flooding_wide_kernel(FloodView cv, BpParams p, BpIO io, float* scratch, long long slice, int track_best)
{
    constexpr int kThreads = flood_threads<D>();
    constexpr bool kSmem = kPlace == Place::kAllSmem;
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ int s_red[kThreads / 32];
    __shared__ int s_next, s_slot;
    const int tid = threadIdx.x;
    const int n = cv.n, m = cv.m, n_pad = (n + 3) & ~3, stride = cv.wide_stride;
    const int words = (n + 31) / 32 + 1;  // the last one stays 0: missing edges of short rows read it
    float* g = scratch + static_cast<size_t>(blockIdx.x) * static_cast<size_t>(slice);
    float* app = g;
    float* best = app + n_pad;  // only when track_best
    float* rest = best + (track_best ? n_pad : 0);
    float* msg = kSmem ? reinterpret_cast<float*>(s_raw + ((static_cast<size_t>(words) * 4 + 15) & ~size_t(15))) : rest;
    float* old = rest + (kSmem ? 0 : static_cast<size_t>(cv.maxdeg) * stride);  // only when kDamp
    uint32_t* hard = reinterpret_cast<uint32_t*>(s_raw);
    if constexpr (kPlace == Place::kSlice)
        hard = reinterpret_cast<uint32_t*>(old + (kDamp ? static_cast<size_t>(cv.maxdeg) * stride : 0));
    const float keep = __fsub_rn(1.0f, p.damping);
    const auto slot = [](int r) { return r ^ ((r >> 5) & 31); };

    auto parity_of = [&](int r) -> unsigned {
        unsigned par = 0u;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            if (j < cv.maxdeg) {
                const unsigned v = __ldg(cv.wide_vars + static_cast<size_t>(j) * m + r);
                par ^= hard[v >> 5] >> (v & 31u);
            }
        }
        return par & 1u;
    };
    // Syndrome weight; without tracking, any nonzero value when it is not zero.
    auto syndrome = [&]() -> int {
        int cnt = 0;
        if (track_best) {
            for (int r = tid; r < m; r += kThreads) cnt += static_cast<int>(parity_of(r));
            return cta_sum<kThreads>(cnt, s_red);
        }
        for (int r0 = 0; r0 < m; r0 += kThreads) {
            if (r0 + tid < m) cnt = static_cast<int>(parity_of(r0 + tid));
            if (__syncthreads_or(cnt)) return 1;
        }
        return 0;
    };

    if (tid == 0) hard[words - 1] = 0u;
    for (int c = blockIdx.x; c < io.count; c = wide_next(io, &s_next)) {
        const float* llr = io.llr + static_cast<size_t>(c) * n;
        for (int v0 = 0; v0 < n; v0 += kThreads) {
            const int v = v0 + tid;
            const float x = v < n ? llr[v] : 0.0f;
            if (v < n) {
                if (track_best) best[v] = x;
                const float q = reg::canonical(x);
                const int e1 = __ldg(cv.col_ptr + v + 1);
                for (int e = __ldg(cv.col_ptr + v); e < e1; ++e) {
                    const int at = __ldg(cv.wide_pos + e);
                    msg[at] = q;
                    if constexpr (kDamp) old[at] = q;
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, x < 0.0f);
            if ((tid & 31) == 0 && v < n) hard[v >> 5] = b;
        }
        __syncthreads();
        int best_w = track_best ? syndrome() : 1;
        int iter = 0, w = 0;
        for (;;) {
            // check nodes (L:3033-3060)
            for (int r = tid; r < m; r += kThreads) {
                const int deg = __ldg(cv.row_ptr + r + 1) - __ldg(cv.row_ptr + r), base = slot(r);
                float q[D], out[D];
#pragma unroll
                for (int j = 0; j < D; ++j) q[j] = j < deg ? msg[j * stride + base] : __int_as_float(0x7f800000);
                reg::row_messages<D>(q, p.alpha, p.beta, out);
#pragma unroll
                for (int j = 0; j < D; ++j)
                    if (j < deg) msg[j * stride + base] = out[j];
            }
            __syncthreads();
            // variable nodes (L:3062-3069): llr + sum of messages in row order; the next inputs
            // (L:3076-3081), optional damping
            for (int v0 = 0; v0 < n; v0 += kThreads) {
                const int v = v0 + tid;
                float acc = 0.0f;
                if (v < n) {
                    acc = reg::canonical(__ldg(llr + v));
                    const int e0 = __ldg(cv.col_ptr + v), e1 = __ldg(cv.col_ptr + v + 1);
                    int at[4];  // the first edges' positions (and most columns' all)
                    float r[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        at[i] = e0 + i < e1 ? __ldg(cv.wide_pos + e0 + i) : -1;
                        r[i] = at[i] >= 0 ? msg[at[i]] : 0.0f;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (at[i] >= 0) acc = __fadd_rn(acc, r[i]);
                    for (int e = e0 + 4; e < e1; ++e) acc = __fadd_rn(acc, msg[__ldg(cv.wide_pos + e)]);
                    app[v] = acc;
                    auto next = [&](int pos, float message) {
                        const float fresh = __fsub_rn(acc, message);
                        if constexpr (kDamp) {
                            const float q = reg::canonical(__fadd_rn(__fmul_rn(keep, fresh), __fmul_rn(p.damping, old[pos])));
                            msg[pos] = q;
                            old[pos] = q;
                        } else {
                            msg[pos] = fresh;
                        }
                    };
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (at[i] >= 0) next(at[i], r[i]);
                    for (int e = e0 + 4; e < e1; ++e) {
                        const int pos = __ldg(cv.wide_pos + e);
                        next(pos, msg[pos]);
                    }
                }
                const unsigned b = __ballot_sync(0xffffffffu, acc < 0.0f);
                if ((tid & 31) == 0 && v < n) hard[v >> 5] = b;
            }
            __syncthreads();
            w = syndrome();
            ++iter;
            if (track_best && (w < best_w || (w == 0 && best_w == 0)))
                for (int i = tid; i < n; i += kThreads) best[i] = app[i];
            if (w < best_w) best_w = w;
            if (w == 0 || iter >= p.max_iter) break;
        }
        wide_finish<kThreads>(p, io, c, n, w, iter, PlainApp{app}, best, track_best != 0, s_red, &s_slot);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

namespace {

// Grid of the wide kernels: up to `per_sm` CTAs per SM, no more CTAs than codewords, and
// no more slices than keep the grid's scratch within `l2_budget` bytes (at least one CTA
// per SM).
int wide_grid(int count, int per_sm, size_t slice_bytes)
{
    constexpr size_t l2_budget = size_t(96) << 20;
    const int sms = device_sm_count();
    int ctas = std::max(1, per_sm) * sms;
    const size_t fit = slice_bytes > 0 ? l2_budget / slice_bytes : static_cast<size_t>(ctas);
    ctas = std::min<long long>(ctas, std::max<long long>(sms, static_cast<long long>(fit)));
    return std::max(1, std::min(ctas, count));
}

// Shared memory of the flooding kernel: the packed hard decisions, and the messages when they fit.
size_t flood_hard_bytes(const FloodView& cv) { return (static_cast<size_t>((cv.n + 31) / 32 + 1) * 4 + 15) & ~size_t(15); }
size_t flood_msg_bytes(const FloodView& cv) { return static_cast<size_t>(cv.maxdeg) * cv.wide_stride * sizeof(float); }

template <int D, bool kDamp, Place kPlace>
void launch_flooding_wide_t(const FloodView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    constexpr bool kSmem = kPlace == Place::kAllSmem;
    const auto kernel = bp_flooding_wide_kernel<D, kDamp, kPlace>;
    const size_t smem = (kPlace == Place::kSlice ? 0 : flood_hard_bytes(cv)) + (kSmem ? flood_msg_bytes(cv) : 0);
    check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(kernel), smem), "cudaFuncSetAttribute(bp wide)");
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, flood_threads<D>(), smem) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    const long long n_pad = (cv.n + 3) & ~3, edges = static_cast<long long>(cv.maxdeg) * cv.wide_stride;
    long long slice = n_pad + (track_best ? n_pad : 0) + (kSmem ? 0 : edges) + (kDamp ? edges : 0) +
                      (kPlace == Place::kSlice ? static_cast<long long>(flood_hard_bytes(cv) / sizeof(float)) : 0);
    slice = (slice + 31) & ~31LL;
    const size_t slice_bytes = static_cast<size_t>(slice) * sizeof(float);
    const int ctas = wide_grid(io.count, per_sm, slice_bytes);
    int device = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    void* scratch = nullptr;
    check_cuda(cudaMallocFromPoolAsync(&scratch, std::max<size_t>(slice_bytes * ctas, 16), scratch_pool(device), st),
               "cudaMallocFromPoolAsync(bp wide)");
    kernel<<<ctas, flood_threads<D>(), smem, st>>>(cv, p, io, static_cast<float*>(scratch), slice, track_best ? 1 : 0);
    const cudaError_t err = cudaGetLastError();
    const cudaError_t ferr = cudaFreeAsync(scratch, st);
    check_cuda(err, "bp wide kernel launch");
    check_cuda(ferr, "cudaFreeAsync(bp wide)");
}

template <int D, bool kDamp>
void launch_flooding_wide_d(const FloodView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    constexpr size_t most = 226 * 1024;  // 1 KB of the 227 KB stays for the kernel's static arrays
    if (flood_hard_bytes(cv) + flood_msg_bytes(cv) <= most) launch_flooding_wide_t<D, kDamp, Place::kAllSmem>(cv, p, io, track_best, st);
    else if (flood_hard_bytes(cv) <= most) launch_flooding_wide_t<D, kDamp, Place::kHardSmem>(cv, p, io, track_best, st);
    else launch_flooding_wide_t<27, kDamp, Place::kSlice>(cv, p, io, track_best, st);  // one instance for any degree
}

template <int D>
void launch_flooding_wide(const FloodView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    if (p.damping == 0.0f) launch_flooding_wide_d<D, false>(cv, p, io, track_best, st);
    else launch_flooding_wide_d<D, true>(cv, p, io, track_best, st);
}

template <int D, int kFar>
void launch_layered_wide_t(const LayeredView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    const long long n_pad = (cv.n + 3) & ~3;
    const long long mp = cv.m;
    const int split = wide_split(cv.n);
    const bool all_smem = split > n_pad;
    const size_t smem = static_cast<size_t>(split) * sizeof(float);
    long long slice = (all_smem ? 0 : n_pad + 4) + (track_best ? n_pad : 0) + 4 * mp;
    slice = (slice + 31) & ~31LL;  // 128-byte aligned slices
    const auto kernel = bp_layered_wide_kernel<D, kFar>;
    check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(kernel), smem), "cudaFuncSetAttribute(bp wide)");
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, wide_threads<D>(), smem) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    const size_t slice_bytes = static_cast<size_t>(slice) * sizeof(float);
    const int ctas = wide_grid(io.count, per_sm, slice_bytes);
    int device = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    void* scratch = nullptr;
    check_cuda(cudaMallocFromPoolAsync(&scratch, std::max<size_t>(slice_bytes * ctas, 16), scratch_pool(device), st),
               "cudaMallocFromPoolAsync(bp wide)");
    kernel<<<ctas, wide_threads<D>(), smem, st>>>(cv, p, io, static_cast<float*>(scratch), slice, split, track_best ? 1 : 0);
    const cudaError_t err = cudaGetLastError();
    const cudaError_t ferr = cudaFreeAsync(scratch, st);
    check_cuda(err, "bp wide kernel launch");
    check_cuda(ferr, "cudaFreeAsync(bp wide)");
}

template <int D>
void launch_layered_wide_d(const LayeredView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    if (cv.wide_smem_slots >= D) launch_layered_wide_t<D, 0>(cv, p, io, track_best, st);
    else if (cv.wide_smem_slots >= D - 2) launch_layered_wide_t<D, 2>(cv, p, io, track_best, st);
    else launch_layered_wide_t<D, D>(cv, p, io, track_best, st);
}

}  // namespace

// Posteriors in shared memory (the dummy posterior, padded to 4 floats, after the last): all of
// them up to 200 KB, else the first 56,320 (220 KB; variables beyond and the dummy in the slice).
int wide_split(int n)
{
    const int n_pad = (n + 3) & ~3;
    return (n_pad + 4) * sizeof(float) <= 200 * 1024 ? n_pad + 4 : static_cast<int>(220 * 1024 / sizeof(float));
}

// Edge slots of a row in the wide kernel: the closest compiled degree.
int wide_slots(int maxdeg)
{
    for (int d : {4, 6, 7, 10, 14, 18, 27})
        if (maxdeg <= d) return d;
    return 0;
}

bool layered_needs_wide(const LayeredView& cv, bool track_best)
{
    const int step = std::max(1, 32 / cv.group);
    return layered_smem_bytes(cv, step, track_best, nullptr) > 227 * 1024;
}

bool flooding_needs_wide(const FloodView& cv) { return flooding_smem_bytes(cv, 1, nullptr) > 227 * 1024; }

void launch_bp_layered_wide(const LayeredView& cv, const BpParams& p, const BpIO& io, cudaStream_t st)
{
    if (io.count <= 0) return;
    const bool track_best = p.route_failures_to_osd && io.osd_llr != nullptr;
    if (!io.work_zeroed) check_cuda(cudaMemsetAsync(io.work_counter, 0, sizeof(int), st), "reset work counter");
    switch (wide_slots(cv.maxdeg)) {
        case 4: launch_layered_wide_d<4>(cv, p, io, track_best, st); break;
        case 6: launch_layered_wide_d<6>(cv, p, io, track_best, st); break;
        case 7: launch_layered_wide_d<7>(cv, p, io, track_best, st); break;
        case 10: launch_layered_wide_d<10>(cv, p, io, track_best, st); break;
        case 14: launch_layered_wide_d<14>(cv, p, io, track_best, st); break;
        case 18: launch_layered_wide_d<18>(cv, p, io, track_best, st); break;
        default: launch_layered_wide_d<27>(cv, p, io, track_best, st); break;
    }
}

void launch_bp_flooding_wide(const FloodView& cv, const BpParams& p, const BpIO& io, cudaStream_t st)
{
    if (io.count <= 0) return;
    if (cv.maxdeg > 27) throw InvalidArgument("flooding schedule supports row degree <= 27");
    const bool track_best = p.route_failures_to_osd && io.osd_llr != nullptr;
    if (!io.work_zeroed) check_cuda(cudaMemsetAsync(io.work_counter, 0, sizeof(int), st), "reset work counter");
    if (cv.maxdeg <= 6) launch_flooding_wide<6>(cv, p, io, track_best, st);
    else if (cv.maxdeg <= 10) launch_flooding_wide<10>(cv, p, io, track_best, st);
    else if (cv.maxdeg <= 18) launch_flooding_wide<18>(cv, p, io, track_best, st);
    else launch_flooding_wide<27>(cv, p, io, track_best, st);
}

}  // namespace sicc
