// Register-resident min-sum rows: the parts shared by the single-code kernels
// (bp_reg_layered.cu, bp_reg_flooding.cu) and the mixed-code kernel (engine.cu).
//
// A group of G lanes owns one codeword; lane g owns row slots g, g + G, ... of
// every layer, at most NL rows in all.  A lane keeps its rows' messages in
// registers, one float per edge, and the shared-memory byte offsets of the
// rows' posteriors, so shared memory holds the posteriors only: an edge costs
// one load and one store per update and one load per syndrome.
//
// What bounds it: the ALU pipe (min/max, compare, select and logic run on 16
// lanes per scheduler, half the issue rate), shared memory and plain issue.
// Messages kept as such need no rebuild from a compressed (min1, min2, argmin,
// signs) state.  A row's outgoing messages come as exclusive minima -- over the
// row's other edges, from the minima of groups of two to four edges -- by
// min.xorsign.abs, which takes the smaller magnitude and multiplies the signs
// in one ALU operation: 2.7 to 2.9 per edge for magnitude and sign together,
// against 15 for rebuild, (min1, min2, argmin), compare, select and signs.
// Scaling and additions run on the FMA pipe, which is otherwise idle.
#pragma once

#include "bp_device.cuh"
#include "bp_kernels.h"

#include <algorithm>
#include <cfloat>
#include <type_traits>
#include <utility>

namespace sicc {
namespace reg {

// f(0), f(1), .. f(N - 1) with compile-time arguments (row loops whose register arrays must not
// end up in local memory).
template <int... I, class F>
__device__ __forceinline__ void static_for_(std::integer_sequence<int, I...>, F&& f)
{
    (f(std::integral_constant<int, I>()), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f)
{
    static_for_(std::make_integer_sequence<int, N>(), f);
}

// Edges 0 .. D-1 of a row (D <= 16) in two to four groups of two to four.
template <int D>
struct Split {
    static constexpr int ng = D <= 6 ? 2 : D <= 8 ? 3 : 4;
    __host__ __device__ static constexpr int size(int i) { return D / ng + (i < D % ng ? 1 : 0); }
    __host__ __device__ static constexpr int start(int i) { return i == 0 ? 0 : start(i - 1) + size(i - 1); }
};

// The smaller magnitude of the two (a NaN is passed over), with the product of their signs.
__device__ __forceinline__ float minx(float a, float b)
{
    float d;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}

__device__ __forceinline__ float max3(float a, float b, float c)  // the largest magnitude
{
    float d;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// |m[j]| = min(FLT_MAX, min over i != j of |a[i]|), sign = product of the other
// signs: the magnitude (min1, min2, argmin) tracking from FLT_MAX gives edge j,
// whichever of equal minima it names the argmin.
template <int D>
__device__ __forceinline__ void exclusive_min(const float (&a)[D], float (&m)[D])
{
    if constexpr (D > 16) {  // prefix and suffix minima: three operations per edge, few registers
        float run = FLT_MAX;
#pragma unroll
        for (int j = 0; j < D; ++j) {
            m[j] = run;
            run = minx(run, a[j]);
        }
        run = FLT_MAX;
#pragma unroll
        for (int j = D - 1; j >= 0; --j) {
            m[j] = minx(m[j], run);
            run = minx(run, a[j]);
        }
        return;
    }
    using S = Split<D>;
    float g[4], e[4], pr[4][3];
    static_for<S::ng>([&](auto gi) {
        constexpr int i = decltype(gi)::value, s = S::start(i), size = S::size(i);
        if constexpr (size == 2) {
            g[i] = minx(a[s], a[s + 1]);
        } else if constexpr (size == 3) {
            pr[i][0] = minx(a[s], a[s + 1]);
            pr[i][1] = minx(a[s], a[s + 2]);
            pr[i][2] = minx(a[s + 1], a[s + 2]);
            g[i] = minx(pr[i][0], a[s + 2]);
        } else {
            pr[i][0] = minx(a[s], a[s + 1]);
            pr[i][1] = minx(a[s + 2], a[s + 3]);
            g[i] = minx(pr[i][0], pr[i][1]);
        }
    });
    if constexpr (S::ng == 2) {
        e[0] = minx(g[1], FLT_MAX);
        e[1] = minx(g[0], FLT_MAX);
    } else if constexpr (S::ng == 3) {
        g[1] = minx(g[1], FLT_MAX);
        g[2] = minx(g[2], FLT_MAX);
        e[0] = minx(g[1], g[2]);
        e[1] = minx(g[0], g[2]);
        e[2] = minx(g[0], g[1]);
    } else {
        const float g01 = minx(minx(g[0], g[1]), FLT_MAX), g23 = minx(minx(g[2], g[3]), FLT_MAX);
        e[0] = minx(g[1], g23);
        e[1] = minx(g[0], g23);
        e[2] = minx(g[3], g01);
        e[3] = minx(g[2], g01);
    }
    static_for<S::ng>([&](auto gi) {
        constexpr int i = decltype(gi)::value, s = S::start(i), size = S::size(i);
        if constexpr (size == 2) {
            m[s] = minx(a[s + 1], e[i]);
            m[s + 1] = minx(a[s], e[i]);
        } else if constexpr (size == 3) {
            m[s] = minx(pr[i][2], e[i]);
            m[s + 1] = minx(pr[i][1], e[i]);
            m[s + 2] = minx(pr[i][0], e[i]);
        } else {
            const float u0 = minx(pr[i][1], e[i]), u1 = minx(pr[i][0], e[i]);
            m[s] = minx(a[s + 1], u0);
            m[s + 1] = minx(a[s], u0);
            m[s + 2] = minx(a[s + 3], u1);
            m[s + 3] = minx(a[s + 2], u1);
        }
    });
}

// Outgoing messages of a row with inputs q (none of them -0, NaN only as an
// addition gives it): sign = product of the other inputs' signs (zero counts
// as positive), magnitude = nms_mag of their smallest magnitude.
template <int D>
__device__ __forceinline__ void row_messages(const float (&q)[D], float alpha, float beta, float (&msg)[D])
{
    exclusive_min<D>(q, msg);
    if (beta == 0.0f) {
#pragma unroll
        for (int j = 0; j < D; ++j) msg[j] = __fmul_rn(alpha, msg[j]);
    } else {
#pragma unroll
        for (int j = 0; j < D; ++j)
            msg[j] = __uint_as_float(__float_as_uint(nms_mag(alpha, beta, fabsf(msg[j]))) | (__float_as_uint(msg[j]) & 0x80000000u));
    }
}

// Shared-memory byte offsets of a lane's D posteriors per row: 32 bits each, or
// (above 40 edges per lane, where they would crowd out the messages) two to a
// register.
template <int D, int NL>
struct Rows {
    static constexpr bool kPacked = D * NL > 40;
    static constexpr int kWords = kPacked ? (D + 1) / 2 : D;
    unsigned w[NL][kWords];
    unsigned real;  // bit t: row t of this lane exists (plain codes: every one does)

    __device__ __forceinline__ unsigned off(int t, int j) const
    {
        if constexpr (kPacked) return (j & 1) ? w[t][j >> 1] >> 16 : w[t][j >> 1] & 0xffffu;
        else return w[t][j];
    }

    // Row t: layer t / rpl, slot gl + (t mod rpl) G.  `base`: byte offset of the codeword's
    // posteriors; a missing edge points at posterior `dummy` (+inf: never a row's minimum or
    // sign, never a parity flip, and left at +inf by its update).
    __device__ __forceinline__ void load(const int* __restrict__ vars, int num_layers, int rpl, int width, int maxdeg,
                                         int G, int gl, unsigned base, int dummy)
    {
        real = 0u;
        const int nrows = num_layers * rpl;
        static_for<NL>([&](auto ti) {
            constexpr int t = decltype(ti)::value;
            const int L = t / rpl, rs = gl + (t - L * rpl) * G;
            const bool in = t < nrows && rs < width;
#pragma unroll
            for (int x = 0; x < kWords; ++x) w[t][x] = 0u;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                const int v = (in && j < maxdeg) ? __ldg(vars + (L * maxdeg + j) * width + rs) : -1;
                const unsigned o = base + 4u * static_cast<unsigned>(v >= 0 ? v : dummy);
                if constexpr (kPacked) w[t][j >> 1] |= (j & 1) ? o << 16 : o;
                else w[t][j] = o;
                if (j == 0) real |= v >= 0 ? 1u << t : 0u;
            }
        });
    }
};

__device__ __forceinline__ float lds(const unsigned char* smem, unsigned off)
{
    return *reinterpret_cast<const float*>(smem + off);
}
__device__ __forceinline__ void sts(unsigned char* smem, unsigned off, float v)
{
    *reinterpret_cast<float*>(smem + off) = v;
}

// A received value as the rows take it: -0 to +0 and any NaN to the one that
// additions give, so that a sign bit says "negative" (the values and every
// comparison with them stay the same).
__device__ __forceinline__ float canonical(float x) { return __fadd_rn(x, 0.0f); }

// Layered update of row t.
template <int D, int NL>
__device__ __forceinline__ void update_row(unsigned char* smem, const Rows<D, NL>& r, int t, float alpha, float beta,
                                           float (&msg)[D])
{
    float q[D];
#pragma unroll
    for (int j = 0; j < D; ++j) q[j] = __fsub_rn(lds(smem, r.off(t, j)), msg[j]);
    row_messages<D>(q, alpha, beta, msg);
#pragma unroll
    for (int j = 0; j < D; ++j) sts(smem, r.off(t, j), __fadd_rn(q[j], msg[j]));
}

// Unsatisfied checks among the lane's rows kFrom .. kTo - 1.
template <bool kPlain, int kFrom, int kTo, int D, int NL>
__device__ __forceinline__ unsigned lane_syndrome(const unsigned char* smem, const Rows<D, NL>& r, int nrows)
{
    unsigned cnt = 0u;
    static_for<kTo - kFrom>([&](auto ti) {
        constexpr int t = kFrom + decltype(ti)::value;
        if (kPlain || t < nrows) {
            unsigned par = 0u;
#pragma unroll
            for (int j = 0; j < D; ++j) par ^= __float_as_uint(lds(smem, r.off(t, j)));
            cnt += par >> 31;
        }
    });
    return cnt;
}

// Threads of a CTA: the large shapes hold up to 80 messages and 40 offset words per lane
// (168 registers: three CTAs of 128), the small one 24 and 24 (80: three of 256).
template <int D, int NL>
constexpr int reg_threads() { return D * NL > 40 ? 128 : 256; }

// The lanes of one codeword: G <= 32 lanes of a warp (W = 1) or W whole warps on a named barrier
// (1, 2 for groups of four warps, 3 .. 6 for groups of two: at most 256 threads).
template <int W>
struct Group {
    int G, gl, slot, lane, leader;
    unsigned gmask;
    int* red;  // W > 1: [slots][W + 1] sums, broadcast value

    __device__ __forceinline__ Group(int group, int* red_all)
    {
        lane = threadIdx.x & 31;
        if constexpr (W == 1) {
            G = group;
            gl = lane & (G - 1);
            const int sub = lane / G;
            gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (sub * G));
            leader = sub * G;
        } else {
            G = W * 32;
            gl = threadIdx.x & (G - 1);
            gmask = 0xffffffffu;
            leader = 0;
        }
        slot = threadIdx.x / G;
        red = red_all + slot * (W + 1);
    }
    __device__ __forceinline__ void sync() const
    {
        if constexpr (W == 1) __syncwarp(gmask);
        else asm volatile("bar.sync %0, %1;" ::"r"((W == 2 ? 3 : 1) + slot), "n"(W * 32) : "memory");
    }
    // Sum over the group, in every lane.  W > 1: two sums of a group need a sync() between them.
    __device__ __forceinline__ int sum(unsigned v) const
    {
        v = __reduce_add_sync(gmask, v);
        if constexpr (W > 1) {
            if (lane == 0) red[gl >> 5] = static_cast<int>(v);
            sync();
            v = 0u;
#pragma unroll
            for (int i = 0; i < W; ++i) v += static_cast<unsigned>(red[i]);
        }
        return static_cast<int>(v);
    }
    __device__ __forceinline__ unsigned min(unsigned v) const
    {
        v = __reduce_min_sync(gmask, v);
        if constexpr (W > 1) {
            sync();  // the previous sum is read
            if (lane == 0) red[gl >> 5] = static_cast<int>(v);
            sync();
#pragma unroll
            for (int i = 0; i < W; ++i) v = ::min(v, static_cast<unsigned>(red[i]));
        }
        return v;
    }
    // Lane 0's value, in every lane.
    __device__ __forceinline__ int from_leader(int v) const
    {
        if constexpr (W == 1) return __shfl_sync(gmask, v, leader);
        if (gl == 0) red[W] = v;
        sync();
        v = red[W];
        sync();
        return v;
    }
};

// Channel values of codeword c into app (canonical) and, when given, a plain copy.  The caller's array
// may start at any float (the rows then all start equally far from a 16-byte boundary).
__device__ __forceinline__ void load_llr(const BpIO& io, int c, int n, int gl, int G, float* app, float* plain)
{
    const float* src = io.llr + static_cast<size_t>(c) * n;
    if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        const float4* s4 = reinterpret_cast<const float4*>(src);
        for (int i = gl; i < (n >> 2); i += G) {
            const float4 v = __ldcs(s4 + i);
            reinterpret_cast<float4*>(app)[i] = make_float4(canonical(v.x), canonical(v.y), canonical(v.z), canonical(v.w));
            if (plain) reinterpret_cast<float4*>(plain)[i] = v;
        }
    } else {
        for (int i = gl; i < n; i += G) {
            const float v = __ldcs(src + i);
            app[i] = canonical(v);
            if (plain) plain[i] = v;
        }
    }
}

// Outputs of codeword c, stopped with syndrome weight w after `iter` iterations; `b` is the
// posterior for OSD.
template <int W>
__device__ __forceinline__ void finish(const Group<W>& g, const BpParams& p, const BpIO& io, int c, int n, int w,
                                       int iter, const float* app, const float* b)
{
    bool accept = (w == 0);
    if (accept && p.min_abs_accept > 0.0f) {
        unsigned mn = 0x7f800000u;
        for (int i = g.gl; i < n; i += g.G) mn = ::min(mn, __float_as_uint(fabsf(app[i])));
        accept = __uint_as_float(g.min(mn)) >= p.min_abs_accept;
    }
    const bool route = !accept && p.route_failures_to_osd && io.osd_llr != nullptr;
    if (g.gl == 0) {
        if (io.success) io.success[c] = accept ? 1 : 0;
        if (io.iterations) io.iterations[c] = static_cast<uint8_t>(iter);
        if (io.used_osd) io.used_osd[c] = 0;
    }
    if (io.out_bits) {
        uint8_t* dst = io.out_bits + static_cast<size_t>(c) * io.out_stride;
        for (int i = g.gl; i < io.out_len; i += g.G) dst[i] = app[i] < 0.0f ? 1 : 0;
    }
    if (io.app_out) {
        float* dst = io.app_out + static_cast<size_t>(c) * n;
        for (int i = g.gl; i < n; i += g.G) dst[i] = app[i];
    }
    if (route) {
        const int s = g.from_leader(g.gl == 0 ? atomicAdd(io.osd_count, 1) : 0);
        float* dst = io.osd_llr + static_cast<size_t>(s) * n;
        for (int i = g.gl; i < n; i += g.G) dst[i] = b[i];
        if (g.gl == 0) io.osd_index[s] = c;
    }
}

// Where a group stands; W = 1 keeps a warp's groups in step (one iteration per pass).
template <int W>
__device__ __forceinline__ bool any_active(bool active)
{
    if constexpr (W == 1) return __any_sync(0xffffffffu, active);
    else return active;
}

// dst = src, n_pad floats of two slots of one group.
template <int W>
__device__ __forceinline__ void copy_slot(const Group<W>& g, float* dst, const float* src, int n_pad)
{
    for (int i = g.gl; i < (n_pad >> 2); i += g.G) reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
}

// One codeword's posteriors (and the dummy), in floats; `arrays` such regions per slot.
inline size_t reg_smem(const LayeredView& cv, int slots, int arrays, int* slot_floats)
{
    *slot_floats = pad_slot_stride(((cv.n + 3) & ~3) + 4, cv.reg_group);
    return static_cast<size_t>(slots) * arrays * *slot_floats * sizeof(float);
}

// Codewords per CTA: `wanted` (0: as many as run) within the shape's threads, three CTAs per SM, and the
// posteriors (the first of the arrays) below 64 KB: the large shapes hold their offsets in 16 bits
// (reg_plan has checked that one warp's codewords do).
template <int D, int NL>
int reg_slots(const LayeredView& cv, int wanted, int arrays, int* slot_floats, size_t* smem)
{
    const int step = std::max(1, 32 / cv.reg_group), most = reg_threads<D, NL>() / cv.reg_group;
    int slots = wanted > 0 ? std::min(wanted, most) : most;
    slots = std::max(step, slots - slots % step);
    *smem = reg_smem(cv, slots, arrays, slot_floats);
    while (slots > step && (*smem > 72 * 1024 || *smem / arrays > 65536)) *smem = reg_smem(cv, slots -= step, arrays, slot_floats);
    return slots;
}

template <int D, int NL, class Kernel>
void launch_reg(Kernel kernel, const LayeredView& cv, const BpParams& p, const BpIO& io, const BpLaunch& shape,
                int arrays, bool track_best, cudaStream_t st)
{
    const int G = cv.reg_group;
    int slot_floats = 0;
    size_t smem = 0;
    const int slots = reg_slots<D, NL>(cv, shape.slots_per_cta, arrays, &slot_floats, &smem);
    check_cuda(grant_dynamic_smem(reinterpret_cast<const void*>(kernel), smem), "cudaFuncSetAttribute(bp reg)");
    int ctas = shape.ctas;
    if (ctas <= 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, slots * G, smem) != cudaSuccess || per_sm <= 0)
            per_sm = 1;
        ctas = std::max(1, std::min(per_sm * device_sm_count(), (io.count + slots - 1) / slots));
    }
    kernel<<<ctas, slots * G, smem, st>>>(cv, p, io, slots, slot_floats, track_best ? 1 : 0);
    check_cuda(cudaGetLastError(), "bp reg kernel launch");
}

}  // namespace reg
}  // namespace sicc
