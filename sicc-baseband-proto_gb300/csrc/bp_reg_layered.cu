// Layered min-sum (schedules 2, 3) with register-resident messages (bp_reg.cuh):
// codes whose lanes own few enough rows, any group of up to 128 lanes per
// codeword.  Rows, order and arithmetic are those of bp_layered_kernel
// (bp_kernels.cu).  Groups run persistently and take codewords from a counter.
//
// Measured on GB300 against the kernels before it (compressed row state, in
// registers for the (128,64) code, else in shared memory): 65,536 frames of
// (128,64) at 2 dB 235 -> 120 us (ALU pipe 80% busy before, 46% now; shared-
// memory pipe 58%); 7,680 codewords of (1024,512) at 2 dB 1,000 -> 245 us;
// 1,000 of (2048,1024) at 2.5 dB 645 -> 82 us.
#include "bp_kernels.h"
#include "bp_reg.cuh"

#include <algorithm>
#include <type_traits>

namespace sicc {

namespace {

using namespace reg;

// kPlain: every lane owns exactly NL rows, one per layer (the quasi-cyclic codes): no row tests.
template <int D, int NL, int W, bool kPlain>
__global__ void __launch_bounds__(reg_threads<D, NL>(), 3)
bp_layered_reg_kernel(LayeredView cv, BpParams p, BpIO io, int slots_per_cta, int slot_floats, int track_best)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_red[reg_threads<D, NL>() / 32 * (W + 1)];
    const Group<W> g(cv.reg_group, s_red);
    const int n = cv.n, n_pad = (n + 3) & ~3;
    const int nrows = cv.num_layers * cv.reg_rpl;
    const unsigned base = static_cast<unsigned>(g.slot * slot_floats) * 4u;
    float* app = reinterpret_cast<float*>(smem + base);
    float* best = app + static_cast<size_t>(slots_per_cta) * slot_floats;  // only when track_best

    Rows<D, NL> rows;  // for the whole launch
    rows.load(cv.vars, cv.num_layers, cv.reg_rpl, cv.width, cv.maxdeg, g.G, g.gl, base, n_pad);
    float msg[NL][D];

    const int total_groups = gridDim.x * slots_per_cta;
    int c = blockIdx.x * slots_per_cta + g.slot;
    bool active = c < io.count;
    int iter = 0, best_w = 0;
    auto init = [&](int cw) {
        load_llr(io, cw, n, g.gl, g.G, app, track_best ? best : nullptr);
        static_for<NL>([&](auto ti) {
#pragma unroll
            for (int j = 0; j < D; ++j) msg[decltype(ti)::value][j] = 0.0f;
        });
        g.sync();
        best_w = track_best ? g.sum(lane_syndrome<kPlain, 0, NL>(smem, rows, nrows)) : 1;
        iter = 0;
    };
    if (g.gl == 0) app[n_pad] = __int_as_float(0x7f800000);  // +inf, before init's sync
    if (active) init(c);

    while (any_active<W>(active)) {
        if (!active) continue;
        static_for<NL>([&](auto ti) {
            constexpr int t = decltype(ti)::value;
            if (kPlain || t < nrows) {
                if (kPlain || ((rows.real >> t) & 1u)) update_row(smem, rows, t, p.alpha, p.beta, msg[t]);
                if (kPlain || (t + 1) % cv.reg_rpl == 0) g.sync();  // end of a layer
            }
        });
        // without tracking only "zero or not" matters: a lane's other rows are read only when the
        // group's first rows all hold (7,680 codewords of (1024,512) at 2 dB 300 -> 245 us)
        unsigned bad = lane_syndrome<kPlain, 0, 1>(smem, rows, nrows);
        int w = track_best ? 0 : g.sum(bad);
        if (w == 0) {
            bad += lane_syndrome<kPlain, 1, NL>(smem, rows, nrows);
            if (W > 1 && !track_best) g.sync();  // between two sums
            w = g.sum(bad);
        }
        ++iter;
        // the best posterior so far (a zero syndrome always is, and then it is app itself)
        if (track_best && w < best_w && w != 0) {
            copy_slot(g, best, app, n_pad);
            g.sync();
        }
        best_w = min(best_w, w);
        if (w == 0 || iter >= p.max_iter) {
            finish(g, p, io, c, n, w, iter, app, (track_best && w != 0) ? best : app);
            c = g.from_leader(g.gl == 0 ? total_groups + atomicAdd(io.work_counter, 1) : 0);
            active = c < io.count;
            g.sync();
            if (active) init(c);
        }
    }
}

template <int D, int NL, bool kPlain>
void launch_shape(const LayeredView& cv, const BpParams& p, const BpIO& io, const BpLaunch& shape, bool track_best,
                  cudaStream_t st)
{
    const int arrays = track_best ? 2 : 1;
    if constexpr (kPlain) {
        if (cv.reg_group == 64) {
            launch_reg<D, NL>(bp_layered_reg_kernel<D, NL, 2, true>, cv, p, io, shape, arrays, track_best, st);
            return;
        }
        if (cv.reg_group == 128) {
            launch_reg<D, NL>(bp_layered_reg_kernel<D, NL, 4, true>, cv, p, io, shape, arrays, track_best, st);
            return;
        }
    }
    launch_reg<D, NL>(bp_layered_reg_kernel<D, NL, 1, kPlain>, cv, p, io, shape, arrays, track_best, st);
}

// The shapes compiled: for plain codes the row counts and degrees of the 4-, 5- and 8-layer
// quasi-cyclic codes, rounded up to (6,4), (14,4), (14,5), (10,8); for ragged ones (layers of
// different widths, or several rows of a layer per lane) the closest of three with row tests.
// f(D, NL, plain) as integral constants for the code's shape.
template <class F>
void with_shape(const LayeredView& cv, F&& f)
{
    const auto call = [&](auto d, auto nl) {
        if (cv.reg_plain) f(d, nl, std::true_type());
        else f(d, nl, std::false_type());
    };
    const int rows = cv.num_layers * cv.reg_rpl;
    using std::integral_constant;
    const bool small = cv.maxdeg <= 6 && (cv.reg_plain ? rows == 4 : rows <= 4);
    if (small) call(integral_constant<int, 6>(), integral_constant<int, 4>());
    else if (cv.reg_plain && rows == 4) f(integral_constant<int, 14>(), integral_constant<int, 4>(), std::true_type());
    else if (cv.reg_plain ? rows == 5 : cv.maxdeg > 10) call(integral_constant<int, 14>(), integral_constant<int, 5>());
    else call(integral_constant<int, 10>(), integral_constant<int, 8>());
}

}  // namespace

void launch_bp_layered_reg(const LayeredView& cv, const BpParams& p, const BpIO& io, const BpLaunch& shape,
                           bool track_best, cudaStream_t st)
{
    with_shape(cv, [&](auto d, auto nl, auto plain) {
        launch_shape<decltype(d)::value, decltype(nl)::value, decltype(plain)::value>(cv, p, io, shape, track_best, st);
    });
}

int layered_reg_default_slots(const LayeredView& cv, bool track_best)
{
    int slots = 0;
    with_shape(cv, [&](auto d, auto nl, auto) {
        int slot_floats = 0;
        size_t smem = 0;
        slots = reg_slots<decltype(d)::value, decltype(nl)::value>(cv, 0, track_best ? 2 : 1, &slot_floats, &smem);
    });
    return slots;
}

void reg_plan(LayeredView& cv, int widest, int narrowest, int group)
{
    cv.reg_group = cv.reg_rpl = cv.reg_plain = 0;
    const bool fixed = group > 0;
    if (!fixed) {
        group = 1;
        while (group < widest && group < 128) group <<= 1;
    }
    int rpl = (widest + group - 1) / group;
    const bool plain = rpl == 1 && narrowest == group &&
                       ((cv.num_layers == 8 && cv.maxdeg <= 10) || (cv.num_layers == 4 && cv.maxdeg <= 14) ||
                        (cv.num_layers == 5 && cv.maxdeg <= 14));
    if (!plain) {  // ragged codes: within a warp
        group = std::min(group, 32);
        rpl = (widest + group - 1) / group;
        const int rows = cv.num_layers * rpl;
        if (!(cv.maxdeg <= 10 && rows <= 8) && !(cv.maxdeg <= 14 && rows <= 5)) return;
    }
    // a CTA's posteriors sit at 16-bit byte offsets in the large shapes; one warp's codewords
    // (three regions each at most) have to fit a CTA's shared memory
    const size_t n_pad = (cv.n + 3) & ~3, slots = std::max(1, 32 / group);
    if (slots * (n_pad + 36) * sizeof(float) >= 65536) return;
    cv.reg_group = group;
    cv.reg_rpl = rpl;
    cv.reg_plain = plain ? 1 : 0;
}

}  // namespace sicc
