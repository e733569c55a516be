// Flooding min-sum (schedules 0, 1) with register-resident messages (bp_reg.cuh):
// the reference CPU decoder (uhd_ldpc_ofdm_link.cpp:3013-3094) with the damping
// of cpu_bp_osd_decode.m:180-183 and best-syndrome tracking (:160-171), run over
// row layers: runs of consecutive rows without a shared variable.  A variable's
// messages are added layer by layer, which is increasing row order, so every
// sum rounds as the reference's.  Groups run persistently and take codewords
// from a counter.
//
// Measured on GB300 against bp_flooding_kernel (bp_kernels.cu, which walks the
// edge lists and stays for codes that do not fit): 8,191 frames of (128,64) at
// 2 dB 230 -> 44 us; 2,001 codewords of (1024,768) at 3.5 dB, damped, 1,434 ->
// 76 us as a call (kernel 55).  The damped form keeps the inputs and recomputes the messages,
// so the large shapes take two CTAs per SM there: at three they spill (2,000 of
// (1024,512): 189 us against 151).
#include "bp_kernels.h"
#include "bp_reg.cuh"

#include <algorithm>
#include <type_traits>

namespace sicc {

namespace {

using namespace reg;

// The inputs q of a lane's rows are the state; kDamp: they are needed again beside the new
// posteriors, so the messages are recomputed from them instead of taking their registers.
// Plain codes only: every lane owns exactly NL rows, one per layer.
template <int D, int NL, int W, bool kDamp>
__global__ void __launch_bounds__(reg_threads<D, NL>(), (kDamp && D * NL > 40) ? 2 : 3)
bp_flooding_reg_kernel(LayeredView cv, BpParams p, BpIO io, int slots_per_cta, int slot_floats, int track_best)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_red[reg_threads<D, NL>() / 32 * (W + 1)];
    const Group<W> g(cv.reg_group, s_red);
    const int n = cv.n, n_pad = (n + 3) & ~3;
    const unsigned base = static_cast<unsigned>(g.slot * slot_floats) * 4u;
    float* app = reinterpret_cast<float*>(smem + base);
    float* llr = app + static_cast<size_t>(slots_per_cta) * slot_floats;
    float* best = llr + static_cast<size_t>(slots_per_cta) * slot_floats;  // only when track_best
    const float keep = __fsub_rn(1.0f, p.damping);

    Rows<D, NL> rows;
    rows.load(cv.vars, cv.num_layers, cv.reg_rpl, cv.width, cv.maxdeg, g.G, g.gl, base, n_pad);
    float q[NL][D];

    const int total_groups = gridDim.x * slots_per_cta;
    int c = blockIdx.x * slots_per_cta + g.slot;
    bool active = c < io.count;
    int iter = 0, best_w = 0;
    auto init = [&](int cw) {
        load_llr(io, cw, n, g.gl, g.G, app, track_best ? best : nullptr);
        g.sync();
        copy_slot(g, llr, app, n_pad);
        unsigned cnt = 0u;
        static_for<NL>([&](auto ti) {
            constexpr int t = decltype(ti)::value;
            unsigned par = 0u;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                q[t][j] = lds(smem, rows.off(t, j));
                par ^= __float_as_uint(q[t][j]);
            }
            cnt += par >> 31;
        });
        best_w = g.sum(cnt);
        g.sync();  // app is read before the first layer adds to it
        iter = 0;
    };
    if (g.gl == 0) app[n_pad] = __int_as_float(0x7f800000);  // +inf, before init's sync
    if (active) init(c);

    while (any_active<W>(active)) {
        if (!active) continue;
        // check nodes, and the variable sums llr + messages in row order (app holds llr)
        static_for<NL>([&](auto ti) {
            constexpr int t = decltype(ti)::value;
            float msg[D];
            row_messages<D>(q[t], p.alpha, p.beta, msg);
#pragma unroll
            for (int j = 0; j < D; ++j) {
                sts(smem, rows.off(t, j), __fadd_rn(lds(smem, rows.off(t, j)), msg[j]));
                if constexpr (!kDamp) q[t][j] = msg[j];
            }
            g.sync();  // end of a layer
        });
        // syndrome of the new posteriors and the next inputs from them
        unsigned cnt = 0u;
        static_for<NL>([&](auto ti) {
            constexpr int t = decltype(ti)::value;
            [[maybe_unused]] float msg[D];
            if constexpr (kDamp) row_messages<D>(q[t], p.alpha, p.beta, msg);
            unsigned par = 0u;
#pragma unroll
            for (int j = 0; j < D; ++j) {
                const float x = lds(smem, rows.off(t, j));
                par ^= __float_as_uint(x);
                if constexpr (kDamp)
                    q[t][j] = canonical(__fadd_rn(__fmul_rn(keep, __fsub_rn(x, msg[j])), __fmul_rn(p.damping, q[t][j])));
                else
                    q[t][j] = __fsub_rn(x, q[t][j]);
            }
            cnt += par >> 31;
        });
        const int w = g.sum(cnt);
        ++iter;
        if (track_best && w < best_w && w != 0) copy_slot(g, best, app, n_pad);
        best_w = min(best_w, w);
        g.sync();
        if (w == 0 || iter >= p.max_iter) {
            finish(g, p, io, c, n, w, iter, app, (track_best && w != 0) ? best : app);
            c = g.from_leader(g.gl == 0 ? total_groups + atomicAdd(io.work_counter, 1) : 0);
            active = c < io.count;
            g.sync();
            if (active) init(c);
        } else {
            copy_slot(g, app, llr, n_pad);
            g.sync();
        }
    }
}

template <int D, int NL, bool kDamp>
void launch_shape(const LayeredView& cv, const BpParams& p, const BpIO& io, bool track_best, cudaStream_t st)
{
    const int arrays = track_best ? 3 : 2;
    const BpLaunch shape{};
    if (cv.reg_group <= 32)
        launch_reg<D, NL>(bp_flooding_reg_kernel<D, NL, 1, kDamp>, cv, p, io, shape, arrays, track_best, st);
    else if (cv.reg_group == 64)
        launch_reg<D, NL>(bp_flooding_reg_kernel<D, NL, 2, kDamp>, cv, p, io, shape, arrays, track_best, st);
    else
        launch_reg<D, NL>(bp_flooding_reg_kernel<D, NL, 4, kDamp>, cv, p, io, shape, arrays, track_best, st);
}

}  // namespace

void launch_bp_flooding_reg(const LayeredView& cv, const BpParams& p, const BpIO& io, cudaStream_t st)
{
    if (io.count <= 0) return;
    const bool track_best = p.route_failures_to_osd && io.osd_llr != nullptr;
    if (!io.work_zeroed) check_cuda(cudaMemsetAsync(io.work_counter, 0, sizeof(int), st), "reset work counter");
    const auto go = [&](auto damp) {
        constexpr bool kDamp = decltype(damp)::value;
        if (cv.num_layers == 4 && cv.maxdeg <= 6) launch_shape<6, 4, kDamp>(cv, p, io, track_best, st);
        else if (cv.num_layers == 4) launch_shape<14, 4, kDamp>(cv, p, io, track_best, st);
        else if (cv.num_layers == 5) launch_shape<14, 5, kDamp>(cv, p, io, track_best, st);
        else launch_shape<10, 8, kDamp>(cv, p, io, track_best, st);
    };
    if (p.damping == 0.0f) go(std::false_type());
    else go(std::true_type());
}

}  // namespace sicc
