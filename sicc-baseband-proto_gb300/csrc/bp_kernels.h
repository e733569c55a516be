// Launch interface of the belief-propagation and OSD kernels.
#pragma once

#include "sicc_common.h"

namespace sicc {

constexpr int kBpThreads = 256;

// Launch shape of the persistent layered kernel; zero fields take defaults.
// Slot stride (floats) of codewords that share a warp, G lanes each: groups sit
// max(G, 4) banks apart, so their simultaneous gathers of the same table column
// do not collide, and every slot stays 16-byte aligned for the float4 copies of
// the posteriors (`floats` is a multiple of 4 on entry).
inline int pad_slot_stride(int floats, int group)
{
    if (group >= 32) return floats;
    const int bank = group < 4 ? 4 : group;
    return floats + ((bank - floats % 32) + 32) % 32;
}

struct BpLaunch {
    int slots_per_cta = 0;    // codewords resident per CTA (multiple of 32/group)
    int ctas = 0;             // grid size (persistent CTAs)
    int osd_share_rounds = 0; // warp OSD: candidate passes between best-metric exchanges (0 = 1)
    int osd_ctas = 0;         // warp OSD grid size (0 = occupancy x SMs)
};

// All launchers are asynchronous on `st`; io.work_counter must point at one
// device int (reset by the launcher).
void launch_bp_layered(const LayeredView& cv, const BpParams& p, const BpIO& io, const BpLaunch& shape,
                       cudaStream_t st);
void launch_bp_flooding(const FloodView& cv, const BpParams& p, const BpIO& io, cudaStream_t st);
// Register-resident messages (bp_reg.cuh).  reg_plan sets cv.reg_* for a code with layers of
// `narrowest` to `widest` rows: `group` lanes per codeword if positive, else the smallest power of
// two covering the widest layer, up to 128; reg_group stays 0 when the code fits no compiled
// shape.  The flooding launcher takes plain codes only.  The layered one expects
// io.work_counter reset.
void reg_plan(LayeredView& cv, int widest, int narrowest, int group);
void launch_bp_layered_reg(const LayeredView& cv, const BpParams& p, const BpIO& io, const BpLaunch& shape,
                           bool track_best, cudaStream_t st);
int layered_reg_default_slots(const LayeredView& cv, bool track_best);  // codewords per CTA, the most it runs
void launch_bp_flooding_reg(const LayeredView& cv, const BpParams& p, const BpIO& io, cudaStream_t st);
size_t layered_smem_bytes(const LayeredView& cv, int slots, bool track_best, int* slot_floats_out);
int layered_default_slots(const LayeredView& cv, bool track_best);
size_t flooding_smem_bytes(const FloodView& cv, int warps, int* slot_floats_out);

// Long codes whose state does not fit one CTA's shared memory (bp_wide.cu): one CTA per
// codeword, state in an L2-sized global scratch block.  launch_bp_layered /
// launch_bp_flooding hand such codes to these.
bool layered_needs_wide(const LayeredView& cv, bool track_best);
int wide_split(int n);          // posteriors the layered wide kernel keeps in shared memory
int wide_slots(int maxdeg);     // edge slots of its row table
bool flooding_needs_wide(const FloodView& cv);
void launch_bp_layered_wide(const LayeredView& cv, const BpParams& p, const BpIO& io, cudaStream_t st);
void launch_bp_flooding_wide(const FloodView& cv, const BpParams& p, const BpIO& io, cudaStream_t st);

// OSD over a device work list; `warps_per_cta`/`ctas` <= 0 take defaults.
void launch_osd(const OsdView& ov, const OsdIO& io, int max_items, cudaStream_t st, int warps_per_cta = 0,
                int ctas = 0);

// OSD of long codes, one CTA per codeword (io.hviews for mixed batches, else
// `hv`); nmax/mmax/poolmax bound the codes of the launch.
// Launch bounds of the large-code OSD over a set of codes.
struct OsdHBounds {
    int nmax = 0, mmax = 0, poolmax = 0;
    void add(int n, int m, int pool);
    bool empty() const { return nmax == 0; }
};
// The large-code OSD runs in classes by m, each with the shared memory its longest code needs, so that
// up to m = 640 two CTAs of 320 threads share an SM (a round's serial pivot choice leaves issue slots
// that only another CTA fills); above, T fills the SM's shared memory and a CTA has 512 threads.
constexpr int kOsdHClasses = 4;
constexpr int kOsdHClassMaxM[kOsdHClasses] = {256, 512, 640, 1024};
inline int osd_h_class(int m) { return m <= 256 ? 0 : m <= 512 ? 1 : m <= 640 ? 2 : 3; }
// Large-code OSD over the items of io, one launch per class present in cls[kOsdHClasses]; with more
// than one class and side streams given (kOsdHClasses - 1 of them, and as many join events), the
// classes run side by side, forked from `st` and joined back to it.
void launch_osd_h(const OsdHBounds* cls, const OsdIO& io, int max_items, cudaStream_t st,
                  const cudaStream_t* side = nullptr, cudaEvent_t fork = nullptr, const cudaEvent_t* join = nullptr);
size_t osd_h_smem_bytes(int nmax, int mmax, int poolmax);

}  // namespace sicc
