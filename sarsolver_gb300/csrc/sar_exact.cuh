// sar_exact.cuh -- exact nearest-bin decisions of the grid kernels.
#pragma once

#include "sar_pipe.cuh"

namespace sar {

// Nearest-bin sampling on the grid paths.  The FP32 bin coordinate s (about the chosen bin, in
// [-0.5, 0.5]) is within ~5e-6 bins of the FP64 position (split bins, sar_geom.cuh); where |s|
// exceeds kNearEdge the bin is decided again from the per-pixel double-float range with the
// unstructured path's exact rule (exact_bin: FP64 rounding of the same value, ties away from
// zero), so the grid kernels pick the bins the per-pixel path picks.  About 1e-4 of the
// pixel·pulses take this branch.
constexpr float kNearEdge = 0.49995f;

// Stored-span index (bins from bg0) and, with PHASE, phase (turns) of grid pixel (i, j, k) for pulse s under nearest
// rule `rule`: pixel offset from the grid origin in FP64 as the host forms it, then the double-float range and
// rounding of the per-pixel kernels (eval_point).
struct ExactSample {
    int gi;
    float f;
};
template <bool PHASE>
__device__ __noinline__ ExactSample exact_grid_sample(const double* __restrict__ steps, const PulseGeom* __restrict__ pulses,
                                                      const float4* __restrict__ alpha2, df kappa, df sr, int bg0, int rule,
                                                      int i, int j, int k, int s) {
    double q[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        q[c] = __dadd_rn(__dadd_rn(__dmul_rn((double)i, steps[c]), __dmul_rn((double)j, steps[3 + c])),
                         __dmul_rn((double)k, steps[6 + c]));
    const double qq = __dadd_rn(__dadd_rn(__dmul_rn(q[0], q[0]), __dmul_rn(q[1], q[1])), __dmul_rn(q[2], q[2]));
    PointGeom pt;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        pt.qh[c] = __double2float_rn(q[c]);
        pt.ql[c] = __double2float_rn(__dsub_rn(q[c], (double)pt.qh[c]));
    }
    pt.qh[3] = __double2float_rn(qq);
    pt.ql[3] = __double2float_rn(__dsub_rn(qq, (double)pt.qh[3]));
    const PulseGeom pg = load_pulse(pulses + s);
    const float4 a2 = __ldg(alpha2 + s);
    df r = point_range(pulse_tx(pg), df_make(a2.x, a2.y), pt);
    if (pg.monostatic != 0.0f)
        r = df_mulf(r, 2.0f);
    else
        r = df_add(r, point_range(pulse_rx(pg), df_make(a2.z, a2.w), pt));
    r = df_sub(r, df_make(pg.rref_hi, pg.rref_lo));
    const df V = df_sub(df_mul(sr, r), df_make((float)bg0, 0.0f));
    ExactSample e;
    float sf;
    exact_bin(V, bg0, rule, &e.gi, &sf);
    e.f = PHASE ? df_frac(df_mul(kappa, r)) : 0.f;
    return e;
}

// Deferred re-decisions.  A pixel-pulse near a rounding boundary is taken at its FP32 bin with the others and noted
// in a queue of its warp's; 32 notes at a time (and the rest at the end) are decided exactly, a lane each, and where
// the exact bin differs (about 2 % of the notes) the sample moves there.  Decided on the spot, one lane would go
// through the double-float range and the FP64 pipe with its warp waiting.
constexpr int kNearQueue = 64;   // notes a warp's queue holds

}  // namespace sar
