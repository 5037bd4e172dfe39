// sar_gather.cuh -- backprojection gather along iso-range lines (sar_gather.cu): layout and launch.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "sar_kernels.cuh"
#include "sar_lattice.h"

namespace sar {

constexpr int kGatherLines = 32;   // lattice lines of a tile: a lane each
constexpr int kGatherWalk = 16;    // pixels of a line one thread keeps

// How samples find their bins: runs of pixels within three plain bins, or a bin per pixel with split bins, linear
// or nearest.
enum { GATHER_RUNS = 0, GATHER_NEAREST = 1, GATHER_LINEAR = 2 };

// Tiles of kGatherLines x (16 warps) lattice pixels (split bins: `across` warps on the lattice's first axis, the
// others on its second), the pulses of a stage and the CTAs (parts) that share a
// tile's pulses.
struct GatherLayout {
    Lattice lattice;
    int bins = GATHER_RUNS;
    int warps = 8;    // gathering warps per CTA: 8 or 4
    int across = 1;
    int ctas = 2;     // CTAs an SM holds
    int ww = 0;       // window (bins) staged per pulse
    int pb = 16;      // pulses per stage
    int parts = 1;    // CTAs per tile for all S pulses
    bool ok = false;
    std::vector<int4> tiles;   // (a0, b0, plane, 0)
};

struct GatherArgs {
    GridConst img;              // the image grid (positions)
    GridConst lat;              // the same with steps v, w (expansions)
    const PulseGeom* pulses;    // [S]
    const float2* prof;         // [S][Lg] plain values (kProfValues)
    float2* x;
    float2* partial;            // [parts][pixels], parts > 1
    const int4* tiles;
    unsigned* flags;
    const double* steps = nullptr;    // exact bins (nearest), as BpGridArgs
    const float4* alpha2 = nullptr;
    int bins = GATHER_RUNS;
    int num_tiles, S, Lg, bg0, ww, pb, warps, across, parts, accumulate;
    int vx, vy, wx, wy;
    size_t pixels;
    long long wait_budget = kDefaultWaitBudgetCycles;
    int hold_first_stage = 0;   // test aid, as BpGridArgs
};

// Layout for the sampling `bins`; not ok where the lattice or the windows do not fit.
GatherLayout gather_layout(int bins, const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                           const double* ey, const double* ez, int nx, int ny, int nz, double s_r, double kappa);
// Parts for `count` pulses (at most the layout's).
int gather_parts(const GatherLayout& L, size_t count, size_t pixels);
cudaError_t launch_gather(const GatherArgs& a, cudaStream_t st);

}  // namespace sar
