// sar_scatter.cuh -- forward scatter with a pulse per lane (sar_scatter.cu): layout and launch.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "sar_geom.cuh"
#include "sar_lattice.h"

namespace sar {

constexpr int kWalk = 16;             // pixels of a line within a block
constexpr int kScatterWarps = 4;    // warps (groups of 32 pulses) per CTA

// How a scatter walks its lattice: blocks of `lines` lines (along v) of kWalk pixels along w.
struct ScatterLayout {
    Lattice lattice;
    int lines = 16;
    int half = 0;     // bins a block reaches on either side of its anchor's bin
    int slots = 0;    // window slots per pulse
    bool ok = false;
    std::vector<int4> items;   // (a0, b0, blocks along w, plane) of each CTA's run of blocks
};

struct ScatterArgs {
    GridConst img;              // the image grid (positions)
    GridConst lat;              // the same with steps v, w (expansions)
    const PulseGeom* pulses;    // [S]
    const float2* x;            // image
    float2* acc;                // [S][Lg], pre-zeroed
    const int4* items;
    unsigned* flags;
    int num_items, S, Lg, bg0;
    int vx, vy, wx, wy, lines, half, slots;
};

// How the tile kernel would scatter the same: image steps along its lanes (v) and its walk (w), lines of 32 x 32 tiles, the
// tiles of a line, and pixels of tiles per image pixel.
struct ScatterTiles {
    Lattice axes;
    int lines = 1, along = 1;
    double cover = 1.0;
};

// Host-side choice of lattice, block and segments for linear sampling without split bins (see sar_scatter.cu); not ok
// where the tile kernel is expected to be clearly faster.
ScatterLayout scatter_layout(const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                             const double* ey, const double* ez, int nx, int ny, int nz, double s_r, double kappa,
                             const ScatterTiles& tiles);
cudaError_t launch_scatter(const ScatterArgs& a, cudaStream_t st);

}  // namespace sar
