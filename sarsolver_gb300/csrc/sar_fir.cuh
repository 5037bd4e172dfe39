// sar_fir.cuh -- range-profile upsampling / downsampling by a twice-oversampled transform and a short
// filter (sar_fir.cu): layout, tables and launches.
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace sar {

constexpr int kFirTaps = 10;   // width of the interpolation window, base samples
constexpr int kFirRow = 12;    // floats per row of a tap table

// How a stored span [bg0, bg0 + Lg) of a length-M = U N profile lies on its base grid of 2 N points.
struct FirLayout {
    int H = 0;            // fine bins per base step, U / 2
    int groups = 0;       // base steps the span covers
    int w0 = 0;           // bins of the first base step before the span
    int base_len = 0;     // 2 N
    int base0 = 0;        // base point of the first tap of the first step, mod 2 N
    int stage_len = 0;    // base samples the filter reads
    int hshift = -1;      // log2 H, -1 when H is not a power of two
    int fold_phases = 1;  // phases the fold spreads over neighbouring lanes (power of two, divides H)
    int fold_chunk = 0;   // base samples folded at a time
    int fold_buf = 0;     // fused fold: float2 before the folded samples
    bool fused = false;   // one kernel per direction (N = 512 ... 8192)
    size_t up_smem = 0, down_smem = 0;
};

struct FirArgs {
    const float2* y = nullptr;      // [S][N] phase history, fast time fftshifted (upsampling)
    float2* y_out = nullptr;        // the same (downsampling)
    const float2* wave = nullptr;   // [N] waveform / c(k), FFT order
    const float2* half = nullptr;   // [N] e^{2 pi i k / (2 N)}, FFT order (signed k)
    const float2* tw_n = nullptr;   // [N] e^{2 pi i q / N}
    const float2* wfac = nullptr;   // [S] pulse factors; null: 1 (upsampling)
    const float* taps = nullptr;        // [H][kFirRow]
    const float* pair_taps = nullptr;   // [H][2][kFirRow]: mid-bin value, difference to the next bin
    const double* taps64 = nullptr;     // the same in 64 bits (complex128 rows)
    const double* pair_taps64 = nullptr;
    const float2* acc = nullptr;    // [S][Lg] accumulator (downsampling)
    void* prof = nullptr;           // [S][Lg] profiles in `format` (upsampling)
    int Lg = 0, first = 0, format = 0;   // row of the launch's first CTA; kProf... format
    // copied from the layout by the launchers
    int H = 0, groups = 0, w0 = 0, base_len = 0, base0 = 0, stage_len = 0, hshift = -1, fold_phases = 1, fold_chunk = 0,
        fold_buf = 0;
};

__host__ __device__ constexpr int up_pad_count(int n) { return n + n / 16; }

// Whether (and how) the span goes through the base grid: M an even multiple >= 4 of N, and the span
// shorter than the grid.
bool fir_plan(long N, long M, int Lg, long bg0, FirLayout* L);
// FP64-made tables: taps, pair taps and 1 / c(k) in FFT order.
void fir_tables(const FirLayout& L, std::vector<double>* taps, std::vector<double>* pair_taps, std::vector<double>* inv_c);
// Fused kernels for `rows` pulses from args.first (rows addressed absolutely, as sar_kernels.cuh's).
cudaError_t launch_fir_fused(const FirArgs& a, const FirLayout& L, int rows, bool up, cudaStream_t st);
// The filters alone, between transforms of length 2 N: spec rows [rows][2 N] of complex64, or of complex128, which are
// filtered in FP64 and rounded once.
cudaError_t launch_fir_rows(const void* spec, int dbl, const FirArgs& a, const FirLayout& L, int rows, cudaStream_t st);
cudaError_t launch_fir_fold(void* spec, int dbl, const FirArgs& a, const FirLayout& L, int rows, cudaStream_t st);

}  // namespace sar
