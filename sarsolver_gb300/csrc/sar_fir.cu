// sar_fir.cu -- range-profile upsampling and downsampling through a twice-oversampled transform and a
// short interpolation filter (K1 / K4 for even upsampling factors U = M / N >= 4).
//
// The upsampled profile p(b) = sum_k X_k e^{2 pi i k b / M}, k in [-N/2, N/2), is a band-limited
// function sampled U times finer than its band needs.  Instead of U transforms of N points, the
// kernels form it at twice the band (the base grid, 2 N points, H = U / 2 fine bins apart),
//     z(g) = sum_k (X_k / c(k)) e^{2 pi i k g / (2 N)},
// and interpolate: p(g H + q) = sum_{t < 10} psi(q / H + 4 - t) z(g - 4 + t), with the Kaiser-Bessel
// window psi of width 10 and its Fourier transform c(k) divided out of the spectrum beforehand.  With
// the grid oversampled twice, what such a window passes of the images of the band is 7e-10 of the
// signal (2-norm, measured against the 64-bit transform for N = 251 and 2048, U = 8 and 128; width 8
// passes 7e-8), below the FP32 rounding of the transform and of the ten-term sum (9e-8).  The taps
// depend on q only: a table of H x 10 reals made in FP64.
//
// Only the base samples around the stored span are filtered: per row 2 N-point transforms and 20 FMAs
// per stored bin, whatever U, against U N-point transforms (5 U N log2 N operations).  What is left
// is memory traffic: the row of N samples and the span of Lg bins.  The forward projection uses the
// transpose: the accumulated bins are folded onto the base grid with the same taps, then transformed
// and divided by c(k).
//
// N = 512 ... 8192: one kernel per direction (fir_up_kernel / fir_down_kernel, a CTA per pulse row; up
// to N = 2048 the even and the odd base samples are transformed by two groups of N / 16 threads side
// by side).  Other lengths: cuFFT of length 2 N between the packing kernels (sar_kernels.cu) and the
// filters alone (fir_rows_kernel / fir_fold_kernel).
//
// Measured (GB300, pulses x samples, up / down, against the U-transform kernels or cuFFT of length M
// before): 4096 x 4096, U = 8: 136 / 182 us (462 / 536); 2048 x 2048, U = 8: 43 / 53 us; 1024 x 2048, U = 128:
// 78 / 153 us (down 1059); 1024 x 1024, U = 128: 42 / 84 us (409 / 569); 1500 x 2000 (cuFFT), U = 128: 164 / 238 us in
// three kernels (up 3800 with transforms of length 256000).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "sar_fir.cuh"
#include "sar_kernels.cuh"
#include "sar_stockham.cuh"

namespace sar {

namespace {

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
// 8-byte asynchronous copy global -> shared, zero where !in (nothing is read then).
__device__ __forceinline__ void copy8(float2* dst, const float2* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ float2 conj_of(float2 a) { return make_float2(a.x, -a.y); }
// Complex64 rows are filtered in FP32, complex128 rows in FP64.
template <class R>
using Cplx = typename std::conditional<std::is_same<R, double>::value, double2, float2>::type;
__device__ __forceinline__ float2 mad(float h, float2 z, float2 s) { return __ffma2_rn(dup(h), z, s); }
__device__ __forceinline__ double2 mad(double h, double2 z, double2 s) { return make_double2(fma(h, z.x, s.x), fma(h, z.y, s.y)); }
__device__ __forceinline__ float2 wide(float2 v, float) { return v; }
__device__ __forceinline__ double2 wide(float2 v, double) { return make_double2(v.x, v.y); }
template <class T>
__device__ __forceinline__ T times(T c, float2 f) {
    return T{c.x * f.x - c.y * f.y, c.x * f.y + c.y * f.x};
}

// Transforms of a row side by side: two up to N = 2048, which halves a row's chain of passes; from 4096
// on one after the other, so that two CTAs share an SM and one's loads overlap the other's passes
// (4096 rows of 4096, U = 8, when chosen: upsampling 144 against 189 us, downsampling 172 against 340 us).
constexpr int fir_groups(int N) { return N <= 2048 ? 2 : 1; }

template <int N>
struct FirShape {
    static constexpr int T = N / 16;              // threads of one N-point transform
    static constexpr int G = fir_groups(N);       // transforms side by side
    static constexpr int NT = G * T;
    static constexpr int CTAS = NT >= 512 ? 1 : 512 / NT;   // 128 registers per thread
    static constexpr int BUF = up_pad_count(N);   // one transform buffer (float2)
};

// Filtered bins of groups [gbeg, gend) (group g: fine bins g H + q - w0 of the stored row) from base
// samples z (z[g + t] is tap t of group g).  A thread keeps the taps of one phase q and walks
// consecutive groups with the ten (linear pairs: eleven) samples in registers: one shared-memory
// load and 10 (22) packed FMAs per bin.  Consecutive threads take consecutive phases, so loads are
// broadcast and the stores of a warp contiguous for H >= 32.
template <bool PAIRS, class R>
__device__ __forceinline__ void fir_walk(const Cplx<R>* z, const R* __restrict__ taps, int H, int gbeg, int gend,
                                         int w0, int Lg, int format, float4* dst, float2* vdst, int tid, int nt) {
    constexpr int W = PAIRS ? kFirTaps + 1 : kFirTaps;
    const int ch = max(1, nt / H), len = (gend - gbeg + ch - 1) / ch;
    for (int item = tid; item < H * ch; item += nt) {
        const int q = item % H, c = item / H;
        const int a = gbeg + c * len, b = min(gend, a + len);
        if (a >= b) continue;
        const R* row = taps + (size_t)q * (PAIRS ? 2 * kFirRow : kFirRow);
        R h[W], d[W];
#pragma unroll
        for (int t = 0; t < W; ++t) {
            h[t] = __ldg(row + t);
            d[t] = PAIRS ? __ldg(row + kFirRow + t) : R(0);
        }
        Cplx<R> zw[W];
#pragma unroll
        for (int t = 0; t < W - 1; ++t) zw[t] = z[a + t];
        for (int g = a; g < b; g += W) {
#pragma unroll
            for (int j = 0; j < W; ++j) {
                if (g + j >= b) break;
                zw[(j + W - 1) % W] = z[g + j + W - 1];
                Cplx<R> s{0, 0}, e{0, 0};
#pragma unroll
                for (int t = 0; t < W; ++t) {
                    s = mad(h[t], zw[(j + t) % W], s);
                    if (PAIRS) e = mad(d[t], zw[(j + t) % W], e);
                }
                const int w = (g + j) * H + q - w0;
                if (w < 0 || w >= Lg) continue;
                if (PAIRS)
                    dst[w] = make_float4((float)s.x, (float)s.y, (float)e.x, (float)e.y);
                else if (format == kProfValues)
                    vdst[w] = make_float2((float)s.x, (float)s.y);
                else
                    dst[w] = make_float4((float)s.x, (float)s.y, 0.f, 0.f);
            }
        }
    }
}

template <class R>
__device__ __forceinline__ void fir_write(const Cplx<R>* z, const R* taps, const R* pair_taps, const FirArgs& a, int gbeg,
                                          int gend, long row, int tid, int nt) {
    float4* dst = reinterpret_cast<float4*>(a.prof) + row * a.Lg;
    float2* vdst = reinterpret_cast<float2*>(a.prof) + row * a.Lg;
    if (a.format == kProfLinearPairs)
        fir_walk<true, R>(z, pair_taps, a.H, gbeg, gend, a.w0, a.Lg, a.format, dst, vdst, tid, nt);
    else
        fir_walk<false, R>(z, taps, a.H, gbeg, gend, a.w0, a.Lg, a.format, dst, vdst, tid, nt);
}

// Index of fine value e of a staged fold chunk: PS slots of padding per four groups, so that the
// lanes of a half-warp (16 / PS base samples four groups apart, PS phases each) fall on distinct banks.
__device__ __forceinline__ int fold_pad(int e, int H, int hshift, int PS) {
    return e + (hshift >= 0 ? e >> (hshift + 2) : e / (4 * H)) * PS;
}

// The ten taps of a phase: FP32 from shared memory, FP64 (whose sums take far longer than the loads) from the table.
__device__ __forceinline__ void tap_row(const float4* taps, int p, float (&h)[kFirTaps]) {
    const float4 *hr = taps + p * (kFirRow / 4), h0 = hr[0], h1 = hr[1], h2 = hr[2];
    const float v[kFirTaps] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w, h2.x, h2.y};
#pragma unroll
    for (int t = 0; t < kFirTaps; ++t) h[t] = v[t];
}
__device__ __forceinline__ void tap_row(const double* taps, int p, double (&h)[kFirTaps]) {
#pragma unroll
    for (int t = 0; t < kFirTaps; ++t) h[t] = __ldg(taps + (size_t)p * kFirRow + t);
}

// The tap table into shared memory (the caller's next barrier publishes it).
__device__ __forceinline__ void load_taps(float4* taps, const FirArgs& a, int tid, int nt) {
    for (int i = tid; i < a.H * (kFirRow / 4); i += nt) taps[i] = __ldg(reinterpret_cast<const float4*>(a.taps) + i);
}

// Base samples i0 .. i0 + gc - 1 (gc a multiple of 4; sample i is base point gb0 - 4 + i) folded from
// the fine bins of one accumulator row: z(i) = sum_{t, q} h_q(t) acc(group i - t, bin q).  A thread
// owns four consecutive samples and every PS-th phase: 13 loads feed 40 packed FMAs, and the PS
// partial sums are added with shuffles.  `buf` holds the chunk's bins, `taps` the tap table (FP32: shared
// memory, where eight rows of 48 bytes fall on distinct banks); every thread of the CTA calls.
template <class R, class TAPS, class STORE>
__device__ __forceinline__ void fir_fold(const float2* __restrict__ arow, float2* buf, TAPS taps, const FirArgs& a,
                                         int i0, int gc, int tid, int nt, STORE store) {
    const int H = a.H, PS = a.fold_phases;
    const int first = (i0 - (kFirTaps - 1)) * H - a.w0, count = (gc + kFirTaps - 1) * H;
    for (int e = tid; e < count; e += nt) {
        const int w = first + e;
        const bool in = w >= 0 && w < a.Lg;
        copy8(buf + fold_pad(e, H, a.hshift, PS), arow + (in ? w : 0), in);
    }
    copies_done();
    __syncthreads();
    const int items = (gc / 4) * PS, stride = 4 * H + PS;
    for (int item = tid; item < ((items + 31) & ~31); item += nt) {
        const bool live = item < items;
        const int sb = live ? item / PS : 0, q = item & (PS - 1);
        Cplx<R> o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = Cplx<R>{0, 0};
        if (live)
            for (int p = q; p < H; p += PS) {
                R h[kFirTaps];
                tap_row(taps, p, h);
                const float2* b = buf + sb * stride + p;
#pragma unroll
                for (int gg = 0; gg < kFirTaps + 3; ++gg) {
                    const Cplx<R> v = wide(b[gg * H + (gg >> 2) * PS], R(0));
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int t = k + kFirTaps - 1 - gg;
                        if (t >= 0 && t < kFirTaps) o[k] = mad(h[t], v, o[k]);
                    }
                }
            }
        for (int s = 1; s < PS; s *= 2)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                o[k].x += __shfl_xor_sync(0xffffffffu, o[k].x, s);
                o[k].y += __shfl_xor_sync(0xffffffffu, o[k].y, s);
            }
        if (live && q == 0)
#pragma unroll
            for (int k = 0; k < 4; ++k) store(i0 + 4 * sb + k, o[k]);
    }
}

}  // namespace

// K1, N = 512 ... 8192: phase-history row -> stored span.  Bound: shared-memory latency of the two
// transforms' passes (three or four with a barrier each); the span's stores are next.
template <int N>
__global__ void __launch_bounds__(FirShape<N>::NT, FirShape<N>::CTAS) fir_up_kernel(const FirArgs a) {
    using Sh = FirShape<N>;
    constexpr int T = Sh::T, G = Sh::G, NT = Sh::NT;
    extern __shared__ __align__(16) float2 fsm[];
    const int tid = threadIdx.x, t = tid % T, grp = tid / T;
    float2* A = fsm + grp * 2 * Sh::BUF;
    float2* B = A + Sh::BUF;
    float2* stage = fsm + G * 2 * Sh::BUF;
    const long s = (long)a.first + blockIdx.x;
    const float2 f = a.wfac ? __ldg(a.wfac + s) : make_float2(1.f, 0.f);
    const float2* yr = a.y + s * N;
    // conj(W) y / c, read once per row (the row may be host memory read over the link)
#pragma unroll
    for (int e = 0; e < N / NT; ++e) {
        const int kp = tid + NT * e;
        const float2 yv = yr[(kp + N / 2) & (N - 1)];
        const float2 w = __ldg(a.wave + kp);
        fsm[up_pad(kp)] = make_float2(w.x * yv.x + w.y * yv.y, w.x * yv.y - w.y * yv.x);
    }
    __syncthreads();
    float2 X[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) X[e] = fsm[up_pad(t + T * e)];
    __syncthreads();
#pragma unroll
    for (int pass = 0; pass < 2 / G; ++pass) {
        const int r = G == 2 ? grp : pass;   // base samples 2 j + r
        float2 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = r ? cmulf(X[e], __ldg(a.half + t + T * e)) : X[e];
        up_first_pass<N>(v, A, t);
        __syncthreads();
        const float2* F = up_passes<N, false>(A, B, a.tw_n, t);
        for (int i = ((r ^ a.base0) & 1) + 2 * t; i < a.stage_len; i += 2 * T) {
            const float2 c = F[up_pad(((a.base0 + i) & (2 * N - 1)) >> 1)];
            stage[i] = make_float2(c.x * f.x - c.y * f.y, c.x * f.y + c.y * f.x);
        }
        __syncthreads();
    }
    fir_write<float>(stage, a.taps, a.pair_taps, a, 0, a.groups, s, tid, NT);
}

// K4, N = 512 ... 8192: accumulator row -> phase-history row, the transpose of fir_up_kernel.
template <int N>
__global__ void __launch_bounds__(FirShape<N>::NT, FirShape<N>::CTAS) fir_down_kernel(const FirArgs a) {
    using Sh = FirShape<N>;
    constexpr int T = Sh::T, G = Sh::G, NT = Sh::NT;
    extern __shared__ __align__(16) float2 fsm[];
    const int tid = threadIdx.x, t = tid % T, grp = tid / T;
    float2* A = fsm + grp * 2 * Sh::BUF;
    float2* B = A + Sh::BUF;
    float2* z = fsm + a.fold_buf;
    const long s = (long)a.first + blockIdx.x;
    const float2* arow = a.acc + s * a.Lg;
    const int nb = a.groups + kFirTaps - 1;
    float4* taps = reinterpret_cast<float4*>(z + ((nb + 3) & ~3));
    load_taps(taps, a, tid, NT);
    for (int i0 = 0; i0 < nb; i0 += a.fold_chunk) {
        const int gc = min(a.fold_chunk, (nb - i0 + 3) & ~3);
        fir_fold<float>(arow, fsm, taps, a, i0, gc, tid, NT, [&](int i, float2 v) { z[i] = v; });
        __syncthreads();
    }
    float2 acc[16];
#pragma unroll
    for (int pass = 0; pass < 2 / G; ++pass) {
        const int r = G == 2 ? grp : pass;
        float2 v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {   // conj of base sample 2 j + r
            const int i = (2 * (t + T * e) + r - a.base0) & (2 * N - 1);
            v[e] = i < nb ? conj_of(z[i]) : make_float2(0.f, 0.f);
        }
        up_first_pass<N>(v, B, t);
        __syncthreads();
        float2* F = up_passes<N, true>(B, A, a.tw_n, t);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const float2 c = F[up_pad(t + T * e)];
            const float2 m = r ? cmulf(c, __ldg(a.half + t + T * e)) : c;
            if (G == 2) {
                if (r) F[up_pad(t + T * e)] = m;
            } else {
                acc[e] = pass ? make_float2(acc[e].x + m.x, acc[e].y + m.y) : m;
            }
        }
        __syncthreads();
    }
    const float2 f = __ldg(a.wfac + s);
    // the transform's buffer: B after two radix-16 passes, A after three
    const float2* F0 = fsm + (UpShape<N>::P == 3 ? 0 : Sh::BUF);
#pragma unroll
    for (int e = 0; e < N / NT; ++e) {
        const int i = tid + NT * e;
        float2 k;
        if (G == 2) {
            const float2 u = F0[up_pad(i)], v = F0[2 * Sh::BUF + up_pad(i)];
            k = make_float2(u.x + v.x, -(u.y + v.y));
        } else {
            k = conj_of(acc[e]);
        }
        const float2 w = __ldg(a.wave + i);
        const float2 m = make_float2(w.x * k.x - w.y * k.y, w.x * k.y + w.y * k.x);
        a.y_out[s * N + ((i + N / 2) & (N - 1))] = make_float2(m.x * f.x - m.y * f.y, m.x * f.y + m.y * f.x);
    }
}

constexpr int kFirThreads = 256;

// Any N: the filter from transformed rows spec[row][2 N] (float2, or double2) to the stored span; grid
// (chunks of groups, rows).  The FP64 form, taken where the transform itself is complex128, is bound by the FP64 pipe
// (two operations a cycle and SM): 1500 x 1999, U = 128, 51860 bins a row: 5.8 ms up and 7.5 ms down with the
// transforms, of which FP64 filters 2.8 and 4.5; transforms of length M took 293 ms.
template <class T>
__global__ void __launch_bounds__(kFirThreads) fir_rows_kernel(const T* __restrict__ spec, const FirArgs a, int chunk) {
    extern __shared__ __align__(16) unsigned char rsm[];
    T* zs = reinterpret_cast<T*>(rsm);
    const long s = (long)a.first + blockIdx.y;
    const int g0 = blockIdx.x * chunk, g1 = min(a.groups, g0 + chunk);
    const float2 f = a.wfac ? __ldg(a.wfac + s) : make_float2(1.f, 0.f);
    const T* row = spec + (size_t)blockIdx.y * a.base_len;
    for (int i = threadIdx.x; i < g1 - g0 + kFirTaps; i += kFirThreads) {
        int n = a.base0 + g0 + i;
        if (n >= a.base_len) n -= a.base_len;
        zs[i] = times(row[n], f);
    }
    __syncthreads();
    if constexpr (std::is_same<T, double2>::value)
        fir_write<double>(zs - g0, a.taps64, a.pair_taps64, a, g0, g1, s, threadIdx.x, kFirThreads);
    else
        fir_write<float>(zs - g0, a.taps, a.pair_taps, a, g0, g1, s, threadIdx.x, kFirThreads);
}

// Any N: the fold of an accumulator row onto rows spec[row][2 N], zero outside the span.
template <class T>
__global__ void __launch_bounds__(kFirThreads) fir_fold_kernel(T* __restrict__ spec, const FirArgs a) {
    extern __shared__ __align__(16) float2 fsm[];
    const long s = (long)a.first + blockIdx.y;
    const int nb = a.groups + kFirTaps - 1, i0 = blockIdx.x * a.fold_chunk;
    T* row = spec + (size_t)blockIdx.y * a.base_len;
    auto put = [&](int i, T v) {
        if (i >= a.base_len) return;
        int n = a.base0 + i;
        if (n >= a.base_len) n -= a.base_len;
        row[n] = v;
    };
    if (i0 < nb) {
        if constexpr (std::is_same<T, double2>::value) {
            fir_fold<double>(a.acc + s * a.Lg, fsm, a.taps64, a, i0, a.fold_chunk, threadIdx.x, kFirThreads, put);
        } else {
            float4* taps = reinterpret_cast<float4*>(fsm + a.fold_buf);
            load_taps(taps, a, threadIdx.x, kFirThreads);
            fir_fold<float>(a.acc + s * a.Lg, fsm, taps, a, i0, a.fold_chunk, threadIdx.x, kFirThreads, put);
        }
        return;
    }
    for (int i = i0 + threadIdx.x; i < i0 + a.fold_chunk; i += kFirThreads) put(i, T{0, 0});
}

// ------------------------------------------------------------------ host side
namespace {

constexpr size_t kFirSmem = 220 * 1024;
constexpr size_t kFirFoldBytes = 32 * 1024;   // fold buffer where the transform buffers are smaller

double bessel_i0(double x) {   // power series sum (x^2 / 4)^m / (m!)^2
    double term = 1.0, sum = 1.0;
    for (int m = 1; term > 1e-18 * sum; ++m) {
        term *= 0.25 * x * x / ((double)m * m);
        sum += term;
    }
    return sum;
}

size_t fold_values(int gc, int H, int PS) {
    const size_t n = (size_t)(gc + kFirTaps - 1) * H;
    return n + (n / (4 * (size_t)H) + 1) * PS;
}

size_t transform_values(int N) { return (size_t)(2 * fir_groups(N)) * (size_t)(N + N / 16); }

// Largest fold chunk (multiple of 4 base samples) whose bins fit `values` float2; 0 if none.
int fold_chunk_for(size_t values, int H, int PS, int most) {
    int gc = most & ~3;
    while (gc >= 4 && fold_values(gc, H, PS) > values) gc = gc > 64 ? (gc / 2) & ~3 : gc - 4;
    return gc >= 4 ? gc : 0;
}

}  // namespace

bool fir_plan(long N, long M, int Lg, long bg0, FirLayout* L) {
    if (N < 1 || M % N || N > (1 << 24)) return false;
    const long U = M / N;
    // odd factors have no whole number of bins per base step; at U = 2 the base grid is the fine one
    if (U < 4 || (U & 1) || U / 2 > 4096 || Lg < 1) return false;
    const int H = (int)(U / 2);
    auto floor_div = [](long a, long b) { return a >= 0 ? a / b : -((-a + b - 1) / b); };
    const long gb0 = floor_div(bg0, H), gl = floor_div(bg0 + Lg - 1, H);
    const long groups = gl - gb0 + 1;
    if (groups + kFirTaps + 1 > 2 * N) return false;   // the span wraps around the base grid
    L->H = H;
    L->groups = (int)groups;
    L->w0 = (int)(bg0 - gb0 * H);
    L->base_len = (int)(2 * N);
    L->base0 = (int)(((gb0 - 4) % (2 * N) + 2 * N) % (2 * N));
    L->stage_len = (int)groups + kFirTaps;   // linear pairs read one base sample more
    L->hshift = -1;
    for (int b = 0; b < 13; ++b)
        if (H == (1 << b)) L->hshift = b;
    L->fold_phases = 1;
    while (L->fold_phases < 8 && H % (2 * L->fold_phases) == 0) L->fold_phases *= 2;
    L->fused = false;
    const int nb = ((int)groups + kFirTaps - 1 + 3) & ~3;
    if (fused_fft_length((int)N)) {
        const size_t tv = transform_values((int)N);
        const size_t fold = (std::max(tv, kFirFoldBytes / sizeof(float2)) + 1) & ~(size_t)1;
        const int gc = fold_chunk_for(fold, H, L->fold_phases, nb);
        const size_t up = (tv + L->stage_len) * sizeof(float2);
        const size_t down = (fold + nb) * sizeof(float2) + (size_t)H * kFirRow * sizeof(float);
        if (gc && up <= kFirSmem && down <= kFirSmem) {
            L->fused = true;
            L->fold_chunk = gc;
            L->fold_buf = (int)fold;
            L->up_smem = up;
            L->down_smem = down;
            return true;
        }
    }
    const int gc = fold_chunk_for(kFirFoldBytes / sizeof(float2), H, L->fold_phases, std::max(64, (4096 / H) & ~3));
    if (!gc) return false;
    L->fold_chunk = gc;
    L->fold_buf = (int)((fold_values(gc, H, L->fold_phases) + 1) & ~(size_t)1);
    L->up_smem = 0;
    L->down_smem = (size_t)L->fold_buf * sizeof(float2) + (size_t)H * kFirRow * sizeof(float);
    return true;
}

void fir_tables(const FirLayout& L, std::vector<double>* taps, std::vector<double>* pair_taps, std::vector<double>* inv_c) {
    const int W = kFirTaps, H = L.H;
    const double pi = 3.14159265358979323846;
    // Kaiser-Bessel window of width W on a grid oversampled twice: Jackson et al., IEEE Trans. Med. Imaging 10 (1991), its
    // shape parameter by Beatty, Nishimura and Pauly, ibid. 24 (2005), beta = pi sqrt((W / a)^2 (a - 1/2)^2 - 0.8), a = 2
    const double beta = pi * std::sqrt(0.5625 * W * W - 0.8), i0b = bessel_i0(beta);
    auto psi = [&](double x) {
        const double u = 2.0 * x / W;
        return u * u < 1.0 ? bessel_i0(beta * std::sqrt(1.0 - u * u)) / i0b : 0.0;
    };
    std::vector<double> h((size_t)(H + 1) * (W + 1), 0.0);   // [q][t]; q = H is phase 0 one sample on
    for (int q = 0; q <= H; ++q)
        for (int t = 0; t <= W; ++t) h[(size_t)q * (W + 1) + t] = psi((double)q / H + 4.0 - t);
    taps->assign((size_t)H * kFirRow, 0.0);
    pair_taps->assign((size_t)H * 2 * kFirRow, 0.0);
    for (int q = 0; q < H; ++q)
        for (int t = 0; t <= W; ++t) {
            const double a = h[(size_t)q * (W + 1) + t], b = h[(size_t)(q + 1) * (W + 1) + t];
            if (t < W) (*taps)[(size_t)q * kFirRow + t] = a;
            (*pair_taps)[(size_t)(2 * q) * kFirRow + t] = 0.5 * (a + b);
            (*pair_taps)[(size_t)(2 * q + 1) * kFirRow + t] = b - a;
        }
    // 1 / c(k) at FFT index i of N: the window's Fourier transform at k / (2 N) cycles per base sample
    const int N = L.base_len / 2;
    inv_c->resize(N);
    for (int i = 0; i < N; ++i) {
        const int k = i < N - N / 2 ? i : i - N;
        const double x = pi * W * (double)k / (2.0 * N), r = std::sqrt(beta * beta - x * x);
        (*inv_c)[i] = i0b * r / (W * std::sinh(r));
    }
}

template <int N>
static cudaError_t launch_fir_t(const FirArgs& a, const FirLayout& L, int rows, bool up, cudaStream_t st) {
    auto go = [&](auto kern, size_t smem) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<rows, FirShape<N>::NT, smem, st>>>(a);
        return cudaGetLastError();
    };
    return up ? go(fir_up_kernel<N>, L.up_smem) : go(fir_down_kernel<N>, L.down_smem);
}

static FirArgs with_layout(FirArgs a, const FirLayout& L) {
    a.H = L.H;
    a.groups = L.groups;
    a.w0 = L.w0;
    a.base_len = L.base_len;
    a.base0 = L.base0;
    a.stage_len = L.stage_len;
    a.hshift = L.hshift;
    a.fold_phases = L.fold_phases;
    a.fold_chunk = L.fold_chunk;
    a.fold_buf = L.fold_buf;
    return a;
}

cudaError_t launch_fir_fused(const FirArgs& args, const FirLayout& L, int rows, bool up, cudaStream_t st) {
    if (!L.fused || rows < 1) return cudaErrorInvalidValue;
    const FirArgs a = with_layout(args, L);
    switch (L.base_len / 2) {
        case 512: return launch_fir_t<512>(a, L, rows, up, st);
        case 1024: return launch_fir_t<1024>(a, L, rows, up, st);
        case 2048: return launch_fir_t<2048>(a, L, rows, up, st);
        case 4096: return launch_fir_t<4096>(a, L, rows, up, st);
        case 8192: return launch_fir_t<8192>(a, L, rows, up, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_fir_rows(const void* spec, int dbl, const FirArgs& args, const FirLayout& L, int rows, cudaStream_t st) {
    const FirArgs a = with_layout(args, L);
    const int chunk = std::max(32, 4096 / L.H);   // groups per CTA
    const dim3 grid((unsigned)((L.groups + chunk - 1) / chunk), (unsigned)rows);
    const size_t smem = (size_t)(chunk + kFirTaps + 1) * (dbl ? sizeof(double2) : sizeof(float2));
    if (dbl)
        fir_rows_kernel<<<grid, kFirThreads, smem, st>>>((const double2*)spec, a, chunk);
    else
        fir_rows_kernel<<<grid, kFirThreads, smem, st>>>((const float2*)spec, a, chunk);
    return cudaGetLastError();
}

cudaError_t launch_fir_fold(void* spec, int dbl, const FirArgs& args, const FirLayout& L, int rows, cudaStream_t st) {
    const FirArgs a = with_layout(args, L);
    const dim3 grid((unsigned)((L.base_len + L.fold_chunk - 1) / L.fold_chunk), (unsigned)rows);
    if (dbl)
        fir_fold_kernel<<<grid, kFirThreads, L.down_smem, st>>>((double2*)spec, a);
    else
        fir_fold_kernel<<<grid, kFirThreads, L.down_smem, st>>>((float2*)spec, a);
    return cudaGetLastError();
}

}  // namespace sar
