// sar_resample.cu -- dataset resampling on the GPU: SRP phase ramps, fast-frequency downsampling
// and the slow-time downsampling filter (sar_move_srps, sar_fast_freq_downsample,
// sar_resample_phase_history in include/sargpu.h).
//
// Follows the reference's utilities and resampling loop (src/sarsolver/utils/geodesy.py:33-73,
// utils/signal.py:45-77, numpy/measurement.py:342-458), restructured for the device.  The reference rephases and
// downsamples every pulse of every window and then filters; both the downsampling and the filter are linear and act
// on different axes, so here the filter comes first, fused with the rephasing, and only the output pulses are
// transformed (1 / D of the input pulses):
//   filter:    z[t][f] = sum_k kernel[k] ph[row0[t] + k][f] exp(2 pi i (dR_s / c) (bb_f - sign fc)),
//              bb_f = (f - N/2) fs / N  (phase in turns from a per-pulse constant reduced in FP64 on the host
//              plus an error-free split product for the per-bin slope, good to ~1e-7 turns at hundreds of turns;
//              a thread takes f = t + T e, e < 16: one sine / cosine per thread and pulse times sixteen
//              thread-independent factors)
//   downsample: ifftshift, inverse FFT / N, keep the n/2 lowest and n - n/2 highest modes times the fftshifted
//              Tukey window, forward FFT, fftshift -- the last as a phase ramp of the kept modes, folded into
//              the window, so the forward transform runs in place in the output
// N = 512 ... 8192 runs the filter, the inverse transform and the crop in one kernel per output pulse
// (filter_crop_kernel); other lengths filter into work rows, chunk by chunk, for cuFFT.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "../../include/sargpu.h"
#include "sar_kernels.cuh"
#include "sar_stockham.cuh"

namespace {

int err(int code, const char* msg) {
    sar::sar_internal_set_error(msg);
    return code;
}
int cuda_err(cudaError_t e, const char* what) {
    char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
    return err(e == cudaErrorMemoryAllocation ? SAR_ERR_OUT_OF_MEMORY : SAR_ERR_CUDA, buf);
}
#define R_CUDA(call, what)                                 \
    do {                                                   \
        cudaError_t _e = (call);                           \
        if (_e != cudaSuccess) return cuda_err(_e, what);  \
    } while (0)
#define R_CALL(call)          \
    do {                      \
        int _rc = (call);     \
        if (_rc) return _rc;  \
    } while (0)

unsigned blocks_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 65535u * 8); }

// out[s][j] = in[s][(j + shift_in) % N] * exp(2 pi i phase(s, f)) * scale, where f is the natural
// (fftshifted) frequency index of the value read and phase = b_s + a_s f in turns.  coef[s] =
// (b_s, a_hi_s, a_lo_s, the tail of b_s); a_hi * f is formed with its exact FMA remainder.
__global__ void rephase_kernel(const float2* __restrict__ in, float2* __restrict__ out, const float4* __restrict__ coef,
                               int S, int N, int shift_in, float scale) {
    const size_t total = (size_t)S * N;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const int s = (int)(e / N), j = (int)(e % N);
        int f = j + shift_in;
        if (f >= N) f -= N;
        const float2 v = in[(size_t)s * N + f];
        float2 r = v;
        if (coef) {
            const float4 c = __ldg(coef + s);
            const float ff = (float)f;
            const float p = c.y * ff;
            const float pe = fmaf(c.y, ff, -p);          // exact remainder of the product
            float t = (p - rintf(p)) + pe + c.z * ff + c.x;
            t -= rintf(t);
            float sn, cs;
            sincospif(2.0f * t, &sn, &cs);
            r = make_float2(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
        }
        out[e] = make_float2(r.x * scale, r.y * scale);
    }
}

// dst[s][j] = window[j] * src[s][j < lo ? j : N - (n - j)]  (modes kept by the downsampling).
__global__ void crop_window_kernel(const float2* __restrict__ src, float2* __restrict__ dst, const float2* __restrict__ window,
                                   int S, int N, int n) {
    const int lo = n / 2;
    for (int s = blockIdx.y; s < S; s += gridDim.y)
        for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
            const int k = j < lo ? j : N - (n - j);
            dst[(size_t)s * n + j] = sar::cmulf(__ldg(window + j), src[(size_t)s * N + k]);
        }
}

constexpr int kStepRows = 32;   // pulses whose step factors are formed at a time

// What the slow-time filter reads; all arrays on the device.
struct FilterArgs {
    const float2* ph;      // [S][N]
    const float4* coef;    // [S] phase coefficients, or null
    const float2* kern;    // [L]
    const int* row0;       // [T]
    const float2* window;  // [n] window times the output shift's ramp
    float2* out;
    int N, L, n;
    float scale;
};

// exp(2 pi i ((hi + lo) f + b + b_lo)).  The large terms are added without error and reduced to half a turn before the small
// ones join them, so that the phase is rounded once (to 1.5e-8 turns at most): the factors of a sample are two of these,
// multiplied, and held to the accuracy of one phase formed in plain FP32 sums.
__device__ __forceinline__ float2 unit(float hi, float lo, float f, float b, float b_lo) {
    const float p = hi * f, pe = fmaf(hi, f, -p);   // exact remainder of the product
    const float r = p - rintf(p), s = r + b, bb = s - r, e = (r - (s - bb)) + (b - bb);   // s + e = r + b
    float t = (s - rintf(s)) + (e + (pe + fmaf(lo, f, b_lo)));
    t -= rintf(t);
    float2 v;
    sincospif(2.0f * t, &v.y, &v.x);
    return v;
}

// acc[e] = sum_k kern[k] phase ph[first + k][t + T e] for the sixteen bins of thread t (bins >= N are left zero).
// `steps` holds the pulses' factors exp(2 pi i a_s T e); every thread of the CTA calls.
__device__ __forceinline__ void filtered_bins(const FilterArgs& a, int first, int t, int T, float2 (*steps)[16],
                                              float2 (&acc)[16]) {
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = make_float2(0.f, 0.f);
    for (int kb = 0; kb < a.L; kb += kStepRows) {
        const int nk = min(kStepRows, a.L - kb);
        if (a.coef) {
            __syncthreads();   // the previous batch's readers
            for (int i = threadIdx.x; i < nk * 16; i += blockDim.x) {
                const float4 c = __ldg(a.coef + first + kb + i / 16);
                steps[i / 16][i % 16] = unit(c.y, c.z, (float)(T * (i % 16)), 0.f, 0.f);
            }
            __syncthreads();
        }
        for (int k = 0; k < nk; ++k) {
            const int s = first + kb + k;
            const float2* row = a.ph + (size_t)s * a.N + t;
            float2 w = __ldg(a.kern + kb + k);
            if (a.coef) {
                const float4 c = __ldg(a.coef + s);
                w = sar::cmulf(w, unit(c.y, c.z, (float)t, c.x, c.w));
            }
            float2 v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = t + T * e < a.N ? __ldg(row + T * e) : make_float2(0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float2 m = a.coef ? sar::cmulf(w, steps[k][e]) : w;
                acc[e].x = fmaf(m.x, v[e].x, fmaf(-m.y, v[e].y, acc[e].x));
                acc[e].y = fmaf(m.x, v[e].y, fmaf(m.y, v[e].x, acc[e].y));
            }
        }
    }
}

// N = 512 ... 8192: one output pulse per CTA, from the phase history to its kept modes.
template <int N>
__global__ void __launch_bounds__(N / 16, 8192 / N) filter_crop_kernel(const FilterArgs a, const float2* __restrict__ tw_n) {
    constexpr int T = N / 16;
    extern __shared__ __align__(16) float2 rsm[];
    __shared__ float2 steps[kStepRows][16];
    float2* A = rsm;
    float2* B = rsm + sar::up_pad(N);
    const int t = threadIdx.x;
    float2 z[16], x[16];
    filtered_bins(a, __ldg(a.row0 + blockIdx.x), t, T, steps, z);
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = make_float2(z[(e + 8) & 15].x * a.scale, z[(e + 8) & 15].y * a.scale);   // ifftshift
    sar::up_first_pass<N>(x, A, t);
    __syncthreads();
    const float2* F = sar::up_passes<N, true>(A, B, tw_n, t);
    const int lo = a.n / 2;
    for (int j = t; j < a.n; j += T)
        a.out[(size_t)blockIdx.x * a.n + j] = sar::cmulf(__ldg(a.window + j), F[sar::up_pad(j < lo ? j : N - (a.n - j))]);
}

// Any N: filtered rows in FFT order, work[blockIdx.y][j]; blockIdx.x covers ceil(N / 16) threads.
__global__ void __launch_bounds__(256) filter_rows_kernel(const FilterArgs a, float2* __restrict__ work, int first_row) {
    __shared__ float2 steps[kStepRows][16];
    const int T = (a.N + 15) / 16, t = blockIdx.x * 256 + threadIdx.x;
    float2 z[16];
    filtered_bins(a, __ldg(a.row0 + first_row + blockIdx.y), min(t, a.N), T, steps, z);
    if (t >= T) return;
    float2* dst = work + (size_t)blockIdx.y * a.N;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        const int f = t + T * e;
        if (f >= a.N) continue;
        const int j = f < a.N / 2 ? f + (a.N - a.N / 2) : f - a.N / 2;   // natural bin f is FFT index (f - N/2) mod N
        dst[j] = make_float2(z[e].x * a.scale, z[e].y * a.scale);
    }
}

// Per-pulse phase coefficients in turns: phase(s, f) = b_s + a_s f with a_s = dR_s fs / (c N)
// and b_s = frac(dR_s (-(N/2) fs / N - sign fc) / c), reduced in FP64; a_s is passed as an FP32
// head and tail (the kernel forms head * f with its exact FMA remainder).
std::vector<float4> phase_coefficients(const double* dr, size_t S, size_t N, double fc, double fs, double sign,
                                       double c_eff) {
    std::vector<float4> co(S);
    for (size_t s = 0; s < S; ++s) {
        const double a = dr[s] * fs / (c_eff * (double)N);
        double b = dr[s] * (-(double)(N / 2) * fs / (double)N - sign * fc) / c_eff;
        b -= std::nearbyint(b);
        const float a_hi = (float)a;
        const float a_lo = (float)(a - (double)a_hi);
        co[s] = make_float4((float)b, a_hi, a_lo, (float)(b - (double)(float)b));
    }
    return co;
}

struct DevBuf {
    void* p = nullptr;
    cudaStream_t st = nullptr;
    ~DevBuf() {
        if (p) cudaFreeAsync(p, st);
    }
};

// Batched C2C plans by (device, length, rows), made on first use and kept for the process (plan
// creation costs milliseconds; resampling jobs repeat the same shapes).  A plan has one work area and one
// stream, so its uses follow each other: the mutex covers setting the stream and queueing the transform,
// and a use on another stream waits on the device for the event that the last one left behind.
struct FftPlan {
    bool made = false;
    cufftHandle handle = 0;
    cudaEvent_t last = nullptr;   // end of the plan's last use
};
std::mutex g_plan_mu;
std::map<std::tuple<int, int, int>, FftPlan> g_plans;

int fft_rows(void* data, int n, int rows, int direction, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_plan_mu);
    FftPlan& plan = g_plans[std::make_tuple(dev, n, rows)];
    if (!plan.last) R_CUDA(cudaEventCreateWithFlags(&plan.last, cudaEventDisableTiming), "resampling FFT event");
    if (!plan.made) {
        int dims[1] = {n};
        if (cufftPlanMany(&plan.handle, 1, dims, nullptr, 1, n, nullptr, 1, n, CUFFT_C2C, rows) != CUFFT_SUCCESS)
            return err(SAR_ERR_CUFFT, "resampling FFT plan");
        plan.made = true;
    }
    R_CUDA(cudaStreamWaitEvent(st, plan.last, 0), "resampling FFT order");
    cufftResult r = cufftSetStream(plan.handle, st);
    if (r == CUFFT_SUCCESS)
        r = cufftExecC2C(plan.handle, (cufftComplex*)data, (cufftComplex*)data, direction);
    const cudaError_t e = cudaEventRecord(plan.last, st);   // also after an error: part of it may be queued
    if (r != CUFFT_SUCCESS) return err(SAR_ERR_CUFFT, "resampling FFT");
    R_CUDA(e, "resampling FFT order");
    return SAR_OK;
}

// Window times the ramp that shifts the n-point transform's output by (n + 1) / 2 (numpy's fftshift), FP64-made.
std::vector<float2> shifted_window(const double* window, size_t n) {
    std::vector<float2> w(n);
    for (size_t j = 0; j < n; ++j) {   // exp(-2 pi i j shift / n) = (-1)^j, times exp(-pi i j / n) when n is odd
        const double m = (j & 1) ? -window[j] : window[j];
        if (n & 1) {
            const double angle = -3.14159265358979323846 * (double)j / (double)n;
            w[j] = make_float2((float)(m * std::cos(angle)), (float)(m * std::sin(angle)));
        } else {
            w[j] = make_float2((float)m, 0.f);
        }
    }
    return w;
}

// e^{2 pi i q / N}, q < N, FP64-made once per transform length of the fused kernel (five lengths, 124 KB in all).
const std::vector<float2>& twiddles(size_t N) {
    static std::mutex mu;
    static std::map<size_t, std::vector<float2>> tables;
    std::lock_guard<std::mutex> lock(mu);
    std::vector<float2>& t = tables[N];
    if (t.empty()) {
        t.resize(N);
        for (size_t q = 0; q < N; ++q) {
            const double angle = 6.283185307179586476925286766559 * (double)q / (double)N;
            t[q] = make_float2((float)std::cos(angle), (float)std::sin(angle));
        }
    }
    return t;
}

// Host arrays of one call packed for a single copy; each on a 16-byte boundary.
struct Packed {
    std::vector<unsigned char> bytes;
    size_t add(const void* p, size_t n) {
        const size_t at = bytes.size();
        bytes.resize(at + ((n + 15) & ~(size_t)15));
        memcpy(bytes.data() + at, p, n);
        return at;
    }
};

// Rows of `N` filtered at a time for cuFFT: about 32 MB, which stay in L2 until they are cropped, and at most the
// 65535 that gridDim.y takes.
size_t work_rows(size_t N, size_t T) {
    return std::min({T, std::max<size_t>(1, ((size_t)32 << 20) / (N * sizeof(float2))), (size_t)65535});
}

size_t packed_bytes(size_t S, size_t N, size_t n, size_t L, size_t T) {
    auto up = [](size_t b) { return (b + 15) & ~(size_t)15; };
    return up(S * sizeof(float4)) + up(n * sizeof(float2)) + up(L * sizeof(float2)) + up(T * sizeof(int)) +
           (sar::fused_fft_length((int)N) ? up(N * sizeof(float2)) : 0);
}

template <int N>
cudaError_t launch_filter_crop(const FilterArgs& a, const float2* tw_n, int rows, cudaStream_t st) {
    const size_t smem = sizeof(float2) * 2 * (N + N / 16);
    cudaError_t e = cudaFuncSetAttribute(filter_crop_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    filter_crop_kernel<N><<<rows, N / 16, smem, st>>>(a, tw_n);
    return cudaGetLastError();
}

// The whole resampling with `ws` as device scratch (sar_resample_workspace bytes).
int resample(const float2* ph, size_t S, size_t N, const double* delta_range, double fc, double fs, double sign, double c_eff,
             size_t n, const double* window, const double* kernel, size_t L, const int* row0, size_t T, float2* out,
             unsigned char* ws, cudaStream_t st) {
    const bool fused = sar::fused_fft_length((int)N);
    Packed host;
    size_t at_coef = 0, at_tw = 0;
    if (delta_range) {
        const std::vector<float4> co = phase_coefficients(delta_range, S, N, fc, fs, sign, c_eff);
        at_coef = host.add(co.data(), sizeof(float4) * S);
    }
    const size_t at_win = host.add(shifted_window(window, n).data(), sizeof(float2) * n);
    std::vector<float2> k(L);
    for (size_t i = 0; i < L; ++i) k[i] = make_float2((float)kernel[2 * i], (float)kernel[2 * i + 1]);
    const size_t at_kern = host.add(k.data(), sizeof(float2) * L), at_row = host.add(row0, sizeof(int) * T);
    if (fused) {
        const std::vector<float2>& tw = twiddles(N);
        at_tw = host.add(tw.data(), sizeof(float2) * N);
    }
    R_CUDA(cudaMemcpyAsync(ws, host.bytes.data(), host.bytes.size(), cudaMemcpyHostToDevice, st), "resampling tables");
    cudaEvent_t copied = nullptr;
    R_CUDA(cudaEventCreateWithFlags(&copied, cudaEventDisableTiming), "resampling event");
    cudaEventRecord(copied, st);
    FilterArgs a;
    a.ph = ph;
    a.coef = delta_range ? reinterpret_cast<const float4*>(ws + at_coef) : nullptr;
    a.kern = reinterpret_cast<const float2*>(ws + at_kern);
    a.row0 = reinterpret_cast<const int*>(ws + at_row);
    a.window = reinterpret_cast<const float2*>(ws + at_win);
    a.out = out;
    a.N = (int)N;
    a.L = (int)L;
    a.n = (int)n;
    a.scale = 1.0f / (float)N;   // numpy's ifft scale
    auto work = [&]() -> int {
        if (fused) {
            const float2* tw = reinterpret_cast<const float2*>(ws + at_tw);
            cudaError_t e = cudaSuccess;
            switch (N) {
                case 512: e = launch_filter_crop<512>(a, tw, (int)T, st); break;
                case 1024: e = launch_filter_crop<1024>(a, tw, (int)T, st); break;
                case 2048: e = launch_filter_crop<2048>(a, tw, (int)T, st); break;
                case 4096: e = launch_filter_crop<4096>(a, tw, (int)T, st); break;
                default: e = launch_filter_crop<8192>(a, tw, (int)T, st); break;
            }
            R_CUDA(e, "slow-time filter");
        } else {
            float2* rows = reinterpret_cast<float2*>(ws + ((packed_bytes(S, N, n, L, T) + 255) & ~(size_t)255));
            const size_t chunk = work_rows(N, T);
            for (size_t first = 0; first < T; first += chunk) {
                const int count = (int)std::min(chunk, T - first);
                const dim3 grid((unsigned)(((N + 15) / 16 + 255) / 256), (unsigned)count);
                filter_rows_kernel<<<grid, 256, 0, st>>>(a, rows, (int)first);
                R_CUDA(cudaGetLastError(), "slow-time filter");
                R_CALL(fft_rows(rows, (int)N, count, CUFFT_INVERSE, st));
                const dim3 crop((unsigned)std::min<size_t>((n + 255) / 256, 1024), (unsigned)count);
                crop_window_kernel<<<crop, 256, 0, st>>>(rows, out + first * n, a.window, count, (int)N, (int)n);
                R_CUDA(cudaGetLastError(), "crop");
            }
        }
        return fft_rows(out, (int)n, (int)T, CUFFT_FORWARD, st);
    };
    const int rc = work();
    cudaEventSynchronize(copied);   // the packed host tables go out of scope; the kernels keep running
    cudaEventDestroy(copied);
    return rc;
}

int check_sizes(size_t S, size_t N) {
    if (!S || !N || S > ((size_t)1 << 30) || N > ((size_t)1 << 28) || S * N > ((size_t)1 << 34))
        return err(SAR_ERR_INVALID_ARGUMENT, "bad phase history shape");
    return SAR_OK;
}

}  // namespace

extern "C" int sar_move_srps(const void* ph_dev, void* out_dev, size_t S, size_t N, const double* delta_range,
                             double centre_freq, double sample_bandwidth, double sign_multiplier, double c_eff,
                             void* stream) {
    if (!ph_dev || !out_dev || !delta_range) return err(SAR_ERR_INVALID_ARGUMENT, "null argument");
    R_CALL(check_sizes(S, N));
    cudaStream_t st = (cudaStream_t)stream;
    const std::vector<float4> co = phase_coefficients(delta_range, S, N, centre_freq, sample_bandwidth, sign_multiplier, c_eff);
    DevBuf dc;
    dc.st = st;
    R_CUDA(cudaMallocAsync(&dc.p, sizeof(float4) * S, st), "phase coefficients");
    R_CUDA(cudaMemcpyAsync(dc.p, co.data(), sizeof(float4) * S, cudaMemcpyHostToDevice, st), "phase coefficients");
    rephase_kernel<<<blocks_for(S * N), 256, 0, st>>>((const float2*)ph_dev, (float2*)out_dev, (const float4*)dc.p, (int)S,
                                                     (int)N, 0, 1.0f);
    R_CUDA(cudaGetLastError(), "rephase");
    R_CUDA(cudaStreamSynchronize(st), "rephase");   // host coefficient array goes out of scope
    return SAR_OK;
}

extern "C" int sar_fast_freq_downsample(const void* ph_dev, void* out_dev, size_t S, size_t N, size_t new_N,
                                        const double* window, void* stream) {
    if (!ph_dev || !out_dev || !window) return err(SAR_ERR_INVALID_ARGUMENT, "null argument");
    R_CALL(check_sizes(S, N));
    // new_N > N keeps overlapping modes, as the reference's slicing does; beyond 2 N no mode is left
    if (!new_N || new_N > 2 * N) return err(SAR_ERR_INVALID_ARGUMENT, "new_N must be in [1, 2 N]");
    cudaStream_t st = (cudaStream_t)stream;
    const std::vector<float2> w = shifted_window(window, new_N);
    DevBuf dw, spec;
    dw.st = spec.st = st;
    R_CUDA(cudaMallocAsync(&dw.p, sizeof(float2) * new_N, st), "window");
    R_CUDA(cudaMemcpyAsync(dw.p, w.data(), sizeof(float2) * new_N, cudaMemcpyHostToDevice, st), "window");
    R_CUDA(cudaMallocAsync(&spec.p, sizeof(float2) * S * N, st), "resampling work rows");
    float2* sp = (float2*)spec.p;
    // ifftshift: FFT-order index j reads natural index (j + N/2) mod N; 1/N is numpy's ifft scale
    rephase_kernel<<<blocks_for(S * N), 256, 0, st>>>((const float2*)ph_dev, sp, nullptr, (int)S, (int)N, (int)(N / 2),
                                                     1.0f / (float)N);
    R_CUDA(cudaGetLastError(), "shift");
    R_CALL(fft_rows(sp, (int)N, (int)S, CUFFT_INVERSE, st));
    const dim3 crop((unsigned)std::min<size_t>((new_N + 255) / 256, 1024), (unsigned)std::min<size_t>(S, 65535));
    crop_window_kernel<<<crop, 256, 0, st>>>(sp, (float2*)out_dev, (const float2*)dw.p, (int)S, (int)N, (int)new_N);
    R_CUDA(cudaGetLastError(), "crop");
    R_CALL(fft_rows((float2*)out_dev, (int)new_N, (int)S, CUFFT_FORWARD, st));
    R_CUDA(cudaStreamSynchronize(st), "fast_freq_downsample");   // the host window goes out of scope
    return SAR_OK;
}

static int check_resample(const void* ph_dev, size_t S, size_t N, size_t new_N, const double* window, const double* kernel,
                          size_t kernel_length, const int* row0, size_t num_rows, const void* out_dev) {
    if (!ph_dev || !out_dev || !window || !kernel || !row0) return err(SAR_ERR_INVALID_ARGUMENT, "null argument");
    R_CALL(check_sizes(S, N));
    if (!new_N || new_N > N) return err(SAR_ERR_INVALID_ARGUMENT, "new_N must be in [1, N]");
    if (!kernel_length || kernel_length > S) return err(SAR_ERR_INVALID_ARGUMENT, "bad kernel length");
    for (size_t t = 0; t < num_rows; ++t)
        if (row0[t] < 0 || (size_t)row0[t] + kernel_length > S) return err(SAR_ERR_INVALID_ARGUMENT, "window outside the pulses");
    return SAR_OK;
}

extern "C" size_t sar_resample_workspace(size_t S, size_t N, size_t new_N, size_t kernel_length, size_t num_rows) {
    const size_t tables = (packed_bytes(S, N, new_N, kernel_length, num_rows) + 255) & ~(size_t)255;
    return tables + (sar::fused_fft_length((int)std::min<size_t>(N, 1u << 30)) ? 0 : work_rows(std::max<size_t>(N, 1), num_rows) * N * sizeof(float2));
}

extern "C" int sar_resample_phase_history_ws(const void* ph_dev, size_t S, size_t N, const double* delta_range,
                                             double centre_freq, double sample_bandwidth, double sign_multiplier,
                                             double c_eff, size_t new_N, const double* window, const double* kernel,
                                             size_t kernel_length, const int* row0, size_t num_rows, void* out_dev,
                                             void* workspace_dev, size_t workspace_bytes, void* stream) {
    R_CALL(check_resample(ph_dev, S, N, new_N, window, kernel, kernel_length, row0, num_rows, out_dev));
    if (!num_rows) return SAR_OK;
    if (!workspace_dev || ((uintptr_t)workspace_dev & 255) ||
        workspace_bytes < sar_resample_workspace(S, N, new_N, kernel_length, num_rows))
        return err(SAR_ERR_INVALID_ARGUMENT, "workspace too small or not on a 256-byte boundary");
    return resample((const float2*)ph_dev, S, N, delta_range, centre_freq, sample_bandwidth, sign_multiplier, c_eff, new_N,
                    window, kernel, kernel_length, row0, num_rows, (float2*)out_dev, (unsigned char*)workspace_dev,
                    (cudaStream_t)stream);
}

extern "C" int sar_resample_phase_history(const void* ph_dev, size_t S, size_t N, const double* delta_range,
                                          double centre_freq, double sample_bandwidth, double sign_multiplier,
                                          double c_eff, size_t new_N, const double* window, const double* kernel,
                                          size_t kernel_length, const int* row0, size_t num_rows, void* out_dev,
                                          void* stream) {
    R_CALL(check_resample(ph_dev, S, N, new_N, window, kernel, kernel_length, row0, num_rows, out_dev));
    if (!num_rows) return SAR_OK;
    cudaStream_t st = (cudaStream_t)stream;
    DevBuf ws;
    ws.st = st;
    R_CUDA(cudaMallocAsync(&ws.p, sar_resample_workspace(S, N, new_N, kernel_length, num_rows), st), "resampling workspace");
    R_CALL(resample((const float2*)ph_dev, S, N, delta_range, centre_freq, sample_bandwidth, sign_multiplier, c_eff, new_N,
                    window, kernel, kernel_length, row0, num_rows, (float2*)out_dev, (unsigned char*)ws.p, st));
    R_CUDA(cudaStreamSynchronize(st), "resample");
    return SAR_OK;
}
