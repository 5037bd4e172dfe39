// sar_stockham.cuh -- N-point Stockham transforms in shared memory, N = 512 ... 8192: the passes the
// fused range-profile kernels share (sar_kernels.cu, sar_fir.cu).
#pragma once

#include <cuda_runtime.h>

namespace sar {

template <int N>
struct UpShape {
    static constexpr int T = N / 16;                // threads per row: one radix-16 butterfly each
    static constexpr int P = N >= 8192 ? 3 : 2;     // radix-16 passes after the first
    static constexpr int R0 = N / (P == 3 ? 4096 : 256);   // radix of the first pass: 2, 4, 8 or 16
    static constexpr int NB = 16 / R0;              // first-pass butterflies per thread
    static_assert(R0 >= 2 && R0 <= 16 && R0 * (P == 3 ? 4096 : 256) == N, "unsupported transform length");
};

__device__ __forceinline__ int up_pad(int x) { return x + (x >> 4); }   // one slot per 16: no bank conflicts
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ void dft4_inv(float2& x0, float2& x1, float2& x2, float2& x3) {
    const float2 t0 = make_float2(x0.x + x2.x, x0.y + x2.y), t1 = make_float2(x0.x - x2.x, x0.y - x2.y);
    const float2 t2 = make_float2(x1.x + x3.x, x1.y + x3.y);
    const float2 t3 = make_float2(-(x1.y - x3.y), x1.x - x3.x);   // i (x1 - x3)
    x0 = make_float2(t0.x + t2.x, t0.y + t2.y);
    x1 = make_float2(t1.x + t3.x, t1.y + t3.y);
    x2 = make_float2(t0.x - t2.x, t0.y - t2.y);
    x3 = make_float2(t1.x - t3.x, t1.y - t3.y);
}
// v[k] <- sum_n v[n] e^{+2 pi i n k / 16}: n = 4 n1 + n2, k = k1 + 4 k2 (two radix-4 stages).
__device__ __forceinline__ void dft16_inv(float2 (&v)[16]) {
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4_inv(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);   // -> Y[n2][k1] at v[4 k1 + n2]
    const float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
    // W16^(n2 k1) for (n2, k1) in {1,2,3} x {1,2,3}: exponents 1 2 3 / 2 4 6 / 3 6 9
    v[4 + 1] = cmulf(v[4 + 1], make_float2(c1, s1));
    v[8 + 1] = cmulf(v[8 + 1], make_float2(h, h));
    v[12 + 1] = cmulf(v[12 + 1], make_float2(s1, c1));
    v[4 + 2] = cmulf(v[4 + 2], make_float2(h, h));
    v[8 + 2] = make_float2(-v[8 + 2].y, v[8 + 2].x);   // W16^4 = i
    v[12 + 2] = cmulf(v[12 + 2], make_float2(-h, h));
    v[4 + 3] = cmulf(v[4 + 3], make_float2(s1, c1));
    v[8 + 3] = cmulf(v[8 + 3], make_float2(-h, h));
    v[12 + 3] = cmulf(v[12 + 3], make_float2(-c1, -s1));
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4_inv(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // now v[4 k1 + k2] holds X[k1 + 4 k2]: transpose the 4x4 index to natural order
    float2 t[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) t[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = t[k];
}

// v[k] <- sum_n v[n] e^{+2 pi i n k / 8}: n = 2 n1 + n2, k = k1 + 4 k2 (radix 4, then radix 2).
__device__ __forceinline__ void dft8_inv(float2 (&v)[8]) {
    dft4_inv(v[0], v[2], v[4], v[6]);   // n2 = 0: Y0[k1] at v[2 k1]
    dft4_inv(v[1], v[3], v[5], v[7]);   // n2 = 1: Y1[k1] at v[2 k1 + 1]
    const float h = 0.70710678118654752f;
    v[3] = cmulf(v[3], make_float2(h, h));            // W8^1
    v[5] = make_float2(-v[5].y, v[5].x);              // W8^2 = i
    v[7] = cmulf(v[7], make_float2(-h, h));           // W8^3
    float2 t[8];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
        const float2 a = v[2 * k1], b = v[2 * k1 + 1];
        t[k1] = make_float2(a.x + b.x, a.y + b.y);
        t[k1 + 4] = make_float2(a.x - b.x, a.y - b.y);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = t[k];
}

// First Stockham pass (sub-transform length 1) on the 16 values x[e] = element t + T e a thread
// holds: butterfly j = t + T e1 (e1 < NB) combines elements j + 256 m (m < R0), which are
// x[e1 + NB m], and writes out[j R0 + m].
template <int N>
__device__ __forceinline__ void up_first_pass(const float2 (&x)[16], float2* out, int t) {
    constexpr int T = UpShape<N>::T, R0 = UpShape<N>::R0, NB = UpShape<N>::NB;
#pragma unroll
    for (int e1 = 0; e1 < NB; ++e1) {
        const int j = t + T * e1;
        if constexpr (R0 == 16) {
            float2 v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = x[m];
            dft16_inv(v);
#pragma unroll
            for (int m = 0; m < 16; ++m) out[up_pad(j * 16 + m)] = v[m];
        } else if constexpr (R0 == 8) {
            float2 v[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) v[m] = x[e1 + NB * m];
            dft8_inv(v);
#pragma unroll
            for (int m = 0; m < 8; ++m) out[up_pad(j * 8 + m)] = v[m];
        } else if constexpr (R0 == 4) {
            float2 a = x[e1], b = x[e1 + NB], c = x[e1 + 2 * NB], d = x[e1 + 3 * NB];
            dft4_inv(a, b, c, d);
            out[up_pad(j * 4)] = a;
            out[up_pad(j * 4 + 1)] = b;
            out[up_pad(j * 4 + 2)] = c;
            out[up_pad(j * 4 + 3)] = d;
        } else {
            const float2 a = x[e1], b = x[e1 + NB];
            out[up_pad(j * 2)] = make_float2(a.x + b.x, a.y + b.y);
            out[up_pad(j * 2 + 1)] = make_float2(a.x - b.x, a.y - b.y);
        }
    }
}

// v[r] *= w^r for r = 1..15.  Built from w alone, w^r has r times w's rounding error, which was most of a transform's:
// range profiles of N = 512 ... 8192, 2-norm, 2.7e-7 to 3.7e-7.  From the table's w and w^4 (upsampling): 1.5e-7 to 2.0e-7;
// from w, w^2, w^4 and w^8 (FOUR; downsampling, whose few values leave the twiddles most of the error): 1.4e-7 to 1.7e-7,
// and 8e-8 for 9.5e-8 downsampled at U = 128.  4096 rows of 4096: upsampling 133, 138 and 148 us, downsampling 174, 180 and 182.
__device__ __forceinline__ void apply_powers(float2 (&v)[16], float2 w, float2 w2, float2 w4, float2 w8) {
    const float2 w3 = cmulf(w2, w), w5 = cmulf(w4, w), w6 = cmulf(w4, w2), w7 = cmulf(w4, w3);
    v[1] = cmulf(v[1], w);
    v[2] = cmulf(v[2], w2);
    v[3] = cmulf(v[3], w3);
    v[4] = cmulf(v[4], w4);
    v[5] = cmulf(v[5], w5);
    v[6] = cmulf(v[6], w6);
    v[7] = cmulf(v[7], w7);
    v[8] = cmulf(v[8], w8);
    v[9] = cmulf(v[9], cmulf(w8, w));
    v[10] = cmulf(v[10], cmulf(w8, w2));
    v[11] = cmulf(v[11], cmulf(w8, w3));
    v[12] = cmulf(v[12], cmulf(w8, w4));
    v[13] = cmulf(v[13], cmulf(w8, w5));
    v[14] = cmulf(v[14], cmulf(w8, w6));
    v[15] = cmulf(v[15], cmulf(w8, w7));
}

// e^{2 pi i k r / M} for the 16 frequencies k = t + T e of thread t (signed: minus N for e >= 8),
// 0 <= r < 2U, as the product of e^{2 pi i t r / M} (tw_m[t r]) and the thread-independent factor
// tw_e[16 r + e] = e^{2 pi i (T e - N [e >= 8]) r / M} (stored after the M entries of tw_m).
template <int N>
__device__ __forceinline__ void residue_twiddles(const float2* __restrict__ tw_m, long M, int t, int r,
                                                 float2 (&w)[16]) {
    const float2 a = __ldg(tw_m + t * r);
    const float2* __restrict__ b = tw_m + M + 16 * r;
#pragma unroll
    for (int e = 0; e < 16; ++e) w[e] = cmulf(a, __ldg(b + e));
}

// Radix-16 Stockham pass over N points (sub-transform length ns = N / 256 or N / 16 before it) by the
// N / 16 threads j of one transform.
template <int N, bool FOUR>
__device__ __forceinline__ void up_pass(const float2* in, float2* out, int ns, const float2* __restrict__ tw_n,
                                        int j) {
    float2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = in[up_pad(j + r * (N / 16))];
    const int k = j & (ns - 1);
    const int q = k * (N / (ns * 16));   // w = e^{2 pi i k / (16 ns)}; 8 q < N / 2
    if constexpr (FOUR) {
        apply_powers(v, __ldg(tw_n + q), __ldg(tw_n + 2 * q), __ldg(tw_n + 4 * q), __ldg(tw_n + 8 * q));
    } else {
        const float2 w = __ldg(tw_n + q), w4 = __ldg(tw_n + 4 * q);
        apply_powers(v, w, cmulf(w, w), w4, cmulf(w4, w4));
    }
    dft16_inv(v);
    const int base = (j / ns) * ns * 16 + k;
#pragma unroll
    for (int r = 0; r < 16; ++r) out[up_pad(base + r * ns)] = v[r];
}

// The radix-16 passes after the first (from `in`, ping-ponging with `tmp`): returns the buffer that
// holds the transform.  The caller synchronises before; each pass ends with a barrier.
template <int N, bool FOUR>
__device__ __forceinline__ float2* up_passes(float2* in, float2* tmp, const float2* __restrict__ tw_n, int j) {
    constexpr int R0 = UpShape<N>::R0;
    up_pass<N, FOUR>(in, tmp, R0, tw_n, j);
    __syncthreads();
    up_pass<N, FOUR>(tmp, in, 16 * R0, tw_n, j);
    __syncthreads();
    if constexpr (UpShape<N>::P == 3) {
        up_pass<N, FOUR>(in, tmp, 256 * R0, tw_n, j);
        __syncthreads();
        return tmp;
    }
    return in;
}

static inline bool fused_fft_length(int N) { return N == 512 || N == 1024 || N == 2048 || N == 4096 || N == 8192; }

}  // namespace sar
