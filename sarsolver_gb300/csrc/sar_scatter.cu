// sar_scatter.cu -- forward scatter of a regular grid, linear sampling: a pulse per lane (K3).
//
// A warp owns 32 consecutive pulses, one per lane, and walks blocks of 16 x 16 pixels; every lane adds
// each pixel to its own pulse's range window in shared memory.  The windows lie interleaved,
// [slot][lane], so an access is free of bank conflicts whatever the lanes' bins, no two lanes ever
// write the same slot (no atomics, no distinct-bin guarantee, no pixel order to respect), the
// coefficients of a (block, pulse) live in the lane's registers, and the pixel value is one
// broadcast load for 32 pulses.  With a pixel per lane (fp_grid_ws_kernel) the lanes of a row must fall
// on distinct bins, which away from the grid axes left two conflicting read-modify-writes per pixel
// and pulse (L1 data pipe at 96 %).
//
// Because the order of a block's pixels is free, its lines follow the lattice direction w = (p, q),
// p^2 + q^2 <= 5, along which range changes least.  Down a line of 16 pixels the bin then usually moves
// by less than one: the line's taps lie in three consecutive bins, its sums are kept in registers as
// moments C = sum c, D = sum a c, E = sum |a| c (a the tap position about the middle bin: the three
// linear weights are (|a| - a) / 2, 1 - |a|, (|a| + a) / 2), and three slots are updated once per line (per 8 or 4
// pixels where the bin moves faster; both taps of every pixel where no run is short enough).  Two
// neighbouring lines share each packed FP32 instruction.
//
// Windows: `slots` bins around the block's anchor bin, a ring per lane.  From block to block along w the
// anchor moves by a few bins; the slots left behind are added to the accumulator and cleared, the
// rest at the end of the CTA's run.  Each lane bounds its block's bins against the ring
// before it walks (FLAG_STRIP_WINDOW otherwise, and the block is dropped).
//
// Bound: the FMA pipe and the special-function pipe alike (15 packed FMAs and 4 sine / cosine
// operations per two pixel-pulses).  Measured figures stand at launch_scatter.
#include <algorithm>
#include <cmath>

#include "sar_host_prep.h"
#include "sar_kernels.cuh"
#include "sar_scatter.cuh"

namespace sar {

namespace {

#define SC_TWO_PI 6.28318530717958647692f

__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }

__device__ __forceinline__ PulseGeom load_pulse(const PulseGeom* p) {
    const float4* v = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(v), b = __ldg(v + 1), c = __ldg(v + 2), d = __ldg(v + 3);
    PulseGeom g;
    g.atx_hi[0] = a.x; g.atx_hi[1] = a.y; g.atx_hi[2] = a.z; g.atx_lo[0] = a.w;
    g.atx_lo[1] = b.x; g.atx_lo[2] = b.y; g.arx_hi[0] = b.z; g.arx_hi[1] = b.w;
    g.arx_hi[2] = c.x; g.arx_lo[0] = c.y; g.arx_lo[1] = c.z; g.arx_lo[2] = c.w;
    g.rref_hi = d.x; g.rref_lo = d.y; g.monostatic = d.z; g.pad = d.w;
    return g;
}

constexpr float kRunSpan = 0.98f;   // bins a run of pixels may span (its taps then lie in three bins)
constexpr float kDip = 0.1f;        // bins a run may fall below its end points (curvature)

// Terms of two neighbouring lines (a, a + 1): phase cph + b1 d + b2 d^2 + c9 d^3 in radians and bin
// cv + bv1 d + bv2 d^2, d the offset along the line.
struct LinePair {
    float2 cph, b1, b2, c9, cv, bv1, bv2;
};

__device__ __forceinline__ LinePair line_pair(const Coeffs& co, float di) {
    const float2 D = mk(di, di + 1.f), K = dup(SC_TWO_PI), SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
    LinePair t;
    float2 ph = fma2(fma2(fma2(dup(co.c[6]), D, dup(co.c[3])), D, dup(co.c[1])), D, dup(co.c[0]));
    ph = fma2(add2(add2(ph, SH), NSH), M1, ph);   // mod 1: the line's phases stay below ~5 cycles
    t.cph = mul2(ph, K);
    t.b1 = mul2(fma2(fma2(dup(co.c[7]), D, dup(co.c[4])), D, dup(co.c[2])), K);
    t.b2 = mul2(fma2(dup(co.c[8]), D, dup(co.c[5])), K);
    t.c9 = dup(co.c[9] * SC_TWO_PI);
    t.cv = fma2(fma2(dup(co.v[3]), D, dup(co.v[1])), D, dup(co.v[0]));
    t.bv1 = fma2(dup(co.v[4]), D, dup(co.v[2]));
    t.bv2 = dup(co.v[5]);
    return t;
}

// c = x exp(i phase) for the two lines' pixels at offset d (XN = -im).
__device__ __forceinline__ void contribution(const LinePair& t, float2 d, float4 X, float2 XN, float2* cr, float2* ci) {
    const float2 ph = fma2(fma2(fma2(t.c9, d, t.b2), d, t.b1), d, t.cph);
    float2 sn, cn;
    __sincosf(ph.x, &sn.x, &cn.x);
    __sincosf(ph.y, &sn.y, &cn.y);
    *cr = fma2(mk(X.x, X.y), cn, mul2(XN, sn));
    *ci = fma2(mk(X.x, X.y), sn, mul2(mk(X.z, X.w), cn));
}

// Ring slot of x in [0, 2 W).
__device__ __forceinline__ int wrap(int x, int W) { return (int)min((unsigned)x, (unsigned)(x - W)); }

// A block's lines with runs of G pixels; dip bounds how far the bin falls below a run's end points.
template <int G>
__device__ __forceinline__ void walk_runs(const Coeffs& co, const float4* xs, const float2* xn, float2* win, int off, int W,
                                          int lines) {
    const float2 SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
    const float2 ndip = dup(-0.25f * (G - 1) * (G - 1) * fabsf(co.v[5]));
#pragma unroll 1
    for (int l = 0; l < lines / 2; ++l) {
        const LinePair t = line_pair(co, (float)(2 * l - lines / 2));
        const float4* xl = xs + l * kWalk;
        const float2* nl = xn + l * kWalk;
#pragma unroll
        for (int g0 = 0; g0 < kWalk; g0 += G) {
            const float2 da = dup((float)(g0 - 8)), db = dup((float)(g0 + G - 9));
            const float2 va = fma2(fma2(t.bv2, da, t.bv1), da, t.cv), vb = fma2(fma2(t.bv2, db, t.bv1), db, t.cv);
            const float2 r = add2(add2(mk(fminf(va.x, vb.x), fminf(va.y, vb.y)), ndip), SH);
            // a = v - (n0 + 1/2)
            const float2 cva = fma2(add2(r, NSH), M1, add2(t.cv, dup(-0.5f)));
            float2 Cr = dup(0.f), Ci = Cr, Dr = Cr, Di = Cr, Er = Cr, Ei = Cr;
#pragma unroll
            for (int rr = g0; rr < g0 + G; ++rr) {
                const float2 d = dup((float)(rr - 8));
                float2 cr, ci;
                contribution(t, d, xl[rr], nl[rr], &cr, &ci);
                const float2 av = fma2(fma2(t.bv2, d, t.bv1), d, cva);
                const float2 aa = mk(fabsf(av.x), fabsf(av.y));
                Cr = add2(Cr, cr);
                Ci = add2(Ci, ci);
                Dr = fma2(av, cr, Dr);
                Di = fma2(av, ci, Di);
                Er = fma2(aa, cr, Er);
                Ei = fma2(aa, ci, Ei);
            }
            const float2 h = dup(0.5f);
            const float2 s0r = mul2(fma2(Dr, M1, Er), h), s0i = mul2(fma2(Di, M1, Ei), h);
            const float2 s1r = fma2(Er, M1, Cr), s1i = fma2(Ei, M1, Ci);
            const float2 s2r = mul2(add2(Er, Dr), h), s2i = mul2(add2(Ei, Di), h);
            {
                const int p0 = wrap(__float_as_int(r.x) - SAR_SHIFTER_BITS + off, W), p1 = wrap(p0 + 1, W), p2 = wrap(p1 + 1, W);
                const float2 u0 = win[p0 * 32], u1 = win[p1 * 32], u2 = win[p2 * 32];
                win[p0 * 32] = add2(u0, mk(s0r.x, s0i.x));
                win[p1 * 32] = add2(u1, mk(s1r.x, s1i.x));
                win[p2 * 32] = add2(u2, mk(s2r.x, s2i.x));
            }
            {
                const int p0 = wrap(__float_as_int(r.y) - SAR_SHIFTER_BITS + off, W), p1 = wrap(p0 + 1, W), p2 = wrap(p1 + 1, W);
                const float2 u0 = win[p0 * 32], u1 = win[p1 * 32], u2 = win[p2 * 32];
                win[p0 * 32] = add2(u0, mk(s0r.y, s0i.y));
                win[p1 * 32] = add2(u1, mk(s1r.y, s1i.y));
                win[p2 * 32] = add2(u2, mk(s2r.y, s2i.y));
            }
        }
    }
}

// Both taps of every pixel (the bin moves too fast for runs).
__device__ __forceinline__ void walk_taps(const Coeffs& co, const float4* xs, const float2* xn, float2* win, int off, int W,
                                          int lines) {
    const float2 SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
#pragma unroll 1
    for (int l = 0; l < lines / 2; ++l) {
        const LinePair t = line_pair(co, (float)(2 * l - lines / 2));
        const float4* xl = xs + l * kWalk;
        const float2* nl = xn + l * kWalk;
#pragma unroll 4
        for (int rr = 0; rr < kWalk; ++rr) {
            const float2 d = dup((float)(rr - 8));
            float2 cr, ci;
            contribution(t, d, xl[rr], nl[rr], &cr, &ci);
            const float2 v = fma2(fma2(t.bv2, d, t.bv1), d, t.cv);
            const float2 r = add2(v, SH);
            const float2 s = fma2(add2(r, NSH), M1, v);
            const float2 w0 = fma2(s, M1, dup(0.5f)), w1 = add2(s, dup(0.5f));
            {
                const int p0 = wrap(__float_as_int(r.x) - SAR_SHIFTER_BITS + off, W), p1 = wrap(p0 + 1, W);
                const float2 u0 = win[p0 * 32], u1 = win[p1 * 32], c = mk(cr.x, ci.x);
                win[p0 * 32] = fma2(dup(w0.x), c, u0);
                win[p1 * 32] = fma2(dup(w1.x), c, u1);
            }
            {
                const int p0 = wrap(__float_as_int(r.y) - SAR_SHIFTER_BITS + off, W), p1 = wrap(p0 + 1, W);
                const float2 u0 = win[p0 * 32], u1 = win[p1 * 32], c = mk(cr.y, ci.y);
                win[p0 * 32] = fma2(dup(w0.y), c, u0);
                win[p1 * 32] = fma2(dup(w1.y), c, u1);
            }
        }
    }
}

// Shared memory of a CTA: [warps][slots][32] windows, two image buffers (value pairs of two lines, and the
// negated imaginary parts), two anchors.
struct ScatterSmem {
    size_t xs, xn, anchors, total;
};
__host__ __device__ inline ScatterSmem scatter_smem(int slots, int lines) {
    ScatterSmem L;
    L.xs = (size_t)kScatterWarps * slots * 32 * sizeof(float2);
    L.xn = L.xs + (size_t)2 * (lines / 2) * kWalk * sizeof(float4);
    L.anchors = L.xn + (size_t)2 * (lines / 2) * kWalk * sizeof(float2);
    L.total = L.anchors + 2 * sizeof(df3);
    return L;
}

}  // namespace

__global__ void __launch_bounds__(32 * kScatterWarps, 4) scatter_kernel(const ScatterArgs a) {
    extern __shared__ __align__(16) unsigned char ssm[];
    constexpr int NT = 32 * kScatterWarps;
    const ScatterSmem L = scatter_smem(a.slots, a.lines);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = a.slots;
    const int pairs = a.lines / 2, block_px = pairs * kWalk;   // pixel pairs of a block, at most 128
    float2* win = reinterpret_cast<float2*>(ssm) + (size_t)warp * W * 32 + lane;
    float4* xs = reinterpret_cast<float4*>(ssm + L.xs);
    float2* xn = reinterpret_cast<float2*>(ssm + L.xn);
    df3* anchors = reinterpret_cast<df3*>(ssm + L.anchors);
    const int4 item = __ldg(a.items + blockIdx.x);
    const int s = (int)blockIdx.y * NT + (int)threadIdx.x;   // this lane's pulse
    const bool live = s < a.S;
    float2* arow = a.acc + (size_t)(live ? s : 0) * a.Lg;
    const PulseGeom pg = load_pulse(a.pulses + (live ? s : a.S - 1));

    // this thread's pixel pair of a block: lines 2 l, 2 l + 1 at offset b
    const int l = (int)threadIdx.x % pairs, b = (int)threadIdx.x / pairs;
    auto fetch = [&](int blk, float2* p, float2* q) {
        *p = *q = make_float2(0.f, 0.f);
        if (b >= kWalk || blk >= item.z) return;
        const int la = item.x + 2 * l, lb = item.y + blk * kWalk + b;
        const int i0 = a.vx * la + a.wx * lb, j0 = a.vy * la + a.wy * lb, i1 = i0 + a.vx, j1 = j0 + a.vy;
        const float2* plane = a.x + (size_t)item.w * a.img.ny * a.img.nx;
        if (i0 >= 0 && i0 < a.img.nx && j0 >= 0 && j0 < a.img.ny) *p = __ldg(plane + (size_t)j0 * a.img.nx + i0);
        if (i1 >= 0 && i1 < a.img.nx && j1 >= 0 && j1 < a.img.ny) *q = __ldg(plane + (size_t)j1 * a.img.nx + i1);
    };
    auto stage = [&](int blk, float2 p, float2 q) {
        if (blk >= item.z) return;
        const int o = (blk & 1) * block_px;
        if (b < kWalk) {
            xs[o + l * kWalk + b] = make_float4(p.x, q.x, p.y, q.y);
            xn[o + l * kWalk + b] = make_float2(-p.y, -q.y);
        }
        if (threadIdx.x == 0) {   // anchor: line `lines / 2`, offset 8
            const int la = item.x + pairs, lb = item.y + blk * kWalk + 8;
            anchors[blk & 1] = pixel_position(a.vx * la + a.wx * lb, a.vy * la + a.wy * lb, item.w, a.img);
        }
    };
    float2 p, q;
    fetch(0, &p, &q);
    for (int w = 0; w < W; ++w) win[w * 32] = make_float2(0.f, 0.f);
    stage(0, p, q);
    __syncthreads();

    auto flush = [&](int bin, int slot) {
        const float2 v = win[slot * 32];
        win[slot * 32] = make_float2(0.f, 0.f);
        if (v.x == 0.f && v.y == 0.f) return;
        const long gi = (long)bin - a.bg0;
        if (gi < 0 || gi >= a.Lg) {
            if (live) atomicOr(a.flags, FLAG_STRIP_WINDOW);
            return;
        }
        if (live) atomicAdd(arow + gi, v);
    };
    int lo = 0, rot = 0;   // the ring holds bins [lo, lo + W), bin lo in slot rot
    for (int blk = 0; blk < item.z; ++blk) {
        fetch(blk + 1, &p, &q);   // in flight while this block is walked
        AnchorExpansion ae = expand_anchor(anchors[blk & 1], pg, a.lat);
        Coeffs co;
        phase_coeffs(ae, a.lat, co.c);
        const df vb = anchor_bin(ae, a.lat);
        const int base = base_bin_of(vb, 1.0f);
        bin_coeffs(ae, vb, base, a.lat, co);
        // move the ring to [base - half, ...)
        const int want = base - a.half;
        if (blk == 0) lo = want;
        const int shift = want - lo, n = min(abs(shift), W);
        for (int k = 0; k < n; ++k) {
            const int at = shift > 0 ? k : W - 1 - k;
            flush(lo + at, wrap(rot + at, W));
        }
        lo = want;
        rot = (rot + shift) % W;
        if (rot < 0) rot += W;
        // every tap of the block inside the ring: the bin polynomial's largest excursion over the block, then
        // half a bin of rounding, a run's fall below its end points (< kDip) and two further taps
        const float hl = 0.5f * (float)a.lines;
        const float ext = fabsf(co.v[1]) * hl + fabsf(co.v[2]) * 8.f + fabsf(co.v[3]) * hl * hl + fabsf(co.v[4]) * 8.f * hl +
                          fabsf(co.v[5]) * 64.f;
        if (!(co.v[0] - ext - 0.5f - kDip >= -(float)a.half && co.v[0] + ext + 2.5f <= (float)(W - a.half - 1))) {
            if (live) atomicOr(a.flags, FLAG_STRIP_WINDOW);
            co = Coeffs{};
        }
        // runs: the bin moves by less than kRunSpan over G pixels of a line (|rate| over the block, plus the
        // fall below the end points)
        const float rate = fabsf(co.v[2]) + 8.f * fabsf(co.v[4]) + 16.f * fabsf(co.v[5]), c2 = fabsf(co.v[5]);
        const int off = rot + a.half;   // slot of bin n (about the base) is wrap(n + off)
        const float4* bx = xs + (blk & 1) * block_px;
        const float2* bn = xn + (blk & 1) * block_px;
        if (__all_sync(0xffffffffu, 15.f * rate + 56.25f * c2 < kRunSpan && 56.25f * c2 < kDip))
            walk_runs<16>(co, bx, bn, win, off, W, a.lines);
        else if (__all_sync(0xffffffffu, 7.f * rate + 12.25f * c2 < kRunSpan && 12.25f * c2 < kDip))
            walk_runs<8>(co, bx, bn, win, off, W, a.lines);
        else if (__all_sync(0xffffffffu, 3.f * rate + 2.25f * c2 < kRunSpan && 2.25f * c2 < kDip))
            walk_runs<4>(co, bx, bn, win, off, W, a.lines);
        else
            walk_taps(co, bx, bn, win, off, W, a.lines);
        stage(blk + 1, p, q);   // the other buffer: its last readers passed the previous barrier
        __syncthreads();
    }
    for (int k = 0; k < W; ++k) flush(lo + k, wrap(rot + k, W));
}

// Measured (GB300, this kernel alone, against a pixel per lane in fp_grid_ws_kernel before): 2048^2 x 4096 pulses
// 12.3 ms (16.6); 1300 x 901 x 1200 looking at 27 degrees 1.34 ms (4.22); 1024^2 x 2048 1.55 ms (2.02); 512^2 x
// 1024 0.21 ms (0.28); 256^2 x 128 20 us (33).  15 instructions per pixel-pulse (26 before), issue 48 %, FMA
// pipe 60 % of its cycles.  Tried: loops of 2 / 4 / 8 pixels instead of whole lines in straight code (14.4 / 14.2 /
// 13.8 ms: less to overlap the sine latency with); one body of 8 pixels for both run lengths 13.2 ms; 8 warps per
// CTA 12.7 ms; one warp per CTA 13.9 ms (nothing keeps warps on the same instructions); 20 warps per SM at 96
// registers 12.7 ms; 8 lines per block, and so four CTAs per SM, 13.6 ms.
cudaError_t launch_scatter(const ScatterArgs& a, cudaStream_t st) {
    if (a.lines < 2 || a.lines > 16 || (a.lines & 1) || a.num_items < 1) return cudaErrorInvalidValue;
    const size_t smem = scatter_smem(a.slots, a.lines).total;
    cudaError_t e = cudaFuncSetAttribute(scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int per = 32 * kScatterWarps;
    const dim3 grid((unsigned)a.num_items, (unsigned)((a.S + per - 1) / per));
    scatter_kernel<<<grid, per, smem, st>>>(a);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ layout
namespace {

// Instructions per pixel-pulse by run length, for the choice of lattice only.
double run_cost(double rate) {
    return 15.0 * rate < kRunSpan ? 16.0 : 7.0 * rate < kRunSpan ? 20.0 : 3.0 * rate < kRunSpan ? 27.0 : 34.0;
}

}  // namespace

// The CTAs' runs of blocks: for every strip of `lines` lattice lines the interval of offsets that holds
// image pixels, cut into segments so that a launch has about five waves of CTAs.
static void scatter_items(size_t S, int nx, int ny, int nz, ScatterLayout* L) {
    const int vx = L->vx, vy = L->vy, wx = L->wx, wy = L->wy, det = vx * wy - vy * wx;
    int a_lo = 0, a_hi = 0;
    for (int corner = 0; corner < 4; ++corner) {
        const int i = (corner & 1) ? nx - 1 : 0, j = (corner & 2) ? ny - 1 : 0, a = det * (wy * i - wx * j);
        a_lo = corner ? std::min(a_lo, a) : a;
        a_hi = corner ? std::max(a_hi, a) : a;
    }
    auto clip = [](int v, int w, int a, int n, long* lo, long* hi) {   // 0 <= v a + w b <= n - 1
        const long p = (long)v * a;
        if (w == 0) {
            if (p < 0 || p > n - 1) *hi = *lo - 1;
            return;
        }
        long l = -p, h = n - 1 - p;   // bounds of w b
        if (w < 0) {
            std::swap(l, h);
            l = -l;
            h = -h;
        }
        const long q = std::abs(w);
        *lo = std::max(*lo, l >= 0 ? (l + q - 1) / q : -((-l) / q));
        *hi = std::min(*hi, h >= 0 ? h / q : -((-h + q - 1) / q));
    };
    std::vector<int4> strips;
    long total = 0;
    for (int a0 = a_lo; a0 <= a_hi; a0 += L->lines) {
        long b0 = 0, b1 = -1;
        bool any = false;
        for (int a = a0; a < a0 + L->lines; ++a) {
            long lo = -(1L << 40), hi = 1L << 40;
            clip(vx, wx, a, nx, &lo, &hi);
            if (lo <= hi) clip(vy, wy, a, ny, &lo, &hi);
            if (lo > hi) continue;
            b0 = any ? std::min(b0, lo) : lo;
            b1 = any ? std::max(b1, hi) : hi;
            any = true;
        }
        if (!any) continue;
        const int n = (int)((b1 - b0) / kWalk) + 1;
        total += n;
        strips.push_back(make_int4(a0, (int)b0, n, 0));
    }
    const size_t groups = (S + 32 * kScatterWarps - 1) / (32 * kScatterWarps);
    const long len = std::max<long>(1, (long)((double)total * nz * groups / (152.0 * 12 / kScatterWarps * 5)));
    L->items.clear();
    for (int k = 0; k < nz; ++k)
        for (const int4& t : strips) {
            const int cuts = (int)((t.z + len - 1) / len);
            for (int c = 0; c < cuts; ++c) {
                const int p = (int)((long)t.z * c / cuts), q = (int)((long)t.z * (c + 1) / cuts);
                L->items.push_back(make_int4(t.x, t.y + p * kWalk, q - p, k));
            }
        }
}

ScatterLayout scatter_layout(const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                             const double* ey, const double* ez, int nx, int ny, int nz, double s_r) {
    ScatterLayout best;
    double c0[3];
    for (int d = 0; d < 3; ++d)
        c0[d] = origin[d] + 0.5 * ((nx - 1) * ex[d] + (ny - 1) * ey[d] + (nz - 1) * ez[d]);
    // bin rates along x and y at the scene centre, per pulse
    std::vector<double> gx(S), gy(S);
    for (size_t s = 0; s < S; ++s) {
        gx[s] = gy[s] = 0.0;
        for (int ant = 0; ant < 2; ++ant) {
            const double* p = (ant ? rx : tx) + 3 * s;
            const double w[3] = {c0[0] - p[0], c0[1] - p[1], c0[2] - p[2]};
            const double r = std::sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
            if (!(r > 0.0)) return best;
            gx[s] += s_r * (w[0] * ex[0] + w[1] * ex[1] + w[2] * ex[2]) / r;
            gy[s] += s_r * (w[0] * ey[0] + w[1] * ey[1] + w[2] * ey[2]) / r;
        }
        if (!std::isfinite(gx[s]) || !std::isfinite(gy[s])) return best;
    }
    // directions w of at most length sqrt(5) with an axis v that completes them to a basis
    const int cand[8][4] = {{0, 1, 1, 0}, {1, 0, 0, 1}, {1, 1, 1, 0}, {-1, 1, 1, 0},
                            {2, 1, 1, 0}, {-2, 1, 1, 0}, {1, 2, 0, 1}, {-1, 2, 0, 1}};
    double least = INFINITY;
    for (const auto& c : cand) {
        double cost = 0.0;
        for (size_t s = 0; s < S; ++s) cost += run_cost(std::fabs(c[0] * gx[s] + c[1] * gy[s]));
        // blocks that straddle the image's edges: their extent along x and y, over the image's
        const double bx = 16.0 * (std::abs(c[0]) + std::abs(c[2])), by = 16.0 * (std::abs(c[1]) + std::abs(c[3]));
        cost *= (1.0 + 0.5 * bx / nx) * (1.0 + 0.5 * by / ny);
        if (cost < least) {
            least = cost;
            best.wx = c[0];
            best.wy = c[1];
            best.vx = c[2];
            best.vy = c[3];
        }
    }
    // Window: for a pixel at d from its block's anchor (|line| <= lines / 2, |offset| <= 8) an antenna's range
    // moves by at most |u.d| + |d|^2 / (2 R), u the unit vector at the anchor.  u is taken at the centres
    // of 4 x 4 cells of the scene, where it changes by at most Dc / R towards any anchor of the cell (Dc its
    // half-diagonal and a block's).  Lines are halved until the windows leave room for three CTAs per SM.
    double ea[3], eb[3];
    for (int d = 0; d < 3; ++d) {
        ea[d] = best.vx * ex[d] + best.vy * ey[d];
        eb[d] = best.wx * ex[d] + best.wy * ey[d];
    }
    auto len = [](const double* v) { return std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]); };
    const double block = 8.0 * (len(ea) + len(eb));
    const double Dc = 0.125 * (nx * len(ex) + ny * len(ey)) + 0.5 * nz * len(ez) + 2.0 * block;
    std::vector<double> ra(S, 0.0), rb(S, 0.0), rest(S, 0.0);   // largest rates and D / R of each pulse
    double nearest = INFINITY;
    for (size_t s = 0; s < S; ++s)
        for (int cell = 0; cell < 16; ++cell) {
            const double fx = ((cell & 3) + 0.5) / 4.0 * (nx - 1), fy = ((cell >> 2) + 0.5) / 4.0 * (ny - 1);
            double a = 0.0, b = 0.0, q = 0.0;
            for (int ant = 0; ant < 2; ++ant) {
                const double* p = (ant ? rx : tx) + 3 * s;
                double u[3];
                for (int d = 0; d < 3; ++d)
                    u[d] = p[d] - (origin[d] + fx * ex[d] + fy * ey[d] + 0.5 * (nz - 1) * ez[d]);
                const double r = len(u), R = r - Dc;
                if (!(R > 0.0)) return best;
                nearest = std::min(nearest, R);
                a += std::fabs(u[0] * ea[0] + u[1] * ea[1] + u[2] * ea[2]) / r;
                b += std::fabs(u[0] * eb[0] + u[1] * eb[1] + u[2] * eb[2]) / r;
                q += Dc / R;
            }
            ra[s] = std::max(ra[s], a);
            rb[s] = std::max(rb[s], b);
            rest[s] = std::max(rest[s], q);
        }
    for (best.lines = 16; best.lines >= 2; best.lines /= 2) {
        const double ha = 0.5 * best.lines, hb = 8.0, reach = ha * len(ea) + hb * len(eb);
        double h = 0.0;
        for (size_t s = 0; s < S; ++s)
            h = std::max(h, ha * ra[s] + hb * rb[s] + reach * rest[s] + reach * reach / nearest);
        h = h * s_r + 0.1;
        if (!(h < 4096.0)) continue;
        // taps from half a bin (the anchor's fraction), half a bin of rounding and kDip below to two bins above
        best.half = (int)std::ceil(h + 1.0 + kDip);
        best.slots = best.half + (int)std::ceil(h + 4.0);
        if (scatter_smem(best.slots, best.lines).total <= 75 * 1024) {
            best.ok = true;
            break;
        }
    }
    if (best.ok) scatter_items(S, nx, ny, nz, &best);
    return best;
}

}  // namespace sar
