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

#include "sar_kernels.cuh"
#include "sar_pipe.cuh"
#include "sar_scatter.cuh"

namespace sar {

namespace {

#define SC_TWO_PI 6.28318530717958647692f

__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }

constexpr float kRunSpan = 0.98f;   // bins a run of pixels may span (its taps then lie in three bins)
constexpr float kDip = 0.1f;        // bins a run may fall below its end points (curvature)

// A block's set with the phase's linear coefficients reduced: c1 = c1' + w1 with |c1'| <= 1/8 and w1 a multiple of 1/4
// (w1 di is exact and dropped to its fraction); c2 = c2' + w2 with |c2'| <= 1/4 and w2 a multiple of 1/2, whose part
// w2 d is a whole number of turns at even offsets and h = w2 mod 1 at odd ones.  A line's phases stay below ~2.5
// turns instead of 4.5, and FP32 rounds them to half the error (512^2 x 1024 against 64 bits: 5.5e-7 instead of 7.8e-7).
struct BlockSet {
    Coeffs co;
    float w1, h;
};

__device__ __forceinline__ void reduce_turns(BlockSet& q) {
    q.w1 = 0.25f * rintf(4.f * q.co.c[1]);
    const float w2 = 0.5f * rintf(2.f * q.co.c[2]);
    q.co.c[1] -= q.w1;
    q.co.c[2] -= w2;
    q.h = w2 - rintf(w2);
}

// Terms of two neighbouring lines (a, a + 1): phase cph[d mod 2] + b1 d + b2 d^2 + c9 d^3 in radians and bin
// cv + bv1 d + bv2 d^2, d the offset along the line.
struct LinePair {
    float2 cph[2], b1, b2, c9, cv, bv1, bv2;
};

__device__ __forceinline__ LinePair line_pair(const BlockSet& q, float di) {
    const Coeffs& co = q.co;
    const float2 D = mk(di, di + 1.f), K = dup(SC_TWO_PI), SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
    LinePair t;
    float2 w = mul2(dup(q.w1), D);
    w = fma2(add2(add2(w, SH), NSH), M1, w);   // mod 1, exact
    const float2 ph = add2(fma2(fma2(fma2(dup(co.c[6]), D, dup(co.c[3])), D, dup(co.c[1])), D, dup(co.c[0])), w);
    t.cph[0] = mul2(ph, K);
    t.cph[1] = mul2(add2(ph, dup(q.h)), K);
    t.b1 = mul2(fma2(fma2(dup(co.c[7]), D, dup(co.c[4])), D, dup(co.c[2])), K);
    t.b2 = mul2(fma2(dup(co.c[8]), D, dup(co.c[5])), K);
    t.c9 = dup(co.c[9] * SC_TWO_PI);
    t.cv = fma2(fma2(dup(co.v[3]), D, dup(co.v[1])), D, dup(co.v[0]));
    t.bv1 = fma2(dup(co.v[4]), D, dup(co.v[2]));
    t.bv2 = dup(co.v[5]);
    return t;
}

// c = x exp(i phase) for the two lines' pixels at offset rr - 8 (XN = -im).
__device__ __forceinline__ void contribution(const LinePair& t, int rr, float2 d, float4 X, float2 XN, float2* cr, float2* ci) {
    const float2 ph = fma2(fma2(fma2(t.c9, d, t.b2), d, t.b1), d, t.cph[rr & 1]);
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
__device__ __forceinline__ void walk_runs(const BlockSet& q, const float4* xs, const float2* xn, float2* win, int off, int W,
                                          int lines) {
    const float2 SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
    const float2 ndip = dup(-0.25f * (G - 1) * (G - 1) * fabsf(q.co.v[5]));
#pragma unroll 1
    for (int l = 0; l < lines / 2; ++l) {
        const LinePair t = line_pair(q, (float)(2 * l - lines / 2));
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
                contribution(t, rr, d, xl[rr], nl[rr], &cr, &ci);
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
__device__ __forceinline__ void walk_taps(const BlockSet& q, const float4* xs, const float2* xn, float2* win, int off, int W,
                                          int lines) {
    const float2 SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
#pragma unroll 1
    for (int l = 0; l < lines / 2; ++l) {
        const LinePair t = line_pair(q, (float)(2 * l - lines / 2));
        const float4* xl = xs + l * kWalk;
        const float2* nl = xn + l * kWalk;
#pragma unroll 4
        for (int rr = 0; rr < kWalk; ++rr) {
            const float2 d = dup((float)(rr - 8));
            float2 cr, ci;
            contribution(t, rr, d, xl[rr], nl[rr], &cr, &ci);
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
        BlockSet set;
        Coeffs& co = set.co;
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
        reduce_turns(set);
        // runs: the bin moves by less than kRunSpan over G pixels of a line (|rate| over the block, plus the
        // fall below the end points)
        const float rate = fabsf(co.v[2]) + 8.f * fabsf(co.v[4]) + 16.f * fabsf(co.v[5]), c2 = fabsf(co.v[5]);
        const int off = rot + a.half;   // slot of bin n (about the base) is wrap(n + off)
        const float4* bx = xs + (blk & 1) * block_px;
        const float2* bn = xn + (blk & 1) * block_px;
        if (__all_sync(0xffffffffu, 15.f * rate + 56.25f * c2 < kRunSpan && 56.25f * c2 < kDip))
            walk_runs<16>(set, bx, bn, win, off, W, a.lines);
        else if (__all_sync(0xffffffffu, 7.f * rate + 12.25f * c2 < kRunSpan && 12.25f * c2 < kDip))
            walk_runs<8>(set, bx, bn, win, off, W, a.lines);
        else if (__all_sync(0xffffffffu, 3.f * rate + 2.25f * c2 < kRunSpan && 2.25f * c2 < kDip))
            walk_runs<4>(set, bx, bn, win, off, W, a.lines);
        else
            walk_taps(set, bx, bn, win, off, W, a.lines);
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
// The CTAs' runs of blocks: each strip of `lines` lattice lines cut into segments so that a launch has about
// five waves of CTAs.
static long segment_blocks(long blocks, size_t S, int nz) {
    const size_t groups = (S + 32 * kScatterWarps - 1) / (32 * kScatterWarps);
    return std::max<long>(1, (long)((double)blocks * nz * groups / (152.0 * 3 * 5)));
}

static void scatter_items(size_t S, int nx, int ny, int nz, ScatterLayout* L) {
    const std::vector<LatticeStrip> strips = lattice_strips(L->lattice, L->lines, nx, ny);
    long total = 0;
    for (const LatticeStrip& t : strips) total += (t.b1 - t.b0) / kWalk + 1;
    const long len = segment_blocks(total, S, nz);
    L->items.clear();
    for (int k = 0; k < nz; ++k)
        for (const LatticeStrip& t : strips) {
            const long n = (t.b1 - t.b0) / kWalk + 1, cuts = (n + len - 1) / len;
            for (long c = 0; c < cuts; ++c) {
                const long p = n * c / cuts, q = n * (c + 1) / cuts;
                L->items.push_back(make_int4(t.a0, (int)(t.b0 + p * kWalk), (int)(q - p), k));
            }
        }
}

// Lines per block: halved until the windows leave room for three CTAs per SM.  h: bins from a block's anchor to its pixels.
static bool fit_lines(ScatterLayout* L, int lines, double h) {
    if (!(h < 4096.0)) return false;
    L->lines = lines;
    // taps from half a bin (the anchor's fraction), half a bin of rounding and kDip below to two bins above
    L->half = (int)std::ceil(h + 1.0 + kDip);
    L->slots = L->half + (int)std::ceil(h + 4.0);
    return scatter_smem(L->slots, lines).total <= 75 * 1024;
}

// Estimated seconds on a lattice, from the rates alone: the blocks' pixel-pulses by run length (0.4 ps with runs of 16, 0.9
// with two taps a pixel), what a block costs by itself (spread over its lines), and the slots it flushes: those the anchor
// leaves behind, and a whole window at the end of a segment.  Fitted to 840 launches, every lattice of 380 geometries
// forced in turn: 9 % rms.  Lines count most: with large rates along them 16 lines a block take 1.4 ps, two lines 10 ps.
static double scatter_seconds(const Lattice& lattice, const std::vector<LatticeRate>& rates, size_t S, int nx, int ny, int nz) {
    double v = 0.0, w = 0.0, mean = 0.0, unit = 0.0;
    for (const LatticeRate& r : rates) {
        v = std::max(v, r.v);
        w = std::max(w, r.w);
        mean += r.w / rates.size();
        unit += (15.0 * r.w < kRunSpan ? 0.42 : 7.0 * r.w < kRunSpan ? 0.6 : 3.0 * r.w < kRunSpan ? 0.64 : 0.93) / rates.size();
    }
    ScatterLayout L;
    int lines = 16;
    while (lines >= 2 && !fit_lines(&L, lines, 0.5 * lines * v + 8.0 * w + 0.1)) lines /= 2;
    if (lines < 2) return INFINITY;
    long blocks = 0;
    for (const LatticeStrip& t : lattice_strips(lattice, lines, nx, ny)) blocks += (t.b1 - t.b0) / kWalk + 1;
    const double groups = (double)((S + 32 * kScatterWarps - 1) / (32 * kScatterWarps)), len = (double)segment_blocks(blocks, S, nz);
    const double flushed = (L.slots / len + kWalk * mean) / (kWalk * lines);   // slots per pixel-pulse
    const double pulses = groups * 32 * kScatterWarps, work = (double)blocks * nz * kWalk * lines * pulses;
    const double per_sm = (double)std::min<size_t>(4, 227 * 1024 / (scatter_smem(L.slots, lines).total + 1024));
    const double waves = std::ceil(blocks * nz / len) * groups / (152.0 * per_sm);
    // few waves: a partly filled GPU, and the last wave's share
    const double fill = waves < 1.0 ? 0.6 + 0.5 / waves : waves < 1.6 ? 1.3 : waves < 3.0 ? 1.07 : 1.0;
    return 1.0e-12 * work * (unit + 2.0 * flushed + 4.1 / lines) * fill;
}

// The same for the tile kernel: 1.05, 1.2 and 1.4 ps a pixel-pulse with run windows of 16, 8 and 4 pixels along its walk,
// else 2.4 ps, or 4.8 where neighbouring lanes fall on one bin (atomics).  Strips are cut where their window, of some 480
// bins, ends.
static double tile_seconds(const ScatterTiles& t, const std::vector<LatticeRate>& rates, size_t S, size_t pixels) {
    double v = 0.0, v_mean = 0.0, w = 0.0, unit = 0.0;
    for (const LatticeRate& r : rates) {
        v = std::max(v, r.v);
        w = std::max(w, r.w);
        v_mean += r.v / rates.size();
        unit += (15.0 * r.w < kRunSpan ? 1.05 : 7.0 * r.w < kRunSpan ? 1.2 : 3.0 * r.w < kRunSpan ? 1.4 : 2.4) / rates.size();
    }
    if (unit > 1.4 && v_mean < 1.1) unit = 4.8;
    const double seg = std::max(1.0, std::floor((440.0 - 32.0 * v) / (32.0 * std::max(w, 1.0e-3))));
    const double waves = std::ceil(t.along / std::min(seg, (double)t.along)) * t.lines * std::ceil(S / 16.0) / 304.0;
    return 5.0e-6 + 1.0e-12 * S * pixels * t.cover * unit * (waves < 1.0 ? 0.75 + 0.25 / waves : 1.0);
}

// The tile kernel is taken where it is estimated at less than 0.9 of the lattice's time: mostly small images with four and
// more bins a pixel, whose blocks of few lines, a segment each, are all flush (192 x 192 x 400 pulses, 0.3 m, U = 16, 78
// degrees off an axis: 45 against 72 us), and looks along an axis with run windows.  Of 336 geometries it is a seventh;
// with the line at 1 the errors of both estimates cost what they gain.
ScatterLayout scatter_layout(const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                             const double* ey, const double* ez, int nx, int ny, int nz, double s_r, double kappa,
                             const ScatterTiles& tiles) {
    ScatterLayout L;
    const SceneRates rates = scene_rates(tx, rx, S, origin, ex, ey, ez, nx, ny, nz, s_r);
    auto seconds = [&](const Lattice& l, const std::vector<LatticeRate>& r) { return scatter_seconds(l, r, S, nx, ny, nz); };
    L.lattice = choose_lattice(rates, ex, ey, kappa, seconds);
    if (!L.lattice.ok) return L;
    const double lattice = seconds(L.lattice, lattice_rates(rates, L.lattice));
    if (tile_seconds(tiles, lattice_rates(rates, tiles.axes), S, (size_t)nx * ny * nz) < 0.9 * lattice) return L;
    const LatticeBounds B = lattice_bounds(L.lattice, tx, rx, S, origin, ex, ey, ez, nx, ny, nz, 8.0, 8.0);
    if (!B.ok) return L;
    for (int lines = 16; lines >= 2 && !L.ok; lines /= 2) L.ok = fit_lines(&L, lines, B.excursion(0.5 * lines, 8.0, s_r) + 0.1);
    if (L.ok) scatter_items(S, nx, ny, nz, &L);
    return L;
}

}  // namespace sar
