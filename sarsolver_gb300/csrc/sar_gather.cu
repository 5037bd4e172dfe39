// sar_gather.cu -- backprojection of a regular grid, linear sampling with plain bins: gather along iso-range lines (K2).
//
// A thread keeps 16 pixels of one lattice line (sar_lattice.h: the lines follow the direction along which range
// changes least) and runs over the pulses.  Down such a line a pulse's range bin usually moves by less than one,
// so the 16 samples interpolate between three neighbouring bins p0, p1, p2, loaded once: with a the sample's
// position about the middle one,
//     value = p1 + a (p2 - p0) / 2 + |a| ((p0 + p2) / 2 - p1),
// two FMAs per component and no address, no load and no rounding per pixel.  Where the bin moves faster the line
// is cut into runs of 8 or 4 pixels, and where it moves by most of a bin per pixel each sample loads its own two.
// Two neighbouring pixels share each packed FP32 instruction.
//
// CTA: a tile of 32 lines x 16 pixels per gathering warp (8 or 4 warps; a lane per line, so the lanes' window
// loads run along the range axis), and one producer warp per four.  The producers expand range about the centre
// of every 16 x 16 sub-tile and pulse (as the other grid kernels), classify the runs, and copy each pulse's
// profile window (plain values) with a bulk copy on the stage's mbarrier; stages are double buffered.  Every wait
// is bounded (FLAG_WAIT_TIMEOUT), and each sub-tile's bins are proven to lie in the window (FLAG_GATHER_WINDOW,
// the set then zeroed).
//
// Where the tiles do not fill the GPU, `parts` CTAs share a tile's pulses; each writes its own partial image and
// a second kernel adds them in a fixed order, so results are bitwise reproducible for any number of parts.
//
// Bound: the special-function and FMA pipes (4 sine / cosine operations and 13 packed FMAs per two pixel-pulses).
// Measured figures stand at launch_gather.
#include <algorithm>
#include <cmath>

#include "sar_gather.cuh"
#include "sar_pipe.cuh"

namespace sar {

namespace {

#define GA_TWO_PI 6.28318530717958647692f

constexpr float kRunSpan = 0.98f;   // bins a run of pixels may span (its taps then lie in three bins)
constexpr float kDip = 0.1f;        // bins a run may fall below its end points (curvature)
constexpr int kSumPulses = 512;     // pulses summed in registers at a time
constexpr int kSetFloats = 20;      // floats per coefficient set (neighbouring sets then fall on distinct banks)

__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }

// One pulse onto a thread's 16 pixels (pairs ar[k], ai[k]: offsets 2 k - 8, 2 k - 7).  cs: the sub-tile's set
// [c0 .. c9 v0 .. v5 h], all phase coefficients but c0, c1, c3, c6 in radians; u: the line's offset; w: the pulse's
// window at its base bin.  G: pixels per run, 0: two loads per pixel.
//
// c2 is reduced to half turns: c2 = c2' + w2 with |c2'| <= 1/4 and w2 a multiple of 1/2, whose part w2 d is a whole
// number of turns at even offsets and h = w2 mod 1 at odd ones, the two halves of a pair.  A line's phases stay
// below ~2.5 turns instead of 4.5, and FP32 rounds them to half the error (512^2 x 1024 against 64 bits: 5.5e-7
// instead of 7.2e-7; quarter turns of c1 and c2: 5.3e-7, 2 % slower).
template <int G>
__device__ __forceinline__ void gather_line(const float4* cs, float u, const float2* w, float2 (&ar)[8], float2 (&ai)[8]) {
    const float4 A = cs[0], B = cs[1], C = cs[2], D = cs[3];
    const float h = reinterpret_cast<const float*>(cs)[16];
    float p0 = fmaf(fmaf(fmaf(B.z, u, A.w), u, A.y), u, A.x);
    p0 -= rintf(p0);
    const float2 P0 = mul2(mk(p0, p0 + h), dup(GA_TWO_PI));
    const float2 P1 = dup(fmaf(fmaf(B.w, u, B.x), u, A.z)), P2 = dup(fmaf(C.x, u, B.y)), P3 = dup(C.y);
    const float cv = fmaf(fmaf(D.y, u, C.w), u, C.z), bv1 = fmaf(D.z, u, D.x), bv2 = D.w;
    const float2 V1 = dup(bv1), V2 = dup(bv2);
    auto add = [&](int k, float2 d, float2 re, float2 im) {
        const float2 ph = fma2(fma2(fma2(P3, d, P2), d, P1), d, P0);
        float2 sn, cn;
        __sincosf(ph.x, &sn.x, &cn.x);
        __sincosf(ph.y, &sn.y, &cn.y);
        ar[k] = fma2(re, cn, fma2(im, sn, ar[k]));
        ai[k] = fma2(im, cn, fma2(mk(-re.x, -re.y), sn, ai[k]));
    };
    if constexpr (G > 0) {
        constexpr int GG = G > 0 ? G : 1;
        const float dip = 0.25f * (G - 1) * (G - 1) * fabsf(bv2);
#pragma unroll
        for (int g0 = 0; g0 < kGatherWalk; g0 += GG) {
            const float da = (float)(g0 - 8), db = (float)(g0 + G - 9);
            const float r = (fminf(fmaf(fmaf(bv2, da, bv1), da, cv), fmaf(fmaf(bv2, db, bv1), db, cv)) - dip) + SAR_SHIFTER;
            const float2* q = w + (__float_as_int(r) - SAR_SHIFTER_BITS);
            const float2 q0 = q[0], q1 = q[1], q2 = q[2];
            const float2 VA = dup((cv - (r - SAR_SHIFTER)) - 0.5f);   // a = v - (n0 + 1/2)
            const float2 h0 = mul2(q0, dup(0.5f)), h2 = mul2(q2, dup(0.5f));
            const float2 slope = add2(h2, mk(-h0.x, -h0.y)), kink = add2(add2(h0, h2), mk(-q1.x, -q1.y));
            const float2 Ar = dup(q1.x), Ai = dup(q1.y), Br = dup(slope.x), Bi = dup(slope.y), Cr = dup(kink.x), Ci = dup(kink.y);
#pragma unroll
            for (int k = g0 / 2; k < (g0 + G) / 2; ++k) {
                const float2 d = mk((float)(2 * k - 8), (float)(2 * k - 7));
                const float2 av = fma2(fma2(V2, d, V1), d, VA), aa = mk(fabsf(av.x), fabsf(av.y));
                add(k, d, fma2(av, Br, fma2(aa, Cr, Ar)), fma2(av, Bi, fma2(aa, Ci, Ai)));
            }
        }
    } else {
        const float2 CV = dup(cv), SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float2 d = mk((float)(2 * k - 8), (float)(2 * k - 7));
            const float2 v = fma2(fma2(V2, d, V1), d, CV), r = add2(v, SH);
            const float2 t = add2(fma2(add2(r, NSH), M1, v), dup(0.5f));
            const float2 *qa = w + (__float_as_int(r.x) - SAR_SHIFTER_BITS), *qb = w + (__float_as_int(r.y) - SAR_SHIFTER_BITS);
            const float2 a0 = qa[0], a1 = qa[1], b0 = qb[0], b1 = qb[1];
            add(k, d, fma2(t, mk(a1.x - a0.x, b1.x - b0.x), mk(a0.x, b0.x)), fma2(t, mk(a1.y - a0.y, b1.y - b0.y), mk(a0.y, b0.y)));
        }
    }
}

struct GatherSmem {
    size_t coef, meta, bars, anchors, total;
    int wst;   // float2 per window: ww + 2 values, so that every copy can start at an even bin
};
__host__ __device__ inline GatherSmem gather_smem(int warps, int ww, int pb) {
    GatherSmem L;
    L.wst = ww + 2;
    L.coef = (size_t)2 * pb * L.wst * sizeof(float2);
    L.meta = L.coef + (size_t)2 * pb * 2 * warps * kSetFloats * sizeof(float);
    L.bars = L.meta + (size_t)2 * pb * sizeof(int4);
    L.anchors = L.bars + 4 * sizeof(uint64_t);
    L.total = L.anchors + (size_t)2 * warps * sizeof(df3);
    return L;
}

}  // namespace

template <int NW>
__global__ void __launch_bounds__(32 * (NW + NW / 4), NW == 8 ? 2 : 4) gather_kernel(const GatherArgs a) {
    extern __shared__ __align__(16) unsigned char gsm[];
    constexpr int NP = NW / 4, NS = 2 * NW, PP = 32 / NS;   // producer warps, sub-tiles, pulses per producer pass
    const GatherSmem L = gather_smem(NW, a.ww, a.pb);
    const int pb = a.pb, ww = a.ww;
    float2* win0 = reinterpret_cast<float2*>(gsm);
    float* coef0 = reinterpret_cast<float*>(gsm + L.coef);
    int4* meta0 = reinterpret_cast<int4*>(gsm + L.meta);   // (base bin, then bits 2 w: warp w runs 16 / 8 / 4)
    uint64_t* bars = reinterpret_cast<uint64_t*>(gsm + L.bars);   // full[0..1], empty[2..3]
    df3* anchors = reinterpret_cast<df3*>(gsm + L.anchors);
    const int4 tile = __ldg(a.tiles + blockIdx.x / a.parts);
    const int part = blockIdx.x % a.parts;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < NS) {
        const int la = tile.x + 8 + 16 * (threadIdx.x & 1), lb = tile.y + 8 + 16 * (threadIdx.x >> 1);
        anchors[threadIdx.x] = pixel_position(a.vx * la + a.wx * lb, a.vy * la + a.wy * lb, tile.z, a.img);
    }
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], NP);
        mbar_init(&bars[1], NP);
        mbar_init(&bars[2], NW);
        mbar_init(&bars[3], NW);
        mbar_fence_init();
    }
    __syncthreads();
    // this CTA's share of the pulse stages: global stage st0 + st for local stage st
    const int nst_all = (a.S + pb - 1) / pb;
    const int st0 = (int)((long)part * nst_all / a.parts), nst = (int)((long)(part + 1) * nst_all / a.parts) - st0;

    if (warp >= NW) {
        // ----------------------------------------------------------- producers
        const int pw = warp - NW, q = lane % NS;
        const df3 anchor = anchors[q];
        bool ok = true;
        int issued = 0;
        for (int st = 0; st < nst; ++st) {
            const int b = st & 1;
            if (st >= 2 && !mbar_wait(&bars[2 + b], ((st - 2) >> 1) & 1, 128, 2048, a.wait_budget)) {
                ok = false;
                break;
            }
            if (st == 0 && a.hold_first_stage) {   // nothing computed, copied or arrived for it
                issued = 1;
                continue;
            }
            const int s0 = (st0 + st) * pb, npb = min(pb, a.S - s0);
            float* coef = coef0 + (size_t)b * pb * NS * kSetFloats;
            int4* meta = meta0 + b * pb;
            int mine = 0;   // pulses of this stage staged by this warp
            for (int pass = pw * PP; pass < npb; pass += NP * PP) {
                const int pi = pass + lane / NS;
                const bool valid = pi < npb;
                const PulseGeom pg = load_pulse(a.pulses + s0 + min(pi, npb - 1));
                const AnchorExpansion ae = expand_anchor(anchor, pg, a.lat);
                Coeffs co;
                phase_coeffs(ae, a.lat, co.c);
                const df vb = anchor_bin(ae, a.lat);
                df sum = vb;   // the tile's base bin: floor of the sub-tiles' mean
#pragma unroll
                for (int o = 1; o < NS; o *= 2)
                    sum = df_add(sum, df_make(__shfl_xor_sync(0xffffffffu, sum.hi, o), __shfl_xor_sync(0xffffffffu, sum.lo, o)));
                const int base = __shfl_sync(0xffffffffu, base_bin_of(sum, (float)NS), lane - q);
                bin_coeffs(ae, vb, base, a.lat, co);
                // every tap (n0 .. n0 + 2) inside the staged window [-ww / 2, ww / 2]
                const float ext = 8.f * (fabsf(co.v[1]) + fabsf(co.v[2])) + 64.f * (fabsf(co.v[3]) + fabsf(co.v[4]) + fabsf(co.v[5]));
                if (!(co.v[0] - ext - 0.5f - kDip >= -(float)(ww / 2) && co.v[0] + ext + 2.5f <= (float)(ww / 2))) {
                    if (valid) raise_flag(a.flags, FLAG_GATHER_WINDOW);
                    co = Coeffs{};   // invalid result (flagged); every index is then the window's middle
                }
                // runs: the bin moves by less than kRunSpan over G pixels of a line
                const float rate = fabsf(co.v[2]) + 8.f * fabsf(co.v[4]) + 16.f * fabsf(co.v[5]), c2 = fabsf(co.v[5]);
                const unsigned m16 = __ballot_sync(0xffffffffu, 15.f * rate + 56.25f * c2 < kRunSpan && 56.25f * c2 < kDip);
                const unsigned m8 = __ballot_sync(0xffffffffu, 7.f * rate + 12.25f * c2 < kRunSpan && 12.25f * c2 < kDip);
                const unsigned m4 = __ballot_sync(0xffffffffu, 3.f * rate + 2.25f * c2 < kRunSpan && 2.25f * c2 < kDip);
                if (valid) {
                    float4* dst = reinterpret_cast<float4*>(coef + (size_t)(pi * NS + q) * kSetFloats);
                    const float K = GA_TWO_PI;
                    const float w2 = 0.5f * rintf(2.f * co.c[2]);
                    reinterpret_cast<float*>(dst)[16] = w2 - rintf(w2);
                    dst[0] = make_float4(co.c[0], co.c[1], (co.c[2] - w2) * K, co.c[3]);
                    dst[1] = make_float4(co.c[4] * K, co.c[5] * K, co.c[6], co.c[7] * K);
                    dst[2] = make_float4(co.c[8] * K, co.c[9] * K, co.v[0], co.v[1]);
                    dst[3] = make_float4(co.v[2], co.v[3], co.v[4], co.v[5]);
                    if (q == 0) {
                        const int sh = lane;   // this pulse's sub-tiles are ballot bits lane .. lane + NS - 1
                        auto both = [&](unsigned m) { m >>= sh; return (int)(m & (m >> 1)); };
                        meta[pi] = make_int4(base, both(m16), both(m8), both(m4));
                    }
                }
                mine += min(PP, npb - pass);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_expect_tx(&bars[b], (uint32_t)(mine * L.wst * sizeof(float2)));
            for (int pass = pw * PP; pass < npb; pass += NP * PP) {
                const int pi = pass + lane;
                if (lane < PP && pi < npb) {
                    long g0 = ((long)meta[pi].x - ww / 2 - a.bg0) & ~1L;
                    const long last = ((long)a.Lg - L.wst) & ~1L;
                    if (g0 < 0 || g0 > last) {
                        raise_flag(a.flags, FLAG_TILE_WINDOW);
                        g0 = g0 < 0 ? 0 : last;
                    }
                    fence_proxy_async_smem();
                    bulk_g2s(win0 + (size_t)(b * pb + pi) * L.wst, a.prof + (size_t)(s0 + pi) * a.Lg + g0,
                             (uint32_t)(L.wst * sizeof(float2)), &bars[b]);
                }
            }
            issued = st + 1;
        }
        // drain: wait (with the full budget) for this warp's own copies of the last two stages, so that no bulk
        // copy into this CTA's shared memory is in flight when it exits
        for (int st = max(0, issued - 2); st < issued; ++st)
            if (!(st == 0 && a.hold_first_stage) && !mbar_wait(&bars[st & 1], (st >> 1) & 1, 128, 2048)) ok = false;
        if (!ok && lane == 0) raise_flag(a.flags, FLAG_WAIT_TIMEOUT);
        return;
    }

    // -------------------------------------------------------------- gathering warps
    const int half = lane >> 4;
    const float u = (float)(lane - 8 - 16 * half);
    float2 ar[8], ai[8];
    // one FP32 sum over thousands of pulses would lose accuracy: after every kSumPulses the sums are added to the
    // thread's pixels in memory and start from zero
    const int every = max(1, kSumPulses / pb);
    for (int st = 0; st < nst;) {
        const int begin = st, end = min(nst, st + every);
#pragma unroll
        for (int k = 0; k < 8; ++k) ar[k] = ai[k] = dup(0.f);
        for (; st < end; ++st) {
            const int b = st & 1;
            if (!mbar_wait(&bars[b], (st >> 1) & 1, 32, 256, a.wait_budget)) {
                if (lane == 0) raise_flag(a.flags, FLAG_WAIT_TIMEOUT);
                return;
            }
            const int npb = min(pb, a.S - (st0 + st) * pb);
            const float4* cs = reinterpret_cast<const float4*>(coef0 + ((size_t)b * pb * NS + 2 * warp + half) * kSetFloats);
            const float2* win = win0 + (size_t)b * pb * L.wst + ww / 2;
            const int4* meta = meta0 + b * pb;
#pragma unroll 1
            for (int pi = 0; pi < npb; ++pi) {
                const int4 m = meta[pi];
                const float2* w = win + ((m.x - ww / 2 - a.bg0) & 1);   // the copy starts at an even bin
                if ((m.y >> (2 * warp)) & 1)
                    gather_line<16>(cs, u, w, ar, ai);
                else if ((m.z >> (2 * warp)) & 1)
                    gather_line<8>(cs, u, w, ar, ai);
                else if ((m.w >> (2 * warp)) & 1)
                    gather_line<4>(cs, u, w, ar, ai);
                else
                    gather_line<0>(cs, u, w, ar, ai);
                cs += NS * kSetFloats / 4;
                win += L.wst;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[2 + b]);
        }
        float2* out = a.parts > 1 ? a.partial + (size_t)part * a.pixels : a.x;
        const bool add = begin > 0 || (a.parts == 1 && a.accumulate);
        // (opaque: 16 addresses computed ahead of the pulse loop would not fit its registers)
        int la = tile.x + lane, lb = tile.y + kGatherWalk * warp;
        asm volatile("" : "+r"(la), "+r"(lb));
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int i = a.vx * la + a.wx * (lb + k), j = a.vy * la + a.wy * (lb + k);
            if (i < 0 || i >= a.img.nx || j < 0 || j >= a.img.ny) continue;
            float2 v = (k & 1) ? mk(ar[k / 2].y, ai[k / 2].y) : mk(ar[k / 2].x, ai[k / 2].x);
            float2* dst = out + ((size_t)tile.z * a.img.ny + j) * a.img.nx + i;
            if (add) v = add2(v, *dst);
            *dst = v;
        }
    }
}

// x (+)= sum of the partial images, in order.
__global__ void __launch_bounds__(256) sum_parts_kernel(const float2* __restrict__ partial, float2* __restrict__ x,
                                                        size_t pixels, int parts, int accumulate) {
    for (size_t p = blockIdx.x * (size_t)256 + threadIdx.x; p < pixels; p += (size_t)gridDim.x * 256) {
        float2 v = accumulate ? x[p] : make_float2(0.f, 0.f);
        for (int k = 0; k < parts; ++k) {
            const float2 q = __ldg(partial + (size_t)k * pixels + p);
            v.x += q.x;
            v.y += q.y;
        }
        x[p] = v;
    }
}

cudaError_t launch_sum_parts(const float2* partial, float2* x, size_t pixels, int parts, int accumulate, cudaStream_t st) {
    sum_parts_kernel<<<(unsigned)std::min<size_t>((pixels + 255) / 256, 152 * 8), 256, 0, st>>>(partial, x, pixels, parts,
                                                                                             accumulate);
    return cudaGetLastError();
}

// Measured (GB300, this kernel alone, against the tile gather before): 2048^2 x 4096 pulses 12.4 ms (14.3);
// 1024^2 x 2048 1.52 ms (1.88); 512^2 x 1024 0.22 ms (0.28).  19.6 instructions per pixel-pulse, of which the
// producers' about 2; issue 64 %, FMA pipe 62 %, special functions 57 % of their cycles.  Tried: sign and
// magnitude on the integer pipe, 3 % slower; without the phase's cubic term along the line 2 % faster (not kept: a
// second copy of the body); totals in shared memory instead of the image every 512 pulses, 13.7 ms (registers).
cudaError_t launch_gather(const GatherArgs& a, cudaStream_t st) {
    if (a.num_tiles < 1 || a.parts < 1 || (a.parts > 1 && !a.partial) || (a.Lg & 1) || a.Lg < a.ww + 2) return cudaErrorInvalidValue;
    const size_t smem = gather_smem(a.warps, a.ww, a.pb).total;
    auto go = [&](auto kern, int threads) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)(a.num_tiles * a.parts), threads, smem, st>>>(a);
        return cudaGetLastError();
    };
    cudaError_t e = a.warps == 8 ? go(gather_kernel<8>, 320) : a.warps == 4 ? go(gather_kernel<4>, 160) : cudaErrorInvalidValue;
    return e != cudaSuccess || a.parts == 1 ? e : launch_sum_parts(a.partial, a.x, a.pixels, a.parts, a.accumulate, st);
}

// ------------------------------------------------------------------ layout
namespace {

constexpr size_t kPartialBytes = (size_t)256 << 20;   // partial images of a plan

// Instructions per pixel-pulse by run length, for the choice of lattice only.
double run_cost(double rate) {
    return 15.0 * rate < kRunSpan ? 14.0 : 7.0 * rate < kRunSpan ? 16.0 : 3.0 * rate < kRunSpan ? 20.0 : 26.0;
}

// Estimated seconds of `count` pulses over `tiles` tiles with `parts` CTAs each: whole waves of CTAs at 1.5e12
// pixel-pulses per second, one stage to fill each CTA's pipeline, and the sum of the partial images.
double gather_seconds(size_t tiles, int warps, int pb, size_t count, int parts, size_t pixels) {
    const double slots = 152.0 * (warps == 8 ? 2 : 4), nst = std::ceil((double)count / pb);
    const double stage = pb * (double)kGatherLines * kGatherWalk * warps * slots / 1.5e12;
    return std::ceil(tiles * (double)parts / slots) * (std::ceil(nst / parts) + 1.0) * stage +
           (parts > 1 ? 2e-6 + 16.0 * pixels * parts / 5e12 : 0.0);
}

int best_parts(size_t tiles, int warps, int pb, size_t count, size_t pixels, int most, double* seconds) {
    const int nst = (int)((count + pb - 1) / pb);
    int best = 1;
    *seconds = INFINITY;
    for (int p = 1; p <= std::min(most, nst); ++p) {
        const double t = gather_seconds(tiles, warps, pb, count, p, pixels);
        if (t < *seconds * 0.99) {
            *seconds = t;
            best = p;
        }
    }
    return best;
}

}  // namespace

int gather_parts(const GatherLayout& L, size_t count, size_t pixels) {
    double t;
    return best_parts(L.tiles.size(), L.warps, L.pb, count, pixels, L.parts, &t);
}

GatherLayout gather_layout(const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                           const double* ey, const double* ez, int nx, int ny, int nz, double s_r) {
    GatherLayout best;
    const Lattice lattice = choose_lattice(tx, rx, S, origin, ex, ey, ez, nx, ny, nz, s_r, kGatherLines, 64, run_cost);
    if (!lattice.ok) return best;
    const size_t pixels = (size_t)nx * ny * nz;
    const int most = (int)std::min<size_t>(16, std::max<size_t>(1, kPartialBytes / (pixels * sizeof(float2))));
    double least = INFINITY;
    for (int warps : {8, 4}) {
        const LatticeBounds B = lattice_bounds(lattice, tx, rx, S, origin, ex, ey, ez, nx, ny, nz, 16.0, 8.0 * warps);
        if (!B.ok) return best;
        // a tap from the excursion of the tile's pixels about its mean bin, plus the base's fraction and rounding
        const double h = B.excursion(16.0, 8.0 * warps, s_r) + 0.1;
        if (!(h < 4096.0)) continue;
        const int ww = 2 * (int)std::ceil(h + 3.5 + kDip);
        std::vector<int4> tiles;
        for (int k = 0; k < nz; ++k)
            for (const LatticeStrip& t : lattice_strips(lattice, kGatherLines, nx, ny))
                for (long b = t.b0; b <= t.b1; b += kGatherWalk * warps) tiles.push_back(make_int4(t.a0, (int)b, k, 0));
        for (int pb : {16, 8, 4}) {
            if (gather_smem(warps, ww, pb).total > (size_t)(warps == 8 ? 110 : 55) * 1024) continue;
            double t;
            const int parts = best_parts(tiles.size(), warps, pb, S, pixels, most, &t);
            if (t < 0.97 * least) {
                least = t;
                best.warps = warps;
                best.ww = ww;
                best.pb = pb;
                best.parts = parts;
                best.tiles = tiles;
                best.ok = true;
            }
        }
    }
    best.lattice = lattice;
    return best;
}

}  // namespace sar
