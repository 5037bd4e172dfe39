// sar_gather.cu -- backprojection of a regular grid: gather along iso-range lines (K2).
//
// Linear sampling with plain bins.  A thread keeps 16 pixels of one lattice line (sar_lattice.h: the lines follow the direction along which range
// changes least) and runs over the pulses.  Down such a line a pulse's range bin usually moves by less than one,
// so the 16 samples interpolate between three neighbouring bins p0, p1, p2, loaded once: with a the sample's
// position about the middle one,
//     value = p1 + a (p2 - p0) / 2 + |a| ((p0 + p2) / 2 - p1),
// two FMAs per component and no address, no load and no rounding per pixel.  Where the bin moves faster the line
// is cut into runs of 8 or 4 pixels, and where it moves by most of a bin per pixel each sample loads its own two.
// Two neighbouring pixels share each packed FP32 instruction.
//
// Nearest bins, and linear sampling of so fine bins that FP32 does not hold them (split bins: an exact integer part
// and a fraction).  Every sample loads its own bin, and many bins lie between neighbouring pixels across the lines.
// Here the lanes run along the line, so that their loads fall on neighbouring bins, and a thread keeps 16 pixels
// across it.  Nearest samples close to a rounding boundary are noted and decided exactly (sar_exact.cuh) after the
// sums have been written, where the noted samples are moved in memory.
//
// CTA: a tile of 32 lines x 16 pixels per gathering warp (8 or 4 warps; a lane per line, so the lanes' window
// loads run along the range axis; split bins: tiles 32 or 16 pixels across the lines, the rest of the warps along
// them), and one producer warp per four.  The producers expand range about the centre
// of every 16 x 16 sub-tile and pulse (as the other grid kernels), classify the runs, and copy each pulse's
// profile window (plain values) with a bulk copy on the stage's mbarrier; stages are double buffered.  Every wait
// is bounded (FLAG_WAIT_TIMEOUT), and each sub-tile's bins are proven to lie in the window (FLAG_GATHER_WINDOW,
// the set then zeroed).
//
// Where the tiles do not fill the GPU, `parts` CTAs share a tile's pulses; each writes its own partial image and
// a second kernel adds them in a fixed order, so results are bitwise reproducible for any number of parts.
//
// Bound: instruction issue, then the FMA and special-function pipes (4 sine / cosine operations and 13 packed FMAs
// per two pixel-pulses; split bins: 9 packed and 8 plain FMAs).
// Measured figures stand at launch_gather.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "sar_exact.cuh"
#include "sar_gather.cuh"
#include "sar_pipe.cuh"

namespace sar {

namespace {

#define GA_TWO_PI 6.28318530717958647692f

constexpr float kRunSpan = 0.98f;   // bins a run of pixels may span (its taps then lie in three bins)
constexpr float kDip = 0.1f;        // bins a run may fall below its end points (curvature)
constexpr int kSumPulses = 512;     // pulses summed in registers at a time
constexpr int kSetFloats = 24;      // floats per coefficient set, split bins
constexpr int kRunSetFloats = 20;   // floats per coefficient set, plain bins (neighbouring sets fall on distinct banks)

__device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }

// Offsets of the pixel pairs of a line, read by the packed instructions as constant operands (as immediates they
// would be moved into register pairs: 1 % of the run kernel's time, 3 % of the split ones').
__constant__ float2 kOffsets[8] = {{-8.f, -7.f}, {-6.f, -5.f}, {-4.f, -3.f}, {-2.f, -1.f}, {0.f, 1.f}, {2.f, 3.f}, {4.f, 5.f}, {6.f, 7.f}};

// One pulse onto a thread's 16 pixels (pairs ar[k], ai[k]: offsets 2 k - 8, 2 k - 7).  cs: the sub-tile's set
// [c0 .. c9 v0 .. v5 h n], all phase coefficients but c0, c1, c3, c6 in radians; u: the line's offset; w: the pulse's
// window at its base bin, n (an integer) the sub-tile's distance from it: FP32 then rounds bins of the sub-tile's own
// excursion, not of its tile's up to 128 pixels.  G: pixels per run, 0: two loads per pixel.
//
// c2 is reduced to half turns: c2 = c2' + w2 with |c2'| <= 1/4 and w2 a multiple of 1/2, whose part w2 d is a whole
// number of turns at even offsets and h = w2 mod 1 at odd ones, the two halves of a pair.  A line's phases stay
// below ~2.5 turns instead of 4.5, and FP32 rounds them to half the error (512^2 x 1024 against 64 bits: 5.5e-7
// instead of 7.2e-7; quarter turns of c1 and c2: 5.3e-7, 2 % slower).
template <int G>
__device__ __forceinline__ void gather_line(const float4* cs, float u, const float2* w, float2 (&ar)[8], float2 (&ai)[8]) {
    const float4 A = cs[0], B = cs[1], C = cs[2], D = cs[3];
    const float2 E = reinterpret_cast<const float2*>(cs)[8];
    const float h = E.x;
    w += __float_as_int(E.y);
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
                const float2 d = kOffsets[k];
                const float2 av = fma2(fma2(V2, d, V1), d, VA), aa = mk(fabsf(av.x), fabsf(av.y));
                add(k, d, fma2(av, Br, fma2(aa, Cr, Ar)), fma2(av, Bi, fma2(aa, Ci, Ai)));
            }
        }
    } else {
        const float2 CV = dup(cv), SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float2 d = kOffsets[k];
            const float2 v = fma2(fma2(V2, d, V1), d, CV), r = add2(v, SH);
            const float2 t = add2(fma2(add2(r, NSH), M1, v), dup(0.5f));
            const float2 *qa = w + (__float_as_int(r.x) - SAR_SHIFTER_BITS), *qb = w + (__float_as_int(r.y) - SAR_SHIFTER_BITS);
            const float2 a0 = qa[0], a1 = qa[1], b0 = qb[0], b1 = qb[1];
            add(k, d, fma2(t, mk(a1.x - a0.x, b1.x - b0.x), mk(a0.x, b0.x)), fma2(t, mk(a1.y - a0.y, b1.y - b0.y), mk(a0.y, b0.y)));
        }
    }
}

__device__ __forceinline__ float2 lds2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}

// Split bins: a line's bin polynomial, whose FP32 part stays below some ten bins, and its exact integer part
// nb + step d.  Coefficient sets hold [.. h i0 ia ib w0 .. w3] after the plain ones.
struct SplitLine {
    float cv, b1, b2, b3;
    int nb, step;   // nb without the shifter's bits
};
__device__ __forceinline__ SplitLine split_terms(const float4* cs, float u) {
    const float4 C = cs[2], D = cs[3], E = cs[4], F = cs[5];
    SplitLine t;
    t.cv = fmaf(fmaf(fmaf(F.x, u, D.y), u, C.w), u, C.z);
    t.b1 = fmaf(fmaf(F.y, u, D.z), u, D.x);
    t.b2 = fmaf(F.z, u, D.w);
    t.b3 = F.w;
    t.nb = __float_as_int(__fadd_rn(fmaf(E.z, u, E.y), SAR_SHIFTER)) - 2 * SAR_SHIFTER_BITS;
    t.step = __float_as_int(E.w + SAR_SHIFTER) - SAR_SHIFTER_BITS;
    return t;
}
// Bin of the line's pixel k about the window's base, and its distance s from it.
__device__ __forceinline__ int split_bin(const SplitLine& t, int k, float* s) {
    const float d = (float)(k - 8), v = fmaf(fmaf(fmaf(t.b3, d, t.b2), d, t.b1), d, t.cv), r = __fadd_rn(v, SAR_SHIFTER);
    *s = v - __fadd_rn(r, -SAR_SHIFTER);
    return __float_as_int(r) + t.nb + t.step * (k - 8);
}

// One pulse onto a thread's 16 pixels with split bins, nearest or linear; w: the pulse's window at its base bin.
// Returns the largest distance of a pixel from its bin.
template <bool NEAREST>
__device__ __forceinline__ float gather_split(const float4* cs, float u, const float2* w, float2 (&ar)[8], float2 (&ai)[8]) {
    const SplitLine t = split_terms(cs, u);
    const float4 A = cs[0], B = cs[1], C = cs[2];
    const float h = reinterpret_cast<const float*>(cs)[16];
    float p0 = fmaf(fmaf(fmaf(B.z, u, A.w), u, A.y), u, A.x);
    p0 -= __fadd_rn(__fadd_rn(p0, SAR_SHIFTER), -SAR_SHIFTER);
    const float2 P0 = mul2(mk(p0, p0 + h), dup(GA_TWO_PI));
    const float2 P1 = dup(fmaf(fmaf(B.w, u, B.x), u, A.z)), P2 = dup(fmaf(C.x, u, B.y)), P3 = dup(C.y);
    const float2 CV = dup(t.cv), V1 = dup(t.b1), V2 = dup(t.b2), V3 = dup(t.b3);
    const float2 SH = dup(SAR_SHIFTER), NSH = dup(-SAR_SHIFTER), M1 = dup(-1.f);
    // 32-bit shared-memory addresses: a shift-add and a multiply-add per load
    const uint32_t q = smem_addr(w) + 8u * (uint32_t)t.nb, step = 8u * (uint32_t)t.step;
    float far = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float2 d = kOffsets[k];
        const float2 v = fma2(fma2(fma2(V3, d, V2), d, V1), d, CV), r = add2(v, SH);
        const float2 e = fma2(add2(r, NSH), M1, v);
        const uint32_t qa = q + step * (uint32_t)(2 * k - 8) + 8u * (uint32_t)__float_as_int(r.x);
        const uint32_t qb = q + step * (uint32_t)(2 * k - 7) + 8u * (uint32_t)__float_as_int(r.y);
        float2 pa = lds2(qa), pb = lds2(qb);
        if (NEAREST) {
            far = fmaxf(far, fmaxf(fabsf(e.x), fabsf(e.y)));
        } else {
            const float2 a1 = lds2(qa + 8), b1 = lds2(qb + 8);
            const float ta = e.x + 0.5f, tb = e.y + 0.5f;
            pa = fma2(dup(ta), add2(a1, mk(-pa.x, -pa.y)), pa);
            pb = fma2(dup(tb), add2(b1, mk(-pb.x, -pb.y)), pb);
        }
        const float2 ph = fma2(fma2(fma2(P3, d, P2), d, P1), d, P0);
        float2 sn, cn;
        __sincosf(ph.x, &sn.x, &cn.x);
        __sincosf(ph.y, &sn.y, &cn.y);
        ar[k].x = fmaf(pa.x, cn.x, fmaf(pa.y, sn.x, ar[k].x));
        ar[k].y = fmaf(pb.x, cn.y, fmaf(pb.y, sn.y, ar[k].y));
        ai[k].x = fmaf(pa.y, cn.x, fmaf(-pa.x, sn.x, ai[k].x));
        ai[k].y = fmaf(pb.y, cn.y, fmaf(-pb.x, sn.y, ai[k].y));
    }
    return far;
}

struct GatherSmem {
    size_t coef, meta, bars, anchors, queue, total;
    int wst;    // float2 per window: ww + 2 values, so that every copy can start at an even bin
    int group;  // stages whose coefficients are made together
    int ring;   // such groups held
};
__host__ __device__ inline GatherSmem gather_smem(int bins, int warps, int ww, int pb) {
    GatherSmem L;
    // split bins, one producer: a pass of its lanes makes the coefficients of four pulses
    L.group = bins != GATHER_RUNS && warps == 4 && pb < 4 ? 4 / pb : 1;
    L.ring = bins == GATHER_RUNS || L.group > 1 ? 2 : 4;
    const int held = L.ring * L.group * pb;   // pulses' coefficients held
    L.wst = ww + 2;
    L.coef = (size_t)2 * pb * L.wst * sizeof(float2);
    L.meta = L.coef + (size_t)held * 2 * warps * (bins == GATHER_RUNS ? kRunSetFloats : kSetFloats) * sizeof(float);
    L.bars = L.meta + (size_t)held * sizeof(int4);
    L.anchors = L.bars + 4 * sizeof(uint64_t);
    L.queue = (L.anchors + (size_t)2 * warps * sizeof(df3) + 7) & ~(size_t)7;
    L.total = L.queue + (bins == GATHER_NEAREST ? (size_t)warps * kNearQueue * sizeof(int2) : 0);
    return L;
}

}  // namespace

template <int NW, int BINS>
__global__ void __launch_bounds__(32 * (NW + NW / 4), NW == 8 ? 2 : 4) gather_kernel(const GatherArgs a) {
    extern __shared__ __align__(16) unsigned char gsm[];
    constexpr int NP = NW / 4, NS = 2 * NW, PP = 32 / NS;   // producer warps, sub-tiles, pulses per producer pass
    constexpr bool SPLIT = BINS != GATHER_RUNS;
    constexpr int SF = SPLIT ? kSetFloats : kRunSetFloats;
    const GatherSmem L = gather_smem(BINS, NW, a.ww, a.pb);
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
        const int w = threadIdx.x >> 1;
        const int la = tile.x + 8 + 32 * (SPLIT ? w % a.across : 0) + 16 * (threadIdx.x & 1);
        const int lb = tile.y + 8 + kGatherWalk * (SPLIT ? w / a.across : w);
        anchors[threadIdx.x] = pixel_position(a.vx * la + a.wx * lb, a.vy * la + a.wy * lb, tile.z, a.img);
    }
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], SPLIT ? 1 : NP);
        mbar_init(&bars[1], SPLIT ? 1 : NP);
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
        // Plain bins: all producers share a stage.  Split bins, whose wide windows leave room for few pulses a stage:
        // two producers take the stages in turn (so each has its own window buffer and barriers), one makes the
        // coefficients of a group of G stages together; either way before waiting for the windows' buffers.  The ring's
        // next buffer is then free: with G > 1, copying the last stage of group g - 1 has shown the end of the stage
        // two before it, in group g - 2; with single stages the end of stage g - 4 has been seen in the same way.
        const int G = L.group, step = SPLIT ? G * NP : 1;
        for (int st = SPLIT ? pw * G : 0; st < nst; st += step) {
            auto buffer_free = [&](int t) {
                return t < 2 || mbar_wait(&bars[2 + (t & 1)], ((t - 2) >> 1) & 1, 128, 2048, a.wait_budget);
            };
            if (!SPLIT && !buffer_free(st)) {
                ok = false;
                break;
            }
            if (st == 0 && a.hold_first_stage) {   // nothing computed, copied or arrived for it
                issued = 1;
                continue;
            }
            const int s0 = (st0 + st) * pb, npb = min(min(G, nst - st) * pb, a.S - s0);
            const int held = (SPLIT ? st / G % L.ring : st & 1) * G * pb;
            float* coef = coef0 + (size_t)held * NS * SF;
            int4* meta = meta0 + held;
            int mine = 0;   // pulses of this stage staged by this warp
            for (int pass = SPLIT ? 0 : pw * PP; pass < npb; pass += (SPLIT ? 1 : NP) * PP) {
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
                // every tap inside the staged window [-ww / 2, ww / 2]: n0 .. n0 + 2, nearest n0 alone (its bins lie a bin
                // higher than linear ones, whose offset is -1/2, so the window's two further taps are not all left over)
                float lo, hi;
                if (SPLIT) {
                    bin_extent(co, &lo, &hi);
                } else {
                    const df rel = df_sub(vb, df_make((float)base, 0.f));
                    co.i0 = round_shift(rel.hi);
                    co.v[0] = ((rel.hi - co.i0) + rel.lo) + a.lat.bin_offset;
                    const float ext = 8.f * (fabsf(co.v[1]) + fabsf(co.v[2])) + 64.f * (fabsf(co.v[3]) + fabsf(co.v[4]) + fabsf(co.v[5]));
                    lo = co.i0 + co.v[0] - ext;
                    hi = co.i0 + co.v[0] + ext;
                }
                if (!(lo - 0.5f - kDip >= -(float)(ww / 2) && hi + (BINS == GATHER_NEAREST ? 1.5f : 2.5f) <= (float)(ww / 2))) {
                    if (valid) raise_flag(a.flags, FLAG_GATHER_WINDOW);
                    co = Coeffs{};   // invalid result (flagged); every index is then the window's middle
                }
                // runs: the bin moves by less than kRunSpan over G pixels of a line
                unsigned m16 = 0, m8 = 0, m4 = 0;
                if (!SPLIT) {
                    const float rate = fabsf(co.v[2]) + 8.f * fabsf(co.v[4]) + 16.f * fabsf(co.v[5]), c2 = fabsf(co.v[5]);
                    m16 = __ballot_sync(0xffffffffu, 15.f * rate + 56.25f * c2 < kRunSpan && 56.25f * c2 < kDip);
                    m8 = __ballot_sync(0xffffffffu, 7.f * rate + 12.25f * c2 < kRunSpan && 12.25f * c2 < kDip);
                    m4 = __ballot_sync(0xffffffffu, 3.f * rate + 2.25f * c2 < kRunSpan && 2.25f * c2 < kDip);
                }
                if (valid) {
                    float4* dst = reinterpret_cast<float4*>(coef + (size_t)(pi * NS + q) * SF);
                    const float K = GA_TWO_PI;
                    const float w2 = 0.5f * rintf(2.f * co.c[2]);
                    if (SPLIT) {
                        dst[4] = make_float4(w2 - rintf(w2), co.i0, co.ia, co.ib);
                        dst[5] = make_float4(co.w[0], co.w[1], co.w[2], co.w[3]);
                    } else {
                        reinterpret_cast<float2*>(dst)[8] = mk(w2 - rintf(w2), __int_as_float((int)co.i0));
                    }
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
            for (int t = st; t < min(nst, st + G); ++t) {
                const int first = (t - st) * pb, n = min(pb, npb - first);   // the stage's pulses of this group
                if (SPLIT && !buffer_free(t)) {
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_arrive_expect_tx(&bars[t & 1], (uint32_t)((SPLIT ? n : mine) * L.wst * sizeof(float2)));
                for (int pass = SPLIT ? 0 : pw * PP; pass < n; pass += (SPLIT ? 1 : NP) * PP) {
                    const int pi = pass + lane;
                    if (lane < PP && pi < n) {
                        long g0 = ((long)meta[first + pi].x - ww / 2 - a.bg0) & ~1L;
                        const long last = ((long)a.Lg - L.wst) & ~1L;
                        if (g0 < 0 || g0 > last) {
                            raise_flag(a.flags, FLAG_TILE_WINDOW);
                            g0 = g0 < 0 ? 0 : last;
                        }
                        fence_proxy_async_smem();
                        bulk_g2s(win0 + (size_t)((t & 1) * pb + pi) * L.wst, a.prof + (size_t)(s0 + first + pi) * a.Lg + g0,
                                 (uint32_t)(L.wst * sizeof(float2)), &bars[t & 1]);
                    }
                }
                issued = t + 1;
            }
            if (!ok) break;
        }
        // drain: wait (with the full budget) for this warp's own copies of the last two stages, so that no bulk
        // copy into this CTA's shared memory is in flight when it exits
        for (int st = max(0, issued - 2); st < issued; ++st)
            if (!(st == 0 && a.hold_first_stage) && !(SPLIT && st / G % NP != pw) && !mbar_wait(&bars[st & 1], (st >> 1) & 1, 128, 2048)) ok = false;
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
    float2* out = a.parts > 1 ? a.partial + (size_t)part * a.pixels : a.x;
    bool add = a.parts == 1 && a.accumulate;
    const int la0 = tile.x + (SPLIT ? 32 * (warp % a.across) : 0), lb0 = tile.y + kGatherWalk * (SPLIT ? warp / a.across : warp);
    auto flush = [&] {
        // (opaque: 16 addresses computed ahead of the pulse loop would not fit its registers)
        int la = la0 + lane, lb = lb0;
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
        add = true;
#pragma unroll
        for (int k = 0; k < 8; ++k) ar[k] = ai[k] = dup(0.f);
    };
    // nearest bins: notes (pulse from s0 on, lane, pixel; bin taken) of samples near a rounding boundary
    int2* queue = reinterpret_cast<int2*>(gsm + L.queue) + warp * kNearQueue;
    int notes = 0;
    auto settle = [&](int s0) {   // after a flush: moves the noted samples in memory, in the notes' order
        __syncwarp();
        for (int n0 = 0; n0 < notes; n0 += 32) {
            float2* dst = nullptr;
            float2 move = dup(0.f);
            if (n0 + lane < notes) {
                const int2 e = queue[n0 + lane];
                const int s = s0 + (e.x >> 9), la = la0 + ((e.x >> 4) & 31), lb = lb0 + (e.x & 15);
                const int i = a.vx * la + a.wx * lb, j = a.vy * la + a.wy * lb;
                if (i >= 0 && i < a.img.nx && j >= 0 && j < a.img.ny) {
                    const ExactSample x = exact_grid_sample<true>(a.steps, a.pulses, a.alpha2, a.img.kappa, a.img.s_r, a.bg0,
                                                                  BIN_ADJ_NEAREST, i, j, tile.z, s);
                    if (x.gi != e.y && min(x.gi, e.y) >= 0 && max(x.gi, e.y) < a.Lg) {
                        const float2 *row = a.prof + (size_t)s * a.Lg, to = __ldg(row + x.gi), from = __ldg(row + e.y);
                        const float re = to.x - from.x, im = to.y - from.y;
                        float sn, cn;
                        __sincosf(GA_TWO_PI * x.f, &sn, &cn);
                        move = mk(fmaf(re, cn, im * sn), fmaf(im, cn, -re * sn));
                        dst = out + ((size_t)tile.z * a.img.ny + j) * a.img.nx + i;
                    }
                }
            }
            for (unsigned m = __ballot_sync(0xffffffffu, dst != nullptr); m; m &= m - 1) {
                if (lane == __ffs(m) - 1) *dst = add2(*dst, move);
                __syncwarp();
            }
        }
        notes = 0;
        __syncwarp();
    };
#pragma unroll
    for (int k = 0; k < 8; ++k) ar[k] = ai[k] = dup(0.f);
    for (int st = 0; st < nst;) {
        const int begin = st, end = min(nst, st + every);
        for (; st < end; ++st) {
            const int b = st & 1;
            if (!mbar_wait(&bars[b], (st >> 1) & 1, 32, 256, a.wait_budget)) {
                if (lane == 0) raise_flag(a.flags, FLAG_WAIT_TIMEOUT);
                return;
            }
            const int npb = min(pb, a.S - (st0 + st) * pb);
            const int held = SPLIT ? (st / L.group % L.ring * L.group + st % L.group) * pb : b * pb;
            const float4* cs = reinterpret_cast<const float4*>(coef0 + ((size_t)held * NS + 2 * warp + half) * SF);
            const float2* win = win0 + (size_t)b * pb * L.wst + ww / 2;
            const int4* meta = meta0 + held;
#pragma unroll 1
            for (int pi = 0; pi < npb; ++pi) {
                const int4 m = meta[pi];
                const float2* w = win + ((m.x - ww / 2 - a.bg0) & 1);   // the copy starts at an even bin
                if (SPLIT) {
                    const float far = gather_split<BINS == GATHER_NEAREST>(cs, u, w, ar, ai);
                    if (BINS == GATHER_NEAREST && __any_sync(0xffffffffu, far > kNearEdge)) {
                        const SplitLine t = split_terms(cs, u);
                        unsigned mask = 0;
                        for (int k = 0; k < 16; ++k) {
                            float s;
                            split_bin(t, k, &s);
                            mask |= (fabsf(s) > kNearEdge ? 1u : 0u) << k;
                        }
                        const int s0 = (st0 + begin) * pb, rel = (st - begin) * pb + pi;
                        for (unsigned who; (who = __ballot_sync(0xffffffffu, mask != 0)); mask &= mask - 1) {
                            if (notes > kNearQueue - 32) {
                                flush();
                                settle(s0);
                            }
                            if (mask) {
                                const int k = __ffs(mask) - 1;
                                float s;
                                const int n = split_bin(t, k, &s);
                                queue[notes + __popc(who & ((1u << lane) - 1))] = make_int2((rel << 9) | (lane << 4) | k, m.x - a.bg0 + n);
                            }
                            notes += __popc(who);
                        }
                    }
                } else if ((m.y >> (2 * warp)) & 1) {
                    gather_line<16>(cs, u, w, ar, ai);
                } else if ((m.z >> (2 * warp)) & 1) {
                    gather_line<8>(cs, u, w, ar, ai);
                } else if ((m.w >> (2 * warp)) & 1) {
                    gather_line<4>(cs, u, w, ar, ai);
                } else {
                    gather_line<0>(cs, u, w, ar, ai);
                }
                cs += NS * SF / 4;
                win += L.wst;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[2 + b]);
        }
        flush();
        if (BINS == GATHER_NEAREST && notes > 0) settle((st0 + begin) * pb);
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

// Measured (GB300, this kernel alone, against the tile gather before): 2048^2 x 4096 pulses 12.1 ms (14.3);
// 1024^2 x 2048 1.50 ms (1.88); 512^2 x 1024 0.22 ms (0.28).  About 19 instructions per pixel-pulse, of which the
// producers' about 2; issue 64 %, FMA pipe 62 %, special functions 57 % of their cycles.  Tried: sign and
// magnitude on the integer pipe, 3 % slower; without the phase's cubic term along the line 2 % faster (not kept: a
// second copy of the body); totals in shared memory instead of the image every 512 pulses, 13.7 ms (registers).
// Nearest bins, 1100 x 1000 x 1500 pulses at upsample 128: 1.58 ms (3.58), 27 instructions per pixel-pulse, issue 66 %,
// FMA pipe 44 %, special functions 40 %, shared memory 37 %; with no sample ever noted 1.51 ms.  Tried: packed sums
// (moves to pair the loaded values), 6 % slower; 64-bit addresses, 3 % slower.  The whole backprojection by look
// direction, against the tile gather: 0 deg 1.78 ms (3.85), 33 deg 2.25 (5.55), 90 deg 1.66 (3.9), bistatic 1.92;
// 0.5 m pixels at 60 deg, whose windows leave one CTA an SM, 4.2 (5.5).  Linear, 2048^2 x 512, upsample 16 and 0.5 m
// pixels: 2.03 ms (2.90).
cudaError_t launch_gather(const GatherArgs& a, cudaStream_t st) {
    if (a.num_tiles < 1 || a.parts < 1 || (a.parts > 1 && !a.partial) || (a.Lg & 1) || a.Lg < a.ww + 2) return cudaErrorInvalidValue;
    if (a.bins == GATHER_NEAREST && (!a.steps || !a.alpha2)) return cudaErrorInvalidValue;
    const size_t smem = gather_smem(a.bins, a.warps, a.ww, a.pb).total;
    auto go = [&](auto kern, int threads) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)(a.num_tiles * a.parts), threads, smem, st>>>(a);
        return cudaGetLastError();
    };
    auto pick = [&](auto bins) {
        constexpr int B = decltype(bins)::value;
        return a.warps == 8 ? go(gather_kernel<8, B>, 320) : a.warps == 4 ? go(gather_kernel<4, B>, 160) : cudaErrorInvalidValue;
    };
    cudaError_t e = a.bins == GATHER_RUNS      ? pick(std::integral_constant<int, GATHER_RUNS>{})
                    : a.bins == GATHER_NEAREST ? pick(std::integral_constant<int, GATHER_NEAREST>{})
                                               : pick(std::integral_constant<int, GATHER_LINEAR>{});
    return e != cudaSuccess || a.parts == 1 ? e : launch_sum_parts(a.partial, a.x, a.pixels, a.parts, a.accumulate, st);
}

// ------------------------------------------------------------------ layout
namespace {

constexpr size_t kPartialBytes = (size_t)256 << 20;   // partial images of a plan

// Split bins, for the choice of lattice only: instructions per pixel-pulse by the rate along a line, whose half-warps'
// loads spread over the banks.
double split_cost(double rate) { return 16.0 + std::min(rate, 8.0); }

// Plain bins: seconds per pixel-pulse of a lattice on a full GPU, by run length; where each sample loads two bins, by the
// bank conflicts of the lanes' loads.  Fitted to 380 geometries with every lattice forced in turn: 0.7 ps with runs of 16,
// 0.95 without runs up to two bins a bank, then 1.3, 1.6 and 2.4 ps at three, four and five.
double run_unit(const std::vector<LatticeRate>& rates) {
    double sum = 0.0;
    for (const LatticeRate& r : rates) {
        const double run = 0.66 + 0.02 * std::min(r.v, 8.0);
        sum += 15.0 * r.w < kRunSpan  ? run
               : 7.0 * r.w < kRunSpan ? run + 0.06
               : 3.0 * r.w < kRunSpan ? run + 0.14
                                      : std::max(0.95, 0.2 + 0.42 * bank_degree(r.v, false));
    }
    return 1.0e-12 * sum / rates.size();
}

// Estimated seconds of `count` pulses over `tiles` tiles with `parts` CTAs each: whole waves of CTAs at 1.5e12
// pixel-pulses per second (split bins: 1.2e12, less with few pulses a stage or few CTAs an SM, or the windows' bytes
// at 8e12 per second where these take longer), one stage to fill each CTA's pipeline, and the sum of the partial images.
double gather_seconds(const GatherLayout& L, size_t tiles, size_t count, int parts, size_t pixels) {
    const double slots = 152.0 * L.ctas, nst = std::ceil((double)count / L.pb);
    const double units = (double)kGatherLines * kGatherWalk * L.warps;
    const double rate = 1.2e12 * std::sqrt(L.ctas * L.warps / 16.0) / (1.0 + 0.12 / L.pb);
    const double pulse = L.bins == GATHER_RUNS ? units / 1.5e12 : std::max(units / rate, 8.0 * L.ww / 8e12);
    return std::ceil(tiles * (double)parts / slots) * (std::ceil(nst / parts) + 1.0) * L.pb * pulse * slots +
           (parts > 1 ? 2e-6 + 16.0 * pixels * parts / 5e12 : 0.0);
}

int best_parts(const GatherLayout& L, size_t tiles, size_t count, size_t pixels, int most, double* seconds) {
    const int nst = (int)((count + L.pb - 1) / L.pb);
    int best = 1;
    *seconds = INFINITY;
    for (int p = 1; p <= std::min(most, nst); ++p) {
        const double t = gather_seconds(L, tiles, count, p, pixels);
        if (t < *seconds * 0.99) {
            *seconds = t;
            best = p;
        }
    }
    return best;
}

// The same of a lattice's layout at `unit` seconds per pixel-pulse, plain bins: with fewer CTAs an SM than it holds, each
// runs faster (one of two: 0.66 of the time).
double lattice_seconds(const GatherLayout& L, size_t tiles, size_t count, size_t pixels, double unit) {
    const size_t ctas = tiles * L.parts, slots = (size_t)152 * L.ctas, rest = ctas % slots;
    const double last = rest ? std::pow((double)((rest + 151) / 152) / L.ctas, 0.6) : 0.0;
    const double nst = std::ceil((double)count / L.pb), pulse = (double)kGatherLines * kGatherWalk * L.warps * unit;
    return ((double)(ctas / slots) + last) * (std::ceil(nst / L.parts) + 1.0) * L.pb * pulse * slots +
           (L.parts > 1 ? 2e-6 + 16.0 * pixels * L.parts / 5e12 : 0.0);
}

// The layout with the least estimate for a lattice; excursion(lines, walk): bins from a tile's mean to its pixels' (not a
// number: no layout at all).  `tiles` of the result, and its tile list's shape, are those of `lines` x `walk` pixels.
struct Shape {
    GatherLayout layout;
    int lines = 0, walk = 0;
    size_t tiles = 0;
};
template <class EXCURSION>
Shape best_shape(int bins, const Lattice& lattice, size_t S, int nx, int ny, int nz, EXCURSION excursion) {
    const bool split = bins != GATHER_RUNS;
    const size_t pixels = (size_t)nx * ny * nz;
    const int most = (int)std::min<size_t>(16, std::max<size_t>(1, kPartialBytes / (pixels * sizeof(float2))));
    Shape best;
    double least = INFINITY;
    for (int shape : {80, 81, 40, 41}) {   // warps, and the warps along the walk: 1 or 2 with split bins, else all
        const int warps = shape / 10, along = split ? 1 + shape % 10 : warps, across = warps / along;
        if (!split && shape % 10) continue;
        const int lines = kGatherLines * across, walk = kGatherWalk * along;
        // a tap from the excursion of the tile's pixels about its mean bin, plus the base's fraction and rounding
        const double h = excursion(lines, walk) + 0.1;
        if (std::isnan(h)) return Shape{};
        if (!(h < 4096.0)) continue;
        const int ww = 2 * (int)std::ceil(h + 3.5 + kDip);
        size_t tiles = 0;
        for (const LatticeStrip& t : lattice_strips(lattice, lines, nx, ny)) tiles += (size_t)((t.b1 - t.b0) / walk + 1) * nz;
        for (int pb : {16, 8, 4, 2, 1}) {
            if (!split && pb < 4) break;
            const int full = warps == 8 ? 2 : 4;   // CTAs an SM: the registers' limit, and the shared memory's
            const int ctas = std::min(full, (int)(227 * 1024 / (gather_smem(bins, warps, ww, pb).total + 1024)));
            if (ctas < (split ? 1 : full)) continue;
            GatherLayout L;
            L.lattice = lattice;
            L.bins = bins;
            L.warps = warps;
            L.across = across;
            L.ctas = ctas;
            L.ww = ww;
            L.pb = pb;
            L.ok = true;
            double t;
            L.parts = best_parts(L, tiles, S, pixels, most, &t);
            if (t < 0.97 * least) {
                least = t;
                best = Shape{L, lines, walk, tiles};
            }
        }
    }
    return best;
}

}  // namespace

int gather_parts(const GatherLayout& L, size_t count, size_t pixels) {
    double t;
    return best_parts(L, L.tiles.size(), count, pixels, L.parts, &t);
}

GatherLayout gather_layout(int bins, const double* tx, const double* rx, size_t S, const double* origin, const double* ex,
                           const double* ey, const double* ez, int nx, int ny, int nz, double s_r, double kappa) {
    const bool split = bins != GATHER_RUNS;
    const size_t pixels = (size_t)nx * ny * nz;
    auto seconds = [&](const Lattice& L, const std::vector<LatticeRate>& rates) {
        double v = 0.0, w = 0.0, cost = 0.0;
        for (const LatticeRate& r : rates) {
            v = std::max(v, r.v);
            w = std::max(w, r.w);
            cost += split_cost(r.w);
        }
        if (split) {   // cost, and the share of the tiles (192 x 16) that straddle the image's edges
            const double bx = 192 * std::abs(L.wx) + kGatherWalk * std::abs(L.vx), by = 192 * std::abs(L.wy) + kGatherWalk * std::abs(L.vy);
            return cost * (1.0 + 0.5 * bx / nx) * (1.0 + 0.5 * by / ny);
        }
        const Shape q = best_shape(bins, L, S, nx, ny, nz, [&](int lines, int walk) { return 0.5 * (lines * v + walk * w); });
        return q.layout.ok ? lattice_seconds(q.layout, q.tiles, S, pixels, run_unit(rates)) : (double)INFINITY;
    };
    Lattice lattice = choose_lattice(scene_rates(tx, rx, S, origin, ex, ey, ez, nx, ny, nz, s_r), ex, ey, kappa, seconds);
    if (!lattice.ok) return GatherLayout{};
    if (split) {   // the lanes along the iso-range lines, 16 pixels per thread across them
        std::swap(lattice.vx, lattice.wx);
        std::swap(lattice.vy, lattice.wy);
    }
    Shape q = best_shape(bins, lattice, S, nx, ny, nz, [&](int lines, int walk) -> double {
        const LatticeBounds B = lattice_bounds(lattice, tx, rx, S, origin, ex, ey, ez, nx, ny, nz, 0.5 * lines, 0.5 * walk);
        if (!B.ok) return NAN;
        // Split bins are held to the FP64 positions: the expansions' fourth-order terms, at most d^4 / (8 R^3) an
        // antenna, may not use up the margin of kNearEdge.
        const double d = 8.0 * (B.len_a + B.len_b);
        if (split && !(d * d * d * d / (4.0 * B.nearest * B.nearest * B.nearest) * s_r < 1.0e-5)) return NAN;
        return B.excursion(0.5 * lines, 0.5 * walk, s_r);
    });
    GatherLayout best = q.layout;
    if (best.ok)
        for (int k = 0; k < nz; ++k)
            for (const LatticeStrip& t : lattice_strips(lattice, q.lines, nx, ny))
                for (long b = t.b0; b <= t.b1; b += q.walk) best.tiles.push_back(make_int4(t.a0, (int)b, k, 0));
    return best;
}

}  // namespace sar
