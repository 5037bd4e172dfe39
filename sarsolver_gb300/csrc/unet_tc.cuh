// unet_tc.cuh -- tensor-core (tcgen05 + TMA) convolution kernels of the learned warm start.
//
// Activations are NHWC bf16 tensors whose channel counts are multiples of 32.  Two kernels cover
// every convolution of the U-Net, forward and backward:
//
//  * conv_fwd_kernel<BK>: implicit GEMM  D[pixel][n] = sum_{tap, c} X[pixel + tap][c] * Wk[n][tap, c]
//    for 3x3 (pad 1) or 1x1 filters over one or two channel-concatenated sources.  M = 128 pixels
//    of one image (a BW x BH box), N = BN output channels, K stepped in blocks of BK channels of
//    one tap.  Each K block is one 4-D TMA box of the source at (c, x + dx, y + dy, image): the
//    tap shift moves the W/H coordinates, and out-of-image rows and columns arrive as zeros (the
//    padding).  Weights come as 2-D TMA boxes of the [N][taps * C] matrix.  Both operands are
//    K-major with a BK * 2-byte swizzle (128 B for BK = 64, 64 B for BK = 32).  The same kernel
//    runs the backward-data pass with the flipped, transposed filter.  The epilogue adds the
//    bias, applies ReLU or a ReLU-derivative mask, splits the
//    columns over two destination tensors (the two halves of a concatenated input) and can write
//    FP32 (the network output).
//  * conv_wgrad_kernel<CIB, COB>: weight gradient  dW[co][tap, ci] = sum_pixel dZ[pixel][co] *
//    X[pixel + tap][ci].  M = 128 rows = (128 / CIB) taps x CIB input channels, N = BN output
//    channels, K = pixels.  Both operands are read MN-major straight from the NHWC tensors
//    (channel rows of 128 pixels, 4-D TMA boxes as above), so no transposed copy is made.  The
//    pixel range is split over CTAs and each CTA adds its FP32 partial sums into dW.
//
// Warp roles (192 threads): warp 0 issues TMA loads into a ring of shared-memory stages, warp 1
// owns the TMEM accumulator and issues tcgen05.mma from one lane, warps 2-5 drain TMEM with
// tcgen05.ld (each warp reads the 32 TMEM lanes its warp index selects).  Stages are handed over
// with mbarriers: TMA completes "full[s]", tcgen05.commit arrives on "empty[s]" once the MMAs
// reading stage s are done, and a final commit arrives on "done".  Every wait is bounded; on
// expiry the kernel sets a flag bit, drains what it issued and frees its TMEM.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace unet {

constexpr int kThreads = 192;
constexpr unsigned kFlagTimeout = 8u;
constexpr long long kWaitCycles = 4000000000ll;   // ~2 s at 2 GHz

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_try_arrive(uint64_t* b) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(su32(b)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on the phase of the given parity (nanosleep back-off between polls).
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, unsigned max_ns) {
    if (bar_try(b, parity)) return true;
    const long long t0 = clock64();
    unsigned ns = 32;
    while (true) {
        __nanosleep(ns);
        if (bar_try(b, parity)) return true;
        if (clock64() - t0 > kWaitCycles) return false;
        ns = min(2 * ns, max_ns);
    }
}

// Position in a ring of stages: slot and times round it, counted up (64-bit divisions by the number of stages took
// longer than a stage's loads).
struct Ring {
    int s = 0;
    unsigned round = 0;
    __device__ __forceinline__ void next(int stages) {
        if (++s == stages) {
            s = 0;
            ++round;
        }
    }
};
// Every load issued into the ring (`full` barriers) has landed: before the CTA may exit.
__device__ __forceinline__ void drain(const Ring& r, uint64_t* full, int stages, unsigned* flags) {
    for (int s = 0; s < stages; ++s) {
        const unsigned rounds = r.round + (s < r.s ? 1u : 0u);
        if (rounds > 0 && !bar_wait(&full[s], (rounds - 1) & 1, 256)) atomicOr(flags, kFlagTimeout);
    }
}

__device__ __forceinline__ void tma_prefetch(const CUtensorMap* m) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ void tma_4d(void* dst, const CUtensorMap* m, int c0, int c1, int c2, int c3, uint64_t* b) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(su32(dst)),
        "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(su32(b))
        : "memory");
}
__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* m, int c0, int c1, uint64_t* b) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            su32(dst)),
        "l"(m), "r"(c0), "r"(c1), "r"(su32(b))
        : "memory");
}

// One lane of the warp, by the instruction that lets the compiler keep the chosen lane's operands in uniform registers
// (tcgen05.mma takes them there): behind `lane == 0` each MMA first moved its descriptors over, 50 to 70 cycles
// against the 40 of an N = 32 MMA.
__device__ __forceinline__ bool elect_lane() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(slot)), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, bf16 inputs, FP32 accumulator (kind::f16).
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
            d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
// Arrive on the mbarrier once all previously issued tcgen05 operations of this thread are done.
__device__ __forceinline__ void mma_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(b))
                 : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading / stride byte offsets (all >> 4), descriptor
// version 1, swizzle layout in bits 61-63 (2 = 128 B, 4 = 64 B).  In halves, so that the lane that issues the MMAs
// only adds to the low one: it is a single thread's serial chain, and forming both descriptors anew for each MMA took
// 200 cycles, several times the MMA's own.
struct Desc {
    uint32_t lo, hi;
    __device__ __forceinline__ Desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout)
        : lo((addr >> 4) | ((lbo >> 4) << 16)), hi((sbo >> 4) | (1u << 14) | (layout << 29)) {}
    __device__ __forceinline__ Desc moved(uint32_t bytes) const {
        Desc d = *this;
        d.lo += bytes >> 4;
        return d;
    }
    __device__ __forceinline__ uint64_t at(uint32_t bytes) const {   // `bytes` further on: a constant
        uint64_t d;
        asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo + (bytes >> 4)), "r"(hi));
        return d;
    }
};
__host__ __device__ constexpr uint32_t swizzle_layout(int row_bytes) { return row_bytes == 128 ? 2u : 4u; }

// Instruction descriptor of kind::f16: FP32 accumulator, bf16 A and B, K- or MN-major operands,
// N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__host__ __device__ constexpr uint32_t tmem_cols(int n) { return n <= 32 ? 32u : n <= 64 ? 64u : n <= 128 ? 128u : 256u; }

// ------------------------------------------------------------------ forward / backward-data conv
struct ConvMaps {
    CUtensorMap src[2];   // 4-D (C, W, H, images), box (BK, BW, BH, 1)
    CUtensorMap wts;      // 2-D (taps * Ctot, Nout), box (BK, BN)
};

struct ConvArgs {
    int nsrc, C0, C1, Ctot, taps, images;
    int W, H, BW, BH, tiles_x, tiles_y;
    int BN, Nout, stages;
    const float* bias;                 // [Nout] or null
    int relu;
    __nv_bfloat16* out[2];             // columns [0, outc[0]) -> out[0], the rest -> out[1]
    int outc[2];
    const __nv_bfloat16* mask[2];      // zero the value where mask <= 0 (same layout as out)
    float* out_f32;                    // when set: columns [0, f32_keep) as FP32 [pixel][f32_keep]
    int f32_keep;
    unsigned* flags;
};

// Epilogue of one output tile: 32 columns at a time from this warp's TMEM lanes, a pixel per lane.  The rounded values
// go through shared memory (2 KB a warp; 16-byte chunks swizzled by the pixel, so that neither side has bank conflicts)
// to a mapping of four lanes per pixel, whose stores fill whole sectors and, with 32 channels, whole lines; stored a
// pixel per lane, each 16-byte piece was a sector of its own, and the epilogue took 2400 cycles a tile.
template <int BK>
__device__ __forceinline__ void conv_epilogue(const ConvArgs& a, uint32_t tacc, int q, int lane, int img, int x0,
                                              int y0, int n0, uint4* stage) {
    const int lw = 31 - __clz(a.BW);   // BW is a power of two
    auto pixel = [&](int row) {
        return ((size_t)img * a.H + y0 + (row >> lw)) * a.W + x0 + (row & (a.BW - 1));
    };
    const int chunk = lane & 3, row0 = lane >> 2;   // of the lane's stores: pixels row0 + 8 j
    for (int c0 = 0; c0 < a.BN; c0 += 32) {
        const int n = n0 + c0, d = n >= a.outc[0] ? 1 : 0, ch = d ? n - a.outc[0] : n;
        uint4 mask[4];
        if (!a.out_f32 && a.mask[d]) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mask[j] = __ldg(reinterpret_cast<const uint4*>(a.mask[d] + pixel(32 * q + row0 + 8 * j) * a.outc[d] + ch) + chunk);
        }
        float v[32];
        tmem_ld32(tacc + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
        if (a.bias && ((uintptr_t)a.bias & 15) == 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 w = __ldg(reinterpret_cast<const float4*>(a.bias + n + i));
                v[i] += w.x;
                v[i + 1] += w.y;
                v[i + 2] += w.z;
                v[i + 3] += w.w;
            }
        } else if (a.bias) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += __ldg(a.bias + n + i);
        }
        if (a.relu) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.f);
        }
        if (a.out_f32) {
            const size_t pix = pixel(32 * q + lane);
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (n + i < a.f32_keep) a.out_f32[pix * a.f32_keep + n + i] = v[i];
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint4 pk;
            __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int i = 0; i < 4; ++i) pb[i] = __floats2bfloat162_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
            stage[4 * lane + (j ^ ((lane >> 1) & 3))] = pk;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = row0 + 8 * j;
            uint4 pk = stage[4 * row + (chunk ^ ((row >> 1) & 3))];
            if (a.mask[d]) {   // zero where mask <= 0 or not a number
                const __nv_bfloat16* mb = reinterpret_cast<const __nv_bfloat16*>(&mask[j]);
                __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(&pk);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (!(__bfloat162float(mb[i]) > 0.f)) pb[i] = __float2bfloat16_rn(0.f);
            }
            *(reinterpret_cast<uint4*>(a.out[d] + pixel(32 * q + row) * a.outc[d] + ch) + chunk) = pk;
        }
        __syncwarp();
    }
}

// Persistent: CTA c handles work items c, c + gridDim.x, ... (item = M tile x N tile).  The TMA
// ring runs on across items, and two TMEM accumulators alternate so that the epilogue of one
// item overlaps the MMAs of the next ("tfull[b]" committed by the MMA lane when accumulator b
// holds a finished item, "tempty[b]" arrived at by the four epilogue warps once they have read it).
template <int BK>
__global__ void __launch_bounds__(kThreads, 1) conv_fwd_kernel(const __grid_constant__ ConvMaps maps, const ConvArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int a_bytes = 128 * BK * 2, b_bytes = a.BN * BK * 2, stage_bytes = a_bytes + b_bytes;
    uint64_t* full = (uint64_t*)(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* tfull = empty + a.stages;   // [2]
    uint64_t* tempty = tfull + 2;         // [2]
    uint32_t* tslot = (uint32_t*)(tempty + 2);
    __shared__ int timed_out;
    __shared__ uint4 stage_out[4][128];

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int per_img = a.tiles_x * a.tiles_y;
    const int ntn = a.Nout / a.BN;
    const int items = a.images * per_img * ntn;
    const uint32_t ncols = tmem_cols(a.BN);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            bar_init(&tfull[b], 1);
            bar_init(&tempty[b], 4);
        }
        bar_fence_init();
        timed_out = 0;
    }
    if (warp == 1) {
        tmem_alloc(tslot, 2 * ncols);
        tmem_relinquish();
    }
    __syncthreads();
    tc_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
    const int kpt = a.Ctot / BK, nkb = a.taps * kpt;

    if (warp == 0 && lane == 0) {
        tma_prefetch(&maps.src[0]);
        if (a.nsrc > 1) tma_prefetch(&maps.src[1]);
        tma_prefetch(&maps.wts);
        Ring r;
        bool stop = false;
        for (int it = blockIdx.x; it < items && !stop; it += gridDim.x) {
            const int mt = it / ntn, n0 = (it % ntn) * a.BN;
            const int img = mt / per_img, rem = mt % per_img;
            const int x0 = (rem % a.tiles_x) * a.BW, y0 = (rem / a.tiles_x) * a.BH;
            int c = 0, dy = a.taps == 9 ? -1 : 0, dx = dy;
            for (int kb = 0; kb < nkb; ++kb) {
                if (r.round > 0 && !bar_wait(&empty[r.s], (uint32_t)((r.round - 1) & 1), 256)) {
                    atomicOr(a.flags, kFlagTimeout);
                    timed_out = 1;
                    stop = true;
                    break;
                }
                const int src = c >= a.C0 ? 1 : 0, cs = src ? c - a.C0 : c;
                uint8_t* st = smem + r.s * stage_bytes;
                bar_expect_tx(&full[r.s], (uint32_t)stage_bytes);
                tma_4d(st, &maps.src[src], cs, x0 + dx, y0 + dy, img, &full[r.s]);
                tma_2d(st + a_bytes, &maps.wts, kb * BK, n0, &full[r.s]);
                r.next(a.stages);
                c += BK;
                if (c == a.Ctot) {
                    c = 0;
                    if (++dx > 1) {
                        dx = -1;
                        ++dy;
                    }
                }
            }
        }
        drain(r, full, a.stages, a.flags);
    } else if (warp == 1 && elect_lane()) {
        const uint32_t idesc = idesc_bf16(128, a.BN, false, false);
        const uint32_t lay = swizzle_layout(BK * 2), sbo = 8 * BK * 2;
        Ring r;
        int i = 0;
        bool stop = false;
        for (int it = blockIdx.x; it < items && !stop; it += gridDim.x, ++i) {
            const int b = i & 1;
            if (i >= 2 && !bar_wait(&tempty[b], (uint32_t)(((i >> 1) - 1) & 1), 256)) {
                atomicOr(a.flags, kFlagTimeout);
                timed_out = 1;
                break;
            }
            tc_after();
            const uint32_t tacc = tmem + (uint32_t)(b * ncols);
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = r.s;
                if (!bar_wait(&full[s], (uint32_t)(r.round & 1), 64)) {
                    atomicOr(a.flags, kFlagTimeout);
                    timed_out = 1;
                    stop = true;
                    break;
                }
                const uint32_t sa = su32(smem + s * stage_bytes), sb = sa + a_bytes;
                const Desc da(sa, 16, sbo, lay), db(sb, 16, sbo, lay);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) mma_bf16(tacc, da.at(32 * k), db.at(32 * k), idesc, (kb | k) != 0);
                mma_commit(&empty[s]);
                r.next(a.stages);
            }
            mma_commit(&tfull[b]);   // also on the timeout path, so the epilogue warps are released
        }
    } else if (warp >= 2) {
        const int q = warp & 3;
        int i = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++i) {
            const int b = i & 1;
            const bool ok = __all_sync(0xffffffffu, bar_wait(&tfull[b], (uint32_t)((i >> 1) & 1), 1024));
            tc_after();
            if (!ok) {
                if (lane == 0) atomicOr(a.flags, kFlagTimeout);
                break;
            }
            if (__shfl_sync(0xffffffffu, timed_out, 0) == 0) {
                const int mt = it / ntn, n0 = (it % ntn) * a.BN;
                const int img = mt / per_img, rem = mt % per_img;
                conv_epilogue<BK>(a, tmem + (uint32_t)(b * ncols), q, lane, img, (rem % a.tiles_x) * a.BW,
                                  (rem / a.tiles_x) * a.BH, n0, stage_out[q]);
            }
            tc_before();
            __syncwarp();
            if (lane == 0) bar_try_arrive(&tempty[b]);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_after();
        tmem_dealloc(tmem, 2 * ncols);
    }
}

// 3x3 convolutions of images at least 128 pixels wide.  An item is 128 pixels of R neighbouring image rows, each row a
// tile with an accumulator of its own.  The nine taps of the R tiles read R + 2 rows of 130 pixels: each is loaded once
// per channel block, and the taps along x are the same box from one pixel further on (the descriptor's start address
// moves by a pixel; the swizzle goes by the address).  Filters that fit are loaded once per CTA and stay; larger ones
// run through a ring of their own, fed by a warp of its own.  A tile's K blocks are summed in the same order as in
// conv_fwd_kernel (taps, then channels), so the results are the same bits.
//
// Bound: the one lane that issues the MMAs.  An N = 32 MMA takes 40 cycles when they follow each other, and some 100 with
// the waits and addresses between them; hence R tiles to one filter block, and several CTAs an SM.
constexpr int kRowThreads = 224;   // and warp 6: the filter's loads
constexpr int kRowPixels = 130;
__host__ __device__ constexpr int row_slot(int bk) { return (kRowPixels * bk * 2 + 1023) & ~1023; }

struct RowRing {
    int rows;        // R
    int na, nb;      // slots of rows (a channel block each) and of filter blocks
    int resident;    // nb holds the whole filter
};

template <int BK, int R>
__global__ void __launch_bounds__(kRowThreads, 3) conv_row_kernel(const __grid_constant__ ConvMaps maps, const ConvArgs a,
                                                                  const RowRing ring) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int SLOT = row_slot(BK), ROW = BK * 2;
    const int b_bytes = a.BN * ROW;
    uint8_t* wts = smem + ring.na * SLOT;
    uint64_t* afull = (uint64_t*)(wts + ring.nb * b_bytes);
    uint64_t* aempty = afull + ring.na;
    uint64_t* bfull = aempty + ring.na;
    uint64_t* bempty = bfull + ring.nb;
    uint64_t* tfull = bempty + ring.nb;   // [2]
    uint64_t* tempty = tfull + 2;         // [2]
    uint32_t* tslot = (uint32_t*)(tempty + 2);
    __shared__ int timed_out;
    __shared__ uint4 stage_out[4][128];

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int groups = (a.H + R - 1) / R;
    const int per_img = a.tiles_x * groups, ntn = a.Nout / a.BN, items = a.images * per_img * ntn;
    const uint32_t ncols = tmem_cols(a.BN);   // of an accumulator; two sets of R
    const int kpt = a.Ctot / BK, nkb = 9 * kpt;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ring.na; ++s) {
            bar_init(&afull[s], 1);
            bar_init(&aempty[s], 1);
        }
        for (int s = 0; s < ring.nb; ++s) {
            bar_init(&bfull[s], 1);
            bar_init(&bempty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            bar_init(&tfull[b], 1);
            bar_init(&tempty[b], 4);
        }
        bar_fence_init();
        timed_out = 0;
    }
    if (warp == 1) {
        tmem_alloc(tslot, 2 * R * ncols);
        tmem_relinquish();
    }
    __syncthreads();
    tc_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);
    auto give_up = [&] {
        atomicOr(a.flags, kFlagTimeout);
        timed_out = 1;
    };

    if (warp == 0 && lane == 0) {
        tma_prefetch(&maps.src[0]);
        if (a.nsrc > 1) tma_prefetch(&maps.src[1]);
        Ring r;
        bool stop = false;
        for (int it = blockIdx.x; it < items && !stop; it += gridDim.x) {
            const int mt = it / ntn, img = mt / per_img, rem = mt % per_img;
            const int x0 = (rem % a.tiles_x) * 128, y0 = rem / a.tiles_x * R;
            for (int row = -1; row <= R && !stop; ++row)
                for (int c = 0; c < a.Ctot; c += BK, r.next(ring.na)) {
                    if (r.round > 0 && !bar_wait(&aempty[r.s], (r.round - 1) & 1, 256)) {
                        give_up();
                        stop = true;
                        break;
                    }
                    const int src = c >= a.C0 ? 1 : 0;
                    bar_expect_tx(&afull[r.s], (uint32_t)(kRowPixels * ROW));
                    tma_4d(smem + r.s * SLOT, &maps.src[src], src ? c - a.C0 : c, x0 - 1, y0 + row, img, &afull[r.s]);
                }
        }
        drain(r, afull, ring.na, a.flags);
    } else if (warp == 6 && lane == 0) {
        tma_prefetch(&maps.wts);
        Ring r;
        bool stop = false;
        for (int it = blockIdx.x; it < items && !stop; it += gridDim.x) {
            const int n0 = (it % ntn) * a.BN;
            for (int kb = 0; kb < nkb; ++kb, r.next(ring.nb)) {
                if (r.round > 0 && !bar_wait(&bempty[r.s], (r.round - 1) & 1, 256)) {
                    give_up();
                    stop = true;
                    break;
                }
                bar_expect_tx(&bfull[r.s], (uint32_t)b_bytes);
                tma_2d(wts + r.s * b_bytes, &maps.wts, kb * BK, n0, &bfull[r.s]);
            }
            if (ring.resident) break;
        }
        drain(r, bfull, ring.nb, a.flags);
    } else if (warp == 1 && elect_lane()) {
        const uint32_t idesc = idesc_bf16(128, a.BN, false, false);
        const uint32_t lay = swizzle_layout(ROW), sbo = 8 * ROW;
        const Desc da0(su32(smem), 16, sbo, lay), db0(su32(wts), 16, sbo, lay);
        Ring rb;
        int first = 0;        // slot of the item's first row
        uint32_t phase = 0;   // a bit per slot of rows: the phase that its next load completes
        int i = 0;
        bool stop = false;
        auto wrap = [&](int s) { return s >= ring.na ? s - ring.na : s; };
        for (int it = blockIdx.x; it < items && !stop; it += gridDim.x, ++i) {
            const int b = i & 1;
            if (i >= 2 && !bar_wait(&tempty[b], (uint32_t)(((i >> 1) - 1) & 1), 256)) {
                give_up();
                break;
            }
            tc_after();
            const uint32_t tacc = tmem + (uint32_t)(b * R) * ncols;
            if (ring.resident) rb = Ring{};
            for (int dy = 0; dy < 3 && !stop; ++dy, first = wrap(first + kpt))   // first: row dy, which tile 0 reads
#pragma unroll
                for (int dx = 0; dx < 3; ++dx)
                    for (int c = 0; c < kpt && !stop; ++c, rb.next(ring.nb)) {
                        if ((!ring.resident || i == 0) && !bar_wait(&bfull[rb.s], rb.round & 1, 64)) stop = true;
                        const Desc db = db0.moved(rb.s * b_bytes);
                        int s = wrap(first + c);
#pragma unroll
                        for (int j = 0; j < R; ++j, s = wrap(s + kpt)) {
                            // a row is first read at dx = 0 by the tile that comes to it first, last at dx = 2
                            if (dx == 0 && (dy == 0 || j == R - 1)) {
                                if (!stop && !bar_wait(&afull[s], phase >> s & 1, 64)) stop = true;
                                phase ^= 1u << s;
                            }
                            if (stop) continue;
                            const Desc da = da0.moved(s * SLOT + dx * ROW);
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k)
                                mma_bf16(tacc + j * ncols, da.at(32 * k), db.at(32 * k), idesc, (dy | dx | c | k) != 0);
                            if (dx == 2 && (dy == 2 || j == 0)) mma_commit(&aempty[s]);
                        }
                        if (!ring.resident) mma_commit(&bempty[rb.s]);
                    }
            if (stop) give_up();
            for (int row = 3; row < R + 2; ++row) first = wrap(first + kpt);
            mma_commit(&tfull[b]);   // also on the timeout path, so the epilogue warps are released
        }
    } else if (warp >= 2 && warp < 6) {
        const int q = warp & 3;
        int i = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++i) {
            const int b = i & 1;
            const bool ok = __all_sync(0xffffffffu, bar_wait(&tfull[b], (uint32_t)((i >> 1) & 1), 1024));
            tc_after();
            if (!ok) {
                if (lane == 0) atomicOr(a.flags, kFlagTimeout);
                break;
            }
            if (__shfl_sync(0xffffffffu, timed_out, 0) == 0) {
                const int mt = it / ntn, img = mt / per_img, rem = mt % per_img;
                const int y0 = rem / a.tiles_x * R;
                for (int j = 0; j < R && y0 + j < a.H; ++j)
                    conv_epilogue<BK>(a, tmem + (uint32_t)(b * R + j) * ncols, q, lane, img, (rem % a.tiles_x) * 128, y0 + j,
                                      (it % ntn) * a.BN, stage_out[q]);
            }
            tc_before();
            __syncwarp();
            if (lane == 0) bar_try_arrive(&tempty[b]);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_after();
        tmem_dealloc(tmem, 2 * R * ncols);
    }
}

// ------------------------------------------------------------------ weight gradient
struct WgradMaps {
    CUtensorMap x[2];   // 4-D (C, W, H, images), box (CIB, BW, BH, 1)
    CUtensorMap dz;     // 4-D (Cout, W, H, images), box (COB, BW, BH, 1)
};

struct WgradArgs {
    int nsrc, C0, C1, Ctot, taps, Cout;
    int W, H, BW, BH, tiles_x, tiles_y;
    int num_tiles, tiles_per_split;
    int BN, stages;
    float* dw;   // FP32 [Cout][taps * Ctot], accumulated
    float* db;   // FP32 [Cout], accumulated, or null
    unsigned* flags;
};

// The bias gradient, db[n] += sum of dZ over this CTA's share of its pixels (the K blocks are dealt out to the CTAs
// that read them, gridDim.y), by the four warps that otherwise wait for the accumulator: FP32 sums of the staged dZ
// boxes, a pair of channels per thread.  Read again by a kernel of its own, dZ took 9 us a layer and a launch.
template <int COB>
__device__ __forceinline__ void sum_dz(const WgradArgs& a, const uint8_t* dz0, int stage_bytes, uint64_t* full,
                                       uint64_t* empty, int nkb, int n0, float* bsum) {
    constexpr int WORDS = COB / 2, LANES = 128 / WORDS;   // channel pairs of a row, rows read at a time
    const int t = threadIdx.x - 64, word = t % WORDS, row0 = t / WORDS, lane = threadIdx.x & 31;
    const int boxes = a.BN / COB;
    float2 sum[4] = {};   // BN <= 128
    for (int i = t; i < a.BN; i += 128) bsum[i] = 0.f;
    Ring r;
    bool ok = true;
    int turn = blockIdx.y;   // K blocks until this CTA's next
    for (int kb = 0; kb < nkb; ++kb, r.next(a.stages)) {
        if (!__all_sync(0xffffffffu, bar_wait(&full[r.s], r.round & 1, 256))) {
            ok = false;
            break;
        }
        if (turn == 0) {
            turn = gridDim.y;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (j >= boxes) break;
                const uint8_t* box = dz0 + r.s * stage_bytes + j * 128 * COB * 2;
#pragma unroll 8
                for (int p = row0; p < 128; p += LANES) {
                    const int chunk = (word >> 2) ^ (COB == 64 ? p & 7 : (p >> 1) & 3);   // the copy's swizzle
                    const float2 v = __bfloat1622float2(
                        *reinterpret_cast<const __nv_bfloat162*>(box + p * COB * 2 + chunk * 16 + (word & 3) * 4));
                    sum[j].x += v.x;
                    sum[j].y += v.y;
                }
            }
        }
        --turn;
        __syncwarp();
        if (lane == 0) bar_try_arrive(&empty[r.s]);
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j >= boxes) break;
        atomicAdd(&bsum[j * COB + 2 * word], sum[j].x);
        atomicAdd(&bsum[j * COB + 2 * word + 1], sum[j].y);
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (ok)
        for (int i = t; i < a.BN; i += 128) atomicAdd(a.db + n0 + i, bsum[i]);
}

template <int CIB, int COB>
__global__ void __launch_bounds__(kThreads, 1) conv_wgrad_kernel(const __grid_constant__ WgradMaps maps,
                                                                  const WgradArgs a) {
    constexpr int TPG = 128 / CIB;                 // taps per 128-row M tile
    constexpr int A_BOX = 128 * CIB * 2;           // one tap's box: 128 pixel rows of CIB channels
    constexpr int B_BOX = 128 * COB * 2;
    constexpr int A_BYTES = TPG * A_BOX;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nb = a.BN / COB;
    const int stage_bytes = A_BYTES + nb * B_BOX;
    uint64_t* full = (uint64_t*)(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* done = empty + a.stages;
    uint32_t* tslot = (uint32_t*)(done + 1);
    __shared__ int timed_out;
    __shared__ float bsum[128];

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int ngroups = (a.taps + TPG - 1) / TPG;
    const int tg = blockIdx.y % ngroups, cb = blockIdx.y / ngroups;
    const int cglob = cb * CIB, src = cglob >= a.C0 ? 1 : 0, cs = src ? cglob - a.C0 : cglob;
    const int n0 = blockIdx.z * a.BN;
    const int t_begin = blockIdx.x * a.tiles_per_split;
    const int t_end = min(a.num_tiles, t_begin + a.tiles_per_split);
    const int nkb = max(0, t_end - t_begin);
    const uint32_t ncols = tmem_cols(a.BN);
    const int per_img = a.tiles_x * a.tiles_y;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], a.db ? 5 : 1);   // the MMAs, and the four warps that sum dZ
        }
        bar_init(done, 1);
        bar_fence_init();
        timed_out = 0;
    }
    if (warp == 1) {
        tmem_alloc(tslot, ncols);
        tmem_relinquish();
    }
    __syncthreads();
    tc_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);

    if (warp == 0 && lane == 0) {
        tma_prefetch(&maps.x[src]);
        tma_prefetch(&maps.dz);
        Ring r;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = r.s;
            if (r.round > 0 && !bar_wait(&empty[s], (r.round - 1) & 1, 256)) {
                atomicOr(a.flags, kFlagTimeout);
                timed_out = 1;
                break;
            }
            const int t = t_begin + kb, img = t / per_img, rem = t % per_img;
            const int x0 = (rem % a.tiles_x) * a.BW, y0 = (rem / a.tiles_x) * a.BH;
            uint8_t* st = smem + s * stage_bytes;
            bar_expect_tx(&full[s], (uint32_t)stage_bytes);
#pragma unroll
            for (int j = 0; j < TPG; ++j) {
                const int tap = tg * TPG + j;
                int dx = 0, dy = 0;
                if (tap >= a.taps) {
                    dy = -4 * a.BH - 8 - y0;   // a box wholly above the image: zeros
                } else if (a.taps == 9) {
                    dy = tap / 3 - 1;
                    dx = tap % 3 - 1;
                }
                tma_4d(st + j * A_BOX, &maps.x[src], cs, x0 + dx, y0 + dy, img, &full[s]);
            }
            for (int j = 0; j < nb; ++j) tma_4d(st + A_BYTES + j * B_BOX, &maps.dz, n0 + j * COB, x0, y0, img, &full[s]);
            r.next(a.stages);
        }
        drain(r, full, a.stages, a.flags);
    } else if (warp == 1 && elect_lane()) {
        const uint32_t idesc = idesc_bf16(128, a.BN, true, true);
        const uint32_t la = swizzle_layout(CIB * 2), lb = swizzle_layout(COB * 2);
        constexpr uint32_t atom_a = 8 * CIB * 2, atom_b = 8 * COB * 2;
        Ring r;
        for (int kb = 0; kb < nkb; ++kb, r.next(a.stages)) {
            const int s = r.s;
            if (!bar_wait(&full[s], r.round & 1, 64)) {
                atomicOr(a.flags, kFlagTimeout);
                timed_out = 1;
                break;
            }
            const uint32_t sa = su32(smem + s * stage_bytes), sb = sa + A_BYTES;
            const Desc da(sa, A_BOX, atom_a, la), db(sb, B_BOX, atom_b, lb);
#pragma unroll
            for (int k = 0; k < 8; ++k)   // 16 pixel rows (two 8-row groups) per MMA
                mma_bf16(tmem, da.at(2 * atom_a * k), db.at(2 * atom_b * k), idesc, (kb | k) != 0);
            mma_commit(&empty[s]);
        }
        mma_commit(done);
    } else if (warp >= 2) {
        if (a.db) sum_dz<COB>(a, smem + A_BYTES, stage_bytes, full, empty, nkb, n0, bsum);
        const bool ok = __all_sync(0xffffffffu, bar_wait(done, 0, 1024));
        const bool go = ok && nkb > 0 && __shfl_sync(0xffffffffu, timed_out, 0) == 0;
        tc_after();
        if (!ok) {
            if (lane == 0) atomicOr(a.flags, kFlagTimeout);
        } else if (go) {
            const int q = warp & 3, row = 32 * q + lane;
            const int tap = tg * TPG + row / CIB, ci = cglob + row % CIB;
            const size_t ktot = (size_t)a.taps * a.Ctot;
            for (int c0 = 0; c0 < a.BN; c0 += 32) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
                if (tap < a.taps) {
                    float* dst = a.dw + (size_t)(n0 + c0) * ktot + (size_t)tap * a.Ctot + ci;
#pragma unroll
                    for (int i = 0; i < 32; ++i) atomicAdd(dst + (size_t)i * ktot, v[i]);
                }
            }
        }
        tc_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc_after();
        tmem_dealloc(tmem, ncols);
    }
}

// The weight gradient of 3x3 filters over images at least 128 pixels wide: a K block is 128 pixels of an image row, and
// a CTA forms the three taps of one filter row from one box of 131 pixels of X (the taps lie a pixel apart in it: the
// leading offset of the descriptor), where conv_wgrad_kernel loads a box per tap.  An M tile holds four taps of 32
// channels or two of 64; those past the third are formed and not stored.
//
// Bound: L2 to shared memory.  32 -> 32 channels, 512^2: 16 KB of X and dZ a K block and filter row, before 40 KB for
// four taps.  Measured figures stand at conv_wgrad (sar_unet.cu).
constexpr int kWgradPixels = 131;

template <int CIB, int COB>
__global__ void __launch_bounds__(kThreads, 1) conv_wgrad_row_kernel(const __grid_constant__ WgradMaps maps,
                                                                  const WgradArgs a) {
    constexpr int ROW = CIB * 2, SLOTS = 128 / CIB;   // bytes of a pixel; taps of a 128-row M tile
    constexpr int MT = CIB == 64 ? 2 : 1;             // M tiles for the three taps of a filter row
    constexpr int B_BOX = 128 * COB * 2;
    constexpr int A_BYTES = (kWgradPixels * ROW + 1023) & ~1023;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int nb = a.BN / COB;
    const int stage_bytes = A_BYTES + nb * B_BOX;
    const uint32_t load_bytes = kWgradPixels * ROW + nb * B_BOX;
    uint64_t* full = (uint64_t*)(smem + a.stages * stage_bytes);
    uint64_t* empty = full + a.stages;
    uint64_t* done = empty + a.stages;
    uint32_t* tslot = (uint32_t*)(done + 1);
    __shared__ int timed_out;
    __shared__ float bsum[128];

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int dy = blockIdx.y % 3, cb = blockIdx.y / 3;   // filter row, channel block
    const int cglob = cb * CIB, src = cglob >= a.C0 ? 1 : 0, cs = src ? cglob - a.C0 : cglob;
    const int n0 = blockIdx.z * a.BN;
    const int t_begin = blockIdx.x * a.tiles_per_split;
    const int t_end = min(a.num_tiles, t_begin + a.tiles_per_split);
    const int nkb = max(0, t_end - t_begin);
    const uint32_t ncols = tmem_cols(a.BN);
    const int per_img = a.tiles_x * a.tiles_y;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], a.db ? 5 : 1);   // the MMAs, and the four warps that sum dZ
        }
        bar_init(done, 1);
        bar_fence_init();
        timed_out = 0;
    }
    if (warp == 1) {
        tmem_alloc(tslot, MT * ncols);
        tmem_relinquish();
    }
    __syncthreads();
    tc_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tslot, 0);

    if (warp == 0 && lane == 0) {
        tma_prefetch(&maps.x[src]);
        tma_prefetch(&maps.dz);
        Ring r;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = r.s;
            if (r.round > 0 && !bar_wait(&empty[s], (r.round - 1) & 1, 256)) {
                atomicOr(a.flags, kFlagTimeout);
                timed_out = 1;
                break;
            }
            const int t = t_begin + kb, img = t / per_img, rem = t % per_img;
            const int x0 = (rem % a.tiles_x) * 128, y0 = rem / a.tiles_x;
            uint8_t* st = smem + s * stage_bytes;
            bar_expect_tx(&full[s], load_bytes);
            tma_4d(st, &maps.x[src], cs, x0 - 1, y0 + dy - 1, img, &full[s]);
            for (int j = 0; j < nb; ++j) tma_4d(st + A_BYTES + j * B_BOX, &maps.dz, n0 + j * COB, x0, y0, img, &full[s]);
            r.next(a.stages);
        }
        drain(r, full, a.stages, a.flags);
    } else if (warp == 1 && elect_lane()) {
        const uint32_t idesc = idesc_bf16(128, a.BN, true, true);
        const uint32_t la = swizzle_layout(ROW), lb = swizzle_layout(COB * 2);
        constexpr uint32_t atom_a = 8 * CIB * 2, atom_b = 8 * COB * 2;
        Ring r;
        for (int kb = 0; kb < nkb; ++kb, r.next(a.stages)) {
            const int s = r.s;
            if (!bar_wait(&full[s], r.round & 1, 64)) {
                atomicOr(a.flags, kFlagTimeout);
                timed_out = 1;
                break;
            }
            const uint32_t sa = su32(smem + s * stage_bytes), sb = sa + A_BYTES;
            const Desc da(sa, ROW, atom_a, la), db(sb, B_BOX, atom_b, lb);
#pragma unroll
            for (int k = 0; k < 8; ++k)   // 16 pixels (two 8-pixel groups) per MMA; the taps of an M tile a pixel apart
#pragma unroll
                for (int m = 0; m < MT; ++m)
                    mma_bf16(tmem + m * ncols, da.at(m * SLOTS * ROW + 2 * atom_a * k), db.at(2 * atom_b * k), idesc, (kb | k) != 0);
            mma_commit(&empty[s]);
        }
        mma_commit(done);
    } else if (warp >= 2) {
        if (a.db) sum_dz<COB>(a, smem + A_BYTES, stage_bytes, full, empty, nkb, n0, bsum);
        const bool ok = __all_sync(0xffffffffu, bar_wait(done, 0, 1024));
        const bool go = ok && nkb > 0 && __shfl_sync(0xffffffffu, timed_out, 0) == 0;
        tc_after();
        if (!ok) {
            if (lane == 0) atomicOr(a.flags, kFlagTimeout);
        } else if (go) {
            const int q = warp & 3, row = 32 * q + lane, ci = cglob + row % CIB;
            const size_t ktot = (size_t)9 * a.Ctot;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int dx = m * SLOTS + row / CIB;
                for (int c0 = 0; c0 < a.BN; c0 += 32) {
                    float v[32];
                    tmem_ld32(tmem + m * ncols + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
                    if (dx < 3) {
                        float* dst = a.dw + (size_t)(n0 + c0) * ktot + (size_t)(3 * dy + dx) * a.Ctot + ci;
#pragma unroll
                        for (int i = 0; i < 32; ++i) atomicAdd(dst + (size_t)i * ktot, v[i]);
                    }
                }
            }
        }
        tc_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc_after();
        tmem_dealloc(tmem, MT * ncols);
    }
}

}  // namespace unet
