// tc_conv.cuh — the learned proposer's 3x3 convolutions on the 5th-generation tensor cores (tcgen05, sm_100a):
// BF16 operands in shared memory, FP32 accumulators in tensor memory (TMEM).
//
// Activation layout ("chunk-major padded"): every sample (one macroblock's input) is a 50 x 50 raster, its
// 48 x 48 interior plus a ring of zeros; rasters follow each other, Q = samples * 2500 pixels in all. A tensor
// of C channels is C / 8 planes, plane c holding channels 8c .. 8c + 7 of every pixel as 16 bytes: element
// (c, q, e) at ((c * Q) + q) * 8 + e. A 3x3 convolution of such a raster is then a 1-D convolution along q with
// the nine shifts (dy - 1) * 50 + (dx - 1): output pixel q reads input pixel q + shift, and a shift never leaves
// the sample's own raster for an interior pixel (outputs on the ring are written as zeros).
//
// A CTA takes tiles of 256 consecutive output pixels. Per tile: TMA box loads bring the input halo (pixels
// q0 - 51 .. q0 + 332 of every plane, zeros beyond the tensor) into shared memory in the same layout;
// every tap's A operand (128 pixels x 16 channels, K-major, no swizzle) is then just another start address into
// the halo, so no im2col copy is made. The weights (B: 32 output channels x CIN input channels per tap, K-major)
// sit in shared memory for the CTA's life. One thread issues 2 x 9 taps x CIN / 16 MMAs of M = 128, N = 32, K = 16
// into a TMEM accumulator (128 lanes x 2 x 32 FP32 columns); the epilogue warps read their 32 lanes (pixels) x 32
// columns (channels) back with tcgen05.ld, add the bias, apply ReLU or a gradient mask, zero the ring, and
// store BF16. Loads, MMAs and epilogues of successive tiles overlap (conv3x3p_kernel, below).
//
// The same kernel is the backward pass's data gradient (the convolution with the weights transposed and the
// taps mirrored, and the mask of the layer's ReLU in the epilogue).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cstdint>

namespace ironav {
namespace tc {

constexpr int RW = 50;                  // raster width (and height): 48 + 2
constexpr int RPIX = RW * RW;           // pixels a sample
constexpr int TILE = 128;               // output pixels a tile (the MMA's M)
constexpr int HALO_LO = RW + 1;         // the most negative shift
constexpr int BOX_PIXELS = 128;         // pixels a TMA box (256 64-bit elements, the limit of a box's side)
constexpr int COUT = 32;                // output channels (the MMA's N)
constexpr unsigned WAIT_LIMIT = 1u << 26;  // polls of an mbarrier before the kernel gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Waits for the mbarrier's phase `parity` to complete, at most WAIT_LIMIT polls; false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
    const uint32_t a = smem_u32(bar);
    for (unsigned i = 0; i < WAIT_LIMIT; i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// TMA: a box of the tensor map (BOX_PIXELS pixels from pixel q, planes from c) into shared memory, completion counted on
// the mbarrier. The map's elements are half pixels, so any pixel is a 16-byte boundary.
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int q, int c, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(2 * q), "r"(c), "r"(smem_u32(bar))
        : "memory");
}

// A shared-memory matrix descriptor for tcgen05.mma (K-major, no swizzle): start address, the byte distance
// between core matrices adjacent in K (lbo) and in M/N (sbo), version 1 (bits 46-47), layout type 0.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) |
           (1ull << 46);
}
// The instruction descriptor of kind::f16 with BF16 A and B, FP32 D, both K-major, M = 128, N = 32.
constexpr uint32_t IDESC_BF16_M128_N32 = (1u << 4) | (1u << 7) | (1u << 10) | ((COUT >> 3) << 17) | ((TILE >> 4) << 24);

// One MMA, issued by the lane whose `issuer` is set. The whole warp walks the issuing loop, so that the descriptors are
// warp-uniform values: a loop under a one-lane branch moved every operand of every MMA to the uniform registers on its
// own, and the issue bound the kernel (8160 samples, 32 and 16 input channels: 583
// and 420 us, now 553 and 346; shared-memory reads of A, 4 KB for 32 columns of output, bound it now).
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t issuer) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %9, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(issuer));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 lanes x 32 consecutive FP32 columns of TMEM into 32 registers of each thread (lane = the warp's lane).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
        "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// The weight gradient of a 3x3 layer: dw[t][o][i] += sum over pixels q of dz[q][o] * x[q + shift_t][i] (FP32,
// accumulated into dw with atomics), and db[o] += sum over q of dz[q][o]. As MMAs: M = 128 rows (a group of
// 128 / CIN taps x CIN input channels), N = 32 output channels, K = pixels; both operands MN-major (a pixel's 8
// channels contiguous, pixels 16 bytes apart), so the chunk-major tensors are their own canonical layout. Per
// tile of KT pixels, TMA stages the nine tap-shifted views of x ([tap slot][plane][pixel][16 B], taps beyond
// 8 stay zero) and the tile of dz; one thread issues groups x KT / 16 MMAs into one TMEM accumulator per group
// (32 columns each), accumulating over all the CTA's tiles; at the end each warp reads its 32 rows and adds them
// to dw. xmap: x with boxes of KT pixels of every plane; zmap: dz with boxes of KT pixels of its 4 planes.
//
// One CTA an SM, warp-specialised: warp 4 streams tiles into a ring of two stages, warp 5 issues their MMAs, warps 0-3 sum
// the bias gradient from the staged dz; a stage is refilled once its MMAs (tcgen05.commit) and the four warps have
// done with it. The waits are bounded as conv3x3p_kernel's: a role that gives up sets the CTA's failure flag, every other
// role stops at its next wait, and the copies and MMAs still in flight are waited for (bounded) before the TMEM is freed.
// 512 samples of 32 channels: 199 us with two CTAs an SM that each loaded, computed and summed one tile after another
// (and copies of 16-byte rows), now 79.
constexpr int WG_KT = BOX_PIXELS;  // pixels a tile (K)
constexpr int WG_STAGES = 2;
constexpr int WG_THREADS = 192;

template <int CIN>
__host__ __device__ constexpr int wgrad3x3_stage_bytes() {
    return ((9 + 128 / CIN - 1) / (128 / CIN)) * 128 * WG_KT * 2 + 4 * WG_KT * 16;
}
template <int CIN>
constexpr int wgrad3x3_smem_bytes() {
    return WG_STAGES * wgrad3x3_stage_bytes<CIN>() + (2 * WG_STAGES + 1) * 8 + 16 + 32 * 4;
}

// MN-major operands for the weight gradient: M (or N) 8 channels of a pixel contiguous, K = pixels 16 bytes apart.
constexpr uint32_t IDESC_BF16_MN_M128_N32 = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((COUT >> 3) << 17) | ((TILE >> 4) << 24);

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int CIN>
__global__ void __launch_bounds__(WG_THREADS, 1) wgrad3x3_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap zmap,
                                                                 float* __restrict__ dw, float* __restrict__ db, int tiles, unsigned* err) {
    constexpr int KC = CIN / 8, TPG = 128 / CIN, NG = (9 + TPG - 1) / TPG;
    constexpr int PLANE = WG_KT * 16;          // bytes of one plane's tile
    constexpr int ABYTES = NG * 16 * PLANE;    // NG groups x 16 planes (TPG taps x KC planes)
    constexpr int SBYTES = wgrad3x3_stage_bytes<CIN>();
    constexpr unsigned TX = (9 * KC + 4) * PLANE;
    constexpr int NCOL = NG * 32 <= 32 ? 32 : (NG * 32 <= 64 ? 64 : 128);
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + WG_STAGES * SBYTES);  // [WG_STAGES]
    uint64_t* empty = full + WG_STAGES;                                       // [WG_STAGES]: the MMAs and warps 0-3
    uint64_t* done = empty + WG_STAGES;                                       // every MMA of the CTA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* dbs = reinterpret_cast<float*>(tmem_slot + 4);
    __shared__ int s_loaded, s_issued;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;  // this CTA's tiles
    // the slots of taps 9.. stay zero (their rows accumulate nothing)
    for (int s = 0; s < WG_STAGES; s++)
        for (int i = tid; i < (NG * TPG - 9) * KC * PLANE / 16; i += WG_THREADS)
            reinterpret_cast<uint4*>(smem + s * SBYTES + 9 * KC * PLANE)[i] = make_uint4(0, 0, 0, 0);
    if (tid < 32) dbs[tid] = 0.f;
    if (tid == 0) {
        for (int s = 0; s < WG_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 5);
        }
        mbar_init(done, 1);
        *failed = 0;
        s_loaded = s_issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(NCOL));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    float dbsum = 0.f;  // warps 0-3: this thread's share of db: channel lane, pixels warp, warp + 4, ...
    if (warp == 4) {
        if (lane == 0) {
            int loaded = 0;
            for (int it = 0; it < ntiles; it++) {
                const int s = it % WG_STAGES, k = it / WG_STAGES;
                if (k > 0 && !mbar_wait(&empty[s], (k - 1) & 1)) {
                    *failed = 1;
                    break;
                }
                if (*failed) break;
                const int q0 = ((int)blockIdx.x + it * (int)gridDim.x) * WG_KT;
                uint8_t* as = smem + s * SBYTES;
                mbar_expect_tx(&full[s], TX);
                for (int t = 0; t < 9; t++)
                    tma_load(as + (t / TPG) * 16 * PLANE + (t % TPG) * KC * PLANE, &xmap, q0 + (t / 3 - 1) * RW + (t % 3 - 1), 0, &full[s]);
                tma_load(as + ABYTES, &zmap, q0, 0, &full[s]);
                loaded = it + 1;
            }
            s_loaded = loaded;
        }
    } else if (warp == 5) {
        const uint32_t issuer = lane == 0;
        int issued = 0;
        for (int it = 0; it < ntiles; it++) {
            const int s = it % WG_STAGES, k = it / WG_STAGES;
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], k & 1))) {
                *failed = 1;
                break;
            }
            if (__any_sync(0xffffffffu, *failed != 0)) break;
            tc_fence_after();
            const uint32_t a0 = smem_u32(smem) + (uint32_t)(s * SBYTES);
            const uint64_t ad0 = smem_desc(a0, 128, PLANE), bd0 = smem_desc(a0 + ABYTES, 128, PLANE);
#pragma unroll
            for (int g = 0; g < NG; g++)
#pragma unroll
                for (int kk = 0; kk < WG_KT / 16; kk++)
                    mma_bf16(tmem + (uint32_t)(g * 32), ad0 + (uint64_t)((g * 16 * PLANE + kk * 256) >> 4), bd0 + (uint64_t)((kk * 256) >> 4),
                             IDESC_BF16_MN_M128_N32, (it != 0 || kk != 0) ? 1u : 0u, issuer);
            if (issuer) mma_commit(&empty[s]);
            __syncwarp();
            issued = it + 1;
        }
        if (issuer) {
            if (issued > 0) mma_commit(done);
            s_issued = issued;
        }
    } else {
        for (int it = 0; it < ntiles; it++) {
            const int s = it % WG_STAGES, k = it / WG_STAGES;
            const bool ok = mbar_wait(&full[s], k & 1);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) *failed = 1;
                break;
            }
            const __nv_bfloat16* z = reinterpret_cast<const __nv_bfloat16*>(smem + s * SBYTES + ABYTES);
#pragma unroll 8
            for (int p = warp; p < WG_KT; p += 4) dbsum += __bfloat162float(z[((lane >> 3) * WG_KT + p) * 8 + (lane & 7)]);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (__any_sync(0xffffffffu, *failed != 0)) break;
        }
    }
    __syncthreads();
    const bool bad = *failed != 0;
    if (tid == 0 && bad) atomicOr(err, 1u);
    // copies issued but never waited for by the MMAs (bounded), then every MMA issued
    if (warp == 4 && lane == 0)
        for (int it = s_issued; it < s_loaded; it++) mbar_wait(&full[it % WG_STAGES], (it / WG_STAGES) & 1);
    const bool computed = s_issued > 0 && mbar_wait(done, 0);
    if (__syncthreads_or(s_issued > 0 && !computed) && tid == 0) atomicOr(err, 1u);
    tc_fence_after();
    if (warp < 4 && !bad && computed) {
        atomicAdd(&dbs[lane], dbsum);
        for (int g = 0; g < NG; g++) {
            float v[32];
            tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(g * 32), v);
            const int m = warp * 32 + lane, t = g * TPG + m / CIN, i = m % CIN;
            if (t < 9)
#pragma unroll
                for (int o = 0; o < 32; o++) atomicAdd(&dw[(t * COUT + o) * CIN + i], v[o]);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid < 32 && !bad && computed && db != nullptr) atomicAdd(&db[tid], dbs[tid]);
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(NCOL));
}



// ---- the pipelined form of the 3x3 convolution ----------------------------------------------------------
//
// The same convolution with the tile loop overlapped: warp-specialised CTAs of 6 warps. Warp 4 (one thread)
// streams the tiles' halos by TMA into a ring of CP_STAGES stages; warp 5 (one thread) issues each tile's
// MMAs into one of two TMEM accumulators as soon as its halo has landed and that accumulator is free, and
// commits them to the stage's "empty" barrier (the halo may be overwritten) and to the accumulator's
// "full" barrier; warps 0-3 read a full accumulator back (each its 32 TMEM lanes), release it at once and run
// the epilogue while the next tile's MMAs fill the other accumulator. Every wait is bounded: a role that
// gives up sets the CTA's failure flag, every other role stops at its next wait, and the tile loop ends; the
// copies and MMAs still in flight are then waited for (bounded) before the TMEM is freed.
constexpr int CP_THREADS = 192;

// A tile of 256 output pixels: two MMAs of M = 128 a tap and K chunk. The halo it stages (51 pixels each side) is each
// plane's three boxes of 128 pixels. Stages: as many as keep two CTAs an SM (3 of 24 KB at CIN 32).
constexpr int CP_MT = 2;
constexpr int CP_PIXELS = CP_MT * TILE;
constexpr int CP_HALO = 3 * BOX_PIXELS;
constexpr int CP_STAGES = 3;
static_assert(CP_HALO >= CP_PIXELS + 2 * HALO_LO, "the halo covers every tap's rows");

template <int CIN>
constexpr int conv3x3p_smem_bytes() {
    return 9 * (CIN / 8) * COUT * 16 + CP_STAGES * (CIN / 8) * CP_HALO * 16 + (2 * CP_STAGES + 4) * 8 + 16;
}

// One 3x3 convolution layer (CIN input channels, 32 output channels) over the chunk-major padded rasters:
// y = act(conv(x, w) + bias), act = ReLU (relu != 0) or the identity, then times (mask > 0) when `mask` is set
// (the gradient through the layer's ReLU); the ring pixels of y are zero. w is [9 taps][32 out][CIN in] BF16,
// tap = 3 * dy + dx. x is read through `map` (BOX_PIXELS pixels of one plane a box); planes of mask and y are Q pixels
// apart, and the launch computes `pixels` of them (whole samples), in tiles = ceil(pixels / CP_PIXELS).
template <int CIN>
__global__ void __launch_bounds__(CP_THREADS, 1) conv3x3p_kernel(const __grid_constant__ CUtensorMap map, const __nv_bfloat16* __restrict__ w,
                                                                 const float* __restrict__ bias, int relu, const __nv_bfloat16* __restrict__ mask,
                                                                 __nv_bfloat16* __restrict__ y, long long Q, long long pixels, int tiles, unsigned* err) {
    constexpr int KC = CIN / 8, MT = CP_MT;
    constexpr int WBYTES = 9 * KC * COUT * 16;
    constexpr int HP = CP_HALO;                                // halo pixels a stage
    constexpr int HBYTES = KC * HP * 16;
    constexpr int TP = CP_PIXELS;                              // output pixels a tile
    constexpr int ACOLS = MT * COUT;                           // TMEM columns an accumulator
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* ws = smem;                                        // weights: [tap][chunk][out][16 B]
    uint8_t* halos = smem + WBYTES;                            // CP_STAGES x [chunk][HP pixels][16 B]
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + WBYTES + CP_STAGES * HBYTES);  // [CP_STAGES]
    uint64_t* empty = full + CP_STAGES;                        // [CP_STAGES]
    uint64_t* accf = empty + CP_STAGES;                        // [2] accumulator written
    uint64_t* acce = accf + 2;                                 // [2] accumulator read back
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acce + 2);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;  // this CTA's tiles

    for (int i = tid; i < 9 * COUT * CIN; i += CP_THREADS) {
        const int t = i / (COUT * CIN), n = (i / CIN) % COUT, k = i % CIN;
        *reinterpret_cast<__nv_bfloat16*>(ws + ((t * KC + k / 8) * COUT + n) * 16 + (k % 8) * 2) = w[i];
    }
    if (tid == 0) {
        for (int s = 0; s < CP_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&accf[a], 1);
            mbar_init(&acce[a], 4);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * ACOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    __shared__ int s_loaded, s_issued;
    if (warp == 4) {
        // the producer: the halo of tile it into stage it % CP_STAGES once the MMAs of its previous use are done
        int loaded = 0;
        if (lane == 0) {
            for (int it = 0; it < ntiles; it++) {
                const int s = it % CP_STAGES, k = it / CP_STAGES;
                if (k > 0 && !mbar_wait(&empty[s], (k - 1) & 1)) {
                    *failed = 1;
                    break;
                }
                if (*failed) break;
                const long long q0 = ((long long)blockIdx.x + (long long)it * gridDim.x) * TP;
                mbar_expect_tx(&full[s], HBYTES);
#pragma unroll
                for (int c = 0; c < KC; c++)
#pragma unroll
                    for (int m = 0; m < HP / BOX_PIXELS; m++)
                        tma_load(halos + s * HBYTES + (c * HP + m * BOX_PIXELS) * 16, &map, (int)(q0 - HALO_LO) + m * BOX_PIXELS, c, &full[s]);
                loaded = it + 1;
            }
            s_loaded = loaded;
        }
    } else if (warp == 5) {
        // the MMA issuer: tile it into accumulator it & 1
        const uint32_t issuer = lane == 0;
        int issued = 0;
        for (int it = 0; it < ntiles; it++) {
            const int s = it % CP_STAGES, k = it / CP_STAGES, a = it & 1, j = it >> 1;
            bool ok = mbar_wait(&full[s], k & 1);
            if (j > 0) ok = mbar_wait(&acce[a], (j - 1) & 1) && ok;
            if (!__all_sync(0xffffffffu, ok)) {
                *failed = 1;
                break;
            }
            if (__any_sync(0xffffffffu, *failed != 0)) break;
            tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(a * ACOLS);
            const uint64_t ad0 = smem_desc(smem_u32(halos) + (uint32_t)(s * HBYTES), HP * 16, 8 * 16);
            const uint64_t bd0 = smem_desc(smem_u32(ws), COUT * 16, 8 * 16);
#pragma unroll
            for (int t = 0; t < 9; t++)
#pragma unroll
                for (int kk = 0; kk < KC / 2; kk++)
#pragma unroll
                    for (int mh = 0; mh < MT; mh++)
                        mma_bf16(d + (uint32_t)(mh * COUT), ad0 + (uint64_t)(2 * kk * HP + HALO_LO + (t / 3 - 1) * RW + (t % 3 - 1) + mh * TILE),
                                 bd0 + (uint64_t)((t * KC + 2 * kk) * COUT), IDESC_BF16_M128_N32, (t | kk) != 0, issuer);
            if (issuer) {
                mma_commit(&empty[s]);
                mma_commit(&accf[a]);
            }
            __syncwarp();
            issued = it + 1;
        }
        if (issuer) s_issued = issued;
    } else {
        // the epilogue: warp w reads TMEM lanes 32w .. 32w + 31 (pixels), releases the accumulator, stores.
        // The bias stays in registers; a pixel's raster position comes from its tile's (one 64-bit remainder
        // a tile, the rest in 32 bits).
        float bv[32];
#pragma unroll
        for (int c = 0; c < 32; c++) bv[c] = bias != nullptr ? bias[c] : 0.f;
        for (int it = 0; it < ntiles; it++) {
            const int a = it & 1, j = it >> 1;
            const bool ok = mbar_wait(&accf[a], j & 1);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) *failed = 1;
                break;
            }
            tc_fence_after();
            float vv[MT][32];
#pragma unroll
            for (int mh = 0; mh < MT; mh++) tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(a * ACOLS + mh * COUT), vv[mh]);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[a]);
            const long long q0 = ((long long)blockIdx.x + (long long)it * gridDim.x) * TP;
            const int r0 = (int)(q0 % RPIX);
#pragma unroll
            for (int mh = 0; mh < MT; mh++) {
                const float (&v)[32] = vv[mh];
                const long long q = q0 + mh * TILE + warp * 32 + lane;
                if (q < pixels) {
                    int p = r0 + mh * TILE + warp * 32 + lane;
                    if (p >= RPIX) p -= RPIX;
                    const int ry = p / RW, rx = p - ry * RW;
                    const bool ring = ry == 0 || ry == RW - 1 || rx == 0 || rx == RW - 1;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        uint4 m4 = make_uint4(0, 0, 0, 0);
                        if (mask != nullptr) m4 = *reinterpret_cast<const uint4*>(mask + ((size_t)c * Q + q) * 8);
                        const __nv_bfloat16* mk = reinterpret_cast<const __nv_bfloat16*>(&m4);
                        __align__(16) __nv_bfloat16 o[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            float f = v[c * 8 + e] + bv[c * 8 + e];
                            if (relu) f = fmaxf(f, 0.f);
                            if (mask != nullptr && !(__bfloat162float(mk[e]) > 0.f)) f = 0.f;
                            o[e] = __float2bfloat16_rn(ring ? 0.f : f);
                        }
                        *reinterpret_cast<uint4*>(y + ((size_t)c * Q + q) * 8) = *reinterpret_cast<const uint4*>(o);
                    }
                }
            }
            if (__any_sync(0xffffffffu, *failed != 0)) break;
        }
    }
    __syncthreads();
    if (tid == 0 && *failed) atomicOr(err, 1u);
    if (warp == 4 && lane == 0) {
        // copies issued but never consumed, then the MMAs' last arrivals on the stages (bounded waits)
        for (int it = s_issued; it < s_loaded; it++) mbar_wait(&full[it % CP_STAGES], (it / CP_STAGES) & 1);
        for (int it = s_issued > CP_STAGES ? s_issued - CP_STAGES : 0; it < s_issued; it++)
            mbar_wait(&empty[it % CP_STAGES], (it / CP_STAGES) & 1);
    }
    if (warp == 5 && lane == 0 && s_issued > 0) mbar_wait(&accf[(s_issued - 1) & 1], ((s_issued - 1) >> 1) & 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * ACOLS));
}

}  // namespace tc
}  // namespace ironav
