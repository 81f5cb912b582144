// proposer.cuh — the learned proposer's kernels that are not contractions: its input from the pictures, the
// linear head (73,728 features -> 13 outputs) forward and backward, the loss, Adam, and the transposed weights
// of the backward convolutions. The network (the north star's form 4): 4 conv3x3 layers of 32 channels with
// ReLU on a 48 x 48 input of two channels — the current macroblock's 16 x 16 luma tiled 3 x 3 (so every
// position of the window meets the current samples) and the co-located 48 x 48 reference window (the macroblock
// at its centre, 16 samples around it, edges repeated) — both u8 / 255, then a linear head giving 4 candidate
// vectors (x, y in units of 32 luma samples: +-1 covers +-32) and 5 partition logits (P_Skip, 16x16, 16x8,
// 8x16, 8x8). Layer 1 takes 16 input channels (two planes) of which channels 0 and 1 carry the input.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

#include "tc_conv.cuh"

namespace ironav {
namespace prop {

constexpr int NOUT = 13;                  // 4 vectors x 2 + 5 logits
constexpr int NFEAT = 32 * 48 * 48;       // the head's inputs: layer 4's 32 channels x 48 x 48
constexpr float MV_SCALE = 128.f;         // quarter samples per output unit (32 luma samples)

// One training or proposal sample: the macroblock (mbx, mby) of the current picture `cur` predicted from `ref`
// (luma w x h, 8-bit; rows `stride` samples apart in cur, `ref_stride` in ref, 0 meaning `stride`).
struct Sample {
    const uint8_t* cur;
    const uint8_t* ref;
    int w, h, stride, mbx, mby, ref_stride;
};

// The input planes (two: channels 0-7 and 8-15, chunk-major padded) of n samples: a thread per pixel.
__global__ void prep_kernel(const Sample* __restrict__ samples, int n, __nv_bfloat16* __restrict__ x) {
    const long long Q = (long long)n * tc::RPIX;
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= Q) return;
    const int s = (int)(q / tc::RPIX), p = (int)(q % tc::RPIX), ry = p / tc::RW, rx = p % tc::RW;
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = __float2bfloat16_rn(0.f);
    if (ry > 0 && ry < tc::RW - 1 && rx > 0 && rx < tc::RW - 1) {
        const Sample S = samples[s];
        const int iy = ry - 1, ix = rx - 1;
        const int cx = min(S.mbx * 16 + (ix & 15), S.w - 1), cy = min(S.mby * 16 + (iy & 15), S.h - 1);
        const int wx = min(max(S.mbx * 16 - 16 + ix, 0), S.w - 1), wy = min(max(S.mby * 16 - 16 + iy, 0), S.h - 1);
        v[0] = __float2bfloat16_rn((float)S.cur[(size_t)cy * S.stride + cx] * (1.f / 255.f));
        v[1] = __float2bfloat16_rn((float)S.ref[(size_t)wy * (S.ref_stride > 0 ? S.ref_stride : S.stride) + wx] * (1.f / 255.f));
    }
    *reinterpret_cast<uint4*>(x + (size_t)q * 8) = *reinterpret_cast<const uint4*>(v);
    *reinterpret_cast<uint4*>(x + ((size_t)Q + q) * 8) = make_uint4(0, 0, 0, 0);
}

// Feature f of the head (channel c = f % 32, interior pixel (iy, ix) = (f / 32) / 48, (f / 32) % 48) of sample s
// in the chunk-major planes of Q pixels.
__device__ __forceinline__ size_t feat_index(int s, int f, long long Q) {
    const int c = f & 31, pix = f >> 5, iy = pix / 48, ix = pix % 48;
    const long long q = (long long)s * tc::RPIX + (iy + 1) * tc::RW + (ix + 1);
    return ((size_t)(c >> 3) * Q + q) * 8 + (c & 7);
}

// out[s][j] = hb[j] + sum_f hw[j][f] * feat(s, f): a CTA of 256 threads per HEAD_SPB samples, so that each
// weight read from L2 serves HEAD_SPB samples (the head's weights are 3.8 MB; every sample needs all of them).
constexpr int HEAD_SPB = 8;

__global__ void __launch_bounds__(256) head_fwd_kernel(const __nv_bfloat16* __restrict__ feat, long long Q, int n, const float* __restrict__ hw,
                                                       const float* __restrict__ hb, float* __restrict__ out) {
    const int s0 = blockIdx.x * HEAD_SPB, tid = threadIdx.x;
    const int ns = min(HEAD_SPB, n - s0);
    float acc[HEAD_SPB][NOUT];
#pragma unroll
    for (int i = 0; i < HEAD_SPB; i++)
#pragma unroll
        for (int j = 0; j < NOUT; j++) acc[i][j] = 0.f;
    for (int f = tid; f < NFEAT; f += 256) {
        float wj[NOUT];
#pragma unroll
        for (int j = 0; j < NOUT; j++) wj[j] = __ldg(&hw[(size_t)j * NFEAT + f]);
#pragma unroll
        for (int i = 0; i < HEAD_SPB; i++) {
            const float v = i < ns ? __bfloat162float(feat[feat_index(s0 + i, f, Q)]) : 0.f;
#pragma unroll
            for (int j = 0; j < NOUT; j++) acc[i][j] += v * wj[j];
        }
    }
    __shared__ float red[8][HEAD_SPB * NOUT];
#pragma unroll
    for (int i = 0; i < HEAD_SPB; i++)
#pragma unroll
        for (int j = 0; j < NOUT; j++) {
            float a = acc[i][j];
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if ((tid & 31) == 0) red[tid >> 5][i * NOUT + j] = a;
        }
    __syncthreads();
    if (tid < HEAD_SPB * NOUT) {
        const int i = tid / NOUT, j = tid % NOUT;
        if (i < ns) {
            float a = hb[j];
            for (int w = 0; w < 8; w++) a += red[w][tid];
            out[(size_t)(s0 + i) * NOUT + j] = a;
        }
    }
}

// The head's weights packed for head_fwd_packed_kernel: hwt[f][16] = hw[j][f] for j < 13, zero after, so that
// a feature's 13 weights are four 16-byte loads.
__global__ void head_pack_kernel(const float* __restrict__ hw, float* __restrict__ hwt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NFEAT * 16) return;
    const int f = i >> 4, j = i & 15;
    hwt[i] = j < NOUT ? hw[(size_t)j * NFEAT + f] : 0.f;
}

// Two FP32 multiply-adds an instruction (each lane of the pair is an IEEE fma): the head's kernels are bound by
// instruction issue, and the pair halves it.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_pack(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(F2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// The two BF16 values of a word as FP32.
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// 16 bytes from global to shared memory, asynchronously, and the waits for all but the newest N groups of them. A lane of
// the head's kernels stages what it alone reads, so its own wait orders the copy; the ring's depth, not the
// registers, then sets how many bytes an SM has in flight.
__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int HEAD_CHUNK = 16;    // pixels whose packed weights a CTA holds in shared memory at a time
constexpr int HEAD_WPIX = 32 * 4 + 1;  // float4s a pixel's weights take in shared memory: 32 channels x 4, and a
                                       // pad that puts a warp's four pixels on different banks
constexpr int HEAD_SPL = 8;       // samples a lane
constexpr int HEAD_SAMPLES = 512; // samples a CTA (8 warps of 8 x HEAD_SPL samples x 4 pixels)

// The head: CTA (x, y) takes samples 512x .. 512x + 511 and interior pixels pix * y .. pix * (y + 1) - 1. Lane
// l of warp w takes samples 512x + 64w + 8 (l / 4) + k (k < 8) and every fourth pixel from l % 4, so a warp's
// feature loads are 64 contiguous bytes a sample (four pixels of one plane), and each weight read from shared
// memory serves eight samples: with four, the shared-memory reads took as long as the multiply-adds. The CTA stages
// the packed weights of HEAD_CHUNK pixels at a time in shared memory (coalesced); a warp reads four pixels' weights at
// once (four addresses on different banks). Outputs go in pairs (f2_fma; the 14th's weights are zero). The four lanes
// of a sample are summed by shuffles and added to out (which CTAs y = 0 start from the bias; out must be zero before
// the launch). The pixels a CTA takes are the launch's choice, so that few samples still fill the chip (at 512 samples
// 18 slices of 128 pixels kept 36 SMs busy: 191 us, now 52). A step's samples are loaded a step ahead.
// 8160 samples: 525 us with four samples a lane and scalar multiply-adds, 495 with eight and pairs, 381 with the loads ahead.
__global__ void __launch_bounds__(256, 1) head_fwd_packed_kernel(const __nv_bfloat16* __restrict__ feat, long long Q, int n,
                                                                 const float4* __restrict__ hwt, const float* __restrict__ hb,
                                                                 float* __restrict__ out, int pix) {
    __shared__ float4 ws[HEAD_CHUNK * HEAD_WPIX];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pl = lane & 3;
    const int s0 = blockIdx.x * HEAD_SAMPLES + warp * (8 * HEAD_SPL) + (lane >> 2) * HEAD_SPL;
    const int p0 = blockIdx.y * pix, p1 = min(p0 + pix, 48 * 48);
    F2 acc[HEAD_SPL][7];
#pragma unroll
    for (int k = 0; k < HEAD_SPL; k++)
#pragma unroll
        for (int j = 0; j < 7; j++) acc[k][j] = 0ull;
    uint4 ahead[HEAD_SPL];
    auto load = [&](uint4 (&v)[HEAD_SPL], int c, int px) {
        const int iy = px / 48, rq = (iy + 1) * tc::RW + (px - iy * 48) + 1;
#pragma unroll
        for (int k = 0; k < HEAD_SPL; k++)
            v[k] = s0 + k < n ? *reinterpret_cast<const uint4*>(feat + ((size_t)c * Q + (long long)(s0 + k) * tc::RPIX + rq) * 8)
                              : make_uint4(0, 0, 0, 0);
    };
    load(ahead, 0, p0 + pl);
    for (int c0 = p0; c0 < p1; c0 += HEAD_CHUNK) {
        const int np = min(HEAD_CHUNK, p1 - c0);  // a multiple of 4: 2304, pix and the chunk are
        __syncthreads();
        for (int i = threadIdx.x; i < np * 128; i += 256) ws[(i >> 7) * HEAD_WPIX + (i & 127)] = __ldg(hwt + (size_t)c0 * 128 + i);
        __syncthreads();
        for (int pp = pl; pp < np; pp += 4) {
            const int px = c0 + pp;
            const float4* wp = ws + pp * HEAD_WPIX;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                // this step's samples, loaded a step ago, and the next step's (the next plane, or the next pixel's first)
                uint4 raw[HEAD_SPL];
#pragma unroll
                for (int k = 0; k < HEAD_SPL; k++) raw[k] = ahead[k];
                if (c < 3) load(ahead, c + 1, px);
                else if (pp + 4 < np || c0 + HEAD_CHUNK < p1) load(ahead, 0, px + 4);
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const float4* wf = wp + ((c * 8 + e) << 2);
                    const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(wf), wb = *reinterpret_cast<const ulonglong2*>(wf + 1),
                                     wc = *reinterpret_cast<const ulonglong2*>(wf + 2);
                    const F2 wd = *reinterpret_cast<const F2*>(wf + 3);
#pragma unroll
                    for (int k = 0; k < HEAD_SPL; k++) {
                        const uint32_t word = e < 2 ? raw[k].x : (e < 4 ? raw[k].y : (e < 6 ? raw[k].z : raw[k].w));
                        const float x = (e & 1) ? bf_hi(word) : bf_lo(word);
                        const F2 xx = f2_pack(x, x);
                        acc[k][0] = f2_fma(xx, wa.x, acc[k][0]);
                        acc[k][1] = f2_fma(xx, wa.y, acc[k][1]);
                        acc[k][2] = f2_fma(xx, wb.x, acc[k][2]);
                        acc[k][3] = f2_fma(xx, wb.y, acc[k][3]);
                        acc[k][4] = f2_fma(xx, wc.x, acc[k][4]);
                        acc[k][5] = f2_fma(xx, wc.y, acc[k][5]);
                        acc[k][6] = f2_fma(xx, wd, acc[k][6]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < HEAD_SPL; k++) {
        float o[14];
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const float2 v = f2_unpack(acc[k][j]);
            o[2 * j] = v.x;
            o[2 * j + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < NOUT; j++) {
            o[j] += __shfl_xor_sync(0xffffffffu, o[j], 1);
            o[j] += __shfl_xor_sync(0xffffffffu, o[j], 2);
        }
        if (pl == 0 && s0 + k < n)
#pragma unroll
            for (int j = 0; j < NOUT; j++) atomicAdd(&out[(size_t)(s0 + k) * NOUT + j], o[j] + (blockIdx.y == 0 ? hb[j] : 0.f));
    }
}

// The loss of n samples and its gradient d_out (already divided by n): winner-takes-all L1 on the vectors (the
// candidate nearest the target, plus 0.05 of every candidate's distance so that none is left untrained) and
// cross-entropy on the partition logits. target_mv in quarter samples; target_part in 0..4. sums[0] += the
// vector loss, sums[1] += the partition loss, sums[2] += the partition hits (top-1).
__global__ void loss_kernel(const float* __restrict__ out, const int16_t* __restrict__ target_mv, const uint8_t* __restrict__ target_part, int n,
                            float* __restrict__ dout, float* __restrict__ sums) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float* o = out + (size_t)s * NOUT;
    float* d = dout + (size_t)s * NOUT;
    const float tx = target_mv[2 * s] / MV_SCALE, ty = target_mv[2 * s + 1] / MV_SCALE;
    int best = 0;
    float bd = 1e30f, dist[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        dist[k] = fabsf(o[2 * k] - tx) + fabsf(o[2 * k + 1] - ty);
        if (dist[k] < bd) bd = dist[k], best = k;
    }
    float lmv = bd;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        lmv += 0.05f * dist[k];
        const float wk = (k == best ? 1.f : 0.f) + 0.05f;
        d[2 * k] = wk * (o[2 * k] > tx ? 1.f : (o[2 * k] < tx ? -1.f : 0.f)) / n;
        d[2 * k + 1] = wk * (o[2 * k + 1] > ty ? 1.f : (o[2 * k + 1] < ty ? -1.f : 0.f)) / n;
    }
    float m = o[8];
    int arg = 0;
    for (int c = 1; c < 5; c++)
        if (o[8 + c] > m) m = o[8 + c], arg = c;
    float z = 0.f;
    for (int c = 0; c < 5; c++) z += __expf(o[8 + c] - m);
    const int t = target_part[s];
    const float lce = logf(z) - (o[8 + t] - m);
    for (int c = 0; c < 5; c++) d[8 + c] = (__expf(o[8 + c] - m) / z - (c == t ? 1.f : 0.f)) / n;
    atomicAdd(&sums[0], lmv);
    atomicAdd(&sums[1], lce);
    atomicAdd(&sums[2], arg == t ? 1.f : 0.f);
}

constexpr int HB_CHUNK = 128;  // samples whose output gradients a CTA of the head's backward kernels holds at a time
constexpr int HB_SLICE = 64;   // samples a CTA of head_dgrad_kernel takes
constexpr int HB_RING = 8;     // samples a lane of head_dgrad_kernel has staged or in flight
constexpr int HB_UNITS = 128;  // (plane, raster pixel) units a CTA of head_dgrad_kernel takes

// A pixel's 8 channels of one plane; features that are not 16-byte aligned (a caller's own buffer) by halfwords.
__device__ __forceinline__ uint4 ld8(const __nv_bfloat16* p, bool aligned) {
    if (aligned) return *reinterpret_cast<const uint4*>(p);
    const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
    return make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16, h[6] | (uint32_t)h[7] << 16);
}

// Samples s0 .. s0 + k - 1's output gradients into d, each doubled for f2_fma (13 of them and a zero). Returns whether this thread
// saw one that is not finite.
__device__ __forceinline__ bool stage_dout(F2 (*d)[14], const float* __restrict__ dout, int s0, int k) {
    bool odd = false;
    for (int i = threadIdx.x; i < k * 14; i += blockDim.x) {
        const int s = i / 14, j = i - s * 14;
        const float v = j < NOUT ? dout[(size_t)(s0 + s) * NOUT + j] : 0.f;
        d[s][j] = f2_pack(v, v);
        odd |= !isfinite(v);
    }
    return odd;
}

// The head's weight and bias gradients: ghw[j][f] += sum_s dout[s][j] * feat(s, f). Lane l of a CTA's 8 warps takes the
// 8 channels of one (plane, interior pixel), 16 bytes a sample in runs of 512 a warp, with 8 x 13 sums in
// registers; the warps split the samples and add their sums through shared memory, so each gradient is written
// once. (A thread a feature read 2 bytes a sample 16 apart: 381 us at 512 samples; now 58.)
__global__ void __launch_bounds__(256) head_wgrad_kernel(const __nv_bfloat16* __restrict__ feat, long long Q, int n, const float* __restrict__ dout,
                                                         float* __restrict__ ghw, float* __restrict__ ghb) {
    __shared__ __align__(16) F2 d[HB_CHUNK][14];
    __shared__ float red[8][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u = blockIdx.x * 32 + lane, c = u / 2304, pix = u - c * 2304, iy = pix / 48, ix = pix - iy * 48;
    const __nv_bfloat16* base = feat + ((size_t)c * Q + (iy + 1) * tc::RW + (ix + 1)) * 8;
    const bool aligned = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;
    F2 acc[NOUT][4];
#pragma unroll
    for (int j = 0; j < NOUT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[j][e] = 0ull;
    bool odd = false;
    for (int s0 = 0; s0 < n; s0 += HB_CHUNK) {
        const int k = min(HB_CHUNK, n - s0);
        __syncthreads();
        odd |= stage_dout(d, dout, s0, k);
        __syncthreads();
#pragma unroll 4
        for (int s = warp; s < k; s += 8) {
            const uint4 r = ld8(base + (size_t)(s0 + s) * (tc::RPIX * 8), aligned);
            const F2 x[4] = {f2_pack(bf_lo(r.x), bf_hi(r.x)), f2_pack(bf_lo(r.y), bf_hi(r.y)), f2_pack(bf_lo(r.z), bf_hi(r.z)),
                             f2_pack(bf_lo(r.w), bf_hi(r.w))};
#pragma unroll
            for (int j = 0; j < NOUT; j++) {
                const F2 dj = d[s][j];
#pragma unroll
                for (int e = 0; e < 4; e++) acc[j][e] = f2_fma(x[e], dj, acc[j][e]);
            }
        }
    }
    if (__syncthreads_or(odd)) {
        // an output gradient that is not finite belongs to the features that are not zero alone (0 times it is no number): once more,
        // feature by feature
#pragma unroll
        for (int j = 0; j < NOUT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[j][e] = 0ull;
        for (int s = warp; s < n; s += 8) {
            const uint4 r = ld8(base + (size_t)s * (tc::RPIX * 8), aligned);
            const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int j = 0; j < NOUT; j++) {
                const float dj = dout[(size_t)s * NOUT + j];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float x0 = bf_lo(rr[e]), x1 = bf_hi(rr[e]);
                    acc[j][e] = f2_fma(f2_pack(x0, x1), f2_pack(x0 != 0.f ? dj : 0.f, x1 != 0.f ? dj : 0.f), acc[j][e]);
                }
            }
        }
    }
    // thread t sums feature t % 8 of unit t / 8 over the warps
    const int u2 = blockIdx.x * 32 + (threadIdx.x >> 3), c2 = u2 / 2304, pix2 = u2 - c2 * 2304;
    float* g = ghw + (size_t)pix2 * 32 + c2 * 8 + (threadIdx.x & 7);
#pragma unroll
    for (int j = 0; j < NOUT; j++) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; e++) *reinterpret_cast<F2*>(&red[warp][lane * 8 + 2 * e]) = acc[j][e];
        __syncthreads();
        float a = 0.f;
#pragma unroll
        for (int w = 0; w < 8; w++) a += red[w][threadIdx.x];
        g[(size_t)j * NFEAT] += a;
    }
    if (blockIdx.x == 0 && ghb != nullptr)
        for (int j = warp; j < NOUT; j += 8) {
            float a = 0.f;
            for (int s = lane; s < n; s += 32) a += dout[(size_t)s * NOUT + j];
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (lane == 0) ghb[j] += a;
        }
}

// The gradient into layer 4's output through its ReLU: dz(s, f) = (feat(s, f) > 0) * sum_j dout[s][j] hw[j][f],
// into the chunk-major planes dz, the ring's zeros included: a thread per (plane, raster pixel) and HB_SLICE
// samples, its 8 channels' 13 weights in registers, 16 bytes read and written a sample. (A thread a
// (sample, feature), 2 bytes each and the weights from L2, after a pass that cleared dz: 217 + 10 us at 512 samples; now 67.)
__global__ void __launch_bounds__(HB_UNITS) head_dgrad_kernel(const __nv_bfloat16* __restrict__ feat, long long Q, int n, const float* __restrict__ dout,
                                                              const float* __restrict__ hw, __nv_bfloat16* __restrict__ dz) {
    __shared__ __align__(16) F2 d[HB_SLICE][14];
    __shared__ __align__(16) uint4 ring[HB_RING][HB_UNITS];
    const int s0 = blockIdx.x * HB_SLICE, k = min(HB_SLICE, n - s0);
    stage_dout(d, dout, s0, k);
    __syncthreads();
    const int u = blockIdx.y * HB_UNITS + threadIdx.x;
    if (u >= 4 * tc::RPIX) return;
    const int c = u / tc::RPIX, p = u - c * tc::RPIX, ry = p / tc::RW, rx = p - ry * tc::RW;
    const size_t at = ((size_t)c * Q + (size_t)s0 * tc::RPIX + p) * 8;
    if (ry == 0 || ry == tc::RW - 1 || rx == 0 || rx == tc::RW - 1) {
        for (int s = 0; s < k; s++) *reinterpret_cast<uint4*>(dz + at + (size_t)s * (tc::RPIX * 8)) = make_uint4(0, 0, 0, 0);
        return;
    }
    const bool aligned = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;
    auto issue = [&](int s) {
        if (s < k) {
            const __nv_bfloat16* g = feat + at + (size_t)s * (tc::RPIX * 8);
            if (aligned) cp16(&ring[s % HB_RING][threadIdx.x], g);
            else ring[s % HB_RING][threadIdx.x] = ld8(g, false);
        }
        cp_commit();
    };
#pragma unroll
    for (int i = 0; i < HB_RING - 1; i++) issue(i);
    const bool waligned = (reinterpret_cast<uintptr_t>(hw) & 15) == 0;
    F2 w[NOUT][4];
    const float* wsrc = hw + (size_t)((ry - 1) * 48 + rx - 1) * 32 + c * 8;
#pragma unroll
    for (int j = 0; j < NOUT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float* q = wsrc + (size_t)j * NFEAT + 2 * e;
            if (!waligned) w[j][e] = f2_pack(__ldg(q), __ldg(q + 1));
            else if (e % 2 == 0) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(q));
                w[j][e] = f2_pack(v.x, v.y);
                w[j][e + 1] = f2_pack(v.z, v.w);
            }
        }
    for (int s = 0; s < k; s++) {
        issue(s + HB_RING - 1);
        cp_wait<HB_RING - 1>();
        const uint4 r = ring[s % HB_RING][threadIdx.x];
        F2 a[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
        for (int j = 0; j < NOUT; j++) {
            const F2 dj = d[s][j];
#pragma unroll
            for (int e = 0; e < 4; e++) a[e] = f2_fma(dj, w[j][e], a[e]);
        }
        const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 v = f2_unpack(a[e]);
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(bf_lo(rr[e]) > 0.f ? v.x : 0.f, bf_hi(rr[e]) > 0.f ? v.y : 0.f);
            o[e] = *reinterpret_cast<const uint32_t*>(&b2);
        }
        *reinterpret_cast<uint4*>(dz + at + (size_t)s * (tc::RPIX * 8)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// Adam (bias-corrected) on a flat parameter vector; the gradient is cleared after its use.
__global__ void adam_kernel(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, long long n, float lr,
                            float b1, float b2, float c1, float c2, float eps) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    g[i] = 0.f;
}

// The BF16 weights of a layer for its forward convolution ([9][32][cin], as the master) and, when wt is set, the
// transposed and mirrored ones of its data gradient: wt[t][i][o] = w[8 - t][o][i] (cin = 32).
__global__ void weights_kernel(const float* __restrict__ w, int cin, __nv_bfloat16* __restrict__ wf, __nv_bfloat16* __restrict__ wt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 9 * 32 * cin) return;
    wf[i] = __float2bfloat16_rn(w[i]);
    if (wt != nullptr) {
        const int t = i / (32 * cin), o = (i / cin) % 32, k = i % cin;
        wt[((8 - t) * 32 + k) * 32 + o] = __float2bfloat16_rn(w[i]);
    }
}

// The judge's inputs: 4 vectors in quarter samples (the outputs times MV_SCALE, rounded to nearest, clamped to
// the search's range) and the class of largest logit (the first on ties) when its softmax probability is at
// least min_conf, else 5 (unsure), a thread per sample.
__global__ void propose_kernel(const float* __restrict__ out, int n, float min_conf, int16_t* __restrict__ cands, uint8_t* __restrict__ cls) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const float* o = out + (size_t)s * NOUT;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float x = fminf(fmaxf(rintf(o[2 * k] * MV_SCALE), -2048.f), 2047.f);
        const float y = fminf(fmaxf(rintf(o[2 * k + 1] * MV_SCALE), -512.f), 511.f);
        cands[(size_t)s * 8 + 2 * k] = (int16_t)x;
        cands[(size_t)s * 8 + 2 * k + 1] = (int16_t)y;
    }
    int arg = 0;
    float m = o[8];
    for (int c = 1; c < 5; c++)
        if (o[8 + c] > m) m = o[8 + c], arg = c;
    float z = 0.f;
    for (int c = 0; c < 5; c++) z += __expf(o[8 + c] - m);
    cls[s] = (uint8_t)(1.f / z >= min_conf ? arg : 5);
}

}  // namespace prop
}  // namespace ironav
