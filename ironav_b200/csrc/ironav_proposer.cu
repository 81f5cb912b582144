// ironav_proposer.cu — the learned proposer's kernels behind the C ABI (the north star's form 4): its 3x3
// convolutions and their weight gradients on the tensor cores (tc_conv.cuh), and its input, head, loss and
// optimizer on the CUDA cores (proposer.cuh). Every entry point queues its work on the given stream and
// returns; a device wait that gave up sets bit 0 of the caller's error word `err` (device memory), which the
// caller reads once a step. The TMA tensor maps are made on the host, through the driver's
// cuTensorMapEncodeTiled reached via the runtime (no link against libcuda).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../include/ironav_inter.h"
#include "proposer.cuh"
#include "tc_conv.cuh"

using namespace ironav::tc;
namespace prop = ironav::prop;

static_assert(sizeof(ironav_prop_sample) == sizeof(prop::Sample), "ironav_prop_sample layout");

namespace {

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return IRONAV_OK;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver || e == cudaErrorNoKernelImageForDevice)
        return IRONAV_HARDWARE_UNAVAILABLE;
    return IRONAV_INTERNAL;
}

#define CK(x)                                          \
    do {                                               \
        cudaError_t e_ = (x);                          \
        if (e_ != cudaSuccess) return cuda_status(e_); \
    } while (0)

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                 CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver, through the runtime.
EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// The tensor map of `pixels` pixels of a chunk-major padded tensor (planes of Q pixels x 8 BF16) from `base`, read in
// boxes of BOX_PIXELS pixels of `box_planes` planes. A plane's pixels are one run of 16-byte pieces, so the map calls
// it a row of 64-bit elements, two a pixel: dims (2 * pixels, planes), byte stride 16 Q, and a box moves rows of 2 KB.
// (With the 8 channels as the innermost dimension a box moved rows of 16 bytes, a piece a clock: 512 samples' weight
// gradient of 32 channels took 199 us, and with this map and the pipeline around it 79 us; the convolution 631 -> 583 us at 8160.)
// Out-of-range pixels read as zeros.
int plane_map(CUtensorMap* map, const void* base, long long Q, long long pixels, int planes, int box_planes) {
    EncodeTiled enc = encode_fn();
    if (!enc) return IRONAV_HARDWARE_UNAVAILABLE;
    if (reinterpret_cast<uintptr_t>(base) & 15) return IRONAV_INVALID_ARGUMENT;
    const cuuint64_t dims[2] = {(cuuint64_t)pixels * 2, (cuuint64_t)planes};
    const cuuint64_t strides[1] = {(cuuint64_t)Q * 16};
    const cuuint32_t box[2] = {2 * BOX_PIXELS, (cuuint32_t)box_planes};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? IRONAV_OK : IRONAV_INVALID_ARGUMENT;
}

// Samples a launch takes: a box's first element (two a pixel) is a 32-bit coordinate, so a larger batch goes in several launches.
// A sample's interior pixels depend on its own raster only, so a batch may be cut between any two samples.
constexpr long long LAUNCH_SAMPLES = 400000;
static_assert(LAUNCH_SAMPLES * RPIX * 2 < (1ll << 31), "box coordinates fit 32 bits");

int sm_count(int* nsm) {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev));
    return IRONAV_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// A batch of the convolution in launches of at most `per_launch` samples.
int conv3x3(const void* d_x, int cin, long long samples, const void* d_w, const float* d_bias, int relu, const void* d_mask, void* d_y, unsigned* d_err,
            void* stream, long long per_launch) {
    if (!d_x || !d_w || !d_y || !d_err || (cin != 16 && cin != 32) || samples < 1 || samples > (1ll << 22)) return IRONAV_INVALID_ARGUMENT;
    if (!aligned16(d_y) || !aligned16(d_mask)) return IRONAV_INVALID_ARGUMENT;
    const long long Q = samples * RPIX;
    int nsm = 0;
    int s = sm_count(&nsm);
    if (s != IRONAV_OK) return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(d_w);
    for (long long s0 = 0; s0 < samples; s0 += per_launch) {
        const long long q0 = s0 * RPIX, pixels = std::min(samples - s0, per_launch) * RPIX;
        const int tiles = (int)((pixels + CP_PIXELS - 1) / CP_PIXELS);
        CUtensorMap map;
        if ((s = plane_map(&map, static_cast<const uint8_t*>(d_x) + q0 * 16, Q, pixels, cin / 8, 1)) != IRONAV_OK) return s;
        // two persistent CTAs an SM
        const int grid = std::min(tiles, nsm * 2);
        const __nv_bfloat16* mask = d_mask ? static_cast<const __nv_bfloat16*>(d_mask) + q0 * 8 : nullptr;
        __nv_bfloat16* y = static_cast<__nv_bfloat16*>(d_y) + q0 * 8;
        if (cin == 32) {
            constexpr int bytes = conv3x3p_smem_bytes<32>();
            CK(cudaFuncSetAttribute(conv3x3p_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
            conv3x3p_kernel<32><<<grid, CP_THREADS, bytes, st>>>(map, w, d_bias, relu, mask, y, Q, pixels, tiles, d_err);
        } else {
            constexpr int bytes = conv3x3p_smem_bytes<16>();
            CK(cudaFuncSetAttribute(conv3x3p_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
            conv3x3p_kernel<16><<<grid, CP_THREADS, bytes, st>>>(map, w, d_bias, relu, mask, y, Q, pixels, tiles, d_err);
        }
        CK(cudaGetLastError());
    }
    return IRONAV_OK;
}

// A batch of the weight gradient in launches of at most `per_launch` samples.
int wgrad3x3(const void* d_x, int cin, const void* d_dz, long long samples, float* d_dw, float* d_db, unsigned* d_err, void* stream,
             long long per_launch) {
    if (!d_x || !d_dz || !d_dw || !d_err || (cin != 16 && cin != 32) || samples < 1 || samples > (1ll << 22)) return IRONAV_INVALID_ARGUMENT;
    const long long Q = samples * RPIX;
    int nsm = 0;
    int s = sm_count(&nsm);
    if (s != IRONAV_OK) return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (long long s0 = 0; s0 < samples; s0 += per_launch) {
        const long long q0 = s0 * RPIX, pixels = std::min(samples - s0, per_launch) * RPIX;
        const int tiles = (int)((pixels + WG_KT - 1) / WG_KT);
        CUtensorMap xmap, zmap;
        s = plane_map(&xmap, static_cast<const uint8_t*>(d_x) + q0 * 16, Q, pixels, cin / 8, cin / 8);
        if (s == IRONAV_OK) s = plane_map(&zmap, static_cast<const uint8_t*>(d_dz) + q0 * 16, Q, pixels, 4, 4);
        if (s != IRONAV_OK) return s;
        const int grid = std::min(tiles, nsm);
        if (cin == 32) {
            constexpr int bytes = wgrad3x3_smem_bytes<32>();
            CK(cudaFuncSetAttribute(wgrad3x3_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
            wgrad3x3_kernel<32><<<grid, WG_THREADS, bytes, st>>>(xmap, zmap, d_dw, d_db, tiles, d_err);
        } else {
            constexpr int bytes = wgrad3x3_smem_bytes<16>();
            CK(cudaFuncSetAttribute(wgrad3x3_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
            wgrad3x3_kernel<16><<<grid, WG_THREADS, bytes, st>>>(xmap, zmap, d_dw, d_db, tiles, d_err);
        }
        CK(cudaGetLastError());
    }
    return IRONAV_OK;
}

}  // namespace

extern "C" {

int ironav_prop_conv3x3(const void* d_x, int cin, long long samples, const void* d_w, const float* d_bias, int relu, const void* d_mask,
                        void* d_y, unsigned* d_err, void* stream) {
    return conv3x3(d_x, cin, samples, d_w, d_bias, relu, d_mask, d_y, d_err, stream, LAUNCH_SAMPLES);
}

int ironav_prop_wgrad3x3(const void* d_x, int cin, const void* d_dz, long long samples, float* d_dw, float* d_db, unsigned* d_err,
                         void* stream) {
    return wgrad3x3(d_x, cin, d_dz, samples, d_dw, d_db, d_err, stream, LAUNCH_SAMPLES);
}

// Test hooks (not in the public header): the same with the samples a launch takes.
int ironav_debug_prop_conv3x3(const void* d_x, int cin, long long samples, const void* d_w, const float* d_bias, int relu, const void* d_mask,
                              void* d_y, unsigned* d_err, void* stream, long long per_launch) {
    if (per_launch < 1 || per_launch > LAUNCH_SAMPLES) return IRONAV_INVALID_ARGUMENT;
    return conv3x3(d_x, cin, samples, d_w, d_bias, relu, d_mask, d_y, d_err, stream, per_launch);
}

int ironav_debug_prop_wgrad3x3(const void* d_x, int cin, const void* d_dz, long long samples, float* d_dw, float* d_db, unsigned* d_err,
                               void* stream, long long per_launch) {
    if (per_launch < 1 || per_launch > LAUNCH_SAMPLES) return IRONAV_INVALID_ARGUMENT;
    return wgrad3x3(d_x, cin, d_dz, samples, d_dw, d_db, d_err, stream, per_launch);
}

int ironav_prop_prep(const ironav_prop_sample* d_samples, int n, void* d_x, void* stream) {
    if (!d_samples || !d_x || n < 1 || n > (1 << 22) || !aligned16(d_x)) return IRONAV_INVALID_ARGUMENT;
    const long long Q = (long long)n * RPIX;
    prop::prep_kernel<<<(unsigned)((Q + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const prop::Sample*>(d_samples), n, static_cast<__nv_bfloat16*>(d_x));
    return cuda_status(cudaGetLastError());
}

int ironav_prop_head_fwd(const void* d_feat, int n, const float* d_hw, const float* d_hb, float* d_out, void* stream) {
    if (!d_feat || !d_hw || !d_hb || !d_out || n < 1 || n > (1 << 22)) return IRONAV_INVALID_ARGUMENT;
    prop::head_fwd_kernel<<<(n + prop::HEAD_SPB - 1) / prop::HEAD_SPB, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(d_feat), (long long)n * RPIX, n, d_hw, d_hb, d_out);
    return cuda_status(cudaGetLastError());
}

int ironav_prop_head_pack(const float* d_hw, float* d_hwt, void* stream) {
    if (!d_hw || !d_hwt || !aligned16(d_hwt)) return IRONAV_INVALID_ARGUMENT;
    prop::head_pack_kernel<<<(prop::NFEAT * 16 + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_hw, d_hwt);
    return cuda_status(cudaGetLastError());
}

int ironav_prop_head_fwd_packed(const void* d_feat, int n, const float* d_hwt, const float* d_hb, float* d_out, void* stream) {
    if (!d_feat || !d_hwt || !d_hb || !d_out || n < 1 || n > (1 << 22) || !aligned16(d_hwt)) return IRONAV_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CK(cudaMemsetAsync(d_out, 0, (size_t)n * prop::NOUT * sizeof(float), st));
    int nsm = 0;
    const int r = sm_count(&nsm);
    if (r != IRONAV_OK) return r;
    // pixels a CTA: as few as give two waves of CTAs (one an SM), in whole chunks; at most 128, which the sums over a
    // picture's samples (two waves already) are fastest with
    const int sg = (n + prop::HEAD_SAMPLES - 1) / prop::HEAD_SAMPLES, slices = std::max(1, std::min(144, 2 * nsm / sg));
    const int pix = std::min(128, (2304 / prop::HEAD_CHUNK + slices - 1) / slices * prop::HEAD_CHUNK);
    prop::head_fwd_packed_kernel<<<dim3(sg, (2304 + pix - 1) / pix), 256, 0, st>>>(static_cast<const __nv_bfloat16*>(d_feat), (long long)n * RPIX, n,
                                                                                    reinterpret_cast<const float4*>(d_hwt), d_hb, d_out, pix);
    return cuda_status(cudaGetLastError());
}

int ironav_prop_loss(const float* d_out, const int16_t* d_target_mv, const uint8_t* d_target_part, int n, float* d_dout, float* d_sums,
                     void* stream) {
    if (!d_out || !d_target_mv || !d_target_part || !d_dout || !d_sums || n < 1) return IRONAV_INVALID_ARGUMENT;
    prop::loss_kernel<<<(n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(d_out, d_target_mv, d_target_part, n, d_dout, d_sums);
    return cuda_status(cudaGetLastError());
}

int ironav_prop_head_bwd(const void* d_feat, int n, const float* d_dout, const float* d_hw, float* d_ghw, float* d_ghb, void* d_dz,
                         void* stream) {
    if (!d_feat || !d_dout || !d_hw || !d_ghw || !d_dz || n < 1 || n > (1 << 22) || !aligned16(d_dz)) return IRONAV_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long Q = (long long)n * RPIX;
    const __nv_bfloat16* feat = static_cast<const __nv_bfloat16*>(d_feat);
    prop::head_wgrad_kernel<<<4 * 2304 / 32, 256, 0, st>>>(feat, Q, n, d_dout, d_ghw, d_ghb);
    const dim3 grid((n + prop::HB_SLICE - 1) / prop::HB_SLICE, (4 * RPIX + prop::HB_UNITS - 1) / prop::HB_UNITS);
    prop::head_dgrad_kernel<<<grid, prop::HB_UNITS, 0, st>>>(feat, Q, n, d_dout, d_hw, static_cast<__nv_bfloat16*>(d_dz));
    return cuda_status(cudaGetLastError());
}

int ironav_prop_adam(float* d_p, float* d_g, float* d_m, float* d_v, long long n, float lr, float beta1, float beta2, int step, float eps,
                     void* stream) {
    if (!d_p || !d_g || !d_m || !d_v || n < 1 || step < 1) return IRONAV_INVALID_ARGUMENT;
    const float c1 = 1.f - std::pow(beta1, (float)step), c2 = 1.f - std::pow(beta2, (float)step);
    prop::adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(d_p, d_g, d_m, d_v, n, lr, beta1, beta2, c1,
                                                                                                   c2, eps);
    return cuda_status(cudaGetLastError());
}

int ironav_prop_weights(const float* d_w, int cin, void* d_wf, void* d_wt, void* stream) {
    if (!d_w || !d_wf || (cin != 16 && cin != 32) || (d_wt && cin != 32)) return IRONAV_INVALID_ARGUMENT;
    prop::weights_kernel<<<(9 * 32 * cin + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        d_w, cin, static_cast<__nv_bfloat16*>(d_wf), static_cast<__nv_bfloat16*>(d_wt));
    return cuda_status(cudaGetLastError());
}

int ironav_prop_propose(const float* d_out, int n, float min_conf, int16_t* d_cands, uint8_t* d_cls, void* stream) {
    if (!d_out || !d_cands || !d_cls || n < 1 || n > (1 << 22) || !(min_conf >= 0.f && min_conf <= 1.f)) return IRONAV_INVALID_ARGUMENT;
    prop::propose_kernel<<<(n + 127) / 128, 128, 0, static_cast<cudaStream_t>(stream)>>>(d_out, n, min_conf, d_cands, d_cls);
    return cuda_status(cudaGetLastError());
}

}  // extern "C"
