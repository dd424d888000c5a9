// NVFP4 quantisation of a weight matrix (fp32 [rows, K]): E2M1 codes, E4M3 block scales in the 128x4 atom layout, one fp32
// tensor scale. The offline path and the fake quantisation of evaluations; the arithmetic is that of quant_math.cuh, one IEEE
// fp32 operation at a time, so the bytes equal the torch restatement's (fp4.quantize_nvfp4 on the CPU) and the oracle's.
//
// Two launches: the maximum (one partial per CTA), then the blocks, one thread each -- the second read of a matrix of up to
// about 100 MB comes from L2. Bound by instruction issue (about 350 instructions per 16-element block with the "mse" rule) a
// little before HBM: 9728 x 2560 52 us (4170 us as some hundred torch operations), floor 17 us: 17 for the maximum, 38 for the blocks.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/biloco_b200.h"
#include "ptx.cuh"
#include "quant_math.cuh"

extern "C" int biloco_internal_use_pdl();
extern "C" void biloco_internal_mark_relayout(cudaStream_t stream);      // (fused_linear.cu: the next fused launch on this stream starts plain)

namespace {

constexpr int WQ_THREADS = 256;
constexpr int WQ_PMAX = 592;             // partial maxima (CTAs of the first launch)

using biloco::qm::max_nan;               // (a NaN reaches the tensor's maximum, which then gives a tensor scale of 1)

__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

__global__ void __launch_bounds__(WQ_THREADS) weight_amax_kernel(const float4* __restrict__ X, float* __restrict__ pmax, long long nvec) {
    __shared__ float red[WQ_THREADS / 32];
    biloco::griddep_launch_dependents();
    biloco::griddep_wait();
    float m = 0.f;
    const long long stride = (long long)gridDim.x * WQ_THREADS;
#pragma unroll 8
    for (long long i = (long long)blockIdx.x * WQ_THREADS + threadIdx.x; i < nvec; i += stride) {
        const float4 a = X[i];
        m = max_nan(m, max_nan(max_nan(fabsf(a.x), fabsf(a.y)), max_nan(fabsf(a.z), fabsf(a.w))));
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < WQ_THREADS / 32; ++i) m = max_nan(m, red[i]);
        pmax[blockIdx.x] = m;
    }
}

// npmax = 0: the tensor scale is given in gscale.
__global__ void __launch_bounds__(WQ_THREADS) weight_quant_kernel(const float* __restrict__ X, const float* __restrict__ pmax, int npmax, float* __restrict__ gscale,
                                                                  uint8_t* __restrict__ codes, uint8_t* __restrict__ sf, int rows, int K, int rule, float target) {
    __shared__ float red[WQ_THREADS / 32];
    biloco::griddep_launch_dependents();     // (a fused launch, which reads the codes ahead of its wait, goes out plain after this: mark_relayout)
    biloco::griddep_wait();
    float gs;
    if (npmax > 0) {
        float m = 0.f;
        for (int i = threadIdx.x; i < npmax; i += WQ_THREADS) m = max_nan(m, pmax[i]);
        m = warp_max(m);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        m = red[0];
#pragma unroll
        for (int i = 1; i < WQ_THREADS / 32; ++i) m = max_nan(m, red[i]);
        gs = m > 0.f ? __fdiv_rn(m, 6.0f * target) : 1.0f;
        if (blockIdx.x == 0 && threadIdx.x == 0) gscale[0] = gs;
    } else {
        gs = gscale[0];
    }
    // blocks of the padded scale matrix (rows to a multiple of 128, blocks per row to a multiple of 4): padding gets zero scales
    const int kb = K >> 4, kbp = (kb + 3) & ~3, rows_p = (rows + 127) & ~127;
    const unsigned total = (unsigned)rows_p * (unsigned)kbp;
    for (unsigned i = blockIdx.x * WQ_THREADS + threadIdx.x; i < total; i += gridDim.x * WQ_THREADS) {
        const unsigned row = i / (unsigned)kbp, b = i - row * (unsigned)kbp;
        uint8_t s = 0;
        if (row < (unsigned)rows && b < (unsigned)kb) {
            const float4* src = reinterpret_cast<const float4*>(X + (size_t)row * K + b * 16);
            float x[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 a = src[q];
                x[4 * q] = a.x; x[4 * q + 1] = a.y; x[4 * q + 2] = a.z; x[4 * q + 3] = a.w;
            }
            uint2 c;
            biloco::qm::quant_block16<true>(x, gs, rule, c, s);
            *reinterpret_cast<uint2*>(codes + (size_t)row * (K >> 1) + b * 8) = c;
        }
        sf[((size_t)(row >> 7) * (kbp >> 2) + (b >> 2)) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4 + (b & 3)] = s;
    }
}

}  // namespace

extern "C" size_t biloco_b200_weight_quant_ws_bytes(void) { return WQ_PMAX * sizeof(float); }

extern "C" int biloco_b200_weight_quant(const float* X, void* ws, void* codes, void* sf, float* gscale, int rows, int K, int rule, biloco_stream_t stream) {
    if (!X || !ws || !codes || !sf || !gscale) return BILOCO_ERR_NULL;
    const bool given = (rule & BILOCO_RULE_GIVEN_SCALE) != 0;
    rule &= ~BILOCO_RULE_GIVEN_SCALE;
    if (rule != BILOCO_RULE_STATIC_6 && rule != BILOCO_RULE_STATIC_4 && rule != BILOCO_RULE_MSE) return BILOCO_ERR_MODE;
    if (rows < 1 || K < 16 || (K % 16) || (long long)(rows + 127) * (K / 16 + 3) >= (1ll << 31)) return BILOCO_ERR_SHAPE;
    if (((uintptr_t)X & 15) || ((uintptr_t)codes & 7) || ((uintptr_t)ws & 3)) return BILOCO_ERR_ALIGN;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return BILOCO_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(WQ_THREADS);
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = attr;
    cfg.numAttrs = biloco_internal_use_pdl() ? 1 : 0;
    const long long nvec = (long long)rows * K / 4;
    long long g = (nvec + WQ_THREADS * 8 - 1) / (WQ_THREADS * 8);
    const int g1 = given ? 0 : (int)(g > WQ_PMAX ? WQ_PMAX : g);
    if (!given) {
        cfg.gridDim = dim3((unsigned)g1);
        if (cudaLaunchKernelEx(&cfg, weight_amax_kernel, (const float4*)X, (float*)ws, nvec) != cudaSuccess) return BILOCO_ERR_CUDA;
    }
    const long long total = (long long)((rows + 127) / 128 * 128) * ((K / 16 + 3) / 4 * 4);
    g = (total + WQ_THREADS - 1) / WQ_THREADS;
    if (g > 8ll * sms) g = 8ll * sms;
    cfg.gridDim = dim3((unsigned)g);
    if (cudaLaunchKernelEx(&cfg, weight_quant_kernel, X, (const float*)ws, g1, gscale, (uint8_t*)codes, (uint8_t*)sf, rows, K, rule,
                           rule == BILOCO_RULE_STATIC_6 ? 448.0f : 256.0f) != cudaSuccess)
        return BILOCO_ERR_CUDA;
    biloco_internal_mark_relayout((cudaStream_t)stream);
    return BILOCO_OK;
}
