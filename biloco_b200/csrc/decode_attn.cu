// One decode step of attention for M <= 32 sequences, the step between the stacked q/k/v launch and the output
// projection: optional per-head RMS norm of q and k, rotary embedding at the current position, the new key and value
// written into the cache, and attention of every query head over the cache up to that position. One launch replaces the
// few dozen element-wise kernels a framework issues for these steps (each a launch of a few microseconds on a vector of
// a few thousand elements). Not part of the fused linear; a piece of the decode step around it.
//
// Arithmetic (mirrors the composition in plain tensor operations, so that the two can be compared closely):
//     norm:   x * rsqrt(mean(x^2) + eps) in fp32, rounded to bf16, times the bf16 weight, rounded to bf16
//     rotary: halves (x1, x2) of the head: (x1*cos - x2*sin, x2*cos + x1*sin), separate fp32 multiplies and adds, rounded to bf16
//     scores: fp32 dot products of bf16 q and k, times 1/sqrt(D); softmax and the weighted sum of v in fp32; output bf16
// Work split: a CTA takes HPC query heads (up to four) that share one KV head of one sequence, so that the cache is read once
// for them, and a cluster of up to eight CTAs shares the positions; their (maximum, sum, weighted values) meet in the first
// CTA's shared memory. The current position's key and value are formed in the launch (the unit's first CTA stores them), so no
// CTA reads cache entries written in it. Within a warp eight lanes hold a position (sixteen elements each at D = 128), four
// positions at a time, two such sets in flight and two more requested: a dot product ends with three shuffles for all
// four positions, and the accumulators are rescaled only when a maximum rises.
// Bound: HBM at long contexts (keys and values once), latency at short ones. Per launch (32 / 8 heads of 128, one CTA per query
// head and sequence and one position per warp step before): 8 sequences of 3001 positions: step of four layers 1994 -> 1107 us, one of
// 384: 562 -> 469.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "../../include/biloco_b200.h"
#include "ptx.cuh"

extern "C" int biloco_internal_use_pdl();

namespace {

constexpr int AT_THREADS = 256;
constexpr int AT_WARPS = AT_THREADS / 32;
constexpr int AT_MAX_CLUSTER = 8;

struct AttnParams {
    const __nv_bfloat16* qkv;       // [M, (H + 2*KVH) * D]: q heads, then k heads, then v heads
    const __nv_bfloat16* q_norm;    // [D] or null
    const __nv_bfloat16* k_norm;    // [D] or null
    const float* cos;               // [max_len, D/2]
    const float* sin;
    const long long* pos;           // device scalar: the position being written
    __nv_bfloat16* k_cache;         // [M, KVH, max_len, D]
    __nv_bfloat16* v_cache;
    __nv_bfloat16* out;             // [M, H * D]
    int M, H, KVH, max_len;
    int wide;                       // caches aligned to 16 bytes (else to 8)
    int split;                      // CTAs (of one cluster) that share a unit's positions
    float eps, scale;               // (scale: 1/sqrt(D) in units of log2)
};

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// one head vector (D elements in shared memory, one warp): optional norm, then rotary at (cs, sn)
template <int D>
__device__ __forceinline__ void norm_rope(float* x, const __nv_bfloat16* w, float eps, const float* cs, const float* sn, int lane) {
    if (w) {
        float ss = 0.f;
#pragma unroll
        for (int i = lane; i < D; i += 32) ss = fmaf(x[i], x[i], ss);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = rsqrtf(ss / (float)D + eps);
#pragma unroll
        for (int i = lane; i < D; i += 32) x[i] = bf16r(__fmul_rn(bf16r(__fmul_rn(x[i], inv)), __bfloat162float(w[i])));
        __syncwarp();
    }
#pragma unroll
    for (int i = lane; i < D / 2; i += 32) {
        const float x1 = x[i], x2 = x[i + D / 2], c = cs[i], s = sn[i];
        x[i] = bf16r(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
        x[i + D / 2] = bf16r(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s)));
    }
    __syncwarp();
}

__device__ __forceinline__ void unpack16(const uint4& a, const uint4& b, float (&x)[16]) {
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) { x[2 * i] = __uint_as_float(w[i] << 16); x[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
}

// 16 bytes at an address that is 16-byte aligned (wide) or only 8-byte aligned
__device__ __forceinline__ uint4 load16(const void* src, int wide) {
    if (wide) return *reinterpret_cast<const uint4*>(src);
    const uint2 a = reinterpret_cast<const uint2*>(src)[0], b = reinterpret_cast<const uint2*>(src)[1];
    return make_uint4(a.x, a.y, b.x, b.y);
}

// (m, l, acc) of one set of positions joined with another's
template <int HPC>
__device__ __forceinline__ void join_lanes(float (&mx)[HPC], float (&l)[HPC], float (&acc)[HPC][16], int mask) {
#pragma unroll
    for (int h = 0; h < HPC; ++h) {
        const float om = __shfl_xor_sync(0xffffffffu, mx[h], mask), ol = __shfl_xor_sync(0xffffffffu, l[h], mask);
        const float nm = fmaxf(mx[h], om), fa = exp2f(mx[h] - nm), fb = exp2f(om - nm);
        l[h] = l[h] * fa + ol * fb;
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[h][e] = acc[h][e] * fa + __shfl_xor_sync(0xffffffffu, acc[h][e], mask) * fb;
        mx[h] = nm;
    }
}

template <int D, int HPC>
__global__ void __launch_bounds__(AT_THREADS, 1) decode_attention_kernel(const __grid_constant__ AttnParams p) {
    constexpr int LPP = D / 16;                      // lanes per position: elements 8 sl .. 8 sl + 7 of both halves of the row
    constexpr int SLOTS = 32 / LPP;                  // positions per warp step
    constexpr int UNR = 2;
    __shared__ float q_s[HPC][D], k_s[D], v_s[D];
    __shared__ float w_m[AT_WARPS][HPC], w_l[AT_WARPS][HPC], w_acc[AT_WARPS][HPC][D];
    __shared__ float c_m[AT_MAX_CLUSTER][HPC], c_l[AT_MAX_CLUSTER][HPC], c_acc[AT_MAX_CLUSTER][HPC][D];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.split, rank = S > 1 ? (int)(blockIdx.x % (unsigned)S) : 0;
    const int unit = blockIdx.x / (unsigned)S;       // (sequence, KV head, set of HPC of its query heads)
    const int sets = p.H / p.KVH / HPC;
    const int m = unit / (p.KVH * sets), rest = unit - m * p.KVH * sets, g = rest / sets, set = rest - g * sets;
    const int h0 = (g * sets + set) * HPC;
    biloco::griddep_launch_dependents();             // the next kernel of the stream may start its preamble
    biloco::griddep_wait();                          // q/k/v come from the previous kernel
    const long long pos_ll = p.pos[0];
    if (pos_ll < 0 || pos_ll >= p.max_len) return;   // (nothing sensible to do; uniform over the grid)
    const int pos = (int)pos_ll;
    // (the peers' shared memory may be written once every CTA of the cluster has passed this point)
    if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    // cached positions of this CTA: [a, b), dealt to the warps in steps of SLOTS * UNR
    const int per = (pos + S - 1) / S;
    const int a = rank * per < pos ? rank * per : pos, b = a + per < pos ? a + per : pos;
    const int slot = lane / LPP, sl = lane - slot * LPP;
    const size_t cache_row = ((size_t)m * p.KVH + g) * p.max_len;
    const __nv_bfloat16* kb = p.k_cache + cache_row * D + sl * 8;
    const __nv_bfloat16* vb = p.v_cache + cache_row * D + sl * 8;
    uint4 kq[UNR][2], vq[UNR][2];
    auto request = [&](int p0) {                     // keys and values of positions p0 + slot, p0 + SLOTS + slot
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            const int pp = p0 + u * SLOTS + slot;
            if (pp < b) {
                kq[u][0] = load16(kb + (size_t)pp * D, p.wide);
                kq[u][1] = load16(kb + (size_t)pp * D + D / 2, p.wide);
                vq[u][0] = load16(vb + (size_t)pp * D, p.wide);
                vq[u][1] = load16(vb + (size_t)pp * D + D / 2, p.wide);
            } else {
                kq[u][0] = kq[u][1] = vq[u][0] = vq[u][1] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    int p0 = a + warp * SLOTS * UNR;
    request(p0);                                     // (in flight while the query is formed)
    const __nv_bfloat16* row = p.qkv + (size_t)m * (p.H + 2 * p.KVH) * D;
    for (int i = tid; i < HPC * D; i += AT_THREADS) q_s[i / D][i % D] = __bfloat162float(row[h0 * D + i]);
    if (tid < D) {
        k_s[tid] = __bfloat162float(row[(p.H + g) * D + tid]);
        v_s[tid] = __bfloat162float(row[(p.H + p.KVH + g) * D + tid]);
    }
    __syncthreads();
    const float* cs = p.cos + (size_t)pos * (D / 2);
    const float* sn = p.sin + (size_t)pos * (D / 2);
    if (warp < HPC) norm_rope<D>(q_s[warp], p.q_norm, p.eps, cs, sn, lane);
    if (warp == HPC) norm_rope<D>(k_s, p.k_norm, p.eps, cs, sn, lane);
    __syncthreads();
    if (rank == 0 && set == 0 && tid < D) {
        p.k_cache[(cache_row + pos) * D + tid] = __float2bfloat16_rn(k_s[tid]);      // (exact: bf16 values)
        p.v_cache[(cache_row + pos) * D + tid] = __float2bfloat16_rn(v_s[tid]);
    }
    float q[HPC][16], acc[HPC][16], mx[HPC], l[HPC];
#pragma unroll
    for (int h = 0; h < HPC; ++h) {
        mx[h] = -FLT_MAX;
        l[h] = 0.f;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            q[h][e] = q_s[h][(e >> 3) * (D / 2) + sl * 8 + (e & 7)];
            acc[h][e] = 0.f;
        }
    }
    // scores (in units of log2) of UNR positions per slot, then their weights and values
    auto step = [&](float (&sc)[UNR][HPC], const float (&v)[UNR][16]) {
#pragma unroll
        for (int o = 1; o < LPP; o <<= 1)
#pragma unroll
            for (int u = 0; u < UNR; ++u)
#pragma unroll
                for (int h = 0; h < HPC; ++h) sc[u][h] += __shfl_xor_sync(0xffffffffu, sc[u][h], o);
        bool rise = false;                           // (a score is scaled and rounded once: the largest has the weight 1 whatever its size)
#pragma unroll
        for (int h = 0; h < HPC; ++h) {
#pragma unroll
            for (int u = 0; u < UNR; ++u) {
                sc[u][h] = __fmul_rn(sc[u][h], p.scale);
                rise |= sc[u][h] > mx[h];
            }
        }
        if (__any_sync(0xffffffffu, rise)) {
#pragma unroll
            for (int h = 0; h < HPC; ++h) {
                float nm = mx[h];
#pragma unroll
                for (int u = 0; u < UNR; ++u) nm = fmaxf(nm, sc[u][h]);
                const float corr = exp2f(mx[h] - nm);
                l[h] *= corr;
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[h][e] *= corr;
                mx[h] = nm;
            }
        }
#pragma unroll
        for (int u = 0; u < UNR; ++u)
#pragma unroll
            for (int h = 0; h < HPC; ++h) {
                const float w = exp2f(__fsub_rn(sc[u][h], mx[h]));
                l[h] += w;
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[h][e] = fmaf(w, v[u][e], acc[h][e]);
            }
    };
#pragma unroll 1
    for (; p0 < b; p0 += AT_WARPS * SLOTS * UNR) {
        float sc[UNR][HPC], v[UNR][16];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
            float k[16];
            unpack16(kq[u][0], kq[u][1], k);
            unpack16(vq[u][0], vq[u][1], v[u]);
            const bool live = p0 + u * SLOTS + slot < b;
#pragma unroll
            for (int h = 0; h < HPC; ++h) {
                float d = 0.f;
#pragma unroll
                for (int e = 0; e < 16; ++e) d = fmaf(q[h][e], k[e], d);
                sc[u][h] = live ? d : -INFINITY;
            }
        }
        request(p0 + AT_WARPS * SLOTS * UNR);
        step(sc, v);
    }
    if (rank == 0 && warp == 0) {                    // the position being written: slot 0, first of its two
        float sc[UNR][HPC], v[UNR][16];
#pragma unroll
        for (int u = 0; u < UNR; ++u) {
#pragma unroll
            for (int e = 0; e < 16; ++e) v[u][e] = u == 0 && slot == 0 ? v_s[(e >> 3) * (D / 2) + sl * 8 + (e & 7)] : 0.f;      // (0 * an infinity is no zero)
#pragma unroll
            for (int h = 0; h < HPC; ++h) {
                float d = 0.f;
#pragma unroll
                for (int e = 0; e < 16; ++e) d = fmaf(q[h][e], k_s[(e >> 3) * (D / 2) + sl * 8 + (e & 7)], d);
                sc[u][h] = (u == 0 && slot == 0) ? d : -INFINITY;
            }
        }
        step(sc, v);
    }
#pragma unroll
    for (int o = LPP; o < 32; o <<= 1) join_lanes<HPC>(mx, l, acc, o);
    if (slot == 0) {
#pragma unroll
        for (int h = 0; h < HPC; ++h) {
            if (sl == 0) { w_m[warp][h] = mx[h]; w_l[warp][h] = l[h]; }
#pragma unroll
            for (int e = 0; e < 16; ++e) w_acc[warp][h][(e >> 3) * (D / 2) + sl * 8 + (e & 7)] = acc[h][e];
        }
    }
    __syncthreads();
    if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int i = tid; i < HPC * D; i += AT_THREADS) {
        const int h = i / D, d = i - h * D;
        float gm = -FLT_MAX, num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w) gm = fmaxf(gm, w_m[w][h]);
#pragma unroll
        for (int w = 0; w < AT_WARPS; ++w) {
            const float f = exp2f(w_m[w][h] - gm);
            num += f * w_acc[w][h][d];
            den += f * w_l[w][h];
        }
        if (S > 1) {
            biloco::st_cluster_f32(biloco::map_to_cta(biloco::smem_u32(&c_acc[rank][h][d]), 0), num);
            if (d == 0) {
                biloco::st_cluster_f32(biloco::map_to_cta(biloco::smem_u32(&c_m[rank][h]), 0), gm);
                biloco::st_cluster_f32(biloco::map_to_cta(biloco::smem_u32(&c_l[rank][h]), 0), den);
            }
        } else {
            p.out[((size_t)m * p.H + h0) * D + i] = __float2bfloat16_rn(num / den);
        }
    }
    if (S == 1) return;
    __syncwarp();
    biloco::cluster_sync_all();
    if (rank != 0) return;
    for (int i = tid; i < HPC * D; i += AT_THREADS) {
        const int h = i / D, d = i - h * D;
        float gm = -FLT_MAX, num = 0.f, den = 0.f;
        for (int r = 0; r < S; ++r) gm = fmaxf(gm, c_m[r][h]);
        for (int r = 0; r < S; ++r) {
            const float f = exp2f(c_m[r][h] - gm);
            num += f * c_acc[r][h][d];
            den += f * c_l[r][h];
        }
        p.out[((size_t)m * p.H + h0) * D + i] = __float2bfloat16_rn(num / den);
    }
}

template <int D>
static cudaError_t launch_attention(const cudaLaunchConfig_t* cfg, int hpc, const AttnParams& p) {
    switch (hpc) {
        case 4: return cudaLaunchKernelEx(cfg, decode_attention_kernel<D, 4>, p);
        case 2: return cudaLaunchKernelEx(cfg, decode_attention_kernel<D, 2>, p);
        default: return cudaLaunchKernelEx(cfg, decode_attention_kernel<D, 1>, p);
    }
}

}  // namespace

extern "C" int biloco_b200_decode_attention(const void* qkv_bf16, const void* q_norm_bf16, const void* k_norm_bf16, float eps,
                                            const float* cos_table, const float* sin_table, const long long* pos_dev,
                                            void* k_cache_bf16, void* v_cache_bf16, void* out_bf16, int M, int H, int KVH, int D,
                                            int max_len, biloco_stream_t stream) {
    if (!qkv_bf16 || !cos_table || !sin_table || !pos_dev || !k_cache_bf16 || !v_cache_bf16 || !out_bf16) return BILOCO_ERR_NULL;
    if (M < 1 || M > 65535 || H < 1 || KVH < 1 || (H % KVH) != 0 || (D != 64 && D != 128) || max_len < 1) return BILOCO_ERR_SHAPE;
    if (((uintptr_t)qkv_bf16 & 7) || ((uintptr_t)k_cache_bf16 & 7) || ((uintptr_t)v_cache_bf16 & 7)) return BILOCO_ERR_ALIGN;
    AttnParams p;
    p.qkv = (const __nv_bfloat16*)qkv_bf16;
    p.q_norm = (const __nv_bfloat16*)q_norm_bf16;
    p.k_norm = (const __nv_bfloat16*)k_norm_bf16;
    p.cos = cos_table; p.sin = sin_table; p.pos = pos_dev;
    p.k_cache = (__nv_bfloat16*)k_cache_bf16; p.v_cache = (__nv_bfloat16*)v_cache_bf16; p.out = (__nv_bfloat16*)out_bf16;
    p.M = M; p.H = H; p.KVH = KVH; p.max_len = max_len;
    p.eps = eps;
    p.scale = 1.4426950408889634f / sqrtf((float)D);
    // query heads per CTA: as many of a KV head's group as divide it, at most four; positions: over as many CTAs of a cluster as
    // fill the device once, with at least a warp step (16 or 32 positions per warp) of the longest context for each
    const int group = H / KVH, hpc = group % 4 == 0 ? 4 : (group % 2 == 0 ? 2 : 1);
    p.wide = (((uintptr_t)k_cache_bf16 | (uintptr_t)v_cache_bf16) & 15) == 0;
    const long long units = (long long)M * (H / hpc);
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return BILOCO_ERR_CUDA;
    p.split = 1;
    while (p.split < AT_MAX_CLUSTER && units * p.split * 2 <= sms && max_len > p.split * 64) p.split *= 2;
    if (units * p.split > 0x7fffffffll) return BILOCO_ERR_SHAPE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * p.split));
    cfg.blockDim = dim3(AT_THREADS);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (biloco_internal_use_pdl()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (p.split > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.split;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t e = D == 128 ? launch_attention<128>(&cfg, hpc, p) : launch_attention<64>(&cfg, hpc, p);
    return e == cudaSuccess ? BILOCO_OK : BILOCO_ERR_CUDA;
}
