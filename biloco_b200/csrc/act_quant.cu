// NVFP4 activation quantiser: bf16 [M,K] -> E2M1 codes (two per byte, element 2j in bits 0-3), E4M3 block
// scales per 16 elements in the 128x4 atom layout, one fp32 decode scale per call.
//
// Arithmetic contract (every step is a single IEEE fp32 operation, so a CPU restatement reproduces it bit
// for bit):
//     xs   = bf16_rn(x / smooth)            (only when a smoothing vector is given)
//     gs   = amax / (6 * target)            target = 448 (static_6) or 256 (static_4, mse); gs = 1 if amax == 0
//     t    = bmax / gs                      per 16-element block
//     sfD  = e4m3_rn_sat(t / D)             D = 6 or 4
//     d    = f32(sfD) * gs
//     code = e2m1_rn(xs / d)                round-to-nearest-even on {0,.5,1,1.5,2,3,4,6}, saturating; 0 if d == 0, sign only if xs is NaN
//     mse rule: err_D = sum_{j=0..15} (xs_j - value(code_j) * d)^2 in index order (separate mul and add);
//               the block takes D = 4 iff err_4 < err_6.
// One launch of ONE cluster (up to sixteen CTAs of 256 or 512 threads): a decode batch is at most a few hundred KB and the
// launch a chain of latencies, so every element is read once and stays on the SM from there on. Groups of 256 threads take a
// row, a segment of a row (several groups per row at few rows) or several rows; a thread holds 8 elements at a time, two
// neighbouring lanes a block. The activation is formed (RMS norm, SwiGLU, smoothing) in shared memory, the maxima of the CTAs meet
// in distributed shared memory, the blocks are quantised from shared memory. In the RMS form every group of a row adds up the
// whole row's squares, in one fixed order (which the fused linear's own activation prologue, slab_kernel.cuh, follows).
// Against the form with one lane per element, four passes over global memory and the maximum of everything in every cluster, its
// cost in the captured decode step of four layers (8 sequences): 1107 -> 869 us, one sequence 469 -> 425; in a layer of 8192 x 8192 with
// smoothing at 27 rows 87 -> 57 us.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/biloco_b200.h"
#include "ptx.cuh"
#include "quant_math.cuh"

extern "C" int biloco_internal_use_pdl();

namespace {

constexpr int GROUP = 256;               // threads of a group
constexpr int Q_MAX_CLUSTER = 16;        // (more than eight CTAs: non-portable, asked of the driver first)
constexpr int MAX_GPC = 2;               // groups per CTA

using biloco::qm::e4m3_to_float;
using biloco::qm::float_to_e4m3_sat;

struct QParams {
    const __nv_bfloat16* X;              // [M, K] ([M, 2K] = [gate | up] for SwiGLU)
    const __nv_bfloat16* norm_w;
    const __nv_bfloat16* smooth;
    __nv_bfloat16* Xs;                   // the activation that is quantised, or null
    uint8_t *codes, *sf, *rec;
    float *a_gscale, *alpha;
    const float* w_gscale;
    int M, A_rows, K, rule, given_scale, n_alpha;
    int csize, gpc, seg, per, rpg;       // CTAs, groups per CTA, groups per row, vectors per segment, rows per group
    int staged;                          // the group's share fits shared memory; otherwise it is read from global memory again
    float eps, target;
};

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ void unpack8(const uint4& a, float (&v)[8]) {
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { v[2 * e] = __uint_as_float(w[e] << 16); v[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u); }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {      // (exact: bf16 values)
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) w[e] = (__float_as_uint(v[2 * e]) >> 16) | (__float_as_uint(v[2 * e + 1]) & 0xFFFF0000u);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Half a block per lane (lanes 2i and 2i + 1 hold one block): this lane's eight codes and, in both lanes, the block's scale.
__device__ __forceinline__ uint32_t quant_half(const float (&x)[8], int lane, float gs, int rule, uint8_t& sf) {
    uint32_t keep = 0xffffffffu, sign = 0u;
    float bmax = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) bmax = biloco::qm::max_nan(bmax, fabsf(x[j]));
    if (bmax != bmax) {
        const biloco::qm::NanHalf n = biloco::qm::nan_half(x);
        bmax = n.bmax; keep = n.keep; sign = n.sign;
    }
    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 1));
    const float t = __fdiv_rn(bmax, gs);
    uint32_t c[2] = {0u, 0u};
    uint8_t s[2] = {0, 0};
    float e[2] = {0.f, 0.f};
#pragma unroll
    for (int cand = 0; cand < 2; ++cand) {
        if (cand == 0 && rule == BILOCO_RULE_STATIC_4) continue;
        if (cand == 1 && rule == BILOCO_RULE_STATIC_6) continue;
        s[cand] = float_to_e4m3_sat(__fdiv_rn(t, cand == 0 ? 6.0f : 4.0f));
        const float d = __fmul_rn(e4m3_to_float(s[cand]), gs);
        c[cand] = biloco::qm::codes8(x, d, keep, sign);
        if (rule == BILOCO_RULE_MSE) {
            float v[8], sq[8];
            biloco::qm::e2m1_unpack8(c[cand], v);
            float err = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float diff = __fsub_rn(x[j], __fmul_rn(v[j], d));
                sq[j] = __fmul_rn(diff, diff);
                err = __fadd_rn(err, sq[j]);
            }
            const float first = __shfl_xor_sync(0xffffffffu, err, 1);      // index order: the odd lane goes on from the even lane's sum
            float rest = first;
#pragma unroll
            for (int j = 0; j < 8; ++j) rest = __fadd_rn(rest, sq[j]);
            const float other = __shfl_xor_sync(0xffffffffu, rest, 1);
            e[cand] = (lane & 1) ? rest : other;
        }
    }
    const bool four = rule == BILOCO_RULE_STATIC_4 || (rule == BILOCO_RULE_MSE && e[1] < e[0]);
    sf = four ? s[1] : s[0];
    return four ? c[1] : c[0];
}

// PRO: 0 the activation as it is (or smoothed), 1 RMS norm in front, 2 silu(gate) * up in front. PAD: the zero padding is written too (a
// form of its own: its code in the launches that skip it cost them 0.5 us: decode step of one sequence 434 -> 424).
template <int PRO, bool PAD>
__global__ void __launch_bounds__(GROUP * MAX_GPC) act_quant_kernel(const __grid_constant__ QParams p) {
    extern __shared__ uint4 stage_raw[];                     // [group][row][vector of the segment]
    __shared__ float red[GROUP * MAX_GPC / 32];
    __shared__ float cl_max[Q_MAX_CLUSTER];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int crank = p.csize > 1 ? (int)(blockIdx.x % (unsigned)p.csize) : 0;
    const int gl = warp >> 3, gw = warp & 7;                 // group within the CTA, warp within the group
    const int grp = crank * p.gpc + gl;
    const int nv = p.K >> 3;
    // rows and vectors of this group
    const int row0 = p.seg > 1 ? grp / p.seg : grp * p.rpg;
    const int sgm = p.seg > 1 ? grp - row0 * p.seg : 0;
    const int nrows = row0 < p.M ? (p.M - row0 < p.rpg ? p.M - row0 : p.rpg) : 0;
    const int lo = sgm * p.per, hi = lo + p.per < nv ? lo + p.per : nv;
    uint4* stage = stage_raw + (size_t)gl * p.rpg * p.per;
    const uint4* smooth = reinterpret_cast<const uint4*>(p.smooth);
    biloco::griddep_launch_dependents();                     // the consumer may start its own preamble (weight prefetch)
    if (p.csize > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // (every CTA runs before a peer writes to it)
    biloco::griddep_wait();                                  // nothing of the activation is read before the previous kernel has completed
    const int kg = p.K >> 6, mma_n = p.M <= 8 ? 8 : (p.M <= 16 ? 16 : 32), rec_bytes = mma_n * 128 + 2048;
    // ---- zero padding, 16 bytes at a time: block scales of rows M .. 127 (a 16-byte chunk of an atom holds rows r, r + 32, r + 64,
    //      r + 96), codes of rows M .. A_rows, the record's rest ----
    if constexpr (PAD) {
        const int nth = p.csize * blockDim.x, at = crank * blockDim.x + tid;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        auto pad_chunk = [&](uint8_t* atom, int r) {         // chunk r of an atom
            if (r >= p.M && ((uintptr_t)atom & 15) == 0) *reinterpret_cast<uint4*>(atom + r * 16) = zero;
            else
                for (int q = 0; q < 4; ++q)
                    if (r + 32 * q >= p.M) *reinterpret_cast<uint32_t*>(atom + r * 16 + q * 4) = 0u;
        };
        for (int i = at; i < kg * 32; i += nth) pad_chunk(p.sf + (size_t)(i >> 5) * 512, i & 31);
        const long long ncode = (long long)(p.A_rows - p.M) * (p.K >> 4);
        uint2* cz = reinterpret_cast<uint2*>(p.codes + (size_t)p.M * (p.K >> 1));
        for (long long i = at; i < ncode; i += nth) cz[i] = make_uint2(0u, 0u);
        if (p.rec) {
            for (int i = at; i < kg * 32; i += nth) pad_chunk(p.rec + (size_t)(i >> 7) * rec_bytes + mma_n * 128 + ((i >> 5) & 3) * 512, i & 31);
            const int tile = (mma_n - p.M) * 8;              // 16-byte chunks of a tile's rows M .. mma_n - 1
            for (int i = at; i < (p.K >> 8) * tile; i += nth) {
                const int kt = i / tile, c = i - kt * tile;
                *reinterpret_cast<uint4*>(p.rec + (size_t)kt * rec_bytes + p.M * 128 + c * 16) = zero;
            }
        }
    }
    float amax = 0.f;
#pragma unroll 1
    for (int r = 0; r < p.rpg; ++r) {
        const int row = row0 + r;
        const bool live = r < nrows;
        float inv = 0.f;
        if constexpr (PRO == 1) {
            float ss = 0.f;
            const uint4* xr = reinterpret_cast<const uint4*>(p.X + (size_t)row * p.K);
            if (live) {
#pragma unroll 4
                for (int i = tid & (GROUP - 1); i < nv; i += GROUP) {
                    const uint4 a = xr[i];
                    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
                    if (p.staged && i >= lo && i < hi) stage[r * p.per + i - lo] = a;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float l = __uint_as_float(w[e] << 16), h = __uint_as_float(w[e] & 0xFFFF0000u);
                        ss = fmaf(l, l, ss);
                        ss = fmaf(h, h, ss);
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) red[warp] = ss;
            __syncthreads();
            float tot = 0.f;
#pragma unroll
            for (int i = 0; i < GROUP / 32; ++i) tot += red[gl * (GROUP / 32) + i];
            inv = rsqrtf(tot / (float)p.K + p.eps);
        }
        // the activation of the segment -> shared memory (a thread reads back only what it wrote, except under the norm above)
        if (live) {
            uint4* xo = p.Xs ? reinterpret_cast<uint4*>(p.Xs + (size_t)row * p.K) : nullptr;
            const uint4* xr = reinterpret_cast<const uint4*>(p.X + (size_t)row * p.K * (PRO == 2 ? 2 : 1));
#pragma unroll 2
            for (int i = lo + (tid & (GROUP - 1)); i < hi; i += GROUP) {
                float v[8];
                uint4 raw;
                if (PRO == 1 && p.staged) raw = stage[r * p.per + i - lo];
                else raw = xr[i];
                unpack8(raw, v);
                if constexpr (PRO == 1) {
                    float g[8];
                    unpack8(reinterpret_cast<const uint4*>(p.norm_w)[i], g);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = bf16r(bf16r(v[e] * inv) * g[e]);
                }
                if constexpr (PRO == 2) {                    // silu(g) = g / (1 + exp(-g)) in fp32, the roundings of the separate kernels it replaces
                    float u[8];
                    unpack8(xr[nv + i], u);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = bf16r(__fmul_rn(bf16r(__fdiv_rn(v[e], __fadd_rn(1.0f, expf(-v[e])))), u[e]));
                }
                if (smooth) {
                    float s[8];
                    unpack8(smooth[i], s);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = bf16r(__fdiv_rn(v[e], s[e]));
                }
                if (PRO != 0 || smooth) raw = pack8(v);
                if (p.staged) stage[r * p.per + i - lo] = raw;
                if (xo) xo[i] = raw;
#pragma unroll
                for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
            }
        }
        if constexpr (PRO == 1) __syncthreads();             // (red is used again)
    }
    __syncwarp();
    // ---- tensor scale ----
    float gs;
    if (!p.given_scale) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (lane == 0) red[warp] = amax;
        __syncthreads();
        if (warp == 0) {
            float v = lane < p.gpc * (GROUP / 32) ? red[lane] : 0.f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (p.csize > 1) {                               // lane r hands this CTA's maximum to CTA r of the cluster
                asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
                if (lane < p.csize) biloco::st_cluster_f32(biloco::map_to_cta(biloco::smem_u32(&cl_max[crank]), (uint32_t)lane), v);
                __syncwarp();
            } else if (lane == 0) {
                cl_max[0] = v;
            }
        } else if (p.csize > 1) {
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        if (p.csize > 1) biloco::cluster_sync_all();         // (release/acquire: the peers' values are in cl_max)
        else __syncthreads();
        float v = 0.f;
        for (int r = 0; r < p.csize; ++r) v = fmaxf(v, cl_max[r]);
        gs = v > 0.f ? __fdiv_rn(v, 6.0f * p.target) : 1.0f;
    } else {
        if (p.csize > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        gs = p.a_gscale[0];
    }
    if (crank == 0 && tid == 0 && blockIdx.x == 0) {
        if (!p.given_scale) p.a_gscale[0] = gs;
        if (p.alpha && p.w_gscale)
            for (int i = 0; i < p.n_alpha; ++i) p.alpha[i] = __fmul_rn(p.w_gscale[i], gs);      // one per consumer of this activation
    }
    // ---- codes and scales (all lanes of a warp stay together: the block's two lanes exchange) ----
#pragma unroll 1
    for (int r = 0; r < nrows; ++r) {
        const int row = row0 + r;
        const int rsf = (row & 31) * 16 + ((row >> 5) & 3) * 4;
#pragma unroll 1
        for (int i0 = lo + gw * 32; i0 < hi; i0 += GROUP) {
            const int i = i0 + lane;
            const bool on = i < hi;                          // (hi - lo is even: a block's two lanes agree)
            float x[8];
            uint4 raw = make_uint4(0u, 0u, 0u, 0u);
            if (on) raw = p.staged ? stage[r * p.per + i - lo] : reinterpret_cast<const uint4*>((p.Xs ? p.Xs : p.X) + (size_t)row * p.K)[i];
            unpack8(raw, x);
            if (PRO == 0 && smooth && !p.staged && !p.Xs && on) {      // (the smoothed activation was kept nowhere)
                float s[8];
                unpack8(smooth[i], s);
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] = bf16r(__fdiv_rn(x[e], s[e]));
            }
            uint8_t sfb;
            const uint32_t w = quant_half(x, lane, gs, p.rule, sfb);
            if (!on) continue;
            const int kb = i >> 1;
            *reinterpret_cast<uint32_t*>(p.codes + (size_t)row * (p.K >> 1) + i * 4) = w;
            if (!(lane & 1)) p.sf[((size_t)(row >> 7) * kg + (kb >> 2)) * 512 + rsf + (kb & 3)] = sfb;
            if (p.rec) {      // the same where the fused kernel's stage wants it (128-byte swizzle: chunk c of row r at c ^ (r & 7))
                uint8_t* rk = p.rec + (size_t)(kb >> 4) * rec_bytes;
                const int b = (i & 31) * 4;                  // byte of the word within the tile row
                *reinterpret_cast<uint32_t*>(rk + row * 128 + (((b >> 4) ^ (row & 7)) << 4) + (b & 15)) = w;
                if (!(lane & 1)) rk[mma_n * 128 + ((kb >> 2) & 3) * 512 + rsf + (kb & 3)] = sfb;
            }
        }
    }
}

template <int PRO, bool PAD>
static cudaError_t launch_form(cudaLaunchConfig_t* cfg, const QParams& p, int dev) {
    static bool ready[64] = {false};
    if (dev >= 0 && dev < 64 && !ready[dev]) {
        cudaFuncSetAttribute(act_quant_kernel<PRO, PAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        cudaFuncSetAttribute(act_quant_kernel<PRO, PAD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaGetLastError();
        ready[dev] = true;
    }
    return cudaLaunchKernelEx(cfg, act_quant_kernel<PRO, PAD>, p);
}
template <int PRO>
static cudaError_t launch_pro(cudaLaunchConfig_t* cfg, const QParams& p, int dev, bool pad) {      // (pad: not with BILOCO_RULE_PADDED)
    return pad ? launch_form<PRO, true>(cfg, p, dev) : launch_form<PRO, false>(cfg, p, dev);
}

// Whether the device takes a cluster of sixteen such CTAs (asked once per device; the answer depends on how its SMs are grouped).
static bool sixteen_fit(int dev) {
    static int known[64] = {0};
    if (dev < 0 || dev >= 64) return false;
    if (known[dev] == 0) {
        int n = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 16;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(16);
        cfg.blockDim = dim3(GROUP * MAX_GPC);
        cfg.dynamicSmemBytes = 96 * 1024;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        bool ok = cudaFuncSetAttribute(act_quant_kernel<0, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) == cudaSuccess &&
                  cudaFuncSetAttribute(act_quant_kernel<0, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&n, act_quant_kernel<0, false>, &cfg) == cudaSuccess && n >= 1;
        cudaGetLastError();
        known[dev] = ok ? 1 : -1;
    }
    return known[dev] > 0;
}

}  // namespace

static int launch_act_quant(const void* X_bf16, const void* norm_w, float eps, const void* smooth_bf16, void* Xs_bf16, void* A_codes,
                            void* A_sf, void* A_rec, float* a_gscale, float* alpha_out, const float* w_gscale, int n_alpha, int M,
                            int A_rows, int K, int rule, biloco_stream_t stream, int swiglu = 0) {
    if (swiglu && (!Xs_bf16 || norm_w)) return BILOCO_ERR_NULL;
    if (A_rec && (M > 32 || (K % 256) != 0 || ((uintptr_t)A_rec & 15))) return BILOCO_ERR_SHAPE;
    if (!X_bf16 || !A_codes || !A_sf || !a_gscale) return BILOCO_ERR_NULL;
    if (norm_w && !Xs_bf16) return BILOCO_ERR_NULL;
    if (n_alpha < 1 || n_alpha > 16) return BILOCO_ERR_SHAPE;
    if ((uintptr_t)norm_w & 15) return BILOCO_ERR_ALIGN;
    if (M < 1 || A_rows < M || A_rows > 128 || K < 64 || (K % 64) != 0) return BILOCO_ERR_SHAPE;
    const bool given_scale = (rule & BILOCO_RULE_GIVEN_SCALE) != 0, padded = (rule & BILOCO_RULE_PADDED) != 0;
    rule &= ~(BILOCO_RULE_GIVEN_SCALE | BILOCO_RULE_PADDED);
    if (rule != BILOCO_RULE_STATIC_6 && rule != BILOCO_RULE_STATIC_4 && rule != BILOCO_RULE_MSE) return BILOCO_ERR_MODE;
    if (((uintptr_t)A_codes & 7) || ((uintptr_t)X_bf16 & 15) || ((uintptr_t)smooth_bf16 & 15) || ((uintptr_t)Xs_bf16 & 15))
        return BILOCO_ERR_ALIGN;
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return BILOCO_ERR_CUDA;
    QParams p;
    p.X = (const __nv_bfloat16*)X_bf16; p.norm_w = (const __nv_bfloat16*)norm_w; p.smooth = (const __nv_bfloat16*)smooth_bf16;
    p.Xs = (__nv_bfloat16*)Xs_bf16;
    p.codes = (uint8_t*)A_codes; p.sf = (uint8_t*)A_sf; p.rec = (uint8_t*)A_rec;
    p.a_gscale = a_gscale; p.alpha = alpha_out; p.w_gscale = w_gscale;
    p.M = M; p.A_rows = A_rows; p.K = K; p.rule = rule; p.given_scale = given_scale ? 1 : 0; p.n_alpha = n_alpha;
    p.eps = eps; p.target = rule == BILOCO_RULE_STATIC_6 ? 448.0f : 256.0f;
    // groups: about one vector of 8 elements per thread, up to two groups in each of sixteen CTAs
    const int nv = K >> 3;
    const long long nvec = (long long)M * nv;
    int ng = 1, cmax = nvec > 4096 && sixteen_fit(dev) ? 16 : 8;
    while (ng < cmax * MAX_GPC && (ng * GROUP < nvec || ng < M)) ng *= 2;
    p.csize = ng < cmax ? ng : cmax;
    p.gpc = ng / p.csize;
    p.seg = ng >= M ? ng / M : 1;
    p.rpg = ng >= M ? 1 : (M + ng - 1) / ng;
    p.per = ((nv + p.seg - 1) / p.seg + 1) & ~1;
    size_t smem = (size_t)p.gpc * p.rpg * p.per * 16;
    p.staged = smem <= 96 * 1024 ? 1 : 0;
    if (!p.staged) smem = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.csize);
    cfg.blockDim = dim3((unsigned)(GROUP * p.gpc));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (biloco_internal_use_pdl()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (p.csize > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)p.csize;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    const cudaError_t e = norm_w ? launch_pro<1>(&cfg, p, dev, !padded) : (swiglu ? launch_pro<2>(&cfg, p, dev, !padded) : launch_pro<0>(&cfg, p, dev, !padded));
    return e == cudaSuccess ? BILOCO_OK : BILOCO_ERR_CUDA;
}

extern "C" int biloco_b200_act_quant(const void* X_bf16, const void* smooth_bf16, void* Xs_bf16, void* A_codes, void* A_sf,
                                     float* a_gscale, float* alpha_out, const float* w_gscale, int M, int A_rows, int K,
                                     int rule, biloco_stream_t stream) {
    return launch_act_quant(X_bf16, nullptr, 0.f, smooth_bf16, Xs_bf16, A_codes, A_sf, nullptr, a_gscale, alpha_out, w_gscale, 1, M, A_rows,
                            K, rule, stream);
}

extern "C" int biloco_b200_norm_act_quant(const void* X_bf16, const void* norm_weight_bf16, float eps, const void* smooth_bf16,
                                          void* Xn_bf16, void* A_codes, void* A_sf, void* A_rec, float* a_gscale, float* alpha_out,
                                          const float* w_gscale, int n_alpha, int M, int A_rows, int K, int rule,
                                          biloco_stream_t stream) {
    return launch_act_quant(X_bf16, norm_weight_bf16, eps, smooth_bf16, Xn_bf16, A_codes, A_sf, A_rec, a_gscale, alpha_out, w_gscale,
                            n_alpha, M, A_rows, K, rule, stream);
}

extern "C" int biloco_b200_swiglu_act_quant(const void* GU_bf16, const void* smooth_bf16, void* Xa_bf16, void* A_codes, void* A_sf,
                                            void* A_rec, float* a_gscale, float* alpha_out, const float* w_gscale, int n_alpha, int M,
                                            int A_rows, int K, int rule, biloco_stream_t stream) {
    return launch_act_quant(GU_bf16, nullptr, 0.f, smooth_bf16, Xa_bf16, A_codes, A_sf, A_rec, a_gscale, alpha_out, w_gscale, n_alpha, M,
                            A_rows, K, rule, stream, 1);
}
