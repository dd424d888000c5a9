// The linear for MORE than 32 activation rows (a prompt, an evaluation block):
//
//     Y[m,n] = bf16( alpha * sum_k A[m,k] W[n,k]  +  sum_i z[m,i] sign(U[i,n])  (+ bias[n]) ),   z = S .* (X sign(V)^T)
//
// with ONE tensor scale for all rows, as the reference quantises a call. Decode launches take 32 rows each and stream every
// weight again for every 32 rows; here the rows are the MMA's 128-row operand and the work is a contraction, in four launches
// chained by programmatic dependent launch:
//
//   amax_kernel      max |x / smooth| per CTA (and the smoothed activation, when there is smoothing)
//   quant_kernel     tensor scale, NVFP4 codes and block scales, one thread per 16-element block, written as the records the
//                    GEMM stages: per 128 rows and 256 k [codes, 128-byte swizzle applied | four scale atoms], 18 KB
//   z_gemm_kernel    z on the tensor cores (bf16 x +-1 images of the V bits, K split over a cluster and added through
//                    distributed shared memory in rank order), divided by alpha and written as bf16 high part + remainders
//   gemm_kernel      NVFP4 GEMM and, into the SAME accumulator, z times +-1 images of the U bits; epilogue alpha * acc + bias
//
// The low-rank term shares the accumulator because z is divided by alpha beforehand (fp32; high + low part keep 2^-17, a third part,
// where there is one, all of it): a second accumulator would not fit TMEM beside 256 columns and the scale factors.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/biloco_b200.h"
#include "ptx.cuh"
#include "quant_math.cuh"

extern "C" int biloco_internal_use_pdl();
extern "C" unsigned long long biloco_internal_wait_ns();
extern "C" int biloco_internal_skip_publish();
extern "C" int biloco_internal_encode_map(void* map, int bf16, const void* ptr, int rows, int cols, int box_cols, int box_rows);

namespace biloco {
namespace prompt {

constexpr int TM = 128;                          // activation rows per tile
constexpr int KT = 256;                          // k per stage of the GEMM
constexpr int A_REC = TM * 128 + 2048;           // codes of 128 rows x 256 k, then four 512-byte scale atoms
constexpr int Z_REC = 2 * TM * 128;              // 64 ranks: high parts of 128 rows x 128 bytes, then the remainders
constexpr int AUX_WARPS = 8;                     // scale factors -> TMEM, sign images, epilogue
constexpr int PRODUCER_WARP = 8;
constexpr int MMA_WARP = 9;
constexpr int WPROD_WARP = 10;                   // GEMM only: the weights' copies, beside the activations' from PRODUCER_WARP
constexpr int Z_NT = 320, G_NT = 352;            // threads of the z kernel and of the GEMM

__device__ int32_t g_status[16];                 // the device's first wait that ran out since the last reading: code, CTA, kernel, role

struct Ctrl {
    uint64_t full[8], empty[8], aux[8];
    uint64_t acc_full, acc_empty;
    uint32_t tmem_base;
    volatile int abort;
    int32_t* status;                             // the caller's status words, or null
};
constexpr int CTRL_BYTES = 1024;
static_assert(sizeof(Ctrl) <= CTRL_BYTES, "control block too large");

// What bounds these pipelines is the serial cost of synchronisation in the warp that issues the MMAs, not the MMAs: a try_wait
// that succeeds at once takes about 100 cycles (160 inside a called function), tcgen05.commit 46, a tcgen05 fence 23,
// __syncwarp 37 (measured alone on an SM; more beside busy warps), four 128 x 128 MMAs 264. Hence: stages of eight MMAs where
// they fit, ONE barrier per stage for the MMA warp (the auxiliary warps pass on the arrival of the copies with their own), the
// next stage's barrier tested before this stage's MMAs are issued, waits inlined up to their first try. Stages of four
// MMAs with two waits each took 1220 cycles in the z kernel (2048 x 5120 x 512: 37 us).

// One arrival for the warp, after what all its lanes did before.
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}

// Bounded mbarrier wait: false when the budget ran out or another role gave up.
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, Ctrl* c, unsigned long long ns, int which, int role) {
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 3u) == 3u) {
            if (c->abort) return false;
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > ns) {
                c->abort = 1;
                for (int32_t* st : {g_status, c->status})
                    if (st && atomicCAS(&st[0], 0, 120 + which) == 0) { st[1] = (int)blockIdx.x; st[2] = which; st[3] = role; }
                return false;
            }
        }
    }
}
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, Ctrl* c, unsigned long long ns, int which, int role) {
    return mbar_try_wait(bar, parity) || wait_slow(bar, parity, c, ns, which, role);
}
// The same for a whole warp that goes on to warp-wide (.aligned) instructions: one result for all lanes, and all lanes together again.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, Ctrl* c, unsigned long long ns, int which, int role) {
    return __all_sync(0xffffffffu, wait(bar, parity, c, ns, which, role));
}

// ------------------------------------------------------------------------------------------------------------
// Tensor scale
// ------------------------------------------------------------------------------------------------------------
constexpr int Q_THREADS = 256;

// pmax[CTA] = max |x| over the CTA's share; with smoothing Xs = bf16(x / smooth) is formed here (the maximum is its maximum).
// A NaN is the maximum and makes the tensor scale 1 (fp4.activation_scale_from_amax).
__global__ void __launch_bounds__(Q_THREADS) amax_kernel(const uint4* __restrict__ X, const uint4* __restrict__ smooth, uint4* __restrict__ Xs,
                                                         float* __restrict__ pmax, long long nvec, int kvec) {
    __shared__ float red[Q_THREADS / 32];
    griddep_launch_dependents();
    griddep_wait();
    float m = 0.f;
    const long long stride = (long long)gridDim.x * Q_THREADS;
#pragma unroll 4
    for (long long i = (long long)blockIdx.x * Q_THREADS + threadIdx.x; i < nvec; i += stride) {
        const uint4 a = X[i];
        uint4 c = make_uint4(0u, 0u, 0u, 0u);
        if (smooth) c = smooth[(int)(i % kvec)];
        const uint32_t w[4] = {a.x, a.y, a.z, a.w}, v[4] = {c.x, c.y, c.z, c.w};
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float lo, hi;
            qm::unpack_smoothed(w[e], v[e], smooth != nullptr, lo, hi);
            m = qm::max_nan(m, qm::max_nan(fabsf(lo), fabsf(hi)));
            o[e] = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xFFFF0000u);
        }
        if (smooth) Xs[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = qm::max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 1; i < Q_THREADS / 32; ++i) m = qm::max_nan(m, red[i]);
        pmax[blockIdx.x] = m;
    }
}

// One thread per block of sixteen elements; consecutive threads take consecutive blocks of a row.
__global__ void __launch_bounds__(Q_THREADS) quant_kernel(const __nv_bfloat16* __restrict__ X, const float* __restrict__ pmax, int npmax,
                                                          const float* __restrict__ w_gscale, float* __restrict__ alpha_out,
                                                          uint8_t* __restrict__ rec, int rows, int K, int rule, float target) {
    __shared__ float red[Q_THREADS / 32];
    griddep_launch_dependents();
    griddep_wait();
    float m = 0.f;
    for (int i = threadIdx.x; i < npmax; i += Q_THREADS) m = qm::max_nan(m, pmax[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = qm::max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int i = 1; i < Q_THREADS / 32; ++i) m = qm::max_nan(m, red[i]);
    const float gs = m > 0.f ? __fdiv_rn(m, 6.0f * target) : 1.0f;
    // An alpha that underflows to zero leaves the low-rank term alone: zero codes, and 1 as the factor that z is divided by and the
    // accumulator multiplied with.
    const float alpha = __fmul_rn(w_gscale[0], gs);
    const bool lr_alone = alpha == 0.f;
    if (blockIdx.x == 0 && threadIdx.x == 0) alpha_out[0] = lr_alone ? 1.0f : alpha;
    const int kb_row = K >> 4, nkt = K >> 8;
    const long long total = (long long)rows * kb_row, stride = (long long)gridDim.x * Q_THREADS;
    for (long long i = (long long)blockIdx.x * Q_THREADS + threadIdx.x; i < total; i += stride) {
        const int row = (int)(i / kb_row), kb = (int)(i - (long long)row * kb_row);
        const uint4* src = reinterpret_cast<const uint4*>(X + (size_t)row * K + kb * 16);
        const uint4 a = src[0], b = src[1];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float x[16];
#pragma unroll
        for (int e = 0; e < 8; ++e) { x[2 * e] = __uint_as_float(w[e] << 16); x[2 * e + 1] = __uint_as_float(w[e] & 0xFFFF0000u); }
        uint2 c;
        uint8_t sf;
        qm::quant_block16<false>(x, gs, rule, c, sf);
        if (lr_alone) { c = make_uint2(0u, 0u); sf = 0; }
        const int r = row & 127, b16 = kb & 15, ch = b16 >> 1;
        uint8_t* out = rec + ((size_t)(row >> 7) * nkt + (kb >> 4)) * A_REC;
        *reinterpret_cast<uint2*>(out + r * 128 + ((ch ^ (r & 7)) << 4) + (b16 & 1) * 8) = c;
        out[TM * 128 + (b16 >> 2) * 512 + (r & 31) * 16 + (r >> 5) * 4 + (b16 & 3)] = sf;
    }
}

// Sign bits (set = +1) of eight consecutive elements -> 16 bytes of bf16 +-1.0. One multiplication takes a pair's two bits to
// bits 15 and 31 (and to others that the mask drops): three instructions per pair.
__device__ __forceinline__ uint4 signs8(uint32_t bits) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = (((bits & (3u << (2 * i))) * (0x40008000u >> (2 * i))) & 0x80008000u) ^ 0xBF80BF80u;
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// One step of the transposition of four 16-byte pieces over four lanes: the lane without the bit keeps `a` and trades `b` for
// its partner's `a`.
__device__ __forceinline__ void swap_pieces(uint4& a, uint4& b, bool hi, int mask) {
    const uint4 give = hi ? a : b;
    uint4 got;
    got.x = __shfl_xor_sync(0xffffffffu, give.x, mask);
    got.y = __shfl_xor_sync(0xffffffffu, give.y, mask);
    got.z = __shfl_xor_sync(0xffffffffu, give.z, mask);
    got.w = __shfl_xor_sync(0xffffffffu, give.w, mask);
    if (hi) a = got; else b = got;
}

// ------------------------------------------------------------------------------------------------------------
// z = S .* (X sign(V)^T) / alpha
// ------------------------------------------------------------------------------------------------------------
// Tile = 128 rows x NR ranks, K cut into stages of 128 elements that the CTAs of a cluster share. Per stage: X by TMA (two boxes
// of 64 elements, 128-byte swizzle), the sign image written by 128 of the 256 auxiliary threads (the two halves take stages in
// turn), eight MMAs. The partial sums meet in distributed shared memory: CTA q of the cluster adds columns
// [q NR / c, (q + 1) NR / c) over the CTAs in order.
struct ZParams {
    const uint8_t* Vp;
    const __nv_bfloat16* S;
    const float* alpha;
    uint8_t *zrec, *z3;             // z3: third parts of the last row tile, or null
    int32_t* status;
    int skip;                       // test aid: this CTA's copies are left out (-1: none)
    unsigned long long wait_ns;
    int rows, K, R, nrt, ntr, cs;   // ntr: rank tiles
};
template <int NR> struct ZCfg {
    static constexpr int STAGE = 2 * (TM + NR) * 128;         // [X of two chunks | sign images of two chunks]
    static constexpr int ST = NR == 128 ? 3 : 4;
    static constexpr int SMEM = 1024 + ST * STAGE + CTRL_BYTES;
    static_assert(ST * STAGE >= TM * NR * 4, "the exchange of the partial sums reuses the ring");
};

// THIRD: the last row tile gets third parts.
template <int NR, bool THIRD>
__global__ void __launch_bounds__(Z_NT, 1) z_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ ZParams p) {
    using C = ZCfg<NR>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(sm + C::ST * C::STAGE);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int q = blockIdx.x % p.cs, tile = blockIdx.x / p.cs;
    const int rt = tile / p.ntr, rb = tile - rt * p.ntr;
    const int nch = p.K >> 7, c0 = q * nch / p.cs, c1 = (q + 1) * nch / p.cs;      // stages of this CTA
    if (tid == 0) {
        for (int s = 0; s < C::ST; ++s) {
            mbar_init(smem_u32(&ctrl->full[s]), 1);
            mbar_init(smem_u32(&ctrl->empty[s]), 1);
            mbar_init(smem_u32(&ctrl->aux[s]), 4);       // one arrival per warp of the group
        }
        mbar_init(smem_u32(&ctrl->acc_full), 1);
        ctrl->abort = 0;
        ctrl->status = p.status;
        fence_mbar_init();
        prefetch_tmap(&tmX);
    }
    if (warp == MMA_WARP) { tmem_alloc(smem_u32(&ctrl->tmem_base), NR); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    griddep_launch_dependents();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
    griddep_wait();
    if (warp == PRODUCER_WARP) {
        if (lane == 0 && (int)blockIdx.x != p.skip) {
            fence_proxy_async_global();
            int s = 0;
            uint32_t par = 1u;
            for (int c = c0; c < c1; ++c) {
                if (c - c0 >= C::ST && !wait(smem_u32(&ctrl->empty[s]), par, ctrl, p.wait_ns, 1, 8)) break;
                const uint32_t bar = smem_u32(&ctrl->full[s]), st = base + s * C::STAGE;
                mbar_arrive_expect_tx(bar, 2 * TM * 128);
                tma_load_2d(st, &tmX, c * 128, rt * TM, bar);
                tma_load_2d(st + TM * 128, &tmX, c * 128 + 64, rt * TM, bar);
                if (++s == C::ST) { s = 0; par ^= 1u; }
            }
        }
    } else if (warp == MMA_WARP) {
        constexpr uint32_t idesc = make_idesc_bf16(TM, NR);
        int s = 0;
        uint32_t par = 0u;
        bool ready = false;
        for (int c = c0; c < c1; ++c) {
            if (!ready && !warp_wait(smem_u32(&ctrl->aux[s]), par, ctrl, p.wait_ns, 1, 9)) break;
            const int sn = s + 1 == C::ST ? 0 : s + 1;
            const uint32_t pn = sn == 0 ? par ^ 1u : par;
            ready = __all_sync(0xffffffffu, mbar_test_wait(smem_u32(&ctrl->aux[sn]), pn));
            tc_fence_after_sync();
            if (elect_one()) {
                const uint64_t ad = make_smem_desc(base + s * C::STAGE, 1024, 2), bd = make_smem_desc(base + s * C::STAGE + 2 * TM * 128, 1024, 2);
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    tc_mma_bf16(tmem, ad + (k >> 2) * (TM * 128 / 16) + 2 * (k & 3), bd + (k >> 2) * (NR * 128 / 16) + 2 * (k & 3), idesc,
                                (c > c0 || k > 0) ? 1u : 0u);
                if (c + C::ST < c1) tc_commit(smem_u32(&ctrl->empty[s]));
                if (c == c1 - 1) tc_commit(smem_u32(&ctrl->acc_full));
            }
            __syncwarp();
            s = sn;
            par = pn;
        }
    } else {
        // sign images: group g takes stages c0 + g, c0 + g + 2, ...; thread = rank (NR = 128) or one of a rank's two chunks (NR = 64)
        const int g = warp >> 2, t = tid & 127;
        const int r = NR == 128 ? t : t >> 1, h0 = NR == 128 ? 0 : t & 1;
        constexpr int NH = NR == 128 ? 2 : 1;            // chunks per thread
        const int rank = rb * NR + r;
        const bool live = rank < p.R;
        const uint8_t* vrow = p.Vp + (size_t)(live ? rank : 0) * (p.K >> 3);
        int s = g;
        uint32_t par = 1u;
        bool ok = true;
        // (the words of two images are requested while the two before them are written, into registers of their own: moving a
        // requested word to another register waits for it)
        constexpr int BATCH = 2;
        uint2 cur[BATCH][NH], nxt[BATCH][NH];
        auto words = [&](int c, uint2 (&v)[NH]) {
#pragma unroll
            for (int h = 0; h < NH; ++h)
                v[h] = (live && c < c1) ? *reinterpret_cast<const uint2*>(vrow + (size_t)c * 16 + (h0 + h) * 8) : make_uint2(0u, 0u);
        };
#pragma unroll
        for (int i = 0; i < BATCH; ++i) words(c0 + g + 2 * i, cur[i]);
        for (int cb = c0 + g; ok && cb < c1; cb += 2 * BATCH) {
#pragma unroll
            for (int i = 0; i < BATCH; ++i) words(cb + 2 * (BATCH + i), nxt[i]);
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int c = cb + 2 * i;
                if (c < c1 && ok) {
                    if (c - c0 >= C::ST) ok = warp_wait(smem_u32(&ctrl->empty[s]), par, ctrl, p.wait_ns, 1, g);
                    if (ok) {
#pragma unroll
                        for (int h = 0; h < NH; ++h) {
                            uint8_t* row = sm + s * C::STAGE + 2 * TM * 128 + (h0 + h) * NR * 128 + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
                            for (int pc = 0; pc < 8; ++pc) {
                                const uint32_t bits = (pc < 4 ? cur[i][h].x : cur[i][h].y) >> (8 * (pc & 3));
                                *reinterpret_cast<uint4*>(row + ((pc ^ (r & 7)) << 4)) = live ? signs8(bits) : make_uint4(0u, 0u, 0u, 0u);
                            }
                        }
                        fence_proxy_async();
                        ok = warp_wait(smem_u32(&ctrl->full[s]), par ^ 1u, ctrl, p.wait_ns, 1, 2 + g);
                        warp_arrive(smem_u32(&ctrl->aux[s]), lane);
                    }
                    s += 2;
                    if (s >= C::ST) { s -= C::ST; par ^= 1u; }
                }
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i)
#pragma unroll
                for (int h = 0; h < NH; ++h) cur[i][h] = nxt[i][h];
        }
        if (!warp_wait(smem_u32(&ctrl->acc_full), 0, ctrl, p.wait_ns, 1, 11)) ctrl->abort = 1;
        tc_fence_after_sync();
    }
    // ---- partial sums -> the cluster's CTAs: [source CTA][column][row] of the ring memory, which nobody uses any more ----
    __syncwarp();
    __syncthreads();
    if (p.cs > 1) cluster_sync_all();
    const int W = NR / p.cs;                             // columns per CTA
    const int row = tid & 127, half = tid >> 7;
    if (warp < AUX_WARPS) {
#pragma unroll 1
        for (int j = 0; j < NR / 2; j += 16) {
            const int col = half * (NR / 2) + j;
            float d[16];
            tmem_ld_x16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + col, d);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int cc = col + i, t = cc / W;
                st_cluster_f32(map_to_cta(base + (uint32_t)((q * W + cc - t * W) * TM + row) * 4u, (uint32_t)t), d[i]);
            }
        }
        tc_fence_before_sync();
    }
    __syncwarp();
    if (p.cs > 1) cluster_sync_all();
    else __syncthreads();
    if (warp < AUX_WARPS && !ctrl->abort) {
        const float alpha = *p.alpha;
        const float* part_sums = reinterpret_cast<const float*>(sm);
        const int nlr = (p.R + 63) >> 6;
        const bool third = p.z3 != nullptr && rt == p.nrt - 1;
#pragma unroll 1
        for (int j = half; j < W / 4; j += 2) {          // four ranks at a time
            uint32_t part[3][2];
            const int col = q * W + 4 * j;               // column of the rank tile
            const int rank = rb * NR + col;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float a = 0.f;
                for (int src = 0; src < p.cs; ++src) a = __fadd_rn(a, part_sums[(src * W + 4 * j + i) * TM + row]);
                float z = 0.f;
                if (rank + i < p.R) z = __fdiv_rn(__fmul_rn(a, __bfloat162float(p.S[rank + i])), alpha);
#pragma unroll
                for (int k = 0; k < (THIRD ? 3 : 2); ++k) {          // (the remainders are exact; an infinity has none)
                    const __nv_bfloat16 h = __float2bfloat16_rn(z);
                    const uint32_t hb = __bfloat16_as_ushort(h);
                    z = THIRD && fabsf(__bfloat162float(h)) == INFINITY ? 0.f : z - __bfloat162float(h);
                    if (i & 1) part[k][i >> 1] |= hb << 16; else part[k][i >> 1] = hb;
                }
            }
            if (rank < nlr * 64) {
                const int at = row * 128 + (((((rank & 63) >> 3)) ^ (row & 7)) << 4) + (rank & 4) * 2;
                uint8_t* o = p.zrec + ((size_t)rt * nlr + (rank >> 6)) * Z_REC + at;
                *reinterpret_cast<uint2*>(o) = make_uint2(part[0][0], part[0][1]);
                *reinterpret_cast<uint2*>(o + TM * 128) = make_uint2(part[1][0], part[1][1]);
                if (THIRD && third) *reinterpret_cast<uint2*>(p.z3 + (size_t)(rank >> 6) * (TM * 128) + at) = make_uint2(part[2][0], part[2][1]);
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (ctrl->abort) {      // copies may still be in flight towards the stages
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) { }
    }
    __syncwarp();
    if (p.cs > 1) cluster_sync_all();
    if (warp == MMA_WARP) { tc_fence_after_sync(); tmem_dealloc(tmem, NR); }
}

// ------------------------------------------------------------------------------------------------------------
// GEMM
// ------------------------------------------------------------------------------------------------------------
struct GParams {
    const uint8_t* arec;
    const uint8_t *zrec, *z3;       // (z3: third parts of z, last row tile only, or null)
    const uint8_t* W_sf;
    const int32_t* Ucol;
    const float* alpha;
    const __nv_bfloat16* bias;
    __nv_bfloat16* Y;
    int32_t* status;
    int skip;                       // test aid: this CTA's copies are left out (-1: none)
    unsigned long long wait_ns;
    int rows, N, K, R, Rw, nrt, nnt, nlr;
};
// NT = output columns per tile. A stage holds KS k-tiles of the NVFP4 operands (256 k each) or 64 ranks of the low-rank ones.
template <int NT> struct GCfg {
    static constexpr int KS = NT == 256 ? 1 : 2;
    static constexpr int SFB_BLOCKS = NT >= 128 ? NT / 128 : 1;
    static constexpr int SFB_OFF = KS * A_REC;                                 // [k-tile][block] 2 KB
    static constexpr int B_OFF = SFB_OFF + KS * SFB_BLOCKS * 2048;             // [k-tile] NT x 128 bytes
    static constexpr int FP4_BYTES = B_OFF + KS * NT * 128;
    static constexpr int LR_BYTES = Z_REC + NT * 128;                          // z's two parts, sign image
    static constexpr bool Z3_FITS = LR_BYTES + TM * 128 <= FP4_BYTES;          // (a third part behind them)
    static constexpr int STAGE = FP4_BYTES > LR_BYTES ? FP4_BYTES : LR_BYTES;
    static constexpr int ST = 3;
    static constexpr int SMEM = 1024 + ST * STAGE + CTRL_BYTES;
    static constexpr int SFB_STEP = NT == 256 ? 8 : 4;             // TMEM columns per MMA
    static constexpr int SET = NT == 256 ? 64 : 32;                // TMEM columns of a k-tile's scale factors
    static constexpr int TMEM = NT + ST * KS * SET <= 256 ? 256 : 512;
    static_assert(STAGE % 1024 == 0 && B_OFF % 1024 == 0, "operands of the 128-byte swizzle start on 1024 bytes");
    static_assert(NT + ST * KS * SET <= TMEM, "TMEM columns");
    static_assert(SMEM <= 227 * 1024, "shared memory");
};

// THIRD: the last row tile has third parts of z.
template <int NT, bool THIRD>
__global__ void __launch_bounds__(G_NT, 1) gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ GParams p) {
    using C = GCfg<NT>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(sm + C::ST * C::STAGE);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nkt = p.K >> 8, nfs = (nkt + C::KS - 1) / C::KS, ntiles = p.nrt * p.nnt;      // nfs: NVFP4 stages
    // Stages of a tile: NVFP4, then 64 ranks each. Where z has a third part (rows of the last row tile) it comes with them, or, where a
    // stage has no room for it, in stages of its own behind them.
    auto third_part = [&](int rt) { return THIRD && rt == p.nrt - 1; };
    auto stages = [&](int rt) { return nfs + p.nlr + (!C::Z3_FITS && third_part(rt) ? p.nlr : 0); };
    auto rank_stage = [&](int j) { return !THIRD || C::Z3_FITS || j - nfs < p.nlr ? j - nfs : j - nfs - p.nlr; };
    if (tid == 0) {
        for (int s = 0; s < C::ST; ++s) {
            mbar_init(smem_u32(&ctrl->full[s]), 2);      // (both producer warps)
            mbar_init(smem_u32(&ctrl->empty[s]), 1);
            mbar_init(smem_u32(&ctrl->aux[s]), 4);       // one arrival per warp of the group
        }
        mbar_init(smem_u32(&ctrl->acc_full), 1);
        mbar_init(smem_u32(&ctrl->acc_empty), AUX_WARPS);
        ctrl->abort = 0;
        ctrl->status = p.status;
        fence_mbar_init();
        prefetch_tmap(&tmW);
    }
    if (warp == MMA_WARP) { tmem_alloc(smem_u32(&ctrl->tmem_base), C::TMEM); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    griddep_launch_dependents();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
    griddep_wait();
    if (warp == PRODUCER_WARP || warp == WPROD_WARP) {
        // Few and large copies: a wait-and-issue round of one thread takes about 370 cycles and 55 per further copy (measured), a
        // stage's MMAs 200 - 520. One warp brings the activation record (or z), the other the weight rows and their scales.
        if (lane == 0 && (int)blockIdx.x != p.skip) {
            fence_proxy_async_global();
            int s = 0;
            uint32_t par = 1u;
            bool ok = true, first = true;
            for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x) {
                const int nt = tile / p.nrt, rt = tile - nt * p.nrt;
                const int n0 = nt * NT, blk0 = n0 >> 7, nst = stages(rt);
                const int nblk = NT == 256 && (blk0 + 1) * TM < p.N ? 2 : 1;      // scale blocks that exist
                const uint8_t* arec = p.arec + (size_t)rt * nkt * A_REC;
                const uint8_t* zrec = p.zrec + (size_t)rt * p.nlr * Z_REC;
                const uint8_t* wsf = p.W_sf + (size_t)blk0 * (p.K >> 6) * 512;
                for (int j = 0; j < nst; ++j) {
                    if (!first && !wait(smem_u32(&ctrl->empty[s]), par, ctrl, p.wait_ns, 2, 8)) { ok = false; break; }
                    const uint32_t st = base + s * C::STAGE, bar = smem_u32(&ctrl->full[s]);
                    const int kt = j * C::KS, nk = nkt - kt < C::KS ? nkt - kt : C::KS;
                    if (warp == PRODUCER_WARP) {
                        const bool alone = THIRD && !C::Z3_FITS && j >= nfs + p.nlr, with = C::Z3_FITS && j >= nfs && third_part(rt);
                        const uint32_t bytes = j < nfs ? nk * A_REC : (alone ? TM * 128 : Z_REC);
                        const uint8_t* z3 = p.z3 + (size_t)rank_stage(j) * (TM * 128);
                        mbar_arrive_expect_tx(bar, bytes + (with ? TM * 128 : 0));
                        bulk_load(st, j < nfs ? arec + (size_t)kt * A_REC : (alone ? z3 : zrec + (size_t)(j - nfs) * Z_REC), bytes, bar);
                        if (with) bulk_load(st + C::LR_BYTES, z3, TM * 128, bar);
                    } else if (j < nfs) {
                        mbar_arrive_expect_tx(bar, (uint32_t)(nk * (NT * 128 + nblk * 2048)));
                        tma_load_2d(st + C::B_OFF, &tmW, kt * 128, n0, bar);
                        if (C::KS == 2 && nk == 2) tma_load_2d(st + C::B_OFF + NT * 128, &tmW, kt * 128 + 128, n0, bar);
                        bulk_load(st + C::SFB_OFF, wsf + (size_t)kt * 2048, (uint32_t)nk * 2048u, bar);
                        if (nblk == 2) bulk_load(st + C::SFB_OFF + 2048, wsf + (size_t)(p.K >> 6) * 512 + (size_t)kt * 2048, 2048, bar);      // (KS = 1)
                    } else {
                        mbar_arrive(bar);
                    }
                    if (++s == C::ST) { s = 0; par ^= 1u; first = false; }
                }
            }
        }
    } else if (warp == MMA_WARP) {
        constexpr uint32_t id4 = make_idesc_nvf4(TM, NT), id16 = make_idesc_bf16(TM, NT);
        int s = 0, ti = 0;
        uint32_t par = 0u;
        bool ok = true, ready = false;
        for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, ++ti) {
            const int rt = tile % p.nrt, nst = stages(rt);
            const bool third = third_part(rt);
            if (ti > 0 && !warp_wait(smem_u32(&ctrl->acc_empty), (uint32_t)((ti - 1) & 1), ctrl, p.wait_ns, 2, 9)) break;
            for (int j = 0; j < nst; ++j) {
                if (!ready && !(ok = warp_wait(smem_u32(&ctrl->aux[s]), par, ctrl, p.wait_ns, 2, 10))) break;
                const int sn = s + 1 == C::ST ? 0 : s + 1;
                const uint32_t pn = sn == 0 ? par ^ 1u : par;
                ready = __all_sync(0xffffffffu, mbar_test_wait(smem_u32(&ctrl->aux[sn]), pn));
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint32_t st = base + s * C::STAGE;
                    if (j < nfs) {
#pragma unroll
                        for (int kk = 0; kk < C::KS; ++kk) {
                            if (C::KS == 2 && kk == 1 && 2 * j + 1 >= nkt) break;
                            const uint64_t ad = make_smem_desc(st + kk * A_REC, 1024, 2), bd = make_smem_desc(st + C::B_OFF + kk * NT * 128, 1024, 2);
                            const uint32_t sf = tmem + NT + (s * C::KS + kk) * C::SET;
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                tc_mma_nvf4(tmem, ad + 2 * k, bd + 2 * k, id4, sf + 4 * k, sf + 16 + C::SFB_STEP * k, (j > 0 || kk > 0 || k > 0) ? 1u : 0u);
                        }
                    } else {
                        const uint64_t ad = make_smem_desc(st, 1024, 2), ld = make_smem_desc(st + TM * 128, 1024, 2), bd = make_smem_desc(st + Z_REC, 1024, 2),
                                       td = make_smem_desc(st + (C::Z3_FITS ? C::LR_BYTES : 0), 1024, 2);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            tc_mma_bf16(tmem, ad + 2 * k, bd + 2 * k, id16, 1u);
                            if (!THIRD || C::Z3_FITS || j < nfs + p.nlr) tc_mma_bf16(tmem, ld + 2 * k, bd + 2 * k, id16, 1u);
                            if (THIRD && C::Z3_FITS && third) tc_mma_bf16(tmem, td + 2 * k, bd + 2 * k, id16, 1u);
                        }
                    }
                    tc_commit(smem_u32(&ctrl->empty[s]));
                    if (j == nst - 1) tc_commit(smem_u32(&ctrl->acc_full));
                }
                __syncwarp();
                s = sn;
                par = pn;
            }
        }
    } else {
        // ---- auxiliary warps: group g (four warps, one per TMEM quadrant) serves every second stage ----
        const int g = warp >> 2, t = tid & 127;
        const uint32_t quad = (uint32_t)((warp & 3) * 32) << 16;
        const float alpha = *p.alpha;
        int it = 0, s = 0, ti = 0;
        uint32_t par = 0u;
        bool ok = true;
        constexpr int NC = NT >= 128 ? NT / 128 : 1;
        for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, ++ti) {
            const int nt = tile / p.nrt, rt = tile - nt * p.nrt;
            const int n0 = nt * NT, nst = stages(rt);
            // U words of this thread's columns for its next low-rank stage (64 ranks): requested a stage of its group ahead
            uint32_t u[NC][2];
            auto u_words = [&](int w0, uint32_t (&v)[NC][2]) {
#pragma unroll
                for (int i = 0; i < NC; ++i) {
                    const int n = n0 + (NT == 64 ? t >> 1 : i * 128 + t);
#pragma unroll
                    for (int h = 0; h < 2; ++h) v[i][h] = (n < p.N && w0 + h < p.Rw) ? (uint32_t)p.Ucol[(size_t)n * p.Rw + w0 + h] : 0u;
                }
            };
            u_words(2 * rank_stage(nfs + ((it + nfs + g) & 1)), u);      // (its first low-rank stage is the tile's first or second)
            for (int j = 0; j < nst; ++j, ++it) {
                if ((it & 1) == g) {
                    uint8_t* st = sm + s * C::STAGE;
                    // The slot's previous stage was the other group's: until its MMAs are known to be over, the parity of this
                    // stage's full barrier could be that of the lap before.
                    if (it >= C::ST && !(ok = warp_wait(smem_u32(&ctrl->empty[s]), par ^ 1u, ctrl, p.wait_ns, 2, g))) break;
                    if (j < nfs) {
                        // scale factors: lane l of every quadrant holds rows l, l + 32, l + 64, l + 96 of an atom in four consecutive columns
                        if (!(ok = warp_wait(smem_u32(&ctrl->full[s]), par, ctrl, p.wait_ns, 2, g))) break;
                        tc_fence_after_sync();
#pragma unroll
                        for (int kk = 0; kk < C::KS; ++kk) {
                            if (C::KS == 2 && kk == 1 && 2 * j + 1 >= nkt) break;
                            const uint4* fa = reinterpret_cast<const uint4*>(st + kk * A_REC + TM * 128) + lane;
                            const uint4* fb = reinterpret_cast<const uint4*>(st + C::SFB_OFF + kk * C::SFB_BLOCKS * 2048) + lane;
                            const uint32_t set = tmem + quad + NT + (s * C::KS + kk) * C::SET;
                            uint32_t ra[16], rb[4 * C::SFB_STEP];
#pragma unroll
                            for (int a = 0; a < 4; ++a) {
                                const uint4 x = fa[a * 32];
                                ra[4 * a] = x.x; ra[4 * a + 1] = x.y; ra[4 * a + 2] = x.z; ra[4 * a + 3] = x.w;
#pragma unroll
                                for (int b = 0; b < C::SFB_BLOCKS; ++b) {
                                    const uint4 y = fb[b * 128 + a * 32];
                                    uint32_t* o = rb + C::SFB_STEP * a + 4 * b;
                                    if (NT == 64 && (n0 & 64)) { o[0] = y.z; o[1] = y.w; o[2] = 0u; o[3] = 0u; }
                                    else { o[0] = y.x; o[1] = y.y; o[2] = y.z; o[3] = y.w; }
                                }
                            }
                            tmem_st_x16(set, ra);
                            tmem_st_x16(set + 16, rb);
                            if constexpr (NT == 256) tmem_st_x16(set + 32, rb + 16);
                        }
                        tc_wait_st();
                        tc_fence_before_sync();
                    } else {
                        // sign image of 64 ranks: row = output column (NT = 64: two threads per column, 32 ranks each)
                        uint32_t un[NC][2];
                        u_words(2 * rank_stage(j + 2), un);
#pragma unroll
                        for (int i = 0; i < NC; ++i) {
                            const int r = NT == 64 ? t >> 1 : i * 128 + t;
                            uint8_t* row = st + Z_REC + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
                            for (int pc = 0; pc < 8; ++pc) {
                                if (NT == 64 && (pc >> 2) != (t & 1)) continue;
                                *reinterpret_cast<uint4*>(row + ((pc ^ (r & 7)) << 4)) = signs8(u[i][pc >> 2] >> (8 * (pc & 3)));
                            }
                        }
                        fence_proxy_async();
                        if (!(ok = warp_wait(smem_u32(&ctrl->full[s]), par, ctrl, p.wait_ns, 2, 2 + g))) break;
#pragma unroll
                        for (int i = 0; i < NC; ++i) { u[i][0] = un[i][0]; u[i][1] = un[i][1]; }
                    }
                    warp_arrive(smem_u32(&ctrl->aux[s]), lane);
                }
                if (++s == C::ST) { s = 0; par ^= 1u; }
            }
            if (!ok) break;
            // ---- epilogue: TMEM lane = row, this warp's half of the columns, 32 at a time. A lane's 64 bytes of its row are
            // exchanged within groups of four lanes, so that a store instruction writes 64 consecutive bytes of eight rows
            // (16 bytes of 32 rows each took 7600 cycles per 128 x 256 tile) ----
            if (!warp_wait(smem_u32(&ctrl->acc_full), (uint32_t)(ti & 1), ctrl, p.wait_ns, 2, 12)) break;
            tc_fence_after_sync();
            const int m0 = rt * TM + (warp & 3) * 32 + (lane & ~3);
#pragma unroll 1
            for (int c = g * (NT / 2); c < (g + 1) * (NT / 2) && n0 + c < p.N; c += 32) {
                float d[32];
                tmem_ld_x16(tmem + quad + c, d);
                tmem_ld_x16(tmem + quad + c + 16, d + 16);
                uint4 o[4];
                tc_wait_ld();
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    uint4 b = make_uint4(0u, 0u, 0u, 0u);
                    if (p.bias && n0 + c + 8 * h < p.N) b = *reinterpret_cast<const uint4*>(p.bias + n0 + c + 8 * h);      // (N is a multiple of 8)
                    const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const __nv_bfloat162 v = __floats2bfloat162_rn(alpha * d[8 * h + 2 * e] + __uint_as_float(bw[e] << 16),
                                                                       alpha * d[8 * h + 2 * e + 1] + __uint_as_float(bw[e] & 0xFFFF0000u));
                        w[e] = *reinterpret_cast<const uint32_t*>(&v);
                    }
                    o[h] = make_uint4(w[0], w[1], w[2], w[3]);
                }
                swap_pieces(o[0], o[1], lane & 1, 1);
                swap_pieces(o[2], o[3], lane & 1, 1);
                swap_pieces(o[0], o[2], lane & 2, 2);
                swap_pieces(o[1], o[3], lane & 2, 2);
                const int n = n0 + c + 8 * (lane & 3);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (m0 + k < p.rows && n < p.N) *reinterpret_cast<uint4*>(p.Y + (size_t)(m0 + k) * p.N + n) = o[k];
            }
            tc_fence_before_sync();
            warp_arrive(smem_u32(&ctrl->acc_empty), lane);
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (ctrl->abort) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) { }
    }
    if (warp == MMA_WARP) { tc_fence_after_sync(); tmem_dealloc(tmem, C::TMEM); }
}

// ------------------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------------------
struct Layout { size_t alpha, pmax, xs, arec, zrec, z3, total; int nrt, nlr; bool third; };
constexpr int MAX_PMAX = 592;
static Layout layout(int rows, int K, int R, bool smooth) {
    Layout L;
    L.nrt = (rows + TM - 1) / TM;
    L.nlr = (R + 63) / 64;
    auto up = [](size_t x) { return (x + 255) / 256 * 256; };
    size_t o = 0;
    L.alpha = o; o += 256;
    L.pmax = o; o += up(MAX_PMAX * 4);
    L.xs = o; if (smooth) o += up((size_t)rows * K * 2);
    L.arec = o; o += up((size_t)L.nrt * (K / KT) * A_REC);
    L.zrec = o; o += (size_t)L.nrt * L.nlr * Z_REC;
    // One to eight rows behind the last whole 32 have a third part of z, which is then z itself: taken alone (a decode launch) these rows
    // have fp32 z too. It costs their row tile half as many low-rank MMAs again (5120 x 5120, r = 512: 33 rows 28.1 -> 30.2 us,
    // 513 rows 52 -> 57.6, 2049 rows 114 -> 121), and all other row counts nothing.
    L.third = R > 0 && (rows & 31) >= 1 && (rows & 31) <= 8;
    L.z3 = o; if (L.third) o += (size_t)L.nlr * TM * 128;
    L.total = o;
    return L;
}

struct Launch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    Launch(int grid, int block, size_t smem, cudaStream_t s, int cluster = 1) {
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3((unsigned)block);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        int n = 0;
        if (biloco_internal_use_pdl()) {
            attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[n++].val.programmaticStreamSerializationAllowed = 1;
        }
        if (cluster > 1) {
            attr[n].id = cudaLaunchAttributeClusterDimension;
            attr[n].val.clusterDim.x = (unsigned)cluster;
            attr[n].val.clusterDim.y = 1;
            attr[n++].val.clusterDim.z = 1;
        }
        cfg.attrs = attr;
        cfg.numAttrs = (unsigned)n;
    }
};

template <int NR, bool THIRD>
static int launch_z_form(const CUtensorMap& tmX, ZParams z, int nrt, int sms, int dev, cudaStream_t s) {
    static bool ready[64] = {false};
    if (!ready[dev]) {
        if (cudaFuncSetAttribute(z_gemm_kernel<NR, THIRD>, cudaFuncAttributeMaxDynamicSharedMemorySize, ZCfg<NR>::SMEM) != cudaSuccess) return BILOCO_ERR_CUDA;
        ready[dev] = true;
    }
    z.ntr = (z.R + NR - 1) / NR;
    const int tiles = nrt * z.ntr;
    z.cs = 1;
    while (z.cs < 8 && tiles * z.cs * 2 <= sms && (z.K >> 7) >= z.cs * 4) z.cs *= 2;
    Launch l(tiles * z.cs, Z_NT, ZCfg<NR>::SMEM, s, z.cs);
    return cudaLaunchKernelEx(&l.cfg, z_gemm_kernel<NR, THIRD>, tmX, z) == cudaSuccess ? BILOCO_OK : BILOCO_ERR_CUDA;
}
template <int NR>
static int launch_z(const CUtensorMap& tmX, const ZParams& z, int nrt, int sms, int dev, cudaStream_t s) {
    return z.z3 ? launch_z_form<NR, true>(tmX, z, nrt, sms, dev, s) : launch_z_form<NR, false>(tmX, z, nrt, sms, dev, s);
}

template <int NT, bool THIRD>
static int launch_gemm_form(const void* W, GParams g, int sms, int dev, cudaStream_t s) {
    static bool ready[64] = {false};
    if (!ready[dev]) {
        if (cudaFuncSetAttribute(gemm_kernel<NT, THIRD>, cudaFuncAttributeMaxDynamicSharedMemorySize, GCfg<NT>::SMEM) != cudaSuccess) return BILOCO_ERR_CUDA;
        ready[dev] = true;
    }
    CUtensorMap tmW;
    if (biloco_internal_encode_map(&tmW, 0, W, g.N, g.K / 2, 128, NT) != BILOCO_OK) return BILOCO_ERR_CUDA;
    g.nnt = (g.N + NT - 1) / NT;
    const int tiles = g.nrt * g.nnt;
    Launch l(tiles < sms ? tiles : sms, G_NT, GCfg<NT>::SMEM, s);
    return cudaLaunchKernelEx(&l.cfg, gemm_kernel<NT, THIRD>, tmW, g) == cudaSuccess ? BILOCO_OK : BILOCO_ERR_CUDA;
}
template <int NT>
static int launch_gemm(const void* W, const GParams& g, int sms, int dev, cudaStream_t s) {
    return g.z3 ? launch_gemm_form<NT, true>(W, g, sms, dev, s) : launch_gemm_form<NT, false>(W, g, sms, dev, s);
}

// Estimated cycles of the GEMM with NT columns per tile: waves of (k-stages, each the longer of its MMAs and its loads, low-rank
// stages, prologue and epilogue). MMA cycles as measured (see elect_one); loads at about 45 bytes per cycle and SM.
static double gemm_cost(int NT, int mma, int nrt, int N, int nkt, int nlr, int sms, bool third) {
    const int tiles = nrt * ((N + NT - 1) / NT);
    const double load = (A_REC + NT * 128 + (NT >= 128 ? NT / 128 : 1) * 2048) / 45.0, work = 4.0 * mma;
    return (double)((tiles + sms - 1) / sms) * (nkt * (load > work ? load : work) + nlr * 8.0 * mma + 1500.0 + 6.0 * NT)
           + (third ? nlr * (NT == 256 ? 8.0 * mma : 4.0 * mma) : 0.0);      // (one row tile's third parts; stages of their own at 256 columns)
}

}  // namespace prompt
}  // namespace biloco

using namespace biloco;

extern "C" size_t biloco_b200_prompt_ws_bytes(int rows, int N, int K, int R, int smooth) {
    if (rows < 1 || rows > (1 << 22) || N < 8 || (N % 8) || K < 256 || (K % 256) || R < 0) return 0;
    return prompt::layout(rows, K, R, smooth != 0).total;
}

extern "C" int biloco_b200_prompt_linear(const void* W_codes, const void* W_sf, const float* w_gscale, const void* X_bf16, const void* smooth_bf16,
                                         const void* V_packed, const int32_t* U_col32, const void* S_bf16, const void* bias_bf16, void* Y_bf16,
                                         void* ws, size_t ws_bytes, int32_t* status, int rows, int N, int K, int R, int rule, biloco_stream_t stream) {
    if (!W_codes || !W_sf || !w_gscale || !X_bf16 || !Y_bf16 || !ws) return BILOCO_ERR_NULL;
    if (R > 0 && (!V_packed || !U_col32 || !S_bf16)) return BILOCO_ERR_NULL;
    if (rule != BILOCO_RULE_STATIC_6 && rule != BILOCO_RULE_STATIC_4 && rule != BILOCO_RULE_MSE) return BILOCO_ERR_MODE;
    const size_t need = biloco_b200_prompt_ws_bytes(rows, N, K, R, smooth_bf16 != nullptr);
    if (need == 0) return BILOCO_ERR_SHAPE;
    if (ws_bytes < need) return BILOCO_ERR_SCRATCH;
    if (((uintptr_t)W_codes & 15) || ((uintptr_t)W_sf & 15) || ((uintptr_t)X_bf16 & 15) || ((uintptr_t)smooth_bf16 & 15) || ((uintptr_t)bias_bf16 & 15) ||
        ((uintptr_t)Y_bf16 & 15) || ((uintptr_t)ws & 255) || ((uintptr_t)V_packed & 7) || ((uintptr_t)U_col32 & 3) || ((uintptr_t)status & 3))
        return BILOCO_ERR_ALIGN;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return BILOCO_ERR_CUDA;
    cudaStream_t s = (cudaStream_t)stream;
    const prompt::Layout L = prompt::layout(rows, K, R, smooth_bf16 != nullptr);
    uint8_t* w = (uint8_t*)ws;
    float* alpha = (float*)(w + L.alpha);
    float* pmax = (float*)(w + L.pmax);
    const void* X = smooth_bf16 ? w + L.xs : X_bf16;
    const long long nvec = (long long)rows * K / 8;
    long long g1 = (nvec + prompt::Q_THREADS * 4 - 1) / (prompt::Q_THREADS * 4);
    if (g1 > prompt::MAX_PMAX) g1 = prompt::MAX_PMAX;
    {
        prompt::Launch l((int)g1, prompt::Q_THREADS, 0, s);
        if (cudaLaunchKernelEx(&l.cfg, prompt::amax_kernel, (const uint4*)X_bf16, (const uint4*)smooth_bf16, (uint4*)(w + L.xs), pmax, nvec, K / 8) != cudaSuccess)
            return BILOCO_ERR_CUDA;
    }
    {
        long long g2 = ((long long)rows * (K / 16) + prompt::Q_THREADS - 1) / prompt::Q_THREADS;
        if (g2 > 8ll * sms) g2 = 8ll * sms;
        prompt::Launch l((int)g2, prompt::Q_THREADS, 0, s);
        if (cudaLaunchKernelEx(&l.cfg, prompt::quant_kernel, (const __nv_bfloat16*)X, (const float*)pmax, (int)g1, w_gscale, alpha, w + L.arec, rows, K, rule,
                               rule == BILOCO_RULE_STATIC_6 ? 448.0f : 256.0f) != cudaSuccess)
            return BILOCO_ERR_CUDA;
    }
    const unsigned long long ns = biloco_internal_wait_ns();
    if (R > 0) {
        CUtensorMap tmX;
        if (biloco_internal_encode_map(&tmX, 1, X, rows, K, 64, prompt::TM) != BILOCO_OK) return BILOCO_ERR_CUDA;
        prompt::ZParams z = {(const uint8_t*)V_packed, (const __nv_bfloat16*)S_bf16, alpha, w + L.zrec, L.third ? w + L.z3 : nullptr, status, biloco_internal_skip_publish(), ns, rows, K, R, L.nrt, 0, 0};
        // 128 ranks per tile halve the reads of X; 64 where that would leave the device half empty
        const int rc = (R > 64 && L.nrt * ((R + 127) / 128) * 8 >= sms) ? prompt::launch_z<128>(tmX, z, L.nrt, sms, dev, s) : prompt::launch_z<64>(tmX, z, L.nrt, sms, dev, s);
        if (rc != BILOCO_OK) return rc;
    }
    prompt::GParams g = {w + L.arec, w + L.zrec, L.third ? w + L.z3 : nullptr, (const uint8_t*)W_sf, U_col32, alpha, (const __nv_bfloat16*)bias_bf16, (__nv_bfloat16*)Y_bf16, status, biloco_internal_skip_publish(), ns,
                         rows, N, K, R, (R + 31) / 32, L.nrt, 0, L.nlr};
    const double c64 = prompt::gemm_cost(64, 50, L.nrt, N, K / 256, L.nlr, sms, L.third), c128 = prompt::gemm_cost(128, 66, L.nrt, N, K / 256, L.nlr, sms, L.third),
                 c256 = prompt::gemm_cost(256, 130, L.nrt, N, K / 256, L.nlr, sms, L.third);
    if (c256 <= c128 && c256 <= c64) return prompt::launch_gemm<256>(W_codes, g, sms, dev, s);
    if (c128 <= c64) return prompt::launch_gemm<128>(W_codes, g, sms, dev, s);
    return prompt::launch_gemm<64>(W_codes, g, sms, dev, s);
}

// The device's prompt launches since the last reading (synchronises, and clears): word 0 is non-zero if a device-side wait ran out.
extern "C" int biloco_b200_prompt_status(int32_t* out16, biloco_stream_t stream) {
    if (!out16) return BILOCO_ERR_NULL;
    void* words = nullptr;
    if (cudaGetSymbolAddress(&words, prompt::g_status) != cudaSuccess ||
        cudaMemcpyAsync(out16, words, sizeof(int32_t) * 16, cudaMemcpyDeviceToHost, (cudaStream_t)stream) != cudaSuccess ||
        cudaMemsetAsync(words, 0, sizeof(int32_t) * 16, (cudaStream_t)stream) != cudaSuccess)
        return BILOCO_ERR_CUDA;
    return cudaStreamSynchronize((cudaStream_t)stream) == cudaSuccess ? BILOCO_OK : BILOCO_ERR_CUDA;
}
