// The fused linear for 5 to 32 activation rows (schedules 2 and 4): everything that grows with the rows is on the tensor cores.
//
// Work split as in fused_kernel.cuh: units of 128 weight rows x 256 k, an equal contiguous range per CTA (stream-K), the weights
// as the MMA's 128-row operand, 8 / 16 / 32 activation rows as its N operand, one 18 KB record per unit. What is different, and why:
//
//  * z = S .* (X sign(V)^T) by MMAs inside the launch: item (rank block of 128, K slice) builds +-1.0 images of the V bits (before
//    the dependency wait: static) and multiplies them with its slice of X; partial sums go to global memory, every item's CTA adds a
//    share of its rank block's outputs over the slices in order and publishes z. On CUDA cores this took most of a launch
//    from eight rows on, as a launch of its own in front it cost two grid hand-overs.
//  * Expansion by MMAs: +-1.0 images of the U bits times z as a sum of bf16 parts, the parts side by side as ONE operand (an MMA
//    costs 41 cycles at N = 16 and 50 at N = 64, so further parts are nearly free). Up to eight rows three parts, which
//    are z itself, as the tile kernel's fp32 expansion has it (fp32 outputs 1.1e-7 off the 64-bit value, 2.4e-6 with two parts); from
//    nine rows two, which keep 2^-17 of it (2.5e-6). bf16 outputs are 1.66e-3 off either way. The chunks of a round are split
//    into parts by all 256 threads at once: by one group of threads after the other 8 rows of 2560 -> 9728 took 15.2 us instead of 13.4.
//  * A tile's contributors all add: contributor s of n takes words [s w / n, (s + 1) w / n) of the w that a partial sum has. With one finisher
//    per tile the launch was as long as that CTA's n - 1 rounds of dependent loads after everybody else had left.
//  * Nothing is announced, every hand-over is one memory round trip. Partial sums travel as 16-byte words [three rows' sums | launch count]
//    that the reader polls itself (one store and one load each, whole or not there); z carries a validity mark in the lowest
//    mantissa bit (parity of the launch count). The count belongs to this scratch and is kept as eight 64-bit words to which every
//    leaving CTA adds its share of 2^20 (no atomic with a result on the way out). Sums are whole fp32 values: with the mark in their
//    lowest bit too, fp32 outputs of the NVFP4 part alone were 7.8e-8 off (5120 x 5120, 16 rows) instead of 4.9e-8.
//  * Scale factors are moved to TMEM by two groups of four warps in turn (one group's wait - load - store - arrive chain takes
//    longer than a unit arrives at HBM speed), and the MMA warp waits on one barrier per unit.
//
// Measured (us per call, captured chain of distinct layers, K = N = 5120, r = 512, rows 8 / 16 / 32): 12.9 / 13.9 / 16.5 against
// 20.4 / 24.4 / 29.9 with z on CUDA cores (8) or as a launch of its own (16, 32) and one finisher per tile.
#pragma once
#include "fused_cfg.cuh"

namespace biloco {
namespace batch {

constexpr int EPI_WARPS = 8;                     // z, expansion, epilogue (TMEM quadrant = warp % 4)
constexpr int EPI_THREADS = EPI_WARPS * 32;
constexpr int SF_WARP0 = 8;                      // two groups of four: scale factors -> TMEM
constexpr int MMA_WARP = 16;
constexpr int W_WARP = 17, A_WARP = 18;          // weight and activation copies
constexpr int NT = 19 * 32;
constexpr int MAX_RING = 8;
constexpr int IMG = 16384;                       // +-1.0 image: 128 rows x 64 bf16
constexpr int NIMG = 4;                          // images in shared memory at a time
constexpr int TMEM_COLS = 512;
constexpr int SF_COL = 64;                       // scale factors of stage s: 32 columns at 64 + 32 s (after two accumulators of 32)
constexpr int LR_COL = 320;                      // expansion accumulators, 64 columns per segment parity (LR_N of them used); the first also z's
static_assert(SF_COL + 32 * MAX_RING <= LR_COL && LR_COL + 128 <= TMEM_COLS, "TMEM columns");

template <int MMA_N> struct Cfg {
    static constexpr int A_TILE = MMA_N * 128;
    static constexpr int STAGE = W_TILE_BYTES + SF_TILE_BYTES + A_TILE + SF_TILE_BYTES;
    static constexpr int PARTS = MMA_N == 8 ? 3 : 2;                       // bf16 parts of z
    static constexpr int LR_N = MMA_N == 8 ? 32 : PARTS * MMA_N;           // N of the expansion's MMAs: a multiple of 16 (8 rows: columns 24 .. 31 are not read)
    // One z operand: 64 ranks of every part, [part][row] (z stage: the X chunk in the first rows). At 8 rows the MMA's last eight rows are
    // whatever follows (the next operand, the control block): their columns are not read, and 1 KB each would cost a ring stage.
    static constexpr int ZB = PARTS * MMA_N * 128;
    // Rows of a column that a thread reads from TMEM (its half's; all eight at 8 rows), and 16-byte words of three rows' sums per column.
    static constexpr int RH = MMA_N / 2, VR = MMA_N == 8 ? 8 : RH, HW = (RH + 2) / 3, SW = MMA_N == 8 ? 3 : 2 * HW;
    static constexpr int FIXED = 1024 + NIMG * (IMG + ZB) + 1024;
    static constexpr int RING = (SMEM_BUDGET - FIXED) / STAGE < MAX_RING ? (SMEM_BUDGET - FIXED) / STAGE : MAX_RING;
    static constexpr int SMEM = FIXED + RING * STAGE;
    static_assert(STAGE % 1024 == 0 && RING >= 4, "ring");
    static_assert(LR_N * 128 <= ZB + 1024 && ZB % 1024 == 0 && LR_N <= 64, "z operands");
};

// Place of CTA c's partial sums of a tile that it shares, cf being the tile's first contributor: along the units either the CTA or the
// tile of such a segment goes up, so CTA + tile names it, and CTA + first contributor does too (the next shared tile starts with
// the last contributor of this one). G + min(tiles, G) places, where tiles x contributors would be several times as many.
__host__ __device__ constexpr int part_places(int ntile, int G) { return G + (ntile < G ? ntile : G); }
__device__ __forceinline__ int part_base(int t, int cf, int ntile, int G) { return ntile < G ? t : cf; }

constexpr int sum_words(int mma_n) { return mma_n == 8 ? Cfg<8>::SW : (mma_n == 16 ? Cfg<16>::SW : Cfg<32>::SW); }

struct Params {
    const uint8_t *W_tiled, *W_sf, *A_sf, *A_rec;
    const float* alpha;
    const __nv_bfloat16* X;
    const uint8_t* Vp;
    const int32_t* Ucol;
    const __nv_bfloat16 *S, *C;
    void* Y;
    int32_t* status;
    unsigned long long* count;      // eight words: launches completed on this scratch, in bits 20.. of their sum
    float* zbuf;              // [32][Rpad]
    uint4* zpart;             // [item][SW][128]
    uint4* part;              // [part_base(tile) + CTA][SW][128]
    uint2* const* ar_recv;    // row-parallel use, see FusedParams
    const uint32_t* ar_counter;
    int ar_world, ar_rank, ar_slot;
    int M, N, K, R, Rw, Rpad, ngroups, Rg, gtile[3];
    int ntile, nkt, G;        // G: CTAs with units
    int nks, nitems;          // z: K slices per rank block, items in all
    uint32_t epoch;
    int fp32_out;
    int z_cleared;            // zbuf was cleared in front of this launch: its mark is 1, not the count's parity
    int skip_publish;         // test aid: this CTA keeps its partial sums of z to itself (-1: none)
    unsigned long long wait_ns;
};

struct Ctrl {
    uint64_t full[MAX_RING], empty[MAX_RING], sf[MAX_RING];
    uint64_t acc_full[2], acc_empty[2];
    uint64_t lr_free[NIMG];   // the MMAs that read image b have completed
    uint64_t lr_done;         // the last MMAs of a z round or of a segment's expansion have completed
    uint32_t tmem_base, seq, ar_seq;
    volatile int abort;
};
static_assert(sizeof(Ctrl) <= 1024, "control block too large");

__device__ __noinline__ void give_up(Ctrl* c, const Params& p, int code, int role) {
    c->abort = 1;
    if (atomicCAS(p.status, 0, code) == 0) { p.status[1] = (int)blockIdx.x; p.status[2] = (int)p.epoch; p.status[3] = role; }
}
__device__ __noinline__ bool wait_slow(uint32_t bar, uint32_t parity, Ctrl* c, const Params& p, int code, int role) {
    uint64_t t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 3u) == 3u) {
            if (c->abort) return false;
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > p.wait_ns) { give_up(c, p, code, role); return false; }
        }
    }
}
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity, Ctrl* c, const Params& p, int code, int role) {
    return mbar_try_wait(bar, parity) || wait_slow(bar, parity, c, p, code, role);
}
// for a whole warp that goes on to warp-wide instructions
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, Ctrl* c, const Params& p, int code, int role) {
    return __all_sync(0xffffffffu, wait(bar, parity, c, p, code, role));
}
__device__ __forceinline__ void warp_arrive(uint32_t bar, int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void epi_sync() { named_bar_sync(1, EPI_THREADS); }

__device__ __forceinline__ float mark(float v, uint32_t phase) { return __uint_as_float((__float_as_uint(v) & ~1u) | phase); }
__device__ __forceinline__ float unmark(uint32_t w) { return __uint_as_float(w & ~1u); }

// Three rows' sums and the launch count as one 128-bit access.
__device__ __forceinline__ void st_sums(uint4* dst, float a, float b, float c, uint32_t tag) {
    const uint64_t lo = ((uint64_t)__float_as_uint(b) << 32) | __float_as_uint(a), hi = ((uint64_t)tag << 32) | __float_as_uint(c);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(dst), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ uint4 ld_sums(const uint4* src) {
    uint64_t lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}" : "=l"(lo), "=l"(hi) : "l"(src) : "memory");
    return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

// polls a failed attempt's time: true = give up
struct Poll {
    uint64_t t0 = 0;
    uint32_t it = 0;
    __device__ __forceinline__ bool expired(Ctrl* c, const Params& p, int code) {
        if ((it++ & 15u) != 15u) return false;
        if (c->abort) return true;
        const uint64_t now = globaltimer_ns();
        if (t0 == 0) { t0 = now; return false; }
        if (now - t0 > p.wait_ns) { give_up(c, p, code, 0); return true; }
        return false;
    }
};

// Sign bits (set = +1) of eight elements -> eight bf16 +-1.0: one multiplication takes a pair's bits to bits 15 and 31.
__device__ __forceinline__ uint4 signs8(uint32_t bits) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = (((bits & (3u << (2 * i))) * (0x40008000u >> (2 * i))) & 0x80008000u) ^ 0xBF80BF80u;
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// 32 sign bits into half `h` (32 elements) of row r of an image
__device__ __forceinline__ void image_half(uint8_t* img, int r, int h, uint32_t bits) {
    uint8_t* row = img + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(row + (((4 * h + i) ^ (r & 7)) << 4)) = signs8(bits >> (8 * i));
}

// The next bf16 part of two values; what is left of them stays behind (exactly; nothing of an infinity). Three parts are cut off, which
// cannot overflow and leaves nothing after the third; of two the first is rounded, which saves a bit.
template <int PARTS>
__device__ __forceinline__ uint32_t next_part(float& z0, float& z1) {
    uint32_t w;
    if constexpr (PARTS == 3) {
        w = (__float_as_uint(z0) >> 16) | (__float_as_uint(z1) & 0xFFFF0000u);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(z0, z1);
        w = *reinterpret_cast<const uint32_t*>(&h);
    }
    const float f0 = __uint_as_float(w << 16), f1 = __uint_as_float(w & 0xFFFF0000u);
    z0 = fabsf(f0) == INFINITY ? 0.f : z0 - f0;
    z1 = fabsf(f1) == INFINITY ? 0.f : z1 - f1;
    return w;
}

// Words of three rows' sums of a column. 16 and 32 rows: half h's thread holds rows h RH + 3 t + {0, 1, 2} (below the half's end) in word
// h HW + t; 8 rows: rows 3 w + {0, 1, 2} in word w, of half w % 2's thread (three words instead of four). Words without a row below M
// do not exist: `live` of them do, word(i) is the i-th.
template <int MMA_N> struct SumWords {
    using CF = Cfg<MMA_N>;
    int n0, live;
    __device__ __forceinline__ explicit SumWords(int M) {
        n0 = ((MMA_N == 8 || M < CF::RH ? M : CF::RH) + 2) / 3;
        live = n0 + (MMA_N != 8 && M > CF::RH ? (M - CF::RH + 2) / 3 : 0);
    }
    __device__ __forceinline__ int word(int i) const { return i < n0 ? i : CF::HW + i - n0; }
    static __device__ __forceinline__ int row(int w) { return MMA_N == 8 || w < CF::HW ? 3 * w : CF::RH + 3 * (w - CF::HW); }      // the word's first row
    static __device__ __forceinline__ int rows(int w, int M) {                                                                  // and how many it has
        const int left = MMA_N == 8 ? 3 : CF::RH - 3 * (w < CF::HW ? w : w - CF::HW);
        return min(min(3, left), M - row(w));
    }
    static __device__ __forceinline__ void put(uint4* column, const float (&v)[CF::VR], int half, int M, uint32_t tag) {
        constexpr int NW = MMA_N == 8 ? CF::SW : CF::HW;
#pragma unroll
        for (int t = 0; t < NW; ++t) {
            const float b = 3 * t + 1 < CF::VR ? v[3 * t + 1 < CF::VR ? 3 * t + 1 : 0] : 0.f, c = 3 * t + 2 < CF::VR ? v[3 * t + 2 < CF::VR ? 3 * t + 2 : 0] : 0.f;
            if (MMA_N == 8) {
                if ((t & 1) == half && 3 * t < M) st_sums(column + t * 128, v[3 * t], b, c, tag);
            } else if (half * CF::RH + 3 * t < M) {
                st_sums(column + (half * CF::HW + t) * 128, v[3 * t], b, c, tag);
            }
        }
    }
    // Sums of a word over n sources `step` words apart, from source `first` on in cyclic order, each polled until it carries the launch count.
    static __device__ __forceinline__ void add(const uint4* src, int n, size_t step, int first, uint32_t tag, float (&o)[3], Ctrl* c, const Params& p, int code) {
        o[0] = o[1] = o[2] = 0.f;
#pragma unroll 1
        for (int s0 = 0; s0 < n; s0 += 8) {
            uint4 x[8];
            Poll poll;
#pragma unroll 1
            while (true) {
                uint32_t bad = 0u;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    x[j] = make_uint4(0u, 0u, 0u, tag);
                    const int k = s0 + j + first;
                    if (s0 + j < n) x[j] = ld_sums(src + (size_t)(k < n ? k : k - n) * step);
                    bad |= x[j].w ^ tag;
                }
                if (!bad) break;
                if (poll.expired(c, p, code)) break;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (s0 + j < n) {
                    o[0] = __fadd_rn(o[0], __uint_as_float(x[j].x));
                    o[1] = __fadd_rn(o[1], __uint_as_float(x[j].y));
                    o[2] = __fadd_rn(o[2], __uint_as_float(x[j].z));
                }
        }
    }
};

template <int MMA_N>
__device__ __forceinline__ void ld_rows(uint32_t taddr, int half, float (&v)[Cfg<MMA_N>::VR]) {      // this thread's rows of an accumulator
    if constexpr (MMA_N == 8) tmem_ld_x8(taddr, v);
    else if constexpr (MMA_N == 16) tmem_ld_x8(taddr + 8 * half, v);
    else tmem_ld_x16(taddr + 16 * half, v);
    tc_wait_ld();
}

// One output element: residual, rounding, store, and the peers' copies.
template <bool PUSH>
__device__ __forceinline__ void put(const Params& p, const Ctrl* c, int m, int n, float o) {
    const size_t i = (size_t)m * p.N + n;
    if (p.C) o += __bfloat162float(p.C[i]);
    if (!p.fp32_out) { reinterpret_cast<__nv_bfloat16*>(p.Y)[i] = __float2bfloat16(o); return; }
    reinterpret_cast<float*>(p.Y)[i] = o;
    if constexpr (PUSH) {
        const size_t off = (size_t)(c->ar_seq & 1u) * p.ar_world * p.ar_slot + (size_t)p.ar_rank * p.ar_slot + i;
        for (int q = 0; q < p.ar_world; ++q)
            if (q != p.ar_rank)
                asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p.ar_recv[q] + off), "r"(__float_as_uint(o)), "r"(c->ar_seq) : "memory");
    }
}

template <int MMA_N, bool PUSH>
__global__ void __launch_bounds__(NT, 1) batch_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA,
                                                      const __grid_constant__ Params p) {
    using CF = Cfg<MMA_N>;
    constexpr int RING = CF::RING, RH = MMA_N / 2;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    uint8_t* img = sm + RING * CF::STAGE;                    // [NIMG] images
    uint8_t* zop = img + NIMG * IMG;                         // [NIMG] z operands
    Ctrl* ctrl = reinterpret_cast<Ctrl*>(zop + NIMG * CF::ZB);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int cta = blockIdx.x;
    const int T = p.ntile * p.nkt;
    const int u0 = cta < p.G ? sched_first_unit(cta, T, p.G) : 0, u1 = cta < p.G ? sched_first_unit(cta + 1, T, p.G) : 0;
    const int nunits = u1 - u0;
    const int head = SegWalk(u0, u1, p.nkt).head, nhead = u1 - head;      // units [head, u1) go first, then [u0, head)

    if (tid == 0) {
#pragma unroll 1
        for (int s = 0; s < RING; ++s) {
            mbar_init(smem_u32(&ctrl->full[s]), 2);
            mbar_init(smem_u32(&ctrl->empty[s]), 1);
            mbar_init(smem_u32(&ctrl->sf[s]), 4);
        }
#pragma unroll 1
        for (int b = 0; b < 2; ++b) { mbar_init(smem_u32(&ctrl->acc_full[b]), 1); mbar_init(smem_u32(&ctrl->acc_empty[b]), EPI_WARPS); }
#pragma unroll 1
        for (int b = 0; b < NIMG; ++b) mbar_init(smem_u32(&ctrl->lr_free[b]), 1);
        mbar_init(smem_u32(&ctrl->lr_done), 1);
        ctrl->abort = 0;
        fence_mbar_init();
        prefetch_tmap(&tmW);
        prefetch_tmap(&tmA);
    }
    if (warp == MMA_WARP) { tmem_alloc(smem_u32(&ctrl->tmem_base), TMEM_COLS); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    griddep_launch_dependents();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
    auto unit_at = [&](int i) { return i < nhead ? head + i : u0 + (i - nhead); };      // i-th unit in processing order

    if (warp == W_WARP) {
        // ================= weight copies (static: the first ring before the dependency wait) =================
        if (lane == 0) {
            int s = 0;
            uint32_t par = 1u;
#pragma unroll 1
            for (int i = 0; i < nunits; ++i) {
                if (i >= RING && !wait(smem_u32(&ctrl->empty[s]), par, ctrl, p, ST_EMPTY, warp)) break;
                const uint32_t st = base + s * CF::STAGE, bar = smem_u32(&ctrl->full[s]);
                const int u = unit_at(i);
                mbar_arrive_expect_tx(bar, W_TILE_BYTES + SF_TILE_BYTES);
                if (p.W_tiled) {
                    bulk_load(st, p.W_tiled + (size_t)u * (W_TILE_BYTES + SF_TILE_BYTES), W_TILE_BYTES + SF_TILE_BYTES, bar);
                } else {
                    const int t = (int)((unsigned)u / (unsigned)p.nkt), kt = u - t * p.nkt;
                    tma_load_2d(st, &tmW, kt * KT_BYTES, t * TILE_N, bar);
                    bulk_load(st + W_TILE_BYTES, p.W_sf + ((size_t)t * (p.K >> 6) + (size_t)kt * 4) * 512, SF_TILE_BYTES, bar);
                }
                if (++s == RING) { s = 0; par ^= 1u; }
            }
        }
        __syncwarp();
        griddep_wait();
    } else if (warp == A_WARP) {
        // ================= activation copies =================
        griddep_wait();
        if (lane == 0) {
            fence_proxy_async_global();          // the activation was written by ordinary stores of the previous kernel
            int s = 0;
            uint32_t par = 1u;
#pragma unroll 1
            for (int i = 0; i < nunits; ++i) {
                if (i >= RING && !wait(smem_u32(&ctrl->empty[s]), par, ctrl, p, ST_EMPTY, warp)) break;
                const uint32_t st = base + s * CF::STAGE + W_TILE_BYTES + SF_TILE_BYTES, bar = smem_u32(&ctrl->full[s]);
                const int kt = (int)((unsigned)unit_at(i) % (unsigned)p.nkt);
                mbar_arrive_expect_tx(bar, CF::A_TILE + SF_TILE_BYTES);
                if (p.A_rec) {
                    bulk_load(st, p.A_rec + (size_t)kt * (CF::A_TILE + SF_TILE_BYTES), CF::A_TILE + SF_TILE_BYTES, bar);
                } else {
                    tma_load_2d(st, &tmA, kt * KT_BYTES, 0, bar);
                    bulk_load(st + CF::A_TILE, p.A_sf + (size_t)kt * 4 * 512, SF_TILE_BYTES, bar);
                }
                if (++s == RING) { s = 0; par ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        // ================= GEMM MMAs =================
        constexpr uint32_t idesc = make_idesc_nvf4(TILE_N, MMA_N);
        int s = 0, seg = 0;
        uint32_t par = 0u;
        bool ok = true, ready = false;
#pragma unroll 1
        for (SegWalk sw(u0, u1, p.nkt); ok && !sw.done(); sw.next(), ++seg) {
            const int cnt = sw.count(), buf = seg & 1;
            if (seg >= 2 && !warp_wait(smem_u32(&ctrl->acc_empty[buf]), ((seg >> 1) - 1) & 1, ctrl, p, ST_ACC_EMPTY, warp)) break;
#pragma unroll 1
            for (int j = 0; j < cnt; ++j) {
                if (!ready && !(ok = warp_wait(smem_u32(&ctrl->sf[s]), par, ctrl, p, ST_SF_FULL, warp))) break;
                const int sn = s + 1 == RING ? 0 : s + 1;
                const uint32_t pn = sn == 0 ? par ^ 1u : par;
                ready = __all_sync(0xffffffffu, mbar_test_wait(smem_u32(&ctrl->sf[sn]), pn));
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint32_t st = base + s * CF::STAGE, sf = tmem + SF_COL + 32 * s;
                    const uint64_t wd = make_smem_desc(st, 1024, 2), ad = make_smem_desc(st + W_TILE_BYTES + SF_TILE_BYTES, 1024, 2);
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc_mma_nvf4(tmem + 32 * buf, wd + 2 * k, ad + 2 * k, idesc, sf + 4 * k, sf + 16 + 4 * k, (j > 0 || k > 0) ? 1u : 0u);
                    tc_commit(smem_u32(&ctrl->empty[s]));
                    if (j == cnt - 1) tc_commit(smem_u32(&ctrl->acc_full[buf]));
                }
                __syncwarp();
                s = sn;
                par = pn;
            }
        }
    } else if (warp >= SF_WARP0) {
        // ================= scale factors -> TMEM: group g takes units g, g + 2, ... =================
        const int g = (warp - SF_WARP0) >> 2;
        const uint32_t quad = (uint32_t)((warp & 3) * 32) << 16;
        int s = g;
        uint32_t par = 0u;
#pragma unroll 1
        for (int i = g; i < nunits; i += 2) {
            // (the slot's previous unit may have been the other group's: its MMAs first, or the parity could be the last lap's)
            if (i >= RING && !warp_wait(smem_u32(&ctrl->empty[s]), par ^ 1u, ctrl, p, ST_SF_EMPTY, warp)) break;
            if (!warp_wait(smem_u32(&ctrl->full[s]), par, ctrl, p, ST_FULL, warp)) break;
            tc_fence_after_sync();
            const uint8_t* st = sm + s * CF::STAGE;
            const uint4* fa = reinterpret_cast<const uint4*>(st + W_TILE_BYTES) + lane;
            const uint4* fb = reinterpret_cast<const uint4*>(st + W_TILE_BYTES + SF_TILE_BYTES + CF::A_TILE) + lane;
            uint32_t ra[16], rb[16];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const uint4 x = fa[a * 32], y = fb[a * 32];
                ra[4 * a] = x.x; ra[4 * a + 1] = x.y; ra[4 * a + 2] = x.z; ra[4 * a + 3] = x.w;
                rb[4 * a] = y.x; rb[4 * a + 1] = y.y; rb[4 * a + 2] = y.z; rb[4 * a + 3] = y.w;
            }
            const uint32_t set = tmem + quad + SF_COL + 32 * s;
            tmem_st_x16(set, ra);
            tmem_st_x16(set + 16, rb);
            tc_wait_st();
            tc_fence_before_sync();
            warp_arrive(smem_u32(&ctrl->sf[s]), lane);
            s += 2;
            if (s >= RING) { s -= RING; par ^= 1u; }
        }
    } else {
        // ================= z, expansion, epilogue (256 threads) =================
        const int r128 = tid & 127, half = tid >> 7;
        const uint32_t quad = (uint32_t)((warp & 3) * 32) << 16;
        const int kbytes = p.K >> 3, nch = p.K >> 6;
        constexpr uint32_t id_z = make_idesc_bf16(TILE_N, MMA_N < 16 ? 16 : MMA_N), id_lr = make_idesc_bf16(TILE_N, CF::LR_N);
        // (A wait or poll that gives up sets the abort flag, which makes the later ones return at once; nobody leaves early, so that the
        // barriers below always have their 256 threads.)
        uint32_t dpar = 0u, fpar = 0u;           // parity of lr_done's next completion; bit b: of lr_free[b]'s
        // image of chunk c of the V bits of rank block rb: thread = (rank, half of the chunk)
        auto v_image = [&](int rb, int c, int b) {
            const int rank = rb * 128 + r128;
            if (rank < p.R) image_half(img + b * IMG, r128, half, *reinterpret_cast<const uint32_t*>(p.Vp + (size_t)rank * kbytes + c * 8 + half * 4));
            else {
                uint8_t* row = img + b * IMG + (r128 >> 3) * 1024 + (r128 & 7) * 128;
#pragma unroll
                for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(row + (((4 * half + i) ^ (r128 & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
            }
        };
        if (p.R > 0 && cta < p.nitems) {         // the first round's images: static data
            const int rb = cta / p.nks, ks = cta - rb * p.nks;
            const int c0 = ks * nch / p.nks, c1 = (ks + 1) * nch / p.nks;
#pragma unroll 1
            for (int i = 0; i < NIMG && c0 + i < c1; ++i) v_image(rb, c0 + i, i);
        }
        if constexpr (MMA_N == 8) {              // (z's operand has sixteen rows: the upper eight stay zero)
#pragma unroll 1
            for (int i = tid; i < NIMG * 64; i += EPI_THREADS)
                *reinterpret_cast<uint4*>(zop + (i >> 6) * CF::ZB + 1024 + (i & 63) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        griddep_wait();                          // everything below reads what earlier kernels of the stream wrote
        if (tid == 0) {
            unsigned long long n = 0ull;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint4 a = ld_volatile_v4(reinterpret_cast<const uint4*>(p.count) + i);
                n += (((unsigned long long)a.y << 32) | a.x) + (((unsigned long long)a.w << 32) | a.z);
            }
            ctrl->seq = (uint32_t)(n >> 20);
            if (PUSH) ctrl->ar_seq = (ld_volatile_u32(p.ar_counter) >> 20) + 1u;
        }
        const SumWords<MMA_N> words(p.M);
        uint32_t tag = 0u, phase = 0u;          // this launch's number on this scratch (from one), its parity
        // ---- z: partial sums of this CTA's items ----
#pragma unroll 1
        for (int item = cta; p.R > 0 && item < p.nitems; item += gridDim.x) {
            const int rb = item / p.nks, ks = item - rb * p.nks;
            const int c0 = ks * nch / p.nks, c1 = (ks + 1) * nch / p.nks;
#pragma unroll 1
            for (int r0 = c0; r0 < c1; r0 += NIMG) {
                const int nr = c1 - r0 < NIMG ? c1 - r0 : NIMG;
                uint4 xv[NIMG];                  // the round's pieces of X: all requested before any is used
                const int m = tid >> 3, pc = tid & 7;
#pragma unroll
                for (int i = 0; i < NIMG; ++i) {
                    xv[i] = make_uint4(0u, 0u, 0u, 0u);
                    if (i < nr && m < p.M) xv[i] = *reinterpret_cast<const uint4*>(p.X + (size_t)m * p.K + (r0 + i) * 64 + pc * 8);
                }
                if (r0 > c0 || item != cta) {    // (the previous round's MMAs have completed: it waited for them below)
#pragma unroll 1
                    for (int i = 0; i < nr; ++i) v_image(rb, r0 + i, i);
                }
                if (tid < MMA_N * 8) {
#pragma unroll
                    for (int i = 0; i < NIMG; ++i)
                        if (i < nr) *reinterpret_cast<uint4*>(zop + i * CF::ZB + (m >> 3) * 1024 + (m & 7) * 128 + ((pc ^ (m & 7)) << 4)) = xv[i];
                }
                fence_proxy_async();
                epi_sync();
                if (warp == 0 && elect_one()) {
                    tc_fence_after_sync();
#pragma unroll 1
                    for (int i = 0; i < nr; ++i) {
                        const uint64_t ad = make_smem_desc(smem_u32(img + i * IMG), 1024, 2), bd = make_smem_desc(smem_u32(zop + i * CF::ZB), 1024, 2);
#pragma unroll
                        for (int k = 0; k < 4; ++k) tc_mma_bf16(tmem + LR_COL, ad + 2 * k, bd + 2 * k, id_z, (r0 + i > c0 || k > 0) ? 1u : 0u);
                    }
                    tc_commit(smem_u32(&ctrl->lr_done));
                }
                __syncwarp();
                warp_wait(smem_u32(&ctrl->lr_done), dpar, ctrl, p, ST_Z, 1);
                dpar ^= 1u;
            }
            tag = ctrl->seq + 1u;                // (written before the first round's barrier)
            phase = p.z_cleared ? 1u : tag & 1u;
            tc_fence_after_sync();
            float d[CF::VR];
            ld_rows<MMA_N>(tmem + quad + LR_COL, half, d);
            tc_fence_before_sync();
            if (cta != p.skip_publish) SumWords<MMA_N>::put(p.zpart + (size_t)item * CF::SW * 128 + r128, d, half, p.M, tag);
            epi_sync();                          // (the accumulator has been read; the next item may start)
        }
        if (p.R == 0 || cta >= p.nitems) { epi_sync(); tag = ctrl->seq + 1u; phase = p.z_cleared ? 1u : tag & 1u; }
        // ---- z: this CTA's share of the outputs of its items' rank blocks, over the slices in order ----
#pragma unroll 1
        for (int item = cta; p.R > 0 && item < p.nitems; item += gridDim.x) {
            const int rb = item / p.nks, ks = item - rb * p.nks;
            const int E = words.live * 128, e0 = ks * E / p.nks, e1 = (ks + 1) * E / p.nks;
#pragma unroll 1
            for (int e = e0 + tid; e < e1; e += EPI_THREADS) {
                const int w = words.word(e >> 7), r = e & 127, rank = rb * 128 + r, m = words.row(w), nm = words.rows(w, p.M);
                const float coef = rank < p.R ? __bfloat162float(p.S[rank]) : 0.f;
                float t[3];
                words.add(p.zpart + ((size_t)rb * p.nks * CF::SW + w) * 128 + r, p.nks, CF::SW * 128, 0, tag, t, ctrl, p, ST_Z);
                if (rank < p.R) {                // (also after a wait that gave up: every mark has to be this launch's, or the next launch could take an older z for its own)
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        if (i < nm) p.zbuf[(size_t)(m + i) * p.Rpad + rank] = mark(__fmul_rn(t[i], coef), phase);
                }
            }
        }

        // ---- segments: expansion, accumulator, output or partial sum ----
        int seg = 0, ib = 0;                     // ib: images used so far (image ib % NIMG is next)
        int ptile[2], pslot[2], pnc[2], pcf[2], np = 0;      // partial segments of this CTA (its first and last at most)
        uint32_t used = 0u;                      // bit b: image b has been read by expansion MMAs before
#pragma unroll 1
        for (SegWalk sw(u0, u1, p.nkt); !sw.done(); sw.next(), ++seg) {
            const int t = (int)((unsigned)sw.first() / (unsigned)p.nkt), cnt = sw.count(), buf = seg & 1;
            const int cf = sched_cta_of_unit(t * p.nkt, T, p.G), nc = sched_cta_of_unit(t * p.nkt + p.nkt - 1, T, p.G) - cf + 1, slot = cta - cf;
            const int n = t * TILE_N + r128;
            const int grp = (t >= p.gtile[0] ? 1 : 0) + (t >= p.gtile[1] ? 1 : 0) + (t >= p.gtile[2] ? 1 : 0);
            const float alpha = p.alpha[grp];
            const float* zb = p.zbuf + grp * p.Rg;
            const int w0 = slot * p.Rw / nc, w1 = (slot + 1) * p.Rw / nc;      // every contributor expands its share of the rank words
            const uint32_t d2 = tmem + LR_COL + 64 * buf;
            const bool lr = p.R > 0 && w0 < w1;
            if (lr) {
                const int32_t* ucol = p.Ucol + (size_t)(n < p.N ? n : 0) * p.Rw;
                const int nck = (w1 - w0 + 1) >> 1;                            // chunks of 64 ranks (the last may be half)
#pragma unroll 1
                for (int cb = 0; cb < nck; cb += NIMG) {
                    const int nr = nck - cb < NIMG ? nck - cb : NIMG;
                    // sign images: thread = (column, rank word of the chunk); words requested together
                    uint32_t uw[NIMG];
#pragma unroll
                    for (int i = 0; i < NIMG; ++i) {
                        const int w = w0 + 2 * (cb + i) + half;
                        uw[i] = (i < nr && w < w1) ? (uint32_t)ucol[w] : 0u;   // (a missing word meets z = 0)
                    }
#pragma unroll
                    for (int i = 0; i < NIMG; ++i) {
                        const int b = (ib + i) & (NIMG - 1);
                        if (i < nr) {
                            if ((used >> b) & 1u) { warp_wait(smem_u32(&ctrl->lr_free[b]), (fpar >> b) & 1u, ctrl, p, ST_ACC_EMPTY, 1); fpar ^= 1u << b; }
                            used |= 1u << b;
                            image_half(img + b * IMG, r128, half, uw[i]);
                        }
                    }
                    // z pieces: thread = (row, 8 ranks of a chunk), the chunks of a batch over the groups of MMA_N * 8 threads there are (four at 8
                    // rows: splitting z into three parts by one group after another was 20 us of 600 in the decode step of eight sequences);
                    // polled until every value carries this launch's mark
                    constexpr int ZT = MMA_N * 8 < EPI_THREADS ? MMA_N * 8 : EPI_THREADS;
                    const int m = (tid & (ZT - 1)) >> 3, pc = tid & 7;
#pragma unroll 1
                    for (int i = tid / ZT; i < nr; i += EPI_THREADS / ZT) {
                        const int b = (ib + i) & (NIMG - 1), w = w0 + 2 * (cb + i) + (pc >> 2), e0 = 32 * (w0 + 2 * (cb + i)) + 8 * pc;
                        uint32_t part[CF::PARTS][4];
#pragma unroll
                        for (int k = 0; k < CF::PARTS; ++k) part[k][0] = part[k][1] = part[k][2] = part[k][3] = 0u;
                        if (m < p.M && w < w1 && e0 < p.Rg) {
                            const float* src = zb + (size_t)m * p.Rpad + e0;
                            uint32_t v[8];
                            Poll poll;
#pragma unroll 1
                            while (true) {
                                const uint4 a = ld_volatile_v4(src), c = ld_volatile_v4(src + 4);
                                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
                                uint32_t bad = 0u;
#pragma unroll
                                for (int q = 0; q < 8; ++q) bad |= (e0 + q < p.Rg) ? (v[q] ^ phase) : 0u;
                                if (!(bad & 1u)) break;
                                if (poll.expired(ctrl, p, ST_Z)) break;
                            }
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                float z0 = e0 + 2 * q < p.Rg ? unmark(v[2 * q]) : 0.f, z1 = e0 + 2 * q + 1 < p.Rg ? unmark(v[2 * q + 1]) : 0.f;
#pragma unroll
                                for (int k = 0; k < CF::PARTS; ++k) part[k][q] = next_part<CF::PARTS>(z0, z1);
                            }
                        }
                        uint8_t* o = zop + b * CF::ZB + (m >> 3) * 1024 + (m & 7) * 128 + ((pc ^ (m & 7)) << 4);
#pragma unroll
                        for (int k = 0; k < CF::PARTS; ++k)
                            *reinterpret_cast<uint4*>(o + k * MMA_N * 128) = make_uint4(part[k][0], part[k][1], part[k][2], part[k][3]);
                    }
                    fence_proxy_async();
                    epi_sync();
                    if (warp == 0 && elect_one()) {
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int i = 0; i < nr; ++i) {
                            const int b = (ib + i) & (NIMG - 1);
                            const uint64_t ad = make_smem_desc(smem_u32(img + b * IMG), 1024, 2), bd = make_smem_desc(smem_u32(zop + b * CF::ZB), 1024, 2);
#pragma unroll
                            for (int k = 0; k < 4; ++k) tc_mma_bf16(d2, ad + 2 * k, bd + 2 * k, id_lr, (cb + i > 0 || k > 0) ? 1u : 0u);
                            tc_commit(smem_u32(&ctrl->lr_free[b]));
                        }
                        if (cb + nr == nck) tc_commit(smem_u32(&ctrl->lr_done));
                    }
                    __syncwarp();
                    ib += nr;
                }
            }
            warp_wait(smem_u32(&ctrl->acc_full[buf]), (seg >> 1) & 1, ctrl, p, ST_ACC_FULL, warp);
            if (lr) {
                warp_wait(smem_u32(&ctrl->lr_done), dpar, ctrl, p, ST_ACC_FULL, warp);
                dpar ^= 1u;
            }
            epi_sync();
            tc_fence_after_sync();
            float v[CF::VR];
            ld_rows<MMA_N>(tmem + quad + 32 * buf, half, v);
#pragma unroll
            for (int i = 0; i < CF::VR; ++i) v[i] *= alpha;
            if (lr) {
                float a[CF::VR], b[CF::VR];      // the smaller parts first
                ld_rows<MMA_N>(d2 + quad + (CF::PARTS - 1) * MMA_N, half, a);
#pragma unroll
                for (int k = CF::PARTS - 2; k >= 0; --k) {
                    ld_rows<MMA_N>(d2 + quad + k * MMA_N, half, b);
#pragma unroll
                    for (int i = 0; i < CF::VR; ++i) a[i] += b[i];
                }
#pragma unroll
                for (int i = 0; i < CF::VR; ++i) v[i] += a[i];
            }
            tc_fence_before_sync();
            warp_arrive(smem_u32(&ctrl->acc_empty[buf]), lane);
            if (cnt == p.nkt) {
                if (n < p.N && !ctrl->abort) {
#pragma unroll
                    for (int i = 0; i < RH; ++i)
                        if (half * RH + i < p.M) put<PUSH>(p, ctrl, half * RH + i, n, MMA_N == 8 && half ? v[CF::VR - RH + i] : v[i]);
                }
            } else {
                SumWords<MMA_N>::put(p.part + (size_t)(part_base(t, cf, p.ntile, p.G) + cta) * CF::SW * 128 + r128, v, half, p.M, tag);
                if (np == 0) { ptile[0] = t; pslot[0] = slot; pnc[0] = nc; pcf[0] = cf; } else { ptile[1] = t; pslot[1] = slot; pnc[1] = nc; pcf[1] = cf; }
                ++np;
            }
        }
        // ---- this CTA's words of the tiles it shares ----
#pragma unroll 1
        for (int q = 0; q < np; ++q) {
            const int t = q == 0 ? ptile[0] : ptile[1], slot = q == 0 ? pslot[0] : pslot[1], nc = q == 0 ? pnc[0] : pnc[1], cf = q == 0 ? pcf[0] : pcf[1];
            const int n = t * TILE_N + r128;
            const uint4* src = p.part + (size_t)(part_base(t, cf, p.ntile, p.G) + cf) * CF::SW * 128 + r128;
#pragma unroll 1
            for (int i = slot * words.live / nc + half; i < (slot + 1) * words.live / nc; i += 2) {
                const int w = words.word(i), m = words.row(w), nm = words.rows(w, p.M);
                float o[3];
                words.add(src + w * 128, nc, CF::SW * 128, nc - 1, tag, o, ctrl, p, ST_TILE);      // (the tile's last contributor first, as the tile kernel's finisher adds)
                if (n < p.N && !ctrl->abort) {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (k < nm) put<PUSH>(p, ctrl, m + k, n, o[k]);
                }
            }
        }
    }

    // ---------------- common exit ----------------
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (ctrl->abort) {      // give copies that may still be in flight time to land before the shared memory is released
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) { }
    }
    if (tid == 0) {         // this CTA's share of 2^20
        const uint32_t share = (uint32_t)((((unsigned long long)(cta + 1)) << 20) / gridDim.x) - (uint32_t)((((unsigned long long)cta) << 20) / gridDim.x);
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p.count + (cta & 7)), "l"((unsigned long long)share) : "memory");
    }
    if (warp == MMA_WARP) { tc_fence_after_sync(); tmem_dealloc(tmem, TMEM_COLS); }
}

}  // namespace batch
}  // namespace biloco
