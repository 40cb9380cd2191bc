// Linear layers over the packed rows of a step on the 5th-generation tensor cores (sm_100a): TMA -> shared memory -> tcgen05.mma ->
// TMEM -> epilogue.  Stands in for the reference's dequant-to-scratch + cuBLAS GEMM + epilogue pass (rwkv_dequant_int8, cublasGemmEx,
// rwkv_gemm_epilogue; src/backend_cuda.rs:4195-4227, 1254-1368, 4613-4633) and its register-tiled batched GEMVs (gemv_variant_mb,
// gemv_int8_rkv_stage1_batch; :3381-3554, :1665-1910).
//
// Arithmetic.  Weights are never converted: the u8 codes q are the A operand of tcgen05.mma.kind::i8 as they sit in HBM, the
// activation row is four columns of signed base-128 digits of its fixed-point value t (operands.cuh).  The tensor core returns exact
// int32 sums; Q = sum_j 128^(3-j) I_j = sum_k q_k t_k, y = e 2^-27 (s Q + z sum_k t_k): no rounding but the one of t and the one of y, so
// no dependence on how K is split or on the other rows.  (Sums of more than 53 bits pass through fp64 in some kernels, which can turn a tie of the last rounding.)  Files with one (scale, zero) per group of 128 weights (the reference's own) get a fresh accumulator per K block of
// 128 bytes = one group: the epilogue warps fold s_g Q_g + z_g T_g into fp32 registers while the next group is multiplied.  fp16
// weights use kind::f16 with hi + lo halves of the activations.
//
// Work split.  One CTA = one tile of 128 weight rows x up to 64 activation rows x one slice of K; the slices of a tile are a cluster
// of 1, 2, 4 or 8 CTAs that exchange partial sums through distributed shared memory (each CTA finishes its share of the activation
// rows), so that a layer with few tiles still has every SM streaming and no partial sum goes through global memory (the kernel this
// one replaces cut tiles between persistent CTAs and paid a global round trip, an atomic and a serial sum per cut tile).  A CTA takes
// at most half an SM (<= 113 KB shared memory, <= 256 TMEM columns): two are resident, one loads while the other finishes, and the
// next kernel of the step becomes resident early and requests its weights before the dependency wait.  (The exception: split tiles of
// more than 108 rows of fp16 weights, whose partial sums take up to 128 KB; one of them is resident.)
// All problems of a launch are cut alike.  (fp16 rank projections next to int8 matrices were cut in two at most: twenty K blocks through a ring of
// five were the longest chain of the launch with r, k and v; 3 rows, 2560 channels, 32 layers: a step of 1.74 ms, now 1.67.)
// What bounds it: at few rows the chain operand tiles (L2) -> products -> exchange -> store behind the dependency wait, the weights
// are there already; at 64 rows the operand tiles' L2 traffic as well (a 128-row tile re-reads them all).
// In cycles after the wait (3 rows, att.output and ffn.value split in 4 and 8): operand tiles and products 3800 and 5400, two cluster barriers and the partial sums
// between them 2150 and 2500, their addition and the outputs 1500 and 1800; 64 rows, ffn.key split in two: 12000, 5900 and 6000.  Tried without gain: partial
// sums counted by an mbarrier of their receiver instead of the barriers (3 rows 47.0 -> 49.8 us a layer), the epilogue run once on nothing before the wait.
//
// Code size is part of the design.  The kernels of a layer run for a few microseconds each, in turn, on every SM; 32 KB of code run at
// an instruction per cycle, up to 128 KB at a third of that, more at less than a fifth (measured with straight-line kernels), and a
// branch to a line that is not there waits for the L2.  A version of this kernel with its epilogue specialised at compile time and
// unrolled took 150 to 345 KB and 0.5 us for thirty instructions; hence one epilogue, loops that stay loops, and one function per
// activation.
//
// Roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer (+ TMEM owner), warps 2-9 operand construction and epilogue (two per
// TMEM lane quarter).  Every mbarrier wait is bounded; on expiry bit 1 of the status word is raised and the roles drain.
#pragma once
#include <cuda.h>

#include "operands.cuh"
#include "tc_ptx.cuh"

namespace rsv {

constexpr int kRlThreads = 320;
constexpr int kRlEpiWarps = 8;
constexpr int kRlEpiThreads = 32 * kRlEpiWarps;
constexpr int rl_persistent_threads(int epi_warps) { return 64 + 32 * epi_warps; }
constexpr int kRlTileM = 128;
constexpr int kRlABytes = kRlTileM * 128;
constexpr int kRlMaxProb = 8;
constexpr int kRlMaxStages = 8;
constexpr int kRlMaxSplit = 8;

struct RlProb {
    const uint8_t* bimg;    // operand image; null: built in the kernel from x
    const float* xscale;    // [R]
    const long long* tsum;  // [R][tparts] sums over parts of a row
    const float* tgrp;      // [R][kblocks]
    const float *wscale, *wzero;  // RL_I8: [M]
    const uint32_t* szt;          // RL_I8G: [kblocks][M] fp16 scale | fp16 zero << 16
    const float* x;  // BUILD: activations [R, ldx]
    float *y, *y2;
    const float* bias;
    float* ymax;  // optional: [R][M tiles] maxima of |y| over the tile's outputs (EPI_RELU2 only)
    int ldx, ldy, epi, fmt, M, K, kblocks, job0, tparts;
};
struct alignas(64) RlLaunch {
    CUtensorMap amap[kRlMaxProb];
    RlProb p[kRlMaxProb];
    int nprob, R, rt, n_tiles, split, log_split, nt8, nt16, nt_max, ring, tmem_cols;  // ring: bytes of shared memory for stages
    int* status;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, unsigned long long v) { asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <int THREADS = kRlEpiThreads>
__device__ __forceinline__ void rl_epi_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}

// Four outputs at a time (independent chains), one piece of code for all epilogues (bias is 0 where there is none).
__device__ __forceinline__ void rl_activate4(int epi, float (&a)[4], float bias) {
    if (epi == EPI_STORE) return;
    if (epi == EPI_RELU2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = fmaxf(a[i], 0.f);
            a[i] = t * t;
        }
    } else if (epi == EPI_TANH) {
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = tanhf(a[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = sigmoidf_(a[i] + bias);
        if (epi == EPI_DECAY)
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = expf(a[i] * kDecayScale);
    }
}
// Lane i < 4: the warp's maximum of |a[i]| (a NaN counts as 0).
__device__ __forceinline__ float rl_rowmax4(const float (&a)[4], bool mine, int lane) {
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t t = __reduce_max_sync(0xffffffffu, mine ? __float_as_uint(fmaxf(fabsf(a[i]), 0.f)) : 0u);
        if (lane == i) mx = t;
    }
    return __uint_as_float(mx);
}
// exact integer (|q| < 2^51) -> double without the slow 64-bit conversion
__device__ __forceinline__ double rl_ll2d(long long q) { return __longlong_as_double(0x4338000000000000LL + q) - 6755399441055744.0; }
// Per-group weights: columns between the two accumulators (read 32 at a time), and floats between the blocks' activation sums in shared memory.
__host__ __device__ constexpr int rl_group_cols(int nt) { return (nt + 31) / 32 * 32; }
__host__ __device__ constexpr int rl_group_rows(int rt) { return (rt + 3) / 4 * 4; }
// A digit's sum over a group, |i| <= 2^21, as fp32 (the conversion instruction runs at an eighth of this)
__device__ __forceinline__ float rl_small2f(uint32_t i) { return __uint_as_float(0x4B400000u + i) - 12582912.0f; }
// An int8 output from the exact sum Q = sum_k q_k t_k and the row's T = sum_k t_k: xs (ws Q + wz T), xs a power of two, rounded to fp32 once.  The scales are fp16
// numbers: with ws = ms unit and wz = mz unit in whole numbers (ms < 2^11, |mz| < 2^19, the unit a power of two with the sign of ws) ms Q + mz T is an
// integer, under 2^63 for K < 2^16, which the conversion to fp32 rounds (`whole`).  That covers zero points of one to 256 steps of the codes, and none.  fp64 takes the
// others; it holds sums of up to 53 bits.
// In fp64 the arithmetic holds the tensor pipe up.  512 rows of 2560 -> 10240, us: files symmetric around code 128 42.0 and as integers 41.0 (as two fp32 halves, which lost
// the last bit of some sums and more of small negative ones, 40.8), zero points of 96 steps 47.5 and 41.0; 1024 rows of those 84.2 and 72.2.
struct RlScale {
    float ws, wz, unit;
    uint32_t ms;
    int mz;
    bool whole;
};
__device__ __forceinline__ RlScale rl_scale(float ws, float wz) {
    const uint32_t bs = __float_as_uint(ws), bz = __float_as_uint(wz), e = (bs >> 23) & 0xFFu;
    const uint32_t ms = ws == 0.f ? 0u : ((bs & 0x7FFFFFu) | 0x800000u) >> 13, mz = wz == 0.f ? 0u : ((bz & 0x7FFFFFu) | 0x800000u) >> 13;
    const int up = mz ? (int)((bz >> 23) & 0xFFu) - (int)e : 0;
    RlScale w;
    w.ws = ws;
    w.wz = wz;
    w.ms = ms;
    w.whole = (ms | mz) == 0u || (e > 10u && e < 255u && up >= 0 && up <= 8 && !((bs | bz) & 0x1FFFu));
    w.unit = __uint_as_float((bs & 0x80000000u) | (w.whole && ms ? (e - 10u) << 23 : 0u));
    w.mz = w.whole ? (int)(mz << up) : 0;
    if ((int)(bs ^ bz) < 0) w.mz = -w.mz;
    return w;
}
struct RlSum8 {  // of a row of activations: T, and as fp64
    long long t;
    double td;
};
__device__ __forceinline__ float rl_value8(const RlScale& w, float xs, long long q, const RlSum8& row) {
    return xs * (w.whole ? w.unit * (float)(q * (long long)w.ms + row.t * w.mz) : (float)((double)w.ws * rl_ll2d(q) + (double)w.wz * row.td));
}
__device__ __forceinline__ long long rl_digits2q(int i0, int i1, int i2, int i3) {
    return ((long long)i0 * 128 + i1) * 16384 + ((long long)i2 * 128 + i3);
}

// Where a tile's outputs go: row rl of the tile to y + rl ldy (and y2), nr rows.
struct RlOut {
    float *y, *y2;
    size_t ldy;
    int nr, epi;
    float bias;
    bool maxima;
};
__device__ __forceinline__ RlOut rl_out(const RlProb& P, int r0, int nr, int m, float bias) {
    RlOut o;
    o.ldy = (size_t)P.ldy;
    o.y = P.y + (size_t)r0 * P.ldy + m;
    o.y2 = P.y2 ? P.y2 + (size_t)r0 * P.ldy + m : nullptr;
    o.nr = nr;
    o.epi = P.epi;
    o.bias = bias;
    o.maxima = P.ymax != nullptr;
    return o;
}
// The sums of a tile whose K was not split, from tensor memory through the thread's registers to the output, rows rl .. rl + 3 at a time
// (`turn`: the WARPS / 4 warps of a lane quarter take turns).  What bounds this is the latency of its instructions: a warp issues one in eight cycles.
template <int WARPS>
__device__ __forceinline__ void rl_finish(const RlOut& o, bool f16, uint32_t taddr, const float* s_xs, const RlSum8* s_t, float* s_ymax, const RlScale& w, bool mok,
                                          int turn, int lane) {
#pragma unroll 1
    for (int rl = 4 * turn; rl < o.nr; rl += WARPS) {
        float a[4];
        __syncwarp();  // (the loads below want the whole warp, whose lanes may take either form of rl_value8)
        if (f16) {
            uint32_t v[8];
            tmem_ld8(taddr + 2 * rl, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = s_xs[rl + i] * (__uint_as_float(v[2 * i]) + __uint_as_float(v[2 * i + 1]));
        } else {
            uint32_t v[16];
            tmem_ld16(taddr + 4 * rl, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = rl_value8(w, s_xs[rl + i], rl_digits2q((int)v[4 * i], (int)v[4 * i + 1], (int)v[4 * i + 2], (int)v[4 * i + 3]), s_t[rl + i]);
        }
        rl_activate4(o.epi, a, o.bias);
        const int left = o.nr - rl;
        float* p = o.y + (size_t)rl * o.ldy;
        if (mok) {
            p[0] = a[0];
            if (left > 1) p[o.ldy] = a[1];
            if (left > 2) p[2 * o.ldy] = a[2];
            if (left > 3) p[3 * o.ldy] = a[3];
        }
        if (o.y2 && mok) {
            p = o.y2 + (size_t)rl * o.ldy;
            p[0] = a[0];
            if (left > 1) p[o.ldy] = a[1];
            if (left > 2) p[2 * o.ldy] = a[2];
            if (left > 3) p[3 * o.ldy] = a[3];
        }
        if (o.maxima) {
            const float mx = rl_rowmax4(a, mok, lane);
            if (lane < 4) s_ymax[rl + lane] = mx;  // (rows past the end have slots of their own)
        }
    }
}

// The products of one tile: K block after K block through the ring (position s, parity par) into the accumulator at d.
template <bool I8>
__device__ __forceinline__ bool rl_mma_tile(uint64_t* full, uint64_t* empty, uint32_t& s, uint32_t& par, uint32_t NS, int nk, uint32_t smem_addr, uint32_t stage_bytes, uint32_t d,
                                            uint32_t idesc, volatile int* abort_flag) {
#pragma unroll 1
    for (int kb = 0; kb < nk; ++kb) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], par, abort_flag))) return false;
        tc_fence_after();
        const uint32_t a_addr = smem_addr + s * stage_bytes;
        const uint64_t adesc = tc_smem_desc(a_addr), bdesc = tc_smem_desc(a_addr + kRlABytes);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) tc_mma_elect<I8>(d, adesc + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), idesc, (kb == 0 && k4 == 0) ? 0u : 1u);
        tc_commit_elect(&empty[s]);
        if (++s == NS) {
            s = 0;
            par ^= 1u;
        }
    }
    return true;
}
// The same for per-group weights: block j into accumulator j mod 2 (acc_cols apart), handed to the epilogue warps block by block.
__device__ __forceinline__ bool rl_mma_groups(uint64_t* full, uint64_t* empty, uint64_t* acc_full, uint64_t* acc_empty, uint32_t NS, int nk, uint32_t smem_addr, uint32_t stage_bytes, uint32_t tmem,
                                              uint32_t acc_cols, uint32_t idesc, volatile int* abort_flag) {
    uint32_t s = 0, par = 0;
#pragma unroll 1
    for (int j = 0; j < nk; ++j) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s], par, abort_flag))) return false;
        if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[j & 1], (((uint32_t)j >> 1) & 1u) ^ 1u, abort_flag))) return false;
        tc_fence_after();
        const uint32_t a_addr = smem_addr + s * stage_bytes, d = tmem + (uint32_t)(j & 1) * acc_cols;
        const uint64_t adesc = tc_smem_desc(a_addr), bdesc = tc_smem_desc(a_addr + kRlABytes);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) tc_mma_elect<true>(d, adesc + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), idesc, k4 ? 1u : 0u);
        tc_commit_elect(&acc_full[j & 1]);
        tc_commit_elect(&empty[s]);
        if (++s == NS) {
            s = 0;
            par ^= 1u;
        }
    }
    return true;
}

// GROUPED: the launch's int8 problems have per-group weights (RL_I8G), else RL_I8; fp16 problems may be in either kind of launch.
// BUILD (fp16 problems with short rows, not split along K): the operands are built here from fp32 activations, straight into shared
// memory; a kernel of its own would cost more than every CTA converting the few rows again.
template <bool GROUPED, bool BUILD>
__global__ void __launch_bounds__(kRlThreads, 2) rows_linear_kernel(const __grid_constant__ RlLaunch L) {
    extern __shared__ __align__(1024) uint8_t rl_raw[];
    __shared__ __align__(8) uint64_t full[kRlMaxStages], empty[kRlMaxStages], acc_full[2], acc_empty[2], b_ready;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    __shared__ float s_xs[kRlMaxRowsF];
    __shared__ RlSum8 s_t[kRlMaxRows];  // int8
    __shared__ float s_ymax[4][kRlMaxRowsF];  // per lane quarter (32 weight rows)
    uint8_t* smem = (uint8_t*)(((uintptr_t)rl_raw + 1023) & ~(uintptr_t)1023);
    volatile int* abort_flag = &s_abort;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = BUILD ? 1 : L.split, rank = !BUILD && S > 1 ? (int)cluster_rank() : 0;
    const int job = (int)blockIdx.x / S;
    int pi = 0;
#pragma unroll 1
    while (pi + 1 < L.nprob && job >= L.p[pi + 1].job0) ++pi;
    const RlProb& P = L.p[pi];
    const int ltile = job - P.job0, mt = ltile / L.n_tiles, ntile = ltile - mt * L.n_tiles;
    const int fmt = BUILD ? (int)RL_F16 : P.fmt, D = rl_cols(fmt), NT = fmt == RL_F16 ? L.nt16 : L.nt8;
    const int stage_bytes = kRlABytes + (BUILD ? 0 : NT * 128), NS = min(kRlMaxStages, L.ring / stage_bytes);
    const int kb0 = P.kblocks * rank / S, nk = P.kblocks * (rank + 1) / S - kb0;
    const int r0 = ntile * L.rt, nr = min(L.rt, L.R - r0), ncols = nr * D;
    const bool grouped = GROUPED && fmt == RL_I8G;

    // The producer's thread sets the barriers up and requests the first ring pass of weights at once: the block's setup (tensor memory,
    // synchronisation) is hidden behind the copies.  Tiles the ring has no room for yet are requested into L2.
    const int kel = rl_kelems(fmt);
    const uint32_t bbytes = BUILD ? 0u : (uint32_t)(NT * 128);
    uint64_t pol = 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRlMaxStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kRlEpiWarps);
        }
        mbar_init(&b_ready, kRlEpiWarps);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // weights are read once per step: marked evict-first so that activations, states, vectors and the kernels' code stay in L2
        // (several row tiles share a weight tile: then it has to stay until the others have read it)
        pol = L.n_tiles == 1 ? l2_evict_first_policy() : l2_evict_normal_policy();
#pragma unroll 1
        for (int j = 0; j < nk; ++j) {
            if (grouped && (P.M & 3) == 0) l2_prefetch(P.szt + (size_t)(kb0 + j) * P.M + mt * kRlTileM, (uint32_t)min(kRlTileM, P.M - mt * kRlTileM) * 4u);
            if (j < NS) {
                mbar_expect_tx(&full[j], kRlABytes + bbytes);
                tma_load_2d_hint(&L.amap[pi], &full[j], smem + (size_t)j * stage_bytes, (kb0 + j) * kel, mt * kRlTileM, pol);
            } else {
                tma_prefetch_2d(&L.amap[pi], (kb0 + j) * kel, mt * kRlTileM);
            }
        }
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, (uint32_t)L.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- producer: operand tiles behind the dependency wait, then the rest of the ring's traffic ----------------
        if (lane == 0) {
            const uint8_t* bsrc = BUILD ? nullptr : P.bimg + ((size_t)ntile * P.kblocks + kb0) * bbytes;
            const int filled = min(NS, nk);
            uint32_t s = 0, par = 1;  // a fresh barrier passes a wait on parity 1
            int j = 0;
            if (!BUILD) pdl_wait();
#pragma unroll 1
            for (; j < nk; ++j) {
                uint8_t* dst = smem + (size_t)s * stage_bytes;
                if (j >= filled) {
                    if (!mbar_wait(&empty[s], par, abort_flag)) break;
                    mbar_expect_tx(&full[s], kRlABytes + bbytes);
                    tma_load_2d_hint(&L.amap[pi], &full[s], dst, (kb0 + j) * kel, mt * kRlTileM, pol);
                }
                if (!BUILD) bulk_load(dst + kRlABytes, bsrc + (size_t)j * bbytes, bbytes, &full[s]);
                if (++s == (uint32_t)NS) {
                    s = 0;
                    par ^= 1u;
                }
            }
            if (*abort_flag)  // copies in flight land before the CTA may exit
#pragma unroll 1
                for (int q = max(0, j - NS); q < j; ++q)
#pragma unroll 1
                    for (uint32_t i = 0; i < (1u << 16); ++i)
                        if (mbar_try_wait(&full[q % NS], (uint32_t)(q / NS) & 1u)) break;
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the warp runs convergently, one elected lane issues) ----------------
        const uint32_t idesc = tc_idesc(fmt != RL_F16, (ncols + 15) & ~15), smem_addr = smem_u32(smem);
        uint32_t s = 0, par = 0;
        bool ok;
        if (BUILD) {
            const uint32_t bbuf = smem_addr + (uint32_t)L.ring;
            ok = __all_sync(0xffffffffu, mbar_wait(&b_ready, 0u, abort_flag));
            tc_fence_after();
#pragma unroll 1
            for (int j = 0; j < nk && ok; ++j) {
                ok = __all_sync(0xffffffffu, mbar_wait(&full[s], par, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint64_t adesc = tc_smem_desc(smem_addr + s * (uint32_t)stage_bytes), bdesc = tc_smem_desc(bbuf + (uint32_t)(j * NT * 128));
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) tc_mma_elect<false>(tmem, adesc + (uint64_t)(k4 * 2), bdesc + (uint64_t)(k4 * 2), idesc, (j == 0 && k4 == 0) ? 0u : 1u);
                tc_commit_elect(&empty[s]);
                if (++s == (uint32_t)NS) {
                    s = 0;
                    par ^= 1u;
                }
            }
        } else if (grouped) {
            ok = rl_mma_groups(full, empty, acc_full, acc_empty, (uint32_t)NS, nk, smem_addr, (uint32_t)stage_bytes, tmem, rl_group_cols(NT), idesc, abort_flag);
        } else if (fmt != RL_F16) {
            ok = rl_mma_tile<true>(full, empty, s, par, (uint32_t)NS, nk, smem_addr, (uint32_t)stage_bytes, tmem, idesc, abort_flag);
        } else {
            ok = rl_mma_tile<false>(full, empty, s, par, (uint32_t)NS, nk, smem_addr, (uint32_t)stage_bytes, tmem, idesc, abort_flag);
        }
        if (!grouped && ok) tc_commit_elect(&acc_full[0]);
    }
    // epilogue warps: output row m of this thread, and which of the two warps of its lane quarter it is in
    const bool epi = warp >= 2;
    const int et = threadIdx.x - 64, ew = warp - 2, half = (ew >> 2) & 1, quarter = warp & 3, ml = quarter * 32 + lane, m = mt * kRlTileM + ml;
    const bool mok = m < P.M;
    const int sh = L.log_split, slots = (nr + S - 1) >> sh;
    const uint32_t recv = smem_u32(smem);
    float ws = 0.f, wz = 0.f, bias = 0.f;
    constexpr int kGChunks = kRlMaxRowsG / 8 / 2;  // 32-column chunks (eight activation rows) per warp
    float gacc[GROUPED ? kGChunks : 1][8];
    const int tg_rows = rl_group_rows(L.rt);
    uint32_t z0 = 0, z1 = 0;  // grouped: (scale, zero) words of the next two groups
    if (epi) {
        if (mok) {
            if (!BUILD && fmt == RL_I8) {
                ws = P.wscale[m];
                wz = P.wzero[m];
            }
            if (P.bias) bias = P.bias[m];
            if (grouped) {
                z0 = __ldg(P.szt + (size_t)kb0 * P.M + m);
                if (nk > 1) z1 = __ldg(P.szt + (size_t)(kb0 + 1) * P.M + m);
            }
        }
        float* s_tg = reinterpret_cast<float*>(smem + L.ring);  // grouped: [nk][tg_rows]
        pdl_wait();
        if (BUILD) {
            // a warp per row: find the maximum, convert; elements past K are zeros (the tensor map fills the weights there with zeros)
            uint8_t* bb = smem + L.ring;
#pragma unroll 1
            for (int r = ew; r < nr; r += kRlEpiWarps) {
                const float* x = P.x + (size_t)(r0 + r) * P.ldx;
                float am = 0.f, v[2][8];  // the row's first 512 elements stay in registers
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int k = 8 * (lane + 32 * q);
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[q][e] = 0.f;
                    if (k < P.K) rl_load8(v[q], x + k);
#pragma unroll
                    for (int e = 0; e < 8; ++e) am = fmaxf(am, fabsf(v[q][e]));
                }
#pragma unroll 1
                for (int k = 512 + 8 * lane; k < P.K; k += 256) {
                    float t[8];
                    rl_load8(t, x + k);
#pragma unroll
                    for (int e = 0; e < 8; ++e) am = fmaxf(am, fabsf(t[e]));
                }
                const int ex = rl_scale_exp(warp_absmax(am));
                const float mult = rl_mult(RL_F16, ex);
#pragma unroll 1
                for (int c = lane, q = 0; c < nk * 8; c += 32, ++q) {
                    if (q >= 2) {
#pragma unroll
                        for (int e = 0; e < 8; ++e) v[1][e] = 0.f;
                        if (8 * c < P.K) rl_load8(v[1], x + 8 * c);
                    }
                    float t[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) t[e] = q == 0 ? v[0][e] : v[1][e];
                    rl_put8(RL_F16, bb + (size_t)(c >> 3) * (NT * 128), 2 * r, 8 * (c & 7), t, mult);
                }
                if (lane == 0) s_xs[r] = rl_xscale(RL_F16, ex);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tiles are read by the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_ready);
        } else {
            if (et < nr) {
                s_xs[et] = __ldcg(P.xscale + r0 + et);
                if (fmt == RL_I8) {
                    long long t = 0;
#pragma unroll 1
                    for (int i = 0; i < P.tparts; ++i) t += __ldcg(P.tsum + (size_t)(r0 + et) * P.tparts + i);
                    s_t[et] = RlSum8{t, rl_ll2d(t)};
                }
            }
            if (grouped)
#pragma unroll 4
                for (int i = et; i < nk * nr; i += kRlEpiThreads) {
                    const int r = i / nk, kb = i - r * nk;
                    s_tg[kb * tg_rows + r] = __ldcg(P.tgrp + (size_t)(r0 + r) * P.kblocks + kb0 + kb);
                }
        }
        rl_epi_sync();
        if (grouped) {
            // ---- per group: digit sums -> fp32, times the group's scale, plus zero x the group's activation sum ----
            // What bounds it: at few rows the way of a group's word from memory, at many the instructions of the sums.  The words come two groups ahead, the first two before
            // the wait, all of them asked into L2 with the weights; an accumulator is read 32 columns at a time (16 before) and one half of a sum does not go through the
            // conversion unit: a layer of 3 rows of 2560 channels 60.2 -> 54.0 us, of 16 75.2 -> 66.6, a prompt of 201 rows 272 -> 249.
#pragma unroll
            for (int c = 0; c < (GROUPED ? kGChunks : 1); ++c)
#pragma unroll
                for (int i = 0; i < 8; ++i) gacc[c][i] = 0.f;
            auto group = [&](int j, uint32_t& z) -> bool {
                const float gs = __half2float(__ushort_as_half((unsigned short)(z & 0xFFFFu))), gz = __half2float(__ushort_as_half((unsigned short)(z >> 16)));
                if (j + 2 < nk && mok) z = __ldg(P.szt + (size_t)(kb0 + j + 2) * P.M + m);
                if (!__all_sync(0xffffffffu, mbar_wait_parked(&acc_full[j & 1], ((uint32_t)j >> 1) & 1u, abort_flag))) return false;
                tc_fence_after();
                const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((j & 1) * rl_group_cols(NT));
#pragma unroll
                for (int c = 0; c < (GROUPED ? kGChunks : 1); ++c) {
                    const int c0 = (2 * c + half) * 32;
                    if (c0 < ncols) {  // (rows past the end of the tile: sums of nothing, never sent)
                        uint32_t v[32];
                        tmem_ld32(taddr + c0, v);
                        const float4* tg = reinterpret_cast<const float4*>(s_tg + j * tg_rows + (c0 >> 2));
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float4 t4 = tg[h];
                            const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                // |digit sum| <= 2^21: two halves of two digits each, their weighted sum in one fp32 fma.  One half through the conversion unit,
                                // the other beside it (both through it were its whole time: 464 cycles for 29 rows of a block, whose products take 256).
                                const uint32_t* d = v + 16 * h + 4 * i;
                                const float hi = fmaf(rl_small2f(d[0]), 128.0f, rl_small2f(d[1])), lo = (float)((int)d[2] * 128 + (int)d[3]);
                                gacc[c][4 * h + i] = fmaf(gs, fmaf(hi, 16384.0f, lo), fmaf(gz, t[i], gacc[c][4 * h + i]));
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[j & 1]);
                return true;
            };
#pragma unroll 1
            for (int j = 0; j < nk; j += 2) {  // (two groups, so that a word is two groups on its way)
                if (!group(j, z0)) break;
                if (j + 1 < nk && !group(j + 1, z1)) break;
            }
        } else {
            mbar_wait_parked(&acc_full[0], 0u, abort_flag);  // a time-out shows in the abort flag
        }
        tc_fence_after();
    }
    // K in one piece: the sums go from tensor memory through this thread's registers to the output.  Otherwise (and for per-group
    // weights) they are exchanged: row r of the tile is finished by CTA r mod S of the cluster (S = 1: this one); its sums land in the owner's ring as
    // [slice][row / S][128] eight-byte words: the exact integer, the hi and lo sums of an fp16 row, or the fp32 sum of per-group weights.
    if (S > 1) cluster_sync_all();  // every CTA of the cluster is done with its ring
    const bool go = epi && !__any_sync(0xffffffffu, *abort_flag), direct = BUILD || (S == 1 && !grouped);
    const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16);
    if (!BUILD && go && !direct) {
        auto send = [&](int r, unsigned long long v) {
            if (r < nr) st_cluster_u64(map_to_rank(recv + (uint32_t)(((rank * slots + (r >> sh)) * kRlTileM + ml) * 8), (uint32_t)(r & (S - 1))), v);
        };
        if (grouped) {
#pragma unroll
            for (int c = 0; c < (GROUPED ? kGChunks : 1); ++c)
#pragma unroll
                for (int i = 0; i < 8; ++i) send((2 * c + half) * 8 + i, (unsigned long long)__float_as_uint(gacc[c][i]));
        } else {
#pragma unroll 1
            for (int c0 = half * 16; c0 < ncols; c0 += 32) {
                uint32_t v[16];
                tmem_ld16(taddr + c0, v);
                if (fmt == RL_F16) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) send((c0 >> 1) + i, (unsigned long long)v[2 * i] | ((unsigned long long)v[2 * i + 1] << 32));
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) send((c0 >> 2) + i, (unsigned long long)rl_digits2q((int)v[4 * i], (int)v[4 * i + 1], (int)v[4 * i + 2], (int)v[4 * i + 3]));
                }
            }
        }
    }
    if (S > 1) cluster_sync_all();
    else if (GROUPED && epi && !direct) rl_epi_sync();
    const int epi_op = P.epi;
    const RlScale w8{ws, wz, 0.f, 0u, 0, false};  // (no products run beside this: fp64 is the shorter chain, a layer of 3 rows 44.0 us and 44.8, 64 rows 103.7 and 104.6)
    if (go && direct) {
        const RlOut out = rl_out(P, r0, nr, m, bias);
        rl_finish<kRlEpiWarps>(out, BUILD || fmt == RL_F16, taddr, s_xs, s_t, s_ymax[quarter], w8, mok, half, lane);
    } else if (!BUILD && go) {
        // this CTA's share of the rows: slices added in order, scaled, activated, stored (four rows at a time per thread)
        const int mine = nr > rank ? (nr - rank + S - 1) >> sh : 0;
        const size_t stride = (size_t)slots * kRlTileM, ystep = (size_t)P.ldy << sh;
        const size_t y0 = (size_t)(r0 + rank + (4 * half << sh)) * P.ldy + m;
        float *y = P.y + y0, *y2 = P.y2 ? P.y2 + y0 : nullptr;
        const bool maxima = P.ymax != nullptr;
#pragma unroll 1
        for (int rl = 4 * half; rl < mine; rl += 8, y += 8 * ystep) {
            const int left = mine - rl;  // rows past the end repeat the last one
            float a[4];
            const unsigned long long* src = reinterpret_cast<const unsigned long long*>(smem) + (size_t)rl * kRlTileM + ml;
            int r[4], off[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                off[i] = min(i, left - 1) * kRlTileM;
                r[i] = rank + ((rl + min(i, left - 1)) << sh);
            }
            if (fmt != RL_I8) {
                float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};  // (per-group weights: the fp32 sum is in hi, lo is zero)
#pragma unroll 1
                for (int s = 0; s < S; ++s, src += stride)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const unsigned long long t = src[off[i]];
                        hi[i] += __uint_as_float((uint32_t)t);
                        lo[i] += __uint_as_float((uint32_t)(t >> 32));
                    }
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = s_xs[r[i]] * (hi[i] + lo[i]);
            } else {
                long long q[4] = {0, 0, 0, 0};
#pragma unroll 1
                for (int s = 0; s < S; s += 2, src += 2 * stride)  // (S is 2, 4 or 8 here)
#pragma unroll
                    for (int i = 0; i < 4; ++i) q[i] += (long long)src[off[i]] + (long long)src[stride + off[i]];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = rl_value8(w8, s_xs[r[i]], q[i], s_t[r[i]]);
            }
            rl_activate4(epi_op, a, bias);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (mok && i < left) y[i * ystep] = a[i];
            if (y2) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (mok && i < left) y2[i * ystep] = a[i];
                y2 += 8 * ystep;
            }
            if (maxima) {
                const float mx = rl_rowmax4(a, mok, lane);
                if (lane < min(4, left)) s_ymax[quarter][rank + ((rl + lane) << sh)] = mx;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (P.ymax && go && et < nr && (et & (S - 1)) == rank) P.ymax[(size_t)(r0 + et) * ((P.M + kRlTileM - 1) / kRlTileM) + mt] = fmaxf(fmaxf(s_ymax[0][et], s_ymax[1][et]), fmaxf(s_ymax[2][et], s_ymax[3][et]));
    if (threadIdx.x == 0 && *abort_flag) atomicOr(L.status, 2);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)L.tmem_cols);
    }
}

// Several row tiles (per-row int8 weights; fp16 weights in tiles of more than 64 rows or cut for turns), and heads of one row tile: one persistent CTA per SM takes tiles of 128
// weight rows x up to 64 activation rows (fp16: 128) in turn, whole K.  One ring of stages runs through all of them and there are two accumulators, so the
// tensor core works on the next tile while the epilogue warps finish the last one.  With a CTA per tile (two resident) both CTAs of an SM ran in
// step: of a tile's 22 us at K = 2560 the tensor core worked 13 at 85 % of its rate, the rest was the first loads and the epilogue.
// Measured, 2560 x 10240 (ffn.key), int8: 1024 rows 139 us with a CTA per tile, now 72; 512 rows 82 and 41.  Sixteen epilogue warps: eight took longer over a
// tile than the tensor core over its 20 K blocks (512 rows 48; up to 128 rows there are eight all the same, see the launch).
// What bounds it: the products, at the clock that the power limit leaves them (1.75 GHz), and what gets in their way.  512 rows with parts switched off (us): ffn.key
// 41.7, products alone 31, without the copies 34, without the epilogue 37; ffn.value 48.0, 37, 40 and 44 (that GPU's; 44.3 on another, whose clock was higher).  The loop that issues products is a function of its own: inside
// the kernel's control flow it took 600 cycles a K block whose products take 480, as a function those 480 (a bare ring of barriers and products
// does too); with that and the integer epilogue (rl_value8) ffn.key 42.0 -> 41.0 us, ffn.value 45.6 -> 44.3, r, k, v and rank projections 40.8 -> 39.5, at 1024 rows ffn.key 75.6 -> 72.2.
// Tried without gain: four producer threads, six stages instead of four, weights asked into L2 a turn ahead, one warp that waits for an accumulator and wakes
// the others, the next stage's barrier tried ahead.
struct RlCursor {
    int job, pi, kb, nk, mt, ntile;
    __device__ __forceinline__ void set(const RlLaunch& L, int j) {
        job = j;
        kb = 0;
        while (pi + 1 < L.nprob && j >= L.p[pi + 1].job0) ++pi;  // jobs come in ascending order
        const int lt = j - L.p[pi].job0;
        mt = lt / L.n_tiles;
        ntile = lt - mt * L.n_tiles;
        nk = L.p[pi].kblocks;
    }
};
template <int WARPS>
__global__ void __launch_bounds__(rl_persistent_threads(WARPS), 1) rows_linear_persistent_kernel(const __grid_constant__ RlLaunch L, int jobs) {
    extern __shared__ __align__(1024) uint8_t rl_raw[];
    __shared__ __align__(8) uint64_t full[kRlMaxStages], empty[kRlMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    __shared__ float s_xs[kRlMaxRowsF];
    __shared__ RlSum8 s_t[kRlMaxRows];  // int8
    __shared__ float s_ymax[4][kRlMaxRowsF];
    uint8_t* smem = (uint8_t*)(((uintptr_t)rl_raw + 1023) & ~(uintptr_t)1023);
    volatile int* abort_flag = &s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, G = (int)gridDim.x;
    const uint32_t stage_bytes = (uint32_t)(kRlABytes + L.nt_max * 128), acc_cols = (uint32_t)L.tmem_cols / 2;
    const uint32_t NS = min((uint32_t)kRlMaxStages, (uint32_t)L.ring / stage_bytes);
    uint32_t filled = 0;
    uint64_t pol = 0;
    if (threadIdx.x == 0) {
        pol = L.n_tiles == 1 ? l2_evict_first_policy() : l2_evict_normal_policy();  // (see above)
        for (int i = 0; i < kRlMaxStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], WARPS);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // weights of the first ring pass, before the dependency wait
        RlCursor c;
        c.pi = 0;
        c.set(L, (int)blockIdx.x);
#pragma unroll 1
        for (; filled < NS && c.job < jobs; ++filled) {
            const int fmt = L.p[c.pi].fmt;
            mbar_expect_tx(&full[filled], kRlABytes + (uint32_t)(fmt == RL_F16 ? L.nt16 : L.nt8) * 128u);
            tma_load_2d_hint(&L.amap[c.pi], &full[filled], smem + (size_t)filled * stage_bytes, c.kb * rl_kelems(fmt), c.mt * kRlTileM, pol);
            if (++c.kb == c.nk) {
                if (c.job + G >= jobs) {
                    ++filled;
                    break;
                }
                c.set(L, c.job + G);
            }
        }
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, (uint32_t)L.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    RlCursor c;
    c.pi = 0;
    if (warp == 0) {
        if (lane == 0) {
            uint32_t f = 0, s = 0, par = 1;
            bool ok = true;
            pdl_wait();
#pragma unroll 1
            for (int job = (int)blockIdx.x; job < jobs && ok; job += G) {
                c.set(L, job);
                const RlProb& P = L.p[c.pi];
                const int kel = rl_kelems(P.fmt);
                const uint32_t bbytes = (uint32_t)(P.fmt == RL_F16 ? L.nt16 : L.nt8) * 128u;
                const uint8_t* bsrc = P.bimg + (size_t)c.ntile * c.nk * bbytes;
#pragma unroll 1
                for (int kb = 0; kb < c.nk; ++kb, ++f, bsrc += bbytes) {
                    uint8_t* dst = smem + (size_t)s * stage_bytes;
                    if (f >= filled) {
                        if (!mbar_wait(&empty[s], par, abort_flag)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(&full[s], kRlABytes + bbytes);
                        tma_load_2d_hint(&L.amap[c.pi], &full[s], dst, kb * kel, c.mt * kRlTileM, pol);
                    }
                    bulk_load(dst + kRlABytes, bsrc, bbytes, &full[s]);
                    if (++s == NS) {
                        s = 0;
                        par ^= 1u;
                    }
                }
            }
            if (*abort_flag)  // copies in flight land before the CTA may exit
#pragma unroll 1
                for (uint32_t q = f > NS ? f - NS : 0; q < f; ++q)
#pragma unroll 1
                    for (uint32_t i = 0; i < (1u << 16); ++i)
                        if (mbar_try_wait(&full[q % NS], (q / NS) & 1u)) break;
        }
    } else if (warp == 1) {
        const uint32_t smem_addr = smem_u32(smem);
        uint32_t s = 0, par = 0, it = 0;
        bool ok = true;
#pragma unroll 1
        for (int job = (int)blockIdx.x; job < jobs && ok; job += G, ++it) {
            c.set(L, job);
            const int fmt = L.p[c.pi].fmt, nr = min(L.rt, L.R - c.ntile * L.rt);
            const uint32_t idesc = tc_idesc(fmt != RL_F16, (nr * rl_cols(fmt) + 15) & ~15), d = tmem + (it & 1u) * acc_cols;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[it & 1u], ((it >> 1) & 1u) ^ 1u, abort_flag));
            if (ok)
                ok = fmt != RL_F16 ? rl_mma_tile<true>(full, empty, s, par, NS, c.nk, smem_addr, stage_bytes, d, idesc, abort_flag)
                                   : rl_mma_tile<false>(full, empty, s, par, NS, c.nk, smem_addr, stage_bytes, d, idesc, abort_flag);
            if (ok) tc_commit_elect(&acc_full[it & 1u]);
        }
    } else {
        const int et = threadIdx.x - 64, turn = (warp - 2) >> 2, quarter = warp & 3, ml = quarter * 32 + lane;
        uint32_t it = 0;
        pdl_wait();
        // every warp runs every turn (the block barriers below): after a time-out without waiting and without output
#pragma unroll 1
        for (int job = (int)blockIdx.x; job < jobs; job += G, ++it) {
            c.set(L, job);
            const RlProb& P = L.p[c.pi];
            const int r0 = c.ntile * L.rt, nr = min(L.rt, L.R - r0), m = c.mt * kRlTileM + ml;
            const bool mok = m < P.M;
            float ws = 0.f, wz = 0.f, bias = 0.f;
            if (mok) {
                if (P.fmt == RL_I8) {
                    ws = __ldg(P.wscale + m);
                    wz = __ldg(P.wzero + m);
                }
                if (P.bias) bias = __ldg(P.bias + m);
            }
            if (et < nr) {
                const float xs = __ldcg(P.xscale + r0 + et);
                s_xs[et] = xs;
                if (P.fmt == RL_I8) {
                    long long t = 0;
#pragma unroll 1
                    for (int i = 0; i < P.tparts; ++i) t += __ldcg(P.tsum + (size_t)(r0 + et) * P.tparts + i);
                    s_t[et] = RlSum8{t, rl_ll2d(t)};
                }
            }
            const RlScale w8 = rl_scale(ws, wz);
            rl_epi_sync<32 * WARPS>();
            if (!*abort_flag) mbar_wait_parked(&acc_full[it & 1u], (it >> 1) & 1u, abort_flag);
            tc_fence_after();
            if (!__any_sync(0xffffffffu, *abort_flag)) {
                const RlOut out = rl_out(P, r0, nr, m, bias);
                rl_finish<WARPS>(out, P.fmt == RL_F16, tmem + ((uint32_t)(quarter * 32) << 16) + (it & 1u) * acc_cols, s_xs, s_t, s_ymax[quarter], w8, mok, turn, lane);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[it & 1u]);
            rl_epi_sync<32 * WARPS>();
            if (P.ymax && et < nr)
                P.ymax[(size_t)(r0 + et) * ((P.M + kRlTileM - 1) / kRlTileM) + c.mt] = fmaxf(fmaxf(s_ymax[0][et], s_ymax[1][et]), fmaxf(s_ymax[2][et], s_ymax[3][et]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicOr(L.status, 2);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, (uint32_t)L.tmem_cols);
    }
}

}  // namespace rsv
