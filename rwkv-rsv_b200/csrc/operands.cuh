// Activation operands of the tensor-core linear layers (rows_linear.cuh), and the LayerNorm + token-shift kernel that produces most
// of them.
//
// An operand is what an activation matrix x[R, K] becomes before it meets weights on the tensor cores:
//   int8 weights: t = rint(x / e 2^27), e = 2^ceil(log2 max|x_r|) per row r, as four signed base-128 digits = four int8 columns;
//   fp16 weights: x / e split into hi + lo fp16 halves = two columns.
// It is stored as the image of the shared-memory tiles the GEMM reads: [row tile][128-byte block of K][column][128 bytes] with the
// 16-byte chunks of a column permuted as the 128-byte swizzle wants them (chunk ^ (column mod 8)), so that a tile is one untiled
// bulk copy and needs no tensor map, and the same code can write it straight to shared memory inside the GEMM.
// Besides the image a row leaves its scale (xscale), and for int8 the exact sum of its t: over the row (tsum; one (scale, zero) per
// weight row) or per group of 128 (tgrp; one per weight row and group).
#pragma once
#include "kernels.cuh"
#include "row_tiles.hpp"

namespace rsv {

constexpr int kRlP = 7 * kRlDigits - 1;  // fixed-point bits

// smallest ex with 2^ex >= amax (0 for an all-zero or non-finite row)
__device__ __forceinline__ int rl_scale_exp(float amax) {
    const uint32_t b = __float_as_uint(amax);
    if (!(amax > 0.f && amax < 3.0e38f)) return 0;
    const int ex = (int)(b >> 23) - 127 + ((b & 0x7FFFFFu) ? 1 : 0);
    return max(-99, min(99, ex));
}
__device__ __forceinline__ float rl_pow2(int n) { return __int_as_float((n + 127) << 23); }  // -126 <= n <= 127
// fp32 scale of a row: what one unit of its fixed-point (int8) or normalised (fp16) values is worth
__device__ __forceinline__ float rl_xscale(int fmt, int ex) { return rl_pow2(fmt == RL_F16 ? ex : ex - kRlP); }
__device__ __forceinline__ float rl_mult(int fmt, int ex) { return rl_pow2(fmt == RL_F16 ? -ex : kRlP - ex); }

__device__ __forceinline__ void rl_load8(float (&v)[8], const float* p) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p + 4));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// Eight consecutive elements (K index kin .. kin + 7 inside a block, a multiple of 8) of the activation row whose first column in
// the tile is n0.  Returns the sum of the fixed-point values (int8; 0 for fp16).  `tile`: global or shared memory.
__device__ __forceinline__ int rl_put8(int fmt, uint8_t* tile, int n0, int kin, const float (&v)[8], float mult) {
    if (fmt == RL_F16) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float a = v[2 * i] * mult, b = v[2 * i + 1] * mult;
            a = fminf(fmaxf(a, -1.0f), 1.0f);
            b = fminf(fmaxf(b, -1.0f), 1.0f);
            const __half2 h = __floats2half2_rn(a, b);
            const float2 hf = __half22float2(h);
            const __half2 l = __floats2half2_rn(a - hf.x, b - hf.y);
            hi[i] = *reinterpret_cast<const uint32_t*>(&h);
            lo[i] = *reinterpret_cast<const uint32_t*>(&l);
        }
        const int chunk = kin >> 3;
        *reinterpret_cast<uint4*>(tile + n0 * 128 + ((chunk ^ (n0 & 7)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(tile + (n0 + 1) * 128 + ((chunk ^ ((n0 + 1) & 7)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        return 0;
    }
    int ts = 0;
    uint32_t dig[4][2];  // digit j of elements 0-3, 4-7
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int t = __float2int_rn(v[4 * q + i] * mult);  // NaN -> 0
            t = max(-(1 << kRlP), min(1 << kRlP, t));
            ts += t;
            // biased by 64 in each of the three low digits the base-128 fields of t are its balanced digits + 64: one field per byte
            const uint32_t u = (uint32_t)t + 64u * (1u + 128u + 16384u);
            w[i] = (u & 0x7Fu) | ((u << 1) & 0x7F00u) | ((u << 2) & 0x7F0000u) | ((u << 3) & 0xFF000000u);
        }
        // 4 x 4 byte transpose: byte position (low to high) = digit 3, 2, 1, 0
        const uint32_t a01 = __byte_perm(w[0], w[1], 0x5140), b01 = __byte_perm(w[0], w[1], 0x7362);
        const uint32_t a23 = __byte_perm(w[2], w[3], 0x5140), b23 = __byte_perm(w[2], w[3], 0x7362);
        auto unbias = [](uint32_t f) {  // bytes f in 0 .. 127 -> f - 64 as int8
            const uint32_t y = f ^ 0x40404040u;
            return y | ((y & 0x40404040u) << 1);
        };
        dig[3][q] = unbias(__byte_perm(a01, a23, 0x5410));
        dig[2][q] = unbias(__byte_perm(a01, a23, 0x7632));
        dig[1][q] = unbias(__byte_perm(b01, b23, 0x5410));
        dig[0][q] = __byte_perm(b01, b23, 0x7632);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = n0 + j;
        *reinterpret_cast<uint2*>(tile + n * 128 + (((kin >> 4) ^ (n & 7)) << 4) + (kin & 8)) = make_uint2(dig[j][0], dig[j][1]);
    }
    return ts;
}

// Where one operand of a step goes.
struct RlOperandOut {
    const float* mix;  // token-shift mix vector of the operand (null: the normalised row itself)
    uint8_t* img;
    float* xscale;    // [R]
    long long* tsum;  // [R][tparts] (RL_I8)
    float* tgrp;      // [R][kblocks] (RL_I8G)
    int fmt, nt, kblocks, tparts;  // nt: columns of a tile
};
__device__ __forceinline__ uint8_t* rl_tile(const RlOperandOut& o, int rt, int r, int kb) {
    return o.img + ((size_t)(r / rt) * o.kblocks + kb) * (size_t)(o.nt * 128);
}
// sum of ts over the 16 lanes that hold one group of 128 elements (|ts| <= 2^30 per lane)
__device__ __forceinline__ long long rl_group_sum(int ts) {
    int lo = ts & 0xFFFF, hi = ts >> 16;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
        hi += __shfl_xor_sync(0xffffffffu, hi, o);
    }
    return (long long)hi * 65536 + lo;
}

// ---- LayerNorm + token shift -> operands ------------------------------------------------------------------------------------
// One CTA per row (and, with gridDim.y > 1, per output): eight channels per thread, the row lives in registers.
//   cur = LN(x_in[r] (+ delta[r])), prev = LN of row r - 1 when that row is the session's previous token (the same code, hence the
//   same bits) and the slot's shift state otherwise; output o = cur + mix_o (prev - cur), written as an operand.
// Stands in for norm_lerp6(_batch), cmix_norm_lerp(_batch), rwkv_seq_shift(_batch) and rwkv_copy_token(_batch)
// (src/backend_cuda.rs:2412-2549, 1505-1640, 4313-4406; math src/model.rs:402-411, 484-495), and, without shift, for ln_out
// (src/model.rs:507).  `delta` is the pending residual of the linear layer before; the sum goes to x_out, another buffer, because row
// r - 1's sum is needed too while another CTA produces it.  With multi-row segments the new shift state goes to `staging`, because a
// segment's first row still has to read the old one; the CTAs past the rows commit the staging area of the block before this one.
// What bounds it: at few rows the chain load -> mean -> variance -> row maximum -> digits (block-wide reductions); it writes operands instead of fp32 because the
// conversion in a kernel of its own cost a second launch and a second such chain (8 rows, n_embd 2560: 11.0 + 9.2 us for the two kernels it replaces, CUDA events around each).
// Cycles after the dependency wait at 3 rows: loads 1500, two sums of 700, normalising 700, maxima 360, digits 1800, sum of digits 500 (in 64-bit shuffles; two integer reductions
// now, here and in operand_known_kernel: a layer of 3 rows 44.6 -> 44.1 us, 16 58.4 -> 57.6); 512 rows of six outputs are bound by the digits.  The row stays in registers: in shared
// memory the sums took 1.4 us, and the kernel's 20 KB kept the next launch's CTAs off its SMs.  The outputs go one by one with a barrier each, the next one's mix
// vector on its way meanwhile; with all maxima behind one barrier every value was computed twice and every mix vector read twice, which cost more than the barriers, most of all
// in narrow models.  Exclusive us in the step, one output and six, with the row in shared memory, one barrier, as it is: 2560 channels 512 rows 15.2 27.4, 11.6 23.8, 11.0
// 21.3, 1024 rows 25.8 45.3, 23.7 43.1, 22.4 38.5; 1024 channels 512 rows 7.9 15.2, 7.9 19.2, 7.6 17.1, 256 rows 7.2 12.1, 6.4 10.4, 6.1 8.3.
// The variants with 64 registers spill one of them, which costs nothing that shows.
struct LnOperandsArgs {
    const float *x_in, *delta;
    float* x_out;
    const float *lw, *lb;
    const RowMeta* rows;
    const int* row_map;  // not null: LayerNorm of rows row_map[0 .. R), no shift
    float *shift_state, *staging;
    const float* commit_src;  // [nseg, C] -> commit_dst[slot of the segment]
    float* commit_dst;
    const SegMeta* segs;
    int R, C, rt, nseg, nout;
    RlOperandOut out[7];
};
constexpr int kLnMaxThreads = 1024;  // n_embd up to 8192 (ln_operands_wide_kernel: any)
constexpr int kLnSumThreads = 256;  // the wide kernel: threads that take part in the row sums
// Sums over the block of a (the row) and, where `two`, of b (the previous token's row): shuffles, then every warp adds the warps' sums.  The order depends on
// the row's length alone, so a row gives the same bits as itself and as somebody's previous token, whatever the step.
__device__ __forceinline__ void ln_block_sums(float& a, float& b, bool two, float (&red)[2][32], int warp, int lane, int nw) {
    a = warp_sum(a);
    if (two) b = warp_sum(b);
    if (lane == 0) {
        red[0][warp] = a;
        red[1][warp] = b;
    }
    __syncthreads();
    a = warp_sum(lane < nw ? red[0][lane] : 0.f);
    if (two) b = warp_sum(lane < nw ? red[1][lane] : 0.f);
}
__device__ __forceinline__ float ln_sum8(const float (&v)[8]) { return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])); }
__device__ __forceinline__ float ln_square8(const float (&v)[8]) {
    float q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = v[i] * v[i];
    return ln_sum8(q);
}
__device__ __forceinline__ void ln_weights8(float (&v)[8], const float* p) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p + 4));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
// Blocks of the variant with 64 registers a thread (<320, 3>) that an SM holds.  While all rows' blocks are resident at once it is the faster one: the weights are
// there when they are needed.  With more rows the variant with 48 registers, which loads them where it uses them, fits more blocks beside one another: one output and six,
// 512 int8 rows of 2560 channels 12.6 22.6 us and 11.0 21.3; but 384 rows 9.1 17.1 and 10.8 21.1; 592 rows of 2048 channels (256 threads, four blocks) 11.8 18.7 and 11.1
// 21.3, 640 rows 13.2 22.5 and 11.8 21.3; 1024 rows of 512 channels (64 threads, sixteen blocks) 5.8 17.4 and 6.0 21.1.
constexpr int ln_resident_blocks(int threads) { return 1024 / threads; }
template <int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) ln_operands_kernel(const __grid_constant__ LnOperandsArgs A) {
    __shared__ float red[2][2][32];
    __shared__ float redm[7][32];
    __shared__ int2 redt[7][32];  // per output and warp: low 16 bits and the rest of the fixed-point sums, added up
    pdl_launch_dependents();
    const int C = A.C, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    if ((int)blockIdx.x >= A.R) {  // commit CTAs
        pdl_wait();
        if (blockIdx.y == 0) {
            const int sg = (int)blockIdx.x - A.R;
            float* dst = A.commit_dst + (size_t)A.segs[sg].slot * C;
#pragma unroll 1
            for (int i = 4 * tid; i < C; i += 4 * blockDim.x) *reinterpret_cast<float4*>(dst + i) = __ldcg(reinterpret_cast<const float4*>(A.commit_src + (size_t)sg * C + i));
        }
        return;
    }
    const int r = blockIdx.x, k0 = 8 * tid;
    const bool on = k0 < C;
    const int kc = on ? k0 : 0;
    RowMeta rm{0, 0, 0, 0};
    if (A.rows) rm = A.rows[r];
    const size_t row = A.row_map ? (size_t)A.row_map[r] : (size_t)r;
    const bool shift = A.rows != nullptr, pln = shift && rm.has_prev;
    // weights before the dependency wait, or where they are used (see above)
    constexpr bool EARLY = BLOCKS < 4;
    float lw[8], lb[8], mx[8];
    const int o0 = blockIdx.y, step = gridDim.y;
    if (EARLY) {
        ln_weights8(lw, A.lw + kc);
        ln_weights8(lb, A.lb + kc);
        if (A.out[o0].mix) ln_weights8(mx, A.out[o0].mix + kc);
    }
    const int rloc = r % A.rt, rtile = r / A.rt;
    pdl_wait();
    const float* xr = A.x_in + row * C + kc;
    const float* dr = A.delta ? A.delta + row * C + kc : nullptr;
    float x[8], xp[8];
    rl_load8(x, xr);
#pragma unroll
    for (int i = 0; i < 8; ++i) xp[i] = 0.f;
    if (shift) rl_load8(xp, pln ? xr - C : A.shift_state + (size_t)rm.slot * C + kc);
    if (dr) {
        float d[8];
        rl_load8(d, dr);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] += d[i];
        if (pln) {
            rl_load8(d, dr - C);
#pragma unroll
            for (int i = 0; i < 8; ++i) xp[i] += d[i];
        }
    }
    if (A.x_out && on && o0 == 0) {
        float4* o = reinterpret_cast<float4*>(A.x_out + row * C + k0);
        o[0] = make_float4(x[0], x[1], x[2], x[3]);
        o[1] = make_float4(x[4], x[5], x[6], x[7]);
    }
    float s0 = on ? ln_sum8(x) : 0.f, s1 = on ? ln_sum8(xp) : 0.f;
    ln_block_sums(s0, s1, pln, red[0], warp, lane, nw);
    s0 /= (float)C;
    s1 /= (float)C;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] -= s0;
        if (pln) xp[i] -= s1;
    }
    s0 = on ? ln_square8(x) : 0.f;
    s1 = on ? ln_square8(xp) : 0.f;
    ln_block_sums(s0, s1, pln, red[1], warp, lane, nw);
    s0 = 1.0f / sqrtf(s0 / (float)C + kLnEps);
    s1 = 1.0f / sqrtf(s1 / (float)C + kLnEps);
    if (!EARLY) {
        ln_weights8(lw, A.lw + kc);
        ln_weights8(lb, A.lb + kc);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] = x[i] * s0 * lw[i] + lb[i];                  // cur
        if (pln) xp[i] = xp[i] * s1 * lw[i] + lb[i];  // prev
        xp[i] -= x[i];                                     // prev - cur
    }
    if (shift && rm.is_last && on && o0 == 0) {
        float4* o = reinterpret_cast<float4*>(A.staging + (size_t)rm.seg * C + k0);
        o[0] = make_float4(x[0], x[1], x[2], x[3]);
        o[1] = make_float4(x[4], x[5], x[6], x[7]);
    }
    // output by output; the next one's mix vector is on its way meanwhile
    if (!EARLY && A.out[o0].mix) ln_weights8(mx, A.out[o0].mix + kc);
#pragma unroll 1
    for (int o = o0; o < A.nout; o += step) {
        const RlOperandOut& O = A.out[o];
        float v[8], am = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[i] = O.mix ? x[i] + mx[i] * xp[i] : x[i];
            am = fmaxf(am, fabsf(v[i]));
        }
        if (o + step < A.nout && A.out[o + step].mix) ln_weights8(mx, A.out[o + step].mix + kc);
        am = warp_absmax(on ? am : 0.f);
        if (lane == 0) redm[o][warp] = am;
        __syncthreads();
        const int ex = rl_scale_exp(warp_absmax(lane < nw ? redm[o][lane] : 0.f)), fmt = O.fmt, lk = fmt == RL_F16 ? 6 : 7;
        int ts = 0;
        if (on)
            ts = rl_put8(fmt, O.img + ((size_t)rtile * O.kblocks + (k0 >> lk)) * (size_t)(O.nt * 128), rloc * rl_cols(fmt), k0 & ((1 << lk) - 1), v, rl_mult(fmt, ex));
        if (fmt == RL_I8G) {
            const long long t16 = rl_group_sum(ts);
            if (on && (lane & 15) == 0) O.tgrp[(size_t)r * O.kblocks + k0 / 128] = (float)t16;
        } else if (fmt == RL_I8) {
            const int lo = __reduce_add_sync(0xffffffffu, ts & 0xFFFF), hi = __reduce_add_sync(0xffffffffu, ts >> 16);
            if (lane == 0) redt[o][warp] = make_int2(lo, hi);
        }
        if (tid == 0) O.xscale[r] = rl_xscale(fmt, ex);
    }
    __syncthreads();
#pragma unroll 1
    for (int o = warp; o < A.nout; o += nw)
        if (o % step == o0 && A.out[o].fmt == RL_I8) {
            const int2 t = lane < nw ? redt[o][lane] : make_int2(0, 0);
            const int lo = __reduce_add_sync(0xffffffffu, t.x), hi = __reduce_add_sync(0xffffffffu, t.y);
            if (lane == 0) A.out[o].tsum[r] = (long long)hi * 65536 + lo;
        }
}

// The same for rows that do not fit the block's registers (n_embd above 8192): the row is read again from global memory (L2) for the statistics,
// for every output's maximum and for its digits.  Its sums have an order of their own, which also depends on the length of a row alone.  No model in use is this wide, so nothing is tuned here.
__global__ void __launch_bounds__(kLnMaxThreads) ln_operands_wide_kernel(const __grid_constant__ LnOperandsArgs A) {
    __shared__ float red[2][kLnSumThreads / 32], redm[32];
    __shared__ long long redt[32];
    pdl_launch_dependents();
    pdl_wait();
    const int C = A.C, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    if ((int)blockIdx.x >= A.R) {  // commit CTAs
        if (blockIdx.y == 0) {
            const int sg = (int)blockIdx.x - A.R;
            float* dst = A.commit_dst + (size_t)A.segs[sg].slot * C;
            for (int i = tid; i < C; i += blockDim.x) dst[i] = __ldcg(A.commit_src + (size_t)sg * C + i);
        }
        return;
    }
    const int r = blockIdx.x, rloc = r % A.rt, rtile = r / A.rt;
    RowMeta rm{0, 0, 0, 0};
    if (A.rows) rm = A.rows[r];
    const size_t row = A.row_map ? (size_t)A.row_map[r] : (size_t)r;
    const bool shift = A.rows != nullptr, pln = shift && rm.has_prev;
    const float *xr = A.x_in + row * C, *dr = A.delta ? A.delta + row * C : nullptr, *sr = shift ? A.shift_state + (size_t)rm.slot * C : nullptr;
    auto load8 = [&](float (&v)[8], const float* x, const float* d, int k) {  // eight elements of a row with its pending residual
        rl_load8(v, x + k);
        if (d) {
            float t[8];
            rl_load8(t, d + k);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] += t[i];
        }
    };
    if (A.x_out && blockIdx.y == 0)
        for (int k = 8 * tid; k < C; k += 8 * blockDim.x) {
            float v[8];
            load8(v, xr, dr, k);
            float4* o = reinterpret_cast<float4*>(A.x_out + row * C + k);
            o[0] = make_float4(v[0], v[1], v[2], v[3]);
            o[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
    float mean[2] = {0.f, 0.f}, inv[2] = {0.f, 0.f};
    for (int w = 0; w < (pln ? 2 : 1); ++w)
        for (int pass = 0; pass < 2; ++pass) {
            const float *x = xr - (size_t)w * C, *d = dr ? dr - (size_t)w * C : nullptr;
            if (tid < kLnSumThreads) {
                float a = 0.f;
                for (int i = tid; i < C; i += kLnSumThreads) {
                    const float v = __ldcg(x + i) + (d ? __ldcg(d + i) : 0.f), c = v - mean[w];
                    a += pass ? c * c : v;
                }
                a = warp_sum(a);
                if (lane == 0) red[pass][warp] = a;
            }
            __syncthreads();
            float sum = 0.f;
            for (int i = 0; i < kLnSumThreads / 32; ++i) sum += red[pass][i];
            if (pass == 0)
                mean[w] = sum / (float)C;
            else
                inv[w] = 1.0f / sqrtf(sum / (float)C + kLnEps);
        }
    // cur = LN of the row, and prev - cur, at channels k .. k + 7
    auto normalised = [&](float (&x)[8], float (&xp)[8], int k) {
        float lw[8], lb[8];
        rl_load8(lw, A.lw + k);
        rl_load8(lb, A.lb + k);
        load8(x, xr, dr, k);
        if (pln)
            load8(xp, xr - C, dr ? dr - C : nullptr, k);
        else if (shift)
            rl_load8(xp, sr + k);
        else
            for (int i = 0; i < 8; ++i) xp[i] = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            x[i] = (x[i] - mean[0]) * inv[0] * lw[i] + lb[i];
            if (pln) xp[i] = (xp[i] - mean[1]) * inv[1] * lw[i] + lb[i];
            xp[i] -= x[i];
        }
    };
    if (shift && rm.is_last && blockIdx.y == 0)
        for (int k = 8 * tid; k < C; k += 8 * blockDim.x) {
            float x[8], xp[8];
            normalised(x, xp, k);
            float4* o = reinterpret_cast<float4*>(A.staging + (size_t)rm.seg * C + k);
            o[0] = make_float4(x[0], x[1], x[2], x[3]);
            o[1] = make_float4(x[4], x[5], x[6], x[7]);
        }
    for (int o = blockIdx.y; o < A.nout; o += gridDim.y) {
        const RlOperandOut& O = A.out[o];
        auto mixed = [&](float (&v)[8], int k) {
            float xp[8];
            normalised(v, xp, k);
            if (O.mix) {
                float mx[8];
                rl_load8(mx, O.mix + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = v[i] + mx[i] * xp[i];
            }
        };
        float am = 0.f;
        for (int k = 8 * tid; k < C; k += 8 * blockDim.x) {
            float v[8];
            mixed(v, k);
#pragma unroll
            for (int i = 0; i < 8; ++i) am = fmaxf(am, fabsf(v[i]));
        }
        am = warp_absmax(am);
        if (lane == 0) redm[warp] = am;
        __syncthreads();
        const int ex = rl_scale_exp(warp_absmax(lane < nw ? redm[lane] : 0.f)), fmt = O.fmt, kel = rl_kelems(fmt);
        long long tot = 0;
        for (int k0 = 0; k0 < C; k0 += 8 * blockDim.x) {  // (uniform trip count: the sums below are warp-wide)
            const int k = k0 + 8 * tid;
            int ts = 0;
            if (k < C) {
                float v[8];
                mixed(v, k);
                ts = rl_put8(fmt, O.img + ((size_t)rtile * O.kblocks + k / kel) * (size_t)(O.nt * 128), rloc * rl_cols(fmt), k % kel, v, rl_mult(fmt, ex));
            }
            if (fmt == RL_F16) continue;
            const long long t16 = rl_group_sum(ts);
            if (fmt == RL_I8G && k < C && (lane & 15) == 0) O.tgrp[(size_t)r * O.kblocks + k / 128] = (float)t16;
            tot += t16 + __shfl_xor_sync(0xffffffffu, t16, 16);
        }
        if (lane == 0) redt[warp] = tot;
        __syncthreads();
        if (tid == 0) {
            O.xscale[r] = rl_xscale(fmt, ex);
            if (fmt == RL_I8) {
                long long t = 0;
                for (int i = 0; i < nw; ++i) t += redt[i];
                O.tsum[r] = t;
            }
        }
        __syncthreads();  // redm and redt are written again
    }
}

// ---- operands of activations another kernel left in fp32 ----------------------------------------------------------------------
// Rows whose producer left maxima of |x| over `parts` parts of the row (amax[R][parts]): elementwise, grid (rows, ceil(K / 2048)); every
// CTA leaves the exact sum of its part of the row (tsum[R][gridDim.y]).  Elements between K and the end of the last block are written as
// zeros: the weights there are zero-filled by the tensor map, and 0 x NaN (what another step left in the image) would not be.
constexpr int kOpThreads = 256;
__global__ void __launch_bounds__(kOpThreads) operand_known_kernel(const float* x, int ldx, int K, const float* amax, int parts, int rt,
                                                                   const __grid_constant__ RlOperandOut O) {
    __shared__ int2 red[kOpThreads / 32];
    __shared__ float redm[kOpThreads / 32];
    pdl_launch_dependents();
    const int r = blockIdx.x, k0 = ((int)blockIdx.y * kOpThreads + (int)threadIdx.x) * 8, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();
    float v[8];
    rl_load8(v, x + (size_t)r * ldx + (k0 < K ? k0 : 0));
    float am = 0.f;
#pragma unroll 1
    for (int i = threadIdx.x; i < parts; i += kOpThreads) am = fmaxf(am, __ldcg(amax + (size_t)r * parts + i));
    am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(am)));
    if (lane == 0) redm[warp] = am;
    __syncthreads();
    am = redm[lane & (kOpThreads / 32 - 1)];
    const int ex = rl_scale_exp(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(am)))), kel = rl_kelems(O.fmt);
    int ts = 0;
    if (k0 < K) ts = rl_put8(O.fmt, rl_tile(O, rt, r, k0 / kel), (r % rt) * rl_cols(O.fmt), k0 % kel, v, rl_mult(O.fmt, ex));
    else if (O.fmt == RL_F16 && k0 < O.kblocks * 64) {  // (K of int8 weights is whole blocks)
        uint8_t* col = rl_tile(O, rt, r, k0 / 64) + (r % rt) * 2 * 128;
        const int chunk = (k0 % 64) / 8, n0 = (r % rt) * 2;
        *reinterpret_cast<uint4*>(col + ((chunk ^ (n0 & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(col + 128 + ((chunk ^ ((n0 + 1) & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (O.fmt == RL_I8G) {
        const long long t16 = rl_group_sum(ts);
        if (k0 < K && (lane & 15) == 0) O.tgrp[(size_t)r * O.kblocks + k0 / 128] = (float)t16;
    } else if (O.fmt == RL_I8) {
        const int lo = __reduce_add_sync(0xffffffffu, ts & 0xFFFF), hi = __reduce_add_sync(0xffffffffu, ts >> 16);
        if (lane == 0) red[warp] = make_int2(lo, hi);
        __syncthreads();
        if (warp == 0) {
            const int2 t = lane < kOpThreads / 32 ? red[lane] : make_int2(0, 0);
            const int l = __reduce_add_sync(0xffffffffu, t.x), h = __reduce_add_sync(0xffffffffu, t.y);
            if (lane == 0) O.tsum[(size_t)r * gridDim.y + blockIdx.y] = (long long)h * 65536 + l;
        }
    }
    if (blockIdx.y == 0 && threadIdx.x == 0) O.xscale[r] = rl_xscale(O.fmt, ex);
}

// Short rows (the rank-space vectors; any length works): one warp per (row, matrix) finds the maximum, then converts.  Elements
// between K and the end of the last block are written as zeros, as above.
struct OperandRowsArgs {
    const float* x[4];
    int ldx[4], K[4];
    RlOperandOut out[4];
    int R, rt, n;
};
__global__ void __launch_bounds__(kOpThreads) operand_rows_kernel(const __grid_constant__ OperandRowsArgs A) {
    pdl_launch_dependents();
    const int item = (int)blockIdx.x * (kOpThreads / 32) + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    pdl_wait();
    if (item >= A.R * A.n) return;
    const int r = item / A.n, m = item - r * A.n;
    const RlOperandOut& O = A.out[m];
    const float* x = A.x[m] + (size_t)r * A.ldx[m];
    const int K = A.K[m], kel = rl_kelems(O.fmt), kend = O.kblocks * kel;
    float am = 0.f;
    for (int k = 4 * lane; k < K; k += 128) {
        const float4 t = __ldcg(reinterpret_cast<const float4*>(x + k));
        am = fmaxf(fmaxf(am, fmaxf(fabsf(t.x), fabsf(t.y))), fmaxf(fabsf(t.z), fabsf(t.w)));
    }
    am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(am)));
    const int ex = rl_scale_exp(am);
    const float mult = rl_mult(O.fmt, ex);
    long long tot = 0;
    for (int kk = 0; kk < kend; kk += 256) {  // (uniform trip count: the sums below are warp-wide)
        const int k = kk + 8 * lane;
        int ts = 0;
        if (k < kend) {
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (k < K) rl_load8(v, x + k);
            ts = rl_put8(O.fmt, rl_tile(O, A.rt, r, k / kel), (r % A.rt) * rl_cols(O.fmt), k % kel, v, mult);
        }
        if (O.fmt != RL_F16) {
            const long long t16 = rl_group_sum(ts);
            if (O.fmt == RL_I8G && k < kend && (lane & 15) == 0) O.tgrp[(size_t)r * O.kblocks + k / 128] = (float)t16;
            tot += t16 + __shfl_xor_sync(0xffffffffu, t16, 16);
        }
    }
    if (lane == 0) {
        O.xscale[r] = rl_xscale(O.fmt, ex);
        if (O.fmt == RL_I8) O.tsum[r] = tot;
    }
}

}  // namespace rsv
