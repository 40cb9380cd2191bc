// WKV-7 for a long prompt of one session (or few): sixteen tokens at a time in matrix form.
// Stands in for rwkv_fuse_ka and rwkv_dplr_seq(_batch) (src/backend_cuda.rs:4231-4309, 4436-4575; math src/model.rs:436-471), which walk a segment
// token by token.
//
// One head, state S [64 rows i][64 columns j].  Token t:  u_t = S kk_t;  S <- S diag(w_t) + u_t b_t^T + v_t k_t^T;  y_t = S r_t
// (kk: normalised, b = -kk a, k: k~).  With the running products W_t = w_1 ... w_t of a chunk of T = 16 tokens and
//   kk^_t = W_{t-1} kk_t,  r^_t = W_t r_t,  b^_s = b_s / W_s,  k^_s = k_s / W_s,
//   A_ts = kk^_t . b^_s,  B_ts = kk^_t . k^_s  (s < t),   E_ts = r^_t . b^_s,  F_ts = r^_t . k^_s  (s <= t)
// the chunk is   u_t = S0 kk^_t + sum_{s<t} (A_ts u_s + B_ts v_s),   y_t = S0 r^_t + sum_{s<=t} (E_ts u_s + F_ts v_s),
//                S = S0 diag(W_T) + sum_s (u_s (b_s W_T / W_s)^T + v_s (k_s W_T / W_s)^T).
// The triangular system does not involve the state, so it is solved for the right-hand sides kk^ and B v beforehand:
//   u = S0 K + UV,  y = S0 R + YV   with   K = (1 - A)^-1 kk^,  UV = (1 - A)^-1 B v,  R = r^ + E K,  YV = E UV + F v.
// Precision.  A model's decays lie in (0.545, 1] (exp(-sigmoid / sqrt(e))), so 1 / W stays below 1.7e4 and only products with W_t / W_s <= 1 are ever
// summed.  Everything is fp32 but the running products and the joining of the products' 16-column sums (double), and the sums are cut into short chains (in the
// products, even and odd terms in the solution; the state takes the sums of a chunk over u and over v, two roundings instead of seventeen).  Against the
// recurrence in 64 bits (320 and 512 tokens, 8 heads, normal inputs; 1e-7 relative, token by token in fp32 in brackets):
//   decays uniform in (0.545, 1): y 1.24 (1.30), state 0.72 (0.73);  all 0.545: 1.32 (1.50), 0.64 (0.67);  0.999 to 1: 1.67 (2.38), 1.65 (3.19);
//   those of a random model: 1.36 (1.42), 1.02 (1.12).
//
//   wkv7_prepare_kernel  one CTA per (head, chunk), all chunks of the step at once: the vectors and K, R, UV, YV of a chunk -> scratch
//   wkv7_chunk_kernel    two CTAs per (head, segment), 32 state rows each, chunk after chunk: two products with the state per chunk
// GroupNorm, bonus and gate follow in wkv7_finish_kernel (wkv_seq.cuh).
// What bounds it: shared memory.  A 16-byte read of a warp takes four cycles however many lanes want the same bytes; a chunk's products are 112 of them
// per warp (a lane's tile is four rows x eight tokens, then four rows x four columns), 1800 cycles of the 3400 a chunk takes; the rest is the
// chain products, barrier, sums, barrier, products.  512 tokens, 40 heads: 56 us and 27 to prepare; token by token 130.  201 tokens: 25 + 14 and 51.
// A CTA asks for more than half of the shared memory, so that no two share an SM: what they need (103 KB) leaves room for two, and they were placed in pairs as the
// predecessor's CTAs left, in some runs and not in others (320 tokens 58 us always, 512 tokens 57 or 90; alone 36 and 56).
#pragma once
#include "wkv_seq.cuh"

namespace rsv {

constexpr int kWcT = 16;       // tokens of a chunk
// Tokens of the shortest segment.  A layer in us, token by token and in chunks (8, 40 and 64 heads): 96 tokens 84.8 and 86.1, 128.2 and 133.0, 178.4 and 185.6; 128 tokens
// 98.0 and 96.6, 147.3 and 145.5, 204.3 and 204.9; 160 tokens 108.9 and 100.7, 166.9 and 162.2, 255.3 and 251.9; 256 tokens 138 and 120, 227 and 209, 320 and 309.
constexpr int kWcMinLen = 160;
constexpr int kWcRows = 32;    // state rows of a CTA
constexpr int kWcXStride = 68;  // floats between the rows of K and R: eight lanes read eight rows, 16 bytes each, from different banks
constexpr int kWcConsumers = 128;
constexpr int kWcThreads = kWcConsumers + 32;  // + the producer's warp
constexpr int kWcPrepThreads = 128;
constexpr int kWcStages = 3;
// Scratch of a (chunk, head), in floats: [K 16 rows, R 16 rows][b^ 16, k^ 16 rows of 64][W_16: 64][two parts of: UV, v, YV, each 16 x 32]
constexpr int kWcX = 2 * kWcT * kWcXStride, kWcZ = 2 * kWcT * 64, kWcPart = 3 * kWcT * kWcRows;
constexpr int kWcHeadFloats = kWcX + kWcZ + 64;
constexpr int kWcFloats = kWcHeadFloats + 2 * kWcPart;
constexpr int kWcStageFloats = kWcHeadFloats + kWcPart;
constexpr int kWcSStride = 20;  // floats between rows of a warp's 32 x 16 piece of the state
constexpr int kWcSumStride = 40;  // floats between the tokens of the warps' sums
constexpr size_t kWcSmemBytes = (size_t)(kWcStages * kWcStageFloats + 4 * 2 * kWcT * kWcSumStride + 4 * kWcRows * kWcSStride + kWcT * kWcRows) * 4 + 128;
constexpr size_t kWcSmemAlone = 120 * 1024;  // (see above)
static_assert(kWcSmemBytes <= kWcSmemAlone);

__host__ __device__ inline int wkv_chunks_of(int len) { return (len + kWcT - 1) / kWcT; }

// The inputs of the WKV kernels of a step (token rows [R, C]) and the head parameters [C].
struct WkvArgs {
    const SegMeta* segs;  // chunk0: chunks of the segments before
    const float *r, *k, *v, *vgate, *vfirst, *w, *a;
    const float *k_k, *k_a;
    float *state, *v_first_state, *yg, *tmp;
    int nseg, H, C;
    int* status;
};

// sums of v[0 .. 7] over the warp; lane l holds the one of index (l >> 2) & 7 (bits 4, 3, 2 of the lane: index bits 2, 1, 0)
__device__ __forceinline__ float wc_sum8(float (&v)[8], int lane) {
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) {
        const bool up = lane & (4 * m);
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const float send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * m);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__global__ void __launch_bounds__(kWcPrepThreads, 5) wkv7_prepare_kernel(const __grid_constant__ WkvArgs P) {
    constexpr int N = kHeadSize, T = kWcT;
    __shared__ __align__(16) float xs[2 * T][kWcXStride], zs[2 * T][kWcXStride];  // kk^, r^ / b^, k^
    __shared__ __align__(16) float vs[T][N];
    __shared__ __align__(16) float gram[4][T][T];  // A, B, E, F
    __shared__ float ssp[2][T];
    __shared__ double wtot[2][N];
    const int h = blockIdx.x, chunk = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    int lo = 0, hi = P.nseg;  // the last segment with at most `chunk` chunks before it
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.segs[mid].chunk0 <= chunk) lo = mid;
        else hi = mid;
    }
    const SegMeta sg = P.segs[lo];
    const int t0 = (chunk - sg.chunk0) * T, nt = min(T, sg.len - t0);
    const int c = tid & (N - 1), half = tid >> 6, hc = h * N, C = P.C;  // thread: channel c, tokens 8 half .. 8 half + 7
    const float kkc = P.k_k[hc + c], kac = P.k_a[hc + c];
    pdl_wait();
    const float *r = pdl_fresh(P.r), *k = pdl_fresh(P.k), *v = pdl_fresh(P.v), *vgate = pdl_fresh(P.vgate), *vfirst = pdl_fresh(P.vfirst), *w = pdl_fresh(P.w),
                *a = pdl_fresh(P.a);
    float* out = P.tmp + ((size_t)chunk * P.H + h) * kWcFloats;
    {
        float kv[8], rv[8], wv[8], av[8], vv[8];
        const size_t base = (size_t)(sg.start + t0) * C + hc + c;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = 8 * half + i;
            const size_t p = base + (size_t)min(t, nt - 1) * C;
            kv[i] = k[p];
            rv[i] = r[p];
            wv[i] = w[p];
            av[i] = a[p];
            vv[i] = v[p];
            if (vgate) vv[i] = vv[i] + vgate[p] * (vfirst[p] - vv[i]);
        }
        float sq[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float kk = kv[i] * kkc;
            sq[i] = kk * kk;
        }
        const float s8 = wc_sum8(sq, lane);
        if ((lane & 3) == 0) ssp[warp & 1][8 * half + (lane >> 2)] = s8;
        // products of the decays over this thread's tokens; tokens past the end leave the state as it is
        double W[8], run = 1.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (8 * half + i < nt) run *= wv[i];
            W[i] = run;
        }
        wtot[half][c] = run;
        __syncthreads();
        const double before = half ? wtot[0][c] : 1.0;
        if (half) out[kWcX + kWcZ + c] = (float)(before * run);
        double suf = half ? 1.0 : wtot[1][c];  // product of the decays after the token
#pragma unroll
        for (int i = 7; i >= 0; --i) {
            const int t = 8 * half + i;
            const bool on = t < nt;
            const double wp = before * (i ? W[i - 1] : 1.0), wt = before * W[i];
            double iw = (double)(1.0f / (float)wt);
            iw *= 2.0 - wt * iw;
            const float inv = 1.0f / fmaxf(sqrtf(ssp[0][t] + ssp[1][t]), kL2Eps);
            const float kh = kv[i] * kkc * inv, kt = kv[i] + kac * (kv[i] * av[i] - kv[i]);
            const float bh = on ? kh * (-av[i]) : 0.f, kth = on ? kt : 0.f;
            xs[t][c] = on ? (float)(wp * kh) : 0.f;
            xs[T + t][c] = on ? (float)(wt * rv[i]) : 0.f;
            zs[t][c] = (float)(bh * iw);
            zs[T + t][c] = (float)(kth * iw);
            vs[t][c] = on ? vv[i] : 0.f;
            out[kWcX + t * N + c] = (float)(bh * suf);
            out[kWcX + (T + t) * N + c] = (float)(kth * suf);
            if (on) suf *= wv[i];
            out[kWcHeadFloats + (c >> 5) * kWcPart + (T + t) * kWcRows + (c & 31)] = on ? vv[i] : 0.f;
            if (P.v_first_state && t0 + t == sg.len - 1) P.v_first_state[(size_t)sg.slot * C + hc + c] = vv[i];
        }
    }
    __syncthreads();
    {
        // the four 16 x 16 products: a thread has rows ty of kk^ and of r^, columns tx and tx + 8 of b^ and of k^
        const int ty = tid >> 3, tx = tid & 7;
        double sum[2][4] = {};
#pragma unroll
        for (int j0 = 0; j0 < N; j0 += 16) {
            float acc[2][4][4];
#pragma unroll
            for (int j = j0; j < j0 + 16; j += 4) {
                float4 x[2], z[4];
#pragma unroll
                for (int i = 0; i < 2; ++i) x[i] = *reinterpret_cast<const float4*>(&xs[T * i + ty][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) z[i] = *reinterpret_cast<const float4*>(&zs[8 * i + tx][j]);
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float(&a4)[4] = acc[p][q];
                        const bool first = j == j0;
                        a4[0] = first ? x[p].x * z[q].x : fmaf(x[p].x, z[q].x, a4[0]);
                        a4[1] = first ? x[p].y * z[q].y : fmaf(x[p].y, z[q].y, a4[1]);
                        a4[2] = first ? x[p].z * z[q].z : fmaf(x[p].z, z[q].z, a4[2]);
                        a4[3] = first ? x[p].w * z[q].w : fmaf(x[p].w, z[q].w, a4[3]);
                    }
            }
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) sum[p][q] += (double)((acc[p][q][0] + acc[p][q][1]) + (acc[p][q][2] + acc[p][q][3]));
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) gram[2 * p + (q >> 1)][ty][8 * (q & 1) + tx] = (float)sum[p][q];
    }
    __syncthreads();
    {
        // a thread solves one column of the triangular system: column c of kk^ (half 0) or of B v (half 1)
        // (the solution's even and odd terms are added apart; R and YV, which go into y as they are, in groups of four that are joined in double)
        float* o = half == 0 ? out + c : out + kWcHeadFloats + (c >> 5) * kWcPart + (c & 31);
        const int step = half == 0 ? kWcXStride : kWcRows, second = half == 0 ? T * kWcXStride : 2 * T * kWcRows;
        float x[T], vc[T];
#pragma unroll
        for (int t = 0; t < T; ++t) vc[t] = half ? vs[t][c] : 0.f;
#pragma unroll
        for (int t = 0; t < T; ++t) {
            float p[2] = {0.f, 0.f};
            if (half == 0) {
                x[t] = xs[t][c];
            } else {
                float b[2] = {0.f, 0.f};
#pragma unroll
                for (int s = 0; s < t; ++s) b[s & 1] = fmaf(gram[1][t][s], vc[s], b[s & 1]);
                x[t] = b[0] + b[1];
            }
#pragma unroll
            for (int s = 0; s < t; ++s) p[s & 1] = fmaf(gram[0][t][s], x[s], p[s & 1]);
            x[t] += p[0] + p[1];
            double z = half == 0 ? (double)xs[T + t][c] : 0.0;
#pragma unroll
            for (int s0 = 0; s0 <= t; s0 += 4) {
                float q = 0.f;
#pragma unroll
                for (int s = s0; s < s0 + 4 && s <= t; ++s) q = fmaf(gram[2][t][s], x[s], q);
                z += (double)q;
            }
            if (half)
#pragma unroll
                for (int s0 = 0; s0 <= t; s0 += 4) {
                    float q = 0.f;
#pragma unroll
                    for (int s = s0; s < s0 + 4 && s <= t; ++s) q = fmaf(gram[3][t][s], vc[s], q);
                    z += (double)q;
                }
            o[t * step] = x[t];
            o[second + t * step] = (float)z;
        }
    }
}

// Grid (2 H, segments).  Four consumer warps, one producer.  Warp wc has columns 16 wc .. 16 wc + 15 of the CTA's 32 rows, in registers (four rows x
// four columns per lane) and, for the products with K and R, in shared memory.
__global__ void __launch_bounds__(kWcThreads) wkv7_chunk_kernel(const __grid_constant__ WkvArgs P) {
    constexpr int N = kHeadSize, T = kWcT;
    extern __shared__ __align__(16) float wc_smem[];
    __shared__ __align__(8) uint64_t full[kWcStages], empty[kWcStages];
    __shared__ int s_abort;
    const SegMeta sg = P.segs[blockIdx.y];
    const int h = blockIdx.x >> 1, part = blockIdx.x & 1, H = P.H, C = P.C, tid = threadIdx.x, lane = tid & 31, wc = tid >> 5;
    float* stage = reinterpret_cast<float*>(((uintptr_t)wc_smem + 127) & ~(uintptr_t)127);
    float* sums = stage + kWcStages * kWcStageFloats;     // [warp][token of u, token of y][32 rows], 40 floats apart
    float* pieces = sums + 4 * 2 * T * kWcSumStride;      // [warp][32 rows][16 columns], 20 floats apart
    float* us = pieces + 4 * kWcRows * kWcSStride;        // [token][32 rows]
    volatile int* abort_flag = &s_abort;
    const int nc = (sg.len + T - 1) / T;
    if (tid == 0) {
        for (int i = 0; i < kWcStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], kWcConsumers / 32);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch_dependents();
    const int lr = lane >> 2, lc = lane & 3;  // rows 4 lr .. 4 lr + 3, columns 4 lc .. 4 lc + 3 of the warp's piece
    float* srow = P.state + (((size_t)sg.slot * H + h) * N + part * kWcRows + 4 * lr) * N + 16 * (wc & 3) + 4 * lc;
    float S[4][4];
    if (wc < 4)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4*>(srow + i * N);
            S[i][0] = t.x, S[i][1] = t.y, S[i][2] = t.z, S[i][3] = t.w;
        }
    __syncthreads();  // barriers initialised
    pdl_wait();
    if (wc == 4) {
        // ---- producer: chunk n -> stage n mod 3 ----
        if (lane == 0) {
            const float* src = pdl_fresh(P.tmp) + ((size_t)sg.chunk0 * H + h) * kWcFloats;
            int n = 0;
#pragma unroll 1
            for (; n < nc; ++n, src += (size_t)H * kWcFloats) {
                const int sl = n % kWcStages;
                if (n >= kWcStages && !mbar_wait(&empty[sl], (uint32_t)(n / kWcStages - 1) & 1u, abort_flag)) break;
                float* dst = stage + sl * kWcStageFloats;
                mbar_expect_tx(&full[sl], kWcStageFloats * 4);
                bulk_load(dst, src, kWcHeadFloats * 4, &full[sl]);
                bulk_load(dst + kWcHeadFloats, src + kWcHeadFloats + part * kWcPart, kWcPart * 4, &full[sl]);
            }
            if (*abort_flag)  // copies in flight land before the CTA may exit
                for (int m = max(0, n - kWcStages); m < n; ++m)
                    for (uint32_t i = 0; i < (1u << 16); ++i)
                        if (mbar_try_wait(&full[m % kWcStages], (uint32_t)(m / kWcStages) & 1u)) break;
        }
        return;
    }
    float* piece = pieces + wc * kWcRows * kWcSStride;
    const int so = tid >> 2, sr = 8 * (tid & 3);  // this thread's share of the sums: token so (0-15 u, 16-31 y), rows sr .. sr + 7
    bool ok = true;
    // every warp takes every turn (the barriers below); after a time-out without waiting and without output
#pragma unroll 1
    for (int n = 0; n < nc; ++n) {
        const int sl = n % kWcStages;
        const float* X = stage + sl * kWcStageFloats;
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(piece + (4 * lr + i) * kWcSStride + 4 * lc) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
        __syncwarp();
        ok = ok && mbar_wait(&full[sl], (uint32_t)(n / kWcStages) & 1u, abort_flag);
        {
            // ---- S0 (K, R) over the warp's columns: rows 4 lr .. 4 lr + 3, tokens lc, lc + 4, ... ----
            float acc[4][8] = {};
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                float4 s[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i] = *reinterpret_cast<const float4*>(piece + (4 * lr + i) * kWcSStride + j);
#pragma unroll
                for (int o = 0; o < 8; ++o) {
                    const float4 x = *reinterpret_cast<const float4*>(X + (4 * o + lc) * kWcXStride + 16 * wc + j);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][o] = fmaf(s[i].w, x.w, fmaf(s[i].z, x.z, fmaf(s[i].y, x.y, fmaf(s[i].x, x.x, acc[i][o]))));
                }
            }
#pragma unroll
            for (int o = 0; o < 8; ++o) *reinterpret_cast<float4*>(sums + (wc * 2 * T + 4 * o + lc) * kWcSumStride + 4 * lr) = make_float4(acc[0][o], acc[1][o], acc[2][o], acc[3][o]);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kWcConsumers) : "memory");
        // ---- add the four warps' sums and the part that comes from v ----
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const float* uv = X + kWcHeadFloats + (so < T ? so : so + T) * kWcRows + sr + 4 * q;  // [UV][v][YV]
            float4 t = *reinterpret_cast<const float4*>(uv);
            float4 d[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] = *reinterpret_cast<const float4*>(sums + (i * 2 * T + so) * kWcSumStride + sr + 4 * q);
            t.x += (d[0].x + d[1].x) + (d[2].x + d[3].x);
            t.y += (d[0].y + d[1].y) + (d[2].y + d[3].y);
            t.z += (d[0].z + d[1].z) + (d[2].z + d[3].z);
            t.w += (d[0].w + d[1].w) + (d[2].w + d[3].w);
            if (so < T) {
                *reinterpret_cast<float4*>(us + so * kWcRows + sr + 4 * q) = t;
            } else {
                const int tok = n * T + so - T;
                if (tok < sg.len && ok) *reinterpret_cast<float4*>(P.yg + (size_t)(sg.start + tok) * C + h * N + part * kWcRows + sr + 4 * q) = t;
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kWcConsumers) : "memory");
        // ---- S = S0 diag(W) + (sum u b + sum v k): the old state is rounded once per chunk, whatever its size against the sums ----
        const float *bz = X + kWcX + 16 * wc + 4 * lc, *kz = bz + T * 64, *vr = X + kWcHeadFloats + T * kWcRows + 4 * lr, *ur = us + 4 * lr;
        const float4 W = *reinterpret_cast<const float4*>(X + kWcX + kWcZ + 16 * wc + 4 * lc);
        float B[4][4] = {}, D[4][4] = {};
#pragma unroll
        for (int s = 0; s < T; ++s) {
            const float4 u = *reinterpret_cast<const float4*>(ur + s * kWcRows), v = *reinterpret_cast<const float4*>(vr + s * kWcRows);
            const float4 b = *reinterpret_cast<const float4*>(bz + s * 64), k = *reinterpret_cast<const float4*>(kz + s * 64);
            const float uu[4] = {u.x, u.y, u.z, u.w}, vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                B[i][0] = fmaf(uu[i], b.x, B[i][0]);
                B[i][1] = fmaf(uu[i], b.y, B[i][1]);
                B[i][2] = fmaf(uu[i], b.z, B[i][2]);
                B[i][3] = fmaf(uu[i], b.w, B[i][3]);
                D[i][0] = fmaf(vv[i], k.x, D[i][0]);
                D[i][1] = fmaf(vv[i], k.y, D[i][1]);
                D[i][2] = fmaf(vv[i], k.z, D[i][2]);
                D[i][3] = fmaf(vv[i], k.w, D[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            S[i][0] = fmaf(S[i][0], W.x, B[i][0]) + D[i][0];
            S[i][1] = fmaf(S[i][1], W.y, B[i][1]) + D[i][1];
            S[i][2] = fmaf(S[i][2], W.z, B[i][2]) + D[i][2];
            S[i][3] = fmaf(S[i][3], W.w, B[i][3]) + D[i][3];
        }
        __syncwarp();  // every lane has read the stage and the piece
        if (lane == 0) mbar_arrive(&empty[sl]);
    }
    if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
        for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(srow + i * N) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    } else if (lane == 0) {
        atomicOr(P.status, 16);
    }
}

}  // namespace rsv
