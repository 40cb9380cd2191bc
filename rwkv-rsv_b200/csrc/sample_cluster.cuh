// Sampling with one cluster of CTAs per logits row.  Same specification as sample_rows_kernel (kernels.cuh): penalties -> temperature ->
// top-k -> softmax -> top-p -> draw, the general path of rwkv_sample(_batch) (src/backend_cuda.rs:3741-3769, 3835-3908, 3923-4006).
//
// A row of 65536 logits in one CTA made about ten passes over global memory with 1024 threads: 218 us per step, on one SM per session,
// between two steps that wait for it.  Here a CTA holds 8192 logits in registers (sixteen consecutive ones per thread), a row is a
// cluster of up to eight CTAs, and the logits are read once.  What is left is a chain of block and cluster barriers, so the exchanges
// are built to need few: every CTA reads the others' results through distributed shared memory and repeats the small joint steps
// itself, instead of one CTA doing them and broadcasting.
//   maximum          one value per CTA
//   k-th largest     a histogram of (max - l) in 512 linear bins finds the bin where the k-th largest lies; the elements of the bins up to
//                    it (a few hundred) are collected and sorted by every CTA.  Where the collection would not fit 1024 entries (nearly
//                    equal logits, or a large k) the bits of the k-th largest are found by four 8-bit radix passes instead.
//   top-p            a walk over the sorted list (k <= 512: the top-k list serves both)
//   draw             prefix sums in vocabulary order: thread, block, cluster
// Measured, 65536 logits: one row, top-k 50 + top-p 23 us (218 in one CTA, 24 before the walk below took eight entries at a time and the sort dropped block
// barriers within a warp); 1024 rows of top-p alone 1.09 ms (1.51).
#pragma once
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace rsv {

constexpr int kScThreads = 512;
constexpr int kScPer = 16;                       // consecutive logits per thread
constexpr int kScSeg = kScThreads * kScPer;      // logits per CTA
constexpr int kScMaxCtas = 8;
constexpr int kScMaxV = kScSeg * kScMaxCtas;
constexpr int kScBins = kScThreads;              // one per thread
constexpr int kScList = 1024;

struct ScShared {
    uint32_t hist[kScBins];   // this CTA's histogram (read by the others)
    float local[kScList];     // this CTA's part of the collection (read by the others)
    int local_n;
    float xmax, xsum, xkept;  // this CTA's maximum, sum, kept sum (read by the others)
    int xchosen, xlast;       // this CTA's drawn token (V: none) and its last kept one (-1: none)
    alignas(16) float list[kScList];  // the collection, sorted (every CTA its own copy)
    float red[kScThreads / 32];
    uint32_t ured[kScThreads / 32];
    int cross, before;        // bin that holds the k-th largest; elements in the bins before it
    float cut;
    int chosen;
};

__device__ __forceinline__ uint32_t sc_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void sc_cluster_sync(int S) {
    if (S == 1) {
        __syncthreads();
    } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}
__device__ __forceinline__ uint32_t sc_remote_u32(const void* p, int rank) {
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float sc_remote_f32(const void* p, int rank) { return __uint_as_float(sc_remote_u32(p, rank)); }
__device__ __forceinline__ float sc_block_sum(float v, float* red) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = red[threadIdx.x & 15];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
// exclusive prefix sum of one value per thread over the CTA
__device__ __forceinline__ uint32_t sc_block_prefix(uint32_t v, uint32_t* red) {
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)(threadIdx.x & 31) >= o) incl += t;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 31) red[threadIdx.x >> 5] = incl;
    __syncthreads();
    uint32_t base = 0;
#pragma unroll
    for (int i = 0; i < kScThreads / 32; ++i)
        if (i < (int)(threadIdx.x >> 5)) base += red[i];
    return base + incl - v;
}
__device__ __forceinline__ int sc_bin(float l, float mx) {
    const float d = (mx - l) * 16.0f;  // monotone in l, so the bins are ordered like the values
    return d < (float)(kScBins - 1) ? max((int)d, 0) : kScBins - 1;
}

__global__ void __launch_bounds__(kScThreads, 2) sample_cluster_kernel(const float* __restrict__ logits, int V, const float* __restrict__ sampler8,
                                                                       const uint32_t* __restrict__ hist, int hist_stride, const int* __restrict__ round_cnt,
                                                                       uint32_t* __restrict__ next_tok, uint32_t* __restrict__ seq, int* __restrict__ seq_cnt,
                                                                       int seq_cap, const int* __restrict__ row_map, int S) {
    __shared__ ScShared sh;
    extern __shared__ uint32_t s_counter[];  // [8192] penalty histogram of this CTA's tokens
    const int tid = threadIdx.x, rank = S > 1 ? (int)sc_ctarank() : 0, row = (int)blockIdx.x / S;
    const int ent = row_map ? row_map[row] : row;  // entry of the per-session arrays (sampler rows, history, counters, tokens)
    const float* lg = logits + (size_t)row * V;
    const int i0 = rank * kScSeg + tid * kScPer;
    float x[kScPer];
    if ((V & 3) == 0 && (reinterpret_cast<uintptr_t>(lg) & 15) == 0) {  // (a caller's device array need not start at 16 bytes)
#pragma unroll
        for (int q = 0; q < kScPer / 4; ++q) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i0 + 4 * q < V) t = __ldcg(reinterpret_cast<const float4*>(lg + i0 + 4 * q));
            x[4 * q] = t.x, x[4 * q + 1] = t.y, x[4 * q + 2] = t.z, x[4 * q + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < kScPer; ++q) x[q] = i0 + q < V ? __ldcg(lg + i0 + q) : 0.f;
    }
    const int nv = max(0, min(kScPer, V - i0));  // this thread's logits
    const float* sp = sampler8 + (size_t)ent * 8;
    const float temperature = sp[0], top_p = sp[2], rep = sp[4], freq = sp[5], pres = sp[6];
    const uint32_t top_k = __float_as_uint(sp[1]);
    uint32_t seed = __float_as_uint(sp[3]), hist_len = __float_as_uint(sp[7]);
    if (round_cnt) {  // self-loop: round r uses seed + r and the r tokens generated so far
        const uint32_t round = (uint32_t)round_cnt[ent];
        seed += round;
        hist_len = min(round, (uint32_t)hist_stride);
    }
    const uint32_t* hrow = hist ? hist + (size_t)ent * hist_stride : nullptr;
    if (hist_len > 0u && hrow && (rep != 1.0f || freq != 0.0f || pres != 0.0f)) {
        for (int i = tid; i < kScSeg; i += kScThreads) s_counter[i] = 0u;
        __syncthreads();
        for (int h = tid; h < (int)hist_len; h += kScThreads) {
            const uint32_t t = hrow[h], o = t - (uint32_t)(rank * kScSeg);
            if (t < (uint32_t)V && o < (uint32_t)kScSeg) atomicAdd(&s_counter[o], 1u);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kScPer; ++q) {
            const uint32_t cnt = s_counter[tid * kScPer + q];
            if (cnt > 0u) {
                if (rep != 1.0f) x[q] = x[q] > 0.0f ? x[q] / rep : x[q] * rep;
                if (pres != 0.0f) x[q] -= pres;
            }
            if (freq != 0.0f) x[q] -= freq * (float)cnt;
        }
    }
    const float invT = temperature > 0.0f ? 1.0f / temperature : 1.0f;
    float mx = -1e30f;
#pragma unroll
    for (int q = 0; q < kScPer; ++q) {
        x[q] *= invT;
        if (x[q] < -3.0e38f) x[q] = -1e30f;  // masked tokens (-inf, the lowest float) count as -1e30, so that a row of nothing else is drawn from uniformly
        if (q < nv) mx = fmaxf(mx, x[q]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((tid & 31) == 0) sh.red[tid >> 5] = mx;
    sh.hist[tid] = 0u;
    if (tid == 0) sh.local_n = 0;
    __syncthreads();
    mx = sh.red[tid & 15];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (tid == 0) sh.xmax = mx;
    sc_cluster_sync(S);
#pragma unroll 1
    for (int c = 0; c < S; ++c) mx = fmaxf(mx, sc_remote_f32(&sh.xmax, c));

    // ---- k-th largest, and the sorted list of the elements down to it ----
    const bool use_k = top_k > 0u && top_k < (uint32_t)V, use_p = top_p > 0.0f && top_p < 1.0f;
    float thr = -3.0e38f;
    int m = 0;  // list entries that are >= the k-th largest
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
        // round 0: the top-k threshold; round 1: the 512 largest for top-p, unless the top-k list holds everything that is kept
        int K;
        if (round == 0) {
            if (!use_k) continue;
            K = (int)top_k;
        } else {
            if (!use_p || (use_k && top_k <= (uint32_t)kTopPMaxPicks)) continue;
            K = min(kTopPMaxPicks, V);
            if (use_k) {  // the histogram and the collection are used a second time
                sc_cluster_sync(S);
                sh.hist[tid] = 0u;
                if (tid == 0) sh.local_n = 0;
                __syncthreads();
            }
        }
#pragma unroll
        for (int q = 0; q < kScPer; ++q)
            if (q < nv) atomicAdd(&sh.hist[sc_bin(x[q], mx)], 1u);
        sc_cluster_sync(S);
        uint32_t cnt = 0;
#pragma unroll 1
        for (int c = 0; c < S; ++c) cnt += sc_remote_u32(&sh.hist[tid], c);
        const uint32_t pre = sc_block_prefix(cnt, sh.ured);
        if (pre < (uint32_t)K && pre + cnt >= (uint32_t)K) {  // exactly one thread
            sh.cross = tid;
            sh.before = (int)(pre + cnt);
        }
        __syncthreads();
        const int cross = sh.cross, n_in = sh.before;  // elements in the bins up to the crossing one
        float kth = 0.f;
        int n = n_in;
        if (n_in <= kScList) {
#pragma unroll
            for (int q = 0; q < kScPer; ++q)
                if (q < nv && sc_bin(x[q], mx) <= cross) sh.local[atomicAdd(&sh.local_n, 1)] = x[q];
        } else {
            // radix passes over the keys; a pass's histogram is read by all CTAs before the next one clears it
            uint32_t prefix = 0, mask = 0;
            int krem = K, equal = 0;
#pragma unroll 1
            for (int shift = 24; shift >= 0; shift -= 8) {
                sc_cluster_sync(S);
                sh.hist[tid] = 0u;
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kScPer; ++q) {
                    const uint32_t key = float_key(x[q]);
                    if (q < nv && (key & mask) == prefix) atomicAdd(&sh.hist[255u - ((key >> shift) & 255u)], 1u);
                }
                sc_cluster_sync(S);
                uint32_t c8 = 0;
                if (tid < 256)
#pragma unroll 1
                    for (int c = 0; c < S; ++c) c8 += sc_remote_u32(&sh.hist[tid], c);
                const uint32_t p8 = sc_block_prefix(c8, sh.ured);
                if (p8 < (uint32_t)krem && p8 + c8 >= (uint32_t)krem) {
                    sh.cross = 255 - tid;
                    sh.before = krem - (int)p8;
                    sh.chosen = (int)c8;
                }
                __syncthreads();
                prefix |= (uint32_t)sh.cross << shift;
                mask |= 255u << shift;
                krem = sh.before;
                equal = sh.chosen;
                __syncthreads();
            }
            kth = key_float(prefix);
            if (K <= kTopPMaxPicks) {
                // the elements above the k-th (K - krem of them); those equal to it are known without collecting them
#pragma unroll
                for (int q = 0; q < kScPer; ++q)
                    if (q < nv && float_key(x[q]) > prefix) sh.local[atomicAdd(&sh.local_n, 1)] = x[q];
            }
            n = K <= kTopPMaxPicks ? min(kTopPMaxPicks, K - krem + equal) : 0;
        }
        if (n > 0) {
            sc_cluster_sync(S);
            int at = 0;
#pragma unroll 1
            for (int c = 0; c < S; ++c) {
                const int nc = min((int)sc_remote_u32(&sh.local_n, c), kScList);
                for (int i = tid; i < nc; i += kScThreads)
                    if (at + i < kScList) sh.list[at + i] = sc_remote_f32(&sh.local[i], c);
                at += nc;
            }
            int np = 32;
            while (np < n) np <<= 1;
            for (int i = at + tid; i < np; i += kScThreads) sh.list[i] = i < n ? kth : -INFINITY;
            __syncthreads();
            // bitonic sort, descending (np <= 1024: a pair per thread).  Pairs up to 32 apart stay within the 64 entries of a warp: steps that follow
            // each other there need no block barrier (15 of the 55 steps of 1024 entries do).
#pragma unroll 1
            for (int kk = 2; kk <= np; kk <<= 1)
#pragma unroll 1
                for (int j = kk >> 1; j > 0; j >>= 1) {
                    if (tid < np / 2) {
                        const int a = 2 * tid - (tid & (j - 1)), b = a + j;
                        const float va = sh.list[a], vb = sh.list[b];
                        const bool desc = (a & kk) == 0;
                        if (desc ? va < vb : va > vb) {
                            sh.list[a] = vb;
                            sh.list[b] = va;
                        }
                    }
                    if (j > 32 || (j == 1 && kk >= 64))  // (the next step is kk's, j / 2 apart, or after j = 1 that of 2 kk, kk apart)
                        __syncthreads();
                    else
                        __syncwarp();
                }
            __syncthreads();
            kth = sh.list[K - 1];
            // entries >= kth: all of them are in the list
            const int lim = min(n, kTopPMaxPicks);
            m = K;
            while (m < lim && sh.list[m] == kth) ++m;
            m = min(m, kTopPMaxPicks);
        }
        if (round == 0) thr = kth;
    }

    // ---- softmax over what is kept ----
    float ps = 0.f;
    float e[kScPer];
    const float below = expf(-1e30f - mx);  // what a token under the threshold counts: 0, but 1 in a row of masked tokens only
#pragma unroll
    for (int q = 0; q < kScPer; ++q) {
        e[q] = q >= nv ? 0.f : x[q] < thr ? below : expf(x[q] - mx);  // (most warps have nothing above a top-k threshold and skip the rest)
        ps += e[q];
    }
    ps = sc_block_sum(ps, sh.red);
    if (tid == 0) sh.xsum = ps;
    sc_cluster_sync(S);
    float total = 0.f;
#pragma unroll 1
    for (int c = 0; c < S; ++c) total += sc_remote_f32(&sh.xsum, c);
    const float div = total > 0.0f ? total : 1.0f;
#pragma unroll
    for (int q = 0; q < kScPer; ++q) e[q] = e[q] / div;

    float cutoff = 0.0f;
    if (use_p) {
        for (int i = tid; i < m; i += kScThreads) sh.list[i] = expf(sh.list[i] - mx) / div;
        __syncthreads();
        if (tid == 0) {
            // picks from the largest down until the sum reaches top_p (at most 512); past the list only zeros follow
            // Eight at a time while their sum stays under top_p (the same additions in the same order; the chain is an addition per pick instead of a read, an
            // addition, a comparison and a branch)
            float cum = 0.0f, cut = 0.0f;
            int c = 0;
#pragma unroll 1
            for (; c + 8 <= m; c += 8) {
                const float4 p = *reinterpret_cast<const float4*>(&sh.list[c]), q = *reinterpret_cast<const float4*>(&sh.list[c + 4]);
                const float t = (((((((cum + p.x) + p.y) + p.z) + p.w) + q.x) + q.y) + q.z) + q.w;
                if (!(t < top_p)) break;
                cum = t;
                cut = q.w;
            }
            for (; c < m && cum < top_p; ++c) {
                cut = sh.list[c];
                cum += cut;
            }
            if (cum < top_p && m < min(kTopPMaxPicks, V)) cut = 0.0f;
            sh.cut = cut;
        }
        __syncthreads();
        cutoff = sh.cut;
    }

    // ---- draw: first kept index, in vocabulary order, whose running sum exceeds u ----
    // Sums put together from different parts round differently, so a thread without kept tokens can start above what the one before it
    // reached; only kept tokens are looked at.  Where no sum exceeds u (u = the total), the last kept token is the answer.
    float csum = 0.f;
#pragma unroll
    for (int q = 0; q < kScPer; ++q) {
        if (e[q] < cutoff) e[q] = 0.0f;
        csum += e[q];
    }
    float incl = csum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if ((tid & 31) >= o) incl += t;
    }
    __syncthreads();
    if ((tid & 31) == 31) sh.red[tid >> 5] = incl;
    if (tid == 0) {
        sh.xchosen = V;
        sh.xlast = -1;
    }
    __syncthreads();
    float wbase = 0.f, kept = 0.f;
#pragma unroll
    for (int i = 0; i < kScThreads / 32; ++i) {
        if (i < (tid >> 5)) wbase += sh.red[i];
        kept += sh.red[i];
    }
    if (tid == 0) sh.xkept = kept;
    sc_cluster_sync(S);
    float base = 0.f, total2 = 0.f;
#pragma unroll 1
    for (int c = 0; c < S; ++c) {
        const float t = sc_remote_f32(&sh.xkept, c);
        if (c < rank) base += t;
        total2 += t;
    }
    const float u = u01(seed) * total2;
    float acc = base + wbase + incl - csum;  // exclusive prefix of this thread's range
    int mine = V, last = -1;
#pragma unroll
    for (int q = 0; q < kScPer; ++q) {
        acc += e[q];
        if (e[q] > 0.0f) {
            last = i0 + q;
            if (acc > u && mine == V) mine = i0 + q;
        }
    }
    if (mine < V) atomicMin(&sh.xchosen, mine);
    last = __reduce_max_sync(0xffffffffu, last);
    if ((tid & 31) == 0 && last >= 0) atomicMax(&sh.xlast, last);
    sc_cluster_sync(S);
    if (rank == 0 && tid == 0) {
        int tok = V;
#pragma unroll 1
        for (int c = 0; c < S; ++c) tok = min(tok, (int)sc_remote_u32(&sh.xchosen, c));
        if (tok == V) {
            tok = -1;
#pragma unroll 1
            for (int c = 0; c < S; ++c) tok = max(tok, (int)sc_remote_u32(&sh.xlast, c));
            if (tok < 0 || total2 != total2) tok = V - 1;  // nothing was kept, or a NaN among the probabilities
        }
        next_tok[ent] = (uint32_t)tok;
        if (seq) {
            const int c = seq_cnt[ent];
            if (c < seq_cap) seq[(size_t)ent * seq_cap + c] = (uint32_t)tok;
            seq_cnt[ent] = c + 1;
        }
    }
    sc_cluster_sync(S);  // no CTA leaves while its shared memory may be read
}

}  // namespace rsv
