// Batch-1 decode as a row-owner weight-streaming matrix-vector product inside one persistent launch.
//
// One cooperative launch runs n tokens x L layers x (head, arg-max) for ONE session: the launch stands in for the
// reference's captured-graph decode step (forward_token / forward_layer / selfloop_step, src/gpu_model.rs:1879-2392)
// and its weight-streaming GEMVs (gemv_variant, gemv_int8_rkv_stage1, gemv_f16; src/backend_cuda.rs:3229-3373,
// 2949-3152, 1421-1498), which read 4 rows per block with the dequantisation fused into the load.
//
// Decomposition.  CTA c (one per SM) owns output rows [c M / G, (c+1) M / G) of every matrix for the WHOLE K: no
// partial sums ever cross a CTA, so a phase is  activation vector -> dot products -> tagged stores.
//   warp 0      producer (its warpgroup's other warps idle).  Walks the fixed sequence of weight chunks this CTA will ever need - token after token, layer
//               after layer, phase after phase - and streams them with bulk asynchronous copies (cp.async.bulk) into a
//               byte-granular ring in shared memory; a chunk = one tile of up to 16 rows x one piece of K, one mbarrier
//               per chunk.  It never waits for other CTAs, only for ring space, so HBM keeps streaming while the other
//               warps wait for activations.
//   warps 4-19  consumers.  Warp w of them owns the w-th sixteenth of K of every matrix: it turns its sixteenth of the activation
//               vector into operand fragments itself (LayerNorm, token shift, fixed-point digits; only the row statistics
//               and the maximum cross warps) and multiplies its columns of every tile.  So all sixteen warps work on a
//               tile at once, an operand is read only by the warp that wrote it, and chunks are released in the order they
//               came.  The sixteen partial sums of a row meet in shared memory; four lanes per row add them and store.
// The weights are stored a second time in the order of the stream, each chunk as the A fragments of the matrix
// instruction ([step of 32 bytes][row][thread of the quad][8 bytes]: rows 0-7 of the tile, then rows 8-15), so a lane's
// operand is one conflict-free 8-byte read and a tile of fewer than 16 rows takes no padding.
// Arithmetic.  int8 matrices: the u8 codes q are multiplied as they are (m16n8k32, u8 x s8 -> s32) with the four
// signed base-256 digits of the fixed-point activation t = rint(x / e 2^30), e = 2^ceil(log2 max|x|) (the digits are
// the bytes of (t + 0x808080) ^ 0x808080); the four int32 sums recombine to Q = sum_k q_k t_k exactly (int64), and
// with the container's per-row (scale s, zero z)  y = e 2^-30 (s Q + z T), T = sum_k t_k: no accumulation rounding,
// no dependence on the schedule.  Rows with a (scale, zero) per group of 128 close the integer sums at every group
// boundary and accumulate in fp32.  fp16 matrices (head, rank projections, fp16 checkpoints): m16n8k16 f16 x f16 -> f32
// with x / e split into hi + lo halves (two operand columns).  These are 8-column problems that stream weights at
// HBM speed; the tensor pipe is nearly idle, which is why the warp-level instruction is the right size here and the
// tcgen05 kernels take over once several rows make the product a dense contraction.
// Phases per layer:
//   1  LN1 + token shift -> r, k, v and the four rank projections (tanh / sigmoid applied)
//   2  one CTA per head: rank back-projections (their rows arrive through the ring too), decay / a / v-gate / g,
//      WKV-7 state update in place, GroupNorm, bonus, gate
//   3  att.output, x += ...      4  LN2 + shift -> relu(ffn.key)^2      5  ffn.value, x += ...
// then ln_out + head -> logits, arg-max across CTAs, next token.
// Exchange between CTAs.  There is no grid barrier between the phases: every exchanged value carries the number of the layer it belongs
// to (8 bytes: value, tag; the non-negative hidden values of the ffn carry the parity of that number in their sign bit), and a
// reader polls the values it needs.  A barrier costs a release fence, an atomic, a poll and then the load of the data, 2.9 us from the
// last store to the data in registers with the weight stream running; polling the data is one store and one load.  A buffer may be
// overwritten for the next layer without further ado: nobody can produce a value of the next use before everybody has consumed this
// one (every output of a phase depends on every input of it).  State that is read a token later (the shift states) is ordered by the one
// grid barrier at the end of a token.
// What bounds it: the dependent chain of a layer, not HBM.  Its code is therefore written once and looped (phases 1, 3, 4, 5 and the
// head are the same code with other pointers): 32 KB of code run at an instruction per cycle, 128 KB at a third of that, more at less
// than a fifth; and nothing should spill: with the shared memory taken, the threads' stacks do not fit L1 and every spill is an L2 round
// trip (0.07 ms of a token's 1.40 with 128 bytes of spills; up to 2560 channels nothing does, the 4096-channel instantiation spills as much).
// Measured per token at 2560 channels, 32 layers, 65536 rows of vocabulary: int8 1.30 ms (3.0 GB: 0.47 ms at copy bandwidth), fp16
// 1.81 ms; 1.49 and 1.90 ms with a grid barrier after every phase and a tile of rows per warp; int8 per group 1.53 ms.  512 channels, 4 layers:
// 0.09 ms (0.13).  4096 channels, 32 layers: int8 2.47 ms.
// All waits are bounded; on expiry bit 5 of the status word is set (and the word after it says which wait), every role drains its copies in flight and exits.
#pragma once
#include <cstddef>

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace rsv {

constexpr int kDsConsumerWarps = 16;
constexpr int kDsConsumers = kDsConsumerWarps * 32;  // 512
constexpr int kDsThreads = kDsConsumers + 128;       // + the producer's warpgroup, of which one warp works
// Registers per thread.  Seventeen warps put five on one scheduler, so a thread can be launched with 96, and the consumers spilled; the
// producer's warpgroup gives some of its own to them (both then fit without a spill up to 2560 channels).
constexpr int kDsLaunchRegs = 96, kDsProducerRegs = 40, kDsConsumerRegs = 104;
static_assert(128 * kDsProducerRegs + kDsConsumers * kDsConsumerRegs <= kDsThreads * kDsLaunchRegs, "register split");
constexpr int kDsBars = 32;                          // chunks in flight (mbarrier pairs)
constexpr int kDsTileRows = 16;                      // rows of a tile (the m dimension of the matrix instruction)
constexpr int kDsPad = 0;                            // bytes between the rows of a chunk
constexpr int kDsMaxPiece = 2560;                    // bytes of K per piece: the head's rows
constexpr int kDsRankPiece = 1280;                   // ... the rank projections'
constexpr int kDsLayerPiece = 640;                   // ... the layers' big matrices (unless a sixteenth of K is longer)
constexpr int kDsPartInt = kDsConsumerWarps * 16 + 64;  // bytes per row of partial sums: four int32 digit sums per warp (+ padding against bank conflicts) ...
constexpr int kDsPartF32 = kDsConsumerWarps * 4 + 16;   // ... or one fp32 sum per warp
constexpr int kDsPartBytes = 5 * kDsTileRows * kDsPartInt;  // partial sums of a batch of tiles
constexpr int kDsRankTiles = 2;                      // tiles of rank-projection rows per CTA
constexpr int kDsMergeBytes = 24 * 1024;             // a tile of at most this many bytes is one chunk
constexpr int kDsMaxRank = 512;                      // longest rank-space vector
constexpr int kDsMaxSlice = 32;                      // channels of the residual stream per CTA
constexpr int kDsP = 30;                             // fixed-point bits of the activation digits
constexpr uint32_t kDsBarSpin = 1u << 22;

// What a finished dot product becomes.
enum DsOut : int { DSO_R = 0, DSO_K, DSO_V, DSO_MID_TANH, DSO_MID, DSO_MID_SIG, DSO_XADD, DSO_H, DSO_LOGITS };

// One matrix of a phase.
struct DsEntry {
    const char* base;     // fp16 [M,K] or u8 [M,K], row-major
    const float* wscale;  // int8: [M] per-row scale and zero of the container
    const float* wzero;
    const float* mix;     // rank projections: the token-shift mix vector of their input; null otherwise
    const uint32_t* sz;   // int8 with one (scale, zero) per row and group of 128 (is_i8 == 2): the container's [M, K/128] words, fp16 scale | fp16 zero << 16
    int M;                // output rows (0: the entry does not exist in this layer)
    int row_stride;       // bytes between rows
    int piece_bytes;      // bytes of K per piece (a multiple of 128, <= kDsMaxPiece)
    int npieces;          // pieces per row
    int is_i8;            // 0: fp16; 1: int8, one (scale, zero) per row (wscale, wzero); 2: int8, one per row and group of 128 (sz)
    int xvec;             // which vector of the phase's operand area the rows are multiplied with
    int out;              // DsOut
    int out_off;          // offset inside the rank-space vector for DSO_MID*
    int cta0, ncta;       // the rows are split over the ncta CTAs cta0, cta0 + 1, ... (mod G)
};
enum { DSE_W1 = 0, DSE_A1, DSE_G1, DSE_V1, DSE_WR, DSE_WK, DSE_WV, DSE_WO, DSE_WFK, DSE_WFV, DSE_COUNT };
struct DsLayer {
    DsEntry e[DSE_COUNT];
    const __half *w2, *a2, *v2, *g2;  // back-projections [C, mid] fp16
    const float *ln1_w, *ln1_b, *ln2_w, *ln2_b, *lnx_w, *lnx_b;
    const float *x_r, *x_k, *x_v, *ffn_x_k;
    const float *w0, *a0, *v0, *r_k, *k_k, *k_a;
};
struct DsParams {
    const DsLayer* layers;
    DsEntry head;
    const __half* emb;
    const float *ln0_w, *ln0_b, *lno_w, *lno_b;
    int L, C, H, F, V, wm, am, vm, gm;
    int slot;
    long long lay_x, lay_s;        // floats between consecutive layers of the shift states / the WKV states
    float *tmix_x, *wkv, *cmix_x;  // state bases (layer 0, slot 0)
    float* state_vfirst;           // [cap][C]
    // exchanged values: (value, tag) pairs, and for hbuf values with a parity in the sign
    unsigned long long *xa, *xb;   // [C] residual stream after ffn.value / after att.output
    unsigned long long *yg, *vfirst;  // [C]
    unsigned long long* rkv;       // [3][C]
    unsigned long long* mid;       // [wm+am+vm+gm]
    uint32_t* hbuf;                // [F]
    uint32_t epoch;                // tag of layer 0 of the launch's first token; layer l of token t: epoch + t L + l
    uint32_t* tokens;              // [1] current input token (read at start, written after arg-max)
    const uint32_t* tok_list;      // [n_tokens], used when tok_from_list
    uint32_t* seq;
    int* seq_cnt;
    int seq_cap;
    float* logits;  // [V]
    float* cand_val;
    int* cand_idx;  // [G]
    unsigned* grid_bar;
    int* status;
    int n_tokens, tok_from_list, argmax_feed;  // tok_from_list: 0 tokens[0], 1 tok_list, 2 tok0
    uint32_t tok0;
    unsigned bar_base;  // the grid barrier's counter when the launch begins (it only grows)
    const char* wstream;      // the layers' weights in consumption order: region (layer l, CTA c) at (l G + c) wslot
    long long wslot;
    const char* hstream;      // the head's rows in consumption order: region of CTA c at c hslot
    long long hslot;
    int ring_bytes;  // shared-memory ring
    int vec_floats;  // operand area, in 4-byte elements: max(4 C, F)
};

// ---- small helpers ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void ds_consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kDsConsumers) : "memory"); }
// The same, and whether any of the consumers passed `bad`: every exit on an error is taken by all of them together (a warp that left
// alone would leave the others in the next barrier).
__device__ __forceinline__ bool ds_consumer_sync_or(bool bad) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)bad), "n"(kDsConsumers)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ uint32_t ds_lds32(uint32_t saddr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}
__device__ __forceinline__ uint2 ds_lds64(uint32_t saddr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(saddr));
    return v;
}
__device__ __forceinline__ void ds_sts64(uint32_t saddr, uint32_t a, uint32_t b) { asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(saddr), "r"(a), "r"(b) : "memory"); }
__device__ __forceinline__ void ds_sts8(uint32_t saddr, uint32_t a) { asm volatile("st.shared.u8 [%0], %1;" ::"r"(saddr), "r"(a) : "memory"); }
__device__ __forceinline__ void ds_sts16(uint32_t saddr, unsigned short a) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(saddr), "h"(a) : "memory"); }
__device__ __forceinline__ void ds_sts32(uint32_t saddr, uint32_t a) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(saddr), "r"(a) : "memory"); }
// D += A (16 x 32 u8, row-major: sixteen weight rows; lo = rows 0-7, hi = rows 8-15) x B (32 x 8 s8: the activation digits, one per column)
__device__ __forceinline__ void ds_mma_i8(int (&c)[4], uint2 lo, uint2 hi, uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(b.x), "r"(b.y));
}
// D += A (16 x 16 f16: sixteen weight rows) x B (16 x 8 f16: hi and lo halves of the activations), fp32 accumulation
__device__ __forceinline__ void ds_mma_f16(float (&c)[4], uint2 lo, uint2 hi, uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(b.x), "r"(b.y));
}
// Bulk asynchronous copy global -> shared memory of this CTA (16-byte aligned addresses, size a multiple of 16), completion
// counted in bytes on `bar`.  Weights are read once per token: they are marked evict-first in L2 so that the small arrays and
// the recurrent state every phase re-reads stay resident.
__device__ __forceinline__ void ds_bulk_load(uint32_t dst_saddr, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst_saddr), "l"(src),
                 "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void ds_arrive(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// Wait that ignores the abort flag (used to drain copies in flight before leaving); still bounded.
__device__ __forceinline__ void ds_mbar_drain(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 20); ++i)
        if (mbar_try_wait(bar, parity)) return;
}
__device__ __forceinline__ float ds_pow2(int n) { return __int_as_float((n + 127) << 23); }
// exponent e of the power-of-two scale of a vector whose largest magnitude is `amax`
__device__ __forceinline__ int ds_exponent(float amax) {
    if (!(amax >= 1.0e-30f && amax < 3.0e38f)) return 0;
    const int bits = __float_as_int(amax), ex = (bits >> 23) - 127 + ((bits & 0x7FFFFF) ? 1 : 0);
    return max(-90, min(90, ex));
}
// first row of the share of virtual CTA index vc when M rows are split over n CTAs
__host__ __device__ inline int ds_row_begin(int vc, int M, int n) { return (int)(((long long)vc * M) / n); }
// the rows [r0, r0 + n) of entry E that CTA `cta` of G owns (n = 0: none)
__host__ __device__ inline void ds_rows_of(const DsEntry& E, int cta, int G, int& r0, int& n) {
    r0 = n = 0;
    if (E.M <= 0 || E.ncta <= 0) return;
    const int vc = ((cta - E.cta0) % G + G) % G;
    if (vc >= E.ncta) return;
    r0 = ds_row_begin(vc, E.M, E.ncta);
    n = ds_row_begin(vc + 1, E.M, E.ncta) - r0;
}
// bytes of the (scale, zero) words behind a chunk of rows with one per group of 128: [group of the piece][16 rows]
__host__ __device__ inline int ds_sz_bytes(const DsEntry& E) { return E.is_i8 == 2 ? (E.piece_bytes >> 7) * kDsTileRows * 4 : 0; }
__host__ __device__ inline int ds_chunk_bytes(const DsEntry& E, int nr) { return nr * (E.piece_bytes + kDsPad) + ds_sz_bytes(E); }
// the CTA that runs head h of layer l (H <= G: heads spread with a stride, rotated per layer so that the extra bytes of a
// head's back-projection rows do not always land on the same SMs); -1 when CTA `cta` has no head in that layer
__host__ __device__ inline int ds_head_of_cta(int cta, int l, int H, int G) {
    const int stride = G / H;
    const int d = ((cta - (l * 37) % G) % G + G) % G;
    if (d % stride) return -1;
    const int h = d / stride;
    return h < H ? h : -1;
}
__host__ __device__ inline int ds_pad16(int n) { return (n + 15) / 16 * 16; }
// two fp16 packed in a 32-bit register -> two floats
__device__ __forceinline__ float2 ds_half2_bits_to_float2(uint32_t u) {
    float2 f;
    asm("{\n\t.reg .f16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.f32.f16 %0, lo;\n\tcvt.f32.f16 %1, hi;\n\t}" : "=f"(f.x), "=f"(f.y) : "r"(u));
    return f;
}
// A chunk of weight rows: one tile (up to 16 rows of a matrix) x one piece of K.  The chunks a CTA consumes are the same in every
// layer (its row ranges do not change).  The table below lists them: it lays out the second copy of the weights; the decode kernel
// itself walks the same order from each matrix's row count and piece size.
struct DsChunk {
    int cb;            // bytes of the chunk
    int nr_steps;      // rows (<= 16) | 64-byte column steps of the piece << 16
    int piece_np;      // which piece of the rows' K | pieces per row << 16
    int e_flags_row0;  // matrix DSE_* (DSE_COUNT: the head) | flags << 8 (1: int8, 2: absent in layer 0, 4: a (scale, zero) per group) | first row of the tile (from the CTA's first row) << 16
    int stride;        // bytes of a row in the chunk
};
constexpr int kDsMaxChunks = 384;  // table entries per CTA: the chunks of a layer plus the head's
enum { DSP_P1 = 0, DSP_P3, DSP_P4, DSP_P5, DSP_HEAD, DSP_COUNT };
struct DsPlan {
    int er0[DSE_COUNT + 1], en[DSE_COUNT + 1];  // rows [er0, er0 + en) of every matrix (DSE_*; last: the head) this CTA owns: the same in all layers
    int rank_entry;                             // the rank projection whose rows this CTA owns (-1: none)
    int ph0[DSP_COUNT], phn[DSP_COUNT];         // the phases' ranges in ctab
    int phn_l0;                                 // chunks of phase 1 in layer 0 (no v-gate projection there)
    DsChunk ctab[kDsMaxChunks];
};
// Builds a CTA's plan: row ranges (the one place where the rows are divided), then the chunk table phase by phase (matrix after
// matrix, tile after tile, piece after piece).  `ents` = a layer's matrices (one with a v-gate projection).  Returns false when the
// table would overflow.  (The last argument is unused.)
__host__ __device__ inline bool ds_build_plan(DsPlan& pl, const DsEntry* ents, const DsEntry& head, int cta, int G, uint32_t) {
    for (int e = 0; e <= DSE_COUNT; ++e) {
        int r0, n;
        ds_rows_of(e == DSE_COUNT ? head : ents[e], cta, G, r0, n);
        pl.er0[e] = r0;
        pl.en[e] = n;
    }
    pl.rank_entry = -1;
    for (int e = DSE_W1; e <= DSE_V1; ++e)
        if (pl.en[e] > 0 && pl.rank_entry < 0) pl.rank_entry = e;
    const int first[DSP_COUNT] = {DSE_W1, DSE_WO, DSE_WFK, DSE_WFV, DSE_COUNT}, last[DSP_COUNT] = {DSE_WV, DSE_WO, DSE_WFK, DSE_WFV, DSE_COUNT};
    int k = 0;
    bool fits = true;
    pl.phn_l0 = 0;
    for (int ph = 0; ph < DSP_COUNT; ++ph) {
        pl.ph0[ph] = k;
        for (int e = first[ph]; e <= last[ph]; ++e) {
            const DsEntry& E = e == DSE_COUNT ? head : ents[e];
            const int n = pl.en[e];
            for (int row0 = 0; row0 < n; row0 += kDsTileRows) {
                const int nr = n - row0 < kDsTileRows ? n - row0 : kDsTileRows;
                for (int p = 0; p < E.npieces; ++p) {
                    if (k >= kDsMaxChunks) {
                        fits = false;
                        continue;
                    }
                    DsChunk& c = pl.ctab[k++];
                    c.stride = E.piece_bytes + kDsPad;
                    c.cb = ds_chunk_bytes(E, nr);
                    c.nr_steps = nr | ((E.piece_bytes >> 6) << 16);
                    c.piece_np = p | (E.npieces << 16);
                    c.e_flags_row0 = e | ((E.is_i8 ? 1 : 0) << 8) | ((e == DSE_V1 ? 2 : 0) << 8) | ((E.is_i8 == 2 ? 4 : 0) << 8) | (row0 << 16);
                    if (ph == DSP_P1 && e != DSE_V1) ++pl.phn_l0;
                }
            }
        }
        pl.phn[ph] = k - pl.ph0[ph];
    }
    return fits;
}

// What a consumer needs to know about the rows of one matrix (shared memory, filled once per launch).
struct DsRows {
    int r0, n, tiles;  // rows [r0, r0 + n), tiles of 16
    int np, piece;     // pieces per row, bytes per piece
    int steps, spp;    // 32-byte steps of a whole row, of a piece
    int fmt;           // 0 fp16, 1 int8 with a (scale, zero) per row, 2 per group of 128
    int out, out_off;
    int full_bytes, last_bytes;  // bytes of a chunk of 16 rows, and of one of the last tile
    int merged;                  // the last tile's pieces, few rows, come as one chunk: the producer takes about 0.2 us per chunk
};

// ---- shared-memory layout: [ring][operand area: vec_floats x 4 bytes][DsShared] ----------------
constexpr int kDsMaxWarpSteps = 64;  // 32-byte steps of a warp's sixteenth of the longest row
struct DsShared {
    uint64_t full[kDsBars], empty[kDsBars];
    int alloc[kDsBars];     // producer only: bytes (with wrap waste) a chunk in flight holds
    int ring_off[kDsBars];  // where the chunk on a barrier pair landed (written by the producer before it arms the barrier)
    int abort_flag;
    int abort_where;  // which wait gave up first (1 rows: full, 2 producer: empty, 3 grid barrier, 4 heads: full) | detail << 4
    uint32_t tok;
    // Exchanged between the consumer warps, one array per use: 0, 1 row sums (LayerNorm; ||kk||^2 and bonus; arg-max), 2, 3 GroupNorm
    // sums, 2, 5 operand maxima, 4 scales of a head's rank vectors.  An array may be written again only after a barrier that follows its
    // last read; between a head's last sum (3) and the maxima of the next unit (2, 5) there is none.
    float red[6][16];
    int red_i[16];
    long long tsw[16];                       // per warp: exact sum of its fixed-point values
    float tstep[16][kDsMaxWarpSteps];        // per warp and step: the same as fp32 (rows with a (scale, zero) per group)
    float xs_own[kDsMaxSlice];               // this CTA's slice of the residual stream
    float ts_own[kDsMaxSlice];               // pending time-mix shift state of the slice
    float cs_own[kDsMaxSlice];               // pending channel-mix shift state of the slice
    alignas(16) float hv[14 * 64];           // the 64-vectors of a head
    DsRows rows[DSE_COUNT + 1];
    int rank_entry, big_entry;               // the rank projection (-1: none) and the one of receptance, key, value this CTA owns rows of
    alignas(16) char part[kDsPartBytes + kDsRankTiles * kDsTileRows * kDsPartF32];
    DsLayer layer[2];                        // table of the current / next layer
};

// Operand area.  Vector v of a phase (`len` elements) occupies 4 len bytes, stored as the B fragments the consumer lanes read (8 bytes):
//   int8 matrices: [k / 32][digit 0..3][t = (k % 16) / 4][word (k % 32) / 16], the word holding the digit of four consecutive k;
//   fp16 matrices: [k / 16][0 = hi, 1 = lo][t = (k % 8) / 2][word (k % 16) / 8], the word holding the halves of k, k + 1.
// Element k of a vector (32 lanes write 32 consecutive elements: no bank conflicts); returns its fixed-point value (int8).
__device__ __forceinline__ int ds_put(bool i8, uint32_t vec_s, int k, float x, float mult) {
    if (i8) {
        const int t = __float2int_rn(x * mult);  // |t| <= 2^30; a NaN converts to 0
        const uint32_t u = ((uint32_t)t + 0x00808080u) ^ 0x00808080u;  // bytes = signed base-256 digits of t
        const uint32_t dst = vec_s + (uint32_t)(k >> 5) * 128u + (uint32_t)((k >> 2) & 3) * 8u + (uint32_t)((k >> 4) & 1) * 4u + (uint32_t)(k & 3);
        ds_sts8(dst, u);
        ds_sts8(dst + 32, u >> 8);
        ds_sts8(dst + 64, u >> 16);
        ds_sts8(dst + 96, u >> 24);
        return t;
    }
    const float f = fminf(fmaxf(x * mult, -1.0f), 1.0f);
    const __half hi = __float2half_rn(f), lo = __float2half_rn(f - __half2float(hi));
    const uint32_t dst = vec_s + (uint32_t)(k >> 4) * 64u + (uint32_t)((k >> 1) & 3) * 8u + (uint32_t)((k >> 3) & 1) * 4u + (uint32_t)(k & 1) * 2u;
    ds_sts16(dst, __half_as_ushort(hi));
    ds_sts16(dst + 32, __half_as_ushort(lo));
    return 0;
}
// exact sum over the warp
__device__ __forceinline__ long long ds_warp_sum_int(int v) {
    const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)(v & 0xFFFF));
    const int hi = __reduce_add_sync(0xffffffffu, v >> 16);
    return (long long)hi * 65536 + (long long)lo;
}

// ---- exchanged values --------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long ds_pair(float v, uint32_t tag) { return (unsigned long long)__float_as_uint(v) | ((unsigned long long)tag << 32); }
__device__ __forceinline__ void ds_put_pair(unsigned long long* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(ds_pair(v, tag)) : "memory");
}
__device__ __forceinline__ unsigned long long ds_get_pair(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ds_get_word(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// A spin loop's turn: false when the limit is reached or another role gave up (then `where` is recorded).
__device__ __forceinline__ bool ds_spin_ok(DsShared* S, uint32_t& turns, int where) {
    if (++turns < kDsBarSpin && !((turns & 255u) == 255u && *(volatile int*)&S->abort_flag)) return true;
    atomicCAS(&S->abort_where, 0, where);
    *(volatile int*)&S->abort_flag = 1;
    return false;
}
// N elements base[first + 32 i] (i < N, those below end) carrying `tag`: all are requested at once, those that are not there yet again.
template <int N>
__device__ __forceinline__ bool ds_poll_pairs(DsShared* S, const unsigned long long* base, int first, int end, uint32_t tag, float (&v)[N], int where) {
    unsigned long long r[N];
    uint32_t turns = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = first + 32 * i < end ? ds_get_pair(base + first + 32 * i) : (unsigned long long)tag << 32;
    for (;;) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < N; ++i) all = all && (uint32_t)(r[i] >> 32) == tag;
        if (all) break;
        if (!ds_spin_ok(S, turns, where)) {
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = 0.f;
            return false;
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            if ((uint32_t)(r[i] >> 32) != tag) r[i] = ds_get_pair(base + first + 32 * i);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __uint_as_float((uint32_t)r[i]);
    return true;
}

// Steps [0, ns) of one tile with fp16 weights: lo / hi = this lane's addresses in rows 0-7 / 8-15, advancing by lstep / hstep per step.
__device__ __forceinline__ void ds_tile_f16(float (&c)[4], uint32_t lo, uint32_t lstep, uint32_t hi, uint32_t hstep, uint32_t b, int ns) {
    float c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = 0.f;
    int s = 0;
#pragma unroll 2
    for (; s + 2 <= ns; s += 2) {
        const uint2 al = ds_lds64(lo), ah = ds_lds64(hi), bb = ds_lds64(b);
        const uint2 bl = ds_lds64(lo + lstep), bh = ds_lds64(hi + hstep), b2 = ds_lds64(b + 64);
        ds_mma_f16(c, al, ah, bb);
        ds_mma_f16(c1, bl, bh, b2);
        lo += 2 * lstep;
        hi += 2 * hstep;
        b += 128;
    }
    if (s < ns) ds_mma_f16(c, ds_lds64(lo), ds_lds64(hi), ds_lds64(b));
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += c1[i];
}

// Tiles [tile0, tile1) of one matrix: this warp's sixteenth of K of every tile, partial sums to `part_s` ([row from tile0][warp]).
// J = the launch's index of the first chunk of tile0; a tile has np chunks, of which the warp reads one, shared with 16 / np - 1
// neighbours (a last tile of few rows is one chunk).  Lanes of rows that a tile does not have read another row's data; their sums are never looked at.  Returns false after a
// timeout.
__device__ __forceinline__ bool ds_multiply(DsShared* S, const DsRows* E, uint32_t ring_s, uint32_t vec_s, uint32_t part_s, uint32_t J, int tile0, int tile1, int w, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const int np = E->np, steps = E->steps, spp = E->spp, w0 = (w * steps) >> 4, piece = (w * np) >> 4, s0 = w0 - piece * spp, ns = (((w + 1) * steps) >> 4) - w0;
    const int fmt = E->fmt, n = E->n, merged = E->merged ? E->tiles - 1 : -1;
    const uint32_t bb = vec_s + (uint32_t)w0 * (fmt ? 128u : 64u) + (uint32_t)(g & (fmt ? 3 : 1)) * 32u + (uint32_t)t * 8u;
    uint32_t j = J + (uint32_t)piece;
    uint32_t dst = part_s + (fmt == 1 ? (uint32_t)(g * kDsPartInt + w * 16 + t * 8) : (uint32_t)(g * kDsPartF32 + w * 4));
#pragma unroll 1
    for (int tile = tile0; tile < tile1; ++tile, j += (uint32_t)np) {
        const bool one = tile == merged;
        if (one) j -= (uint32_t)piece;
        const int slot = (int)(j % kDsBars);
        const bool got = mbar_wait(&S->full[slot], (j / kDsBars) & 1u, (volatile int*)&S->abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
            if (lane == 0) atomicCAS(&S->abort_where, 0, 1 | (int)((j & 0xFFFF) << 4));
            return false;
        }
        const uint32_t base = ring_s + (uint32_t)S->ring_off[slot] + (one ? (uint32_t)(piece * E->last_bytes) : 0u);
        const int nr = min(kDsTileRows, n - tile * kDsTileRows), nlo = min(8, nr), nhi = nr > 8 ? nr - 8 : nlo;
        const uint32_t lstep = (uint32_t)nlo * 32u, hstep = (uint32_t)nhi * 32u;
        uint32_t lo = base + (uint32_t)(s0 * nlo + min(g, nlo - 1)) * 32u + (uint32_t)t * 8u;
        uint32_t hi = nr > 8 ? base + (uint32_t)(spp * nlo + s0 * nhi + min(g, nhi - 1)) * 32u + (uint32_t)t * 8u : lo;
        uint32_t b = bb;
        if (fmt == 1) {
            int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
            int s = 0;
#pragma unroll 2
            for (; s + 2 <= ns; s += 2) {
                const uint2 al = ds_lds64(lo), ah = ds_lds64(hi), b0 = ds_lds64(b);
                const uint2 bl = ds_lds64(lo + lstep), bh = ds_lds64(hi + hstep), b1 = ds_lds64(b + 128);
                ds_mma_i8(c0, al, ah, b0);
                ds_mma_i8(c1, bl, bh, b1);
                lo += 2 * lstep;
                hi += 2 * hstep;
                b += 256;
            }
            if (s < ns) ds_mma_i8(c0, ds_lds64(lo), ds_lds64(hi), ds_lds64(b));
            // lane (g, t < 2): digits 2 t, 2 t + 1 of rows g and g + 8
            if (t < 2) {
                ds_sts64(dst, (uint32_t)(c0[0] + c1[0]), (uint32_t)(c0[1] + c1[1]));
                ds_sts64(dst + 8 * kDsPartInt, (uint32_t)(c0[2] + c1[2]), (uint32_t)(c0[3] + c1[3]));
            }
            dst += kDsTileRows * kDsPartInt;
        } else {
            float a0, a1;
            if (fmt == 0) {
                float c[4];
                ds_tile_f16(c, lo, lstep, hi, hstep, b, ns);
                a0 = c[0] + c[1];  // columns 0, 1 = hi, lo (lanes t = 0)
                a1 = c[2] + c[3];
            } else {
                // int8 rows with a (scale, zero) per group of 128 (four steps): the integer sums of the warp's steps of a group are weighted by
                // the digits' powers of 256 in fp32 (exact: |sum| < 2^23, power-of-two weights), multiplied by the group's scale and
                // accumulated in fp32 together with zero x (sum of those steps' activations)
                const float w_lo = t == 0 ? 1.0f : 65536.0f, w_hi = w_lo * 256.0f;
                const uint32_t sz = base + (uint32_t)(nr * E->piece) + (uint32_t)g * 4u;  // [group of the piece][16 rows] words behind the rows
                a0 = a1 = 0.f;
                int c[4] = {0, 0, 0, 0};
                float tsum = 0.f;
#pragma unroll 1
                for (int s = 0; s < ns; ++s) {
                    const uint2 al = ds_lds64(lo), ah = ds_lds64(hi), b0 = ds_lds64(b);
                    ds_mma_i8(c, al, ah, b0);
                    tsum += S->tstep[w][s];
                    lo += lstep;
                    hi += hstep;
                    b += 128;
                    if (((w0 + s) & 3) == 3 || s + 1 == ns) {
                        const uint32_t zo = sz + (uint32_t)((s0 + s) >> 2) * 64u;
                        const float2 fa = ds_half2_bits_to_float2(ds_lds32(zo)), fb = ds_half2_bits_to_float2(ds_lds32(zo + 32u));  // (scale, zero) of rows g, g + 8
                        const float tz = t == 0 ? tsum : 0.f;
                        a0 = fmaf(fa.x, fmaf((float)c[1], w_hi, (float)c[0] * w_lo), fmaf(fa.y, tz, a0));
                        a1 = fmaf(fb.x, fmaf((float)c[3], w_hi, (float)c[2] * w_lo), fmaf(fb.y, tz, a1));
                        c[0] = c[1] = c[2] = c[3] = 0;
                        tsum = 0.f;
                    }
                }
                a0 += __shfl_xor_sync(0xffffffffu, a0, 1);  // lanes t = 0, 1 hold two digits each
                a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
            }
            if (t == 0) {
                ds_sts32(dst, __float_as_uint(a0));
                ds_sts32(dst + 8 * kDsPartF32, __float_as_uint(a1));
            }
            dst += kDsTileRows * kDsPartF32;
        }
        __syncwarp();
        if (lane == 0) ds_arrive(&S->empty[slot], one ? 1u : (uint32_t)np);  // 16 / np warps share the chunk; the barrier counts 16
    }
    return true;
}

// One finished output: row rl of this CTA's rows of matrix E.  `xout`: where the phase's residual stream goes.
__device__ __forceinline__ void ds_store(const DsParams& P, DsShared* S, const DsRows* E, int rl, float y, uint32_t tag, unsigned long long* xout) {
    const int m = E->r0 + rl, out = E->out;
    if (out == DSO_LOGITS) {
        P.logits[m] = y;
        return;
    }
    if (out == DSO_H) {
        const float a = fmaxf(y, 0.f);
        asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(P.hbuf + m), "r"((__float_as_uint(a * a) & 0x7FFFFFFFu) | (tag << 31)) : "memory");
        return;
    }
    unsigned long long* dst = P.rkv + (size_t)out * P.C + m;  // DSO_R, DSO_K, DSO_V
    if (out == DSO_XADD) {
        y += S->xs_own[rl];
        S->xs_own[rl] = y;
        dst = xout + m;
    } else if (out > DSO_V) {
        if (out == DSO_MID_TANH) y = tanhf(y);
        if (out == DSO_MID_SIG) y = 1.0f / (1.0f + expf(-y));
        dst = P.mid + E->out_off + m;
    }
    ds_put_pair(dst, y, tag);
}

__device__ __forceinline__ float4 ds_ldcg4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float ds_sum4(float4 v) { return (v.x + v.y) + (v.z + v.w); }
// Sum / maximum over the 512 consumer threads through a 16-entry array: one barrier per call.  Calls that follow each other must use
// different arrays (a thread may enter the next call while another still reads this one's array).
__device__ __forceinline__ float ds_block_sum(float v, float* arr, int w, int lane) {
    v = warp_sum(v);
    if (lane == 0) arr[w] = v;
    ds_consumer_sync();
    float s = arr[lane & 15];  // one read per lane, then a fixed shuffle tree over the 16 warp sums
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// CMAX: the largest n_embd the instantiation handles (it sizes the per-thread register arrays of the activation vectors)
template <int CMAX>
__global__ void __launch_bounds__(kDsThreads, 1) decode_stream_kernel(const __grid_constant__ DsParams P) {
    constexpr int NE = CMAX / 512;  // channels per lane (a warp holds C / 16); four times that of the F = 4 C hidden values
    extern __shared__ __align__(1024) uint8_t ds_smem_raw[];
    uint8_t* ring = (uint8_t*)(((uintptr_t)ds_smem_raw + 127) & ~(uintptr_t)127);
    DsShared* S = reinterpret_cast<DsShared*>(reinterpret_cast<float*>(ring + P.ring_bytes) + P.vec_floats);  // 16-byte aligned: ring and operand area are multiples of 16 bytes
    const uint32_t ring_s = smem_u32(ring), vec_s = ring_s + (uint32_t)P.ring_bytes, part_s = smem_u32(S->part);
    volatile int* abort_flag = (volatile int*)&S->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = gridDim.x, cta = blockIdx.x;
    const int C = P.C, L = P.L;
    // fp16 back-projection rows of a head in fragment order, rank dimensions padded to whole steps
    const int wmp = ds_pad16(P.wm), amp = ds_pad16(P.am), vmp = ds_pad16(P.vm), gmp = ds_pad16(P.gm);

    if (threadIdx.x < kDsBars) {
        mbar_init(&S->full[threadIdx.x], 1);
        mbar_init(&S->empty[threadIdx.x], kDsConsumerWarps);
        if (threadIdx.x == 0) {
            S->abort_flag = 0;
            S->abort_where = 0;
            S->rank_entry = -1;
            S->big_entry = DSE_WR;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x <= DSE_COUNT) {
        // layer 1's table when there is one: layer 0 has no v-gate projection, otherwise all layers split alike
        const int e = threadIdx.x;
        const DsEntry& E = e == DSE_COUNT ? P.head : P.layers[L > 1 ? 1 : 0].e[e];
        DsRows r;
        ds_rows_of(E, cta, G, r.r0, r.n);
        r.tiles = (r.n + kDsTileRows - 1) / kDsTileRows;
        r.np = E.npieces;
        r.piece = E.piece_bytes;
        r.steps = E.row_stride >> 5;
        r.spp = E.piece_bytes >> 5;
        r.fmt = E.is_i8;
        r.out = E.out;
        r.out_off = E.out_off;
        r.full_bytes = ds_chunk_bytes(E, kDsTileRows);
        r.last_bytes = ds_chunk_bytes(E, r.n - (r.tiles - 1) * kDsTileRows);
        r.merged = r.np * r.last_bytes <= kDsMergeBytes;
        S->rows[e] = r;
        if (r.n > 0 && e <= DSE_V1) S->rank_entry = e;
        if (r.n > 0 && e >= DSE_WR && e <= DSE_WV) S->big_entry = e;
    }
    __syncthreads();

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kDsProducerRegs));
        if (warp == 0) {
            // =========================== producer ===========================
            const uint64_t pol = l2_evict_first_policy();
            const int R = P.ring_bytes;
            int head = 0, used = 0;
            uint32_t j = 0, tail = 0;
            bool ok = true;
            const int rank_e = S->rank_entry, big_e = S->big_entry;
            // The weights lie in the stream in the order they are consumed: every chunk is one bulk copy from a running pointer.
#pragma unroll 1
            for (int t = 0; t < P.n_tokens && ok; ++t) {
                const bool do_head = P.argmax_feed || t == P.n_tokens - 1;
#pragma unroll 1
                for (int l = 0; l < L + (do_head ? 1 : 0) && ok; ++l) {
                    const char* src = l < L ? P.wstream + ((size_t)l * G + cta) * (size_t)P.wslot : P.hstream + (size_t)cta * (size_t)P.hslot;
                    const bool has_head = l < L && ds_head_of_cta(cta, l, P.H, G) >= 0;
                    // a layer: rank rows, r / k / v rows, a head's three chunks (w2 + a2 | v2 (layers > 0) + half of g2 | the other half), att.output, ffn.key, ffn.value
#pragma unroll 1
                    for (int item = 0; item < 8 && ok; ++item) {
                        int nfull, nlast = 0, fb, lb = 0;
                        if (item >= 2 && item <= 4) {
                            nfull = has_head ? 1 : 0;
                            fb = item == 2 ? 128 * (wmp + amp) : 64 * gmp + (item == 3 && l > 0 ? 128 * vmp : 0);
                        } else {
                            int e = l == L ? (item == 0 ? DSE_COUNT : -1) : item == 0 ? rank_e : item == 1 ? big_e : item - 5 + DSE_WO;
                            if (e == DSE_V1 && l == 0) e = -1;
                            if (e < 0) continue;
                            const DsRows& E = S->rows[e];
                            nlast = E.tiles > 0 ? (E.merged ? 1 : E.np) : 0;
                            nfull = max(E.tiles - 1, 0) * E.np;
                            fb = E.full_bytes;
                            lb = E.merged ? E.np * E.last_bytes : E.last_bytes;
                        }
                        if (l == L && item > 0) break;
#pragma unroll 1
                        for (int q = 0; q < nfull + nlast; ++q) {
                            const int bytes = q < nfull ? fb : lb;
                            // room in the ring (waiting for the oldest chunks to be released); a chunk that does not fit behind the last one goes to the start
                            const bool wrap = head + bytes > R;
                            const int waste = wrap ? R - head : 0;
                            while (used + waste + bytes > R || j - tail >= (uint32_t)kDsBars) {
                                const bool w = mbar_wait(&S->empty[tail % kDsBars], (tail / kDsBars) & 1u, abort_flag);
                                if (!__all_sync(0xffffffffu, w)) {
                                    if (lane == 0) atomicCAS(&S->abort_where, 0, 2 | (int)((j & 0xFFFF) << 4));
                                    ok = false;
                                    break;
                                }
                                used -= S->alloc[tail % kDsBars];
                                ++tail;
                            }
                            if (!ok) break;
                            if (wrap) head = 0;
                            const int slot = (int)(j % kDsBars);
                            if (lane == 0) {
                                S->alloc[slot] = waste + bytes;
                                S->ring_off[slot] = head;
                                mbar_expect_tx(&S->full[slot], (uint32_t)bytes);  // a release: the offset is visible to whoever sees the barrier complete
                                ds_bulk_load(ring_s + (uint32_t)head, src, (uint32_t)bytes, &S->full[slot], pol);
                            }
                            __syncwarp();
                            used += waste + bytes;
                            head += bytes;
                            src += bytes;
                            ++j;
                        }
                    }
                }
            }
            // copies still in flight must land before the CTA may exit (only after an abort: otherwise every chunk was consumed)
            if (!ok)
                for (; tail < j; ++tail) ds_mbar_drain(&S->full[tail % kDsBars], (tail / kDsBars) & 1u);
        }
    } else {
        // =========================== consumers ===========================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDsConsumerRegs));
        const int wtid = threadIdx.x - 128, w = wtid >> 5;
        uint32_t J = 0;  // chunks of this CTA consumed so far (the producer numbers them the same way)
        unsigned bar_target = P.bar_base;
        bool ok = true;
        const int r0o = S->rows[DSE_WO].r0, nown = S->rows[DSE_WO].n;  // this CTA's slice of the channels = its rows of att.output / ffn.value
        uint32_t lt = 0;  // layers run so far: the table of the current layer sits in S->layer[lt & 1]

        auto stage_layer = [&](int l, uint32_t slot) {
            static_assert(sizeof(DsLayer) % 4 == 0, "DsLayer is copied word by word");
            const uint32_t* src = reinterpret_cast<const uint32_t*>(P.layers + l);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&S->layer[slot & 1]);
            for (int i = wtid; i < (int)(sizeof(DsLayer) / 4); i += kDsConsumers) dst[i] = __ldg(src + i);
        };
        // Grid barrier.  The counter only ever grows; a CTA sees barrier n complete before it arrives on barrier n + 1.
        auto bar_wait = [&]() -> bool {
            if (wtid == 0) {
                bool got = false;
                for (uint32_t i = 0; i < kDsBarSpin; ++i) {
                    unsigned v;
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(P.grid_bar) : "memory");
                    if ((int)(v - bar_target) >= 0) {
                        got = true;
                        break;
                    }
                    if ((i & 255u) == 255u && *abort_flag) break;
                }
                if (!got) {
                    atomicCAS(&S->abort_where, 0, 3 | (int)((bar_target & 0xFFFF) << 4));
                    *abort_flag = 1;
                }
            }
            return !ds_consumer_sync_or(*abort_flag != 0);
        };
        auto bar_arrive = [&]() {
            ds_consumer_sync();
            if (wtid == 0) {
                // one release operation instead of a fence and a relaxed atomic (the bar.sync above ordered the other warps' stores
                // before this thread)
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.grid_bar) : "memory");
            }
            bar_target += (unsigned)G;
        };

#pragma unroll 1
        for (int t = 0; t < P.n_tokens && ok; ++t) {
            const bool do_head = P.argmax_feed || t == P.n_tokens - 1;
            if (wtid == 0) {
                uint32_t tk = (P.argmax_feed && t > 0) ? S->tok : (P.tok_from_list == 2 ? P.tok0 : P.tok_from_list ? P.tok_list[t] : P.tokens[0]);
                if (tk >= (uint32_t)P.V) {
                    atomicOr(P.status, 1);
                    tk = 0;
                }
                S->tok = tk;
            }
            if (t == 0) stage_layer(0, 0);
            ds_consumer_sync();
            float best = -1e30f;  // arg-max over the head rows this thread finished
            int best_i = 0x7fffffff;

            // ---- units: phase 1, 3, 4, 5 of every layer (phase 2, the heads, follows phase 1), then the vocabulary head ----
#pragma unroll 1
            for (int u = 0; u < 4 * L + (do_head ? 1 : 0) && ok; ++u) {
                const int l = u >> 2, ph = l == L ? 4 : (u & 3);
                const DsLayer& Ly = S->layer[lt & 1];
                const size_t lx = (size_t)l * P.lay_x + (size_t)P.slot * C;
                const int eA = ph == 0 ? S->big_entry : ph == 4 ? (int)DSE_COUNT : DSE_WO + ph - 1;
                int eB = ph == 0 ? S->rank_entry : -1;
                if (eB == DSE_V1 && l == 0) eB = -1;
                const DsRows *A = &S->rows[eA], *B = eB >= 0 ? &S->rows[eB] : nullptr;
                const DsEntry& EA = ph == 4 ? P.head : Ly.e[eA];
                const bool ln = ph != 1 && ph != 3, i8 = A->fmt != 0, pg = A->fmt == 2;
                if (ph == 2) stage_layer(l + 1 < L ? l + 1 : 0, lt + 1);  // the table of the layer that runs next (the first one again after the last)
                const uint32_t tag = P.epoch + (uint32_t)(t * L + l);
                // ---- requested before the wait: (scale, zero) of the row this thread will finish, LayerNorm and mix vectors, shift state ----
                float ws = 0.f, wz = 0.f;
                if (A->fmt == 1 && (wtid >> 2) < A->n) {
                    ws = __ldg(EA.wscale + A->r0 + (wtid >> 2));
                    wz = __ldg(EA.wzero + A->r0 + (wtid >> 2));
                }
                const int per = ph == 3 ? C / 4 : C / 16, first = w * per + lane, end = (w + 1) * per;  // this lane's elements: first, first + 32, ...
                const int where = 3 | ((u & 0xFFFF) << 4);
                // The warp's sixteenth of operand A (and B: phase 1, the rank projection's input) is put into the operand area as fp32 first and
                // converted in place, 32 elements at a time, when the vector's maximum is known.
                const uint32_t rawA = vec_s + 4u * (uint32_t)first, rawB = rawA + 4u * (uint32_t)C;
                float am0 = 0.f, am1 = 0.f;
                if (ln) {
                    const float* shift = ph == 0 ? P.tmix_x + lx : ph == 2 ? P.cmix_x + lx : nullptr;
                    const float* mixA = ph == 0 ? EA.mix : ph == 2 ? Ly.ffn_x_k : nullptr;
                    const float* mixB = eB >= 0 ? Ly.e[eB].mix : mixA;
                    const float* lw = ph == 0 ? Ly.ln1_w : ph == 2 ? Ly.ln2_w : P.lno_w;
                    const float* lb = ph == 0 ? Ly.ln1_b : ph == 2 ? Ly.ln2_b : P.lno_b;
                    float pw[NE], pb[NE], pv[NE], mA[NE], mB[NE], x[NE];
#pragma unroll
                    for (int i = 0; i < NE; ++i) {
                        const int k = min(first + 32 * i, end - 1);
                        pw[i] = __ldg(lw + k);
                        pb[i] = __ldg(lb + k);
                        pv[i] = mA[i] = mB[i] = 0.f;
                        if (shift) {
                            pv[i] = __ldcg(shift + k);
                            mA[i] = __ldg(mixA + k);
                            mB[i] = __ldg(mixB + k);
                        }
                    }
                    if (u == 0) {
                        // x = LN0(embedding row), every CTA builds the whole vector
#pragma unroll
                        for (int i = 0; i < NE; ++i) x[i] = __half2float(P.emb[(size_t)S->tok * C + min(first + 32 * i, end - 1)]);
                    } else {
                        ok = ds_poll_pairs<NE>(S, ph == 2 ? P.xb : P.xa, first, end, ph == 2 ? tag : tag - 1u, x, where);
                    }
                    float inv;
#pragma unroll 1
                    for (int pass = u == 0 ? 0 : 1; pass < 2; ++pass) {
                        float a = 0.f;
#pragma unroll
                        for (int i = 0; i < NE; ++i)
                            if (first + 32 * i < end) a += x[i];
                        const float mean = ds_block_sum(a, S->red[0], w, lane) / (float)C;
                        a = 0.f;
#pragma unroll
                        for (int i = 0; i < NE; ++i) {
                            x[i] -= mean;
                            if (first + 32 * i < end) a += x[i] * x[i];
                        }
                        inv = 1.0f / sqrtf(ds_block_sum(a, S->red[1], w, lane) / (float)C + kLnEps);
                        if (pass == 0) {
#pragma unroll
                            for (int i = 0; i < NE; ++i) {
                                const int k = min(first + 32 * i, end - 1);
                                x[i] = x[i] * inv * __ldg(P.ln0_w + k) + __ldg(P.ln0_b + k);
                                if (first + 32 * i < end && (unsigned)(k - r0o) < (unsigned)nown) S->xs_own[k - r0o] = x[i];
                            }
                        }
                    }
                    float* own = ph == 0 ? S->ts_own : S->cs_own;  // LN(x): the new shift state, stored once everybody has read the old one
#pragma unroll
                    for (int i = 0; i < NE; ++i) {
                        const float c = x[i] * inv * pw[i] + pb[i], d = shift ? pv[i] - c : 0.f;
                        const int k = first + 32 * i;
                        if (k < end) {
                            if (shift && (unsigned)(k - r0o) < (unsigned)nown) own[k - r0o] = c;
                            const float a = c + mA[i] * d, b = c + mB[i] * d;
                            am0 = fmaxf(am0, fabsf(a));
                            am1 = fmaxf(am1, fabsf(b));
                            ds_sts32(rawA + 128u * i, __float_as_uint(a));
                            if (B) ds_sts32(rawB + 128u * i, __float_as_uint(b));
                        }
                    }
                } else if (ph == 1) {
                    float x[NE];
                    ok = ds_poll_pairs<NE>(S, P.yg, first, end, tag, x, where);
#pragma unroll
                    for (int i = 0; i < NE; ++i)
                        if (first + 32 * i < end) {
                            am0 = fmaxf(am0, fabsf(x[i]));
                            ds_sts32(rawA + 128u * i, __float_as_uint(x[i]));
                        }
                } else {
                    // hidden values: the sign bit is the parity of the layer's tag
                    uint32_t r[4 * NE], turns = 0;
                    const uint32_t* src = P.hbuf + first;
#pragma unroll
                    for (int i = 0; i < 4 * NE; ++i) r[i] = first + 32 * i < end ? ds_get_word(src + 32 * i) : tag << 31;
                    for (;;) {
                        bool all = true;
#pragma unroll
                        for (int i = 0; i < 4 * NE; ++i) all = all && (r[i] >> 31) == (tag & 1u);
                        if (all) break;
                        if (!ds_spin_ok(S, turns, where)) {
                            ok = false;
                            break;
                        }
#pragma unroll
                        for (int i = 0; i < 4 * NE; ++i)
                            if ((r[i] >> 31) != (tag & 1u)) r[i] = ds_get_word(src + 32 * i);
                    }
#pragma unroll
                    for (int i = 0; i < 4 * NE; ++i)
                        if (first + 32 * i < end) {
                            const uint32_t x = r[i] & 0x7FFFFFFFu;
                            am0 = fmaxf(am0, __uint_as_float(x));
                            ds_sts32(rawA + 128u * i, x);
                        }
                }
                // ---- operands: one scale per vector; every warp writes (and later reads) its own sixteenth ----
                am0 = warp_absmax(am0);
                am1 = warp_absmax(am1);
                if (lane == 0) {
                    S->red[2][w] = am0;
                    S->red[5][w] = am1;  // (not [3]: a head's last sum before this unit may still be being read there)
                }
                if (!(ok = !ds_consumer_sync_or(!ok))) break;
                // the shift state this CTA owns: this phase's input is complete, so everybody has read the old one
                if (wtid < nown) {
                    if (ph == 1) (P.tmix_x + lx)[r0o + wtid] = S->ts_own[wtid];
                    if (ph == 3) (P.cmix_x + lx)[r0o + wtid] = S->cs_own[wtid];
                }
                const int ex0 = ds_exponent(warp_absmax(S->red[2][lane & 15])), ex1 = ds_exponent(warp_absmax(S->red[5][lane & 15]));
                {
                    long long ts = 0;
#pragma unroll 1
                    for (int i0 = 0; i0 < (B ? 2 : 1) * ((per + 31) / 32); i0 += NE) {  // (operand B: a second round of NE)
                        const bool second = B && i0 >= (per + 31) / 32, q8 = !second && i8;
                        const int k0 = second ? first : first + 32 * i0;
                        const uint32_t vs = second ? vec_s + 4u * (uint32_t)C : vec_s;
                        const float mult = second ? ds_pow2(-ex1) : ds_pow2((i8 ? kDsP : 0) - ex0);
                        float x[NE];
#pragma unroll
                        for (int i = 0; i < NE; ++i) x[i] = k0 + 32 * i < end ? __uint_as_float(ds_lds32(vs + 4u * (uint32_t)(k0 + 32 * i))) : 0.f;
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < NE; ++i) {
                            int tv = 0;
                            if (k0 + 32 * i < end) tv = ds_put(q8, vs, k0 + 32 * i, x[i], mult);
                            ts += tv;
                            if (pg && q8) {  // 32 consecutive elements: the sum of a step
                                const long long t32 = ds_warp_sum_int(tv);
                                if (lane == 0) S->tstep[w][i0 + i] = (float)t32;
                            }
                        }
                    }
                    if (A->fmt == 1) {
                        const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)(ts & 0xFFFF));
                        const int hi = __reduce_add_sync(0xffffffffu, (int)(ts >> 16));
                        if (lane == 0) S->tsw[w] = (long long)hi * 65536 + (long long)lo;
                    }
                }
                __syncwarp();
                // ---- rows, in batches of tiles whose partial sums fit ----
                const int tile_bytes = kDsTileRows * (A->fmt == 1 ? kDsPartInt : kDsPartF32), batch = kDsPartBytes / tile_bytes;
#pragma unroll 1
                for (int tile0 = 0; tile0 < A->tiles; tile0 += batch) {
                    const int tile1 = min(A->tiles, tile0 + batch), base = tile0 * kDsTileRows, nA = min(A->n - base, (tile1 - tile0) * kDsTileRows);
                    if (tile0) ds_consumer_sync();  // the previous batch's sums have been read
#pragma unroll 1
                    for (int which = B && tile0 == 0 ? 0 : 1; which < 2; ++which) {  // phase 1: the rank rows come first
                        const DsRows* E = which ? A : B;
                        const int e0 = which ? tile0 : 0, e1 = which ? tile1 : E->tiles;
                        ok = ok && ds_multiply(S, E, ring_s, which ? vec_s : vec_s + 4u * (uint32_t)C, which ? part_s : part_s + kDsPartBytes, J, e0, e1, w, lane);
                        J += (uint32_t)((e1 - e0) * E->np - (e1 == E->tiles && E->merged ? E->np - 1 : 0));
                    }
                    if (!(ok = !ds_consumer_sync_or(!ok))) break;
                    // four lanes per row add its sixteen sums (rank rows follow the others)
                    const unsigned quad = 0xFu << (lane & 28);
                    const int q = lane & 3, nB = B && tile0 == 0 ? B->n : 0;
#pragma unroll 1
                    for (int rr = wtid >> 2; rr < ((nA + nB + 7) & ~7); rr += kDsConsumers / 4) {  // (whole warps: shuffles below)
                        const bool isB = rr >= nA;
                        const int r = min(isB ? rr - nA : rr, max((isB ? nB : nA) - 1, 0));
                        float y;
                        if (!isB && A->fmt == 1) {
                            const char* src = S->part + (size_t)r * kDsPartInt + q * 16;
                            int d[4] = {0, 0, 0, 0};
                            long long T = 0;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int4 v = *reinterpret_cast<const int4*>(src + i * 64);
                                d[0] += v.x, d[1] += v.y, d[2] += v.z, d[3] += v.w;
                                T += S->tsw[q + 4 * i];
                            }
                            long long Q = (long long)d[0] + ((long long)d[1] << 8) + ((long long)d[2] << 16) + ((long long)d[3] << 24);
#pragma unroll
                            for (int o = 1; o < 4; o <<= 1) {
                                Q += __shfl_xor_sync(quad, Q, o);
                                T += __shfl_xor_sync(quad, T, o);
                            }
                            if (tile0 || rr >= kDsConsumers / 4) {  // not the prefetched row
                                ws = __ldg(EA.wscale + A->r0 + base + r);
                                wz = __ldg(EA.wzero + A->r0 + base + r);
                            }
                            y = (float)((double)ds_pow2(ex0 - kDsP) * ((double)ws * (double)Q + (double)wz * (double)T));
                        } else {
                            const float4 v = *reinterpret_cast<const float4*>(S->part + (isB ? kDsPartBytes : 0) + (size_t)r * kDsPartF32 + q * 16);
                            y = ds_sum4(v);
                            y += __shfl_xor_sync(quad, y, 1);
                            y += __shfl_xor_sync(quad, y, 2);
                            y *= ds_pow2(isB ? ex1 : ex0 - (pg ? kDsP : 0));
                        }
                        if (q == 0 && rr < nA + nB) {
                            ds_store(P, S, isB ? B : A, isB ? r : base + r, y, tag, ph == 1 ? P.xb : P.xa);
                            if (ph == 4 && y > best) {  // a thread's rows ascend: ties keep the smaller index
                                best = y;
                                best_i = A->r0 + base + r;
                            }
                        }
                    }
                }
                if (!ok) break;
                if (ph == 3) ++lt;
                if (ph != 0) continue;

                // ================= phase 2: one CTA per head =================
                const int h = ds_head_of_cta(cta, l, P.H, G);
                if (h >= 0) {
                    // state: 8 threads per row, 8 columns each (the same CTA and threads as in the previous token: no barrier needed)
                    const int rrow = wtid >> 3, oct = wtid & 7, ch = h * 64 + rrow, cc = h * 64 + (wtid & 63);
                    float* srow = P.wkv + (size_t)l * P.lay_s + ((size_t)P.slot * P.H + h) * 4096 + (size_t)rrow * 64 + oct * 8;
                    const float4 s4a = ds_ldcg4(srow), s4b = ds_ldcg4(srow + 4);
                    const float p_gw = __ldg(Ly.lnx_w + ch), p_gb = __ldg(Ly.lnx_b + ch);
                    float p_w0 = 0.f, p_a0 = 0.f, p_kk = 0.f, p_ka = 0.f, p_rk = 0.f, p_v0 = 0.f;
                    if (wtid < 64) {
                        p_w0 = __ldg(Ly.w0 + cc), p_a0 = __ldg(Ly.a0 + cc), p_kk = __ldg(Ly.k_k + cc), p_ka = __ldg(Ly.k_a + cc), p_rk = __ldg(Ly.r_k + cc);
                        if (l > 0) p_v0 = __ldg(Ly.v0 + cc);
                    }
                    const int vdim = w == 0 ? P.wm : w == 1 ? P.am : w == 2 ? P.vm : P.gm;                      // rank-space vector of warps 0-3
                    const int voff = w == 0 ? 0 : w == 1 ? P.wm : w == 2 ? P.wm + P.am : P.wm + P.am + P.vm;    // its place in P.mid
                    const uint32_t o_w = vec_s, o_a = o_w + 4u * wmp, o_v = o_a + 4u * amp, o_g = o_v + 4u * vmp;  // fragments of the four vectors
                    if (w < 4) {
                        // hi + lo halves of a rank-space vector, zeros up to a whole step
                        const uint32_t dst = w == 0 ? o_w : w == 1 ? o_a : w == 2 ? o_v : o_g;
                        const int padded = w == 2 && l == 0 ? 0 : ds_pad16(vdim);  // layer 0 has no v gate
                        float x[kDsMaxRank / 32], am = 0.f;
                        ok = ds_poll_pairs<kDsMaxRank / 32>(S, P.mid + voff, lane, w == 2 && l == 0 ? 0 : vdim, tag, x, where);
#pragma unroll
                        for (int i = 0; i < kDsMaxRank / 32; ++i) am = fmaxf(am, fabsf(x[i]));  // (zeros past the end)
                        const int ex = ds_exponent(warp_absmax(am));
#pragma unroll
                        for (int i = 0; i < kDsMaxRank / 32; ++i)
                            if (lane + 32 * i < padded) ds_put(false, dst, lane + 32 * i, x[i], ds_pow2(-ex));
                        if (lane == 0) S->red[4][w] = ds_pow2(ex);
                    } else if (w < 10) {
                        const int i = wtid - 128;
                        float x[1];
                        ok = ds_poll_pairs<1>(S, P.rkv + (size_t)(i >> 6) * C + h * 64, i & 63, 64, tag, x, where);
                        S->hv[i] = x[0];  // r, k, v of the head
                    } else if (w < 12 && l > 0) {
                        float x[1];
                        ok = ds_poll_pairs<1>(S, P.vfirst + h * 64, wtid - 320, 64, tag - (uint32_t)l, x, where);
                        S->hv[13 * 64 + wtid - 320] = x[0];
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!(ok = !ds_consumer_sync_or(!ok))) break;
                    // back-projections: warp = (tile of 16 channels, part): part 0 decay, 1 a, 2 v gate and the first part of the output gate, 3 the rest of it
                    const int tile = w >> 2, part = w & 3, g = lane >> 2, tq = lane & 3;
                    const int sg = gmp / 16, sv = l > 0 ? vmp / 16 : 0, gsplit = max(0, (sg - sv) / 2);
                    const uint32_t lane_off = (uint32_t)(g * 32 + tq * 8), b_off = (uint32_t)((g & 1) * 32 + tq * 8);
#pragma unroll 1
                    for (int c = 0; c < 3 && ok; ++c) {
                        const uint32_t jc = J + (uint32_t)c;
                        const int slot = (int)(jc % kDsBars);
                        const bool need = c == 0 ? part < 2 : c == 1 ? (part == 2 || (part == 3 && tile < 2)) : (part >= 2 && tile >= 2);
                        if (need) {
                            const bool got = mbar_wait(&S->full[slot], (jc / kDsBars) & 1u, abort_flag);
                            if (!__all_sync(0xffffffffu, got)) {
                                if (lane == 0) atomicCAS(&S->abort_where, 0, 4 | (int)((jc & 0xFFFF) << 4));
                                ok = false;
                                break;
                            }
                            const uint32_t base = ring_s + (uint32_t)S->ring_off[slot] + lane_off;
                            const uint32_t gbase = base + (c == 1 && l > 0 ? 128u * (uint32_t)vmp : 0u) + (uint32_t)(tile & 1) * 32u * (uint32_t)gmp;
#pragma unroll 1
                            for (int k = 0; k < 2; ++k) {
                                // k = 0: decay / a / v gate; k = 1: output gate
                                uint32_t lo, bf;
                                int steps, ns, slot_hv;
                                if (k == 0) {
                                    if (c == 0) {
                                        const int mp = part == 0 ? wmp : amp;
                                        lo = base + (part ? 128u * (uint32_t)wmp : 0u) + (uint32_t)tile * 32u * (uint32_t)mp;
                                        bf = part ? o_a : o_w;
                                        steps = ns = mp / 16;
                                    } else if (c == 1 && part == 2 && l > 0) {
                                        lo = base + (uint32_t)tile * 32u * (uint32_t)vmp;
                                        bf = o_v;
                                        steps = ns = sv;
                                    } else {
                                        continue;
                                    }
                                    slot_hv = 3 + part;
                                } else {
                                    if (c == 0 || (tile >> 1) != c - 1) continue;
                                    const int from = part == 2 ? 0 : gsplit;
                                    lo = gbase + (uint32_t)from * 256u;
                                    bf = o_g + (uint32_t)from * 64u;
                                    steps = sg;
                                    ns = part == 2 ? gsplit : sg - gsplit;
                                    slot_hv = 4 + part;
                                }
                                float cs[4];
                                ds_tile_f16(cs, lo, 256u, lo + (uint32_t)steps * 256u, 256u, bf + b_off, ns);
                                const float sc = S->red[4][k ? 3 : part];
                                if (tq == 0) {
                                    S->hv[slot_hv * 64 + tile * 16 + g] = (cs[0] + cs[1]) * sc;
                                    S->hv[slot_hv * 64 + tile * 16 + g + 8] = (cs[2] + cs[3]) * sc;
                                }
                            }
                        }
                        __syncwarp();
                        if (lane == 0) ds_arrive(&S->empty[slot], 1u);  // all sixteen warps release the chunk, those that do not read it at once
                    }
                    J += 3;
                    if (!(ok = !ds_consumer_sync_or(!ok))) break;
                    // per-channel quantities of the head (warps 0, 1); ||kk||^2 and the bonus sum over the 64 channels
                    if (wtid < 64) {
                        const float aa = 1.0f / (1.0f + expf(-(S->hv[4 * 64 + wtid] + p_a0)));
                        const float wdec = expf((1.0f / (1.0f + expf(-(S->hv[3 * 64 + wtid] + p_w0)))) * kDecayScale);
                        const float rr = S->hv[wtid], kk0 = S->hv[64 + wtid];
                        float vv0 = S->hv[128 + wtid];
                        if (l == 0) {
                            ds_put_pair(P.vfirst + cc, vv0, tag);
                            P.state_vfirst[(size_t)P.slot * C + cc] = vv0;
                        } else {
                            const float gate = 1.0f / (1.0f + expf(-(S->hv[5 * 64 + wtid] + p_v0)));
                            vv0 = vv0 + gate * (S->hv[13 * 64 + wtid] - vv0);
                        }
                        const float kkj = kk0 * p_kk, kt = kk0 + p_ka * (kk0 * aa - kk0);
                        S->hv[8 * 64 + wtid] = wdec;
                        S->hv[9 * 64 + wtid] = kkj;
                        S->hv[10 * 64 + wtid] = aa;
                        S->hv[11 * 64 + wtid] = kt;
                        S->hv[12 * 64 + wtid] = vv0;
                        const float ssp = warp_sum(kkj * kkj), srp = warp_sum(rr * kt * p_rk);
                        if (lane == 0) {
                            S->red[0][w] = ssp;
                            S->red[1][w] = srp;
                        }
                    }
                    ds_consumer_sync();
                    const float ss = S->red[0][0] + S->red[0][1], srk = S->red[1][0] + S->red[1][1];
                    const float invn = 1.0f / fmaxf(sqrtf(ss), kL2Eps);
                    const float vv_row = S->hv[12 * 64 + rrow];
                    float St[8] = {s4a.x, s4a.y, s4a.z, s4a.w, s4b.x, s4b.y, s4b.z, s4b.w};
                    // this thread's eight columns of the head's vectors (16-byte reads)
                    auto ld8 = [&](int arr, float (&o)[8]) {
                        const float4 lo = *reinterpret_cast<const float4*>(&S->hv[arr * 64 + oct * 8]), hi = *reinterpret_cast<const float4*>(&S->hv[arr * 64 + oct * 8 + 4]);
                        o[0] = lo.x, o[1] = lo.y, o[2] = lo.z, o[3] = lo.w, o[4] = hi.x, o[5] = hi.y, o[6] = hi.z, o[7] = hi.w;
                    };
                    float kkh[8], wv[8], av[8], ktv[8], rv[8], sa = 0.f;
                    ld8(9, kkh);
                    ld8(8, wv);
                    ld8(10, av);
                    ld8(11, ktv);
                    ld8(0, rv);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        kkh[q] *= invn;
                        sa = fmaf(St[q], kkh[q], sa);
                    }
                    sa += __shfl_xor_sync(0xffffffffu, sa, 1);
                    sa += __shfl_xor_sync(0xffffffffu, sa, 2);
                    sa += __shfl_xor_sync(0xffffffffu, sa, 4);
                    float y = 0.f;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float bq = kkh[q] * (-av[q]);
                        St[q] = fmaf(St[q], wv[q], fmaf(sa, bq, vv_row * ktv[q]));
                        y = fmaf(St[q], rv[q], y);
                    }
                    y += __shfl_xor_sync(0xffffffffu, y, 1);
                    y += __shfl_xor_sync(0xffffffffu, y, 2);
                    y += __shfl_xor_sync(0xffffffffu, y, 4);
                    *reinterpret_cast<float4*>(srow) = make_float4(St[0], St[1], St[2], St[3]);
                    *reinterpret_cast<float4*>(srow + 4) = make_float4(St[4], St[5], St[6], St[7]);
                    const float gmean = ds_block_sum(oct == 0 ? y : 0.f, S->red[2], w, lane) / 64.0f;
                    const float d = y - gmean;
                    const float var = ds_block_sum(oct == 0 ? d * d : 0.f, S->red[3], w, lane) / 64.0f + kGnEps;
                    if (oct == 0) ds_put_pair(P.yg + ch, (d * (1.0f / sqrtf(var)) * p_gw + p_gb + srk * vv_row) * (S->hv[6 * 64 + rrow] + S->hv[7 * 64 + rrow]), tag);
                }
            }
            if (!ok) break;

            // the token's one grid barrier: orders the shift states for the next token, and the arg-max candidates
            if (!P.argmax_feed) {
                if (t + 1 < P.n_tokens) {
                    bar_arrive();
                    if (!(ok = bar_wait())) break;
                }
            } else {
                // arg-max: lanes -> warp -> CTA -> grid; ties go to the smaller index
                auto reduce = [&](float& bv, int& bi) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                        if (ov > bv || (ov == bv && oi < bi)) {
                            bv = ov;
                            bi = oi;
                        }
                    }
                };
                reduce(best, best_i);
                if (lane == 0) {
                    S->red[0][w] = best;
                    S->red_i[w] = best_i;
                }
                ds_consumer_sync();
                best = S->red[0][lane & 15];
                best_i = S->red_i[lane & 15];
                reduce(best, best_i);
                if (wtid == 0) {
                    P.cand_val[cta] = best;
                    P.cand_idx[cta] = best_i;
                }
                bar_arrive();
                if (!(ok = bar_wait())) break;
                // every CTA reduces the candidates itself: no further barrier before the next token
                if (w == 0) {
                    best = -1e30f;
                    best_i = 0x7fffffff;
#pragma unroll 1
                    for (int c = lane; c < G; c += 32) {
                        const float ov = __ldcg(P.cand_val + c);
                        const int oi = __ldcg(P.cand_idx + c);
                        if (ov > best || (ov == best && oi < best_i)) {
                            best = ov;
                            best_i = oi;
                        }
                    }
                    reduce(best, best_i);
                    if (lane == 0) {
                        if (best_i == 0x7fffffff) best_i = 0;
                        S->tok = (uint32_t)best_i;
                        if (cta == 0) {
                            P.tokens[0] = (uint32_t)best_i;
                            if (P.seq) {
                                const int cnt = P.seq_cnt[0];
                                if (cnt < P.seq_cap) P.seq[cnt] = (uint32_t)best_i;
                                P.seq_cnt[0] = cnt + 1;
                            }
                        }
                    }
                }
                ds_consumer_sync();
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) {
        atomicOr(P.status, 32);
        // where: a CTA that gave up on its own chunks or ring outranks the CTAs that gave up on the grid barrier because of it
        if (S->abort_where) atomicMax(P.status + 1, (((S->abort_where & 15) == 3 ? 1 : 2) << 28) | (cta << 20) | (S->abort_where & 0xFFFFF));
    }
}

// Writes the second copy of the weights: for every layer and every CTA of the decode kernel, the CTA's chunks in the order it
// consumes them (fragment order, see above), the head's rows in a region of their own.  Launched once per model with the decode
// kernel's grid size; CTA c lays out the region of decode CTA c.
__global__ void __launch_bounds__(256) ds_retile_kernel(const __grid_constant__ DsParams P, char* wstream, long long wslot, char* hstream, long long hslot) {
    __shared__ DsPlan pl;
    const int G = gridDim.x, cta = blockIdx.x;
    if (threadIdx.x == 0) ds_build_plan(pl, P.layers[P.L > 1 ? 1 : 0].e, P.head, cta, G, 0u);
    __syncthreads();
    // `nr` rows (row_stride bytes apart), `steps` steps of 32 bytes from byte `col` on -> fragments; bytes past row_bytes are zeros
    auto fragments = [&](const char* rows, size_t row_stride, int row_bytes, int nr, int col, int steps, char* dst) {
        const int nlo = min(8, nr), nhi = nr - nlo;
        for (int i = threadIdx.x; i < nr * steps * 4; i += blockDim.x) {
            const bool hi = i >= nlo * steps * 4;
            const int q = hi ? i - nlo * steps * 4 : i, n = hi ? nhi : nlo, tq = q & 3, g = (q >> 2) % n, s = (q >> 2) / n;
            const char* src = rows + (size_t)(g + (hi ? 8 : 0)) * row_stride;
            const int c0 = col + s * 32 + 4 * tq, c1 = c0 + 16;
            uint2 v = make_uint2(0u, 0u);
            if (c0 < row_bytes) v.x = *reinterpret_cast<const uint32_t*>(src + c0);
            if (c1 < row_bytes) v.y = *reinterpret_cast<const uint32_t*>(src + c1);
            *reinterpret_cast<uint2*>(dst + (size_t)i * 8) = v;
        }
    };
    auto copy_chunk = [&](const DsEntry& E, const DsChunk& c, char* dst) {
        const int nr = c.nr_steps & 0xFFFF, piece = c.piece_np & 0xFFFF, e = c.e_flags_row0 & 0xFF, row0 = c.e_flags_row0 >> 16, r = pl.er0[e] + row0;
        fragments(E.base + (size_t)r * (size_t)E.row_stride, (size_t)E.row_stride, E.row_stride, nr, piece * E.piece_bytes, E.piece_bytes >> 5, dst);
        if (E.is_i8 == 2) {  // the rows' (scale, zero) words of this piece's groups: [group][16 rows], zero for rows past nr
            const int ngp = E.piece_bytes >> 7, kgroups = E.row_stride >> 7;
            uint32_t* zd = reinterpret_cast<uint32_t*>(dst + (size_t)nr * c.stride);
            for (int i = threadIdx.x; i < ngp * kDsTileRows; i += blockDim.x) {
                const int gi = i / kDsTileRows, row = i % kDsTileRows;
                zd[i] = row < nr ? E.sz[(size_t)(r + row) * kgroups + (size_t)piece * ngp + gi] : 0u;
            }
        }
    };
    // tiles [tile0, tile1) of 16 rows of one head of a back-projection matrix [C, mid]
    auto copy_back = [&](const __half* W, int h, int mid, int tile0, int tile1, char*& dst) {
        for (int tile = tile0; tile < tile1; ++tile) {
            fragments(reinterpret_cast<const char*>(W + (size_t)(h * 64 + tile * 16) * mid), (size_t)mid * 2, mid * 2, 16, 0, ds_pad16(mid) / 16, dst);
            dst += 32 * ds_pad16(mid);
        }
    };
    for (int l = 0; l < P.L; ++l) {
        const DsLayer& Ly = P.layers[l];
        char* dst = wstream + ((size_t)l * G + cta) * (size_t)wslot;
        for (int ph = DSP_P1; ph <= DSP_P5; ++ph) {
            for (int k = pl.ph0[ph]; k < pl.ph0[ph] + pl.phn[ph]; ++k) {
                const DsChunk& c = pl.ctab[k];
                if (l == 0 && ((c.e_flags_row0 >> 8) & 2)) continue;
                copy_chunk(Ly.e[c.e_flags_row0 & 0xFF], c, dst);
                dst += c.cb;
            }
            if (ph == DSP_P1) {
                const int h = ds_head_of_cta(cta, l, P.H, G);
                if (h >= 0) {  // the head's back-projection rows: w2, a2 | v2 (layers > 0), first 32 g2 rows | the other 32 g2 rows
                    copy_back(Ly.w2, h, P.wm, 0, 4, dst);
                    copy_back(Ly.a2, h, P.am, 0, 4, dst);
                    if (l > 0) copy_back(Ly.v2, h, P.vm, 0, 4, dst);
                    copy_back(Ly.g2, h, P.gm, 0, 4, dst);
                }
            }
        }
    }
    char* dst = hstream + (size_t)cta * (size_t)hslot;
    for (int k = pl.ph0[DSP_HEAD]; k < pl.ph0[DSP_HEAD] + pl.phn[DSP_HEAD]; ++k) {
        copy_chunk(P.head, pl.ctab[k], dst);
        dst += pl.ctab[k].cb;
    }
}

}  // namespace rsv
