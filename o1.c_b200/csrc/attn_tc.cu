// Prefix-causal flash attention on the sm_100a tensor cores.  Replaces the
// cuDNN SDPA graphs (o1.c src/cuda/hd_cudnn_sdpa.cu:114-441) and the eager
// S x S path (src/cuda/attn.cu:22-174): scores are never written to HBM.
//
//   out[s, h, :] = softmax_t( q[s,h,:] . k[t,kh,:] / sqrt(128) + mask[s,t] ) v[t,kh,:]
//   kh = h / (heads / kv_heads); mask: rows s < ar_len see keys t <= s,
//   rows s >= ar_len see every key (o1.c src/runtime/sequence.c:120-142).
//
// Two kernels.  flash_attn1_kernel is the one that runs: one query tile per CTA with triple-buffered scores (described at the kernel).
// The other, where a program asks for it (attention_tile_mode), flash_attn_kernel:
// one CTA = 256 query rows of one head: two query tiles of 128 rows that share every K/V tile
// brought into shared memory (half the K/V fill per query row of a one-tile CTA, and the two tiles'
// softmax and MMA phases overlap each other).  Operands stay seq-major ([S, heads*128]); head split /
// merge (attn.cu:180-218) disappear into the TMA coordinates and the output addressing.
//   warp 0     : TMA producer (two Q tiles once, then K tiles (2 stages) and V tiles (3 stages))
//   warp 1     : tcgen05.mma issuer: S_g = Q_g K_j^T into TMEM, O_g += P_g V_j with P_g read from
//                tensor memory and V as an MN-major operand, alternating between the groups
//   warps 2..17: two softmax groups of eight warps, one group per query tile, two threads per query
//                row (TMEM lane == row; the warps w and w+4 of a group own the same 32 lanes and
//                take 64 score columns each): fp32 scores -> running max (halves exchanged through
//                shared memory) / sum in the exp2 domain -> bf16 P written back into tensor memory
//                over the scores.  The softmax -> PV -> next-scores round trip of a group is the
//                critical path of the kernel, which is why a row is split over two threads.
// An accumulator is only rescaled when its running max grows by more than 2^8 (sum and
// accumulator share the same stale max, so the final division is still exact).
#include <cstdlib>
#include "common.cuh"
#include "ptx.cuh"
#include "kernels.h"

namespace o1 {

static constexpr int AQ = 128;      // query rows per softmax group
static constexpr int AQ2 = 256;     // query rows per CTA (two groups)
static constexpr int AKV = 128;     // keys per tile
static constexpr int AD = 128;      // head dim
static constexpr int TILE_BYTES = 128 * 128 * 2;   // 32 KB: two 64-column panels of 16 KB
static constexpr int PANEL_BYTES = 128 * 64 * 2;
static constexpr int K_STAGES = 2;
static constexpr int V_STAGES = 3;
static constexpr int ATTN_THREADS = 576;   // TMA warp, MMA warp, two softmax groups of eight warps
// Q x2 | K x2 | V x3 (P lives in tensor memory) + 192 B of barriers / slots + row-max exchange
static constexpr int ATTN_XCH = 2 * 2 * 128 * 4;   // [group][column half][row] floats
static constexpr int ATTN_SMEM = TILE_BYTES * (2 + K_STAGES + V_STAGES) + 192 + ATTN_XCH;

// n / d for 0 <= n < 2^31 without a division (Granlund and Montgomery, PLDI 1994: multiply by 2^32 (2^s - d) / d + 1, add n, shift
// by s = ceil(log2 d)): a work unit takes four divisions, some 150 cycles each, before its first copy can start.
struct FastDiv {
    uint32_t mul, shift;
    void set(int d) {
        shift = 0;
        while ((1ll << shift) < d) ++shift;
        mul = (uint32_t)((((1ull << shift) - (uint64_t)d) << 32) / (uint64_t)d + 1);
    }
    __device__ __forceinline__ int div(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shift); }
};

struct AttnArgs {
    uint16_t* out;
    int ldo;
    int S, heads, kv_heads, ar_len;
    int row_lo, row_hi; // only query rows in [row_lo, row_hi) are computed and written (whole range: 0, S)
    float scale_log2;   // scale * log2(e)
    // head h of q sits at TMA coordinates (h*q_hc + d, h*q_hr + s); same for k/v with
    // the kv head.  seq-major [S, H*128]: hc = 128, hr = 0; head-major [H,S,128]: hc = 0, hr = S.
    int q_hc, q_hr, kv_hc, kv_hr;
    long out_hoff;      // element offset of head h in the output: h * out_hoff
    int* err;
    // out_rows > 0: output rows [b*out_rows, (b+1)*out_rows) are written to out_tab[b] (possibly another
    // GPU's memory) instead of out
    int out_rows;
    uint16_t* out_tab[8];
    // Work items: item = head * nqb + query block.  The first n_plain items are one CTA each.  Each of the
    // remaining (tail) items is cut along the keys into `ways` CTAs that leave unnormalised partial results
    // (accumulator, running max, row sum) in part_o / part_ml for attn_merge_kernel, so that the last,
    // partly filled wave of CTAs is short.  ways == 1: no tail.
    int nqb, n_plain, ways;
    // One-tile kernel (unit_at()): query blocks [qb0, qb0 + nqb), the first nc of them all causal; n_full of the plain items see every
    // key, n_long work units with the parts of the tail, and n_short causal items.
    int qb0, nc, n_full, n_long, n_short;
    int out_copy;       // all rows go to `out`: they leave through a tensor map
    int hf, hr;         // the plain items are hf whole heads and the first hr query blocks of another
    FastDiv by_full, by_nqb, by_ways, by_hf, by_hf1, by_group;    // nqb - nc, nqb, ways, hf, hf + 1, query heads per key head
    float* part_o;      // [slot][rows of an item][128] fp32, slot = (item - n_plain) * ways + part
    float* part_ml;     // [slot][rows of an item][2]: max (exp2 domain) the partial is relative to, row sum
};

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Packed fp32 pairs (one issue slot for two lanes' worth of FMA / ADD): the softmax warps are bound by
// instruction issue and latency, not by a pipe, so halving the FMA and ADD count of the exp2 loop is time saved.
__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// P = exp2(s * scale - m) for this thread's 64 scores, rounded to bf16 pairs and written to 32 tensor-memory
// columns at t_p; returns the fp32 sum of the unrounded values.
__device__ __forceinline__ float softmax_exp_store(const uint32_t (&r)[2][32], uint64_t scale2, uint64_t negm2, uint32_t t_p) {
    uint64_t lsa = pack_f32x2(0.f, 0.f), lsb = lsa;     // two independent chains of pair sums
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])),
                                          scale2, negm2);
            float x0, x1;
            unpack_f32x2(x2, x0, x1);
            const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
            if (i & 1) lsb = add_f32x2(lsb, pack_f32x2(p0, p1));
            else lsa = add_f32x2(lsa, pack_f32x2(p0, p1));
            pk[i] = cvt_bf16x2(p0, p1);
        }
        tmem_st16(t_p + c * 16, pk);
    }
    tmem_st_wait();
    float s0, s1;
    unpack_f32x2(add_f32x2(lsa, lsb), s0, s1);
    return s0 + s1;
}

__global__ void __launch_bounds__(ATTN_THREADS, 1)
flash_attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const AttnArgs a) {
    // 7 tiles of 32 KB fill the SM's shared memory, so there is no room for an alignment pad or
    // static arrays: the dynamic window itself is declared 1024-byte aligned (checked below).
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_s = smem;                               // two query tiles
    uint8_t* k_s = q_s + 2 * TILE_BYTES;
    uint8_t* v_s = k_s + K_STAGES * TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + V_STAGES * TILE_BYTES);
    uint64_t* q_full = bars;                // 1
    uint64_t* k_full = bars + 1;            // K_STAGES
    uint64_t* k_empty = k_full + K_STAGES;
    uint64_t* v_full = k_empty + K_STAGES;  // V_STAGES
    uint64_t* v_empty = v_full + V_STAGES;
    uint64_t* s_full = v_empty + V_STAGES;  // 2 (one per group)
    uint64_t* p_ready = s_full + 2;         // 2
    uint64_t* o_done = p_ready + 2;         // 1
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 1);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    float* xch = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 192);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    int item = blockIdx.x, part = 0, ways = 1;
    if (item >= a.n_plain) {
        const int t = item - a.n_plain;
        item = a.n_plain + t / a.ways;
        part = t - (t / a.ways) * a.ways;
        ways = a.ways;
    }
    const int h = item / a.nqb;
    const int q0 = (item - h * a.nqb) * AQ2;
    const int kh = h / (a.heads / a.kv_heads);
    if (q0 + AQ2 <= a.row_lo || q0 >= a.row_hi) { grid_dep_wait(); return; }   // no row of this block is wanted (whole CTA, before any set-up)

    // keys this pair of query tiles can see (the second tile's range covers the first's)
    int kv_end = a.S;
    if (q0 + AQ2 - 1 < a.ar_len) kv_end = q0 + AQ2;   // all rows causal: keys <= last row
    if (kv_end > a.S) kv_end = a.S;
    const int tiles_all = (kv_end + AKV - 1) / AKV;
    const int j0 = (int)((long)part * tiles_all / ways);                  // first key tile of this CTA
    const int n_tiles = (int)((long)(part + 1) * tiles_all / ways) - j0;  // and how many it covers
    if (n_tiles <= 0) {
        // a part of a tail item that has fewer key tiles than parts: an empty partial (max -inf, sum 0), nothing else
        grid_dep_wait();
        if (threadIdx.x < AQ2) {
            const int slot = (item - a.n_plain) * ways + part;
            *reinterpret_cast<float2*>(a.part_ml + ((size_t)slot * AQ2 + threadIdx.x) * 2) = make_float2(-INFINITY, 0.f);
        }
        return;
    }

    if (threadIdx.x == 0) {
        int ab = error_word(a.err);
        if (ab == 0 && (smem_u32(smem) & 1023u) != 0) { ab = 20; atomicExch(a.err, 20); }
        *s_abort = ab;
    }
    __syncthreads();
    if (*s_abort != 0) { grid_dep_wait(); return; }

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < K_STAGES; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
        for (int s = 0; s < V_STAGES; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_ready[s], 8); }
        mbar_init(o_done, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_S = tmem_base;         // scores of the two groups: columns [0,128) and [128,256)
    const uint32_t tmem_O = tmem_base + 256;   // output accumulators of the two groups: [256,384), [384,512)

    if (warp == 0) {
        // -------------------------------------------------------- TMA producer
        if (elect_one()) {
            tma_prefetch_desc(&tmQ);
            tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmV);
            mbar_expect_tx(q_full, 2 * TILE_BYTES);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                tma_load_2d(q_s + g * TILE_BYTES, &tmQ, q_full, h * a.q_hc, h * a.q_hr + q0 + g * AQ);
                tma_load_2d(q_s + g * TILE_BYTES + PANEL_BYTES, &tmQ, q_full, h * a.q_hc + 64,
                            h * a.q_hr + q0 + g * AQ);
            }
            auto load_k = [&](int j) -> bool {
                const int st = j % K_STAGES;
                if (!mbar_wait(&k_empty[st], ((j / K_STAGES) & 1) ^ 1)) { atomicExch(a.err, 11); return false; }
                mbar_expect_tx(&k_full[st], TILE_BYTES);
                tma_load_2d(k_s + st * TILE_BYTES, &tmK, &k_full[st], kh * a.kv_hc, kh * a.kv_hr + (j0 + j) * AKV);
                tma_load_2d(k_s + st * TILE_BYTES + PANEL_BYTES, &tmK, &k_full[st], kh * a.kv_hc + 64,
                            kh * a.kv_hr + (j0 + j) * AKV);
                return true;
            };
            auto load_v = [&](int j) -> bool {
                const int st = j % V_STAGES;
                if (!mbar_wait(&v_empty[st], ((j / V_STAGES) & 1) ^ 1)) { atomicExch(a.err, 12); return false; }
                mbar_expect_tx(&v_full[st], TILE_BYTES);
                tma_load_2d(v_s + st * TILE_BYTES, &tmV, &v_full[st], kh * a.kv_hc, kh * a.kv_hr + (j0 + j) * AKV);
                tma_load_2d(v_s + st * TILE_BYTES + PANEL_BYTES, &tmV, &v_full[st], kh * a.kv_hc + 64,
                            kh * a.kv_hr + (j0 + j) * AKV);
                return true;
            };
            // load order follows the consumer: K0, then per tile V(j), K(j+1)
            bool ok = load_k(0);
            for (int j = 0; j < n_tiles && ok; ++j) {
                ok = load_v(j);
                if (ok && j + 1 < n_tiles) ok = load_k(j + 1);
            }
        }
    } else if (warp == 1) {
        // -------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0);
            constexpr uint32_t idesc_pv = umma_idesc_bf16(128, 128, 0, 1);  // V is MN-major
            bool ok = mbar_wait(q_full, 0);
            if (!ok) atomicExch(a.err, 13);
            // S_g = Q_g K_j^T; one descriptor per operand tile, the eight K steps only move its
            // 16-byte-unit address field
            auto issue_qk = [&](int g, uint64_t k_desc) {
                const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s + g * TILE_BYTES), 16, 1024);
#pragma unroll
                for (int kk = 0; kk < AD / 16; ++kk) {
                    const uint64_t off = (uint64_t)(((kk >> 2) * PANEL_BYTES + (kk & 3) * 32) >> 4);
                    umma_ss(tmem_S + g * 128, q_desc + off, k_desc + off, idesc_qk, kk != 0);
                }
                umma_commit(&s_full[g]);
            };
            auto k_ready = [&](int j, uint64_t& k_desc) -> bool {
                const int st = j % K_STAGES;
                if (!mbar_wait(&k_full[st], (j / K_STAGES) & 1)) { atomicExch(a.err, 14); return false; }
                tc_fence_after();
                k_desc = umma_desc_sw128(smem_u32(k_s + st * TILE_BYTES), 16, 1024);
                return true;
            };
            uint64_t k_desc = 0;
            if (ok) ok = k_ready(0, k_desc);
            if (ok) {
                issue_qk(0, k_desc);
                issue_qk(1, k_desc);
                umma_commit(&k_empty[0]);
            }
            // Per key tile j and group g: O_g += P_g(j) V_j, then S_g = Q_g K_{j+1}^T.  P_g overlays S_g in
            // tensor memory: MMAs of one thread execute in issue order, so the next score product
            // overwrites it only after the PV product has consumed it.  While group g runs its softmax
            // the tensor pipe works on the other group.
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int vst = j % V_STAGES;
                if (!mbar_wait(&v_full[vst], (j / V_STAGES) & 1)) { atomicExch(a.err, 15); ok = false; break; }
                const uint64_t v_desc = umma_desc_sw128(smem_u32(v_s + vst * TILE_BYTES), PANEL_BYTES, 1024);
                const bool more = j + 1 < n_tiles;
                if (more && !k_ready(j + 1, k_desc)) { ok = false; break; }
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    if (!mbar_wait(&p_ready[g], j & 1)) { atomicExch(a.err, 16); ok = false; break; }
                    tc_fence_after();
                    const uint32_t p_tmem = tmem_S + g * 128;   // bf16 P in the first 64 score columns
#pragma unroll
                    for (int kk = 0; kk < AKV / 16; ++kk)       // 16 keys down per step, 128 B per key row
                        umma_ts(tmem_O + g * 128, p_tmem + kk * 8, v_desc + (uint64_t)((kk * 16 * 128) >> 4),
                                idesc_pv, (j | kk) != 0);
                    if (more) issue_qk(g, k_desc);
                }
                if (!ok) break;
                umma_commit(&v_empty[vst]);
                if (more) umma_commit(&k_empty[(j + 1) % K_STAGES]);
            }
            umma_commit(o_done);
        }
    } else {
        // -------------------------------------------------------- softmax groups + output
        const int grp = (warp - 2) >> 3;         // which of the CTA's two query tiles
        const int half = ((warp - 2) >> 2) & 1;  // which 64 score / output columns of the row
        const int qd = warp & 3;                 // TMEM lane quadrant this warp may access
        const int row = qd * 32 + lane;          // row within the query tile
        const int qg0 = q0 + grp * AQ;           // first row of this group's tile
        const int row_g = qg0 + row;             // global query index
        const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
        const bool tile_has_causal = qg0 < a.ar_len;
        const bool row_causal = row_g < a.ar_len;
        const uint32_t t_s = tmem_S + grp * 128 + lane_off;
        const uint32_t t_o = tmem_O + grp * 128 + half * 64 + lane_off;
        float* x_mine = xch + (grp * 2 + half) * 128 + row;
        const float* x_other = xch + (grp * 2 + (half ^ 1)) * 128 + row;
        const int bar_id = 1 + grp;              // named barrier of the group's 256 threads
        constexpr int BAR_THREADS = 256;
        float m_used = -INFINITY;                // max the stored P / l / O of this row are relative to
        float l = 0.f;                           // this thread's share of the row sum
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int kv0 = (j0 + j) * AKV + half * 64;
            if (!mbar_wait(&s_full[grp], j & 1)) { atomicExch(a.err, 17); ok = false; break; }
            tc_fence_after();
            const bool need_mask = (kv0 + 64 > a.S) || (tile_has_causal && kv0 + 63 > qg0);
            // this thread's 64 fp32 scores go to registers with one wait
            uint32_t r[2][32];
            tmem_ld32(t_s + half * 64, r[0]);
            tmem_ld32(t_s + half * 64 + 32, r[1]);
            tmem_ld_wait();
            if (need_mask) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = kv0 + c * 32 + i;
                        const bool allow = key < a.S && (!row_causal || key <= row_g);
                        if (!allow) r[c][i] = 0xff800000u;   // -inf
                    }
            }
            float mx;
            {
                // three-input max: 64 scores in 32 instructions, four independent chains
                float mxa = -INFINITY, mxb = -INFINITY, mxc = -INFINITY, mxd = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    mxa = max3(mxa, __uint_as_float(r[0][2 * i]), __uint_as_float(r[0][2 * i + 1]));
                    mxb = max3(mxb, __uint_as_float(r[0][16 + 2 * i]), __uint_as_float(r[0][16 + 2 * i + 1]));
                    mxc = max3(mxc, __uint_as_float(r[1][2 * i]), __uint_as_float(r[1][2 * i + 1]));
                    mxd = max3(mxd, __uint_as_float(r[1][16 + 2 * i]), __uint_as_float(r[1][16 + 2 * i + 1]));
                }
                mx = max3(mxa, mxb, fmaxf(mxc, mxd));
            }
            // row max over both halves: the partner thread's value comes through shared memory.  The slot
            // is rewritten one tile later, after the partner has arrived on p_ready and a new s_full
            // has come round, so one barrier per tile is enough.
            *x_mine = mx;
            asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(BAR_THREADS) : "memory");
            mx = fmaxf(mx, *x_other);
            const float m_tile = mx * a.scale_log2;
            const bool grow = (m_tile - m_used) > 8.0f;      // also true while m_used == -inf
            if (__any_sync(0xffffffffu, grow)) {
                float alpha = 1.0f;
                if (grow) {
                    alpha = ex2_approx(m_used - m_tile);         // 0 on the first tile
                    m_used = m_tile;
                    l *= alpha;
                }
                if (j >= 1) {
                    // PV_g(j-1) was issued before QK_g(j), whose completion s_full just reported: O is
                    // complete and idle until PV_g(j), which waits for p_ready.  Each thread scales its
                    // own 64 output columns.
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[16];
                        tmem_ld16(t_o + c * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st16(t_o + c * 16, o);
                    }
                    tmem_st_wait();
                }
            }
            // P = exp2(s * scale_log2 - m_used) as packed bf16 pairs, written over the score columns
            // (this half's 64 scores are in registers by now, and the partner only writes after the
            // barrier above, i.e. after both loads): 64 scores become 32 columns at [half*32, +32).
            // A causal row may have no visible key in this tile and none before: m_used is still -inf
            // then and every score is masked; 0 keeps exp2(-inf + 0) = 0 instead of exp2(-inf + inf)
            const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
            const uint64_t scale2 = pack_f32x2(a.scale_log2, a.scale_log2), negm2 = pack_f32x2(neg_m, neg_m);
            l += softmax_exp_store(r, scale2, negm2, t_s + half * 32);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[grp]);
        }
        // ---- output: O / l -> bf16 -> out[row_g, h*128 + half*64 ..]
        if (ok && n_tiles > 0) {
            const int failed = error_word(a.err);
            if (!mbar_wait(o_done, 0)) { atomicExch(a.err, 19); ok = false; }
            tc_fence_after();
            if (failed) ok = false;
        }
        // the row sum is the two threads' shares together (same exchange slots; every thread of the
        // group reaches this barrier: a failed wait above fails for the whole group alike)
        *x_mine = l;
        asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(BAR_THREADS) : "memory");
        l += *x_other;
        if (ok && ways > 1) {
            // partial result of a key range: accumulator as it is (relative to m_used), max and row sum
            const int slot = (item - a.n_plain) * ways + part;
            const int prow = grp * AQ + row;
            float* po = a.part_o + ((size_t)slot * AQ2 + prow) * AD + half * 64;
            if (half == 0) {
                float2 ml = make_float2(m_used, l);
                *reinterpret_cast<float2*>(a.part_ml + ((size_t)slot * AQ2 + prow) * 2) = ml;
            }
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t o[32];
                tmem_ld32(t_o + c * 32, o);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    *reinterpret_cast<uint4*>(po + c * 32 + i * 4) = make_uint4(o[i * 4], o[i * 4 + 1], o[i * 4 + 2], o[i * 4 + 3]);
            }
        } else if (ok && a.out_rows > 0) {
            // Row blocks of the output live in other GPUs' memory: leave as full 128-byte row segments (4 rows
            // per store instruction) instead of 16-byte pieces of 32 rows.  The staging slice is this warp's
            // 4 KB of the Q tiles, which no MMA reads any more once o_done has completed.
            const float inv_l = 1.0f / l;
            uint8_t* stg = q_s + (warp - 2) * (32 * 128);
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t o[32];
                tmem_ld32(t_o + c * 32, o);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint4 pk;
                    pk.x = cvt_bf16x2(__uint_as_float(o[i * 8 + 0]) * inv_l, __uint_as_float(o[i * 8 + 1]) * inv_l);
                    pk.y = cvt_bf16x2(__uint_as_float(o[i * 8 + 2]) * inv_l, __uint_as_float(o[i * 8 + 3]) * inv_l);
                    pk.z = cvt_bf16x2(__uint_as_float(o[i * 8 + 4]) * inv_l, __uint_as_float(o[i * 8 + 5]) * inv_l);
                    pk.w = cvt_bf16x2(__uint_as_float(o[i * 8 + 6]) * inv_l, __uint_as_float(o[i * 8 + 7]) * inv_l);
                    const int j = c * 4 + i;
                    *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) * 16)) = pk;
                }
            }
            __syncwarp();
            const int ch = lane & 7;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int rr = k * 4 + (lane >> 3);
                const uint4 v = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((ch ^ (rr & 7)) * 16));
                const int rg = qg0 + qd * 32 + rr;
                if (rg < a.row_hi && rg >= a.row_lo) {
                    const int blk = rg / a.out_rows;
                    uint16_t* dst = a.out_tab[blk] + (size_t)(rg - blk * a.out_rows) * a.ldo + (size_t)h * a.out_hoff +
                                    half * 64 + ch * 8;
                    *reinterpret_cast<uint4*>(dst) = v;
                }
            }
        } else if (ok) {
            const float inv_l = 1.0f / l;
            uint16_t* dst = a.out + (size_t)row_g * a.ldo + (size_t)h * a.out_hoff + half * 64;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t o[32];
                tmem_ld32(t_o + c * 32, o);
                tmem_ld_wait();
                if (row_g < a.row_hi && row_g >= a.row_lo) {
                    uint4* d4 = reinterpret_cast<uint4*>(dst + c * 32);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 pk;
                        pk.x = cvt_bf16x2(__uint_as_float(o[i * 8 + 0]) * inv_l, __uint_as_float(o[i * 8 + 1]) * inv_l);
                        pk.y = cvt_bf16x2(__uint_as_float(o[i * 8 + 2]) * inv_l, __uint_as_float(o[i * 8 + 3]) * inv_l);
                        pk.z = cvt_bf16x2(__uint_as_float(o[i * 8 + 4]) * inv_l, __uint_as_float(o[i * 8 + 5]) * inv_l);
                        pk.w = cvt_bf16x2(__uint_as_float(o[i * 8 + 6]) * inv_l, __uint_as_float(o[i * 8 + 7]) * inv_l);
                        d4[i] = pk;
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ---------------------------------------------------------------------------------------------------------------
// One query tile at a time, scores triple-buffered: work items of 128 rows fill 148 SMs at short sequences too (S = 1280: 320
// instead of 160), and no serial chain as in the two-tile kernel.  Tensor memory: three score buffers of 128 columns + one output accumulator.  The MMA
// thread issues S(g+3) = Q K^T right after PV(g), so the scores of the next two key tiles are always there or on their
// way and the softmax warps never wait for a score product that waits for them.  Warps 2..9 and 10..17 are two softmax
// sets that take alternate key tiles (two threads per row, as above); they agree on the running max through shared
// memory: the set that takes tile g waits for the other set's decision for tile g-1 (made early in its phase) before it
// decides for tile g.
// A CTA stays on its SM and takes one work unit after the other (unit_at()): the key tiles of its units are ONE stream, counted by g,
// that copies, score products and softmax sets run through without a stop.  The next unit's Q, K and first three score products are
// there before this one's last PV, the set that did not take the last key tile goes on with the next unit at once, and the other one
// leaves this unit's rows in its Q tile, from where another warp takes them to memory.  What stays between two units is the
// accumulator, which PV of the next one may only overwrite once it has been read.
// A CTA for each item (barriers, tensor memory, first copies and the way out for each) / units in a stream, 32 / 8 heads, us: 592
// rows 18.8 / 14.9, 1280 rows 39.2 / 31.9, 3157 rows 175 / 152, 8000 rows 960 / 852, 16640 rows alike (3.7 to 3.9 ms at the power cap), all rows
// causal 1280 rows 29.6 / 20.5, 3157 rows 115 / 88; the tower's 16 heads of 72 at 4096 patches 124 / 107; one unit for each CTA (200
// rows) 6.5 / 6.5.  The same bits.  A key tile takes 1340 to 1410 cycles (1560 before), 1250 of which shared memory needs for the
// operands (160 KB: Q and K 64, V 32, the copies 64); storing the rows by the set itself cost 2 to 5 % of these times.
// EXACT: the reference max is a row's exact score, as in the two-tile kernel, so that P of that key is exactly 1; from T1_EXACT_ROWS
// rows on, where that kernel used to run.  Else the max is rounded up to bf16 (half the exchange): the error against 64 bits is 6 %
// larger (16640 rows 2.20e-3 against 2.06e-3, alike from 592 rows on).  The time is the same, 600 to 4500 rows 1 % longer; shorter
// sequences keep it because 36 blocks carry a change of single roundings as far as 4e-2 (2-norm), and their results stay
// what they have always been.
// Measured against the two-tile kernel: see attention_tile_mode().
static constexpr int T1_ROWS = 128;       // query rows per work item
static constexpr int T1_THREADS = ATTN_THREADS + 32;    // (and the store warp)
static constexpr int T1_Q_STAGES = 2;
static constexpr int T1_K_STAGES = 2;
static constexpr int T1_V_STAGES = 3;
static constexpr int T1_S_BUFS = 3;       // score buffers in tensor memory
static constexpr int T1_EXACT_ROWS = 8192;
static constexpr int T1_BARS = 256, T1_UNITS = 4;     // (unit table: see T1_UNITS x 32 bytes behind the barriers)
// row-max exchange ([set][use][half][row] bf16, EXACT: [set][half][row] floats); behind it (not EXACT) the max in force, [tile parity][row]
static constexpr int T1_XCH = 2048;
static constexpr int T1_SMEM = TILE_BYTES * (T1_Q_STAGES + T1_K_STAGES + T1_V_STAGES) + T1_BARS + T1_UNITS * 32 + T1_XCH + 512;

// bounded wait with one outcome for the whole warp (the code behind it issues warp-wide tensor-memory accesses)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}

// DH: columns of a head that hold data.  72 (the vision tower; heads stored 128 apart, columns 72..79 zero) takes five of
// the eight K steps of Q K^T and 80 of the 128 output columns; what the second panels hold beyond that is never read.
// NSEG: sequences in one launch (the two branches of a guided step: at 296 rows each has 96 work items for 148 SMs).
template <int NSEG>
struct Attn1Params {
    CUtensorMap q[NSEG], k[NSEG], v[NSEG], o[NSEG];
    AttnArgs a[NSEG];
};

// A work unit: a query tile of a head with all the keys it sees, or one of the parts of a tail item.
struct alignas(16) AttnUnit {
    int h, q0;       // head (-1: no unit, the CTA is done), first query row
    int kv_c, kv_r;  // tensor-map coordinates of its first key tile
    int j0, n;       // first key tile, and how many (0: a part of an item that has fewer key tiles than parts)
    int slot;        // where a part's results go; -1: a whole item
    int seg;         // sequence
};
// Unit u of a launch.  CTA b takes the units b, b + grid, ...: those that see every key (and the parts) come first, those of causal
// query tiles, which stop at the diagonal, after them with the longest in front, so that the rounds' sums are even (1280
// rows, of which 256 causal, 32 heads: at most 22 key tiles for a CTA; in the order of the heads 30).
template <int NSEG>
__device__ __forceinline__ AttnUnit unit_at(const Attn1Params<NSEG>& par, int u) {
    int seg = 0;
    if (NSEG > 1) {
        const int l0 = par.a[0].n_long, l1 = par.a[NSEG - 1].n_long, s0 = par.a[0].n_short;
        if (u >= l0 + l1) {
            u -= l1;
            if (u >= l0 + s0) { u += l1 - l0 - s0; seg = 1; }
        } else if (u >= l0) { u -= l0; seg = 1; }
    }
    const AttnArgs& a = par.a[seg];
    AttnUnit un;
    un.seg = seg;
    int qb, part = 0;
    un.slot = -1;
    if (u < a.n_full) {
        un.h = a.by_full.div(u);
        qb = a.nc + u - un.h * (a.nqb - a.nc);
    } else if (u < a.n_long) {
        un.slot = u - a.n_full;
        const int i = a.by_ways.div(un.slot), item = a.n_plain + i;
        part = un.slot - i * a.ways;
        un.h = a.by_nqb.div(item);
        qb = item - un.h * a.nqb;
    } else {
        // hf causal tiles of each number from hr on, one more of each below
        int v = u - a.n_long, top = a.nc;
        if (top > a.hr && v >= (top - a.hr) * a.hf) { v -= (top - a.hr) * a.hf; top = a.hr; }
        const int cnt = a.hf + (top <= a.hr), c = top <= a.hr ? a.by_hf1.div(v) : a.by_hf.div(v);
        un.h = v - c * cnt;
        qb = top - 1 - c;
    }
    un.q0 = (a.qb0 + qb) * T1_ROWS;
    // keys this query tile can see
    int kv_end = a.S;
    if (un.q0 + T1_ROWS - 1 < a.ar_len) kv_end = un.q0 + T1_ROWS;   // all rows causal: keys <= last row
    if (kv_end > a.S) kv_end = a.S;
    const int tiles = (kv_end + AKV - 1) / AKV;
    un.j0 = 0;
    un.n = tiles;
    if (un.slot >= 0) {
        un.j0 = a.by_ways.div(part * tiles);
        un.n = a.by_ways.div((part + 1) * tiles) - un.j0;
    }
    const int kh = a.by_group.div(un.h);
    un.kv_c = kh * a.kv_hc;
    un.kv_r = kh * a.kv_hr + un.j0 * AKV;
    return un;
}
// The end of a unit: the rows of one of its warps, O / l -> bf16 -> the unit's Q tile, from where the store warp takes them (a part's
// results go out from here).  stg: 4 KB of the warp's own (32 rows of half a head, 128-byte swizzle), at their beginning the shares
// of the rows' sums.  (16 columns at a time: with 32 the compiler puts values of the loop over the key tiles into local memory, and
// with all but a few KB of the SM's memory taken by tiles that made the whole kernel 1.5 times as slow.)
__device__ __forceinline__ void attn_stage_rows(uint8_t* stg, uint32_t t_o, uint64_t* o_free, uint64_t* o_staged, float m_used, float* part_o,
                                             float* part_ml /* of the warp's first row; null: a whole item, or not wanted */, bool whole) {
    const int lane = threadIdx.x & 31;
    const float* sh = reinterpret_cast<const float*>(stg) + lane;
    const float lsum = (sh[0] + sh[32]) + (sh[64] + sh[96]);
    const float inv_l = 1.0f / lsum;
    // partial result of a key range: accumulator as it is (relative to the max), max and row sum
    if (part_ml) *reinterpret_cast<float2*>(part_ml + lane * 2) = make_float2(m_used, lsum);
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
        uint32_t o[16];
        tmem_ld16(t_o + c * 16, o);
        tmem_ld_wait();
        if (c == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free);
        }
        if (whole) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                uint4 pk;
                pk.x = cvt_bf16x2(__uint_as_float(o[i * 8 + 0]) * inv_l, __uint_as_float(o[i * 8 + 1]) * inv_l);
                pk.y = cvt_bf16x2(__uint_as_float(o[i * 8 + 2]) * inv_l, __uint_as_float(o[i * 8 + 3]) * inv_l);
                pk.z = cvt_bf16x2(__uint_as_float(o[i * 8 + 4]) * inv_l, __uint_as_float(o[i * 8 + 5]) * inv_l);
                pk.w = cvt_bf16x2(__uint_as_float(o[i * 8 + 6]) * inv_l, __uint_as_float(o[i * 8 + 7]) * inv_l);
                *reinterpret_cast<uint4*>(stg + lane * 128 + (((c * 2 + i) ^ (lane & 7)) * 16)) = pk;
            }
        } else if (part_o) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<uint4*>(part_o + lane * AD + c * 16 + i * 4) = make_uint4(o[i * 4], o[i * 4 + 1], o[i * 4 + 2], o[i * 4 + 3]);
        }
    }
    // (for the copy that takes the rows out, and the one that fills the place again)
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(o_staged);
}

template <int DH, int NSEG, bool EXACT>
__global__ void __launch_bounds__(T1_THREADS, 1) flash_attn1_kernel(const __grid_constant__ Attn1Params<NSEG> par) {
    constexpr int DN = (DH + 15) & ~15;      // columns the MMAs work on
    // Q x2 | K x2 | V x3: 7 tiles of 32 KB again, the window 1024-byte aligned (checked below)
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_s = smem;
    uint8_t* k_s = q_s + T1_Q_STAGES * TILE_BYTES;
    uint8_t* v_s = k_s + T1_K_STAGES * TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + T1_V_STAGES * TILE_BYTES);
    uint64_t* q_full = bars;                   // T1_Q_STAGES, by unit
    uint64_t* q_empty = q_full + T1_Q_STAGES;  // T1_Q_STAGES: the unit's score products are done and its rows have left
    uint64_t* k_full = q_empty + T1_Q_STAGES;  // T1_K_STAGES, by tile
    uint64_t* k_empty = k_full + T1_K_STAGES;
    uint64_t* v_full = k_empty + T1_K_STAGES;  // T1_V_STAGES
    uint64_t* v_empty = v_full + T1_V_STAGES;
    uint64_t* s_full = v_empty + T1_V_STAGES;  // T1_S_BUFS (one per score buffer)
    uint64_t* p_ready = s_full + T1_S_BUFS;    // T1_S_BUFS
    uint64_t* m_pub = p_ready + T1_S_BUFS;     // 2 (one per softmax set)
    uint64_t* l_full = m_pub + 2;              // 2, by unit: all shares of the row sums are there
    uint64_t* o_free = l_full + 2;             // 1: the accumulator has been read
    uint64_t* u_full = o_free + 1;             // T1_UNITS: the unit stands in the table
    uint64_t* o_staged = u_full + T1_UNITS;    // 2, by unit: its rows lie in its Q tile
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_staged + 2);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    // The CTA's units as the producer comes to them, the last entry with n = 0.  It is at most three ahead of the unit whose rows
    // are being stored: it waits for a place for Q.
    AttnUnit* units = reinterpret_cast<AttnUnit*>(reinterpret_cast<uint8_t*>(bars) + T1_BARS);
    float* xch = reinterpret_cast<float*>(units + T1_UNITS);

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    int* const err = par.a[0].err;

    // (the error word and the descriptors are on their way while the barriers and tensor memory are set up)
    if (threadIdx.x == 96) {
        int ab = error_word(err);
        if (ab == 0 && (smem_u32(smem) & 1023u) != 0) { ab = 20; atomicExch(err, 20); }
        *s_abort = ab;
    }
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < NSEG; ++i) {
            tma_prefetch_desc(&par.q[i]);
            tma_prefetch_desc(&par.k[i]);
            tma_prefetch_desc(&par.v[i]);
            if (par.a[i].out_copy) tma_prefetch_desc(&par.o[i]);
        }
    }
    if (threadIdx.x == 64) {
        for (int s = 0; s < T1_Q_STAGES; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 2); }
        for (int s = 0; s < T1_K_STAGES; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
        for (int s = 0; s < T1_V_STAGES; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        for (int s = 0; s < T1_S_BUFS; ++s) { mbar_init(&s_full[s], 1); mbar_init(&p_ready[s], 8); }
        for (int s = 0; s < 2; ++s) { mbar_init(&m_pub[s], 8); mbar_init(&l_full[s], 16); mbar_init(&o_staged[s], 8); }
        mbar_init(o_free, 8);
        for (int s = 0; s < T1_UNITS; ++s) mbar_init(&u_full[s], 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    AttnUnit un;                 // (the producer's first one: known before the kernel in front of this one has ended)
    if (warp == 0) un = unit_at<NSEG>(par, blockIdx.x);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    if (*s_abort != 0) {
        if (warp == 1) tmem_dealloc(tmem_base, 512);
        return;
    }
    const uint32_t tmem_S = tmem_base;         // three score buffers: columns [0,128), [128,256), [256,384)
    const uint32_t tmem_O = tmem_base + 384;   // output accumulator: [384,512)

    if (warp == 0) {
        // -------------------------------------------------------- TMA producer
        if (elect_one()) {
            auto tile = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
                mbar_expect_tx(bar, TILE_BYTES);
                tma_load_2d(dst, map, bar, c0, c1);
                tma_load_2d(dst + PANEL_BYTES, map, bar, c0 + 64, c1);
            };
            int u = blockIdx.x, ki = 0, jk = 0, i = 0;       // K: unit, its number among this CTA's, key tile in it, tile of the stream
            int vi = 0, jv = 0, vn = 0;
            bool more = true, first = true;
            if (un.n > 0) {
                // (the first two copies by themselves: nothing else to do in front of them)
                const AttnArgs& a = par.a[NSEG > 1 ? un.seg : 0];
                tile(q_s, &par.q[NSEG > 1 ? un.seg : 0], &q_full[0], un.h * a.q_hc, un.h * a.q_hr + un.q0);
                tile(k_s, &par.k[NSEG > 1 ? un.seg : 0], &k_full[0], un.kv_c, un.kv_r);
                units[0] = un;
                mbar_arrive(&u_full[0]);
                first = false;
                i = 1;
                if (un.n == 1) ki = 1; else jk = 1;
            }
            AttnUnit vun = un;
            int total = 0;
            for (int k = 0; k < NSEG; ++k) total += par.a[k].n_long + par.a[k].n_short;
            // the stream: K0 K1 V0 K2 V1 K3 ..; a unit's first K waits for a place for its Q, and V must not wait with it
            for (;; ++i) {
                if (i >= 2) {
                    const int g = i - 2, st = g % T1_V_STAGES;
                    if (jv == 0) { vun = units[vi % T1_UNITS]; vn = vun.n; }
                    if (vn == 0) break;
                    if (!mbar_wait(&v_empty[st], ((g / T1_V_STAGES) & 1) ^ 1)) { atomicExch(err, 12); break; }
                    tile(v_s + st * TILE_BYTES, &par.v[NSEG > 1 ? vun.seg : 0], &v_full[st], vun.kv_c, vun.kv_r + jv * AKV);
                    if (++jv == vn) { jv = 0; ++vi; }
                }
                if (!more) continue;
                if (jk == 0) {
                    while (true) {
                        if (!first) {
                            u += (int)gridDim.x;
                            if (u < total) un = unit_at<NSEG>(par, u);
                            else { un.n = 0; un.h = -1; }
                        }
                        first = false;
                        if (un.n > 0 || un.h < 0) break;
                        // a part of a tail item without key tiles: an empty partial (max -inf, sum 0), nothing else
                        for (int r = 0; r < T1_ROWS; ++r)
                            *reinterpret_cast<float2*>(par.a[NSEG > 1 ? un.seg : 0].part_ml + ((size_t)un.slot * T1_ROWS + r) * 2) = make_float2(-INFINITY, 0.f);
                    }
                    units[ki % T1_UNITS] = un;
                    mbar_arrive(&u_full[ki % T1_UNITS]);
                    if (un.n == 0) { more = false; continue; }
                    const int st = ki & 1;
                    if (!mbar_wait(&q_empty[st], ((ki >> 1) & 1) ^ 1)) { atomicExch(err, 10); break; }
                    const AttnArgs& a = par.a[NSEG > 1 ? un.seg : 0];
                    tile(q_s + st * TILE_BYTES, &par.q[NSEG > 1 ? un.seg : 0], &q_full[st], un.h * a.q_hc, un.h * a.q_hr + un.q0);
                }
                const int st = i % T1_K_STAGES;
                if (!mbar_wait(&k_empty[st], ((i / T1_K_STAGES) & 1) ^ 1)) { atomicExch(err, 11); break; }
                tile(k_s + st * TILE_BYTES, &par.k[NSEG > 1 ? un.seg : 0], &k_full[st], un.kv_c, un.kv_r + jk * AKV);
                if (++jk == un.n) { jk = 0; ++ki; }
            }
        }
    } else if (warp == 1) {
        // -------------------------------------------------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128, 0, 0);
            constexpr uint32_t idesc_pv = umma_idesc_bf16(128, DN, 0, 1);  // V is MN-major
            int gq = 0, qi = 0, jq = 0, qn = 0;      // score products: tile of the stream, unit, tile in it, tiles it has
            int pi = 0, jp = 0, pn = 0;              // the same of P V
            bool ok = true, more = true;
            // Per key tile g: S = Q K^T up to g + T1_S_BUFS - 1, the last of them into the buffer P(g - 1) leaves (MMAs of one
            // thread execute in issue order), then O += P(g) V_g.  The scores of the next T1_S_BUFS - 1 tiles are already there
            // or on their way, so the softmax warps never wait for a score product that waits for them.
            for (int g = 0; ok; ++g) {
                while (more && gq < g + T1_S_BUFS) {
                    const int qs = qi & 1, st = gq % T1_K_STAGES, b = gq % T1_S_BUFS;
                    if (jq == 0) {
                        // A unit's first product waits for the place for Q of the unit two before it, which is free once that one's
                        // rows have left, so that one's last P V has to be on its way (units of a single key tile).
                        if (qi >= pi + 2) break;
                        if (!mbar_wait(&u_full[qi % T1_UNITS], (qi / T1_UNITS) & 1)) { atomicExch(err, 23); ok = false; break; }
                        qn = units[qi % T1_UNITS].n;
                        if (qn == 0) { more = false; break; }
                        if (!mbar_wait(&q_full[qs], (qi >> 1) & 1)) { atomicExch(err, 13); ok = false; break; }
                    }
                    if (!mbar_wait(&k_full[st], (gq / T1_K_STAGES) & 1)) { atomicExch(err, 14); ok = false; break; }
                    tc_fence_after();
                    // one descriptor per operand tile, the eight K steps only move its 16-byte-unit address field
                    const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s + qs * TILE_BYTES), 16, 1024);
                    const uint64_t k_desc = umma_desc_sw128(smem_u32(k_s + st * TILE_BYTES), 16, 1024);
#pragma unroll
                    for (int kk = 0; kk < DN / 16; ++kk) {
                        const uint64_t off = (uint64_t)(((kk >> 2) * PANEL_BYTES + (kk & 3) * 32) >> 4);
                        umma_ss(tmem_S + b * 128, q_desc + off, k_desc + off, idesc_qk, kk != 0);
                    }
                    umma_commit(&s_full[b]);
                    umma_commit(&k_empty[st]);
                    ++gq;
                    if (++jq == qn) { umma_commit(&q_empty[qs]); jq = 0; ++qi; }
                }
                if (!ok) break;
                const int vst = g % T1_V_STAGES, b = g % T1_S_BUFS;
                if (jp == 0) {
                    if (qi == pi && jq == 0) break;      // the stream has ended
                    pn = units[pi % T1_UNITS].n;
                    if (pi > 0 && !mbar_wait(o_free, (pi - 1) & 1)) { atomicExch(err, 22); break; }
                }
                if (!mbar_wait(&v_full[vst], (g / T1_V_STAGES) & 1)) { atomicExch(err, 15); break; }
                const uint64_t v_desc = umma_desc_sw128(smem_u32(v_s + vst * TILE_BYTES), PANEL_BYTES, 1024);
                if (!mbar_wait(&p_ready[b], (g / T1_S_BUFS) & 1)) { atomicExch(err, 16); break; }
                tc_fence_after();
                const uint32_t p_tmem = tmem_S + b * 128;   // bf16 P in the first 64 columns of the buffer
#pragma unroll
                for (int kk = 0; kk < AKV / 16; ++kk)       // 16 keys down per step, 128 B per key row
                    umma_ts(tmem_O, p_tmem + kk * 8, v_desc + (uint64_t)((kk * 16 * 128) >> 4), idesc_pv, (jp | kk) != 0);
                umma_commit(&v_empty[vst]);
                if (++jp == pn) { jp = 0; ++pi; }
            }
        }
    } else if (warp == T1_THREADS / 32 - 1) {
        // -------------------------------------------------------- store warp
        // The unit's rows leave its Q tile: as one copy for each half of the head, or, where a range of rows is wanted or they go to
        // other GPUs' memory, as segments of 128 bytes (4 rows per store instruction).
        for (int index = 0;; ++index) {
            if (!mbar_wait_warp(&u_full[index % T1_UNITS], (index / T1_UNITS) & 1)) { atomicExch(err, 25); break; }
            const AttnUnit w = units[index % T1_UNITS];
            if (w.n == 0) break;
            const int failed = error_word(err);
            if (!mbar_wait_warp(&o_staged[index & 1], (index >> 1) & 1)) { atomicExch(err, 26); break; }
            const AttnArgs& a = par.a[NSEG > 1 ? w.seg : 0];
            const uint8_t* rows_s = q_s + (index & 1) * TILE_BYTES;
            if (w.slot < 0 && !failed) {
                if (a.out_copy) {
                    if (elect_one()) {
                        tma_store_3d(&par.o[NSEG > 1 ? w.seg : 0], rows_s, 0, w.q0, w.h);
                        tma_store_3d(&par.o[NSEG > 1 ? w.seg : 0], rows_s + PANEL_BYTES, 64, w.q0, w.h);
                        bulk_commit();
                        bulk_wait_read();
                    }
                } else {
                    const int ch = lane & 7;
                    for (int k = lane >> 3; k < 2 * T1_ROWS; k += 4) {
                        const int hf = k / T1_ROWS, rr = k - hf * T1_ROWS, rg = w.q0 + rr;
                        const uint4 v = *reinterpret_cast<const uint4*>(rows_s + hf * PANEL_BYTES + rr * 128 + ((ch ^ (rr & 7)) * 16));
                        if (hf * 64 + ch * 8 < DH && rg < a.row_hi && rg >= a.row_lo) {
                            uint16_t* dst = a.out + (size_t)rg * a.ldo;
                            if (a.out_rows > 0) {
                                const int blk = rg / a.out_rows;
                                dst = a.out_tab[blk] + (size_t)(rg - blk * a.out_rows) * a.ldo;
                            }
                            *reinterpret_cast<uint4*>(dst + (size_t)w.h * a.out_hoff + hf * 64 + ch * 8) = v;
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_empty[index & 1]);
        }
        bulk_wait_all();
    } else {
        // -------------------------------------------------------- softmax sets + output
        const int set = (warp - 2) >> 3;         // set 0 takes the stream's even key tiles, set 1 the odd ones
        const int half = ((warp - 2) >> 2) & 1;  // which 64 score / output columns of the row
        const int qd = warp & 3;                 // TMEM lane quadrant this warp may access
        const int row = qd * 32 + lane;          // row within the query tile
        const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
        const uint32_t t_o = tmem_O + half * 64 + lane_off;
        // The max of a row's scores in a tile, half a row by each of its two threads, in shared memory.
        // EXACT, [set][half][row]: the two threads read both halves, and so do those of the other set, which follow this set's decision
        // by the same arithmetic.  All eight warps of a set arrive on m_pub once they have read; a set writes again after the other's
        // arrival for the tile in between, which comes after its own for the tile before, so an entry is not overwritten
        // before all four threads have it.
        // Else [set][use parity][half][row] in bf16, beside it [tile parity][row] the max in force after a tile (every stored P, partial
        // sum and O is relative to it) as the unscaled score it came from.  Both threads of a row read the previous tile's
        // entry and one writes this tile's, so the two lie in different places, and all eight warps of a set
        // arrive on m_pub: an entry is not overwritten before it is read.
        // Each set waits for every tile of the other one, a unit's last one included, so this holds from unit to unit.
        float *x_mine = xch + set * 256 + half * 128 + row, *x_half = xch + set * 256 + (half ^ 1) * 128 + row;
        const float* x_set = xch + (set ^ 1) * 256 + row;
        uint16_t* x16 = reinterpret_cast<uint16_t*>(xch) + set * 512 + row;
        uint16_t* m_sh = reinterpret_cast<uint16_t*>(xch + T1_XCH / 4);
        const int bar_id = 1 + set;              // named barrier of the set's 256 threads
        constexpr int BAR_THREADS = 256;
        const float scale_log2 = par.a[0].scale_log2;      // (of all sequences)
        bool ok = true;
        int g = 0;                               // the unit's first tile in the stream
        for (int index = 0;; ++index) {
        const AttnUnit* unit = units + index % T1_UNITS;
        {
            // the set goes on to a unit, or stops, as one
            uint32_t got = mbar_wait(&u_full[index % T1_UNITS], (index / T1_UNITS) & 1);
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %0, 0;\n\tbarrier.cta.red.and.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "+r"(got) : "r"(bar_id), "n"(BAR_THREADS) : "memory");
            if (!got) { atomicExch(err, 24); break; }
        }
        const int g_end = g + unit->n;
        if (g_end == g) break;
        // last key this row sees, counted from the unit's first key tile
        int k_last;
        {
            const AttnArgs& a = par.a[NSEG > 1 ? unit->seg : 0];
            const int row_g = unit->q0 + row;
            k_last = (row_g < a.ar_len && row_g < a.S ? row_g : a.S - 1) - unit->j0 * AKV;
        }
        float m_mine = -INFINITY;                // max this thread's partial sum is relative to
        uint32_t m_raw = 0xff800000u;            // (not EXACT) the score it came from
        float l = 0.f;                           // this thread's share of the row sum
        // the max in force after the other set's tile gj: the sum follows where that set raised it
        auto follow = [&](int gj) {
            float m_tile;
            bool raised;
            if constexpr (EXACT) {
                m_tile = fmaxf(x_set[0], x_set[128]) * scale_log2;
                raised = (m_tile - m_mine) > 8.0f;
            } else {
                const uint32_t raw = (uint32_t)m_sh[(gj & 1) * T1_ROWS + row] << 16;
                m_tile = __uint_as_float(raw) * scale_log2;
                raised = raw != m_raw;
                m_raw = raw;
            }
            if (raised) {
                l *= ex2_approx(m_mine - m_tile);     // m_mine == -inf: l is 0 and stays 0
                m_mine = m_tile;
            }
        };
        for (int gj = g + ((g ^ set) & 1); gj < g_end; gj += 2) {
            const int b = gj % T1_S_BUFS;
            const int use = (gj >> 1) & 1;
            const uint32_t t_s = tmem_S + b * 128 + lane_off;
            // A thread whose wait ran out keeps taking part in the set's named barrier (one per tile) and does
            // nothing else, so that no partner is left waiting at a barrier that has no time limit.
            uint32_t r[2][32];
            float mx = -INFINITY;
            if (ok && !mbar_wait_warp(&s_full[b], (gj / T1_S_BUFS) & 1)) { atomicExch(err, 17); ok = false; }
            if (ok) {
            tc_fence_after();
            // this thread's 64 fp32 scores go to registers with one wait
            tmem_ld32(t_s + half * 64, r[0]);
            tmem_ld32(t_s + half * 64 + 32, r[1]);
            tmem_ld_wait();
            const int seen = k_last + 1 - ((gj - g) * AKV + half * 64);      // how many of the 64 keys the row sees
            if (__any_sync(0xffffffffu, seen < 64)) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (c * 32 + i >= seen) r[c][i] = 0xff800000u;   // -inf
            }
            {
                // three-input max: 64 scores in 32 instructions, four independent chains
                float mxa = -INFINITY, mxb = -INFINITY, mxc = -INFINITY, mxd = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    mxa = max3(mxa, __uint_as_float(r[0][2 * i]), __uint_as_float(r[0][2 * i + 1]));
                    mxb = max3(mxb, __uint_as_float(r[0][16 + 2 * i]), __uint_as_float(r[0][16 + 2 * i + 1]));
                    mxc = max3(mxc, __uint_as_float(r[1][2 * i]), __uint_as_float(r[1][2 * i + 1]));
                    mxd = max3(mxd, __uint_as_float(r[1][16 + 2 * i]), __uint_as_float(r[1][16 + 2 * i + 1]));
                }
                mx = max3(mxa, mxb, fmaxf(mxc, mxd));
            }
            // Row max over both halves: the partner thread's value comes through shared memory.
            if constexpr (EXACT) {
                if (gj > g && !mbar_wait_warp(&m_pub[set ^ 1], ((gj - 1) >> 1) & 1)) { atomicExch(err, 18); ok = false; }
                if (ok) *x_mine = mx;
            } else {
                // The reference value only has to be the same for both threads and not below the true max, so it travels as a
                // bf16 rounded toward +inf (+inf / NaN cannot occur in a score).  A slot is rewritten two uses later, after a
                // barrier the partner only reaches once it has read this use's value.
                const uint32_t mb = __float_as_uint(mx);
                mx = __uint_as_float(((int32_t)mb >= 0 ? mb + 0xffffu : mb) & 0xffff0000u);
                x16[use * 256 + half * 128] = (uint16_t)(__float_as_uint(mx) >> 16);
            }
            }
            asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(BAR_THREADS) : "memory");
            if (!ok) continue;
            mx = fmaxf(mx, EXACT ? *x_half : __uint_as_float((uint32_t)x16[use * 256 + (half ^ 1) * 128] << 16));
            const float m_tile = mx * scale_log2;
            // the max in force after the previous tile, which the other set decided
            if (gj > g) {
                if (!EXACT && !mbar_wait_warp(&m_pub[set ^ 1], ((gj - 1) >> 1) & 1)) { atomicExch(err, 18); ok = false; continue; }
                follow(gj - 1);
            }
            const bool grow = (m_tile - m_mine) > 8.0f;      // also true while m_mine == -inf
            float alpha = 1.0f;
            if (grow) {
                alpha = ex2_approx(m_mine - m_tile);         // 0 on the first tile
                m_mine = m_tile;
                m_raw = __float_as_uint(mx);
                l *= alpha;
            }
            if (!EXACT && half == 0) m_sh[(gj & 1) * T1_ROWS + row] = (uint16_t)(m_raw >> 16);
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_pub[set]);
            if (gj > g && __any_sync(0xffffffffu, grow)) {
                // O must hold all of PV(gj-1) and nothing of PV(gj): the first is what v_empty of tile gj-1 reports,
                // the second waits for this set's p_ready.  Each thread scales its own 64 output columns.
                if (!mbar_wait_warp(&v_empty[(gj - 1) % T1_V_STAGES], ((gj - 1) / T1_V_STAGES) & 1)) { atomicExch(err, 21); ok = false; continue; }
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < 4 && half * 64 + c * 16 < DN; ++c) {
                    uint32_t o[16];
                    tmem_ld16(t_o + c * 16, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_st16(t_o + c * 16, o);
                }
                tmem_st_wait();
            }
            // P = exp2(s * scale_log2 - m) as packed bf16 pairs, written over the score columns (this half's 64
            // scores are in registers by now, and the partner only writes after the barrier above, i.e. after
            // both loads): 64 scores become 32 columns at [half*32, +32).  A causal row may have no visible key
            // in this tile and none before: m is still -inf then and every score is masked; 0 keeps
            // exp2(-inf + 0) = 0 instead of exp2(-inf + inf)
            const float neg_m = (m_mine == -INFINITY) ? 0.f : -m_mine;
            const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2), negm2 = pack_f32x2(neg_m, neg_m);
            l += softmax_exp_store(r, scale2, negm2, t_s + half * 32);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        const int gl = g_end - 1;                // the unit's last tile
        const bool mine = (gl & 1) == set;       // the set that took it stores the unit's rows
        g = g_end;
        // ---- the sums of the other set follow its max
        if (ok && !mine) {
            if (!mbar_wait_warp(&m_pub[set ^ 1], (gl >> 1) & 1)) { atomicExch(err, 18); ok = false; }
            if (ok) follow(gl);
        }
        if (!ok) continue;
        // The row sum is the four threads' shares together.  They meet in the unit's Q tile, which no MMA reads any more (the scores
        // of the last tile are there), in the 4 KB that each storing warp has for its rows: [set, half][lane], behind l_full.
        // The shares of unit i and of unit i + 2 go through the same barrier: before a warp comes to the second it has seen the
        // other set decide on a tile behind the first.
        uint8_t* slices = q_s + (index & 1) * TILE_BYTES + qd * 4096;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
            *reinterpret_cast<float*>(slices + hh * 4 * 4096 + (set * 2 + half) * 128 + lane * 4) = l;
        __syncwarp();
        if (lane == 0) mbar_arrive(&l_full[index & 1]);
        if (!mine) continue;
        // ---- output: O / l -> bf16 -> out[row, h*128 + half*64 ..]
        const int failed = error_word(err);
        // (v_empty of the last tile: its PV is done)
        if (!mbar_wait_warp(&l_full[index & 1], (index >> 1) & 1) ||
            !mbar_wait_warp(&v_empty[gl % T1_V_STAGES], (gl / T1_V_STAGES) & 1)) { atomicExch(err, 19); ok = false; continue; }
        tc_fence_after();
        const int slot = unit->slot;
        const AttnArgs& a = par.a[NSEG > 1 ? unit->seg : 0];
        const size_t prow = (size_t)slot * T1_ROWS + qd * 32;
        attn_stage_rows(slices + half * 4 * 4096, tmem_O + half * 64 + lane_off, o_free, &o_staged[index & 1], m_mine,
                        slot >= 0 && !failed ? a.part_o + prow * AD + half * 64 : nullptr,
                        slot >= 0 && !failed && half == 0 ? a.part_ml + prow * 2 : nullptr, slot < 0);
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// Combines the partial results of the tail items: out = sum_i O_i 2^(m_i - M) / sum_i l_i 2^(m_i - M).
// One block per query row, one thread per output column.
__global__ void __launch_bounds__(AD) attn_merge_kernel(const AttnArgs a, int n_tail, int AQ2 /* rows per item */) {
    grid_dep_launch();
    grid_dep_wait();
    const int ti = blockIdx.x / AQ2, r = blockIdx.x - ti * AQ2;
    if (ti >= n_tail) return;
    const int item = a.n_plain + ti;
    const int h = item / a.nqb;
    const int row_g = (item - h * a.nqb) * AQ2 + r;
    if (row_g >= a.S) return;
    const int col = threadIdx.x;
    float M = -INFINITY;
    for (int i = 0; i < a.ways; ++i) M = fmaxf(M, a.part_ml[((size_t)(ti * a.ways + i) * AQ2 + r) * 2]);
    float num = 0.f, den = 0.f;
    for (int i = 0; i < a.ways; ++i) {
        const size_t pr = (size_t)(ti * a.ways + i) * AQ2 + r;
        const float m = a.part_ml[pr * 2];
        if (m == -INFINITY) continue;           // this key range held no visible key for the row
        const float wgt = exp2f(m - M);
        num = fmaf(a.part_o[pr * AD + col], wgt, num);
        den = fmaf(a.part_ml[pr * 2 + 1], wgt, den);
    }
    const float v = num * (1.0f / den);
    uint16_t* dst = a.out + (size_t)row_g * a.ldo + (size_t)h * a.out_hoff;
    if (a.out_rows > 0) {
        const int blk = row_g / a.out_rows;
        dst = a.out_tab[blk] + (size_t)(row_g - blk * a.out_rows) * a.ldo + (size_t)h * a.out_hoff;
    }
    dst[col] = f32_to_bf16(v);
}

// Number of key-range parts for the tail items: the last (total % SMs) items would otherwise be a round of their own.  Cost of the tail in
// item durations: rounds it needs, ceil(rem * w / SMs), times the duration of a part, 1/w plus a fixed share, which the rule
// takes as twelve key tiles' worth for 128-row items.  That share was measured with a CTA for each item (its set-up, copies, drain and the
// merge launch); as units of a stream the parts have less of it, and the rule is right more often than it thinks.  After full rounds the
// SMs have drifted apart and a tail of a few items costs next to nothing: split from a fifth of a round on, or after one round at
// most.  Unsplit / split, units in a stream, us: 4 heads 10496 rows (32 tail items after two rounds) 193 / 171, 16640 rows (76 after three)
// 476 / 462, 8 heads 8192 rows (68 after three) 248 / 236, 12356 rows (36 after five) 555 / 504, 16 heads 12356 rows (72 after
// ten) 1027 / 999; left alone: 8 heads 16640 rows (4 after seven) 990, 16 heads 8192 rows (136 after six) 426.
// Below T1_EXACT_ROWS rows the share is four key tiles, as measured with the two-tile kernel's 256-row items (which keep it),
// and the tail a quarter of a round: like the max there, the choice decides the bits of a forward, so it stays although most tails are better left
// whole now: 4 heads 5500 rows (24 after one) 71.9 / 60.7 us, but 16 heads 1280 rows (12 after one) 22.3 / 24.6, 8 heads 6000 rows (80 after
// two) 143 / 156, 32 heads 3157 rows (60 after five) 132 / 137, 8000 rows (92 after thirteen) 823 / 831.
// Every part keeps at least two key tiles.
static int g_tail_ways = 0;   // 0: choose; 1: never split; n > 1: n parts whenever they fit
void attention_tail_ways(int ways) { g_tail_ways = ways < 0 ? 0 : ways; }
// Which kernel: 0 and 2 = one query tile per CTA, 1 = two.  One is the better form at every length since its issuing threads are
// elected.  Two / one in turn in one process, us: 32 / 8 heads 8192 rows 1077 / 892, 10496 rows 1737 / 1471, 12356 rows 2538 / 2017,
// 16640 rows 4402 / 3476, all rows causal 2301 / 1927; a rank of a sharded forward, whose output leaves through the table (here into
// this GPU's memory), 8192 / 16640 rows: 16 / 4 heads 574 / 426 and 2310 / 1763, 8 / 2 heads 330 / 229 and 1032 / 819, 4 / 1 heads
// 195 / 117 and 676 / 465.  (The row segments it stores there are of 64 bytes where the two-tile kernel's are of 128: a rank
// of eight stores 15 MB in those 465 us, 4 % of what a link carries.)
static int g_tile_mode = -1;    // -1: not yet read from the environment (O1_ATTN_TILE_MODE)
void attention_tile_mode(int mode) { g_tile_mode = (mode < 0 || mode > 2) ? 0 : mode; }
static int tile_mode() {
    if (g_tile_mode < 0) {
        const char* e = getenv("O1_ATTN_TILE_MODE");
        g_tile_mode = (e && (e[0] == '1' || e[0] == '2')) ? e[0] - '0' : 0;
    }
    return g_tile_mode;
}
bool attention_two_tile_only() { return tile_mode() == 1; }

static int choose_tail_ways(int total, int nsm, int min_tiles, size_t scratch_bytes, int rows_item, int S) {
    const int rem = total % nsm;
    if (rem == 0) return 1;
    const size_t part_bytes = (size_t)rows_item * AD * 4 + (size_t)rows_item * 2 * 4;
    if (g_tail_ways >= 1) {
        const bool fits = g_tail_ways * 2 <= min_tiles && (size_t)rem * g_tail_ways * part_bytes <= scratch_bytes;
        return fits ? g_tail_ways : 1;
    }
    const bool long_one = rows_item == T1_ROWS && S >= T1_EXACT_ROWS;
    const double fixed = (long_one ? 12.0 : 4.0) / min_tiles;
    int best = 1;
    double best_cost = 1.0;
    for (int w = 2; w <= 32 && w * 2 <= min_tiles; ++w) {
        if ((size_t)rem * w * part_bytes > scratch_bytes) break;
        const double cost = (double)((rem * w + nsm - 1) / nsm) * (1.0 / w + fixed) + 0.02;
        if (cost < best_cost - 1e-9) { best_cost = cost; best = w; }
    }
    const bool worth = rem * (long_one ? 5 : 4) >= nsm || total / nsm <= 1;
    return (worth && best_cost < 0.9) ? best : 1;
}

// The one-tile kernel's work units: those of the plain items, sorted by how many keys they see, and `parts` of the tail items.
static void set_units(AttnArgs& a, int parts) {
    int nc = a.ar_len / T1_ROWS - a.qb0;       // query blocks whose rows are all causal
    nc = nc < 0 ? 0 : (nc > a.nqb ? a.nqb : nc);
    a.nc = nc;
    a.hf = a.nqb ? a.n_plain / a.nqb : 0;
    a.hr = a.n_plain - a.hf * a.nqb;
    a.n_full = a.hf * (a.nqb - nc) + (a.hr > nc ? a.hr - nc : 0);
    a.by_full.set(a.nqb - nc > 0 ? a.nqb - nc : 1);
    a.by_nqb.set(a.nqb > 0 ? a.nqb : 1);
    a.by_ways.set(a.ways);
    a.by_hf.set(a.hf > 0 ? a.hf : 1);
    a.by_hf1.set(a.hf + 1);
    a.by_group.set(a.heads / a.kv_heads);
    a.n_long = a.n_full + parts;
    a.n_short = a.n_plain - a.n_full;
}

// One sequence, ready to launch.
struct AttnSetup {
    CUtensorMap q, k, v, o;
    AttnArgs a;
    int grid, n_tail, rows_item;
    bool one_tile;
    double work;
};

static bool attention_setup(AttnSetup& s, const void* q, int ldq, const void* k, int ldk, const void* v,
                                 int ldv, void* out, int ldo, int S, int heads, int kv_heads,
                                 int ar_len, float scale, bool in_head_major, bool out_head_major,
                                 void* const* out_tab = nullptr, int out_rows = 0,
                                 void* scratch = nullptr, size_t scratch_bytes = 0, int row_lo = 0, int row_hi = -1) {
    if (out_tab) {
        if (out_rows <= 0 || (S + out_rows - 1) / out_rows > 8 || out_head_major) { set_error("attention: bad output table"); return false; }
        for (int i = 0; i < (S + out_rows - 1) / out_rows; ++i)
            if (!out_tab[i] || (((uintptr_t)out_tab[i]) & 15)) { set_error("attention: output table entry %d unusable", i); return false; }
        out = out_tab[0];
    }
    if (!q || !k || !v || !out || S <= 0 || heads <= 0 || kv_heads <= 0 || (heads % kv_heads) != 0) {
        set_error("attention: bad args");
        return false;
    }
    if ((ldo % 8) != 0 || (((uintptr_t)out) & 15)) { set_error("attention: output not 16-byte aligned"); return false; }
    if (ar_len < 0) ar_len = 0;
    if (ar_len > S) ar_len = S;
    bool maps_ok;
    if (in_head_major) {
        maps_ok = cached_tmap(&s.q, q, (uint64_t)heads * S, AD, AD, 128) &&
                  cached_tmap(&s.k, k, (uint64_t)kv_heads * S, AD, AD, 128) &&
                  cached_tmap(&s.v, v, (uint64_t)kv_heads * S, AD, AD, 128);
    } else {
        maps_ok = cached_tmap(&s.q, q, S, (uint64_t)heads * AD, ldq, 128) &&
                  cached_tmap(&s.k, k, S, (uint64_t)kv_heads * AD, ldk, 128) &&
                  cached_tmap(&s.v, v, S, (uint64_t)kv_heads * AD, ldv, 128);
    }
    if (!maps_ok) return false;
    const bool one_tile = tile_mode() != 1;
    const int rows_item = one_tile ? T1_ROWS : AQ2;
    AttnArgs& a = s.a;
    a.out = (uint16_t*)out; a.ldo = ldo;
    a.S = S; a.heads = heads; a.kv_heads = kv_heads; a.ar_len = ar_len;
    a.row_lo = row_lo < 0 ? 0 : row_lo;
    a.row_hi = (row_hi < 0 || row_hi > S) ? S : row_hi;
    if (a.row_lo != 0 || a.row_hi != S) { scratch = nullptr; scratch_bytes = 0; }   // a row range never splits its tail items
    a.scale_log2 = scale * 1.4426950408889634f;
    a.q_hc = in_head_major ? 0 : AD;  a.q_hr = in_head_major ? S : 0;
    a.kv_hc = a.q_hc;                 a.kv_hr = a.q_hr;
    a.out_hoff = out_head_major ? (long)S * AD : AD;
    if (out_head_major) a.ldo = AD;
    a.err = device_error_word();
    a.out_rows = out_tab ? out_rows : 0;
    for (int i = 0; i < 8; ++i) a.out_tab[i] = nullptr;
    if (out_tab) for (int i = 0; i < (S + out_rows - 1) / out_rows; ++i) a.out_tab[i] = (uint16_t*)out_tab[i];
    a.nqb = (S + rows_item - 1) / rows_item;
    a.qb0 = 0;
    if (one_tile) {       // (the two-tile kernel leaves query blocks out on the device)
        a.qb0 = a.row_lo / rows_item;
        a.nqb = (a.row_hi + rows_item - 1) / rows_item - a.qb0;
        if (a.row_hi <= a.row_lo) a.nqb = 0;
    }
    const int total = a.nqb * heads;
    a.n_plain = total; a.ways = 1; a.part_o = nullptr; a.part_ml = nullptr;
    int n_tail = 0;
    if (scratch && scratch_bytes && (((uintptr_t)scratch) & 15) == 0) {
        const int nsm = sm_count();
        const int rem = total % nsm;
        // fewest key tiles among the tail items (all-causal query blocks stop at the diagonal)
        int min_tiles = 1 << 30;
        for (int it = total - rem; it < total; ++it) {
            const int q0 = (it % a.nqb) * rows_item;
            int kv_end = (q0 + rows_item - 1 < ar_len) ? q0 + rows_item : S;
            if (kv_end > S) kv_end = S;
            const int t = (kv_end + AKV - 1) / AKV;
            // (items of a few key tiles, the fully causal first query tiles, are short anyway: they do not limit
            // the number of parts, and parts of theirs that get no key tile leave an empty partial)
            if (t >= 4 && t < min_tiles) min_tiles = t;
        }
        const int w = (rem && min_tiles < (1 << 30)) ? choose_tail_ways(total, nsm, min_tiles, scratch_bytes, rows_item, S) : 1;
        if (w > 1) {
            n_tail = rem;
            a.n_plain = total - rem;
            a.ways = w;
            a.part_o = (float*)scratch;
            a.part_ml = a.part_o + (size_t)rem * w * rows_item * AD;
        }
    }
    a.out_copy = one_tile && !out_tab && a.row_lo == 0 && a.row_hi == S;
    if (a.out_copy && !cached_tmap_heads(&s.o, out, AD, S, heads, a.ldo, a.out_hoff, T1_ROWS)) return false;
    s.grid = a.n_plain + n_tail * a.ways;
    set_units(a, n_tail * a.ways);
    s.n_tail = n_tail; s.rows_item = rows_item; s.one_tile = one_tile;
    // QK^T + PV over the keys each row can see: 4*heads*128*(ar(ar+1)/2 + (S-ar)*S)
    s.work = 4.0 * heads * 128.0 * (0.5 * ar_len * (ar_len + 1.0) + (double)(S - ar_len) * S);
    return true;
}

// (a failed attribute call has left its own text)
static bool launched(cudaError_t e) {
    if (e != cudaSuccess) set_error("attention: launch: %s", cudaGetErrorString(e));
    return e == cudaSuccess;
}
template <int NSEG, bool EXACT>
static bool launch_one_tile(const AttnSetup* s, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    auto kern = flash_attn1_kernel<AD, NSEG, EXACT>;
    if (!func_attr_once(attr_done, (const void*)kern, T1_SMEM, "attention (one tile)")) return false;
    Attn1Params<NSEG> p;
    int grid = 0;
    for (int i = 0; i < NSEG; ++i) {
        p.q[i] = s[i].q; p.k[i] = s[i].k; p.v[i] = s[i].v; p.o[i] = s[i].o; p.a[i] = s[i].a;
        grid += s[i].grid;
    }
    if (grid == 0) return true;       // an empty range of rows
    if (grid > sm_count()) grid = sm_count();
    return launched(launch_chained(kern, dim3(grid), dim3(T1_THREADS), T1_SMEM, st, 1, p.a[0].S, p));
}
static bool launch_two_tile(const AttnSetup& s, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    if (!func_attr_once(attr_done, (const void*)flash_attn_kernel, ATTN_SMEM, "attention")) return false;
    return launched(launch_chained(flash_attn_kernel, dim3(s.grid), dim3(ATTN_THREADS), ATTN_SMEM, st, 1, s.a.S, s.q, s.k, s.v, s.a));
}
// s[0 .. n): one launch for all of them where all take the one-tile kernel of short sequences
static bool attention_launch(const AttnSetup* s, int n, cudaStream_t st) {
    double work = 0;
    for (int i = 0; i < n; ++i) work += s[i].work;
    prof_before(PROF_ATTN, work, st);
    bool ok = true;
    auto exact = [&](int i) { return s[i].a.S >= T1_EXACT_ROWS; };
    if (n == 2 && s[0].one_tile && s[1].one_tile && !exact(0) && !exact(1)) ok = launch_one_tile<2, false>(s, st);
    else
        for (int i = 0; i < n && ok; ++i)
            ok = !s[i].one_tile ? launch_two_tile(s[i], st) : exact(i) ? launch_one_tile<1, true>(s + i, st) : launch_one_tile<1, false>(s + i, st);
    for (int i = 0; i < n && ok; ++i)
        if (s[i].n_tail)
            ok = launched(launch_chained(attn_merge_kernel, dim3(s[i].n_tail * s[i].rows_item), dim3(AD), 0, st, 1, s[i].a.S, s[i].a,
                                         s[i].n_tail, s[i].rows_item));
    prof_after(st);
    return ok && launched(cudaGetLastError());
}

bool flash_attention_vision(const void* qkv, void* out, int S, float scale, cudaStream_t st) {
    constexpr int H = 16, DH = 72, LD = 3 * H * AD;
    if (!qkv || !out || S <= 0 || (((uintptr_t)out) & 15)) { set_error("attention (vision): bad args"); return false; }
    const uint16_t* q = (const uint16_t*)qkv;
    Attn1Params<1> p = {};
    if (!cached_tmap(&p.q[0], q, S, H * AD, LD, 128) || !cached_tmap(&p.k[0], q + H * AD, S, H * AD, LD, 128) ||
        !cached_tmap(&p.v[0], q + 2 * H * AD, S, H * AD, LD, 128))
        return false;
    static std::atomic<uint64_t> attr_done{0};
    auto kern = flash_attn1_kernel<DH, 1, false>;
    if (!func_attr_once(attr_done, (const void*)kern, T1_SMEM, "attention (vision)")) return false;
    AttnArgs& a = p.a[0];
    a.out = (uint16_t*)out; a.ldo = H * DH; a.out_hoff = DH;
    a.S = S; a.heads = a.kv_heads = H;
    a.row_hi = S;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.q_hc = a.kv_hc = AD;
    a.err = device_error_word();
    a.nqb = (S + T1_ROWS - 1) / T1_ROWS;
    a.n_plain = a.nqb * H; a.ways = 1;
    a.out_copy = 1;
    if (!cached_tmap_heads(&p.o[0], out, DH, S, H, a.ldo, DH, T1_ROWS)) return false;
    set_units(a, 0);
    const int grid = a.n_plain < sm_count() ? a.n_plain : sm_count();
    prof_before(PROF_ATTN, 4.0 * H * DH * (double)S * S, st);
    cudaError_t e = launch_chained(kern, dim3(grid), dim3(T1_THREADS), T1_SMEM, st, 1, p.a[0].S, p);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("attention (vision): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}
bool flash_attention(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv,
                     void* out, int ldo, int S, int heads, int kv_heads, int ar_len, float scale,
                     cudaStream_t st, void* scratch, size_t scratch_bytes) {
    AttnSetup s;
    return attention_setup(s, q, ldq, k, ldk, v, ldv, out, ldo, S, heads, kv_heads, ar_len, scale, false, false, nullptr, 0,
                           scratch, scratch_bytes) &&
           attention_launch(&s, 1, st);
}
// n sequences (1 or 2) whose rows lie behind one another in qkv [rows, q | k | v], out [rows, ldo] and scratch (scratch_row
// bytes per row); each attends to its own rows only, with the results of a call of its own
bool flash_attention_rows(const uint16_t* qkv, int ld, void* out, int ldo, const int* rows, const int* ar_len, int n, int heads,
                          int kv_heads, float scale, cudaStream_t st, void* scratch, size_t scratch_row) {
    if (n < 1 || n > 2) { set_error("attention: one or two sequences"); return false; }
    AttnSetup s[2];
    size_t row0 = 0;
    for (int i = 0; i < n; ++i) {
        const uint16_t* q = qkv + row0 * ld;
        if (!attention_setup(s[i], q, ld, q + heads * AD, ld, q + (heads + kv_heads) * AD, ld, (uint16_t*)out + row0 * ldo, ldo,
                             rows[i], heads, kv_heads, ar_len[i], scale, false, false, nullptr, 0,
                             (uint8_t*)scratch + row0 * scratch_row, rows[i] * scratch_row))
            return false;
        row0 += rows[i];
    }
    return attention_launch(s, n, st);
}
bool flash_attention_tab(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv,
                         void* const* out_tab, int out_rows, int ldo, int S, int heads, int kv_heads,
                         int ar_len, float scale, cudaStream_t st, void* scratch, size_t scratch_bytes) {
    AttnSetup s;
    return attention_setup(s, q, ldq, k, ldk, v, ldv, nullptr, ldo, S, heads, kv_heads, ar_len, scale, false, false, out_tab,
                           out_rows, scratch, scratch_bytes) &&
           attention_launch(&s, 1, st);
}
// q [heads,S,128], k/v [kv_heads,S,128]; out head-major [heads,S,128] or seq-major [S, heads*128]
bool flash_attention_hm(const void* q, const void* k, const void* v, void* out, int S, int heads,
                        int kv_heads, int ar_len, float scale, bool out_head_major, cudaStream_t st,
                        int row_lo, int row_hi) {
    AttnSetup s;
    return attention_setup(s, q, AD, k, AD, v, AD, out, heads * AD, S, heads, kv_heads, ar_len, scale, true, out_head_major,
                           nullptr, 0, nullptr, 0, row_lo, row_hi) &&
           attention_launch(&s, 1, st);
}

}  // namespace o1
