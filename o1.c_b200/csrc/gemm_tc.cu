// Dense linear layer  Y[M,N] = X[M,K] * W[N,K]^T  (bf16 in, fp32 accumulate,
// bf16 out) on the sm_100a tensor cores.  Replaces the cuBLASLt path of
// o1.c's hd_linear (src/cuda/gemm.cu:413-461, 506-525).
//
// Structure: persistent CTAs (one per SM), 128 x BN x 64 tiles.
//   warp 0      : TMA producer  (global -> 128B-swizzled shared, 4-6 stages)
//   warp 1      : tcgen05.mma issuer, accumulators in TMEM, double buffered
//   warps 2..9  : epilogue (tcgen05.ld -> registers -> fused op -> shared memory -> global)
// The epilogue of tile i overlaps the main loop of tile i+1.
//
// Fused epilogues keep the reference's bf16 rounding points:
//   BIAS   : bf16(bf16(acc) + bias)            (gemm.cu:226-236 second pass)
//   RESID  : bf16(bf16(acc) + resid)           (residual.cu:14-23)
//   SWIGLU : B tile = 128 gate rows + 128 up rows of the same columns;
//            bf16(bf16(silu(bf16 g)) * bf16 u) (act.cu:22-34)
//   LORA   : W = bf16(f32(W) + scale*acc)      (lora_merge.cu:26-33), for callers of o1_gemm; hd_lora_merge_gpu has a
//            kernel of its own (lora.cu)
#include <cstdlib>
#include "common.cuh"
#include "ptx.cuh"
#include "kernels.h"

#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

namespace o1 {

static constexpr int BM = 128;
static constexpr int BK = 64;
static constexpr int EPI_WARPS = 8;                       // two per quadrant of tensor memory
static constexpr int EPI_SLICE = 2048 + 64;               // shared memory of a warp: 32 rows x 32 columns, and their bias
static constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
static constexpr int SK_THREADS = 192;                    // narrow tiles: four epilogue warps
static constexpr int PAIR_ALONE = 116 * 1024;             // least shared memory of a CTA of a pair: more than half of an SM's 228 KB, see pair_capacity()

struct GemmArgs {
    int M, N, K;
    uint16_t* out;
    int ldo;
    const uint16_t* bias;
    const uint16_t* resid;
    int ldr;
    const float* rope;     // EPI_QKNORM: cos|sin table [M,128] fp32; EPI_VROPE: cos [M,72]
    const float* rope_sin; // EPI_VROPE: sin [M,72]
    float scale;
    int num_m, num_n, group_m;
    int halves_from;       // gate | up on pairs: the first tile that is taken as two halves
    int prefetch;          // K blocks of weights requested into L2 ahead of their load (0: none)
    // Output column blocks: column c lives at out + (c / o_cb) * o_cb_stride + row * ldo + c % o_cb
    // (o_cb == 0: plain row-major).  Lets a projection write its head groups into per-destination
    // slabs of an all-to-all send buffer.  o_cb must be a multiple of the tile width.
    int o_cb;
    long o_cb_stride;
    // With o_tab_n > 0 block b starts at o_tab[b] instead of out + b * o_cb_stride: the blocks may then
    // live in other GPUs' memory (peer-mapped), which turns the epilogue's stores into the transfer.
    int o_tab_n;
    uint16_t* o_tab[8];
    // Input K blocks: K columns [b*a_kblk, (b+1)*a_kblk) of row r live at x[(b*a_rows + r) * ldx + ...]
    // (a_kblk == 0: plain).  Lets a projection read the slabs an all-to-all received, one per source.
    int a_kblk, a_rows;
    // EPI_QKV: the output columns are three segments [q | k | v] with a weight tensor each (tensor maps B, B2, B3);
    // q and k tiles take the per-head norm + rotary epilogue (norm weights seg_norm[0], [1]), v tiles are stored as
    // they are.  seg_n = columns of q and of k (= v).  With output tables, segment s uses o_tab[8*s ...] and its own
    // block width seg_cb[s].
    int seg_n[2];
    const uint16_t* seg_norm[2];
    int seg_cb[3];
    uint16_t* seg_tab[16];    // tables of segments 1 and 2 (segment 0 uses o_tab)
    int* err;
};

// PAIR: two CTAs (a cluster) work on one 256 x BN tile with cta_group::2 MMAs; each holds its own 128 rows of A and
// of the accumulator and HALF of the B tile, so a stage is a third smaller and a B element is fetched into shared
// memory once per 256 output rows instead of once per 128.
template <int BN, bool PAIR = false>
struct GemmCfg {
    static constexpr int A_BYTES = BM * BK * 2;
    static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = PAIR ? 6 : ((BN == 256) ? 4 : 6);
    static constexpr int STORE_STAGE_BYTES = EPI_WARPS * 4096;   // epilogue staging, 4 KB per warp
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/ + STORE_STAGE_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;
};

__device__ __forceinline__ void tile_coords(int tile, int num_m, int num_n, int group_m, int& mb, int& nb) {
    const int per_group = group_m * num_n;
    const int grp = tile / per_group;
    const int r = tile - grp * per_group;
    const int m_first = grp * group_m;
    int gm = num_m - m_first;
    if (gm > group_m) gm = group_m;
    mb = m_first + r % gm;
    nb = r / gm;
}

// bf16-valued activations -> GELU, as o1.c's vision kernels compute it (src/cuda/vision_kernels.cu:100-133): the tanh
// form of the ViT block MLP or the erf form of the patch mergers, fp32 throughout, rounded by the caller.  One branch for
// all values: with one per value nothing overlaps (a 128 x 128 tile's epilogue took 9 us longer).
template <int N>
__device__ __forceinline__ void gelu_all(float (&v)[N], bool exact) {
    if (exact) {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = 0.5f * v[j] * (1.0f + erff(v[j] * 0.7071067811865476f));
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = gelu_tanh(v[j]);
    }
}
__device__ __forceinline__ void unpack8_bf16(const uint4& o, float* v) {
    v[0] = bf16lo(o.x); v[1] = bf16hi(o.x); v[2] = bf16lo(o.y); v[3] = bf16hi(o.y);
    v[4] = bf16lo(o.z); v[5] = bf16hi(o.z); v[6] = bf16lo(o.w); v[7] = bf16hi(o.w);
}

// ---- epilogues.  A warp holds 32 accumulator rows, one per thread.  What it loads and stores goes through its slice of shared
// memory, so that every access to global memory is of whole row segments of 64 bytes and more: with a thread storing its own row an
// instruction touches 32 lines, and that, four warps instead of eight and SwiGLU's branch per value (its division) made an epilogue
// of 11 us (SwiGLU), 15 (per-head norm) and 5 to 10 (the others) per 256-column tile.  The main loop of the next tile covers that, but
// not a CTA's last tile: q | k | v at 592 rows was 48 us for a round of 25.

// What an epilogue reads per column and per element.  In the others GemmArgs::bias is null (SwiGLU, LoRA) or the norm weight of one
// head (per-head norm), and must not be read by column.
static constexpr bool epi_has_bias(int e) { return e == EPI_BIAS || e == EPI_BIAS_GELU || e == EPI_BIAS_RESID || e == EPI_GATE_RESID; }
static constexpr bool epi_has_resid(int e) { return e == EPI_RESID || e == EPI_BIAS_RESID || e == EPI_GATE_RESID; }
static constexpr bool epi_plain(int e) { return e == EPI_STORE || epi_has_bias(e) || epi_has_resid(e); }

// Groups of 32 columns at c_first, c_first + c_step, ... of a tile, plain row-major output (or column blocks, see GemmArgs).
// LIMIT: rows from row_end on are another CTA's (row_end <= M).  PARTS: the sum lies in `parts` accumulators, part_cols columns apart.
template <int EPI, bool LIMIT = false, bool PARTS = false>
struct PlainEpilogue {
    static_assert(epi_plain(EPI), "this epilogue has no operands by column and element");
    static constexpr bool HAS_BIAS = epi_has_bias(EPI), HAS_RESID = epi_has_resid(EPI);
    // what the next group needs, requested one group ahead: the residual, eight rows of four 16-byte pieces at a time, and the bias
    // (or gate), a piece by each of four lanes
    uint4 rn[4] = {}, bq = {};
    int row_end = 0, parts = 1, part_cols = 0;
    // row0: first of the warp's rows; cols: columns of the tile that exist (a multiple of eight)
    __device__ __forceinline__ void ahead(const GemmArgs& g, int row0, int col0, int cols, int c, int lane) {
        if (HAS_BIAS && lane < 4 && c + lane * 8 < cols) bq = *reinterpret_cast<const uint4*>(g.bias + col0 + c + lane * 8);
        if (!HAS_RESID) return;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int row = row0 + k * 8 + (lane >> 2), col = c + (lane & 3) * 8;
            if (row < (LIMIT ? row_end : g.M) && col < cols) rn[k] = *reinterpret_cast<const uint4*>(g.resid + (size_t)row * g.ldr + col0 + col);
        }
    }
    // the caller has called ahead() for c_first; stg: EPI_SLICE bytes of the warp's own
    __device__ __forceinline__ void run(const GemmArgs& g, uint32_t t_row, int row0, int col0, int cols, int c_first, int c_step,
                                        uint8_t* stg, int lane, bool failed) {
        const int sr = lane >> 2, ch = lane & 3;
        uint4 *own = reinterpret_cast<uint4*>(stg + lane * 64), *bias_s = reinterpret_cast<uint4*>(stg + 2048);
#pragma unroll 1
        for (int c = c_first; c < cols; c += c_step) {
            uint32_t r[32];
            tmem_ld32(t_row + c, r);
            __syncwarp();
            if (HAS_RESID) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    *reinterpret_cast<uint4*>(stg + (k * 8 + sr) * 64 + ((ch ^ ((sr >> 1) & 3)) * 16)) = rn[k];
            }
            if (HAS_BIAS && lane < 4) bias_s[lane] = bq;
            if (HAS_RESID || HAS_BIAS) {
                ahead(g, row0, col0, cols, c + c_step, lane);
                __syncwarp();
            }
            tmem_ld_wait();
            if (PARTS) {
                // (from zero on, in the order of the parts)
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__fadd_rn(0.f, __uint_as_float(r[j])));
#pragma unroll 1
                for (int p = 1; p < parts; ++p) {
                    uint32_t r2[32];
                    tmem_ld32(t_row + p * part_cols + c, r2);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__fadd_rn(__uint_as_float(r[j]), __uint_as_float(r2[j])));
                }
            }
            float v[32];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float b[8] = {}, rs[8] = {};
                if (HAS_BIAS) unpack8_bf16(bias_s[i], b);
                if (HAS_RESID) unpack8_bf16(own[i ^ ((lane >> 1) & 3)], rs);
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    float x = __uint_as_float(r[i * 8 + j]), y = __uint_as_float(r[i * 8 + j + 1]);
                    if (EPI != EPI_STORE) bf16_round2(x, y);
                    if (EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESID) { x += b[j]; y += b[j + 1]; }
                    if (EPI == EPI_GATE_RESID) { x *= b[j]; y *= b[j + 1]; }
                    // linear + bias stored as bf16, then GELU or the residual add of src/cuda/residual.cu:14-23
                    if (EPI == EPI_BIAS_GELU || EPI == EPI_BIAS_RESID || EPI == EPI_GATE_RESID) bf16_round2(x, y);
                    if (HAS_RESID) { x += rs[j]; y += rs[j + 1]; }
                    v[i * 8 + j] = x; v[i * 8 + j + 1] = y;
                }
            }
            if (EPI == EPI_BIAS_GELU) gelu_all(v, g.scale != 0.f);
            store_group(g, v, stg, row0, col0 + c, cols - c, lane, failed, row_end);
        }
    }
    // this thread's row of 32 columns -> the warp's rows as segments of 64 bytes
    static __device__ __forceinline__ void store_group(const GemmArgs& g, const float (&v)[32], uint8_t* stg, int row0, int col, int cols,
                                                       int lane, bool failed, int row_end = 0) {
        const int sr = lane >> 2, ch = lane & 3;
        uint4* own = reinterpret_cast<uint4*>(stg + lane * 64);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* x = v + i * 8;
            own[i ^ ((lane >> 1) & 3)] = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]),
                                                    pack_bf16x2(x[6], x[7]));
        }
        __syncwarp();
        // (a group of 32 columns never straddles an output block)
        uint16_t* out = g.out + (g.o_cb ? (size_t)(col / g.o_cb) * g.o_cb_stride + col % g.o_cb : (size_t)col) + ch * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int row = row0 + k * 8 + sr;
            const uint4 o = *reinterpret_cast<const uint4*>(stg + (k * 8 + sr) * 64 + ((ch ^ ((sr >> 1) & 3)) * 16));
            if (!failed && row < (LIMIT ? row_end : g.M) && ch * 8 < cols) *reinterpret_cast<uint4*>(out + (size_t)row * g.ldo) = o;
        }
    }
};

// SwiGLU of 32 columns: bf16(silu(g)) * u with silu(g) = g * (1 / (1 + e^-g)).  The quotient is the IEEE one, by Markstein's step from
// the approximate reciprocal (P. Markstein, IBM J. Res. Dev. 34, 1990); the division itself, which branches for each value, is left
// to warps that hold a gate below -80, where 1 + e^-g comes near the largest number, or a NaN.
template <int N>       // v: gates, then results; u: what they multiply; all of them bf16 values, results to be rounded by the caller
__device__ __forceinline__ void swiglu_vals(float (&v)[N], const float (&u)[N]) {
    bool plain = true;
#pragma unroll
    for (int j = 0; j < N; j += 2) plain = plain && fminf(v[j], v[j + 1]) > -80.f && v[j] == v[j] && v[j + 1] == v[j + 1];
    if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            float s[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float x = 1.0f + expf(-v[j + i]);
                const float y = __fdividef(1.0f, x);
                s[i] = v[j + i] * __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
            }
            bf16_round2(s[0], s[1]);
            v[j] = s[0] * u[j]; v[j + 1] = s[1] * u[j + 1];
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float sg = 1.0f / (1.0f + expf(-v[j]));
            v[j] = bf16_round(v[j] * sg) * u[j];
        }
    }
}
__device__ __forceinline__ void swiglu_all(const uint32_t (&rg)[32], const uint32_t (&ru)[32], float (&v)[32]) {
    float u[32];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
        v[j] = __uint_as_float(rg[j]); v[j + 1] = __uint_as_float(rg[j + 1]);
        u[j] = __uint_as_float(ru[j]); u[j + 1] = __uint_as_float(ru[j + 1]);
        bf16_round2(v[j], v[j + 1]);
        bf16_round2(u[j], u[j + 1]);
    }
    swiglu_vals(v, u);
}

// (head_epilogue()'s arithmetic for one row, by eight lanes, in gemm_rows_kernel; as a function that one uses too it costs its launches
// 0.5 us.)  Each lane takes 8 + 8 of its bf16 values from shared memory, from column 8 t and 64 + 8 t on.
__device__ __forceinline__ void head_row(const GemmArgs& g, const uint8_t* s_lo, const uint8_t* s_hi, const float (&wl)[8], const float (&wh)[8],
                                         int row, bool row_ok, uint16_t* obase, int t) {
    const float* cs = g.rope + (size_t)(row_ok ? row : 0) * 128 + 8 * t;
    const float4 ca = *reinterpret_cast<const float4*>(cs), cb = *reinterpret_cast<const float4*>(cs + 4);
    const float4 sa = *reinterpret_cast<const float4*>(cs + 64), sb = *reinterpret_cast<const float4*>(cs + 68);
    float lo[8], hi[8];
    unpack8_bf16(*reinterpret_cast<const uint4*>(s_lo), lo);
    unpack8_bf16(*reinterpret_cast<const uint4*>(s_hi), hi);
    float sq = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) sq = __fadd_rn(sq, __fmaf_rn(hi[j], hi[j], __fmul_rn(lo[j], lo[j])));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, o));
    const float inv = rsqrtf(sq / 128.0f + g.scale);
    const float cc[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    const float ss[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
    float ol[8], oh[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float a = bf16_round(wl[j] * lo[j] * inv);
        const float b = bf16_round(wh[j] * hi[j] * inv);
        ol[j] = bf16_round(a * cc[j]) - bf16_round(b * ss[j]);
        oh[j] = bf16_round(b * cc[j]) + bf16_round(a * ss[j]);
    }
    if (row_ok) {
        uint16_t* o = obase + (size_t)row * g.ldo + 8 * t;
        *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16x2(ol[0], ol[1]), pack_bf16x2(ol[2], ol[3]), pack_bf16x2(ol[4], ol[5]), pack_bf16x2(ol[6], ol[7]));
        *reinterpret_cast<uint4*>(o + 64) = make_uint4(pack_bf16x2(oh[0], oh[1]), pack_bf16x2(oh[2], oh[3]), pack_bf16x2(oh[4], oh[5]), pack_bf16x2(oh[6], oh[7]));
    }
}
// Per-head RMSNorm + rotary on a projection's output (o1.c src/model/block.c:266-289 runs head split, hd_rmsnorm, hd_apply_rotary as
// separate passes).  The 128 values of a head are rounded to bf16 (the projection's stored result) and pass through shared memory, 16
// rows at a time; then eight lanes take a row: each sums 8 + 8 elements, the pairwise tree over the lanes is the order of
// qk_norm_rope_kernel, so that both paths agree bit for bit, and cos | sin and the result are whole lines.  half_lo .. half_hi: which
// of the warp's two groups of 16 rows; obase: the head's first column of row 0.
__device__ __forceinline__ void head_epilogue(const GemmArgs& g, uint32_t t_head, int row0, int rows, uint16_t* obase,
                                              const uint16_t* norm_w, int half_lo, int half_hi, uint8_t* stg, int lane) {
    const int t = lane & 7, sub = lane >> 3;
    float wl[8], wh[8];
    unpack8_bf16(*reinterpret_cast<const uint4*>(norm_w + 8 * t), wl);
    unpack8_bf16(*reinterpret_cast<const uint4*>(norm_w + 64 + 8 * t), wh);
#pragma unroll 1
    for (int hf = half_lo; hf < half_hi; ++hf) {
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(t_head + c * 32, r);
            tmem_ld_wait();
            if ((lane >> 4) == hf) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint4 o;
                    o.x = pack_bf16x2(__uint_as_float(r[8 * i]), __uint_as_float(r[8 * i + 1]));
                    o.y = pack_bf16x2(__uint_as_float(r[8 * i + 2]), __uint_as_float(r[8 * i + 3]));
                    o.z = pack_bf16x2(__uint_as_float(r[8 * i + 4]), __uint_as_float(r[8 * i + 5]));
                    o.w = pack_bf16x2(__uint_as_float(r[8 * i + 6]), __uint_as_float(r[8 * i + 7]));
                    *reinterpret_cast<uint4*>(stg + (lane & 15) * 256 + (((c * 4 + i) ^ (lane & 7)) * 16)) = o;
                }
            }
        }
        __syncwarp();
#pragma unroll 2
        for (int it = 0; it < 4; ++it) {
            const int rr = it * 4 + sub, row = row0 + hf * 16 + rr;
            const bool row_ok = row < rows;
            const float* cs = g.rope + (size_t)(row_ok ? row : 0) * 128 + 8 * t;
            const float4 ca = *reinterpret_cast<const float4*>(cs), cb = *reinterpret_cast<const float4*>(cs + 4);
            const float4 sa = *reinterpret_cast<const float4*>(cs + 64), sb = *reinterpret_cast<const float4*>(cs + 68);
            float lo[8], hi[8];
            unpack8_bf16(*reinterpret_cast<const uint4*>(stg + rr * 256 + ((t ^ (rr & 7)) * 16)), lo);
            unpack8_bf16(*reinterpret_cast<const uint4*>(stg + rr * 256 + (((8 + t) ^ (rr & 7)) * 16)), hi);
            float sq = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) sq = __fadd_rn(sq, __fmaf_rn(hi[j], hi[j], __fmul_rn(lo[j], lo[j])));
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) sq = __fadd_rn(sq, __shfl_xor_sync(0xffffffffu, sq, o));
            const float inv = rsqrtf(sq / 128.0f + g.scale);
            const float cc[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
            const float ss[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
            float ol[8], oh[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float a = bf16_round(wl[j] * lo[j] * inv);
                const float b = bf16_round(wh[j] * hi[j] * inv);
                ol[j] = bf16_round(a * cc[j]) - bf16_round(b * ss[j]);
                oh[j] = bf16_round(b * cc[j]) + bf16_round(a * ss[j]);
            }
            if (row_ok) {
                uint16_t* o = obase + (size_t)row * g.ldo + 8 * t;
                *reinterpret_cast<uint4*>(o) = make_uint4(pack_bf16x2(ol[0], ol[1]), pack_bf16x2(ol[2], ol[3]), pack_bf16x2(ol[4], ol[5]), pack_bf16x2(ol[6], ol[7]));
                *reinterpret_cast<uint4*>(o + 64) = make_uint4(pack_bf16x2(oh[0], oh[1]), pack_bf16x2(oh[2], oh[3]), pack_bf16x2(oh[4], oh[5]), pack_bf16x2(oh[6], oh[7]));
            }
        }
    }
}

template <int EPI, int BN, bool PAIR>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmB3, const __grid_constant__ CUtensorMap tmB4,
               const GemmArgs g) {
    using Cfg = GemmCfg<BN, PAIR>;
    // gate | up on pairs: the last tiles as halves of 64 columns of each (tmB3, tmB4: boxes of 64 rows), see launch_tc_pair()
    constexpr bool HALVES = PAIR && EPI == EPI_SWIGLU;
    static_assert(!PAIR || BN == 256, "the pair form splits a 256-wide B tile");
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* tfull = empty + STAGES;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    uint8_t* store_stage = smem + STAGES * Cfg::STAGE_BYTES + 256;

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    // (a pair decides together, after its cluster barrier; the word is on its way while barriers and tensor memory are set up)
    __shared__ int s_abort;
    if (threadIdx.x == 64) s_abort = error_word(g.err);
    const uint32_t rank = PAIR ? cluster_rank() : 0u;    // 0: the CTA that issues the pair's MMAs
    if (PAIR) cluster_arrive();

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (EPI == EPI_SWIGLU || EPI == EPI_QKV) tma_prefetch_desc(&tmB2);
        if (EPI == EPI_QKV) tma_prefetch_desc(&tmB3);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], PAIR ? 2 * EPI_WARPS : EPI_WARPS);    // the epilogue warps of both CTAs arrive on the first CTA's
        }
        fence_mbar_init();
    }
    if (PAIR) cluster_wait();
    if (warp == 1) {
        if (PAIR) tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
        else { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();           // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    if (PAIR && warp == 1) tmem_relinquish_pair();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    bool live = s_abort == 0;
    if (PAIR) live = (s_abort | ld_cluster_s32(map_to_rank(smem_u32(&s_abort), rank ^ 1u))) == 0;

    // the pair form walks tiles of 256 rows: row tile 2 * mb2 + rank of each belongs to this CTA
    const int sched_m = PAIR ? (g.num_m + 1) / 2 : g.num_m;
    const int sched_group = PAIR ? (g.group_m + 1) / 2 : g.group_m;
    // (HALVES: units from halves_from on are halves, two to a tile)
    const int halves_from = HALVES ? g.halves_from : 0;
    const int num_tiles = sched_m * g.num_n + (HALVES ? sched_m * g.num_n - halves_from : 0);
    const int tile0 = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int tile_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int kblocks = (g.K + BK - 1) / BK;   // a ragged last K block is zero-filled by TMA in both operands

    if (!live) {
        // nothing to do: straight to the common teardown
    } else if (warp == 0) {
        // ------------------------------------------------------ TMA producer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                int mb, nb;
                const bool is_half = HALVES && tile >= halves_from;
                tile_coords(is_half ? halves_from + ((tile - halves_from) >> 1) : tile, sched_m, g.num_n, sched_group, mb, nb);
                if (PAIR) mb = mb * 2 + (int)rank;
                const uint32_t pair_bytes = 2 * (is_half ? Cfg::STAGE_BYTES - 64 * BK * 2 : Cfg::STAGE_BYTES);      // both CTAs' halves
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1)) { ok = false; atomicExch(g.err, 1); break; }
                    uint8_t* a_s = smem + stage * Cfg::STAGE_BYTES;
                    uint8_t* b_s = a_s + Cfg::A_BYTES;
                    if (!PAIR) mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
                    else if (rank == 0) mbar_expect_tx(&full[stage], pair_bytes);
                    int a_c0 = kb * BK, a_c1 = mb * BM;
                    if (g.a_kblk > 0) {
                        const int blk = a_c0 / g.a_kblk;
                        a_c0 -= blk * g.a_kblk;
                        a_c1 += blk * g.a_rows;
                    }
                    if (PAIR) {
                        // this CTA's 128 rows of A and its 128 of the tile's 256 B rows (second half for the second CTA)
                        tma_load_2d_pair(a_s, &tmA, &full[stage], a_c0, a_c1);
                        if (is_half) {
                            tma_load_2d_pair(b_s, rank == 0 ? &tmB3 : &tmB4, &full[stage], kb * BK, nb * 128 + ((tile - halves_from) & 1) * 64);
                        } else if (EPI == EPI_SWIGLU) {
                            tma_load_2d_pair(b_s, rank == 0 ? &tmB : &tmB2, &full[stage], kb * BK, nb * 128);
                        } else if (EPI == EPI_QKV) {
                            const int col0 = nb * BN;
                            const int seg = col0 >= g.seg_n[0] + g.seg_n[1] ? 2 : (col0 >= g.seg_n[0] ? 1 : 0);
                            const int lrow = col0 - (seg == 2 ? g.seg_n[0] + g.seg_n[1] : (seg == 1 ? g.seg_n[0] : 0));
                            const CUtensorMap* mB = seg == 0 ? &tmB : (seg == 1 ? &tmB2 : &tmB3);
                            tma_load_2d_pair(b_s, mB, &full[stage], kb * BK, lrow + (int)rank * 128);
                        } else {
                            tma_load_2d_pair(b_s, &tmB, &full[stage], kb * BK, nb * BN + (int)rank * 128);
                        }
                        if (++stage == STAGES) { stage = 0; phase ^= 1; }
                        continue;
                    }
                    tma_load_2d(a_s, &tmA, &full[stage], a_c0, a_c1);
                    if (EPI == EPI_SWIGLU) {
                        // 128 gate rows then 128 up rows of the same output columns
                        tma_load_2d(b_s, &tmB, &full[stage], kb * BK, nb * 128);
                        tma_load_2d(b_s + 128 * BK * 2, &tmB2, &full[stage], kb * BK, nb * 128);
                    } else if (EPI == EPI_QKV) {
                        // the weight tensor of the segment this column tile lies in, at the segment's own row
                        const int col0 = nb * BN;
                        const int seg = col0 >= g.seg_n[0] + g.seg_n[1] ? 2 : (col0 >= g.seg_n[0] ? 1 : 0);
                        const int lrow = col0 - (seg == 2 ? g.seg_n[0] + g.seg_n[1] : (seg == 1 ? g.seg_n[0] : 0));
                        const CUtensorMap* mB = seg == 0 ? &tmB : (seg == 1 ? &tmB2 : &tmB3);
#pragma unroll
                        for (int h = 0; h < BN / 128; ++h)
                            tma_load_2d(b_s + h * 128 * BK * 2, mB, &full[stage], kb * BK, lrow + h * 128);
                    } else {
#pragma unroll
                        for (int h = 0; h < BN / 128; ++h)
                            tma_load_2d(b_s + h * 128 * BK * 2, &tmB, &full[stage], kb * BK,
                                        nb * BN + h * 128);
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc_full = umma_idesc_bf16(PAIR ? 2 * BM : BM, BN, 0, 0), idesc_half = umma_idesc_bf16(2 * BM, BN / 2, 0, 0);
            int stage = 0;
            uint32_t phase = 0;
            int as = 0;
            uint32_t aphase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                const uint32_t idesc = HALVES && tile >= halves_from ? idesc_half : idesc_full;
                if (!mbar_wait(&tempty[as], aphase ^ 1)) { atomicExch(g.err, 2); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * BN;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&full[stage], phase)) { ok = false; atomicExch(g.err, 3); break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + stage * Cfg::STAGE_BYTES);
                    const uint64_t ad = umma_desc_sw128(a_addr, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + Cfg::A_BYTES, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {  // 32 bytes per K step = 2 units of the address field
                        if (PAIR) umma_ss_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                        else umma_ss(d_tmem, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                    }
                    if (PAIR) umma_commit_pair(&empty[stage]);
                    else umma_commit(&empty[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (PAIR) umma_commit_pair(&tfull[as]);
                else umma_commit(&tfull[as]);
                if (++as == 2) { as = 0; aphase ^= 1; }
            }
        }
    } else {
        // ------------------------------------------------------ epilogue
        const int q = warp & 3;                  // TMEM lane quadrant this warp may access
        const int half = (warp - 2) >> 2;        // which of the quadrant's two warps
        uint8_t* stg = store_stage + (warp - 2) * 4096;
        int as = 0;
        uint32_t aphase = 0;
        const int failed = error_word(g.err);
        for (int tile = tile0; tile < num_tiles; tile += tile_step) {
            int mb, nb;
            const bool is_half = HALVES && tile >= halves_from;
            tile_coords(is_half ? halves_from + ((tile - halves_from) >> 1) : tile, sched_m, g.num_n, sched_group, mb, nb);
            if (PAIR) mb = mb * 2 + (int)rank;
            const int rows = failed ? 0 : g.M;
            const int row0 = mb * BM + q * 32;
            const int cols = g.N - nb * BN < BN ? g.N - nb * BN : BN;      // (plain epilogues: N may be ragged, N % 8 == 0)
            // (v of q | k | v is stored as it is; the other epilogues do not use this one)
            PlainEpilogue<epi_plain(EPI) ? EPI : (int)EPI_STORE> plain;
            plain.ahead(g, row0, nb * BN, cols, half * 32, lane);
            const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull[as], aphase));
            if (!got) { atomicExch(g.err, 4); break; }
            tc_fence_after();
            const uint32_t t_row = tmem_base + as * BN + ((uint32_t)(q * 32) << 16);
            // EPI_QKV: which segment this column tile lies in decides the epilogue (warp-uniform); everything
            // below addresses the output through (seg_col0 + column inside the segment) or the segment's tables
            int seg = 0, seg_col0 = 0, lcol0 = nb * BN, cb = g.o_cb;
            uint16_t* const* tab = g.o_tab;
            const uint16_t* norm_w = g.bias;
            if (EPI == EPI_QKV) {
                seg = lcol0 >= g.seg_n[0] + g.seg_n[1] ? 2 : (lcol0 >= g.seg_n[0] ? 1 : 0);
                seg_col0 = seg == 2 ? g.seg_n[0] + g.seg_n[1] : (seg == 1 ? g.seg_n[0] : 0);
                lcol0 -= seg_col0;
                cb = g.seg_cb[seg];
                if (seg > 0) tab = g.seg_tab + (seg - 1) * 8;
                norm_w = g.seg_norm[seg == 1 ? 1 : 0];
            }
            const int epi_eff = (EPI == EPI_QKV) ? (seg < 2 ? (int)EPI_QKNORM : (int)EPI_STORE) : EPI;
            if (EPI == EPI_SWIGLU) {
                const int width = is_half ? 64 : 128, col0 = nb * 128 + (is_half ? ((tile - halves_from) & 1) * 64 : 0);
#pragma unroll 1
                for (int c = half * 32; c < width; c += 64) {
                    uint32_t rg[32], ru[32];
                    tmem_ld32(t_row + c, rg);
                    tmem_ld32(t_row + width + c, ru);
                    tmem_ld_wait();
                    float v[32];
                    swiglu_all(rg, ru, v);
                    __syncwarp();
                    PlainEpilogue<EPI_STORE>::store_group(g, v, stg, row0, col0 + c, 32, lane, failed);
                }
            } else if (epi_eff == EPI_STORE && g.o_tab_n) {
                // Blocks of the output live in other GPUs' memory.  One thread per row would put 16-byte
                // pieces of 32 different rows into every store instruction; over NVLink each piece is a
                // packet of its own.  So 64 columns at a time go through the swizzled shared-memory slice of
                // this warp and leave as full 128-byte row segments (4 rows per instruction).
#pragma unroll 1
                for (int c2 = half; c2 < BN / 64; c2 += 2) {
                    uint32_t r0[32], r1[32];
                    tmem_ld32(t_row + c2 * 64, r0);
                    tmem_ld32(t_row + c2 * 64 + 32, r1);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t* src = j < 4 ? &r0[(j & 3) * 8] : &r1[(j & 3) * 8];
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(src[0]), __uint_as_float(src[1]));
                        o.y = pack_bf16x2(__uint_as_float(src[2]), __uint_as_float(src[3]));
                        o.z = pack_bf16x2(__uint_as_float(src[4]), __uint_as_float(src[5]));
                        o.w = pack_bf16x2(__uint_as_float(src[6]), __uint_as_float(src[7]));
                        *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) * 16)) = o;
                    }
                    __syncwarp();
                    const int col = lcol0 + c2 * 64;        // a 64-column group never straddles a block (cb % 128 == 0)
                    uint16_t* obase = tab[col / cb] + (col % cb);
                    const int ch = lane & 7;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int rr = k * 4 + (lane >> 3);
                        const uint4 o = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((ch ^ (rr & 7)) * 16));
                        if (row0 + rr < rows) *reinterpret_cast<uint4*>(obase + (size_t)(row0 + rr) * g.ldo + ch * 8) = o;
                    }
                    __syncwarp();
                }
            } else if (epi_eff == EPI_QKNORM) {
                // two heads: one for each of a quadrant's warps; one head: 16 rows each
                const int hb = BN == 256 ? half : 0, col = lcol0 + hb * 128;
                uint16_t* obase;
                if (g.o_tab_n) obase = tab[col / cb] + (col % cb);       // (a head never straddles a destination block)
                else {
                    const int c = seg_col0 + col;
                    obase = g.out + (g.o_cb ? (size_t)(c / g.o_cb) * g.o_cb_stride + (c % g.o_cb) : (size_t)c);
                }
                head_epilogue(g, t_row + hb * 128, row0, rows, obase, norm_w, BN == 256 ? 0 : half, BN == 256 ? 2 : half + 1, stg, lane);
            } else if (EPI == EPI_LORA) {
                // In-place update of W.  The contraction is short (9 x rank), so this epilogue's read-modify-write of W bounds
                // the kernel: a row's W values of two 32-column groups are requested before the first is used.
                const int row = row0 + lane;
                const bool row_ok = row < rows;
#pragma unroll 1
                for (int c4 = 0; c4 < BN / 128; ++c4) {
                    uint4 wv[2][4];
                    const int at = c4 * 128 + half * 64;
                    const uint16_t* wrow = g.out + (size_t)row * g.ldo + nb * BN + at;
                    if (row_ok) {
#pragma unroll
                        for (int c = 0; c < 2; ++c)
#pragma unroll
                            for (int i = 0; i < 4; ++i) wv[c][i] = reinterpret_cast<const uint4*>(wrow + c * 32)[i];
                    }
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        uint32_t r[32];
                        tmem_ld32(t_row + at + c * 32, r);
                        tmem_ld_wait();
                        if (row_ok) {
                            uint4* dst = reinterpret_cast<uint4*>(g.out + (size_t)row * g.ldo + nb * BN + at + c * 32);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint4 o = wv[c][i];
                                uint4 n;
                                n.x = pack_bf16x2(bf16lo(o.x) + g.scale * __uint_as_float(r[i * 8 + 0]),
                                                  bf16hi(o.x) + g.scale * __uint_as_float(r[i * 8 + 1]));
                                n.y = pack_bf16x2(bf16lo(o.y) + g.scale * __uint_as_float(r[i * 8 + 2]),
                                                  bf16hi(o.y) + g.scale * __uint_as_float(r[i * 8 + 3]));
                                n.z = pack_bf16x2(bf16lo(o.z) + g.scale * __uint_as_float(r[i * 8 + 4]),
                                                  bf16hi(o.z) + g.scale * __uint_as_float(r[i * 8 + 5]));
                                n.w = pack_bf16x2(bf16lo(o.w) + g.scale * __uint_as_float(r[i * 8 + 6]),
                                                  bf16hi(o.w) + g.scale * __uint_as_float(r[i * 8 + 7]));
                                dst[i] = n;
                            }
                        }
                    }
                }
            } else if constexpr (epi_plain(EPI) || EPI == EPI_QKV) {
                plain.run(g, t_row, row0, nb * BN, cols, half * 32, 64, stg, lane, failed);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster(map_to_rank(smem_u32(&tempty[as]), 0));
                else mbar_arrive(&tempty[as]);
            }
            if (++as == 2) { as = 0; aphase ^= 1; }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still signal it or feed an MMA
    tc_fence_after();
    if (warp == 1) {
        if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
        else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// ---------------------------------------------------------------- few tiles
// A problem with few output tiles leaves most SMs idle in the persistent kernel: a 77-row projection is 32 tiles of 128
// columns, the tower's fc2 at 520 rows 45 tiles of 68 K blocks.  This kernel takes one narrower tile (32 or 96 columns) per CTA, two CTAs
// per SM (one's epilogue runs under the other's main loop): the same sum for every element, for callers that rely on it.
// gemm_few_pair_kernel is its form on CTA pairs, and the one that sums a long K in parts.
// K blocks of weights requested into L2 ahead of their load, before the wait for the previous grid to begin with: three to
// five stages do not cover the way from memory (the persistent kernel's six do, and there the requests only cost: 24 -> 32 us at
// 77 x 4096 x 4096).  The row tiles of a column share them: the thread of the first one alone took 18 x 145 cycles for a K of 1152, and
// found room for them only where the kernel before left some (the tower of 520 patches 1777 -> 1764 us).
static constexpr int SK_PREFETCH = 24;
// KPS: K blocks per stage.  Two where an SM has one CTA anyway: the trip through a stage's barriers then counts half (a K
// block of a 32-column tile takes 290 cycles instead of 390-430; 77 x 4096 x 4096 17.8 -> 12.7 us).
template <int BN, int KPS>
struct SplitCfg {
    static constexpr int STAGES = BN <= 32 ? 5 : 3;      // with KPS = 1 as many as leave room for a second CTA
    static constexpr int STAGE_BYTES = KPS * (BM + BN) * BK * 2;
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /*align*/ + 128 /*barriers*/;
    static constexpr int TMEM_COLS = BN == 32 ? 32 : (BN == 96 ? 128 : 256);
    // (32 columns are one group for each quadrant; two CTAs of 144 have no registers for more)
    static constexpr int THREADS = BN == 96 || (BN == 144 && KPS == 2) ? GEMM_THREADS : SK_THREADS;
};
// The tower's q | k | v projection takes the same kernel unsplit with tiles of 144 columns, two whole heads of 72: a
// thread then holds both halves of its row's heads and the rotary is part of the epilogue (3456 = 24 tiles exactly).
static constexpr int VQ_BN = 144;
static constexpr int VQ_PITCH = 168;     // bytes of a staged row of one head: 16 lanes' 8-byte pieces meet 32 different banks

// Bias, rotary and the spacing of the tower's heads, for one head of 72 columns and the 32 rows of a warp.  bs: the head's bias; vcs, vsn: cos and
// sin of this thread's row; stg: 32 x VQ_PITCH bytes of the warp's own.
__device__ __forceinline__ void vrope_head(const GemmArgs& g, uint32_t t_head, int col, const uint2* bs, const float (&vcs)[36], const float (&vsn)[36],
                                           uint8_t* stg, int row0, bool failed, int lane) {
    const int which = col / 1152, h = (col - which * 1152) / 72;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; ++k) {      // twelve columns and their partners 36 further
        uint32_t rl[3][4], rh[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            tmem_ld4(t_head + k * 12 + i * 4, rl[i]);
            tmem_ld4(t_head + 36 + k * 12 + i * 4, rh[i]);
        }
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const uint2 bl = bs[k * 3 + i], bh = bs[9 + k * 3 + i];
            const float b0[4] = {bf16lo(bl.x), bf16hi(bl.x), bf16lo(bl.y), bf16hi(bl.y)};
            const float b1[4] = {bf16lo(bh.x), bf16hi(bh.x), bf16lo(bh.y), bf16hi(bh.y)};
            float lo[4], hi[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = bf16_round(bf16_round(__uint_as_float(rl[i][j])) + b0[j]);
                const float y = bf16_round(bf16_round(__uint_as_float(rh[i][j])) + b1[j]);
                const float c = vcs[(k * 3 + i) * 4 + j], sn = vsn[(k * 3 + i) * 4 + j];
                // fp32 rotary, one rounding (src/cuda/rope.cu:155-178); the table repeats after 36
                lo[j] = which < 2 ? rope_f32(x, c, -y, sn) : x;
                hi[j] = which < 2 ? rope_f32(y, c, x, sn) : y;
            }
            uint2* d = reinterpret_cast<uint2*>(stg + lane * VQ_PITCH) + k * 3 + i;
            d[0] = make_uint2(pack_bf16x2(lo[0], lo[1]), pack_bf16x2(lo[2], lo[3]));
            d[9] = make_uint2(pack_bf16x2(hi[0], hi[1]), pack_bf16x2(hi[2], hi[3]));
        }
    }
    __syncwarp();
    const int rows = failed ? 0 : g.M - row0;
    uint16_t* out = g.out + (size_t)row0 * g.ldo + (which * 16 + h) * 128;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        const int p = i * 32 + lane, r = p / 10, c = p - r * 10;
        const uint2* sp = reinterpret_cast<const uint2*>(stg + r * VQ_PITCH) + c * 2;
        uint4 o = make_uint4(0, 0, 0, 0);          // columns 72..79
        if (c < 9) { const uint2 o0 = sp[0], o1 = sp[1]; o = make_uint4(o0.x, o0.y, o1.x, o1.y); }
        if (r < rows) *reinterpret_cast<uint4*>(out + (size_t)r * g.ldo + c * 8) = o;
    }
}
__device__ __forceinline__ void vrope_tables(const GemmArgs& g, int row, float (&vcs)[36], float (&vsn)[36]) {
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const float4 c4 = *reinterpret_cast<const float4*>(g.rope + (size_t)row * 72 + c * 4);
        const float4 s4 = *reinterpret_cast<const float4*>(g.rope_sin + (size_t)row * 72 + c * 4);
        vcs[c * 4] = c4.x; vcs[c * 4 + 1] = c4.y; vcs[c * 4 + 2] = c4.z; vcs[c * 4 + 3] = c4.w;
        vsn[c * 4] = s4.x; vsn[c * 4 + 1] = s4.y; vsn[c * 4 + 2] = s4.z; vsn[c * 4 + 3] = s4.w;
    }
}

template <int EPI, int BN, int KPS>
__global__ void __launch_bounds__(SplitCfg<BN, KPS>::THREADS, KPS == 1 ? 2 : 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g) {
    static_assert(BN == 32 || BN == 96 || (BN == VQ_BN && EPI == EPI_VROPE), "the tiles there are");
    constexpr int SK_STAGE_BYTES = SplitCfg<BN, KPS>::STAGE_BYTES, SK_STAGES = SplitCfg<BN, KPS>::STAGES, NU = BN / 16;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + SK_STAGES * SK_STAGE_BYTES);
    uint64_t* empty = full + SK_STAGES;
    uint64_t* acc_done = empty + SK_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_done + 1);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    __shared__ uint4 bias_s[BN / 8];
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int nb = (int)(blockIdx.x / g.num_m), mb = (int)blockIdx.x - nb * g.num_m;      // CTAs that share weights run next to each other

    if (threadIdx.x == 64) *s_abort = error_word(g.err);
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < SK_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_done, 1);
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, SplitCfg<BN, KPS>::TMEM_COLS); tmem_relinquish(); }
    const int kblocks = (g.K + BK - 1) / BK;
    // the row tiles share the requests for the weights they all read
    const int span = g.prefetch * g.num_m;
    if (warp == 0 && elect_one())
        for (int i = mb; i < span && i < kblocks; i += g.num_m) tma_prefetch_2d(&tmB, i * BK, nb * BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    // (after a failure no loads and no results)
    bool ok = *s_abort == 0;
    const int failed = warp >= 2 ? error_word(g.err) : 0;

    if (ok && warp == 0) {
        if (elect_one()) {
            for (int i = 0, it = 0; i < kblocks; i += KPS, ++it) {
                const int s = it % SK_STAGES, n = kblocks - i < KPS ? kblocks - i : KPS;
                if (!mbar_wait(&empty[s], ((it / SK_STAGES) & 1) ^ 1)) { atomicExch(g.err, 51); break; }
                uint8_t* a_s = smem + s * SK_STAGE_BYTES;
                mbar_expect_tx(&full[s], n * (SK_STAGE_BYTES / KPS));
                for (int u = 0; u < n; ++u) {
                    if (mb == 0 && span > 0 && i + u + span < kblocks) tma_prefetch_2d(&tmB, (i + u + span) * BK, nb * BN);
                    int a_c0 = (i + u) * BK, a_c1 = mb * BM;
                    if (g.a_kblk > 0) {
                        const int blk = a_c0 / g.a_kblk;
                        a_c0 -= blk * g.a_kblk;
                        a_c1 += blk * g.a_rows;
                    }
                    tma_load_2d(a_s + u * BM * BK * 2, &tmA, &full[s], a_c0, a_c1);
                    tma_load_2d(a_s + KPS * BM * BK * 2 + u * BN * BK * 2, &tmB, &full[s], (i + u) * BK, nb * BN);
                }
            }
        }
    } else if (ok && warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, 0, 0);
            bool good = true;
            for (int i = 0, it = 0; i < kblocks && good; i += KPS, ++it) {
                const int s = it % SK_STAGES;
                if (!mbar_wait(&full[s], (it / SK_STAGES) & 1)) { atomicExch(g.err, 52); good = false; break; }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(smem + s * SK_STAGE_BYTES);
#pragma unroll
                for (int u = 0; u < KPS; ++u) {
                    if (i + u >= kblocks) break;
                    const uint64_t ad = umma_desc_sw128(a_addr + u * BM * BK * 2, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + KPS * BM * BK * 2 + u * BN * BK * 2, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_ss(tmem_base, ad + 2 * k, bd + 2 * k, idesc, (i | u | k) != 0);
                }
                umma_commit(&empty[s]);
            }
            umma_commit(acc_done);
        }
    }
    if constexpr (BN == 96 || (BN == 32 && epi_has_resid(EPI))) {
        // whole K: the epilogue of the persistent kernels, with the stages as its staging once the MMAs are through with them
        // (32 columns without a residual are better stored directly: 77 x 4096 x 4096 12.66 us against 12.81)
        const int row0 = mb * BM + (warp & 3) * 32, col0 = nb * BN, cols = g.N - col0 < BN ? g.N - col0 : BN;
        const int half = (warp - 2) >> 2;        // (always 0 with 32 columns)
        if (ok && warp >= 2) {
            PlainEpilogue<EPI> plain;
            plain.ahead(g, row0, col0, cols, half * 32, lane);
            if (!mbar_wait(acc_done, 0)) { atomicExch(g.err, 53); ok = false; }
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            if (ok) plain.run(g, tmem_base + ((uint32_t)((warp & 3) * 32) << 16), row0, col0, cols, half * 32, 64,
                              smem + (warp - 2) * EPI_SLICE, lane, failed);
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (warp == 1) tmem_dealloc(tmem_base, SplitCfg<BN, KPS>::TMEM_COLS);
        return;
    }
    // (32 columns without a residual, or the tower's 144.)  The tile's bias comes into shared memory while the main loop runs: each of
    // its units of 16 columns would otherwise wait for its own loads.
    constexpr bool HAS_BIAS = epi_has_bias(EPI) || EPI == EPI_VROPE;
    const int q = warp & 3;       // TMEM lane quadrant this warp may access
    const int trow = q * 32 + lane;
    const int row = mb * BM + trow;
    const bool row_ok = row < g.M;
    float vcs[36], vsn[36];      // (EPI_VROPE)
    if (ok && warp >= 2) {
        if (EPI == EPI_VROPE) {
            vrope_tables(g, row_ok ? row : 0, vcs, vsn);
        }
        if (HAS_BIAS && trow * 8 < BN) {
            const int col = nb * BN + trow * 8;
            bias_s[trow] = col < g.N ? *reinterpret_cast<const uint4*>(g.bias + col) : make_uint4(0, 0, 0, 0);
        }
        if (HAS_BIAS) asm volatile("bar.sync 1, %0;" ::"n"(SplitCfg<BN, KPS>::THREADS - 64) : "memory");      // the epilogue warps
    }
    if (ok && warp >= 2) {
        if (!mbar_wait(acc_done, 0)) { atomicExch(g.err, 53); ok = false; }
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
    }
    const bool store = row_ok && !failed;
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
    if constexpr (EPI == EPI_VROPE) {
        // Bias, rotary and the spacing of the heads.  cos and sin of this thread's row have come into registers under the main
        // loop; a head goes through shared memory (the stages are free now) and leaves as whole rows of 160 bytes.  With cos / sin
        // loaded per head and every thread storing its own row, 32 lines to an instruction, this epilogue took three times the
        // main loop's time: the launch 21.4 -> 14.6 us at 520 rows and 60.8 -> 43.8 us at 4096.
        if (ok && warp >= 2) {
            // (with one CTA on an SM a head for each of eight warps)
            uint8_t* stg = smem + (warp - 2) * (32 * VQ_PITCH);
#pragma unroll 1
            for (int hh = (warp - 2) >> 2; hh < 2; hh += SplitCfg<BN, KPS>::THREADS == GEMM_THREADS ? 2 : 1) {
                vrope_head(g, t_row + hh * 72, nb * VQ_BN + hh * 72, reinterpret_cast<const uint2*>(bias_s) + hh * 18, vcs, vsn, stg, mb * BM + q * 32,
                           failed, lane);
            }
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        if (warp == 1) tmem_dealloc(tmem_base, SplitCfg<BN, KPS>::TMEM_COLS);
        return;
    }
    if (ok && warp >= 2) {
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            const int col = nb * BN + u * 16;
            // (N is a multiple of eight: a unit is whole, its first half, or outside)
            const bool h0 = store && col < g.N, h1 = store && col + 8 < g.N;
            uint32_t r[16];
            tmem_ld16(t_row + u * 16, r);
            tmem_ld_wait();
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __fadd_rn(0.f, __uint_as_float(r[j]));
            // the rounding points of gemm_tc_kernel's epilogues
            float b[16];
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (HAS_BIAS) unpack8_bf16(bias_s[2 * u + h], b + h * 8);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (EPI == EPI_BIAS) v[j] = bf16_round(v[j]) + b[j];
                if (EPI == EPI_BIAS_GELU) v[j] = bf16_round(bf16_round(v[j]) + b[j]);
            }
            if (EPI == EPI_BIAS_GELU) gelu_all(v, g.scale != 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float* w = v + h * 8;
                uint4 o;
                o.x = pack_bf16x2(w[0], w[1]); o.y = pack_bf16x2(w[2], w[3]);
                o.z = pack_bf16x2(w[4], w[5]); o.w = pack_bf16x2(w[6], w[7]);
                if (h ? h1 : h0) *reinterpret_cast<uint4*>(g.out + (size_t)row * g.ldo + col + h * 8) = o;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, SplitCfg<BN, KPS>::TMEM_COLS);
}

// ---------------------------------------------------------------- narrow tiles on CTA pairs
// The 32-column form with two CTAs to a tile of 128 rows x 64 to 128 columns: each has half of the rows of the activations, half of the weights
// and, in its tensor memory, its rows of the result; and four K blocks to a copy.  What bounds the narrow tiles is the thread that
// issues the copies, some 145 cycles for each whatever its size (two for a K block, and one for L2), and shared memory: an MMA of 128 x 32 x 16
// reads 5 KB while the copies write as much, the pair's of 128 x 64 x 16 reads and writes 3 KB on an SM.  Same order of the
// sum, so the same bits.
// PARTS: so too where the K of a tile is to be summed in parts.  The parts follow one another, each in an accumulator of its
// own, and the epilogue adds them in their order.  (When the CTAs of a cluster shared them, the exchange took 13,000 of 33,000 cycles at
// 520 x 1152 x 4304, the main loop 11,000.)  fewpair_cols() has both sides' times.
// How many bytes of weights are on their way decides the time (77 x 4096 x 4096: two stages of four K blocks 16.6 us, four 11.3), so a stage
// holds no more rows of the activations than there are: a tile of up to 128 rows is shared evenly, `ra` rows (a multiple of eight)
// to a CTA.  The MMA reads 64, the others from whatever lies behind: their results are not used.
static constexpr int FP_KPS = 4;      // K blocks a stage and copy
static constexpr int FP_MAX_STAGES = 12, FP_ROOM = 216 * 1024;
static constexpr int FP_SMEM = FP_ROOM + 1024 /*align*/ + 256 /*barriers*/;
__host__ __device__ constexpr int fp_stage_bytes(int ra, int fc) { return FP_KPS * (ra + fc) * BK * 2; }

template <int EPI, bool PARTS>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_few_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmA2, const __grid_constant__ CUtensorMap tmB2, const GemmArgs g, const int ra, const int fc,
                     const int stages, const int parts) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + stages * fp_stage_bytes(ra, fc));
    uint64_t* empty = full + FP_MAX_STAGES;
    uint64_t* acc_done = empty + FP_MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_done + 1);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    cluster_arrive();
    const int tile = (int)(blockIdx.x >> 1);
    const int nb = tile / g.num_m, mb = tile - nb * g.num_m;      // CTAs that share weights run next to each other
    const int stage_bytes = fp_stage_bytes(ra, fc), a_bytes = ra * BK * 2;
    const int a_row = mb * 2 * ra + (int)rank * ra, b_row = nb * 2 * fc + (int)rank * fc;

    if (threadIdx.x == 64) *s_abort = error_word(g.err);
    if (threadIdx.x == 96) {
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_done, 1);
        fence_mbar_init();
    }
    cluster_wait();
    if (warp == 1) tmem_alloc_pair(tmem_slot, PARTS ? 512 : 64);
    // whole K blocks come FP_KPS to a copy, a ragged last one by itself (tmA2, tmB2)
    const int kblocks = (g.K + BK - 1) / BK, kwhole = g.K / BK;
    if (warp == 0 && elect_one()) {
        tma_prefetch_desc(&tmB);
        tma_prefetch_desc(&tmA);
        // the row tiles share the requests for the weights they all read; for a long K (PARTS) all of them make as many as one would
        const int most = PARTS ? g.prefetch * g.num_m : g.prefetch;
        for (int i = mb * FP_KPS; i < most && i < kwhole; i += g.num_m * FP_KPS) tma_prefetch_3d(&tmB, 0, b_row, i);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    if (warp == 1) tmem_relinquish_pair();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const bool live = (*s_abort | ld_cluster_s32(map_to_rank(smem_u32(s_abort), rank ^ 1u))) == 0;

    if (live && warp == 0) {
        if (elect_one()) {
            uint32_t phase = 0;
            for (int i = 0, s = 0; i < kblocks;) {
                if (!mbar_wait(&empty[s], phase ^ 1)) { atomicExch(g.err, 91); break; }
                uint8_t* a_s = smem + s * stage_bytes;
                if (i < kwhole) {
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes);      // both CTAs' halves
                    tma_load_3d_pair(a_s, &tmA, &full[s], 0, a_row, i);
                    tma_load_3d_pair(a_s + FP_KPS * a_bytes, &tmB, &full[s], 0, b_row, i);
                    i = i + FP_KPS < kwhole ? i + FP_KPS : kwhole;
                } else {
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes / FP_KPS);
                    tma_load_2d_pair(a_s, &tmA2, &full[s], i * BK, a_row);
                    tma_load_2d_pair(a_s + FP_KPS * a_bytes, &tmB2, &full[s], i * BK, b_row);
                    ++i;
                }
                if (++s == stages) { s = 0; phase ^= 1; }
            }
        }
    } else if (live && warp == 1) {
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc_bf16(BM, 2 * fc, 0, 0);
            uint32_t phase = 0, d = tmem_base;
            int p = 0, p_end = kblocks / parts;      // K part, first K block of the next one
            bool fresh = true;                       // nothing in its accumulator yet
            for (int i = 0, s = 0; i < kblocks;) {
                if (!mbar_wait(&full[s], phase)) { atomicExch(g.err, 92); break; }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(smem + s * stage_bytes);
                const int n = i < kwhole ? (kwhole - i < FP_KPS ? kwhole - i : FP_KPS) : 1;
#pragma unroll
                for (int u = 0; u < FP_KPS; ++u) {
                    if (u >= n) break;
                    if (PARTS && i + u == p_end && p + 1 < parts) { ++p; p_end = (p + 1) * kblocks / parts; d += fc; fresh = true; }
                    const uint64_t ad = umma_desc_sw128(a_addr + u * a_bytes, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + FP_KPS * a_bytes + u * fc * BK * 2, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_ss_pair(d, ad + 2 * k, bd + 2 * k, idesc, k != 0 || !fresh);
                    fresh = false;
                }
                i += n;
                umma_commit_pair(&empty[s]);
                if (++s == stages) { s = 0; phase ^= 1; }
            }
            umma_commit_pair(acc_done);
        }
    } else if (live) {
        // With 64 rows to a CTA the lanes 0..63 of its tensor memory hold the first half of the tile's columns, 64..127 the other half of
        // the same rows.
        const int q = warp & 3, failed = error_word(g.err);
        const int row0 = a_row + (q & 1) * 32;
        const int col0 = nb * 2 * fc + (q >> 1) * fc, cols = g.N - col0 < fc ? g.N - col0 : fc;
        PlainEpilogue<EPI, true, PARTS> plain;
        plain.row_end = a_row + ra < g.M ? a_row + ra : g.M;
        if (PARTS) { plain.parts = parts; plain.part_cols = fc; }
        const int c_first = ((warp - 2) >> 2) * 32, c_step = ((int)blockDim.x - 64) >> 2;     // four or eight warps
        if (cols > c_first) plain.ahead(g, row0, col0, cols, c_first, lane);
        bool ok = mbar_wait(acc_done, 0);
        if (!ok) atomicExch(g.err, 93);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        // (all MMAs are through with the stages, which serve as staging)
        if (ok && cols > c_first) plain.run(g, tmem_base + ((uint32_t)(q * 32) << 16), row0, col0, cols, c_first, c_step, smem + (warp - 2) * EPI_SLICE, lane, failed);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still signal it or feed an MMA
    tc_fence_after();
    if (warp == 1) tmem_dealloc_pair(tmem_base, PARTS ? 512 : 64);
}

// ---------------------------------------------------------------- tiles fitted to the number of SMs
// The persistent kernel with a tile width chosen at run time, a multiple of 16 from 144 to 192 columns: where 128 or 256
// columns leave a last round of few tiles (1280 rows x 4096 columns: 320 tiles for 148 SMs, three rounds for 2.2), some
// width in between often makes whole rounds (144 columns: 290 tiles, two rounds).  A block of 1280 rows went from 539 to
// 503 us, a guided step of 2 x 296 rows from 11.1 to 10.5 ms.  Same warps, same pipeline and the same sums; plain
// row-major output with the bias or residual epilogue.  (The epilogue's slices take 17 KB: 160 columns have five stages where six
// would fit without, 800 x 3072 x 4096 23.7 us with six, 23.6 with five.)
static constexpr int FIT_MAX_STAGES = 6, FIT_ROOM = 208 * 1024 /*stages*/, FIT_SMEM = FIT_ROOM + EPI_WARPS * EPI_SLICE + 1024 /*align*/ + 256 /*barriers*/;

template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_fit_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g, const int bn,
                const int stages) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int stage_bytes = (BM + bn) * BK * 2;      // (bn is a multiple of 16: the stages stay 1024-byte aligned)
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + FIT_ROOM + EPI_WARPS * EPI_SLICE);
    uint64_t* empty = full + FIT_MAX_STAGES;
    uint64_t* tfull = empty + FIT_MAX_STAGES;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 64) *s_abort = error_word(g.err);
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&tfull[s], 1); mbar_init(&tempty[s], EPI_WARPS); }
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const bool live = *s_abort == 0;
    const int num_tiles = g.num_m * g.num_n, kblocks = (g.K + BK - 1) / BK;

    if (live && warp == 0) {
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                int mb, nb;
                tile_coords(tile, g.num_m, g.num_n, g.group_m, mb, nb);
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1)) { ok = false; atomicExch(g.err, 61); break; }
                    uint8_t* a_s = smem + stage * stage_bytes;
                    mbar_expect_tx(&full[stage], stage_bytes);
                    int a_c0 = kb * BK, a_c1 = mb * BM;
                    if (g.a_kblk > 0) {
                        const int blk = a_c0 / g.a_kblk;
                        a_c0 -= blk * g.a_kblk;
                        a_c1 += blk * g.a_rows;
                    }
                    tma_load_2d(a_s, &tmA, &full[stage], a_c0, a_c1);
                    tma_load_2d(a_s + BM * BK * 2, &tmB, &full[stage], kb * BK, nb * bn);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (live && warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_bf16(BM, bn, 0, 0);
            int stage = 0, as = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                if (!mbar_wait(&tempty[as], aphase ^ 1)) { atomicExch(g.err, 62); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * 256;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&full[stage], phase)) { ok = false; atomicExch(g.err, 63); break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
                    const uint64_t ad = umma_desc_sw128(a_addr, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + BM * BK * 2, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_ss(d_tmem, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                    umma_commit(&empty[stage]);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
                umma_commit(&tfull[as]);
                if (++as == 2) { as = 0; aphase ^= 1; }
            }
        }
    } else if (live) {
        const int q = warp & 3, half = (warp - 2) >> 2;       // (as in gemm_tc_kernel)
        uint8_t* stg = smem + FIT_ROOM + (warp - 2) * EPI_SLICE;
        int as = 0;
        uint32_t aphase = 0;
        const int failed = error_word(g.err);
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
            int mb, nb;
            tile_coords(tile, g.num_m, g.num_n, g.group_m, mb, nb);
            const int row0 = mb * BM + q * 32, col0 = nb * bn, cols = g.N - col0 < bn ? g.N - col0 : bn;
            PlainEpilogue<EPI> plain;
            plain.ahead(g, row0, col0, cols, half * 32, lane);
            const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull[as], aphase));
            if (!got) { atomicExch(g.err, 64); break; }
            tc_fence_after();
            plain.run(g, tmem_base + as * 256 + ((uint32_t)(q * 32) << 16), row0, col0, cols, half * 32, 64, stg, lane, failed);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[as]);
            if (++as == 2) { as = 0; aphase ^= 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ---------------------------------------------------------------- CTA pairs with a tile width chosen at run time
// The pair form (256 rows over two CTAs, each with half of the B tile) for any width that is a multiple of 16, any N and every
// epilogue with plain row-major output, and for the tower's q | k | v (EPI_VROPE).  Narrower tiles pay where they make fewer or fuller rounds: a one-CTA tile of 128 x 128
// brings 32 KB into an SM per K block and is bound by that (70 bytes a clock); half a pair tile of 256 x 128 brings 24 KB for the
// same products.
static constexpr int PF_MAX_STAGES = 8, PF_STAGE_ROOM = 192 * 1024, PF_STORE = EPI_WARPS * EPI_SLICE;
static constexpr int PF_SMEM = PF_STAGE_ROOM + PF_STORE + 1024 /*align*/ + 256 /*barriers*/;
// EPI_VROPE: two heads to a tile, one for each of a quadrant's two warps, whose slice holds 32 staged rows of it and its bias.
static constexpr int PFV_STAGES = 7, PFV_ROOM = PFV_STAGES * (BM + VQ_BN / 2) * BK * 2, PFV_SLICE = 32 * VQ_PITCH + 160, PFV_STORE = EPI_WARPS * PFV_SLICE;
static constexpr int PFV_SMEM = PFV_ROOM + PFV_STORE + 1024 /*align*/ + 256 /*barriers*/;

template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_fit_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmArgs g, const int bn,
                     const int stages) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int stage_bytes = (BM + bn / 2) * BK * 2;      // (bn is a multiple of 16: the stages stay 1024-byte aligned)
    uint8_t* store_s = smem + (EPI == EPI_VROPE ? PFV_ROOM : PF_STAGE_ROOM);
    uint64_t* full = reinterpret_cast<uint64_t*>(store_s + (EPI == EPI_VROPE ? PFV_STORE : PF_STORE));
    uint64_t* empty = full + PF_MAX_STAGES;
    uint64_t* tfull = empty + PF_MAX_STAGES;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    cluster_arrive();
    if (threadIdx.x == 64) *s_abort = error_word(g.err);
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&tfull[s], 1); mbar_init(&tempty[s], 2 * EPI_WARPS); }
        fence_mbar_init();
    }
    cluster_wait();
    if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
    const int num_m = (g.num_m + 1) / 2, group_m = (g.group_m + 1) / 2;
    const int num_tiles = num_m * g.num_n, kblocks = (g.K + BK - 1) / BK;
    const int tile0 = (int)(blockIdx.x >> 1), tile_step = (int)(gridDim.x >> 1);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    if (warp == 1) tmem_relinquish_pair();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const bool live = (*s_abort | ld_cluster_s32(map_to_rank(smem_u32(s_abort), rank ^ 1u))) == 0;

    if (live && warp == 0) {
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                int mb, nb;
                tile_coords(tile, num_m, g.num_n, group_m, mb, nb);
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1)) { ok = false; atomicExch(g.err, 71); break; }
                    uint8_t* a_s = smem + stage * stage_bytes;
                    if (rank == 0) mbar_expect_tx(&full[stage], 2 * stage_bytes);      // both CTAs' halves
                    int a_c0 = kb * BK, a_c1 = (mb * 2 + (int)rank) * BM;
                    if (g.a_kblk > 0) {
                        const int blk = a_c0 / g.a_kblk;
                        a_c0 -= blk * g.a_kblk;
                        a_c1 += blk * g.a_rows;
                    }
                    tma_load_2d_pair(a_s, &tmA, &full[stage], a_c0, a_c1);
                    tma_load_2d_pair(a_s + BM * BK * 2, &tmB, &full[stage], kb * BK, nb * bn + (int)rank * (bn / 2));
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (live && warp == 1) {
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc_bf16(2 * BM, bn, 0, 0);
            int stage = 0, as = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                if (!mbar_wait(&tempty[as], aphase ^ 1)) { atomicExch(g.err, 72); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * 256;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&full[stage], phase)) { ok = false; atomicExch(g.err, 73); break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
                    const uint64_t ad = umma_desc_sw128(a_addr, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + BM * BK * 2, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_ss_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                    umma_commit_pair(&empty[stage]);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
                umma_commit_pair(&tfull[as]);
                if (++as == 2) { as = 0; aphase ^= 1; }
            }
        }
    } else if (live) {
        const int q = warp & 3, half = (warp - 2) >> 2;       // (as in gemm_tc_kernel)
        uint8_t* stg = store_s + (warp - 2) * (EPI == EPI_VROPE ? PFV_SLICE : EPI_SLICE);
        int as = 0;
        uint32_t aphase = 0;
        const int failed = error_word(g.err);
        for (int tile = tile0; tile < num_tiles; tile += tile_step) {
            int mb, nb;
            tile_coords(tile, num_m, g.num_n, group_m, mb, nb);
            const int row0 = (mb * 2 + (int)rank) * BM + q * 32;
            const uint32_t t_row = tmem_base + as * 256 + ((uint32_t)(q * 32) << 16);
            if constexpr (EPI == EPI_VROPE) {
                const int col0 = nb * VQ_BN + half * 72;
                float vcs[36], vsn[36];
                vrope_tables(g, row0 + lane < g.M ? row0 + lane : 0, vcs, vsn);
                uint2* bs = reinterpret_cast<uint2*>(stg + 32 * VQ_PITCH);
                if (lane < 18) bs[lane] = *reinterpret_cast<const uint2*>(g.bias + col0 + lane * 4);
                const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull[as], aphase));
                if (!got) { atomicExch(g.err, 74); break; }
                tc_fence_after();
                vrope_head(g, t_row + half * 72, col0, bs, vcs, vsn, stg, row0, failed, lane);
                __syncwarp();      // (the bias and the staged rows have been read)
            } else {
                const int col0 = nb * bn, cols = g.N - col0 < bn ? g.N - col0 : bn;
                PlainEpilogue<EPI> plain;
                plain.ahead(g, row0, col0, cols, half * 32, lane);
                const bool got = __all_sync(0xffffffffu, mbar_wait(&tfull[as], aphase));
                if (!got) { atomicExch(g.err, 74); break; }
                tc_fence_after();
                plain.run(g, t_row, row0, col0, cols, half * 32, 64, stg, lane, failed);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&tempty[as]), 0));
            if (++as == 2) { as = 0; aphase ^= 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still signal it or feed an MMA
    tc_fence_after();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---------------------------------------------------------------- CTA pairs fitted to the number of rows
// Gate | up + SwiGLU and q | k | v have epilogues that fix the columns of a tile, so the pair kernel pays whole 256s of rows: 592 rows
// as 768.  Here the operands change places: 256 rows of WEIGHTS are the M of the MMA (128 in each CTA: 64 gate rows and the 64
// up rows of the same columns, or one head), and the tokens its N, any multiple of 16 up to 256: 592 rows as three tiles of 208.
// The products and the order of their sums are the same, so the bits are.  An accumulator holds a column of the output per lane; 16
// tokens at a time go through shared memory as bf16 (the first rounding of both epilogues) and come back by token, from four warps.
// The rule, and both sides' times: rows_width().
static constexpr int RW_TOK = 16;                          // tokens of a group
static constexpr int RW_STAGE = RW_TOK * 256;              // their 128 columns
static constexpr int RW_STORE = 2 * 2 * RW_STAGE;          // two groups of four warps, two buffers each
static constexpr int RW_SMEM = PF_STAGE_ROOM + RW_STORE + 1024 /*align*/ + 256 /*barriers*/;

template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                 const __grid_constant__ CUtensorMap tmW3, const GemmArgs g, const int bn, const int stages) {
    static_assert(EPI == EPI_SWIGLU || EPI == EPI_QKV, "the other epilogues have tiles of any number of columns");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int stage_bytes = (BM + bn / 2) * BK * 2;      // (bn is a multiple of 16: the stages stay 1024-byte aligned)
    uint8_t* store_s = smem + PF_STAGE_ROOM;
    uint64_t* full = reinterpret_cast<uint64_t*>(store_s + RW_STORE);
    uint64_t* empty = full + PF_MAX_STAGES;
    uint64_t* tfull = empty + PF_MAX_STAGES;
    uint64_t* tempty = tfull + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    cluster_arrive();
    if (threadIdx.x == 64) *s_abort = error_word(g.err);
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmW);
        tma_prefetch_desc(&tmW2);
        if (EPI == EPI_QKV) tma_prefetch_desc(&tmW3);
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&tfull[s], 1); mbar_init(&tempty[s], 2 * EPI_WARPS); }
        fence_mbar_init();
    }
    cluster_wait();
    if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
    const int num_tiles = g.num_m * g.num_n, kblocks = (g.K + BK - 1) / BK;
    const int tile0 = (int)(blockIdx.x >> 1), tile_step = (int)(gridDim.x >> 1);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // both CTAs' barriers exist before either signals the other's
    tc_fence_after();
    if (warp == 1) tmem_relinquish_pair();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem_base = *tmem_slot;
    const bool live = (*s_abort | ld_cluster_s32(map_to_rank(smem_u32(s_abort), rank ^ 1u))) == 0;
    // q | k | v: the weight tensor of this CTA's head and the head's first column in it
    auto segment = [&](int nb, int& lcol0) {
        const int col0 = nb * 256 + (int)rank * 128;
        const int seg = col0 >= g.seg_n[0] + g.seg_n[1] ? 2 : (col0 >= g.seg_n[0] ? 1 : 0);
        lcol0 = col0 - (seg == 2 ? g.seg_n[0] + g.seg_n[1] : (seg == 1 ? g.seg_n[0] : 0));
        return seg;
    };

    if (live && warp == 0) {
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                int mb, nb, lrow = 0;
                tile_coords(tile, g.num_m, g.num_n, g.group_m, mb, nb);
                const int seg = EPI == EPI_QKV ? segment(nb, lrow) : 0;
                const CUtensorMap* mW = seg == 0 ? &tmW : (seg == 1 ? &tmW2 : &tmW3);
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&empty[stage], phase ^ 1)) { ok = false; atomicExch(g.err, 81); break; }
                    uint8_t* a_s = smem + stage * stage_bytes;
                    if (rank == 0) mbar_expect_tx(&full[stage], 2 * stage_bytes);      // both CTAs' halves
                    if (EPI == EPI_SWIGLU) {
                        tma_load_2d_pair(a_s, &tmW, &full[stage], kb * BK, nb * 128 + (int)rank * 64);
                        tma_load_2d_pair(a_s + 64 * BK * 2, &tmW2, &full[stage], kb * BK, nb * 128 + (int)rank * 64);
                    } else {
                        tma_load_2d_pair(a_s, mW, &full[stage], kb * BK, lrow);
                    }
                    tma_load_2d_pair(a_s + BM * BK * 2, &tmX, &full[stage], kb * BK, mb * bn + (int)rank * (bn / 2));
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (live && warp == 1) {
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc_bf16(2 * BM, bn, 0, 0);
            int stage = 0, as = 0;
            uint32_t phase = 0, aphase = 0;
            bool ok = true;
            for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
                if (!mbar_wait(&tempty[as], aphase ^ 1)) { atomicExch(g.err, 82); break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + as * 256;
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (!mbar_wait(&full[stage], phase)) { ok = false; atomicExch(g.err, 83); break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
                    const uint64_t ad = umma_desc_sw128(a_addr, 16, 1024);
                    const uint64_t bd = umma_desc_sw128(a_addr + BM * BK * 2, 16, 1024);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) umma_ss_pair(d_tmem, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
                    umma_commit_pair(&empty[stage]);
                    if (++stage == stages) { stage = 0; phase ^= 1; }
                }
                umma_commit_pair(&tfull[as]);
                if (++as == 2) { as = 0; aphase ^= 1; }
            }
        }
    } else if (live) {
        const int q = warp & 3, grp = (warp - 2) >> 2;       // quadrant of tensor memory, which of the two groups of four warps
        const int tid = q * 32 + lane, tok = tid >> 3, t = tid & 7;      // by token: eight lanes each
        uint8_t* stg = store_s + grp * 2 * RW_STAGE;
        int as = 0, buf = 0;
        uint32_t aphase = 0;
        const int failed = error_word(g.err);
        bool ok = true;       // (a warp whose wait ran out goes on through its group's barriers, and does nothing else)
        for (int tile = tile0; tile < num_tiles; tile += tile_step) {
            int mb, nb, lcol0 = 0;
            tile_coords(tile, g.num_m, g.num_n, g.group_m, mb, nb);
            const int row0 = mb * bn, rows = g.M - row0 < bn ? g.M - row0 : bn;
            const int seg = EPI == EPI_QKV ? segment(nb, lcol0) : 0;
            uint16_t* obase = g.out + (EPI == EPI_SWIGLU ? nb * 128 + (int)rank * 64 : nb * 256 + (int)rank * 128);
            float wl[8], wh[8];
            if (EPI == EPI_QKV && seg < 2) {
                unpack8_bf16(*reinterpret_cast<const uint4*>(g.seg_norm[seg] + 8 * t), wl);
                unpack8_bf16(*reinterpret_cast<const uint4*>(g.seg_norm[seg] + 64 + 8 * t), wh);
            }
            if (ok && !__all_sync(0xffffffffu, mbar_wait(&tfull[as], aphase))) { atomicExch(g.err, 84); ok = false; }
            tc_fence_after();
            const uint32_t t_row = tmem_base + as * 256 + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c = grp * RW_TOK; c < rows; c += 2 * RW_TOK, buf ^= 1) {
                uint8_t* st = stg + buf * RW_STAGE;
                if (ok) {
                    uint32_t r[RW_TOK];
                    tmem_ld16(t_row + c, r);
                    tmem_ld_wait();
                    // this lane's column of 16 tokens: a warp writes 64 bytes of each
#pragma unroll
                    for (int j = 0; j < RW_TOK; j += 2) {
                        const uint32_t p = pack_bf16x2(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
                        *reinterpret_cast<uint16_t*>(st + j * 256 + tid * 2) = (uint16_t)p;
                        *reinterpret_cast<uint16_t*>(st + (j + 1) * 256 + tid * 2) = (uint16_t)(p >> 16);
                    }
                }
                // (one barrier a group: a buffer is written again behind the next one, when all four warps have read it)
                asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory");
                const int row = row0 + c + tok;
                const bool row_ok = ok && !failed && c + tok < rows;
                const uint4* in = reinterpret_cast<const uint4*>(st + tok * 256) + t;
                if (EPI == EPI_SWIGLU) {
                    float v[8], u[8];
                    unpack8_bf16(in[0], v);
                    unpack8_bf16(in[8], u);
                    swiglu_vals(v, u);
                    if (row_ok) *reinterpret_cast<uint4*>(obase + (size_t)row * g.ldo + 8 * t) =
                        make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
                } else if (seg < 2) {
                    head_row(g, reinterpret_cast<const uint8_t*>(in), reinterpret_cast<const uint8_t*>(in + 8), wl, wh, row, row_ok, obase, t);
                } else if (row_ok) {
                    uint4* o = reinterpret_cast<uint4*>(obase + (size_t)row * g.ldo) + t;
                    o[0] = in[0];
                    o[8] = in[8];
                }
            }
            tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&tempty[as]), 0));
            if (++as == 2) { as = 0; aphase ^= 1; }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // neither CTA leaves (or frees tensor memory) while the other may still signal it or feed an MMA
    tc_fence_after();
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---------------------------------------------------------------- SIMT path
// For M < 8 (timestep MLP, M = 1) and for shapes the tensor-core tiles do not cover.  One warp per output column and MR
// rows: bound by the weights' way from memory, so a weight is read once for all its rows, four 16-byte pieces of a lane at
// a time.
// A warp per row needs every warp an SM holds: 36 registers instead of 32, two blocks fewer, cost 10 % (4096 x 4096, 2 rows).
template <int MR>
__global__ void __launch_bounds__(128, MR == 1 ? 16 : 1)
gemm_simt_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w,
                                 const uint16_t* __restrict__ bias, uint16_t* __restrict__ y, int M,
                                 int N, int K, int ldx, int ldy) {
    grid_dep_launch();
    grid_dep_wait();
    const int warps_per_block = blockDim.x >> 5;
    const int n = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
    const int m0 = blockIdx.y * MR;
    const int lane = threadIdx.x & 31;
    if (n >= N) return;
    const uint16_t* xr[MR];
#pragma unroll
    for (int i = 0; i < MR; ++i) xr[i] = x + (size_t)(m0 + i < M ? m0 + i : M - 1) * ldx;
    const uint16_t* wr = w + (size_t)n * K;
    float acc[MR] = {};
    // the rows and the weights lie on 16-byte boundaries
    if (((K | (MR == 1 ? m0 * ldx : ldx)) & 7) == 0 && ((((uintptr_t)x) | ((uintptr_t)w)) & 15) == 0) {
        constexpr int UN = MR == 1 ? 1 : 4;
#pragma unroll 4
        for (int k0 = lane * 8; k0 < K; k0 += 256 * UN) {
            uint4 b[UN];
#pragma unroll
            for (int u = 0; u < UN; ++u)
                b[u] = k0 + u * 256 < K ? *reinterpret_cast<const uint4*>(wr + k0 + u * 256) : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < UN; ++u) {
                if (k0 + u * 256 >= K) break;
#pragma unroll
                for (int i = 0; i < MR; ++i) {
                    const uint4 a = *reinterpret_cast<const uint4*>(xr[i] + k0 + u * 256);
                    acc[i] += bf16lo(a.x) * bf16lo(b[u].x); acc[i] += bf16hi(a.x) * bf16hi(b[u].x);
                    acc[i] += bf16lo(a.y) * bf16lo(b[u].y); acc[i] += bf16hi(a.y) * bf16hi(b[u].y);
                    acc[i] += bf16lo(a.z) * bf16lo(b[u].z); acc[i] += bf16hi(a.z) * bf16hi(b[u].z);
                    acc[i] += bf16lo(a.w) * bf16lo(b[u].w); acc[i] += bf16hi(a.w) * bf16hi(b[u].w);
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32)
#pragma unroll
            for (int i = 0; i < MR; ++i) acc[i] += bf16_to_f32(xr[i][k]) * bf16_to_f32(wr[k]);
    }
#pragma unroll
    for (int i = 0; i < MR; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        if (lane == 0 && m0 + i < M) {
            float v = acc[i];
            if (bias) v = bf16_round(v) + bf16_to_f32(bias[n]);
            y[(size_t)(m0 + i) * ldy + n] = f32_to_bf16(v);
        }
    }
}

// ---------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres);
        if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess) fn = (EncodeTiledFn)p;
    });
    return fn;
}

// Row-major bf16 matrix [rows, cols] with row pitch ld (elements); box is
// 64 columns x box_rows rows, 128-byte swizzle.
bool make_tmap_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("tensor map: cuTensorMapEncodeTiled entry point unavailable"); return false; }
    if ((((uintptr_t)base) & 15) || ((ld * 2) & 15)) {
        set_error("tensor map: base/pitch not 16-byte aligned");
        return false;
    }
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {ld * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("tensor map: encode failed (%d)", (int)r); return false; }
    return true;
}

// [heads][rows][cols] with pitches ld and hoff (elements), boxes of 64 columns x box_rows rows of one head, same swizzle: rows and columns
// of a box that a head does not have are left out of a store
static bool make_tmap_heads(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t heads, uint64_t ld, uint64_t hoff,
                            uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("tensor map: cuTensorMapEncodeTiled entry point unavailable"); return false; }
    if ((((uintptr_t)base) & 15) || ((ld * 2) & 15) || ((hoff * 2) & 15)) { set_error("tensor map: base/pitch not 16-byte aligned"); return false; }
    cuuint64_t dims[3] = {cols, rows, heads};
    cuuint64_t strides[2] = {ld * 2, hoff * 2};
    cuuint32_t box[3] = {64, box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("tensor map: encode failed (%d)", (int)r); return false; }
    return true;
}

// A row-major matrix [rows, cols], cols a multiple of 64, as [cols / 64][rows][64]: boxes of `blocks` K blocks, each box_rows rows of 128 bytes,
// land one behind the other.  (The extents are exactly the matrix's.)
static bool make_tmap_kblocks(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t blocks) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("tensor map: cuTensorMapEncodeTiled entry point unavailable"); return false; }
    if ((((uintptr_t)base) & 15) || ((ld * 2) & 15) || (cols % 64)) { set_error("tensor map: base/pitch not 16-byte aligned"); return false; }
    cuuint64_t dims[3] = {64, rows, cols / 64};
    cuuint64_t strides[2] = {ld * 2, 128};
    cuuint32_t box[3] = {64, box_rows, blocks};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("tensor map: encode failed (%d)", (int)r); return false; }
    return true;
}

// What a map is of: rows x cols; `parts` heads, hoff elements apart; rows x cols in boxes of `parts` K blocks.
enum TmapKind { TMAP_MATRIX, TMAP_HEADS, TMAP_KBLOCKS };
struct TmapKey {
    TmapKind kind; const void* p; uint64_t rows, cols, ld; uint32_t box; uint64_t parts, hoff;
    bool operator<(const TmapKey& o) const {
        return std::tie(kind, p, rows, cols, ld, box, parts, hoff) < std::tie(o.kind, o.p, o.rows, o.cols, o.ld, o.box, o.parts, o.hoff);
    }
};
// Encoding a tensor map costs a few microseconds on the host; weights and
// workspace buffers repeat every block and step, so cache by (ptr, shape).
// The map is copied out under the lock: the cache may be emptied by a later
// call (or another thread) while the caller still holds its copy.
static bool cached(CUtensorMap* out, const TmapKey& k) {
    static std::map<TmapKey, CUtensorMap> cache;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(k);
    if (it != cache.end()) { *out = it->second; return true; }
    if (cache.size() > 8192) cache.clear();
    const bool made = k.kind == TMAP_MATRIX ? make_tmap_bf16(out, k.p, k.rows, k.cols, k.ld, k.box)
                      : k.kind == TMAP_HEADS ? make_tmap_heads(out, k.p, k.cols, k.rows, k.parts, k.ld, k.hoff, k.box)
                                             : make_tmap_kblocks(out, k.p, k.rows, k.cols, k.ld, k.box, (uint32_t)k.parts);
    if (!made) return false;
    cache.emplace(k, *out);
    return true;
}
bool cached_tmap(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    return cached(out, TmapKey{TMAP_MATRIX, base, rows, cols, ld, box_rows, 0, 0});
}
static bool cached_tmap_kblocks(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t blocks) {
    return cached(out, TmapKey{TMAP_KBLOCKS, base, rows, cols, ld, box_rows, blocks, 0});
}
bool cached_tmap_heads(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t heads, uint64_t ld, uint64_t hoff,
                       uint32_t box_rows) {
    return cached(out, TmapKey{TMAP_HEADS, base, rows, cols, ld, box_rows, heads, hoff});
}

// cudaFuncSetAttribute is per device: remember, per kernel instantiation, on which devices it was done.
bool func_attr_once(std::atomic<uint64_t>& done, const void* func, int smem_bytes, const char* what) {
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return true;
    cudaError_t e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("%s: smem attribute: %s", what, cudaGetErrorString(e));
        return false;
    }
    done.fetch_or(bit, std::memory_order_release);
    return true;
}

// 0: single CTAs only, no cluster is launched; else CTA pairs where tile_form() finds them the better form and, for callers
// that allow it, a long K of few tiles in parts (the default)
static int g_pair_mode = -1;
void gemm_pair_mode(int mode) { g_pair_mode = mode; }
static bool pair_wanted() {
    if (g_pair_mode < 0) {
        const char* e = getenv("O1_GEMM_PAIR");
        g_pair_mode = (e && e[0] == '0') ? 0 : 1;
    }
    return g_pair_mode != 0;
}

// Activations of less than 128 KB: loads through a tensor map of so few bytes slow down with the number of CTAs that make them
// (4096 x 4096 as 128 tiles: 15 rows 27.9 us, 16 rows 12.3, wherever the rows lie; the cause is not known).
static bool small_rows(long M, long K) { return M * K * 2 < (128l << 10); }
// A launch of some hundred us counts as one of many rows (see OVERLAP_ROWS): 24576 x 4096 at 3100 rows 501 us overlapped,
// 485 without.  So does one whose loads are slow anyway, if its K is long: 12 x 12288 x 4096 38.0 / 37.1, 10 x 4096 x 4096
// 23.4 / 22.5; but 12 x 8192 x 2048 18.3 / 20.0.
static long overlap_rows(const GemmArgs& g) {
    return (double)g.M * g.N * g.K > 1.5e11 || (small_rows(g.M, g.K) && g.K >= 4096) ? OVERLAP_ROWS + 1 : g.M;
}

// A persistent grid must be co-resident: as many pairs as the device can hold at once (a GPC with an odd number of SMs leaves one
// without a partner), asked once per device.
// Every pair kernel takes more than half of an SM's shared memory (PAIR_ALONE), so that no two CTAs of pairs are ever on an SM, of
// one grid, of the next one in a chain or of another stream.  tcgen05.alloc of a pair needs a turn on both of its SMs (a CTA has it until it gives up its
// permit), and nothing in its definition orders two pairs that begin on the same two SMs: each might have the turn on one of them and
// wait for the other, without a limit.  A single CTA's allocation waits on its own SM only, for CTAs that do not wait for it.
static int pair_capacity(const void* kern, int threads, int smem) {
    static std::atomic<int> max_pairs[64];
    int dev = 0;
    cudaGetDevice(&dev);
    int pairs = max_pairs[dev & 63].load(std::memory_order_acquire);
    if (pairs > 0) return pairs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = sm_count() / 2; }
    if (n > sm_count() / 2) n = sm_count() / 2;
    max_pairs[dev & 63].store(n, std::memory_order_release);
    return n;
}

// gate | up: where at most half of the pairs have a tile in the last round, its tiles are taken as two halves of 64 gate and 64 up columns.
// A half takes some 0.6 of a tile's time (it loads 24 KB for each K block, the tile 32).  Whole tiles / with halves, 12288 columns of each, K =
// 4096, us: 256 rows (1.3 rounds) 71 / 55, 1024 rows 174 / 162, 1280 rows 211 / 195 (170 / 161 at the full clock), 1792 rows 285 / 270, 2048 rows
// 307 / 293, 3500 rows 549 / 532, 4352 rows 650 / 642; last rounds that more than half of the pairs have stay whole (two rounds of halves).
// A block that runs at the power cap gains less (1280 rows: nothing beyond 1 %).
template <int EPI>
static bool launch_tc_pair(const CUtensorMap* tA, const CUtensorMap* tB, const CUtensorMap* tB2, GemmArgs& g,
                           cudaStream_t st, const CUtensorMap* tB3, const CUtensorMap* tB4 = nullptr) {
    using Cfg = GemmCfg<256, true>;
    static_assert(Cfg::SMEM_BYTES >= PAIR_ALONE, "see pair_capacity()");
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_tc_kernel<EPI, 256, true>;
    if (!func_attr_once(attr_done, (const void*)kern, Cfg::SMEM_BYTES, "gemm (pair)")) return false;
    const int tiles = ((g.num_m + 1) / 2) * g.num_n;
    int pairs = pair_capacity((const void*)kern, GEMM_THREADS, Cfg::SMEM_BYTES);
    g.halves_from = tiles;
    if (EPI == EPI_SWIGLU && tiles > pairs && 2 * (tiles % pairs) <= pairs) g.halves_from = tiles - tiles % pairs;
    if (pairs > tiles) pairs = tiles;
    prof_before(EPI == EPI_QKV ? (int)EPI_STORE : EPI, 2.0 * g.M * (double)g.N * g.K * (EPI == EPI_SWIGLU ? 2.0 : 1.0), st);
    cudaError_t e = launch_chained(kern, dim3(2 * pairs), dim3(GEMM_THREADS), Cfg::SMEM_BYTES, st, 2, overlap_rows(g), *tA, *tB, *tB2,
                                   tB3 ? *tB3 : *tB2, tB4 ? *tB4 : *tB2, g);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (pair): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

template <int EPI>
static bool launch_pair_fit(const CUtensorMap* tA, const void* w, GemmArgs& g, int bn, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_pair_fit_kernel<EPI>;
    constexpr int SMEM = EPI == EPI_VROPE ? PFV_SMEM : PF_SMEM, ROOM = EPI == EPI_VROPE ? PFV_ROOM : PF_STAGE_ROOM;
    static_assert(SMEM >= PAIR_ALONE, "see pair_capacity()");
    if (!func_attr_once(attr_done, (const void*)kern, SMEM, "gemm (pair, fitted)")) return false;
    CUtensorMap mB;
    if (!cached_tmap(&mB, w, g.N, g.K, g.K, bn / 2)) return false;
    g.num_n = (g.N + bn - 1) / bn;
    int stages = ROOM / ((BM + bn / 2) * BK * 2);
    if (stages > PF_MAX_STAGES) stages = PF_MAX_STAGES;
    const int tiles = (g.num_m + 1) / 2 * g.num_n;
    int pairs = pair_capacity((const void*)kern, GEMM_THREADS, SMEM);
    if (pairs > tiles) pairs = tiles;
    prof_before(EPI == EPI_BIAS_GELU || EPI == EPI_VROPE ? (int)EPI_BIAS : (EPI == EPI_BIAS_RESID || EPI == EPI_GATE_RESID ? (int)EPI_RESID : EPI),
                2.0 * g.M * (double)g.N * g.K, st);
    cudaError_t e = launch_chained(kern, dim3(2 * pairs), dim3(GEMM_THREADS), SMEM, st, 2, overlap_rows(g), *tA, mB, g, bn, stages);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (pair, fitted): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

// x [M, K] (row pitch ldx) against the weights of `num_n` tiles: gate and up, or q, k and v
template <int EPI>
static bool launch_rows(const void* x, int ldx, const CUtensorMap* mW, const CUtensorMap* mW2, const CUtensorMap* mW3, GemmArgs& g, int bn,
                        cudaStream_t st) {
    static_assert(RW_SMEM >= PAIR_ALONE, "see pair_capacity()");
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_rows_kernel<EPI>;
    if (!func_attr_once(attr_done, (const void*)kern, RW_SMEM, "gemm (pair, rows)")) return false;
    CUtensorMap mX;
    if (!cached_tmap(&mX, x, g.M, g.K, ldx, bn / 2)) return false;
    g.num_m = (g.M + bn - 1) / bn;
    g.num_n = g.N / (EPI == EPI_SWIGLU ? 128 : 256);
    g.group_m = (g.group_m * BM + bn - 1) / bn;
    int stages = PF_STAGE_ROOM / ((BM + bn / 2) * BK * 2);
    if (stages > PF_MAX_STAGES) stages = PF_MAX_STAGES;
    const int tiles = g.num_m * g.num_n;
    int pairs = pair_capacity((const void*)kern, GEMM_THREADS, RW_SMEM);
    if (pairs > tiles) pairs = tiles;
    prof_before(EPI == EPI_QKV ? (int)EPI_STORE : EPI, 2.0 * g.M * (double)g.N * g.K * (EPI == EPI_SWIGLU ? 2.0 : 1.0), st);
    cudaError_t e = launch_chained(kern, dim3(2 * pairs), dim3(GEMM_THREADS), RW_SMEM, st, 2, overlap_rows(g), mX, *mW, *mW2, *mW3, g, bn, stages);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (pair, rows): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

// CTA pairs of the GEMM kernel the current device can hold at once (what the pair form's grid is clamped to)
int gemm_pair_capacity() {
    using Cfg = GemmCfg<256, true>;
    auto kern = gemm_tc_kernel<EPI_STORE, 256, true>;
    if (cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sm_count() / 2));
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); return -1; }
    return n;
}

// Which persistent form takes the fewest (rounds of tiles) x (time of a K block): one CTA per 128 x 128 or 128 x 256 tile,
// or a pair of CTAs per 256 x 256 tile.  The sums are the same in all of them.  A round of tiles with K = 4096 takes 15.6,
// 29 (4096 columns) to 33 (24576) and 25 us; measured at 4096 columns: 592 rows 33.3 / 31.6 / 30.5 us, 1280 rows 51.4 / 60.3 / 54.5, 2242
// rows 73.7 / 64.7 / 59.2, 8192 rows 255 / 197 / 197, and at 6144 columns (q | k | v) 296 rows 24.6 / 38.6 / 40.1, 1280 rows 66.4 / 60.5 / 53.0.  Gate | up as
// pairs instead of one CTA per 128 x 256 tile: 1280 rows 213 / 186 us, a block of 16640 rows 9.24 / 9.02 ms.
enum TileForm { TILE_128, TILE_256, TILE_PAIR };
static constexpr int TILE_COST[3] = {31, 66, 50};
// Those times are the main loop's; below K = 2048 the epilogue counts as much, and finer tiles are the safer choice until
// there are two full waves of wide ones.
static constexpr int LONG_K = 2048;
static TileForm tile_form(int num_m, int N, int K, bool wide_ok, bool pair_ok, long* units = nullptr /*cost by TILE_COST, K >= LONG_K*/) {
    const long sms = sm_count();
    if (!wide_ok) {
        if (units) *units = ((long)num_m * ((N + 127) / 128) + sms - 1) / sms * TILE_COST[TILE_128];
        return TILE_128;
    }
    if (K < LONG_K) {
        if ((long)num_m * (N / 256) < 2 * sms) return TILE_128;
        return pair_ok && pair_wanted() && (long)((num_m + 1) / 2) * (N / 256) >= sms ? TILE_PAIR : TILE_256;
    }
    auto cost = [&](TileForm f, long tiles, long at_once) { return (tiles + at_once - 1) / at_once * TILE_COST[f]; };
    const long c128 = cost(TILE_128, (long)num_m * (N / 128), sms), c256 = cost(TILE_256, (long)num_m * (N / 256), sms);
    const long cp = pair_ok && pair_wanted() ? cost(TILE_PAIR, (long)((num_m + 1) / 2) * (N / 256), sms / 2) : c256 + 1;
    if (units) *units = cp <= c256 && cp <= c128 ? cp : (c256 <= c128 ? c256 : c128);
    if (cp <= c256 && cp <= c128) return TILE_PAIR;
    return c256 <= c128 ? TILE_256 : TILE_128;
}

// Below K = 2048, the plain, bias and residual families: two rounds of pairs against four of 128 columns.  128 columns / pairs:
// 2048 x 4096 x 1024 21.3 / 18.5, with residual 24.4 / 21.4, 1000 x 8192 x 1024 24.6 / 21.7, 4096 x 2048 x 1536 32.5 / 28.0,
// 2242 x 4096 x 512 12.6 / 11.7, but K = 256 9.8 / 9.9; three rounds against four 1100 x 8192 x 1024 24.9 / 27.4, one against two 1000 x
// 4096 x 1024 11.4 / 11.4, K = 512 7.8 / 8.5.  (Their epilogue is short; q | k | v with K = 1024 would be slower, 1300 rows 23.0 / 24.7.)
static bool two_rounds_of_pairs(int num_m, int N, int K) {
    const long sms = sm_count(), pair_tiles = (long)((num_m + 1) / 2) * (N / 256);
    return K >= 512 && K < LONG_K && pair_tiles <= sms / 2 * 2 && (long)num_m * (N / 128) > 3 * sms;
}

// The fitted width for the bias and residual families, or 0 where no width beats the other forms.  A round of bn columns
// takes about 31 (1/4 + 3/4 bn/128) of TILE_COST's units: the copies of A and the trips through the barriers do not grow
// with the tile (nor do they shrink: widths below 128 gain nothing).
static int fit_width(int num_m, int N, int K, double* units) {
    if (K < LONG_K) return 0;
    const long sms = sm_count();
    auto cost = [&](TileForm f, long tiles, long at_once) { return (tiles + at_once - 1) / at_once * TILE_COST[f] * 512; };
    long best = cost(TILE_128, (long)num_m * (N / 128), sms);
    if ((N % 256) == 0) {
        const long c256 = cost(TILE_256, (long)num_m * (N / 256), sms), cp = cost(TILE_PAIR, (long)((num_m + 1) / 2) * (N / 256), sms / 2);
        best = c256 < best ? c256 : best;
        if (pair_wanted() && cp < best) best = cp;
    }
    best -= best / 16;       // (only for a gain that shows)
    int width = 0;
    for (int bn = 144; bn <= 192; bn += 16) {
        const long tiles = (long)num_m * ((N + bn - 1) / bn), c = (tiles + sms - 1) / sms * TILE_COST[TILE_128] * (128 + 3 * bn);
        if (c < best) { best = c; width = bn; *units = c / 512.0; }
    }
    return width;
}
// The width of a pair tile for the linears of long K, or 0 where the other forms' cost `best` (TILE_COST's units) is as good.  A
// round of bn columns takes 0.6 + 0.1 bn us at K = 4096, two of those units per us.  Other forms against this one at 4096 x 4096:
// 300 rows 19.0 / 16.8 us (128 columns), 768 rows 25.8 / 23.2 (176), 1280 rows 37.6 / 35.5 (144), 2600 rows 85 / 76 (160), and at
// 4096 x 12288 62 / 47, 70 / 58, 124 / 101, 265 / 236; 3072 x 4096 at 1000 rows 30.5 / 22.4 (176); where the rule leaves the others,
// 592 rows 21.1 / 22.0, 2242 rows 60.7 / 62.5, 4352 rows 112.7 / 120.
// Epilogues that also have the 256 x 256 pair form go up to 192 columns, the others (GELU, bias or gate + residual) up to 256.
// Form without a pair width / with it, in turn: plain store 592 x 4096 x 4096 29.5 / 21.5 (176), 3000 x 1024 x 3072 23.5 / 17.5; GELU at
// 4096 x 4096: 592 rows 34 / 24.0 (176), 1600 rows 53 / 47.6 (208), 3000 rows 96 / 80.6 (176), 8192 rows 222 / 193 (256; with 128
// columns 230); K in no whole blocks: 300 x 4096 x 3080 22.4 / 18.7 (128), 700 x 4096 x 3080 + residual 29.8 / 24.3 (176),
// 1280 x 4096 x 3080 63.8 / 37.2 (144).  From K = 2048 on pairs would be ahead too (592 x 4096 x 2560 20.2 / 15.1, 1280 x 2048 x 2048
// + residual 16.1 / 13.0), but there the one-CTA widths and the narrow tiles are the rule, as the 128-column tiles are
// for a ragged K or N where 256 does not divide N: only the vision tower's linears, which ask for it (GEMM_TOWER), take pairs.
static constexpr int PAIR_FIT_K = 3072;
static int pair_fit_width(int num_m, int N, double best, int lo, int hi) {
    const long pairs = sm_count() / 2;
    int width = 0;
    best *= 15.0 / 16;       // (only for a gain that shows)
    for (int bn = lo; bn <= hi; bn += 16) {
        const long tiles = (long)((num_m + 1) / 2) * ((N + bn - 1) / bn);
        const double c = (double)((tiles + pairs - 1) / pairs) * (1.2 + 0.2 * bn);
        if (c < best) { best = c; width = bn; }
    }
    return width;
}
// The number of tokens of a tile of gemm_rows_kernel, or 0 where the other forms' cost `best` (TILE_COST's units) is as good.  tiles_w:
// tiles of 256 weight rows.  A round takes as long as one of pair_fit_width()'s columns.  The other forms / this one, us, gate | up with
// SwiGLU (12288 columns of each, K = 4096): 129 rows 61 / 46, 256 rows 73 / 55, 296 rows 75 / 68, 513 rows 117 / 85, 592 rows 120 / 100, 785
// rows 171 / 131, 1030 rows 197 / 157, 1600 rows 273 / 239, 2070 rows 337 / 299; q | k | v of 4096 + 2 x 1024 columns: 64 rows
// 29.6 / 23.5, 256 rows 21.4 / 18.7, 392 rows 34.3 / 23.4, 592 rows 36.3 / 31.3, 925 rows 58.7 / 42.6, 1280 rows 62.9 / 56.3, 1690 rows
// 81.7 / 68.2, 2450 rows 110 / 97, 3970 rows 166 / 147.  Up to 128 rows gate | up is read from memory at 5 TB/s either way (77 rows 40.6
// / 40.5, 100 rows 41.1 / 45.5): swiglu_rows_width().  Whole 256s, and what is near them, stay with the others (2242, 4352 rows).
static int rows_width(int M, int tiles_w, int K, double best) {
    if (K < LONG_K || !pair_wanted()) return 0;
    const long pairs = sm_count() / 2;
    int width = 0;
    best *= 15.0 / 16;       // (only for a gain that shows)
    for (int t = (M + 255) / 256; t <= (M + 255) / 256 + 3; ++t) {
        const int bn = ((M + t - 1) / t + 15) / 16 * 16;
        if (bn < 64) break;
        const double c = (double)((t * tiles_w + pairs - 1) / pairs) * (1.2 + 0.2 * bn);
        if (c < best) { best = c; width = bn; }
    }
    return width;
}
template <int EPI>
static bool launch_fit(const CUtensorMap* tA, const void* w, GemmArgs& g, int bn, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_fit_kernel<EPI>;
    if (!func_attr_once(attr_done, (const void*)kern, FIT_SMEM, "gemm (fitted)")) return false;
    CUtensorMap mB;
    if (!cached_tmap(&mB, w, g.N, g.K, g.K, bn)) return false;
    g.num_n = (g.N + bn - 1) / bn;
    int stages = FIT_ROOM / ((BM + bn) * BK * 2);
    if (stages > FIT_MAX_STAGES) stages = FIT_MAX_STAGES;
    const int tiles = g.num_m * g.num_n, grid = tiles < sm_count() ? tiles : sm_count();
    prof_before(EPI, 2.0 * g.M * (double)g.N * g.K, st);
    cudaError_t e = launch_chained(kern, dim3(grid), dim3(GEMM_THREADS), FIT_SMEM, st, 1, overlap_rows(g), *tA, mB, g, bn, stages);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (fitted): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

template <int EPI, int BN>
static bool launch_tc(const CUtensorMap* tA, const CUtensorMap* tB, const CUtensorMap* tB2,
                      GemmArgs& g, cudaStream_t st, const CUtensorMap* tB3 = nullptr) {
    using Cfg = GemmCfg<BN>;
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_tc_kernel<EPI, BN, false>;
    if (!func_attr_once(attr_done, (const void*)kern, Cfg::SMEM_BYTES, "gemm")) return false;
    const int tiles = g.num_m * g.num_n;
    int grid = sm_count();
    if (grid > tiles) grid = tiles;
    prof_before((EPI == EPI_QKNORM || EPI == EPI_QKV) ? (int)EPI_STORE : (EPI == EPI_BIAS_GELU ? (int)EPI_BIAS : ((EPI == EPI_BIAS_RESID || EPI == EPI_GATE_RESID) ? (int)EPI_RESID : EPI)), 2.0 * g.M * (double)g.N * g.K * (EPI == EPI_SWIGLU ? 2.0 : 1.0), st);
    cudaError_t e = launch_chained(kern, dim3(grid), dim3(GEMM_THREADS), Cfg::SMEM_BYTES, st, 1, overlap_rows(g), *tA, *tB, *tB2,
                                   tB3 ? *tB3 : *tB2, *tB2, g);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm: launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

// Which form for few tiles a problem takes: tile width and parts of K; width 0: the persistent kernel is the
// better one.  Times in us, persistent kernel with 128-column tiles against this one:
//  * 32 columns where that makes at most two CTAs per SM: 77 x 4096 x 4096 19.4 / 12.7, 520 x 1152 x 1152 11.1 / 8.7,
//    130 x 4608 x 4608 23.9 / 20.0; beyond, the activations are read too often: 296 x 4096 x 4096 19.6 / 31.6
//  * 96 columns where the wider tiles need a second round and these do not, and K is short: 2916 x 1152 x 1152 16.0 / 12.5,
//    520 x 4304 x 1152 16.4 / 14.1; 593 x 4096 x 12288 86 / 84, where CTA pairs take 72
//  * a long K in parts (bn 128, ks parts), for callers that allow that order of the sum: what once went over the CTAs of a cluster, where
//    even narrow tiles left a long main loop (520 x 1152 x 4304 23.5 / 18.7, five CTAs; 96 x 1152 x 4304 22.2 / 12.9, six).  Narrow pair
//    tiles take it now with an accumulator for each part (13.5, 10.4), and take half the time whole or in parts; the parts stay, for the
//    tower's bits, and because shorter chains of sums misround less (7,883 of 13.6 M results of the tower's linears against 37,310).
// But few rows of a long K (small_rows()) are read by fewer SMs in wider tiles: by at most half of them from K = 2048 on, by no
// more than all from K = 512 on.  Narrow / 128 columns / before there were narrow ones: 10 x 4096 x 4096 27.4 / 22.5 / 24.6,
// 10 x 6144 x 4096 52.0 / 26.5 / 26.3, 12 x 8192 x 2048 28.7 / 18.3 / 19.7, 33 x 8192 x 1024 13.7 / 9.8 / 12.3, 12 x 8192 x 512
// 9.5 / 6.5 / 8.5, 96 columns at 20 x 24576 x 2048 37.1 / 26.0 / 32.7; but 10 x 2304 x 4096 (72 tiles) 20.5 / 18.6 / 24.6,
// 10 x 1024 x 4096 15.0 / 17.3 / 24.6, 33 x 4096 x 256 4.2 / 4.9 / 7.8, and the tower of 36 patches (135 tiles, K = 1152) 1.78
// / 1.93 / 3.15 ms.  K of no whole 64 columns, whose rows lie across the memory's lines, gains nothing from two CTAs per SM
// (640 x 1152 x 4304 27.0 / 22.5 / 26.7) except where a residual is added (the tower of 832 patches 2.66 / 2.70 ms).
struct SplitPlan { int bn, ks; };
static constexpr int MAX_SPLIT = 6;      // (accumulators of 64 columns at most: 384 of tensor memory's 512)
static SplitPlan split_plan(int M, int N, int K, bool may_split, bool resid) {
    const int sms = sm_count(), kblocks = (K + BK - 1) / BK;
    const long num_m = (M + BM - 1) / BM;
    auto tiles = [&](int bn) { return num_m * ((N + bn - 1) / bn); };
    if (may_split && kblocks >= 32 && tiles(128) * 3 <= sms) {
        const long ks = sms * 8 / 5 / tiles(128);
        return {128, ks > MAX_SPLIT ? MAX_SPLIT : (int)ks};
    }
    const bool small_a = small_rows(M, K);
    long most = 2 * sms;
    if ((K % 64) != 0 && !resid) most = sms;
    if (small_a && K >= 512) most = K >= 2048 ? sms / 2 : sms;
    if (tiles(32) <= most) return {32, 1};
    if (K <= (small_a ? 1024 : 2048) && tiles(128) > sms && tiles(96) <= 2 * sms) return {96, 1};
    return {0, 0};
}

// Narrow tiles on CTA pairs: columns of a CTA, or 0 for the one-CTA forms; K from 256 on.  32 columns where that makes at most one CTA per
// SM, else 48 or 64 (two CTAs of 32 columns on an SM have half the room each for weights on their way).  One CTA per 32 columns / pairs,
// us: 77 x 4096 x 4096 13.2 / 10.1, 16 x 4096 x 4096 13.0 / 9.3, 128 x 4096 x 4096 13.4 / 11.0, 77 x 1024 x 4096 11.5 / 7.4, 300 x 1024 x 4096
// 11.9 / 8.7, 77 x 1024 x 3072 9.4 / 6.0, 16 x 4096 x 1024 8.5 / 4.8, 256 x 1152 x 1152 4.6 / 3.9;
// a short K of more than two row tiles only where 32 columns do not fit: 300 x 1152 x 1152 5.07 / 5.11, 512 x 1152 x 1152 5.26 / 5.61.  (A copy
// for each K block: 77 x 4096 x 4096 12.7, 77 x 1024 x 4096 11.4; stages of 128 rows: 11.2 and 7.8; eight K blocks to a copy and two stages
// 12.3 and 8.8, two and eight 11.7 and 9.7.)  Two CTAs of 32 columns on an SM / pairs of 48 or 64: 130 x 4096 x 4096 16.9 / 12.7, 256 x 4096 x
// 4096 18.3 / 14.3, 520 x 1024 x 4096 17.4 / 10.9, 300 x 3072 x 4096 17.3 / 13.2, 256 x 4608 x 4608 21.9 / 16.2, 520 x 1152 x 1152 6.8 / 5.4, 200 x
// 4096 x 1024 6.2 / 6.0.  K shared by the CTAs of a cluster / the parts' accumulators in one pair: 520 x 1152 x 4304 18.4 / 12.8, 160 x 1152 x
// 4304 17.6 / 11.0, 96 x 1152 x 4304 12.1 / 9.3, 128 x 4608 x 4608 19.3 / 12.3, 128 x 4096 x 4608 18.1 / 12.2, 300 x 1024 x 2112 14.4 / 7.5, 9 x 4096
// x 4104 23.5 / 12.4.  The 96-column form with 96 columns of a pair tile to a CTA (two CTAs per SM, five stages of one block): 520 x 4304 x 1152
// 11.9 / 11.5, x 512 8.5 / 8.9: left alone.
// A short K ends before the pair's set-up (two cluster barriers, and no other pair beside it) has paid: from eight K a row on, up to K = 1024 for 128
// rows and more, and from K = 384 on where the one-CTA tiles leave half of the SMs idle.  One CTA / pairs, 4096 columns: 16 rows K = 256 3.70
// / 3.54, 40 rows K = 384 4.11 / 3.81, 77 rows K = 256 3.05 / 3.70, K = 640 4.50 / 4.43, 128 rows K = 768 4.12 / 4.65, K = 1024 5.00 / 5.16 (3072 columns
// 4.81 / 4.51), 256 rows K = 512 4.25 / 4.56, K = 1024 6.28 / 5.97; 1152 columns: 128 rows K = 256 2.78 / 2.78, K = 384 3.10 / 2.97, K = 768 4.01 / 3.39.
static int fewpair_cols(int M, int N, int K, int parts) {
    if (!pair_wanted() || K < 256) return 0;
    const long num_m = (M + BM - 1) / BM;
    const bool idle = 2 * num_m * ((N + 31) / 32) <= sm_count();
    if (parts == 1 && K < 8 * (M < 128 ? M : 128) && !(idle && K >= 384)) return 0;
    for (int fc = 32; fc <= 64; fc += 16)
        if (2 * num_m * ((N + 2 * fc - 1) / (2 * fc)) <= sm_count()) return fc == 32 && num_m > 2 && K < LONG_K && parts == 1 ? 0 : fc;
    return 0;
}
static int swiglu_rows_width(int M, int N, int K) {
    long units = 0;
    tile_form((M + BM - 1) / BM, 2 * N, K, true, true, &units);
    return M <= BM || K < LONG_K ? 0 : rows_width(M, N / 128, K, (double)units);
}
static int simt_rows(int M, int N, int K);
// The form a GEMM takes.  plain: row-major output; wide_ok: 256-column tiles fit it.
GemmPlan gemm_plan(int M, int N, int K, int epi, int force_bn, bool plain, bool wide_ok, bool blocked_a) {
    if (!gemm_tc_supported(M, N, K, epi)) return {GEMM_ROWS, simt_rows(M, N, K), 1};
    const int num_m = (M + BM - 1) / BM;
    if (epi == EPI_SWIGLU) {     // (2N columns of gate and up; pairs of 256 x 256 or gemm_rows_kernel's of 256 x any)
        const int rows = force_bn <= 0 && !blocked_a ? swiglu_rows_width(M, N, K) : 0;
        const bool pair = force_bn <= 0 && (rows || tile_form(num_m, 2 * N, K, true, true) == TILE_PAIR);
        return {pair ? GEMM_PAIR : GEMM_TILE, 256, pair ? 2 : 1, rows};
    }
    const bool pair_ok = epi == EPI_STORE || epi == EPI_BIAS || epi == EPI_RESID;
    if (force_bn == 128) return {GEMM_TILE, 128, 1};
    if (force_bn == 256) {       // the pair form where that family has two rounds of its tiles
        const bool pair = pair_ok && pair_wanted() && ((num_m + 1) / 2) * (N / 256) >= sm_count();
        return {pair ? GEMM_PAIR : GEMM_TILE, 256, pair ? 2 : 1};
    }
    plain = plain && force_bn <= 0;
    const bool tower = force_bn == GEMM_TOWER;
    const bool resid = epi_has_resid(epi);
    const bool small = plain && (pair_ok || resid || epi == EPI_BIAS_GELU);
    if (small) {
        const SplitPlan p = split_plan(M, N, K, (tower || force_bn == GEMM_SPLIT_K) && pair_wanted(), resid);
        // the tower's long K (the MLP's second linear, the mergers): pair tiles of any width instead of narrow ones, from 257 rows on
        if (p.ks > 1 || (p.bn > 0 && !(tower && pair_wanted() && K >= LONG_K && num_m > 2)))
            return {GEMM_FEW, p.bn, p.ks, p.bn == 96 || blocked_a ? 0 : fewpair_cols(M, N, K, p.ks)};
        // (From 1025 rows on a K of 1024 and more too: the tower of 1200 / 3024 / 4096 patches 2800 / 5600 / 8100 -> 2700 / 5370 / 7820
        // us, but of 832 patches 2165 -> 2197.  Only where 256 does not divide N: with the 256-column forms to choose from, a
        // pair width loses as often as it gains, 1600 x 2304 x 1152 13.5 / 14.5, 1100 x 4096 x 1024 12.6 / 13.7, 4096 rows
        // 36.3 / 40.7, but 1280 rows 14.9 / 12.2.)
        if (tower && pair_wanted() && num_m > (K >= LONG_K ? 2 : 8) && (K >= LONG_K || (K >= 1024 && !wide_ok))) {
            long units = 0;
            tile_form(num_m, N, K, wide_ok, pair_ok, &units);
            const int width = pair_fit_width(num_m, N, p.bn > 0 ? 1e9 : (double)units, 96, 256);
            if (width) return {GEMM_FIT, width, 2};
        }
    }
    long form_units = 0;
    TileForm f = tile_form(num_m, N, K, wide_ok, pair_ok, &form_units);
    if (small && pair_ok && wide_ok && pair_wanted() && two_rounds_of_pairs(num_m, N, K)) f = TILE_PAIR;
    double units = (double)form_units;
    int width = 0;
    if (plain && (N % 128) == 0 && (epi == EPI_RESID || epi == EPI_BIAS)) width = fit_width(num_m, N, K, &units);
    if (small && !tower && K >= PAIR_FIT_K && (wide_ok || ((N % 128) == 0 && (K % BK) == 0)) && pair_wanted() && M > BM) {
        const int w = pair_fit_width(num_m, N, units, 128, pair_ok ? 192 : 256);
        if (w) return {w == 128 ? GEMM_TILE : GEMM_FIT, w, 2};
    }
    if (width) return {GEMM_FIT, width, 1};
    return {f == TILE_PAIR ? GEMM_PAIR : GEMM_TILE, f == TILE_128 ? 128 : 256, f == TILE_PAIR ? 2 : 1};
}

template <int EPI, int BN, int KPS = 1>
static bool launch_split_bn(const CUtensorMap* tA, const CUtensorMap* tB, GemmArgs& g, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    constexpr int SMEM = SplitCfg<BN, KPS>::SMEM;
    auto kern = gemm_split_kernel<EPI, BN, KPS>;
    if (!func_attr_once(attr_done, (const void*)kern, SMEM, "gemm (few tiles)")) return false;
    g.num_n = (g.N + BN - 1) / BN;
    g.prefetch = SK_PREFETCH;
    prof_before((EPI == EPI_BIAS_GELU || EPI == EPI_VROPE) ? (int)EPI_BIAS
                                                           : ((EPI == EPI_BIAS_RESID || EPI == EPI_GATE_RESID) ? (int)EPI_RESID : EPI),
                2.0 * g.M * (double)g.N * g.K, st);
    cudaError_t e = launch_chained(kern, dim3(g.num_m * g.num_n), dim3(SplitCfg<BN, KPS>::THREADS), SMEM, st, 1, g.M, *tA, *tB, g);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (few tiles): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

template <int EPI, bool PARTS>
static bool launch_few_pair(const void* x, int ldx, const void* w, GemmArgs& g, int fc, int parts, cudaStream_t st) {
    static std::atomic<uint64_t> attr_done{0};
    auto kern = gemm_few_pair_kernel<EPI, PARTS>;
    if (!func_attr_once(attr_done, (const void*)kern, FP_SMEM, "gemm (few tiles, pairs)")) return false;
    CUtensorMap mA, mB;
    const int ra = g.num_m > 1 ? BM / 2 : (g.M + 15) / 16 * 8;      // rows of a CTA: half of the tile's, in eights
    int stages = FP_ROOM / fp_stage_bytes(ra, fc);
    if (stages > FP_MAX_STAGES) stages = FP_MAX_STAGES;
    // no more stages than the K blocks take: a short K leaves room for the next kernel's CTAs, but not for another one of this grid
    const int copies = (g.K / BK + FP_KPS - 1) / FP_KPS + (g.K % BK != 0);
    if (stages > copies) stages = copies;
    int smem = stages * fp_stage_bytes(ra, fc) + 1024 /*align*/ + 256 /*barriers*/;
    if (smem < PAIR_ALONE) smem = PAIR_ALONE;
    const int kw = g.K / BK * BK;
    if (!cached_tmap_kblocks(&mA, x, g.M, kw, ldx, ra, FP_KPS) || !cached_tmap_kblocks(&mB, w, g.N, kw, g.K, fc, FP_KPS)) return false;
    CUtensorMap mA2 = mA, mB2 = mB;
    if (kw != g.K && (!cached_tmap(&mA2, x, g.M, g.K, ldx, ra) || !cached_tmap(&mB2, w, g.N, g.K, g.K, fc))) return false;
    g.num_n = (g.N + 2 * fc - 1) / (2 * fc);
    g.prefetch = SK_PREFETCH;
    prof_before(EPI == EPI_BIAS_GELU ? (int)EPI_BIAS : (EPI == EPI_BIAS_RESID || EPI == EPI_GATE_RESID ? (int)EPI_RESID : EPI),
                2.0 * g.M * (double)g.N * g.K, st);
    cudaError_t e = launch_chained(kern, dim3(2 * g.num_m * g.num_n), dim3(fc > 32 ? GEMM_THREADS : SK_THREADS), smem, st, 2, g.M, mA, mB, mA2, mB2, g, ra, fc, stages, parts);
    prof_after(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { set_error("gemm (few tiles, pairs): launch: %s", cudaGetErrorString(e)); return false; }
    return true;
}

template <int EPI>
static bool launch_split(const CUtensorMap* tA, const void* x, int ldx, const void* w, GemmArgs& g, const GemmPlan& p, cudaStream_t st) {
    if (p.pair) return p.ks > 1 ? launch_few_pair<EPI, true>(x, ldx, w, g, p.pair, p.ks, st) : launch_few_pair<EPI, false>(x, ldx, w, g, p.pair, 1, st);
    CUtensorMap mB;
    if (!cached_tmap(&mB, w, g.N, g.K, g.K, p.bn)) return false;
    if (p.bn == 96) return launch_split_bn<EPI, 96>(tA, &mB, g, st);
    if (p.bn == 32) return g.num_m * ((g.N + 31) / 32) <= sm_count() ? launch_split_bn<EPI, 32, 2>(tA, &mB, g, st) : launch_split_bn<EPI, 32>(tA, &mB, g, st);
    set_error("gemm (few tiles): no kernel for %d columns and %d parts of K", p.bn, p.ks);
    return false;
}

// Rows that share a warp of gemm_simt_kernel, which then reads a weight once for all of them; equal groups of at most four.
// us with a warp per row and column against shared rows (before launches overlapped, a warp per row):
//  * K up to 1024: a warp's work is short and what counts is the number of blocks.  4096 x 256: 5 rows 6.4 / 3.6 (6.2), 7 rows
//    8.6 / 4.4 (7.7); 12288 x 512: 2 rows 8.4 / 6.2 (8.2), 7 rows 24.4 / 12.9 (16.4); 4096 x 1024: 2 rows 4.8 / 4.5 (6.2)
//  * beyond, three rows and more where N alone has two waves of blocks: 12288 x 2048: 3 rows 16.9 / 15.9 (19.4), 4 rows
//    20.6 / 17.6 (22.7), 7 rows 31.5 / 28.7 (34.8); 24576 x 1536: 6 rows 48.7 / 37.1 (47.2)
//  * weights beyond L2, which every further row would fetch from memory again: 24576 x 4096: 4 rows 53.2 (117.9)
//  * otherwise a warp per row: a chain of loads per warp and too few warps to hide it cost more than reading the weights from
//    L2 again.  4096 x 4096: 2 rows 8.9 / 13.5 (10.3), 7 rows 19.5 / 23.0 (22.5); 12288 x 2048: 2 rows 13.4 / 14.8 (16.4)
static int simt_rows(int M, int N, int K) {
    const bool share = K <= 1024 || (M >= 3 && N >= 2 * 8 * 4 * sm_count()) || (size_t)N * K * 2 > (126u << 20);
    if (M == 1 || M > 65535 /* no more rows than the grid takes one by one */ || !share) return 1;
    const int groups = (M + 3) / 4;
    return (M + groups - 1) / groups;
}

bool gemm_tc_supported(int M, int N, int K, int epi) {
    // tiny M (timestep MLP, M = 1) is a GEMV: SIMT path.  K only has to keep the rows 16-byte aligned for TMA
    // (the last K block may be ragged: both operands are zero-filled beyond K).
    if (M < 8 || (K % 8) != 0) return false;
    // a ragged right edge (N % 128 != 0, e.g. the 4304-wide MLP of the vision tower) is covered by the plain,
    // bias and bias+GELU epilogues, in steps of eight columns
    if (epi == EPI_STORE || epi == EPI_BIAS || epi == EPI_BIAS_GELU) return (N % 8) == 0;
    return (N % 128) == 0;   // EPI_SWIGLU: N = ff columns of each of gate / up
}

// epi: see Epi.  For EPI_SWIGLU, w = gate weight, w2 = up weight, N = ff.
bool gemm_bf16(const void* x, const void* w, const void* w2, void* y, int M, int N, int K, int epi,
               const void* bias, const void* resid, float scale, int force_bn, cudaStream_t st) {
    return gemm_bf16_ld(x, K, w, w2, y, N, M, N, K, epi, bias, resid, N, scale, force_bn, st);
}

bool gemm_bf16_ld(const void* x, int ldx, const void* w, const void* w2, void* y, int ldy, int M,
                  int N, int K, int epi, const void* bias, const void* resid, int ldr, float scale,
                  int force_bn, cudaStream_t st) {
    return gemm_bf16_ex(x, ldx, w, w2, y, ldy, M, N, K, epi, bias, resid, ldr, scale, force_bn, 0, 0, 0, 0, st);
}

bool gemm_bf16_ex(const void* x, int ldx, const void* w, const void* w2, void* y, int ldy, int M, int N,
                  int K, int epi, const void* bias, const void* resid, int ldr, float scale, int force_bn,
                  int o_cb, long o_cb_stride, int a_kblk, int a_rows, cudaStream_t st, void* const* o_tab) {
    if (!x || !w || (!y && !o_tab) || M <= 0 || N <= 0 || K <= 0) { set_error("gemm: bad args"); return false; }
    if (o_tab && (!o_cb || N / o_cb > 8 || (epi != EPI_STORE && epi != EPI_QKNORM))) {
        set_error("gemm: an output table needs column blocks (at most 8) and the plain or per-head norm epilogue");
        return false;
    }
    if ((o_cb || a_kblk) && !gemm_tc_supported(M, N, K, epi)) {
        set_error("gemm: blocked operand layouts need a tensor-core shape");
        return false;
    }
    if (o_cb && ((o_cb % 128) != 0 || (N % o_cb) != 0 || epi == EPI_SWIGLU)) {
        set_error("gemm: bad output column block %d", o_cb);
        return false;
    }
    if (a_kblk && ((a_kblk % BK) != 0 || (K % a_kblk) != 0)) {
        set_error("gemm: bad input K block %d", a_kblk);
        return false;
    }
    if (!gemm_tc_supported(M, N, K, epi)) {
        if (epi != EPI_STORE && epi != EPI_BIAS) { set_error("gemm: shape unsupported for fused epilogue"); return false; }
        const uint16_t* b = (const uint16_t*)(epi == EPI_BIAS ? bias : nullptr);
        const int mr = simt_rows(M, N, K);
        auto kern = mr == 1 ? gemm_simt_kernel<1> : mr == 2 ? gemm_simt_kernel<2> : mr == 3 ? gemm_simt_kernel<3> : gemm_simt_kernel<4>;
        const cudaError_t e = launch_chained(kern, dim3((N + 3) / 4, (M + mr - 1) / mr), dim3(128), 0, st, 1, M, (const uint16_t*)x,
                                             (const uint16_t*)w, b, (uint16_t*)y, M, N, K, ldx, ldy);
        if (e != cudaSuccess) { set_error("gemm(simt): launch: %s", cudaGetErrorString(e)); return false; }
        return true;
    }
    if ((N % 128) != 0 && ((ldy % 8) != 0 || (((uintptr_t)y) & 15) || (bias && (((uintptr_t)bias) & 15)))) {
        set_error("gemm: a ragged N needs 16-byte aligned output rows and bias");
        return false;
    }
    if ((epi == EPI_BIAS_RESID || epi == EPI_GATE_RESID) && (!bias || !resid || (((uintptr_t)bias) & 15) || (((uintptr_t)resid) & 15) || (ldr % 8))) {
        set_error("gemm: the bias / gate + residual epilogues need both operands, 16-byte aligned");
        return false;
    }
    GemmArgs g = {};
    g.M = M; g.N = N; g.K = K;
    g.out = (uint16_t*)y; g.ldo = ldy;
    g.bias = (const uint16_t*)bias;
    g.resid = (const uint16_t*)resid; g.ldr = ldr;
    g.scale = scale;
    g.rope = g.rope_sin = nullptr;
    if (epi == EPI_QKNORM) {
        // resid carries the cos|sin table, bias the norm weight; every 128 output columns are one head
        if (!bias || !resid || (N % 128) != 0 || (o_cb && (o_cb % 128) != 0) || (((uintptr_t)bias) & 15) ||
            (((uintptr_t)resid) & 15)) {
            set_error("gemm: per-head norm epilogue needs norm weight, cos|sin table and whole heads");
            return false;
        }
        g.rope = (const float*)resid;
        g.resid = nullptr;
    }
    g.err = device_error_word();
    g.num_m = (M + BM - 1) / BM;
    // Row tiles are visited in groups whose activation slab (group_m x 128 rows x K) stays L2-resident
    // (about 48 MB of the 126 MB) while the weights stream past it.
    {
        long gm = (48l << 20) / ((long)BM * K * 2);
        g.group_m = (int)(gm < 4 ? 4 : (gm > 32 ? 32 : gm));
    }
    g.o_cb = o_cb; g.o_cb_stride = o_cb_stride;
    g.o_tab_n = 0;
    for (int i = 0; i < 8; ++i) g.o_tab[i] = nullptr;
    if (o_tab) {
        g.o_tab_n = N / o_cb;
        for (int i = 0; i < g.o_tab_n; ++i) {
            if (!o_tab[i] || (((uintptr_t)o_tab[i]) & 15)) { set_error("gemm: output table entry %d unusable", i); return false; }
            g.o_tab[i] = (uint16_t*)o_tab[i];
        }
    }
    g.a_kblk = a_kblk; g.a_rows = a_rows;
    g.seg_n[0] = g.seg_n[1] = 0;
    g.seg_norm[0] = g.seg_norm[1] = nullptr;
    g.seg_cb[0] = g.seg_cb[1] = g.seg_cb[2] = 0;
    for (int i = 0; i < 16; ++i) g.seg_tab[i] = nullptr;

    CUtensorMap mA, mB, mB2;
    if (!(a_kblk ? cached_tmap(&mA, x, (uint64_t)(K / a_kblk) * a_rows, a_kblk, ldx, 128)
                 : cached_tmap(&mA, x, M, K, ldx, 128)))
        return false;
    if (!cached_tmap(&mB, w, N, K, K, 128)) return false;
    if (epi == EPI_SWIGLU) { if (!cached_tmap(&mB2, w2, N, K, K, 128)) return false; }
    else mB2 = mB;
    const CUtensorMap *tA = &mA, *tB = &mB, *tB2 = &mB2;

    const bool wide_ok = (N % 256) == 0 && (!o_cb || (o_cb % 256) == 0);
    if (epi != EPI_SWIGLU && force_bn == 256 && !wide_ok) {
        set_error("gemm: BN=256 needs N (and the output column block) %% 256 == 0");
        return false;
    }
    const GemmPlan p = gemm_plan(M, N, K, epi, a_kblk && force_bn < 0 ? 0 : force_bn, !o_cb && !o_tab, wide_ok, a_kblk != 0);     // (K in parts: plain rows)
    if (epi == EPI_SWIGLU) {
        if (p.pair) {
            CUtensorMap mG, mU;
            if (!cached_tmap(&mG, w, N, K, K, 64) || !cached_tmap(&mU, w2, N, K, K, 64)) return false;
            return launch_rows<EPI_SWIGLU>(x, ldx, &mG, &mU, &mU, g, p.pair, st);
        }
        g.num_n = N / 128;
        if (p.form != GEMM_PAIR) return launch_tc<EPI_SWIGLU, 256>(tA, tB, tB2, g, st);
        CUtensorMap hG, hU;      // (of half tiles)
        if (!cached_tmap(&hG, w, N, K, K, 64) || !cached_tmap(&hU, w2, N, K, K, 64)) return false;
        return launch_tc_pair<EPI_SWIGLU>(tA, tB, tB2, g, st, &hG, &hU);
    }
    if (p.form == GEMM_FEW) switch (epi) {
        case EPI_STORE: return launch_split<EPI_STORE>(tA, x, ldx, w, g, p, st);
        case EPI_BIAS:  return launch_split<EPI_BIAS>(tA, x, ldx, w, g, p, st);
        case EPI_RESID: return launch_split<EPI_RESID>(tA, x, ldx, w, g, p, st);
        case EPI_BIAS_GELU: return launch_split<EPI_BIAS_GELU>(tA, x, ldx, w, g, p, st);
        case EPI_BIAS_RESID: return launch_split<EPI_BIAS_RESID>(tA, x, ldx, w, g, p, st);
        case EPI_GATE_RESID: return launch_split<EPI_GATE_RESID>(tA, x, ldx, w, g, p, st);
    }
    if (p.ks == 2 && (p.form == GEMM_FIT || p.form == GEMM_TILE)) switch (epi) {
        case EPI_STORE: return launch_pair_fit<EPI_STORE>(tA, w, g, p.bn, st);
        case EPI_BIAS:  return launch_pair_fit<EPI_BIAS>(tA, w, g, p.bn, st);
        case EPI_RESID: return launch_pair_fit<EPI_RESID>(tA, w, g, p.bn, st);
        case EPI_BIAS_GELU: return launch_pair_fit<EPI_BIAS_GELU>(tA, w, g, p.bn, st);
        case EPI_BIAS_RESID: return launch_pair_fit<EPI_BIAS_RESID>(tA, w, g, p.bn, st);
        case EPI_GATE_RESID: return launch_pair_fit<EPI_GATE_RESID>(tA, w, g, p.bn, st);
    }
    if (p.form == GEMM_FIT) return epi == EPI_RESID ? launch_fit<EPI_RESID>(tA, w, g, p.bn, st) : launch_fit<EPI_BIAS>(tA, w, g, p.bn, st);
    const int bn = p.bn;
    if (p.form == GEMM_PAIR) {
        g.num_n = N / 256;
        switch (epi) {
            case EPI_STORE: return launch_tc_pair<EPI_STORE>(tA, tB, tB2, g, st, nullptr);
            case EPI_BIAS:  return launch_tc_pair<EPI_BIAS>(tA, tB, tB2, g, st, nullptr);
            default:        return launch_tc_pair<EPI_RESID>(tA, tB, tB2, g, st, nullptr);
        }
    }
    g.num_n = (N + bn - 1) / bn;
    if (bn == 256) {
        switch (epi) {
            case EPI_STORE: return launch_tc<EPI_STORE, 256>(tA, tB, tB2, g, st);
            case EPI_BIAS:  return launch_tc<EPI_BIAS, 256>(tA, tB, tB2, g, st);
            case EPI_RESID: return launch_tc<EPI_RESID, 256>(tA, tB, tB2, g, st);
            case EPI_LORA:  return launch_tc<EPI_LORA, 256>(tA, tB, tB2, g, st);
            case EPI_QKNORM: return launch_tc<EPI_QKNORM, 256>(tA, tB, tB2, g, st);
            case EPI_BIAS_GELU: return launch_tc<EPI_BIAS_GELU, 256>(tA, tB, tB2, g, st);
            case EPI_BIAS_RESID: return launch_tc<EPI_BIAS_RESID, 256>(tA, tB, tB2, g, st);
            case EPI_GATE_RESID: return launch_tc<EPI_GATE_RESID, 256>(tA, tB, tB2, g, st);
        }
    } else {
        switch (epi) {
            case EPI_STORE: return launch_tc<EPI_STORE, 128>(tA, tB, tB2, g, st);
            case EPI_BIAS:  return launch_tc<EPI_BIAS, 128>(tA, tB, tB2, g, st);
            case EPI_RESID: return launch_tc<EPI_RESID, 128>(tA, tB, tB2, g, st);
            case EPI_LORA:  return launch_tc<EPI_LORA, 128>(tA, tB, tB2, g, st);
            case EPI_QKNORM: return launch_tc<EPI_QKNORM, 128>(tA, tB, tB2, g, st);
            case EPI_BIAS_GELU: return launch_tc<EPI_BIAS_GELU, 128>(tA, tB, tB2, g, st);
            case EPI_BIAS_RESID: return launch_tc<EPI_BIAS_RESID, 128>(tA, tB, tB2, g, st);
            case EPI_GATE_RESID: return launch_tc<EPI_GATE_RESID, 128>(tA, tB, tB2, g, st);
        }
    }
    set_error("gemm: unknown epilogue %d", epi);
    return false;
}

int gemm_qkv_rows(int M, int qc, int kc, int K) {
    const int N = qc + 2 * kc;
    if (N % 256) return 0;
    long units = 0;
    tile_form((M + BM - 1) / BM, N, K, (qc % 256) == 0 && (kc % 256) == 0, true, &units);
    return rows_width(M, N / 256, K, (double)units);
}

// q | k | v projections of one activation matrix as ONE launch: y[M, qc | kc | kc] (row pitch ldy) = x wq^T | x wk^T |
// x wv^T, the per-head RMSNorm + rotary applied to the q and k columns in the epilogue (norm weights q_norm / k_norm
// [128], cos|sin table cs [M,128] fp32).  Three launches of 14.05 + 3.5 + 3.5 waves of tiles (at 16640 rows) become
// one of 21.1; in the sharded forward the gain is larger (fewer rows per rank, the same three partial last waves).
// tq / tk / tv (all or none): per destination rank the base of that rank's q / k / v columns (block widths
// qc/P, kc/P, kc/P); rows then go to the tables instead of y.
bool gemm_qkv(const void* x, int ldx, const void* wq, const void* wk, const void* wv, void* y, int ldy, int M, int qc,
              int kc, int K, const void* q_norm, const void* k_norm, const float* cs, float eps, int n_dst,
              void* const* tq, void* const* tk, void* const* tv, cudaStream_t st) {
    const int N = qc + 2 * kc;
    const bool tabs = n_dst > 0;
    if (!x || !wq || !wk || !wv || (!y && !tabs) || !q_norm || !k_norm || !cs || M < 8 || (K % 8) != 0 || (qc % 128) != 0 ||
        (kc % 128) != 0 || qc <= 0 || kc <= 0 || ((((uintptr_t)q_norm) | ((uintptr_t)k_norm) | ((uintptr_t)cs)) & 15)) {
        set_error("gemm_qkv: bad args");
        return false;
    }
    if (tabs && (n_dst > 8 || !tq || !tk || !tv || (qc % n_dst) != 0 || (kc % n_dst) != 0 || ((qc / n_dst) % 128) != 0 ||
                 ((kc / n_dst) % 128) != 0)) {
        set_error("gemm_qkv: bad destination tables");
        return false;
    }
    GemmArgs g = {};
    g.M = M; g.N = N; g.K = K;
    g.out = (uint16_t*)y; g.ldo = ldy;
    g.bias = (const uint16_t*)q_norm;
    g.resid = nullptr; g.ldr = 0;
    g.rope = cs; g.rope_sin = nullptr;
    g.scale = eps;
    g.err = device_error_word();
    g.num_m = (M + BM - 1) / BM;
    {
        long gm = (48l << 20) / ((long)BM * K * 2);
        g.group_m = (int)(gm < 4 ? 4 : (gm > 32 ? 32 : gm));
    }
    g.o_cb = 0; g.o_cb_stride = 0;
    g.o_tab_n = tabs ? n_dst : 0;
    g.a_kblk = 0; g.a_rows = 0;
    g.seg_n[0] = qc; g.seg_n[1] = kc;
    g.seg_norm[0] = (const uint16_t*)q_norm; g.seg_norm[1] = (const uint16_t*)k_norm;
    g.seg_cb[0] = tabs ? qc / n_dst : 0; g.seg_cb[1] = g.seg_cb[2] = tabs ? kc / n_dst : 0;
    for (int i = 0; i < 8; ++i) g.o_tab[i] = nullptr;
    for (int i = 0; i < 16; ++i) g.seg_tab[i] = nullptr;
    for (int i = 0; i < (tabs ? n_dst : 0); ++i) {
        if (!tq[i] || !tk[i] || !tv[i] || ((((uintptr_t)tq[i]) | ((uintptr_t)tk[i]) | ((uintptr_t)tv[i])) & 15)) {
            set_error("gemm_qkv: destination table entry %d unusable", i);
            return false;
        }
        g.o_tab[i] = (uint16_t*)tq[i]; g.seg_tab[i] = (uint16_t*)tk[i]; g.seg_tab[8 + i] = (uint16_t*)tv[i];
    }
    CUtensorMap mA, mQ, mK, mV;
    if (!cached_tmap(&mA, x, M, K, ldx, 128) || !cached_tmap(&mQ, wq, qc, K, K, 128) ||
        !cached_tmap(&mK, wk, kc, K, K, 128) || !cached_tmap(&mV, wv, kc, K, K, 128))
        return false;
    // 256-wide tiles need every segment (and every destination block) to be a multiple of 256 columns
    bool wide = (qc % 256) == 0 && (kc % 256) == 0;
    if (tabs && (((qc / n_dst) % 256) != 0 || ((kc / n_dst) % 256) != 0)) wide = false;
    const int bn = !tabs && (ldy % 8) == 0 && (((uintptr_t)y) & 15) == 0 ? gemm_qkv_rows(M, qc, kc, K) : 0;
    if (bn) return launch_rows<EPI_QKV>(x, ldx, &mQ, &mK, &mV, g, bn, st);
    const TileForm form = tile_form(g.num_m, N, K, wide, true);
    g.num_n = N / (form == TILE_128 ? 128 : 256);
    if (form == TILE_PAIR) return launch_tc_pair<EPI_QKV>(&mA, &mQ, &mK, g, st, &mV);
    return form == TILE_256 ? launch_tc<EPI_QKV, 256>(&mA, &mQ, &mK, g, st, &mV) : launch_tc<EPI_QKV, 128>(&mA, &mQ, &mK, g, st, &mV);
}

bool gemm_vision_qkv(const void* x, const void* w, const void* b, void* y, int M, const float* cosd, const float* sind,
                     cudaStream_t st) {
    constexpr int K = 1152, N = 3456;
    if (!x || !w || !b || !y || !cosd || !sind || M < 8 ||
        ((((uintptr_t)b) | ((uintptr_t)y) | ((uintptr_t)cosd) | ((uintptr_t)sind)) & 15)) {
        set_error("gemm_vision_qkv: bad args");
        return false;
    }
    GemmArgs g = {};
    g.M = M; g.N = N; g.K = K;
    g.out = (uint16_t*)y; g.ldo = 3 * 16 * 128;
    g.bias = (const uint16_t*)b;
    g.rope = cosd; g.rope_sin = sind;
    g.num_m = (M + BM - 1) / BM;
    g.err = device_error_word();
    CUtensorMap mA, mB;
    if (!cached_tmap(&mA, x, M, K, K, 128)) return false;
    // One CTA per SM: two K blocks a stage, see SplitCfg (the tower at 520 patches 2155 -> 2058 us).  More tiles than that: CTA pairs, which
    // bring three quarters of the bytes into their SMs and have the next tile's products under their epilogue.  Two CTAs of one tile each on an SM /
    // pairs, us: 832 rows 15.2 / 14.1, 1600 rows 25.1 / 18.8, 3024 rows 32.5 / 26.9, 4096 rows 47.0 / 37.4, 8192 rows 94.5 / 70.9; below, one CTA
    // per SM / pairs: 128 rows 8.4 / 9.1, 520 rows 9.1 / 9.8, 768 rows 9.3 / 9.8.
    const bool one_each = g.num_m * (N / VQ_BN) <= sm_count();
    if (!one_each && pair_wanted()) {
        g.group_m = 32;
        return launch_pair_fit<EPI_VROPE>(&mA, w, g, VQ_BN, st);
    }
    if (!cached_tmap(&mB, w, N, K, K, VQ_BN)) return false;
    if (one_each) return launch_split_bn<EPI_VROPE, VQ_BN, 2>(&mA, &mB, g, st);
    return launch_split_bn<EPI_VROPE, VQ_BN>(&mA, &mB, g, st);
}

}  // namespace o1
