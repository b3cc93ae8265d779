// Load-time LoRA merge  W = bf16( f32(W) + s * up @ down ),  s = multiplier*alpha/rank
// (o1.c include/hd_lora.h:10-14, src/model/lora_merge.cu:26-109, where the
// delta is an FP32 cublasSgemm over row chunks followed by an add/cast pass).
//
// One persistent kernel merges up to 16 targets per launch.  What bounds it is HBM: every weight is read once and
// written once, 4 bytes, while the contraction over the rank is short.  So W streams through shared memory on TMA
// loads and stores, and the delta of a 128 x 128 tile is made on the way by the tensor core from the FP32 adapters.
// To keep FP32-grade products on bf16 operands each adapter value is split into three bf16 terms
// (a = a1 + a2 + a3, 24 mantissa bits) and all nine cross terms are summed; every bf16 x bf16 product is exact in the
// FP32 accumulator.  The terms are made inside the kernel, from L2, into the layouts the MMA reads (up rows K-major, down
// rows MN-major, so nothing is transposed): no staging buffer in memory, no allocation, no other launch.
#include "common.cuh"
#include "ptx.cuh"
#include "kernels.h"
#include "../../include/o1_b200.h"

namespace o1 {

static constexpr int LT = 128;                       // tile: 128 rows x 128 columns of W
static constexpr int LR = 64;                        // ranks per chunk
static constexpr int L_TERM_BYTES = LT * LR * 2;     // one bf16 term of an operand tile, one chunk: 16 KB
static constexpr int L_PANEL_BYTES = LT * 64 * 2;    // half a W tile (64 columns): 16 KB
static constexpr int L_GROUP = 16;                   // targets per launch
static constexpr int LORA_THREADS = 448;             // W stream warp, MMA warp, 8 splitter warps, 4 epilogue warps
// NCH chunks of ranks are held at once (one up to rank 64, else two; a higher rank takes several turns per tile): up
// terms, NB buffers of down terms, SLOTS panels of W.  With one chunk the two groups of four splitter warps take
// alternate tiles; with two each takes a chunk.
template <int NCH>
struct LoraCfg {
    static constexpr int NB = NCH == 1 ? 2 : 1, SLOTS = NCH == 1 ? 5 : 2;
    static constexpr int OP_BYTES = 3 * NCH * L_TERM_BYTES;
    static constexpr int SMEM = OP_BYTES * (1 + NB) + SLOTS * L_PANEL_BYTES + 1024 /*align*/ + 256 /*barriers*/;
};

struct LoraTarget {
    const float* up;        // [N, R]
    const float* down;      // [R, K]
    float scale;
    int N, K, R;
    int tiles_n;            // K / 128: tiles of a row block, walked one after the other (the up terms stay)
    int tile0;              // first tile of this target in the launch's list
    int vec;                // adapters can be read 16 bytes at a time
};
struct LoraArgs {
    CUtensorMap tm[L_GROUP];
    LoraTarget t[L_GROUP];
    int count, tiles;
    int* err;
    int* failed;            // host memory: set beside the error word, so that the waiting host need not copy that
};
__device__ __forceinline__ void lora_fail(const LoraArgs& g, int code) {
    atomicExch(g.err, code);
    *reinterpret_cast<volatile int*>(g.failed) = code;
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int32_t c0, int32_t c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
                 "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// eight FP32 values -> one 16-byte chunk per term, the terms `pitch` bytes apart
__device__ __forceinline__ void split8_store(const float (&f)[8], uint8_t* term0, uint32_t off, uint32_t pitch) {
    uint32_t h[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float a = f[2 * j], b = f[2 * j + 1];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const uint32_t p = pack_bf16x2(a, b);
            h[t][j] = p;
            a -= bf16lo(p);
            b -= bf16hi(p);
        }
    }
#pragma unroll
    for (int t = 0; t < 3; ++t)
        *reinterpret_cast<uint4*>(term0 + t * pitch + off) = make_uint4(h[t][0], h[t][1], h[t][2], h[t][3]);
}
__device__ __forceinline__ void lora_load8(const float* p, int n, bool vec, float (&f)[8]) {
    if (vec && n >= 8) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = j < n ? p[j] : 0.f;
    }
}

template <int NCH>
__global__ void __launch_bounds__(LORA_THREADS, 1) lora_merge_kernel(const __grid_constant__ LoraArgs g) {
    using Cfg = LoraCfg<NCH>;
    constexpr int NB = Cfg::NB, L_SLOTS = Cfg::SLOTS, LRC = NCH * LR;
    constexpr uint32_t PITCH = NCH * L_TERM_BYTES;        // from term to term; a term's chunks lie behind one another
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* a_s = smem;                                  // up: three terms, chunks of [128 rows][64 ranks], K-major
    uint8_t* b_s = a_s + Cfg::OP_BYTES;                   // down: NB x three terms, chunks of [64 ranks][2 x 64 columns]
    uint8_t* w_s = b_s + NB * Cfg::OP_BYTES;              // W panels [128 rows][64 columns]
    uint64_t* w_full = reinterpret_cast<uint64_t*>(w_s + L_SLOTS * L_PANEL_BYTES);
    uint64_t* w_done = w_full + L_SLOTS;                  // the panel holds merged weights
    uint64_t* u_full = w_done + L_SLOTS;                  // operand terms of a (tile, LRC ranks) unit, NB buffers
    uint64_t* u_done = u_full + 2;                        // the MMAs that read them are done
    uint64_t* t_full = u_done + 2;                        // accumulator of a tile, two buffers
    uint64_t* t_empty = t_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + 2);
    int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        *s_abort = error_word(g.err);
        if (*s_abort != 0) *reinterpret_cast<volatile int*>(g.failed) = *s_abort;
    }
    __syncthreads();
    if (*s_abort != 0) return;
    if (threadIdx.x == 0) {
        for (int s = 0; s < L_SLOTS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_done[s], 4); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&u_full[s], NCH == 1 ? 4 : 8);
            mbar_init(&u_done[s], 1);
            mbar_init(&t_full[s], 1);
            mbar_init(&t_empty[s], 4);
        }
        fence_mbar_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 2 * LT); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // this CTA's share of the list: consecutive tiles, mostly of one row block
    const int tile_lo = (int)((long)blockIdx.x * g.tiles / gridDim.x);
    const int tile_hi = (int)((long)(blockIdx.x + 1) * g.tiles / gridDim.x);
    int e = 0;
    while (e + 1 < g.count && g.t[e + 1].tile0 <= tile_lo) ++e;

    if (warp == 0) {
        // ------------------------------------------------------ W stream: panels in, merged panels out
        if (elect_one()) {
            const int panels = 2 * (tile_hi - tile_lo);
            // Where the next panel lies: the panels of a row block, the row blocks of a target, one after the other.  (With divisions for
            // each panel, and sizes read from the parameters, this thread was as busy as memory: the seven linears of a block, whole call,
            // 165.7 / 160.3 us at rank 4, 170.7 / 165.8 at 32, from 64 on, where the products count, the same.)
            struct Place { int e, c0, c1, N, K; } in, out;
            const int r0 = tile_lo - g.t[e].tile0;
            in = {e, r0 % g.t[e].tiles_n * LT, r0 / g.t[e].tiles_n * LT, g.t[e].N, g.t[e].K};
            out = in;
            auto next = [&](Place& p) {
                if ((p.c0 += 64) < p.K) return;
                p.c0 = 0;
                if ((p.c1 += LT) < p.N) return;
                p.c1 = 0;
                if (++p.e < g.count) { p.N = g.t[p.e].N; p.K = g.t[p.e].K; }
            };
            auto load = [&](int p) {
                const int s = p % L_SLOTS;
                mbar_expect_tx(&w_full[s], L_PANEL_BYTES);
                tma_load_2d(w_s + s * L_PANEL_BYTES, &g.tm[in.e], &w_full[s], in.c0, in.c1);
                next(in);
            };
            for (int p = 0; p < L_SLOTS && p < panels; ++p) load(p);
            for (int p = 0; p < panels; ++p) {
                const int s = p % L_SLOTS;
                if (!mbar_wait(&w_done[s], (p / L_SLOTS) & 1)) {
                    // give up, but not before the loads still under way have landed
                    lora_fail(g, 41);
                    for (int q = p; q < panels && q < p + L_SLOTS - (p ? 1 : 0); ++q) mbar_wait(&w_full[q % L_SLOTS], (q / L_SLOTS) & 1);
                    break;
                }
                tma_store_2d(&g.tm[out.e], w_s + s * L_PANEL_BYTES, out.c0, out.c1);
                next(out);
                // the slot of the store before this one is free once that store has read it
                if (p >= 1 && p - 1 + L_SLOTS < panels) {
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    load(p - 1 + L_SLOTS);
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = umma_idesc_bf16(128, 128, 0, 1);     // down is MN-major
            int u = 0, te = e;
            bool ok = true;
            for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
                const int i = tile - tile_lo, as = i & 1;
                while (te + 1 < g.count && g.t[te + 1].tile0 <= tile) ++te;
                const int R = g.t[te].R;
                if (!mbar_wait(&t_empty[as], ((i >> 1) & 1) ^ 1)) { lora_fail(g, 42); break; }
                tc_fence_after();
                const uint32_t d = tmem_base + as * LT;
                for (int r0 = 0; r0 < R; r0 += LRC, ++u) {
                    if (!mbar_wait(&u_full[u % NB], (u / NB) & 1)) { lora_fail(g, 43); ok = false; break; }
                    tc_fence_after();
                    const uint64_t ad = umma_desc_sw128(smem_u32(a_s), 16, 1024);
                    const uint64_t bd = umma_desc_sw128(smem_u32(b_s + (u % NB) * Cfg::OP_BYTES), LR * 128, 1024);
                    const int nr = R - r0 < LRC ? R - r0 : LRC;
#pragma unroll
                    for (int c = 0; c < 9; ++c)
                        for (int k = 0; k * 16 < nr; ++k)     // four steps of 16 ranks per chunk
                            umma_ss(d, ad + (uint64_t)(((c / 3) * PITCH + (k >> 2) * L_TERM_BYTES + (k & 3) * 32) >> 4),
                                    bd + (uint64_t)(((c % 3) * PITCH + (k >> 2) * L_TERM_BYTES + (k & 3) * 16 * 128) >> 4),
                                    idesc, (r0 | c | k) != 0);
                    umma_commit(&u_done[u % NB]);
                }
                if (!ok) break;
                umma_commit(&t_full[as]);
            }
        }
    } else if (warp < 10) {
        // ------------------------------------------------------ splitters: FP32 adapters -> bf16 terms
        const int tid = (threadIdx.x - 64) & 127, grp = (warp - 2) >> 2;
        int u = 0, te = e, a_block = -1;      // a_block: the row block of the current target whose up terms are held
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            while (te + 1 < g.count && g.t[te + 1].tile0 <= tile) { ++te; a_block = -1; }
            const LoraTarget& t = g.t[te];
            const int r = tile - t.tile0, row0 = (r / t.tiles_n) * LT, col0 = (r % t.tiles_n) * LT;
            for (int r0 = 0; r0 < t.R; r0 += LRC, ++u) {
                const bool new_a = row0 != a_block || t.R > LRC;
                a_block = row0;
                if (NCH == 1 && (u & 1) != grp) continue;      // the other group's unit
                // this group's ranks: rc .. rc + nr, zero up to the next multiple of 16
                const int rc = r0 + (NCH == 1 ? 0 : grp * LR);
                int nr = t.R - rc < LR ? t.R - rc : LR;
                nr = nr < 0 ? 0 : nr;
                const int ks16 = (nr + 15) & ~15;
                const uint32_t ch = NCH == 1 ? 0u : (uint32_t)grp * L_TERM_BYTES;
                // down rows, eight columns per thread: 16 threads per row
                float f[8][8];
                const int c8 = tid & 15;
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    const int rr = p * 8 + (tid >> 4);
                    if (rr < ks16) lora_load8(t.down + (size_t)(rc + rr) * t.K + col0 + c8 * 8, rr < nr ? 8 : 0, t.vec, f[p]);
                }
                // the buffer's previous unit has been consumed
                if (!mbar_wait(&u_done[u % NB], ((u / NB) & 1) ^ 1)) { lora_fail(g, 44); ok = false; }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                uint8_t* b0 = b_s + (u % NB) * Cfg::OP_BYTES + (c8 >> 3) * (LR * 128);
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                    const int rr = p * 8 + (tid >> 4);
                    if (rr < ks16) split8_store(f[p], b0, ch + (uint32_t)(rr * 128 + (((c8 & 7) ^ (rr & 7)) * 16)), PITCH);
                }
                if (new_a) {
                    // single buffer: the unit before this one must be through with the old terms
                    if (u > 0 && !mbar_wait(&u_done[(u - 1) % NB], ((u - 1) / NB) & 1)) { lora_fail(g, 45); ok = false; }
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const int k8 = tid & 7;
                    if (k8 * 8 < ks16) {
#pragma unroll
                        for (int p = 0; p < 8; ++p) {
                            const int rr = p * 16 + (tid >> 3);
                            int n = row0 + rr < t.N ? nr - k8 * 8 : 0;
                            n = n < 0 ? 0 : n;
                            lora_load8(t.up + (size_t)(row0 + rr) * t.R + rc + k8 * 8, n, t.vec && (t.R & 3) == 0, f[p]);
                        }
#pragma unroll
                        for (int p = 0; p < 8; ++p) {
                            const int rr = p * 16 + (tid >> 3);
                            split8_store(f[p], a_s, ch + (uint32_t)(rr * 128 + ((k8 ^ (rr & 7)) * 16)), PITCH);
                        }
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&u_full[u % NB]);
            }
        }
    } else {
        // ------------------------------------------------------ epilogue: W + scale * delta, in the W panels
        const int qd = warp & 3;                 // TMEM lane quadrant this warp may access
        const int row = qd * 32 + lane;
        int te = e;
        bool ok = true;
        for (int tile = tile_lo; tile < tile_hi && ok; ++tile) {
            const int i = tile - tile_lo, as = i & 1;
            while (te + 1 < g.count && g.t[te + 1].tile0 <= tile) ++te;
            const float scale = g.t[te].scale;
            ok = __all_sync(0xffffffffu, mbar_wait(&t_full[as], (i >> 1) & 1));
            if (!ok) { lora_fail(g, 46); break; }
            tc_fence_after();
            const uint32_t t_row = tmem_base + as * LT + ((uint32_t)(qd * 32) << 16);
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int p = 2 * i + h, s = p % L_SLOTS;
                ok = __all_sync(0xffffffffu, mbar_wait(&w_full[s], (p / L_SLOTS) & 1));
                if (!ok) { lora_fail(g, 47); break; }
                uint32_t r[2][32];
                tmem_ld32(t_row + h * 64, r[0]);
                tmem_ld32(t_row + h * 64 + 32, r[1]);
                tmem_ld_wait();
                uint8_t* wrow = w_s + s * L_PANEL_BYTES + row * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    uint4* q = reinterpret_cast<uint4*>(wrow + ((c ^ (row & 7)) * 16));
                    const uint4 o = *q;
                    const uint32_t* d = &r[c >> 2][(c & 3) * 8];
                    uint4 n;
                    n.x = pack_bf16x2(bf16lo(o.x) + scale * __uint_as_float(d[0]), bf16hi(o.x) + scale * __uint_as_float(d[1]));
                    n.y = pack_bf16x2(bf16lo(o.y) + scale * __uint_as_float(d[2]), bf16hi(o.y) + scale * __uint_as_float(d[3]));
                    n.z = pack_bf16x2(bf16lo(o.z) + scale * __uint_as_float(d[4]), bf16hi(o.z) + scale * __uint_as_float(d[5]));
                    n.w = pack_bf16x2(bf16lo(o.w) + scale * __uint_as_float(d[6]), bf16hi(o.w) + scale * __uint_as_float(d[7]));
                    *q = n;
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_done[s]);
            }
            if (!ok) break;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_empty[as]);
        }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 2 * LT);
}

// shapes the tensor-core tiles do not cover
__global__ void lora_simt_kernel(uint16_t* __restrict__ w, const float* __restrict__ up,
                                 const float* __restrict__ down, int N, int K, int R, float scale) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)N * K) return;
    const int k = (int)(i % K);
    const long n = i / K;
    float acc = 0.f;
    for (int r = 0; r < R; ++r) acc += up[n * R + r] * down[(long)r * K + k];
    w[i] = f32_to_bf16(bf16_to_f32(w[i]) + scale * acc);
}

// The targets collected for one launch.
struct LoraGroup {
    LoraArgs a;
    uintptr_t lo[L_GROUP], hi[L_GROUP];      // address ranges of their weights
    LoraGroup() { a.count = 0; a.tiles = 0; a.err = a.failed = nullptr; }
    // Targets of one launch are merged in no particular order, so a weight that is already in the group (a second
    // adapter for it) has to wait for the next launch: each adapter's result is rounded to bf16 before the next.
    bool clashes(uintptr_t l, uintptr_t h) const {
        for (int i = 0; i < a.count; ++i)
            if (l < hi[i] && lo[i] < h) return true;
        return false;
    }
    bool low_rank = true;                    // up to 64 all of them, or above 64 all of them
    bool launched = false;                   // by any launch of the call
    template <int NCH>
    bool launch_as(cudaStream_t st) {
        static std::atomic<uint64_t> attr_done{0};
        if (!func_attr_once(attr_done, (const void*)lora_merge_kernel<NCH>, LoraCfg<NCH>::SMEM, "lora")) return false;
        const int sms = sm_count();
        lora_merge_kernel<NCH><<<a.tiles < sms ? a.tiles : sms, LORA_THREADS, LoraCfg<NCH>::SMEM, st>>>(a);
        return true;
    }
    bool launch(cudaStream_t st) {
        if (a.count == 0) return true;
        a.err = device_error_word();
        a.failed = device_failed_word();
        if (!a.err || !a.failed) { set_error("lora: no memory for the error word"); return false; }
        if (!(low_rank ? launch_as<1>(st) : launch_as<2>(st))) return false;
        launched = true;
        a.count = a.tiles = 0;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { set_error("lora: launch: %s", cudaGetErrorString(e)); return false; }
        return true;
    }
};

}  // namespace o1

using namespace o1;

extern "C" {

// Returns once the merge is done, so that the caller may release the adapters.  HD_ERR_RUNTIME when it was not: an error of
// the stream, or the device's error word set, in which case the kernel merges nothing (it was set before) or stops on the way
// (one of its waits ran out).  A call whose targets all take the simple kernel (no whole 128-column tiles) only enqueues: it
// takes 4 us instead of 11 and can be captured, and the adapters stay until the stream has come past it.
hd_status hd_lora_merge_gpu(hd_lora_entry* entries, size_t count, void* stream) {
    if (count == 0) return HD_OK;
    if (!entries) { set_error("lora: null entries"); return HD_ERR_MISSING; }
    cudaStream_t st = (cudaStream_t)stream;
    hd_status rc = HD_OK;
    LoraGroup grp;
    for (size_t i = 0; i < count && rc == HD_OK; ++i) {
        hd_lora_entry* e = &entries[i];
        const int R = (int)e->rank, K = (int)e->in_dim, N = (int)e->out_dim;
        if (R <= 0 || K <= 0 || N <= 0 || !e->up_dev || !e->down_dev || !e->base_dev) {
            set_error("lora: bad entry %zu", i);
            rc = HD_ERR_MISMATCH;
            break;
        }
        const float scale = e->multiplier * e->alpha / (float)e->rank;
        const uintptr_t lo = (uintptr_t)e->base_dev, hi = lo + (size_t)N * K * 2;
        // whole 128-column tiles, at least the eight rows of a core matrix, and 16-byte aligned rows for TMA; the
        // number of tiles fits an int
        const bool tc = N >= 8 && (K % LT) == 0 && (lo & 15) == 0 && ((long)(N + LT - 1) / LT) * (K / LT) < (1l << 30);
        if ((grp.a.count == L_GROUP || !tc || (R <= LR) != grp.low_rank || grp.clashes(lo, hi) || grp.a.tiles >= (1 << 30)) && !grp.launch(st)) {
            rc = HD_ERR_RUNTIME;
            break;
        }
        if (!tc) {
            const long tot = (long)N * K;
            lora_simt_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(
                (uint16_t*)e->base_dev, (const float*)e->up_dev, (const float*)e->down_dev, N, K, R, scale);
            if (cudaGetLastError() != cudaSuccess) { set_error("lora: simt launch failed"); rc = HD_ERR_RUNTIME; }
            continue;
        }
        if (!make_tmap_bf16(&grp.a.tm[grp.a.count], e->base_dev, N, K, K, LT)) { rc = HD_ERR_RUNTIME; break; }
        grp.low_rank = R <= LR;
        LoraTarget& t = grp.a.t[grp.a.count];
        t.up = (const float*)e->up_dev;
        t.down = (const float*)e->down_dev;
        t.scale = scale;
        t.N = N; t.K = K; t.R = R;
        t.tiles_n = K / LT;
        t.tile0 = grp.a.tiles;
        t.vec = ((((uintptr_t)e->up_dev) | ((uintptr_t)e->down_dev)) & 15) == 0;
        grp.lo[grp.a.count] = lo; grp.hi[grp.a.count] = hi;
        grp.a.tiles += ((N + LT - 1) / LT) * t.tiles_n;
        ++grp.a.count;
    }
    // (an entry that cannot be used ends the call; the ones before it are merged)
    if (!grp.launch(st) && rc == HD_OK) rc = HD_ERR_RUNTIME;
    if (!grp.launched) return rc;
    const cudaError_t e = cudaStreamSynchronize(st);
    // (a copy of the error word itself would take 7.6 us: 236 -> 244 us for the adapter of a whole block)
    const int word = *(volatile int*)device_failed_word();
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("lora: %s", cudaGetErrorString(e));
    } else if (word != 0) {
        set_error("lora: the device's error word is set (code %d): the weights are not, or not all, merged", word);
    }
    return rc == HD_OK && (e != cudaSuccess || word != 0) ? HD_ERR_RUNTIME : rc;
}

}  // extern "C"
