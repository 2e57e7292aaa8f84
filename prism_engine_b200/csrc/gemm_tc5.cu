// Palettized GEMM on tcgen05 / TMEM:  Y[t][r] = f16( sum_k f32(X[t][k]) * f32(W[r][k]) )
// -- one lut_gemv_cpu per activation row (prefill_cpu, src/lut/engine_impl.rs:1046-1053; the
// reference's never-dispatched kernel for the same job is templates/palettized_gemm.metal:16-117).
//
// A persistent pair of CTAs (cta_group::2) computes tiles of 256 weight rows x nt tokens over a range of K:
//  * weights: the 16 dequantising warps of a CTA expand its 128 rows with lane-private pair tables (one row per
//    lane = one TMEM lane) and store 128 k at a time into a ring of TMEM stages -- the A operand never touches
//    shared memory;
//  * activations: TMA boxes of 64 k x nt/2 tokens straight from X, swizzled; each CTA fetches its half of the
//    tokens and one tcgen05.mma reads both halves, so a token tile crosses L2 once per PAIR;
//  * one thread of the pair issues the products (M = 256, N = nt, K = 16); the fp32 sums (nt TMEM columns) leave
//    through registers: they are taken out of TMEM first, the accumulator goes back to the issuing thread, and the
//    rounding, the residual or the SwiGLU product and the stores run under the next tile's products.  The first
//    stages of that tile are expanded before the sums are waited for.
// Where the tiles do not fill the GPU K is cut into ranges; their fp32 sums meet in scratch memory and the last
// warp to arrive adds them in a fixed order.
// 2-bit tensors (4-entry palettes; BITS = 2) run the same pipeline: a 16-byte index chunk then holds 64 weights of
// a row and expands into two 32-k chunks of the A operand through a 16-entry pair table indexed by nibbles
// (sk_expand2, pair_table.cuh).
// Bound: with many tokens the tensor core under the power cap; with few, the table lookups (256 cycles of the
// shared-memory pipe per 128 x 128 weights) and the latency of a short chain of stages.
// Measured, 4 bit, when it replaced one CTA per 128 x 256 tile whose single issuing thread spent 1 700 cycles on a stage of 1 024
// (waits one after the other, descriptors through vector registers, three commits) and which used as many CTAs as there were
// row tiles: 18944 x 3584, 2048 tokens 266 -> 216 us (1 287 TFLOP/s, 0.78 of measured burst), 512 tokens 67 -> 54, 32 tokens
// 26 -> 19.9; 4608 x 3584, 2048 tokens 72 -> 53, 32 tokens 23.4 -> 15.1; 3584 x 18944, 2048 tokens 320 -> 278, 32 tokens
// 96.5 -> 25.0.  The times before are without the residual or SwiGLU passes and the re-laid activations that went with them.
// A kernel of its own for split K (neither form holds the other's registers: stores of spills at 4 | 2 bits 370 | 322 bytes
// -> none for split K, 70 | 26 for whole K), the first table
// beside the TMEM allocation, the sums of four ranges requested together, and tiles by the fitted estimate of gm_plan: 3584 x 3584
// 15.7 -> 11.5 at 32 tokens, 3584 x 18944 26.5 -> 20.5 at 32, 81 -> 58 at 400, 269 -> 220 at 2048, gate and up of 18944 x 3584 40.1 -> 35.1.
// Every mbarrier wait is bounded; a wait that gives up raises the context's device error word.
#include <algorithm>

#include "common.cuh"
#include "pair_table.cuh"
#include "tc5_ptx.cuh"
#include "tensor_map.cuh"

namespace prism {

constexpr int GM_DEQ_WARPS = 16;
constexpr int GM_MMA_WARP = 16;  // the warp after it loads the activations
constexpr int GM_THREADS = 18 * 32;
constexpr int GM_STAGE_K = 128;               // k of a weight stage: 64 TMEM columns
constexpr int GM_SA = 4;                      // weight stages; a warp of slot j fills every fourth, ring position j
constexpr int GM_D_COL = GM_SA * 64;          // accumulator: up to 256 columns after the A stages
constexpr int GM_SX_MAX = 32;                 // most activation stages, of 64 k each
constexpr int GM_XD = GM_SX_MAX / 2;          // weight stages that many belong to
// The two pair tables start on 64 KB boundaries of the shared-memory window, so that a lookup's address is one
// permute of an index byte; barriers and activation stages lie before and after them.
constexpr uint32_t GM_SBASE = 1024;           // where dynamic shared memory starts (checked)
constexpr uint32_t GM_TBL = 65536;
constexpr uint32_t GM_OUT_LOW = 2048, GM_OUT_LOW_WARPS = 12;      // 1 KB per dequantising warp on the way out: 16 tokens x 32 rows
constexpr uint32_t GM_X_LOW = GM_OUT_LOW + GM_OUT_LOW_WARPS * 1024, GM_X_HIGH = GM_TBL + 2 * 65536;
constexpr uint32_t GM_END = GM_SBASE + 227 * 1024;
constexpr uint32_t GM_OUT_HIGH = GM_END - (GM_DEQ_WARPS - GM_OUT_LOW_WARPS) * 1024;
// barriers (8 B each) at GM_SBASE: afull[SA], done[SA], xfull[SX], xdone[XD], dfull, dempty; error flag, TMEM base.  One commit
// per weight stage gives back its TMEM columns and the activation stages it used; where small token tiles leave room for more
// activation stages than SA weight stages use, another says so on a ring of their length.
constexpr uint32_t GM_STATE = GM_SBASE + 8 * (2 * GM_SA + GM_SX_MAX + GM_XD + 2);
constexpr size_t GM_SMEM_BYTES = GM_END - GM_SBASE;
static_assert(GM_STATE + 16 <= GM_OUT_LOW, "barriers overlap what follows");

enum GemmOut { GM_PLAIN = 0, GM_RESID = 1, GM_SWIGLU = 2 };

struct GemmArgs {
    const uint8_t *idx, *idx2;        // weights: one tensor, or gate and up
    const uint16_t *pal, *pal2;
    uint32_t n_hb, m;                 // half-blocks, valid weight rows
    uint32_t n_ichunks;               // 16-byte index chunks per row (K/32 at 4 bit, K/64 at 2 bit)
    uint32_t n_st;                    // weight stages (K/128)
    uint32_t n_rp, n_tt, splits;      // pairs of 128-row tiles, token tiles, ranges of K
    uint32_t subs;                    // tensors a tile goes through one after the other: 2 for SwiGLU
    uint32_t nt;                      // tokens of a tile, a multiple of 32
    uint32_t sx_low, sx;              // activation stages before the tables, and in all
    uint32_t m_tok, mode;
    uint32_t wide;                    // rows of y (and resid) can be moved 8 values at a time; GM_PLAIN only without
    uint16_t *y;                      // [m_tok][m]
    const uint16_t *resid;            // [m_tok][m] (GM_RESID), may be y
    float *part;                      // [item][CTA][warp][column][lane] sums of a range
    unsigned int *arrived;            // [tile][CTA][warp]
    unsigned int *err;
};

namespace {

__device__ __forceinline__ void gm_mma_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int SLOT>
__device__ __forceinline__ uint32_t gm_lds(uint32_t off) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];\n" : "=r"(v) : "r"(off), "n"(SLOT * 128));
    return v;
}
// The 16 table lookups of one 32-k chunk of a row: bytes of the index words -> half2 entries.
template <int SLOT>
__device__ __forceinline__ void gm_lookup(uint32_t (&A)[16], const uint4 &wv, uint32_t laneq) {
    const uint32_t aw[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
    for (int hh = 0; hh < 4; hh++) {
        A[4 * hh + 0] = gm_lds<SLOT>(__byte_perm(aw[hh], laneq, 0x7604));
        A[4 * hh + 1] = gm_lds<SLOT>(__byte_perm(aw[hh], laneq, 0x7614));
        A[4 * hh + 2] = gm_lds<SLOT>(__byte_perm(aw[hh], laneq, 0x7624));
        A[4 * hh + 3] = gm_lds<SLOT>(__byte_perm(aw[hh], laneq, 0x7634));
    }
}
__device__ __forceinline__ void gm_lookup16(uint32_t (&A)[16], const uint4 &wv, uint32_t laneq, uint32_t slot) {
    if (slot == 0) gm_lookup<0>(A, wv, laneq);
    else gm_lookup<1>(A, wv, laneq);
}

struct GmItem {
    uint32_t rp, tt, k0, k1;  // k in stages
};
template <bool SPLIT>
__device__ __forceinline__ GmItem gm_item(const GemmArgs &a, uint32_t w) {
    if (!SPLIT) return GmItem{w % a.n_rp, w / a.n_rp, 0, a.n_st};
    const uint32_t s = w % a.splits, t = w / a.splits;
    return GmItem{t % a.n_rp, t / a.n_rp, a.n_st * s / a.splits, a.n_st * (s + 1) / a.splits};
}

// 16 tokens of one weight row, rounded (pairs, the first in the low half), where rows of y cannot be moved 8 values at a time.
__device__ __forceinline__ void gm_store(const GemmArgs &a, const uint32_t (&v)[8], uint32_t t0, uint32_t row) {
    if (row >= a.m || t0 >= a.m_tok) return;
    const uint32_t n = min(16u, a.m_tok - t0);
    uint16_t *y = a.y + (size_t)t0 * a.m + row;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++)
        if (i < n) y[(size_t)i * a.m] = (uint16_t)(v[i / 2] >> (16 * (i & 1)));
}
// A whole warp's 32 rows x 16 tokens, 16 bytes a lane: the values change places in the warp's 1 KB of shared memory, so that a
// lane holds 8 rows of a token; with the residual, or the product with silu of the gate values this lane stored for the tile
// before (f16(f16(silu(g)) * u), engine_impl.rs:1355-1366).
__device__ __forceinline__ void gm_store_wide(const GemmArgs &a, const uint32_t (&v)[8], uint32_t t0, uint32_t row0, uint32_t sub, uint8_t *out) {
    const uint32_t lane = threadIdx.x & 31;
    uint16_t *mine = reinterpret_cast<uint16_t *>(out) + lane;
#pragma unroll
    for (uint32_t i = 0; i < 16; i++) mine[i * 32] = (uint16_t)(v[i / 2] >> (16 * (i & 1)));
    __syncwarp();
    const uint32_t r = row0 + (lane & 3) * 8;
    const bool product = a.mode == GM_SWIGLU && sub == 1;
#pragma unroll
    for (uint32_t p = 0; p < 2; p++) {
        const uint32_t t = t0 + p * 8 + (lane >> 2);
        if (t >= a.m_tok || r >= a.m) continue;
        uint4 w = reinterpret_cast<const uint4 *>(out)[p * 32 + lane];
        uint16_t *y = a.y + (size_t)t * a.m + r;
        if (a.mode == GM_RESID || product) {
            const uint4 o = *reinterpret_cast<const uint4 *>(product ? y : a.resid + (size_t)t * a.m + r);
            const uint32_t ov[4] = {o.x, o.y, o.z, o.w};
            uint32_t wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&wv[i])), x = __half22float2(*reinterpret_cast<const __half2 *>(&ov[i]));
                __half2 res;
                if (product)
                    res = __floats2half2_rn(__half2float(__float2half_rn(x.x / (1.0f + expf(-x.x)))) * h.x, __half2float(__float2half_rn(x.y / (1.0f + expf(-x.y)))) * h.y);
                else
                    res = __floats2half2_rn(h.x + x.x, h.y + x.y);
                wv[i] = *reinterpret_cast<const uint32_t *>(&res);
            }
            w = make_uint4(wv[0], wv[1], wv[2], wv[3]);
        }
        *reinterpret_cast<uint4 *>(y) = w;
    }
    __syncwarp();
}
__device__ __forceinline__ uint32_t gm_pack(float x, float y) {
    const __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t *>(&h);
}

}  // namespace

template <int BITS, bool SPLIT>
__global__ void __launch_bounds__(GM_THREADS, 1) lut_gemm_tc5_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(smem);
    if ((smem_base & 0xFFFFu) != GM_SBASE) {  // layout assumption broken: refuse to compute
        if (threadIdx.x == 0) atomicExch(a.err, 1u);
        return;
    }
    uint8_t *const win = smem - GM_SBASE;               // 64 KB-aligned start of the window
    const uint32_t base = smem_base - GM_SBASE;
    // Tables, barriers and TMEM are set up from weights alone while the previous kernel drains.
    pdl_launch_dependents();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), rank = t5::cluster_rank();
    // afull, xfull and dempty: the pair's, in CTA 0 (it issues the products); done and dfull: each CTA's own
    const uint32_t b_afull = base + GM_SBASE, b_done = b_afull + 8 * GM_SA, b_xfull = b_done + 8 * GM_SA,
                   b_xdone = b_xfull + 8 * GM_SX_MAX, b_dfull = b_xdone + 8 * GM_XD, b_dempty = b_dfull + 8;
    const bool deep = a.sx > 2 * GM_SA;
    constexpr int ICPS = BITS == 4 ? 4 : 2;             // 16-byte index chunks per weight stage
    volatile uint32_t *err_flag = reinterpret_cast<volatile uint32_t *>(win + GM_STATE);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(win + GM_STATE + 8);
    const uint32_t n_items = a.n_rp * a.n_tt * a.splits, pair_id = blockIdx.x / 2, n_pairs = gridDim.x / 2;
    const uint32_t xstage = a.nt * 64;                  // bytes of this CTA's half of the tokens
    auto x_addr = [&](uint32_t s) { return base + (s < a.sx_low ? GM_X_LOW + s * xstage : GM_X_HIGH + (s - a.sx_low) * xstage); };

    // Dequantising warps: TMEM lane quarter, slot within the quarter; table area, row slot inside its entries.
    const uint32_t q = warp & 3, j = warp >> 2, area = q & 1, slot = q >> 1;
    uint4 r[ICPS];
    auto row_block = [&](const GmItem &i) { return min(4 * (2 * i.rp + rank) + q, a.n_hb - 1); };
    auto chunks = [&](const GmItem &i, uint32_t sub) { return (sub ? a.idx2 : a.idx) + (size_t)row_block(i) * a.n_ichunks * 512 + lane * 16; };
    auto build_table = [&](const GmItem &it, uint32_t sub) {
        uint8_t *tb = win + GM_TBL + area * 65536 + lane * 4 + slot * 128;
        if (BITS == 4) {
            const uint16_t *prow = (sub ? a.pal2 : a.pal) + ((size_t)row_block(it) * 32 + lane) * 16;
            const uint4 p0 = *reinterpret_cast<const uint4 *>(prow);
            const uint4 p1 = *reinterpret_cast<const uint4 *>(prow + 8);
            const uint32_t cbp[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
            const uint32_t hp0 = reinterpret_cast<const uint32_t *>(prow)[2 * j];
            const uint32_t hp1 = reinterpret_cast<const uint32_t *>(prow)[2 * j + 1];
            tb += j * 16384;
#pragma unroll
            for (int lo = 0; lo < 16; lo++) {
#pragma unroll
                for (int hs = 0; hs < 4; hs++) {
                    const uint32_t sel = (((hs & 1) ? 0x76u : 0x54u) << 8) | ((lo & 1) ? 0x32u : 0x10u);
                    *reinterpret_cast<uint32_t *>(tb + lo * 256 + hs * 4096) = __byte_perm(cbp[lo >> 1], (hs & 2) ? hp1 : hp0, sel);
                }
            }
        } else {
            // 16-entry nibble table: entry e = i0 | i1 << 2 -> half2{pal[i0], pal[i1]}; slot j writes e = 4j..4j+3
            const uint2 pp = *reinterpret_cast<const uint2 *>((sub ? a.pal2 : a.pal) + ((size_t)row_block(it) * 32 + lane) * 4);
            const uint32_t v1 = ((j & 2) ? pp.y : pp.x) >> ((j & 1) * 16) & 0xFFFFu;  // pal[i1], i1 = j
#pragma unroll
            for (uint32_t i0 = 0; i0 < 4; i0++) {
                const uint32_t v0 = ((i0 & 2) ? pp.y : pp.x) >> ((i0 & 1) * 16) & 0xFFFFu;
                *reinterpret_cast<uint32_t *>(tb + (4 * j + i0) * 256) = v0 | (v1 << 16);
            }
        }
    };

    if (tid == GM_THREADS - 32) {
        for (int s = 0; s < GM_SA; s++) { t5::mbar_init(b_afull + 8 * s, 8); t5::mbar_init(b_done + 8 * s, 1); }
        for (int s = 0; s < GM_SX_MAX; s++) t5::mbar_init(b_xfull + 8 * s, 1);
        for (int s = 0; s < GM_XD; s++) t5::mbar_init(b_xdone + 8 * s, 1);
        t5::mbar_init(b_dfull, 1);
        t5::mbar_init(b_dempty, 2 * GM_DEQ_WARPS);
        *err_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == GM_MMA_WARP) t5::tmem_alloc_pair(base + GM_STATE + 8, 512);
    // The first tile's indices and table, beside the allocation: every pair has a tile (the grid is no larger than they are).
    if (warp < GM_DEQ_WARPS) {
        const GmItem it = gm_item<SPLIT>(a, pair_id);
        const uint32_t su = it.k0 + j;
        if (su < it.k1) {
            const uint8_t *sp = chunks(it, 0) + (size_t)su * ICPS * 512;
#pragma unroll
            for (int c = 0; c < ICPS; c++) r[c] = t5::ldg128_nc(sp + c * 512);
        }
        build_table(it, 0);
    }
    t5::fence_before();
    __syncthreads();
    t5::cluster_sync();  // the other CTA's barriers exist before anything arrives there
    t5::fence_after();
    const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);

    if (warp < GM_DEQ_WARPS) {
        // =============================== dequantising warps ===============================
        const uint32_t laneq = base + GM_TBL + area * 65536 + lane * 4;
        const uint32_t tmem_lane = tmem_base + ((q * 32) << 16);
        const uint32_t afull0 = t5::map_rank(b_afull + 8 * j, 0), dempty0 = t5::map_rank(b_dempty, 0);
        uint8_t *out = win + (warp < GM_OUT_LOW_WARPS ? GM_OUT_LOW + warp * 1024 : GM_OUT_HIGH + (warp - GM_OUT_LOW_WARPS) * 1024);
        const uint32_t groups = a.nt / 16;               // of 16 accumulator columns; this warp takes j, j + 4, ...
        uint32_t n = 0, ti = 0, cur = gm_item<SPLIT>(a, pair_id).rp * 2;  // the tables are those of tensor `sub` (lowest bit), row pair
        uint32_t pend_w = 0xFFFFFFFFu, pend_sub = 0;     // the tile whose sums are still in TMEM
        bool waited = false, ahead = true;                // ahead: r holds this slot's first stage of the tile already

        auto epilogue = [&](uint32_t w, uint32_t sub) {
            const GmItem it = gm_item<SPLIT>(a, w);
            const uint32_t row = (2 * it.rp + rank) * 128 + q * 32 + lane, tile = SPLIT ? w / a.splits : w, place = rank * GM_DEQ_WARPS + warp;
            const uint32_t per = (groups + 3) / 4 * 512;  // floats of a warp
            t5::mbar_wait_warp(b_dfull, ti & 1, err_flag);
            t5::fence_after();
            ti++;
            auto store = [&](const uint32_t (&v)[8], uint32_t i) {
                const uint32_t t0 = it.tt * a.nt + (j + 4 * i) * 16;
                if (a.wide) gm_store_wide(a, v, t0, row - lane, sub, out);
                else gm_store(a, v, t0, row);
            };
            if (!SPLIT) {
                uint32_t sums[4][8];
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    if (j + 4 * i >= groups) break;
                    uint32_t v[16];
                    t5::ld16(tmem_lane + GM_D_COL + (j + 4 * i) * 16, v);
                    t5::wait_ld();
#pragma unroll
                    for (uint32_t c = 0; c < 8; c++) sums[i][c] = gm_pack(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]));
                }
                t5::fence_before();
                __syncwarp();
                if (lane == 0) t5::mbar_arrive_tmem(dempty0);
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) {
                    if (j + 4 * i >= groups) break;
                    store(sums[i], i);
                }
            } else {
                for (uint32_t i = 0; j + 4 * i < groups; i++) {
                    uint32_t v[16];
                    t5::ld16(tmem_lane + GM_D_COL + (j + 4 * i) * 16, v);
                    t5::wait_ld();
                    float *mine = a.part + ((size_t)w * 2 * GM_DEQ_WARPS + place) * per + i * 512 + lane;
#pragma unroll
                    for (uint32_t c = 0; c < 16; c++) __stcg(mine + c * 32, __uint_as_float(v[c]));
                }
                t5::fence_before();
                __syncwarp();
                uint32_t before = 0;
                if (lane == 0) {
                    t5::mbar_arrive_tmem(dempty0);
                    __threadfence();
                    before = atomicAdd(a.arrived + (size_t)tile * 2 * GM_DEQ_WARPS + place, 1u);
                    __threadfence();
                }
                if (__shfl_sync(0xFFFFFFFFu, before, 0) != a.splits - 1) return;
                __syncwarp();
                if (lane == 0) a.arrived[(size_t)tile * 2 * GM_DEQ_WARPS + place] = 0;
                const size_t step = (size_t)2 * GM_DEQ_WARPS * per;
                for (uint32_t i = 0; j + 4 * i < groups; i++) {
                    const float *p = a.part + ((size_t)tile * a.splits * 2 * GM_DEQ_WARPS + place) * per + i * 512 + lane;
                    float f[16];
#pragma unroll
                    for (uint32_t c = 0; c < 16; c++) f[c] = 0.0f;
                    for (uint32_t s = 0; s < a.splits; s += 4, p += 4 * step) {  // four ranges requested together, added in order
                        float g[4][16];
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++)
#pragma unroll
                            for (uint32_t c = 0; c < 16; c++) g[u][c] = s + u < a.splits ? __ldcg(p + u * step + c * 32) : 0.0f;
#pragma unroll
                        for (uint32_t u = 0; u < 4; u++)
#pragma unroll
                            for (uint32_t c = 0; c < 16; c++) f[c] += g[u][c];
                    }
                    uint32_t v[8];
#pragma unroll
                    for (uint32_t c = 0; c < 8; c++) v[c] = gm_pack(f[2 * c], f[2 * c + 1]);
                    store(v, i);
                }
            }
            __syncwarp();
        };

        bool late = false;                               // this slot's last stage was one of the last two of its tile
        for (uint32_t w = pair_id, sub = 0;;) {
            const bool over = w >= n_items;              // past the last tile: its sums are still to be stored
            GmItem it = gm_item<SPLIT>(a, w);
            if (over) it.k0 = it.k1 = 0;
            {
                uint32_t su = it.k0 + ((j - n) & 3);     // this slot's first stage: ring position j
                const uint8_t *sp = chunks(it, sub);
                if (su < it.k1 && !ahead)
#pragma unroll
                    for (int c = 0; c < ICPS; c++) r[c] = t5::ldg128_nc(sp + (size_t)(su * ICPS + c) * 512);
                ahead = false;
                if (!over && it.rp * 2 + sub != cur) {  // same decision in all warps: they walk the same item list
                    cur = it.rp * 2 + sub;
                    asm volatile("bar.sync %0, 256;\n" ::"r"(1 + area) : "memory");  // lookups of the previous tile are done
                    build_table(it, sub);
                    asm volatile("bar.sync %0, 256;\n" ::"r"(1 + area) : "memory");
                }
                // Everything so far read weights only.  The waits below depend on the activations: wait for the kernel
                // before this one first, so that no bounded wait runs while it (under tensor parallelism: a late peer) is
                // still at work.
                if (!waited) {
                    pdl_wait();
                    waited = true;
                }
                for (bool first = true; first || su < it.k1 || pend_w != 0xFFFFFFFFu; first = false, su += 4) {
                    // The tile before.  A slot that finished early expands its first stage of this one before it waits for the sums, so
                    // that the tensor core has something to go on with; the slots of the last two stages take the sums out first.  Nobody
                    // comes to a second stage before that: it waits for products that wait for these sums.
                    if (pend_w != 0xFFFFFFFFu && (!first || late || su >= it.k1)) {
                        epilogue(pend_w, pend_sub);
                        pend_w = 0xFFFFFFFFu;
                    }
                    if (su < it.k1) {
                        // what r takes next: this slot's next stage, of this tile or of the one after it
                        const uint8_t *np = sp + (size_t)(su + 4) * ICPS * 512;
                        bool fill = su + 4 < it.k1;
                        if (!fill) {
                            const uint32_t nsub = sub + 1 == a.subs ? 0 : sub + 1, nw = nsub ? w : w + n_pairs;
                            const GmItem ni = gm_item<SPLIT>(a, nw);
                            const uint32_t nsu = ni.k0 + ((j - (n + it.k1 - it.k0)) & 3);
                            ahead = fill = nw < n_items && nsu < ni.k1;
                            np = chunks(ni, nsub) + (size_t)nsu * ICPS * 512;
                            late = su + 2 >= it.k1;
                        }
#pragma unroll
                        for (int half = 0; half < 2; half++) {  // 64 k at a time: 32 registers of weights
                            uint32_t A[2][16];
                            if (BITS == 4) {
#pragma unroll
                                for (int c = 0; c < 2; c++) {
                                    const uint4 wv = r[2 * half + c];
                                    if (fill) r[2 * half + c] = t5::ldg128_nc(np + (2 * half + c) * 512);
                                    gm_lookup16(A[c], wv, laneq, slot);
                                }
                            } else {
                                uint4 pa, pb;
                                sk_expand2(pa, pb, r[half]);
                                if (fill) r[half] = t5::ldg128_nc(np + half * 512);
                                gm_lookup16(A[0], pa, laneq, slot);
                                gm_lookup16(A[1], pb, laneq, slot);
                            }
                            if (half == 0) {
                                t5::mbar_wait_warp(b_done + 8 * j, (((n + su - it.k0) / GM_SA) & 1) ^ 1, err_flag);
                                t5::fence_after();
                            }
                            t5::st16(tmem_lane + j * 64 + half * 32, A[0]);
                            t5::st16(tmem_lane + j * 64 + half * 32 + 16, A[1]);
                        }
                        t5::wait_st();
                        t5::fence_before();
                        if (lane == 0) t5::mbar_arrive_tmem(afull0);
                    }
                }
                if (over) break;
            }
            pend_w = w;
            pend_sub = sub;
            n += it.k1 - it.k0;
            if (++sub == a.subs) {
                sub = 0;
                w += n_pairs;
            }
        }
    } else if (warp == GM_MMA_WARP) {
        // =============================== MMA issuing warp ===============================
        // The whole warp walks the stages, so that the compiler keeps descriptors and addresses in uniform registers, and one
        // elected lane issues.  A test of a barrier takes some 100 to 250 cycles behind the lookups of the other warps: three
        // lanes test the three of the next stage at once.
        if (rank == 0) {
            const uint32_t idesc = t5::idesc_f16(256, a.nt), dcol = tmem_base + GM_D_COL;
            uint32_t n = 0, sx = 0, px = 0, ti = 0;
            pdl_wait();  // see the dequantising warps: no bounded wait before the dependency is met
            uint32_t ready = 0;                            // this stage's weights (1) and activations (2, 4) have been seen to be there
            for (uint32_t w = pair_id; w < n_items; w += n_pairs) {
                const GmItem it = gm_item<SPLIT>(a, w);
                for (uint32_t sub = 0; sub < a.subs; sub++, ti++) {
                    t5::mbar_wait_bounded(b_dempty, (ti & 1) ^ 1, err_flag);  // the sums of the tile before have left D
                    for (uint32_t su = it.k0; su < it.k1; su++, n++) {
                        const uint32_t sa = n % GM_SA, acol = tmem_base + sa * 64;
                        const uint32_t s1 = sx + 1 == a.sx ? 0 : sx + 1, p1 = px ^ (s1 == 0), s2 = s1 + 1 == a.sx ? 0 : s1 + 1,
                                       p2 = p1 ^ (s2 == 0), s3 = s2 + 1 == a.sx ? 0 : s2 + 1, p3 = p2 ^ (s3 == 0);
                        if (!(ready & 1)) t5::mbar_wait_bounded(b_afull + 8 * sa, (n / GM_SA) & 1, err_flag);
                        if (!(ready & 2)) t5::mbar_wait_bounded(b_xfull + 8 * sx, px, err_flag);
                        const uint32_t next = __ballot_sync(0xFFFFFFFFu, t5::mbar_test(lane == 0 ? b_afull + 8 * ((n + 1) % GM_SA) : b_xfull + 8 * (lane == 1 ? s2 : s3),
                                                                                       lane == 0 ? ((n + 1) / GM_SA) & 1 : lane == 1 ? p2 : p3));
                        t5::fence_after();
                        const uint64_t x0 = t5::desc_swizzled<128>(x_addr(sx)), x1 = t5::desc_swizzled<128>(x_addr(s1));
                        if (t5::elect_one()) {
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; kk++)  // 16 k are 32 bytes of the swizzled row
                                gm_mma_pair(dcol, acol + kk * 8, x0 + kk * 2, idesc, kk ? 1u : su - it.k0);
                        }
                        if (!(ready & 4)) t5::mbar_wait_bounded(b_xfull + 8 * s1, p1, err_flag);
                        __syncwarp();
                        t5::fence_after();
                        if (t5::elect_one()) {
#pragma unroll
                            for (uint32_t kk = 0; kk < 4; kk++) gm_mma_pair(dcol, acol + 32 + kk * 8, x1 + kk * 2, idesc, 1u);
                            t5::commit_pair(b_done + 8 * sa);
                            if (deep) t5::commit_pair(b_xdone + 8 * (n % GM_XD));
                        }
                        ready = next;
                        sx = s2; px = p2;
                    }
                    if (t5::elect_one()) t5::commit_pair(b_dfull);
                }
            }
        }
    } else if (lane == 0) {
        // =============================== activation loader ===============================
        const uint32_t full0 = t5::map_rank(b_xfull, 0);
        uint32_t sx = 0, h = 0;                            // h: activation stages so far, two per weight stage
        const uint32_t ring = deep ? GM_XD : GM_SA, b_step = deep ? b_xdone : b_done;
        auto wait_step = [&](uint32_t step) { t5::mbar_wait_bounded(b_step + 8 * (step % ring), (step / ring) & 1, err_flag); };
        pdl_wait();
        for (uint32_t w = pair_id; w < n_items; w += n_pairs) {
            const GmItem it = gm_item<SPLIT>(a, w);
            const int32_t t0 = (int32_t)(it.tt * a.nt + rank * (a.nt / 2));
            for (uint32_t sub = 0; sub < a.subs; sub++) {
                for (uint32_t k = it.k0 * 128; k < it.k1 * 128; k += 64, h++) {
                    if (h >= a.sx) wait_step((h - a.sx) / 2);  // at most `ring` stages back: its barrier has not come round again
                    if (rank == 0) t5::mbar_arrive_expect_tx(b_xfull + 8 * sx, 2 * xstage);
                    t5::tma_2d_pair(x_addr(sx), &xmap, (int32_t)k, t0, full0 + 8 * sx);
                    if (++sx == a.sx) sx = 0;
                }
            }
        }
        // every copy in flight lands before the CTA leaves: a stage is done after its products
        for (uint32_t step = h / 2 > ring ? h / 2 - ring : 0; step < h / 2; step++) wait_step(step);
    }
    t5::fence_before();
    __syncthreads();
    t5::cluster_sync();  // nothing arrives in a CTA that has left
    t5::fence_after();
    if (warp == GM_MMA_WARP) t5::tmem_dealloc_pair(tmem_base, 512);
    if (tid == 0 && *err_flag) atomicExch(a.err, 5u);
}

// ---- host side ---------------------------------------------------------------------------------
bool gemm_tc5_eligible(prism_cuda_ctx *ctx, const LutTensor &t, uint32_t m_tok) {
    // whole weight stages of 128 k (four 32-k chunks: four index chunks at 4 bit, two at 2 bit)
    return ctx->smem_base == (int)GM_SBASE && (t.bits == 4 || t.bits == 2) && t.k % GM_STAGE_K == 0 && m_tok >= 8;
}
bool gemm_tc5_wide(const LutTensor &t, const uint16_t *y) { return t.m % 8 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0; }

// Tokens of a tile and ranges of K with the least estimated cycles: a stage's products or its look-ups and hand-overs, a tile's way
// into and out of the pipeline, a launch, the tables of another pair of row tiles; a split pays for its sums' way through L2 and the
// wait for the last of them.  Fitted to every choice (tiles of 32 to 256 tokens, 1 to 8 ranges) for 17 shapes of 2 and 4 bits and
// 24 to 2048 tokens, cold weights: within 12 % of the times, and what it chooses takes 0.7 % more than the best choice on average,
// 10 % at most.  The estimate before took 5 % more on average and up to 1.5 times as long: it only weighed tiles near 256 tokens
// (3584 x 18944, 2048 tokens: 256 tokens and 112 tiles for 74 pairs 261 us, 224 and 140 220; 8192 x 8192, 100 tokens 39 and 28).
struct GmPlan {
    uint32_t nt = 32, splits = 1;
    double cycles = 1e30;
};
static GmPlan gm_plan(uint32_t pairs, uint32_t n_rp, uint32_t n_st, uint32_t m_tok, uint32_t subs, uint32_t most_splits) {
    GmPlan best;
    const uint32_t top = std::min(256u, round_up_u32(m_tok, 32));
    for (uint32_t nt = top; nt >= 32; nt -= 32) {
        const uint64_t tiles = (uint64_t)n_rp * ((m_tok + nt - 1) / nt);
        for (uint32_t cut = 1; cut <= most_splits && cut <= n_st; cut++) {
            if (cut > 1 && tiles * cut * 256 * nt * 4 > (64u << 20)) break;  // bytes of partial sums
            const uint64_t waves = (tiles * cut + pairs - 1) / pairs, tables = subs == 2 ? 2 * waves : cut > 1 || pairs % n_rp ? waves : 1;
            double t = 4200.0 + (double)waves * subs * ((n_st + cut - 1) / cut * std::max(5.6 * nt, 915.0) + 6800.0) + (double)(tables - 1) * 3800.0;
            if (cut > 1) t += 4000.0 + (double)waves * nt * 17.0 + cut * nt * 7.0;
            if (t < best.cycles * 0.999) {
                best.cycles = t;
                best.nt = nt;
                best.splits = cut;
            }
        }
    }
    return best;
}

template <int BITS>
static int gm_pairs(prism_cuda_ctx *ctx, uint32_t *out) {  // pairs that are resident at once
    static int pairs[PRISM_MAX_DEVICES] = {0};
    if (!pairs[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(lut_gemm_tc5_kernel<BITS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GM_SMEM_BYTES));
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(lut_gemm_tc5_kernel<BITS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GM_SMEM_BYTES));
        const int n = resident_clusters(lut_gemm_tc5_kernel<BITS, true>, 2, GM_THREADS, GM_SMEM_BYTES, 2 * ((uint32_t)ctx->sm_count / 2));
        pairs[ctx->device] = std::max(1, std::min(n, ctx->sm_count / 2));
    }
    *out = (uint32_t)pairs[ctx->device];
    return PRISM_OK;
}

template <int BITS>
static int launch_gm(prism_cuda_ctx *ctx, GemmArgs &a, const LutTensor &t, const uint16_t *X, const GmPlan &p, uint32_t pairs) {
    a.nt = p.nt;
    a.splits = p.splits;
    a.n_tt = (a.m_tok + a.nt - 1) / a.nt;
    a.wide = gemm_tc5_wide(t, a.y) && (reinterpret_cast<uintptr_t>(a.resid) & 15) == 0;
    if (a.mode != GM_PLAIN && !a.wide) return fail(ctx, PRISM_E_ARG, "gemm: a residual or gated product needs rows of a multiple of 8 values, 16-byte aligned");
    const uint32_t xstage = a.nt * 64;
    a.sx_low = std::min((uint32_t)GM_SX_MAX, (GM_TBL - GM_X_LOW) / xstage);
    a.sx = std::min((uint32_t)GM_SX_MAX, a.sx_low + (GM_OUT_HIGH - GM_X_HIGH) / xstage);
    const size_t tiles = (size_t)a.n_rp * a.n_tt;
    if (a.splits > 1) {
        const uint32_t per = (a.nt / 16 + 3) / 4 * 512;
        PRISM_TRY(ensure_splitk(ctx, tiles * a.splits * 2 * GM_DEQ_WARPS * per, tiles * 2 * GM_DEQ_WARPS));
        a.part = ctx->splitk_partials;
        a.arrived = ctx->splitk_counters;
    }
    CUtensorMap xmap;
    PRISM_TRY(encode_tensor_map(ctx, &xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, X, t.k, a.m_tok, t.k, 64, a.nt / 2, CU_TENSOR_MAP_SWIZZLE_128B));
    const uint32_t grid = (uint32_t)std::min<uint64_t>(pairs, (uint64_t)tiles * a.splits);
    launch_cluster_pdl(ctx, a.splits > 1 ? lut_gemm_tc5_kernel<BITS, true> : lut_gemm_tc5_kernel<BITS, false>, dim3(2 * grid), dim3(GM_THREADS), GM_SMEM_BYTES, 2u, a, xmap);
    return after_launch(ctx, "lut_gemm_tc5_kernel");
}

static GemmArgs gm_args(prism_cuda_ctx *ctx, const LutTensor &t, uint32_t m_tok, uint16_t *Y) {
    GemmArgs a{};
    a.idx = t.idx; a.pal = t.pal;
    a.n_st = t.k / GM_STAGE_K; a.n_ichunks = t.n_chunks; a.n_hb = t.n_hb; a.m = t.m;
    a.n_rp = (t.n_hb + 7) / 8;
    a.subs = 1;
    a.m_tok = m_tok;
    a.y = Y; a.err = ctx->dev_err;
    return a;
}
constexpr uint32_t GM_MAX_SPLITS = 8;

template <int BITS>
static int gemm_bits(prism_cuda_ctx *ctx, const LutTensor &t, const uint16_t *X, uint32_t m_tok, uint16_t *Y, const uint16_t *resid) {
    uint32_t pairs = 0;
    PRISM_TRY(gm_pairs<BITS>(ctx, &pairs));
    GemmArgs a = gm_args(ctx, t, m_tok, Y);
    a.mode = resid ? GM_RESID : GM_PLAIN;
    a.resid = resid;
    return launch_gm<BITS>(ctx, a, t, X, gm_plan(pairs, a.n_rp, a.n_st, m_tok, 1, GM_MAX_SPLITS), pairs);
}
int launch_gemm_tc5(prism_cuda_ctx *ctx, const LutTensor &t, const uint16_t *X, uint32_t m_tok, uint16_t *Y, const uint16_t *resid) {
    if (reinterpret_cast<uintptr_t>(X) & 15) return fail(ctx, PRISM_E_ARG, "gemm: X must be 16-byte aligned");
    return t.bits == 2 ? gemm_bits<2>(ctx, t, X, m_tok, Y, resid) : gemm_bits<4>(ctx, t, X, m_tok, Y, resid);
}

// Gate and up of a tile one after the other by the same CTA, whose threads meet their own gate values again.
template <int BITS>
static int swiglu_bits(prism_cuda_ctx *ctx, const LutTensor &tg, const LutTensor &tu, const uint16_t *X, uint32_t m_tok, uint16_t *act) {
    uint32_t pairs = 0;
    PRISM_TRY(gm_pairs<BITS>(ctx, &pairs));
    GemmArgs a = gm_args(ctx, tg, m_tok, act);
    a.idx2 = tu.idx; a.pal2 = tu.pal;
    a.subs = 2;
    a.mode = GM_SWIGLU;
    return launch_gm<BITS>(ctx, a, tg, X, gm_plan(pairs, a.n_rp, a.n_st, m_tok, 2, 1), pairs);
}
int launch_swiglu_tc5(prism_cuda_ctx *ctx, const LutTensor &tg, const LutTensor &tu, const uint16_t *X, uint32_t m_tok, uint16_t *act) {
    if (reinterpret_cast<uintptr_t>(X) & 15) return fail(ctx, PRISM_E_ARG, "gemm: X must be 16-byte aligned");
    return tg.bits == 2 ? swiglu_bits<2>(ctx, tg, tu, X, m_tok, act) : swiglu_bits<4>(ctx, tg, tu, X, m_tok, act);
}
// Gate and up in one launch, or two launches with K cut into ranges and a pass over their outputs (5120 x 2048, 24 tokens 25.0 / 24.3 us,
// 8192 x 4096 38.1 / 34.0; at 256 tokens 32.4 / 38.7 and 51.0 / 60.2).
template <int BITS>
static int gm_swiglu_cycles(prism_cuda_ctx *ctx, const LutTensor &t, uint32_t m_tok, double *fused, double *apart) {
    uint32_t pairs = 0;
    PRISM_TRY(gm_pairs<BITS>(ctx, &pairs));
    const GemmArgs a = gm_args(ctx, t, m_tok, nullptr);
    *fused = gm_plan(pairs, a.n_rp, a.n_st, m_tok, 2, 1).cycles;
    *apart = 2 * gm_plan(pairs, a.n_rp, a.n_st, m_tok, 1, GM_MAX_SPLITS).cycles + 6000.0 + (double)m_tok * t.m * 8.0 / 3500.0;
    return PRISM_OK;
}
int gemm_tc5_cycles(prism_cuda_ctx *ctx, const LutTensor &t, uint32_t m_tok, uint32_t subs, double *cycles) {
    if (subs == 2) {
        double fused = 0, apart = 0;
        PRISM_TRY(t.bits == 2 ? gm_swiglu_cycles<2>(ctx, t, m_tok, &fused, &apart) : gm_swiglu_cycles<4>(ctx, t, m_tok, &fused, &apart));
        *cycles = std::min(fused, apart);
        return PRISM_OK;
    }
    uint32_t pairs = 0;
    PRISM_TRY(t.bits == 2 ? gm_pairs<2>(ctx, &pairs) : gm_pairs<4>(ctx, &pairs));
    const GemmArgs a = gm_args(ctx, t, m_tok, nullptr);
    *cycles = gm_plan(pairs, a.n_rp, a.n_st, m_tok, 1, GM_MAX_SPLITS).cycles;
    return PRISM_OK;
}
int swiglu_tc5_pays(prism_cuda_ctx *ctx, const LutTensor &tg, uint32_t m_tok, bool *pays) {
    double fused = 0, apart = 0;
    PRISM_TRY(tg.bits == 2 ? gm_swiglu_cycles<2>(ctx, tg, m_tok, &fused, &apart) : gm_swiglu_cycles<4>(ctx, tg, m_tok, &fused, &apart));
    *pays = fused <= apart;
    return PRISM_OK;
}

}  // namespace prism
