// Dense bf16 GEMM on tcgen05 / TMEM with the segment epilogues of dense.cuh:
//   y[t][n] = epilogue( sum_k x[t][k] * W[n][k] ),  fp32 accumulate.
//
// dense_gemm_pair_kernel: a persistent pair of CTAs computes tiles of 256 weight rows x NT rows of x with
// tcgen05.mma.cta_group::2: each CTA holds its own 128 weight rows and half of the rows of x, so a tile needs 128 + NT / 2
// rows of operands per SM where one CTA alone would need 128 + NT.  Two accumulators of NT columns alternate in TMEM:
// the epilogue of a tile (eight warps per CTA) runs under the products of the next one.
// What bounds it: the operands' way from L2 -- 32 KB per SM and stage at NT = 256, about 760 cycles where the products
// take 512.  One CTA on 256 x 256 moved as many bytes but left its epilogue exposed: 33280 x 3584 on 2048 rows 420 -> 367
// us (1.33 PFLOP/s), 3584 x 22528 216 -> 204 on average with the other linears of a layer.
// Shapes with few tiles cut k into ranges: 3584 x 22528 on 500 rows 122 -> about 70 us.
// dense_gemm_tc5_kernel: the same on one CTA and 128 weight rows, for shapes with too few pairs of row tiles.
// One warp loads: the weights of a 64-k stage are one contiguous 16 KB run (dense.cuh) that already has the unswizzled
// core-matrix order of the A operand; the rows of x come through a tensor map with the 128-byte swizzle of the B operand
// (rows past the end are filled with zeros).  One thread issues the products; four warps per 128 rows read an
// accumulator back, apply the epilogue of the tile's segment and store.
// Every mbarrier wait is bounded; one that gives up raises the context's device error word.
#include <algorithm>

#include "dense.cuh"
#include "tc5_ptx.cuh"
#include "tensor_map.cuh"

namespace prism {

constexpr int DG_A_BYTES = 128 * 64 * 2;      // weights of a stage and row tile
template <int NT>
struct DgCfg {
    static constexpr int THREADS = 64 + 128;      // loader warp, MMA warp, four epilogue warps
    static constexpr int A_BYTES = DG_A_BYTES, B_BYTES = NT * 128;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int S = (200 * 1024 / STAGE) < 8 ? (200 * 1024 / STAGE) : 8;
    static constexpr int TMEM_COLS = 2 * NT < 32 ? 32 : 2 * NT;
    static constexpr int BAR_OFF = S * STAGE;
    static constexpr int TAB_OFF = BAR_OFF + 8 * (2 * S + 4) + 64;
    static constexpr size_t SMEM = TAB_OFF + 1024;  // + slack for the 1 KB alignment of the stages; experts: + their table
};

template <int NT>
struct DpCfg {
    static constexpr int THREADS = 64 + 256;      // loader warp, MMA warp, eight epilogue warps (two per quarter of the rows)
    static constexpr int B_BYTES = NT / 2 * 128;  // this CTA's half of the rows of x
    static constexpr int STAGE = DG_A_BYTES + B_BYTES;
    static constexpr int S = 200 * 1024 / STAGE;
    static constexpr int TMEM_COLS = 2 * NT;
    static constexpr int BAR_OFF = S * STAGE;
    static constexpr int TAB_OFF = BAR_OFF + 8 * (2 * S + 4) + 64;
    static constexpr size_t SMEM = TAB_OFF + 1024;
};

struct DgArgs {
    const uint8_t *w;
    uint32_t kb;              // 64-k stages per row
    uint32_t n_rt, n_tt, rt_group;  // row tiles (pairs of them), token tiles, row tiles per group of the walk
    uint32_t rows;            // rows of x
    uint32_t types;           // operand types in the instruction descriptor
    unsigned int *err;
    DenseEpi epi;
    uint32_t experts;         // 0: plain; else rows of x are sorted by expert and a token tile belongs to one
    const uint32_t *count;    // [experts] rows
    // pairs of CTAs only: k cut into `splits` ranges, neighbouring items of the walk; every epilogue warp leaves its sums
    // in `part` and the last of a tile's splits to arrive adds them in order, so the result does not depend on timing
    uint32_t splits;
    float *part;              // [item][CTA of the pair][warp][column][lane]
    unsigned int *arrived;    // [tile][CTA][warp], zero between launches
};
constexpr uint32_t DG_MAX_EXPERTS = 1024;

// Walk of the tiles: groups of rt_group row tiles over all token tiles, so that the CTAs of one wave share a
// few weights and a few rows of x in L2.
__device__ __forceinline__ void dg_item(const DgArgs &a, uint32_t w, uint32_t &rt, uint32_t &tt) {
    const uint32_t per = a.rt_group * a.n_tt, g = w / per, rem = w % per;
    const uint32_t gr = min(a.rt_group, a.n_rt - g * a.rt_group);
    rt = g * a.rt_group + rem % gr;
    tt = rem / gr;
}

// Experts, by one warp: running sums of their token tiles and rows.
template <int NT>
__device__ __forceinline__ void dg_expert_table(const DgArgs &a, uint32_t *tile_end, uint32_t *row_end, uint32_t lane) {
    uint32_t tiles = 0, rows = 0;
    for (uint32_t e0 = 0; e0 < a.experts; e0 += 32) {
        uint32_t r = e0 + lane < a.experts ? a.count[e0 + lane] : 0, t = (r + NT - 1) / NT;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, t, o), y = __shfl_up_sync(0xFFFFFFFFu, r, o);
            if ((int)lane >= o) { t += x; r += y; }
        }
        if (e0 + lane < a.experts) { tile_end[e0 + lane] = tiles + t; row_end[e0 + lane] = rows + r; }
        tiles += __shfl_sync(0xFFFFFFFFu, t, 31);
        rows += __shfl_sync(0xFFFFFFFFu, r, 31);
    }
}
// Item w of the walk (RT row tiles of 128): its row tile, that tile's place in the weights (counted over all experts),
// its first row of x and the row of x it ends before.
struct DgItem { uint32_t rt, wt, t0, t_end; };
// First 64-k stage of split s of a segment's k.
__device__ __forceinline__ uint32_t dg_k(const DgArgs &a, const DenseEpiSeg &seg, uint32_t s) { return seg.k / 64 * s / a.splits; }
template <int NT, int RT, bool MOE>
__device__ __forceinline__ DgItem dg_locate(const DgArgs &a, uint32_t w, const uint32_t *tile_end, const uint32_t *row_end) {
    DgItem i;
    if (!MOE) {
        uint32_t tt;
        dg_item(a, w, i.rt, tt);
        i.wt = i.rt * RT;
        i.t0 = tt * NT;
        i.t_end = a.rows;
    } else {
        const uint32_t tt = w / a.n_rt;
        i.rt = w % a.n_rt;
        uint32_t lo = 0, hi = a.experts - 1;  // first expert with tile_end > tt
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (tile_end[mid] > tt) hi = mid; else lo = mid + 1;
        }
        const uint32_t first = lo ? tile_end[lo - 1] : 0, r0 = lo ? row_end[lo - 1] : 0;
        i.wt = (lo * a.n_rt + i.rt) * RT;
        i.t0 = r0 + (tt - first) * NT;
        i.t_end = row_end[lo];
    }
    return i;
}

// The epilogue of dense_store for one weight row (a lane) over the NT tokens of a tile, with what does not change
// along the way decided once: sixteen accumulators are read, the residual's old values requested together, and
// the activation of a bf16 result takes the fast exponential and reciprocal.
template <uint32_t ACT>
__device__ __forceinline__ float act_fast(float z) {
    if (ACT == ACT_NONE) return z;
    if (ACT == ACT_RELU2) return z > 0.0f ? z * z : 0.0f;
    const float u = ACT == ACT_GELU_TANH ? 1.5957691216057308f * (z + 0.044715f * z * z * z) : z;  // (1 + tanh(u / 2)) / 2 = sigmoid(u)
    const float g = __fdividef(1.0f, 1.0f + __expf(-u));
    return ACT == ACT_SIGMOID ? g : z * g;
}
// Where a warp finds its sums: an accumulator, or the parts that the splits of k left in memory, added in their order.
struct DgSums {
    uint32_t taddr;
    const float *part;   // [split][column][lane]
    uint32_t splits, stride;
    __device__ __forceinline__ void request(uint32_t g, uint32_t (&v)[16]) const {
        if (!part) {
            t5::ld16(taddr + g, v);
            return;
        }
        float x[16];
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) x[i] = __ldcg(part + (g + i) * 32);
        for (uint32_t s = 1; s < splits; s++)
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) x[i] += __ldcg(part + (size_t)s * stride + (g + i) * 32);
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) v[i] = __float_as_uint(x[i]);
    }
    __device__ __forceinline__ void arrived() const {
        if (!part) t5::wait_ld();
    }
};
template <int NT, uint32_t ACT, uint32_t STORE>  // NT tokens from t0 on
__device__ __forceinline__ void epilogue_row(const DenseEpiSeg &seg, uint32_t row, bool row_ok, const DgSums &sums, uint32_t t0, uint32_t rows) {
    const float bias = seg.bias && row_ok ? __ldg(seg.bias + row) : 0.0f, mul = seg.mul;
    const uint32_t pitch = seg.pitch;
    bf16 *yh = reinterpret_cast<bf16 *>(seg.p) + (size_t)t0 * pitch + row;
    float *yf = reinterpret_cast<float *>(seg.p) + (size_t)t0 * pitch + row;
    const uint32_t n = rows > t0 ? min(rows - t0, (uint32_t)NT) : 0;
#pragma unroll 1
    for (uint32_t g = 0; g < n; g += 16) {
        uint32_t v[16];
        float old[16];
        sums.request(g, v);
        if (STORE == ST_RESID) {
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) old[i] = row_ok && g + i < n ? yf[(size_t)(g + i) * pitch] : 0.0f;
        }
        sums.arrived();
#pragma unroll
        for (uint32_t i = 0; i < 16; i++) {
            const float y = act_fast<ACT>(__uint_as_float(v[i]) + bias) * mul;
            if (row_ok && g + i < n) {
                if (STORE == ST_ACT) yh[(size_t)(g + i) * pitch] = __float2bfloat16_rn(y);
                else yf[(size_t)(g + i) * pitch] = STORE == ST_RESID ? old[i] + y : y;
            }
        }
        __syncwarp();  // the next TMEM read takes the whole warp
    }
}

template <int NT>
__device__ __forceinline__ void epilogue(const DenseEpiSeg &seg, uint32_t row, bool row_ok, const DgSums &sums, uint32_t t0, uint32_t t_end) {
    switch (seg.store * 8 + seg.act) {
    case ST_ACT * 8 + ACT_NONE: epilogue_row<NT, ACT_NONE, ST_ACT>(seg, row, row_ok, sums, t0, t_end); break;
    case ST_ACT * 8 + ACT_SILU: epilogue_row<NT, ACT_SILU, ST_ACT>(seg, row, row_ok, sums, t0, t_end); break;
    case ST_ACT * 8 + ACT_SIGMOID: epilogue_row<NT, ACT_SIGMOID, ST_ACT>(seg, row, row_ok, sums, t0, t_end); break;
    case ST_ACT * 8 + ACT_GELU_TANH: epilogue_row<NT, ACT_GELU_TANH, ST_ACT>(seg, row, row_ok, sums, t0, t_end); break;
    case ST_ACT * 8 + ACT_RELU2: epilogue_row<NT, ACT_RELU2, ST_ACT>(seg, row, row_ok, sums, t0, t_end); break;
    case ST_F32 * 8 + ACT_NONE: epilogue_row<NT, ACT_NONE, ST_F32>(seg, row, row_ok, sums, t0, t_end); break;
    default: epilogue_row<NT, ACT_NONE, ST_RESID>(seg, row, row_ok, sums, t0, t_end); break;  // the launcher rejects the rest
    }
}

template <int NT, bool MOE>
__global__ void __launch_bounds__(DgCfg<NT>::THREADS, 1) dense_gemm_tc5_kernel(const DgArgs a, const __grid_constant__ CUtensorMap xmap,
                                                                                   const __grid_constant__ CUtensorMap xmap2) {
    using C = DgCfg<NT>;
    extern __shared__ uint8_t dg_smem_raw[];
    uint8_t *smem = dg_smem_raw + (1024 - ((uint32_t)__cvta_generic_to_shared(dg_smem_raw) & 1023u)) % 1024;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    pdl_launch_dependents();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t b_full = base + C::BAR_OFF, b_empty = b_full + 8 * C::S, b_dfull = b_empty + 8 * C::S, b_dempty = b_dfull + 16;
    const uint32_t state = C::BAR_OFF + 8 * (2 * C::S + 4);
    volatile uint32_t *err_flag = reinterpret_cast<volatile uint32_t *>(smem + state);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + state + 8);
    uint32_t n_items = a.n_rt * a.n_tt;
    uint32_t *tile_end = reinterpret_cast<uint32_t *>(smem + C::TAB_OFF), *row_end = tile_end + a.experts;  // experts: running sums of tiles and rows
    if (tid == 0) {
        for (int s = 0; s < C::S; s++) { t5::mbar_init(b_full + 8 * s, 1); t5::mbar_init(b_empty + 8 * s, 1); }
        for (int b = 0; b < 2; b++) { t5::mbar_init(b_dfull + 8 * b, 1); t5::mbar_init(b_dempty + 8 * b, 4); }
        *err_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) t5::tmem_alloc(base + state + 8, C::TMEM_COLS);
    t5::fence_before();
    __syncthreads();
    t5::fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);
    pdl_wait();  // before any bounded wait: the kernel before this one may still be at work
    if (MOE) {
        if (warp == 2) dg_expert_table<NT>(a, tile_end, row_end, lane);
        __syncthreads();
        n_items = a.n_rt * tile_end[a.experts - 1];
    }

    if (warp == 0) {
        if (lane == 0) {
            uint32_t n = 0;
            for (uint32_t w = blockIdx.x; w < n_items; w += gridDim.x) {
                const DgItem it = dg_locate<NT, 1, MOE>(a, w, tile_end, row_end);
                const DenseEpiSeg &seg = dense_seg(a.epi, it.rt * 128);
                const uint32_t kb = seg.k / 64;
                const CUtensorMap *map = seg.in ? &xmap2 : &xmap;
                const uint8_t *wsrc = a.w + (size_t)it.wt * a.kb * DG_A_BYTES;
                for (uint32_t k = 0; k < kb; k++, n++) {
                    const uint32_t s = n % C::S, ph = (n / C::S) & 1, dst = base + s * C::STAGE;
                    t5::mbar_wait_bounded(b_empty + 8 * s, ph ^ 1, err_flag);
                    t5::mbar_arrive_expect_tx(b_full + 8 * s, C::STAGE);
                    t5::bulk_g2s(dst, wsrc + (size_t)k * DG_A_BYTES, DG_A_BYTES, b_full + 8 * s);
                    t5::tma_2d(dst + C::A_BYTES, map, (int32_t)(k * 64), (int32_t)it.t0, b_full + 8 * s);
                }
            }
            // every copy in flight lands before the CTA leaves (a stage's last use is committed to its empty barrier)
            for (uint32_t i = 0; i < (uint32_t)C::S && i < n; i++) {
                const uint32_t m = n - 1 - i, s = m % C::S;
                t5::mbar_wait_bounded(b_full + 8 * s, (m / C::S) & 1, err_flag);
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the stages, so that descriptors stay in uniform registers, and one elected lane issues; the
        // test of the next stage's barrier is under way while the products of this one are issued.
        const uint32_t idesc = t5::idesc_f16(128, NT) | a.types;
        uint32_t n = 0, ti = 0, ready = 0;
        for (uint32_t w = blockIdx.x; w < n_items; w += gridDim.x, ti++) {
            const DgItem it = dg_locate<NT, 1, MOE>(a, w, tile_end, row_end);
            const uint32_t kb = dense_seg(a.epi, it.rt * 128).k / 64, d = tmem + (ti & 1) * NT;
            t5::mbar_wait_bounded(b_dempty + 8 * (ti & 1), ((ti >> 1) & 1) ^ 1, err_flag);
            for (uint32_t k = 0; k < kb; k++, n++) {
                const uint32_t s = n % C::S, sa = base + s * C::STAGE, sb = sa + C::A_BYTES;
                if (!ready) t5::mbar_wait_bounded(b_full + 8 * s, (n / C::S) & 1, err_flag);
                ready = t5::mbar_test(b_full + 8 * ((n + 1) % C::S), ((n + 1) / C::S) & 1);
                __syncwarp();
                t5::fence_after();
                if (t5::elect_one()) {
#pragma unroll
                    for (int j = 0; j < 4; j++)  // 16 k each: two k/8 slabs of 2 KB in A, 32 bytes inside the swizzled rows of B
                        t5::mma_ss(d, t5::smem_desc(sa + j * 4096, 2048, 128), t5::desc_swizzled<128>(sb + j * 32), idesc, j ? 1u : k);
                    t5::commit(b_empty + 8 * s);
                }
            }
            if (t5::elect_one()) t5::commit(b_dfull + 8 * (ti & 1));
        }
    } else {
        const uint32_t q = warp & 3;  // the TMEM lanes a warp may read
        uint32_t ti = 0;
        for (uint32_t w = blockIdx.x; w < n_items; w += gridDim.x, ti++) {
            const DgItem it = dg_locate<NT, 1, MOE>(a, w, tile_end, row_end);
            const uint32_t b = ti & 1, row0 = it.rt * 128;
            const DenseEpiSeg &seg = dense_seg(a.epi, row0);
            const uint32_t row = row0 + q * 32 + lane - seg.row0;
            t5::mbar_wait_warp(b_dfull + 8 * b, (ti >> 1) & 1, err_flag);
            t5::fence_after();
            epilogue<NT>(seg, row, row < seg.rows, DgSums{tmem + ((q * 32) << 16) + b * NT, nullptr, 1, 0}, it.t0, it.t_end);
            t5::fence_before();
            __syncwarp();
            if (lane == 0) t5::mbar_arrive(b_dempty + 8 * b);
        }
    }
    t5::fence_before();
    __syncthreads();
    t5::fence_after();
    if (warp == 1) t5::tmem_dealloc(tmem, C::TMEM_COLS);
    if (tid == 0 && *err_flag) atomicExch(a.err, 5u);
}

template <int NT, bool MOE>
__global__ void __launch_bounds__(DpCfg<NT>::THREADS, 1) dense_gemm_pair_kernel(const DgArgs a, const __grid_constant__ CUtensorMap wmap,
                                                                                const __grid_constant__ CUtensorMap xmap,
                                                                                const __grid_constant__ CUtensorMap xmap2) {
    using C = DpCfg<NT>;
    extern __shared__ uint8_t dg_smem_raw[];
    uint8_t *smem = dg_smem_raw + (1024 - ((uint32_t)__cvta_generic_to_shared(dg_smem_raw) & 1023u)) % 1024;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem), rank = t5::cluster_rank();
    pdl_launch_dependents();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    // full and dempty: the pair's, in CTA 0 (it issues the products); empty and dfull: each CTA's own
    const uint32_t b_full = base + C::BAR_OFF, b_empty = b_full + 8 * C::S, b_dfull = b_empty + 8 * C::S, b_dempty = b_dfull + 16;
    const uint32_t state = C::BAR_OFF + 8 * (2 * C::S + 4);
    volatile uint32_t *err_flag = reinterpret_cast<volatile uint32_t *>(smem + state);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + state + 8);
    uint32_t n_items = a.n_rt * a.n_tt * a.splits;
    uint32_t *tile_end = reinterpret_cast<uint32_t *>(smem + C::TAB_OFF), *row_end = tile_end + a.experts;
    if (tid == 0) {
        for (int s = 0; s < C::S; s++) { t5::mbar_init(b_full + 8 * s, 1); t5::mbar_init(b_empty + 8 * s, 1); }
        for (int b = 0; b < 2; b++) { t5::mbar_init(b_dfull + 8 * b, 1); t5::mbar_init(b_dempty + 8 * b, 16); }
        *err_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) t5::tmem_alloc_pair(base + state + 8, C::TMEM_COLS);
    t5::fence_before();
    __syncthreads();
    t5::cluster_sync();  // the other CTA's barriers exist before anything arrives there
    t5::fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0), pair = blockIdx.x / 2, n_pairs = gridDim.x / 2;
    pdl_wait();  // before any bounded wait: the kernel before this one may still be at work
    if (MOE) {
        if (warp == 2) dg_expert_table<NT>(a, tile_end, row_end, lane);
        __syncthreads();
        n_items = a.n_rt * tile_end[a.experts - 1];
    }

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t full0 = t5::map_rank(b_full, 0);
            uint32_t n = 0;
            for (uint32_t w = pair; w < n_items; w += n_pairs) {
                const DgItem it = dg_locate<NT, 2, MOE>(a, w / a.splits, tile_end, row_end);
                const DenseEpiSeg &seg = dense_seg(a.epi, it.rt * 256);
                const uint32_t w0 = (it.wt + rank) * a.kb, k1 = dg_k(a, seg, w % a.splits + 1);
                const CUtensorMap *map = seg.in ? &xmap2 : &xmap;
                for (uint32_t k = dg_k(a, seg, w % a.splits); k < k1; k++, n++) {
                    const uint32_t s = n % C::S, ph = (n / C::S) & 1, dst = base + s * C::STAGE;
                    t5::mbar_wait_bounded(b_empty + 8 * s, ph ^ 1, err_flag);
                    if (rank == 0) t5::mbar_arrive_expect_tx(b_full + 8 * s, 2 * C::STAGE);
                    t5::tma_2d_pair(dst, &wmap, 0, (int32_t)((w0 + k) * 32), full0 + 8 * s);
                    t5::tma_2d_pair(dst + DG_A_BYTES, map, (int32_t)(k * 64), (int32_t)(it.t0 + rank * (NT / 2)), full0 + 8 * s);
                }
            }
            // every copy in flight lands before the CTA leaves: a stage is given back after its products
            for (uint32_t i = 0; i < (uint32_t)C::S && i < n; i++) {
                const uint32_t m = n - 1 - i, s = m % C::S;
                t5::mbar_wait_bounded(b_empty + 8 * s, (m / C::S) & 1, err_flag);
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {  // as in dense_gemm_tc5_kernel
            const uint32_t idesc = t5::idesc_f16(256, NT) | a.types;
            uint32_t n = 0, ti = 0, ready = 0;
            for (uint32_t w = pair; w < n_items; w += n_pairs, ti++) {
                const DgItem it = dg_locate<NT, 2, MOE>(a, w / a.splits, tile_end, row_end);
                const DenseEpiSeg &seg = dense_seg(a.epi, it.rt * 256);
                const uint32_t kb = dg_k(a, seg, w % a.splits + 1) - dg_k(a, seg, w % a.splits), d = tmem + (ti & 1) * NT;
                t5::mbar_wait_bounded(b_dempty + 8 * (ti & 1), ((ti >> 1) & 1) ^ 1, err_flag);
                for (uint32_t k = 0; k < kb; k++, n++) {
                    const uint32_t s = n % C::S, sa = base + s * C::STAGE, sb = sa + DG_A_BYTES;
                    if (!ready) t5::mbar_wait_bounded(b_full + 8 * s, (n / C::S) & 1, err_flag);
                    ready = t5::mbar_test(b_full + 8 * ((n + 1) % C::S), ((n + 1) / C::S) & 1);
                    __syncwarp();
                    t5::fence_after();
                    if (t5::elect_one()) {
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            t5::mma_ss_pair(d, t5::smem_desc(sa + j * 4096, 2048, 128), t5::desc_swizzled<128>(sb + j * 32), idesc, j ? 1u : k);
                        t5::commit_pair(b_empty + 8 * s);
                    }
                }
                if (t5::elect_one()) t5::commit_pair(b_dfull + 8 * (ti & 1));
            }
        }
    } else {
        const uint32_t q = warp & 3, half = (warp - 2) >> 2, dempty0 = t5::map_rank(b_dempty, 0);
        uint32_t ti = 0;
        for (uint32_t w = pair; w < n_items; w += n_pairs, ti++) {
            const DgItem it = dg_locate<NT, 2, MOE>(a, w / a.splits, tile_end, row_end);
            const uint32_t b = ti & 1, row0 = (it.rt * 2 + rank) * 128;
            const DenseEpiSeg &seg = dense_seg(a.epi, row0);
            const uint32_t row = row0 + q * 32 + lane - seg.row0;
            t5::mbar_wait_warp(b_dfull + 8 * b, (ti >> 1) & 1, err_flag);
            t5::fence_after();
            DgSums sums{tmem + ((q * 32) << 16) + b * NT + half * (NT / 2), nullptr, 1, 0};
            const uint32_t t0 = it.t0 + half * (NT / 2);
            if (MOE || a.splits == 1) {
                epilogue<NT / 2>(seg, row, row < seg.rows, sums, t0, it.t_end);
                t5::fence_before();
                __syncwarp();
                if (lane == 0) t5::mbar_arrive_remote(dempty0 + 8 * b);
                continue;
            }
            constexpr uint32_t PART = NT / 2 * 32;  // floats of a warp
            float *mine = a.part + (((size_t)w * 2 + rank) * 8 + (warp - 2)) * PART + lane;
#pragma unroll 1
            for (uint32_t g = 0; g < NT / 2; g += 16) {
                uint32_t v[16];
                t5::ld16(sums.taddr + g, v);
                t5::wait_ld();
#pragma unroll
                for (uint32_t i = 0; i < 16; i++) __stcg(mine + (g + i) * 32, __uint_as_float(v[i]));
            }
            t5::fence_before();
            __threadfence();
            __syncwarp();
            uint32_t before = 0;
            if (lane == 0) {
                t5::mbar_arrive_remote(dempty0 + 8 * b);
                before = atomicAdd(a.arrived + ((size_t)(w / a.splits) * 2 + rank) * 8 + (warp - 2), 1u);
            }
            if (__shfl_sync(0xFFFFFFFFu, before, 0) == a.splits - 1) {
                __threadfence();
                if (lane == 0) a.arrived[((size_t)(w / a.splits) * 2 + rank) * 8 + (warp - 2)] = 0;
                sums.part = a.part + (((size_t)(w - w % a.splits) * 2 + rank) * 8 + (warp - 2)) * PART + lane;
                sums.splits = a.splits;
                sums.stride = 16 * PART;
                epilogue<NT / 2>(seg, row, row < seg.rows, sums, t0, it.t_end);
            }
        }
    }
    t5::fence_before();
    __syncthreads();
    t5::cluster_sync();  // nothing arrives in a CTA that has left
    t5::fence_after();
    if (warp == 1) t5::tmem_dealloc_pair(tmem, C::TMEM_COLS);
    if (tid == 0 && *err_flag) atomicExch(a.err, 5u);
}

// ---- host side ---------------------------------------------------------------------------------
static int encode_2d(prism_cuda_ctx *ctx, CUtensorMap *map, const void *p, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_cols, uint32_t box_rows,
                     bool swizzle) {
    return encode_tensor_map(ctx, map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p, cols, rows, pitch, box_cols, box_rows,
                             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
}
static int encode_inputs(prism_cuda_ctx *ctx, const DgArgs &a, const DenseIn &in, uint32_t box_rows, CUtensorMap *map, CUtensorMap *map2) {
    uint32_t k[2] = {0, 0};  // columns of each input that a segment reads
    for (uint32_t i = 0; i < a.epi.n; i++) k[a.epi.s[i].in] = std::max(k[a.epi.s[i].in], a.epi.s[i].k);
    PRISM_TRY(encode_2d(ctx, map, in.x, std::max(k[0], 64u), a.rows, in.pitch, 64, box_rows, true));
    if (k[1]) return encode_2d(ctx, map2, in.x2, k[1], a.rows, in.pitch2, 64, box_rows, true);
    *map2 = *map;
    return PRISM_OK;
}
// Tiles of a launch on `slots` resident CTAs (or pairs of them).
template <int NT, bool MOE>
static uint32_t dg_tiles(DgArgs &a, uint32_t n_rt, uint32_t slots) {
    a.n_rt = n_rt;
    if (MOE) {
        a.n_tt = a.rows / NT + std::min(a.rows, a.experts);  // at most
    } else {
        a.n_tt = (a.rows + NT - 1) / NT;
        a.rt_group = std::min(a.n_rt, std::max(1u, (slots + a.n_tt - 1) / a.n_tt));
    }
    return std::min(slots, a.n_rt * a.n_tt * a.splits);
}

template <int NT, bool MOE>
static int launch_dg(prism_cuda_ctx *ctx, const DenseLinear &l, DgArgs &a, const DenseIn &in) {
    using C = DgCfg<NT>;
    const size_t smem = C::SMEM + (MOE ? 8 * DG_MAX_EXPERTS : 0);
    static bool configured[PRISM_MAX_DEVICES] = {false};
    if (!configured[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(dense_gemm_tc5_kernel<NT, MOE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured[ctx->device] = true;
    }
    CUtensorMap map, map2;
    PRISM_TRY(encode_inputs(ctx, a, in, NT, &map, &map2));
    const uint32_t grid = dg_tiles<NT, MOE>(a, l.n_tiles, (uint32_t)ctx->sm_count);
    launch_pdl(ctx, "dense_gemm_tc5_kernel", dense_gemm_tc5_kernel<NT, MOE>, dim3(grid), dim3(C::THREADS), smem, a, map, map2);
    return after_launch(ctx, "dense_gemm_tc5_kernel");
}

template <int NT, bool MOE>
static int launch_dp(prism_cuda_ctx *ctx, const DenseLinear &l, DgArgs &a, const DenseIn &in) {
    using C = DpCfg<NT>;
    const size_t smem = C::SMEM + (MOE ? 8 * DG_MAX_EXPERTS : 0);
    static int pairs[PRISM_MAX_DEVICES] = {0};  // pairs that are resident at once (a GPC with an odd number of SMs leaves one idle)
    if (!pairs[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(dense_gemm_pair_kernel<NT, MOE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const int n = resident_clusters(dense_gemm_pair_kernel<NT, MOE>, 2, C::THREADS, smem, 2 * ((uint32_t)ctx->sm_count / 2));
        pairs[ctx->device] = std::max(1, std::min(n, ctx->sm_count / 2));
    }
    CUtensorMap wmap, map, map2;
    PRISM_TRY(encode_2d(ctx, &wmap, a.w, 256, l.bytes() / 512, 256, 256, 32, false));  // 32 rows of 512 bytes: the 16 KB run of a stage
    PRISM_TRY(encode_inputs(ctx, a, in, NT / 2, &map, &map2));
    const uint32_t grid = dg_tiles<NT, MOE>(a, (l.n_tiles + 1) / 2, (uint32_t)pairs[ctx->device]);
    if (a.splits > 1) {
        const size_t tiles = (size_t)a.n_rt * a.n_tt;
        PRISM_TRY(ensure_splitk(ctx, tiles * a.splits * 256 * NT, tiles * 16));
        a.part = ctx->splitk_partials;
        a.arrived = ctx->splitk_counters;
    }
    launch_cluster_pdl(ctx, dense_gemm_pair_kernel<NT, MOE>, dim3(2 * grid), dim3(C::THREADS), smem, 2u, a, wmap, map, map2);
    return after_launch(ctx, "dense_gemm_pair_kernel");
}

// Tile shape, and for pairs of CTAs the number of ranges k is cut into, with the least estimated time: waves x 64-k
// stages x cycles of a stage, which the tensor core bounds by 2 NT (both kernels: a pair does twice the rows on two SMs)
// and the loads by what L2 delivers to the CTAs at work (about 6000 bytes per cycle in all).  A split pays for its sums'
// way through L2 and the wait for the last of them.  `tt(nt)`: token tiles of nt rows.
constexpr size_t DG_PART_MAX = 64u << 20;  // bytes of partial sums
template <bool MOE, typename F>
static int launch_best(prism_cuda_ctx *ctx, const DenseLinear &l, DgArgs &a, const DenseIn &in, F &&tt) {
    struct Shape { uint32_t nt, rt; };
    static const Shape shapes[] = {{256, 2}, {128, 2}, {64, 2}, {256, 1}, {128, 1}, {64, 1}, {32, 1}, {16, 1}};
    const uint32_t G = (uint32_t)ctx->sm_count;
    uint32_t k_min = ~0u, k_max = 0;
    for (uint32_t i = 0; i < a.epi.n; i++) {
        k_min = std::min(k_min, a.epi.s[i].k / 64);
        k_max = std::max(k_max, a.epi.s[i].k / 64);
    }
    Shape best{16, 1};
    double best_t = 1e30;
    a.splits = 1;
    for (const Shape &s : shapes) {
        // a pair of row tiles lies inside an expert; with few rows of x an expert's weights stream, and the pair, whose two
        // halves wait for each other at every stage, streams slower than two CTAs (16 experts x 25 rows: 3 % of a pass)
        if (MOE && s.rt == 2 && (l.n_tiles % 2 || s.nt < 128)) continue;
        const uint64_t tiles = (uint64_t)((l.n_tiles + s.rt - 1) / s.rt) * tt(s.nt), slots = G / s.rt;
        for (uint32_t cut = 1; cut <= 8; cut++) {
            if (cut > 1 && (MOE || s.rt == 1 || k_min < 8 * cut || tiles * cut * 256 * s.nt * 4 > DG_PART_MAX)) break;
            const uint64_t items = tiles * cut;
            const double bytes = DG_A_BYTES + s.nt * 128.0 / s.rt, act = (double)std::min<uint64_t>(items, slots) * s.rt;
            double t = (double)((items + slots - 1) / slots) * ((k_max + cut - 1) / cut) * std::max({2.0 * s.nt, bytes * act / 6000.0, bytes / 100.0});
            if (cut > 1) t += 4000.0 + items * s.nt * 2048.0 / 6000.0;
            if (t < best_t * 0.999) {
                best_t = t;
                best = s;
                a.splits = cut;
            }
        }
    }
    switch (best.nt * 4 + best.rt) {
    case 256 * 4 + 2: return launch_dp<256, MOE>(ctx, l, a, in);
    case 128 * 4 + 2: return launch_dp<128, MOE>(ctx, l, a, in);
    case 64 * 4 + 2: return launch_dp<64, MOE>(ctx, l, a, in);
    case 256 * 4 + 1: return launch_dg<256, MOE>(ctx, l, a, in);
    case 128 * 4 + 1: return launch_dg<128, MOE>(ctx, l, a, in);
    case 64 * 4 + 1: return launch_dg<64, MOE>(ctx, l, a, in);
    case 32 * 4 + 1: return launch_dg<32, MOE>(ctx, l, a, in);
    default: return launch_dg<16, MOE>(ctx, l, a, in);
    }
}

static int dg_args(prism_cuda_ctx *ctx, const DenseLinear &l, const DenseIn &in, const DenseOut *outs, uint32_t rows, DgArgs &a) {
    a.w = reinterpret_cast<const uint8_t *>(l.w);
    a.kb = l.k_pad / 64;
    a.rows = rows;
    a.err = ctx->dev_err;
    a.types = 1u << 7 | 1u << 10;  // A and B bf16
    a.epi = dense_epi(l, outs);
    for (uint32_t i = 0; i < l.n_segs; i++) {
        const DenseEpiSeg &s = a.epi.s[i];
        const void *x = s.in ? in.x2 : in.x;
        const uint32_t pitch = s.in ? in.pitch2 : in.pitch;
        if (!x || (reinterpret_cast<uintptr_t>(x) & 15) || pitch % 8 || pitch < s.k || s.k % 64)
            return fail(ctx, PRISM_E_ARG, "dense gemm: input rows must be 16-byte aligned and hold the padded k range");
        if (i && (s.in != a.epi.s[i - 1].in || s.k != a.epi.s[i - 1].k) && s.row0 % 256)
            return fail(ctx, PRISM_E_ARG, "dense gemm: a segment with another input must start on an even row tile");
        if (s.store != ST_ACT && s.act != ACT_NONE) return fail(ctx, PRISM_E_ARG, "dense gemm: fp32 outputs take no activation");
    }
    return PRISM_OK;
}

int launch_dense_gemm_tc5(prism_cuda_ctx *ctx, const DenseLinear &l, const DenseIn &in, const DenseOut *outs, uint32_t rows) {
    DgArgs a{};
    PRISM_TRY(dg_args(ctx, l, in, outs, rows, a));
    return launch_best<false>(ctx, l, a, in, [&](uint32_t nt) { return (rows + nt - 1) / nt; });
}

int launch_moe_gemm_tc5(prism_cuda_ctx *ctx, const DenseLinear &l, const MoePlan &plan, const DenseIn &in, const DenseOut &out, uint32_t pairs) {
    if (plan.experts > DG_MAX_EXPERTS || l.n_segs != 1) return fail(ctx, PRISM_E_ARG, "experts: at most 1024 of them");
    DgArgs a{};
    PRISM_TRY(dg_args(ctx, l, in, &out, pairs, a));
    a.experts = plan.experts;
    a.count = plan.count;
    // as if the rows were spread evenly over the experts, plus half a tile each for the ragged ends
    return launch_best<true>(ctx, l, a, in, [&](uint32_t nt) {
        const uint32_t used = std::min(pairs, plan.experts), each = (pairs + used - 1) / used;
        return used * ((each + each / 4 + nt - 1) / nt);
    });
}

}  // namespace prism
