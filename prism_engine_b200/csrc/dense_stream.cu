// Dense bf16 linear of few rows, large weights: y = act(W x) for 1..8 rows as one even stream of weights per SM.
//
// The work is counted in units of 64 k of a row tile (16 KB, one run of the layout) and dealt to two CTAs per SM in equal,
// contiguous ranges, so no SM is left with a last partial wave.  One thread of a CTA keeps a ring of 6 units in flight, a bulk copy of the
// weights and a TMA box of the activations each; the first ring's weights are asked for before the dependency wait, under the
// kernels before this one.  Eight warps take 16 rows of every unit each: eight rows of a k/8 lie together, as ldmatrix reads them.
// A row tile that two or more CTAs share is finished by the warp that delivers last: sums of all contributors in the order of k.
//
// Bound: HBM.  The kernel that takes 32 rows and the whole k per CTA (dense_gemv_kernel) drains its loads at every block and leaves
// a part of its last wave idle.  That one / this, 4 rows, cold weights, us (TB/s): 33280 x 3584 52.4 / 38.7 (6.2), 3584 x 22528 46.3 / 30.5
// (5.3), 19008 x 3584 34.9 / 24.1 (5.6), 12544 x 3584 28.4 / 17.8, 42000 x 8192 143 / 110 (6.3).  One CTA per SM with 11 units in flight
// gives 4.7 TB/s however deep the ring; equal ranges of all units, ends anywhere in a tile, 43.9 for the first of these.
#include <algorithm>

#include "dense.cuh"
#include "tc5_ptx.cuh"
#include "tensor_map.cuh"

namespace prism {

constexpr int DS_CONSUMERS = 8, DS_THREADS = (DS_CONSUMERS + 1) * 32;
constexpr uint32_t DS_X = 16384, DS_STAGE = DS_X + 1024;  // 64 k of a row tile; of eight tokens, swizzled
constexpr uint32_t DS_CTAS = 2, DS_STAGES = 6, DS_RING = 1024;       // barriers before the ring, which the swizzle wants on a multiple of 1 KB
constexpr size_t DS_SMEM = DS_RING + DS_STAGES * (size_t)DS_STAGE + 1024;
static_assert(DS_STAGES * 16 <= DS_RING && DS_CTAS * (DS_SMEM + 1024) <= 228 * 1024, "shared memory");

struct DsArgs {
    const uint8_t *w;
    uint32_t k8, rows, n_units;
    uint32_t share, chunks;                              // CTAs of every row tile and its units; share 0: equal ranges of all units
    uint32_t first[DENSE_MAX_SEGS + 1];                  // units before a segment
    DenseEpi epi;
    float *part;                                         // [CTA][begins | ends a tile][warp][lane][4]
    unsigned int *arrived;                               // [row tile][warp]
    unsigned int *err;
};

namespace {
struct DsTile {
    uint32_t seg, tile, chunk, chunks, valid;            // row tile of the segment, its place in k, rows that there are
};
__device__ __forceinline__ DsTile ds_tile(const DsArgs &a, uint32_t u) {
    DsTile t;
    t.seg = 0;
    while (t.seg + 1 < a.epi.n && u >= a.first[t.seg + 1]) t.seg++;
    const DenseEpiSeg &s = a.epi.s[t.seg];
    t.chunks = s.k / 64;
    t.tile = (u - a.first[t.seg]) / t.chunks;
    t.chunk = (u - a.first[t.seg]) % t.chunks;
    t.valid = min(128u, s.rows - t.tile * 128);
    return t;
}
__device__ __forceinline__ uint32_t ds_start(const DsArgs &a, uint32_t cta) {
    if (!a.share) return (uint32_t)((uint64_t)a.n_units * cta / gridDim.x);
    return cta / a.share * a.chunks + cta % a.share * a.chunks / a.share;
}
// The CTA whose range holds unit u.
__device__ __forceinline__ uint32_t ds_owner(const DsArgs &a, uint32_t u) {
    uint32_t c = (uint32_t)((uint64_t)u * gridDim.x / a.n_units);
    while (ds_start(a, c + 1) <= u) c++;
    while (ds_start(a, c) > u) c--;
    return c;
}
// Every lane waits: what the copies wrote is visible to those that have seen the barrier's phase.
__device__ __forceinline__ void ds_wait(uint32_t addr, uint32_t parity, volatile uint32_t *err_flag) {
    for (uint32_t i = 0; !t5::mbar_try(addr, parity); i++) {
        if ((i & 15) == 15 && *err_flag) break;
        if (i == 4u << 20) {
            *err_flag = 1;
            break;
        }
    }
    __syncwarp();
}
}  // namespace

__global__ void __launch_bounds__(DS_THREADS, DS_CTAS) dense_stream_kernel(const DsArgs a, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap xmap2) {
    extern __shared__ uint8_t dsm[];
    const uint32_t base = ((uint32_t)__cvta_generic_to_shared(dsm) + 1023) & ~1023u;
    const uint32_t b_full = base, b_free = base + 8 * DS_STAGES, ring = base + DS_RING;
    __shared__ uint32_t gave_up;
    volatile uint32_t *err_flag = &gave_up;
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t u0 = ds_start(a, blockIdx.x), u1 = ds_start(a, blockIdx.x + 1);
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < DS_STAGES; s++) {
            t5::mbar_init(b_full + 8 * s, 1);
            t5::mbar_init(b_free + 8 * s, DS_CONSUMERS);
        }
        gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    if (warp == DS_CONSUMERS) {
        // =============================== copies ===============================
        DsTile t = ds_tile(a, u0);
        auto next = [&](uint32_t u) {                    // to unit u, the one after t's
            if (++t.chunk == t.chunks && u < u1) t = ds_tile(a, u);
        };
        auto weights = [&](uint32_t st) {
            if (lane) return;
            t5::mbar_arrive_expect_tx(b_full + 8 * st, DS_STAGE);
            t5::bulk_g2s(ring + st * DS_STAGE, a.w + ((size_t)(a.epi.s[t.seg].row0 / 128 + t.tile) * a.k8 + t.chunk * 8) * 2048, DS_X, b_full + 8 * st);
        };
        auto activations = [&](uint32_t st) {
            if (lane == 0) t5::tma_2d(ring + st * DS_STAGE + DS_X, a.epi.s[t.seg].in ? &xmap2 : &xmap, (int32_t)(t.chunk * 64), 0, b_full + 8 * st);
        };
        const uint32_t early = min(u1, u0 + DS_STAGES);
        for (uint32_t u = u0; u < early; u++) {
            weights(u - u0);
            next(u + 1);
        }
        pdl_wait();
        t = ds_tile(a, u0);
        for (uint32_t u = u0; u < early; u++) {
            activations(u - u0);
            next(u + 1);
        }
        for (uint32_t u = early; u < u1; u++) {
            const uint32_t n = u - u0, st = n % DS_STAGES;
            t5::mbar_wait_warp(b_free + 8 * st, (n / DS_STAGES - 1) & 1, err_flag);
            weights(st);
            activations(st);
            next(u + 1);
        }
        // every copy has landed before the CTA leaves, also when a wait was given up
        for (uint32_t n = u1 - u0 > DS_STAGES ? u1 - u0 - DS_STAGES : 0; n < u1 - u0; n++) {
            uint32_t landed = 0;
            for (uint32_t i = 0; i < 4u << 20 && !landed; i++) landed = t5::mbar_try(b_full + 8 * (n % DS_STAGES), (n / DS_STAGES) & 1);
        }
    } else {
        // =============================== products ===============================
        const uint32_t g8 = lane >> 2, t4 = lane & 3;
        // ldmatrix: lanes 0..7, 8..15, .. give the rows of four 8 x 8 matrices.  Weights: rows 0..7 and 8..15 of a k/8, then of the next;
        // tokens: four k/8
        const uint32_t mat = lane >> 3, a_off = (mat >> 1) * 2048 + (warp * 16 + (mat & 1) * 8 + (lane & 7)) * 16, x_row = DS_X + (lane & 7) * 128;
        pdl_wait();
        DsTile t = ds_tile(a, u0);
        uint32_t began = t.chunk;                        // where this CTA's part of the tile begins
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        auto store = [&](const float (&v)[4]) {
            const DenseEpiSeg &s = a.epi.s[t.seg];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t r = t.tile * 128 + warp * 16 + g8 + 8 * (i >> 1), tok = 2 * t4 + (i & 1);
                if (r < s.rows && tok < a.rows) dense_store<bf16>(s, r, tok, v[i]);
            }
        };
        for (uint32_t u = u0; u < u1; u++) {
            const uint32_t n = u - u0, st = n % DS_STAGES, at = ring + st * DS_STAGE;
            ds_wait(b_full + 8 * st, (n / DS_STAGES) & 1, err_flag);
            if (warp * 16 < t.valid) {
                uint32_t w[4][4], x[2][4];
#pragma unroll
                for (uint32_t h = 0; h < 2; h++) ldsm_x4(x[h], at + x_row + (((4 * h + mat) ^ (lane & 7)) << 4));
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) ldsm_x4(w[i], at + a_off + i * 4096);
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) mma_bf16(acc, w[i], x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1]);
            }
            __syncwarp();
            if (lane == 0) t5::mbar_arrive(b_free + 8 * st);
            const bool last = t.chunk + 1 == t.chunks;
            if (!last && u + 1 < u1) {
                t.chunk++;
                continue;
            }
            if (warp * 16 < t.valid) {
                if (last && began == 0) {
                    store(acc);
                } else {
                    const uint32_t first_unit = u - t.chunk, c0 = ds_owner(a, first_unit), c1 = ds_owner(a, first_unit + t.chunks - 1);
                    auto slot = [&](uint32_t c) { return reinterpret_cast<float4 *>(a.part) + ((size_t)(c * 2 + (c == c0)) * DS_CONSUMERS + warp) * 32 + lane; };
                    __stcg(slot(blockIdx.x), make_float4(acc[0], acc[1], acc[2], acc[3]));
                    __syncwarp();
                    unsigned int before = 0, *count = a.arrived + (size_t)(a.epi.s[t.seg].row0 / 128 + t.tile) * DS_CONSUMERS + warp;
                    if (lane == 0) {
                        __threadfence();
                        before = atomicAdd(count, 1u);
                        __threadfence();
                    }
                    before = __shfl_sync(0xFFFFFFFFu, before, 0);
                    __syncwarp();
                    if (before == c1 - c0) {
                        if (lane == 0) *count = 0;
                        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        for (uint32_t c = c0; c <= c1; c += 8) {  // eight requested together, added in order
                            float4 p[8];
#pragma unroll
                            for (uint32_t i = 0; i < 8; i++) p[i] = c + i <= c1 ? __ldcg(slot(c + i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                            for (uint32_t i = 0; i < 8; i++) { v[0] += p[i].x; v[1] += p[i].y; v[2] += p[i].z; v[3] += p[i].w; }
                        }
                        store(v);
                    }
                }
            }
            acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
            if (u + 1 < u1) t = ds_tile(a, u + 1);
            began = 0;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && gave_up) atomicExch(a.err, 7u);
}

// ---- host side ---------------------------------------------------------------------------------
bool dense_stream_ok(prism_cuda_ctx *ctx, const DenseLinear &l, const DenseIn &in, uint32_t rows) {
    if (rows == 0 || rows > DENSE_GEMV_ROWS || in.norm_w || in.f32 || l.experts != 1 || l.n_segs == 0) return false;
    if ((reinterpret_cast<uintptr_t>(l.w) | reinterpret_cast<uintptr_t>(in.x) | (uintptr_t)in.pitch * 2 | reinterpret_cast<uintptr_t>(in.x2) | (in.x2 ? (uintptr_t)in.pitch2 * 2 : 0)) & 15) return false;
    return l.valid_rows() * l.k_pad >= DENSE_STREAM_LEAST;
}

int launch_dense_stream(prism_cuda_ctx *ctx, const DenseLinear &l, const DenseIn &in, const DenseOut *outs, uint32_t rows) {
    DsArgs a{};
    a.w = reinterpret_cast<const uint8_t *>(l.w);
    a.k8 = l.k_pad / 8;
    a.rows = rows;
    a.epi = dense_epi(l, outs);
    for (uint32_t s = 0; s < l.n_segs; s++) a.first[s + 1] = a.first[s] + (a.epi.s[s].rows + 127) / 128 * (a.epi.s[s].k / 64);
    a.n_units = a.first[l.n_segs];
    a.err = ctx->dev_err;
    // Row tiles of equal length: as many CTAs for each as there are, so that a CTA has one delivery at its end and none between.
    const uint32_t slots = DS_CTAS * (uint32_t)ctx->sm_count;
    uint32_t tiles = 0;
    a.chunks = a.epi.s[0].k / 64;
    bool equal = true;
    for (uint32_t s = 0; s < l.n_segs; s++) {
        tiles += (a.epi.s[s].rows + 127) / 128;
        equal = equal && a.epi.s[s].k / 64 == a.chunks;
    }
    a.share = equal && tiles <= slots ? std::min(slots / tiles, std::max(1u, a.chunks / 4)) : 0;
    const uint32_t grid = a.share ? tiles * a.share : std::min(a.n_units, slots);
    // what any linear of fewer row tiles takes: grown once by the first of a step, not by one after the other (first step of a 7B model 1.9 -> 0.6 ms)
    PRISM_TRY(ensure_splitk(ctx, (size_t)slots * 2 * DS_CONSUMERS * 128, (size_t)std::max(l.n_tiles, slots) * DS_CONSUMERS));
    a.part = ctx->splitk_partials;
    a.arrived = ctx->splitk_counters;
    CUtensorMap xmap, xmap2;
    uint32_t cols[2] = {0, 0};                           // that the segments read of either input
    for (uint32_t s = 0; s < l.n_segs; s++) cols[a.epi.s[s].in ? 1 : 0] = std::max(cols[a.epi.s[s].in ? 1 : 0], a.epi.s[s].k);
    const DenseIn other{in.x2 ? in.x2 : in.x, in.x2 ? in.pitch2 : in.pitch};
    PRISM_TRY(encode_tensor_map(ctx, &xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, in.x, std::max(cols[0], 64u), rows, in.pitch, 64, DENSE_GEMV_ROWS, CU_TENSOR_MAP_SWIZZLE_128B));
    PRISM_TRY(encode_tensor_map(ctx, &xmap2, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, other.x, std::max(cols[1], 64u), rows, other.pitch, 64, DENSE_GEMV_ROWS, CU_TENSOR_MAP_SWIZZLE_128B));
    static bool configured[PRISM_MAX_DEVICES] = {false};
    if (!configured[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(dense_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DS_SMEM));
        configured[ctx->device] = true;
    }
    launch_pdl(ctx, "dense_stream_kernel", dense_stream_kernel, dim3(grid), dim3(DS_THREADS), DS_SMEM, a, xmap, xmap2);
    return after_launch(ctx, "dense_stream_kernel");
}

}  // namespace prism
