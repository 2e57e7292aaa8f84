// Attention of a portion of a prompt on tcgen05 / TMEM: causal softmax attention of T consecutive tokens of each of
// n_seq sequences over the fp16 cache, after their rotated keys and values were appended to it (rope_inplace and
// attention_cpu, src/lut/cpu_fallback.rs:84-143, once per token in the reference).  fp16 q, k, v; fp32 scores,
// softmax and sums.
//
//   prefill_rope_kernel   rotates q in place and k into the cache, copies v: one block per token, so the angles of a
//                         position are computed once for all its heads.
//   prefill_attn_kernel   a CTA takes one query head and QT tiles of 128 query rows (two for heads up to 128 wide: while
//                         the softmax warps of one tile work, the tensor core has the other's products).  Keys and
//                         values come by TMA, 128 positions a stage, straight from the cache (page by page when it is
//                         paged).  S = Q K^T goes to TMEM; a thread owns one query row, so the softmax needs no
//                         exchange; the weights go back to TMEM over the scores they came from, 2^12-fold as TWO fp16
//                         parts (22 bits of each weight down to 2^-15 of the maximum in use, below that to 2^-37 of it,
//                         so that keys beside one that takes nearly all the weight keep theirs) and meet V, read from
//                         shared memory along its rows, in two products each.
//                         The running maximum is only moved when it grows by more than 2^3: O is rescaled a few
//                         times per row tile instead of at every key tile, and a weight is at most 2^15 in the parts.
// Bound: the tensor core -- per 128 x 128 tile and 128-wide head three products of 2*128^3 flops, about 1 570 cycles,
// against about 1 000 for the 16 384 exponentials.  Masked positions carry weight 0; value rows past the portion's
// end (stale cache) are zeroed in shared memory before the product, so no stale NaN meets a zero weight.  A value row of a later
// token that overflowed still does, and an attended one meets the second part of its weight, which may be 0 or negative; scores of
// -inf may leave a row's first tile without a maximum.  Each of these ends in a NaN or an infinity, and a row with one is taken again
// position by position in fp32 over what it may see (pa_plain_row), so a later token's overflow stays out of earlier ones.
// Measured, 28 query / 4 KV heads of 128: the attention of an 8190-token prompt through two layers took 128 ms with one
// cluster of the decode kernel per token, on the CUDA cores; this kernel took 1.87 ms with a single issuing thread (descriptors
// through vector registers), 1.38 with a whole warp walking the tiles.
#include <algorithm>

#include "common.cuh"
#include "tc5_ptx.cuh"
#include "tensor_map.cuh"

namespace prism {

constexpr int PA_K = 128;  // keys of a stage
// A score may lie PA_GROW (in powers of two) above the maximum in use before that is moved; the fp16 parts hold the weights times
// PA_PARTS: at most 2^PA_GROW * PA_PARTS = 2^15.
constexpr float PA_GROW = 3.0f, PA_PARTS = 4096.0f;
template <int HD>
struct PaCfg {
    static constexpr int QT = HD <= 128 ? 2 : 1;           // query tiles of 128 rows
    static constexpr int ROWB = HD >= 64 ? 128 : 64;       // bytes of a swizzled row; wider heads are panels of 64 elements
    static constexpr int PANELS = HD * 2 / ROWB;
    static constexpr int PANEL = 128 * ROWB, TILE = PANELS * PANEL;
    static constexpr int ST = HD == 256 ? 1 : HD == 128 ? 2 : 3;  // stages of keys, and as many of values
    static constexpr int THREADS = QT * 128 + 64;
    static constexpr int K_OFF = QT * TILE, V_OFF = K_OFF + ST * TILE, BAR_OFF = V_OFF + ST * TILE;
    // barriers: kfull[ST], kempty[ST], vfull[ST], vempty[ST], sfull[2], pfull[2], ofull[2], qfull
    static constexpr int STATE_OFF = BAR_OFF + 8 * (4 * ST + 7);
    static constexpr size_t SMEM = STATE_OFF + 16 + 1024;
};

struct PrefillAttnDev {
    uint32_t T, pos0, nh, group;     // tokens and first position of every sequence's portion, query heads, query heads per KV head
    uint32_t seq0;                   // cache sequence of the first one
    uint32_t seq_rows;               // cached rows per sequence (contiguous cache)
    uint32_t box;                    // rows of a copy: 128, or the page where it is smaller
    const int32_t *page_tbl;
    uint32_t page_shift, tbl_stride;
    float scale2;                    // log2(e) / sqrt(head size)
    const uint16_t *q, *kc, *vc;     // rotated queries (rows q_stride apart) and the cache, for the rows taken again
    uint32_t q_stride;
    uint16_t *out;                   // [n_seq * T][nh * HD]
    unsigned int *err;
};

namespace {

__device__ __forceinline__ float pa_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
// Two weights, PA_PARTS-fold, as an fp16 pair (first in the low half) and what that rounding left over as another.
__device__ __forceinline__ void pa_split(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a * PA_PARTS, b * PA_PARTS);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(fmaf(a, PA_PARTS, -f.x), fmaf(b, PA_PARTS, -f.y));
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// Row of the cache that holds position p of cache sequence c.
__device__ __forceinline__ size_t pa_row(const PrefillAttnDev &a, uint32_t c, uint32_t p) {
    if (!a.page_tbl) return (size_t)c * a.seq_rows + p;
    return ((size_t)__ldg(a.page_tbl + (size_t)c * a.tbl_stride + (p >> a.page_shift)) << a.page_shift) + (p & ((1u << a.page_shift) - 1u));
}
// One token's output for one head by one warp, position by position in fp32: a lane takes the scores of every 32nd position and
// HD / 32 columns.  About 20 instructions a position; only rows with infinities or NaN come here.
template <int HD>
__device__ __noinline__ void pa_plain_row(const PrefillAttnDev &a, uint32_t token, uint32_t cseq, uint32_t pos, uint32_t h, uint32_t lane) {
    constexpr uint32_t VEC = HD / 32;
    const uint32_t kh = h / a.group, kvd = a.nh / a.group * HD;
    const uint16_t *q = a.q + (size_t)token * a.q_stride + (size_t)h * HD;
    auto score = [&](uint32_t p) {
        if (p > pos) return -INFINITY;
        const uint4 *k = reinterpret_cast<const uint4 *>(a.kc + pa_row(a, cseq, p) * kvd + (size_t)kh * HD);
        float d = 0.0f;
#pragma unroll 2
        for (uint32_t i = 0; i < HD / 8; i++) {
            const uint4 qv = reinterpret_cast<const uint4 *>(q)[i], kv = k[i];
            const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w}, kw[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&qw[j])), y = __half22float2(*reinterpret_cast<const __half2 *>(&kw[j]));
                d += x.x * y.x;
                d += x.y * y.y;
            }
        }
        return d / sqrtf((float)HD);
    };
    float top = -INFINITY, sum = 0.0f;
    for (uint32_t p = lane; p <= pos; p += 32) top = fmaxf(top, score(p));
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, x));
    for (uint32_t p = lane; p <= pos; p += 32) sum += expf(score(p) - top);
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, x);
    const float inv = 1.0f / (sum + 1e-10f);
    float acc[VEC];
#pragma unroll
    for (uint32_t i = 0; i < VEC; i++) acc[i] = 0.0f;
    for (uint32_t p0 = 0; p0 <= pos; p0 += 32) {
        const float mine = expf(score(p0 + lane) - top);
        for (uint32_t j = 0; j < 32 && p0 + j <= pos; j++) {
            const float e = __shfl_sync(0xFFFFFFFFu, mine, j);
            const uint16_t *v = a.vc + pa_row(a, cseq, p0 + j) * kvd + (size_t)kh * HD + lane;
#pragma unroll
            for (uint32_t i = 0; i < VEC; i++) acc[i] += e * __half2float(__ushort_as_half(v[i * 32])) * inv;
        }
    }
    uint16_t *dst = a.out + (size_t)token * a.nh * HD + (size_t)h * HD + lane;
#pragma unroll
    for (uint32_t i = 0; i < VEC; i++) dst[i * 32] = __half_as_ushort(__float2half_rn(acc[i]));
}

}  // namespace

template <int HD>
__global__ void __launch_bounds__(PaCfg<HD>::THREADS, 1) prefill_attn_kernel(const __grid_constant__ PrefillAttnDev a, const __grid_constant__ CUtensorMap qmap,
                                                                             const __grid_constant__ CUtensorMap kmap,
                                                                             const __grid_constant__ CUtensorMap vmap) {
    using C = PaCfg<HD>;
    constexpr int ST = C::ST, QT = C::QT;
    extern __shared__ uint8_t pa_raw[];
    uint8_t *smem = pa_raw + (1024 - ((uint32_t)__cvta_generic_to_shared(pa_raw) & 1023u)) % 1024;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
    pdl_launch_dependents();
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0);
    const uint32_t b_kfull = base + C::BAR_OFF, b_kempty = b_kfull + 8 * ST, b_vfull = b_kempty + 8 * ST, b_vempty = b_vfull + 8 * ST,
                   b_sfull = b_vempty + 8 * ST, b_pfull = b_sfull + 16, b_ofull = b_pfull + 16, b_qfull = b_ofull + 16;
    volatile uint32_t *err_flag = reinterpret_cast<volatile uint32_t *>(smem + C::STATE_OFF);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::STATE_OFF + 8);
    if (tid == 0) {
        for (int s = 0; s < ST; s++) {
            t5::mbar_init(b_kfull + 8 * s, 1); t5::mbar_init(b_kempty + 8 * s, 1);
            t5::mbar_init(b_vfull + 8 * s, 1); t5::mbar_init(b_vempty + 8 * s, 1);
        }
        for (int q = 0; q < 2; q++) { t5::mbar_init(b_sfull + 8 * q, 1); t5::mbar_init(b_pfull + 8 * q, 4); t5::mbar_init(b_ofull + 8 * q, 1); }
        t5::mbar_init(b_qfull, 1);
        *err_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == QT * 4) t5::tmem_alloc(base + C::STATE_OFF + 8, 512);
    t5::fence_before();
    __syncthreads();
    t5::fence_after();
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *tmem_slot, 0);  // S of tile q at column 128 q, O at 256 + HD q
    pdl_wait();                        // before any bounded wait: the kernel before this one may still be at work

    const uint32_t h = blockIdx.x, kh = h / a.group, sq = blockIdx.y, qb = (gridDim.z - 1 - blockIdx.z) * (QT * 128);
    const uint32_t kv_end = a.pos0 + a.T;  // cached positions of the sequence
    uint32_t n_kt[2] = {0, 0};             // key tiles a query tile sees
#pragma unroll
    for (uint32_t q = 0; q < (uint32_t)QT; q++)
        if (qb + q * 128 < a.T) n_kt[q] = (a.pos0 + min(a.T, qb + q * 128 + 128) + PA_K - 1) / PA_K;
    const uint32_t n = max(n_kt[0], n_kt[1]);

    if (warp < QT * 4) {
        // ================= softmax: thread = query row =================
        const uint32_t q = warp >> 2, row = (warp & 3) * 32 + lane, lanes = ((warp & 3) * 32) << 16;
        const uint32_t s_col = tmem + lanes + q * 128, o_col = tmem + lanes + 256 + q * HD;
        const uint32_t qpos = a.pos0 + qb + q * 128 + row, wpos = qpos - lane;
        float m = -INFINITY, l = 0.0f;
        for (uint32_t j = 0; j < n_kt[q]; j++) {
            if (lane == 0) t5::mbar_wait_bounded(b_sfull + 8 * q, j & 1, err_flag);
            __syncwarp();
            t5::fence_after();
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; c++) t5::ld32(s_col + c * 32, s[c]);
            t5::wait_ld();
            const uint32_t k0 = j * PA_K;
            if (k0 + PA_K - 1 > wpos) {  // some row of the warp does not see the whole tile
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (k0 + c * 32 + i > qpos) s[c][i] = 0xFF800000u;
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                mx[c] = __uint_as_float(s[c][0]);
#pragma unroll
                for (int i = 1; i < 32; i++) mx[c] = fmaxf(mx[c], __uint_as_float(s[c][i]));
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale2;
            const bool grow = top > m + PA_GROW;  // the first tile: m is -inf (every row sees its position 0)
            if (j == 0) {
                m = top;
            } else if (__any_sync(0xFFFFFFFFu, grow)) {
                // the products of the tile before are complete: the scores that were just waited for follow them
                const float f = grow ? pa_ex2(m - top) : 1.0f;
                if (grow) m = top;
                l *= f;
#pragma unroll 1
                for (int c = 0; c < HD / 32; c++) {
                    uint32_t o[32];
                    t5::ld32(o_col + c * 32, o);
                    t5::wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                    t5::st32(o_col + c * 32, o);
                }
            }
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float e0 = pa_ex2(fmaf(__uint_as_float(s[c][2 * i]), a.scale2, -m));
                    const float e1 = pa_ex2(fmaf(__uint_as_float(s[c][2 * i + 1]), a.scale2, -m));
                    sum[i & 3] += e0 + e1;
                    pa_split(e0, e1, hi[i], lo[i]);
                }
                t5::st16(s_col + c * 16, hi);
                t5::st16(s_col + 64 + c * 16, lo);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            t5::wait_st();
            t5::fence_before();
            if (lane == 0) t5::mbar_arrive(b_pfull + 8 * q);
        }
        if (n_kt[q]) {
            t5::mbar_wait_warp(b_ofull + 8 * q, 0, err_flag);
            t5::fence_after();
            const float inv = 1.0f / (l * PA_PARTS);
            const uint32_t t = qb + q * 128 + row;
            uint16_t *dst = a.out + ((size_t)sq * a.T + t) * a.nh * HD + (size_t)h * HD;
            float odd = 0.0f;  // NaN once an output was not finite
#pragma unroll 1
            for (int c = 0; c < HD / 32; c++) {
                uint32_t o[32];
                t5::ld32(o_col + c * 32, o);
                t5::wait_ld();
                uint32_t p[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float x = __uint_as_float(o[2 * i]) * inv, y = __uint_as_float(o[2 * i + 1]) * inv;
                    const __half2 v = __floats2half2_rn(x, y);
                    p[i] = *reinterpret_cast<const uint32_t *>(&v);
                    odd = fmaf(x, 0.0f, fmaf(y, 0.0f, odd));
                }
                if (t < a.T) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        reinterpret_cast<uint4 *>(dst + c * 32)[i] = make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]);
                }
                __syncwarp();  // the next TMEM read takes the whole warp
            }
            for (uint32_t rows = __ballot_sync(0xFFFFFFFFu, t < a.T && odd != 0.0f); rows; rows &= rows - 1) {
                const uint32_t r = __ffs(rows) - 1, tr = t - lane + r;
                pa_plain_row<HD>(a, sq * a.T + tr, a.seq0 + sq, a.pos0 + tr, h, lane);
            }
        }
        t5::fence_before();
    } else if (warp == QT * 4) {
        // ================= copies =================
        if (lane == 0) {
            t5::mbar_arrive_expect_tx(b_qfull, (n_kt[1] ? 2 : 1) * C::TILE);
            for (uint32_t q = 0; q < (uint32_t)QT; q++)
                if (n_kt[q])
                    for (uint32_t p = 0; p < (uint32_t)C::PANELS; p++)
                        t5::tma_2d(base + q * C::TILE + p * C::PANEL, &qmap, (int32_t)(h * HD + p * (C::ROWB / 2)), (int32_t)(sq * a.T + qb + q * 128), b_qfull);
            auto load = [&](const CUtensorMap *map, uint32_t dst, uint32_t k0, uint32_t mbar) {
                const uint32_t rows = min((uint32_t)PA_K, kv_end - k0), boxes = (rows + a.box - 1) / a.box;
                t5::mbar_arrive_expect_tx(mbar, boxes * a.box * HD * 2);
                for (uint32_t b = 0; b < boxes; b++) {
                    const uint32_t pos = k0 + b * a.box;
                    uint32_t r = (a.seq0 + sq) * a.seq_rows + pos;
                    if (a.page_tbl) {
                        const uint32_t page = (uint32_t)__ldg(a.page_tbl + (size_t)(a.seq0 + sq) * a.tbl_stride + (pos >> a.page_shift));
                        r = (page << a.page_shift) + (pos & ((1u << a.page_shift) - 1u));
                    }
                    for (uint32_t p = 0; p < (uint32_t)C::PANELS; p++)
                        t5::tma_2d(dst + p * C::PANEL + b * a.box * C::ROWB, map, (int32_t)(kh * HD + p * (C::ROWB / 2)), (int32_t)r, mbar);
                }
            };
            for (uint32_t j = 0; j < n; j++) {
                const uint32_t st = j % ST, ph = (j / ST) & 1;
                t5::mbar_wait_bounded(b_kempty + 8 * st, ph ^ 1, err_flag);
                load(&kmap, base + C::K_OFF + st * C::TILE, j * PA_K, b_kfull + 8 * st);
                t5::mbar_wait_bounded(b_vempty + 8 * st, ph ^ 1, err_flag);
                load(&vmap, base + C::V_OFF + st * C::TILE, j * PA_K, b_vfull + 8 * st);
            }
            // every copy in flight lands before the CTA leaves
            t5::mbar_wait_bounded(b_qfull, 0, err_flag);
            for (uint32_t j = n > (uint32_t)ST ? n - ST : 0; j < n; j++) {
                t5::mbar_wait_bounded(b_kfull + 8 * (j % ST), (j / ST) & 1, err_flag);
                t5::mbar_wait_bounded(b_vfull + 8 * (j % ST), (j / ST) & 1, err_flag);
            }
        }
        __syncwarp();
    } else {
        // ================= products: the whole warp walks the tiles (descriptors stay in uniform registers), an elected lane
        // issues; all lanes clear stale value rows =================
        const uint32_t id_s = t5::idesc_f16(128, PA_K), id_o = t5::idesc_f16(128, HD) | (1u << 16);  // V is read across its rows
        auto scores = [&](uint32_t q, uint32_t j) {
            const uint32_t qa = base + q * C::TILE, ka = base + C::K_OFF + (j % ST) * C::TILE;
#pragma unroll
            for (int k = 0; k < HD / 16; k++) {
                const uint32_t off = (k * 32 / C::ROWB) * C::PANEL + (k * 32) % C::ROWB;
                t5::mma_ss(tmem + q * 128, t5::desc_swizzled<C::ROWB>(qa + off, 16), t5::desc_swizzled<C::ROWB>(ka + off, 16), id_s, k != 0);
            }
            t5::commit(b_sfull + 8 * q);
        };
        t5::mbar_wait_bounded(b_qfull, 0, err_flag);
        t5::mbar_wait_bounded(b_kfull, 0, err_flag);
        __syncwarp();
        t5::fence_after();
        if (t5::elect_one()) {
            for (uint32_t q = 0; q < (uint32_t)QT; q++)
                if (n_kt[q]) scores(q, 0);
            t5::commit(b_kempty);
        }
        __syncwarp();
        for (uint32_t j = 0; j < n; j++) {
            const uint32_t st = j % ST, ph = (j / ST) & 1, va = base + C::V_OFF + st * C::TILE, jn = j + 1;
            t5::mbar_wait_bounded(b_vfull + 8 * st, ph, err_flag);
            __syncwarp();
            if (kv_end - j * PA_K < (uint32_t)PA_K) {
                const uint32_t first = kv_end - j * PA_K, per = C::ROWB / 16, cells = (PA_K - first) * per * C::PANELS;
                for (uint32_t i = lane; i < cells; i += 32) {
                    const uint32_t p = i / ((PA_K - first) * per), r = i % ((PA_K - first) * per);
                    *reinterpret_cast<uint4 *>(smem + C::V_OFF + st * C::TILE + p * C::PANEL + first * C::ROWB + r * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
            }
            if (jn < n) t5::mbar_wait_bounded(b_kfull + 8 * (jn % ST), (jn / ST) & 1, err_flag);
#pragma unroll
            for (uint32_t q = 0; q < (uint32_t)QT; q++) {
                if (j >= n_kt[q]) continue;
                t5::mbar_wait_bounded(b_pfull + 8 * q, j & 1, err_flag);
                __syncwarp();
                t5::fence_after();
                if (t5::elect_one()) {
#pragma unroll
                    for (int part = 0; part < 2; part++)
#pragma unroll
                        for (int k = 0; k < PA_K / 16; k++)
                            t5::mma_ts(tmem + 256 + q * HD, tmem + q * 128 + part * 64 + k * 8, t5::desc_swizzled<C::ROWB>(va + k * 16 * C::ROWB, C::PANEL), id_o,
                                       part | k ? 1u : j);
                    if (jn < n_kt[q]) scores(q, jn);
                    else t5::commit(b_ofull + 8 * q);
                }
                __syncwarp();
            }
            if (t5::elect_one()) {
                t5::commit(b_vempty + 8 * st);
                if (jn < n) t5::commit(b_kempty + 8 * (jn % ST));
            }
            __syncwarp();
        }
        t5::fence_before();
    }
    __syncthreads();
    t5::fence_after();
    if (warp == QT * 4) t5::tmem_dealloc(tmem, 512);
    if (tid == 0 && *err_flag) atomicExch(a.err, 5u);
}

// Rotation of q (in place) and k (into the cache) and the copy of v, for T tokens of each of n_seq sequences: row
// blockIdx.x is token row % T of sequence row / T.  A thread turns two neighbouring pairs of a head.
__global__ void __launch_bounds__(256) prefill_rope_kernel(uint16_t *qkv, uint32_t stride, uint16_t *kc, uint16_t *vc, uint32_t nh, uint32_t nkv,
                                                           uint32_t hd, uint32_t T, uint32_t pos0, uint32_t seq0, uint32_t seq_rows, uint32_t max_seq,
                                                           uint32_t rope_k, const float *__restrict__ inv_freq,
                                                           const int32_t *__restrict__ page_tbl, uint32_t page_shift, uint32_t tbl_stride) {
    __shared__ float2 cs[128];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t t = blockIdx.x % T, seq = seq0 + blockIdx.x / T, pos = pos0 + t, half = hd / 2;
    for (uint32_t j = threadIdx.x; j < half; j += blockDim.x) {
        float s, c;
        sincosf((float)pos * __ldg(inv_freq + j), &s, &c);
        cs[j] = make_float2(c, s);
    }
    __syncthreads();
    if (pos >= max_seq) return;
    const uint32_t kvd = nkv * hd, qd = nh * hd, quads = hd / 4;
    uint16_t *row = qkv + (size_t)blockIdx.x * stride;
    size_t at = (size_t)seq * seq_rows + pos;
    if (page_tbl) at = ((size_t)__ldg(page_tbl + (size_t)seq * tbl_stride + (pos >> page_shift)) << page_shift) + (pos & ((1u << page_shift) - 1u));
    at *= kvd;
    for (uint32_t i = threadIdx.x; i < (nh + nkv) * quads; i += blockDim.x) {
        const uint32_t head = i / quads, j = 2 * (i % quads);
        uint32_t *src = reinterpret_cast<uint32_t *>(row + (size_t)head * hd + j);
        const uint32_t u = src[0], v = src[half / 2];
        uint32_t ru = u, rv = v;
        if (head < nh || rope_k) {
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u)), b = __half22float2(*reinterpret_cast<const __half2 *>(&v));
            const float2 c0 = cs[j], c1 = cs[j + 1];
            // the reference's order: two products, then their difference / sum, each rounded
            const __half2 x = __floats2half2_rn(__fsub_rn(__fmul_rn(a.x, c0.x), __fmul_rn(b.x, c0.y)), __fsub_rn(__fmul_rn(a.y, c1.x), __fmul_rn(b.y, c1.y)));
            const __half2 y = __floats2half2_rn(__fadd_rn(__fmul_rn(a.x, c0.y), __fmul_rn(b.x, c0.x)), __fadd_rn(__fmul_rn(a.y, c1.y), __fmul_rn(b.y, c1.x)));
            ru = *reinterpret_cast<const uint32_t *>(&x);
            rv = *reinterpret_cast<const uint32_t *>(&y);
        }
        uint32_t *dst = head < nh ? src : reinterpret_cast<uint32_t *>(kc + at + (size_t)(head - nh) * hd + j);
        dst[0] = ru;
        dst[half / 2] = rv;
    }
    const uint4 *vs = reinterpret_cast<const uint4 *>(row + qd + kvd);
    for (uint32_t i = threadIdx.x; i < kvd / 8; i += blockDim.x) reinterpret_cast<uint4 *>(vc + at)[i] = vs[i];
}

// ---- host side ---------------------------------------------------------------------------------
static int encode_rows(prism_cuda_ctx *ctx, CUtensorMap *map, const void *p, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_cols, uint32_t box_rows) {
    return encode_tensor_map(ctx, map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p, cols, rows, pitch, box_cols, box_rows,
                             box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
}

template <int HD>
static int launch_pa(prism_cuda_ctx *ctx, const PrefillAttnDev &d, const PrefillAttn &a) {
    using C = PaCfg<HD>;
    static bool configured[PRISM_MAX_DEVICES] = {false};
    if (!configured[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(prefill_attn_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        configured[ctx->device] = true;
    }
    CUtensorMap q, k, v;
    const uint32_t cols = C::ROWB / 2, kvd = a.nkv * HD;
    PRISM_TRY(encode_rows(ctx, &q, a.qkv, a.nh * HD, (uint64_t)a.n_seq * a.T, a.stride, cols, 128));
    PRISM_TRY(encode_rows(ctx, &k, a.kc, kvd, a.cache_rows, kvd, cols, d.box));
    PRISM_TRY(encode_rows(ctx, &v, a.vc, kvd, a.cache_rows, kvd, cols, d.box));
    const dim3 grid(a.nh, a.n_seq, (a.T + C::QT * 128 - 1) / (C::QT * 128));
    launch_pdl(ctx, "prefill_attn_kernel", prefill_attn_kernel<HD>, grid, dim3(C::THREADS), C::SMEM, d, q, k, v);
    return after_launch(ctx, "prefill_attn_kernel");
}

int launch_prefill_attn(prism_cuda_ctx *ctx, const PrefillAttn &a) {
    if (!(a.hd == 32 || a.hd == 64 || a.hd == 128 || a.hd == 256) || a.stride % 8 || (reinterpret_cast<uintptr_t>(a.qkv) & 15) ||
        (reinterpret_cast<uintptr_t>(a.kc) & 15) || (reinterpret_cast<uintptr_t>(a.vc) & 15))
        return fail(ctx, PRISM_E_ARG, "prefill attention: head_dim 32/64/128/256 and 16-byte rows only");
    const float *inv_freq = nullptr;
    PRISM_TRY(rope_table(ctx, a.hd, a.rope_base, &inv_freq));
    launch_pdl(ctx, "prefill_rope_kernel", prefill_rope_kernel, dim3(a.n_seq * a.T), dim3(256), 0, a.qkv, a.stride, a.kc, a.vc, a.nh, a.nkv, a.hd, a.T,
               a.pos0, a.seq0, a.seq_rows, a.max_seq, a.rope_k, inv_freq, a.page_tbl, a.page_shift, a.tbl_stride);
    PRISM_TRY(after_launch(ctx, "prefill_rope_kernel"));
    PrefillAttnDev d{};
    d.T = a.T; d.pos0 = a.pos0; d.nh = a.nh; d.group = a.nh / a.nkv; d.seq0 = a.seq0; d.seq_rows = a.seq_rows;
    d.page_tbl = a.page_tbl; d.page_shift = a.page_shift; d.tbl_stride = a.tbl_stride;
    d.box = a.page_tbl ? std::min(128u, 1u << a.page_shift) : 128u;
    d.scale2 = 1.4426950408889634f / sqrtf((float)a.hd);
    d.q = a.qkv; d.q_stride = a.stride; d.kc = a.kc; d.vc = a.vc;
    d.out = a.out; d.err = ctx->dev_err;
    switch (a.hd) {
    case 32: return launch_pa<32>(ctx, d, a);
    case 64: return launch_pa<64>(ctx, d, a);
    case 128: return launch_pa<128>(ctx, d, a);
    default: return launch_pa<256>(ctx, d, a);
    }
}

}  // namespace prism
