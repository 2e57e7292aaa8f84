// Fused attention of one decode step: RoPE of q (and of k where the profile asks for it), append
// of the new token's k/v to the fp16 cache, and attention over the cached positions, in ONE
// kernel.  It stands for four nodes of step() (src/lut/engine_impl.rs:1076-1459): Rope(q),
// Rope(k), KVCache::append and Attention (attention_cpu, src/lut/cpu_fallback.rs:84-127;
// rope_inplace, cpu_fallback.rs:131-143), with the same fp16 rounding points: q and k are rounded
// to fp16 after the rotation, the output after the weighted sum.  Scores, softmax and sums are fp32.
//
// A thread-block cluster of S CTAs serves one (KV head, sequence) and up to 8 of the query heads that
// share that KV head, so a cached row is read once per group instead of once per query head.  A WARP owns
// every (warps of the cluster)-th tile of 16 positions: it copies the tile's keys and values into its own part
// of shared memory (two tiles in flight), takes scores = K q^T (m16n8k16: 16 positions x 8 heads) and keeps
// its own running maximum, sum and O^T = V^T p^T; the weights (at most 1) enter that product 2^15-fold as two fp16 parts:
// 21 bits of the fp32 weight down to 2^-18 of the largest, below that to 2^-38 of it, so that keys beside one that takes
// nearly all the weight keep theirs, both positive, so that an infinite value stays one.  So no warp waits for another until the end, where every warp stores its maximum, sum and O
// into the shared memory of the CTA that finishes those outputs, and ONE cluster barrier later they are merged in
// a fixed order.
// Bound: the latency of that chain (dependency wait, rotation, two products, merge) for the contexts of a chat, the
// cache's bytes for long ones.  A launch inside a step, against one warp per cached row, tiles staged by the whole CTA in
// turn and three cluster barriers: 14 heads over 2 of 64 at 160 positions 6.8 -> 4.6 us; 64 over 8 of 128 at 530 13.5 -> 6.3;
// 8 sequences, 28 over 4 of 128, at 215 23.3 -> 6.4; one at 8 200 118 -> 16.8.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "attn_plan.hpp"
#include "common.cuh"
#include "tensor_map.cuh"

namespace cg = cooperative_groups;

namespace prism {

constexpr uint32_t FA_ROWS = 16;     // positions of a tile
constexpr uint32_t FA_MAX_S = 16;    // CTAs of a cluster
constexpr float FA_PARTS = 32768.0f; // weights, at most 1, times this are what the fp16 parts hold
template <int HD>
struct FaCfg {
    static constexpr int WARPS = HD == 256 ? 4 : 8;
    static constexpr int THREADS = WARPS * 32;
    static constexpr int MT = HD / 16;                      // 16-element pieces of a head
    static constexpr int PPR = HD / 8;                      // 16-byte pieces of a row
    static constexpr int TILE = FA_ROWS * HD * 2;           // bytes of a key (or value) tile
    static constexpr int Q_OFF = WARPS * 4 * TILE;          // [8][HD] rotated q, [HD] new k, [HD] new v
    static constexpr int ML_OFF = Q_OFF + 10 * HD * 2;      // [entries][8] maxima, then sums, then weights
    // per warp of the cluster: the O pieces this CTA finishes, 128 floats each
    static __host__ __device__ constexpr uint32_t pieces(uint32_t S) { return (MT + S - 1) / S; }
    static __host__ __device__ constexpr size_t smem(uint32_t S) { return ML_OFF + (size_t)S * WARPS * (3 * 8 * 4 + pieces(S) * 512); }
};

__device__ __forceinline__ float fa_h2f(uint16_t v) { return __half2float(__ushort_as_half(v)); }
__device__ __forceinline__ uint16_t fa_f2h(float v) { return __half_as_ushort(__float2half_rn(v)); }

struct FusedAttnArgs {
    const uint16_t *q, *k, *v;  // this step's projections: rows of nh*hd / nkv*hd halfs, src_stride apart
    uint32_t src_stride;
    uint16_t *kc, *vc;          // fp16 cache of this layer slot: [seq][slot][nkv*hd]
    uint16_t *out;              // [batch][nh*hd]
    const int32_t *pos_dev;     // token position (device scalar, so a captured graph can be replayed)
    uint32_t slot_mul, slot_add;  // cache slot of the new token = pos*slot_mul + slot_add
    uint32_t nh, nkv, batch;
    uint64_t seq_stride;        // halfs between sequences in the cache
    uint32_t max_seq;           // slots per sequence
    uint32_t gt;                // query heads of a cluster, at most 8
    uint32_t rope_k;
    const float *inv_freq;      // [hd/2] rotation frequencies base^(-2j/hd), computed once on the host
    // Paged cache: position p of cache sequence c lives in row (page_tbl[c*tbl_stride + (p >> page_shift)]
    // << page_shift) + (p & (page - 1)) of the layer's page pool; nullptr: one contiguous slab per sequence.
    const int32_t *page_tbl;
    uint32_t page_shift, tbl_stride;
    uint32_t early_cache;       // 1: the kernel before this one in the stream does not write the cache (see the kernel)
};

// Row (in units of cached rows of the layer) of position p of cache sequence c.
__device__ __forceinline__ size_t fa_row(const int32_t *__restrict__ tbl, uint32_t shift, uint32_t tbl_stride, uint64_t seq_rows,
                                         uint32_t c, uint32_t p) {
    if (tbl == nullptr) return (size_t)c * seq_rows + p;
    const uint32_t page = (uint32_t)__ldg(tbl + (size_t)c * tbl_stride + (p >> shift));
    return ((size_t)page << shift) + (p & ((1u << shift) - 1u));
}

// cos / sin of the rotation of the VEC elements a lane owns (elements lane*VEC .. +VEC-1 of a head
// of 32*VEC): the angle depends on the position and the pair index only, so it is computed once
// and applied to every query head and to k.
template <int VEC>
__device__ __forceinline__ void fa_rope_angles(float (&ca)[VEC], float (&sa)[VEC], uint32_t lane, float pos,
                                               const float *__restrict__ inv_freq) {
    constexpr uint32_t half = 16 * VEC;
#pragma unroll
    for (int i = 0; i < VEC; i++) {
        const uint32_t d = lane * VEC + i;
        const uint32_t j = d < half ? d : d - half;
        const float ang = pos * __ldg(inv_freq + j);
        sincosf(ang, &sa[i], &ca[i]);
    }
}

// Rotates a lane's elements; the partner element j +- hd/2 lives in lane ^ 16.
template <int VEC>
__device__ __forceinline__ void fa_rope_apply(float (&x)[VEC], const float (&ca)[VEC], const float (&sa)[VEC], uint32_t lane) {
    constexpr uint32_t half = 16 * VEC;
#pragma unroll
    for (int i = 0; i < VEC; i++) {
        const float other = __shfl_xor_sync(0xFFFFFFFFu, x[i], 16);
        const uint32_t d = lane * VEC + i;
        // d < half: (a, b) = (mine, other) -> a*cos - b*sin;  else (a, b) = (other, mine) -> a*sin + b*cos
        const float r = d < half ? __fsub_rn(__fmul_rn(x[i], ca[i]), __fmul_rn(other, sa[i]))
                                 : __fadd_rn(__fmul_rn(other, sa[i]), __fmul_rn(x[i], ca[i]));
        x[i] = fa_h2f(fa_f2h(r));
    }
}

// 16-byte asynchronous copy global -> shared
__device__ __forceinline__ void fa_cp16(uint32_t dst_smem, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void fa_ldm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void fa_ldm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void fa_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t fa_transpose(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
    return r;
}
// Two weights, FA_PARTS-fold, as an fp16 pair rounded down and what is left over as another.  Both parts of a positive weight
// are positive (at least the smallest fp16 value, 2^-39 of the largest weight), so that an infinite value times the one and the
// other has one sign and is no NaN.
__device__ __forceinline__ void fa_split(float a, float b, uint32_t &hi, uint32_t &lo) {
    a *= FA_PARTS;
    b *= FA_PARTS;
    const uint32_t least = (a > 0.0f ? 1u : 0u) | (b > 0.0f ? 0x10000u : 0u);
    const __half2 floor2 = *reinterpret_cast<const __half2 *>(&least);
    uint32_t d;
    asm("cvt.rz.f16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(b), "f"(a));  // the first source goes to the upper half
    const __half2 h = *reinterpret_cast<const __half2 *>(&d);
    const float2 f = __half22float2(h);
    const __half2 l = __hmax2_nan(__floats2half2_rn(a - f.x, b - f.y), floor2), h1 = __hmax2_nan(h, floor2);
    hi = *reinterpret_cast<const uint32_t *>(&h1);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

template <int HD>
__global__ void __launch_bounds__(FaCfg<HD>::THREADS) attn_fused_kernel(const FusedAttnArgs a) {
    using C = FaCfg<HD>;
    constexpr int VEC = HD / 32, W = C::WARPS, MT = C::MT, PPR = C::PPR;
    pdl_launch_dependents();
    // first half of a cluster barrier that only says "this CTA has started": its second half stands before the
    // first store into a peer's shared memory and has long completed by then
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t S = cluster.dim_blocks().x, rank = cluster.block_rank(), E = S * W;
    extern __shared__ __align__(16) uint8_t fa_smem[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.y;
    uint16_t *qs = reinterpret_cast<uint16_t *>(fa_smem + C::Q_OFF), *newk = qs + 8 * HD, *newv = newk + HD;
    float *mx_all = reinterpret_cast<float *>(fa_smem + C::ML_OFF), *sum_all = mx_all + E * 8, *wgt = sum_all + E * 8;
    float *recv = wgt + E * 8;                     // [entry][piece][lane][4]
    const uint32_t tiles_at = (uint32_t)__cvta_generic_to_shared(fa_smem) + warp * 4 * C::TILE;  // stage s: keys at 2 s, values at 2 s + 1
    const uint32_t g = a.nh / a.nkv, n_ht = (g + a.gt - 1) / a.gt, kvd = a.nkv * HD;
    const uint32_t cl = blockIdx.x / S, kh = cl / n_ht, ht = cl - kh * n_ht;
    const uint32_t h0 = kh * g + ht * a.gt;        // first query head of this cluster
    const uint32_t nhl = min(a.gt, g - ht * a.gt);
    uint16_t *kcb = a.kc + (size_t)kh * HD;
    uint16_t *vcb = a.vc + (size_t)kh * HD;
    const uint64_t seq_rows = a.seq_stride / kvd;  // rows of a sequence's slab (contiguous cache)
    auto row_of = [&](uint32_t p) { return fa_row(a.page_tbl, a.page_shift, a.tbl_stride, seq_rows, b, p) * kvd; };
    auto place_of = [](uint32_t r, uint32_t c) { return r * (HD * 2) + ((PPR >= 8 ? c ^ (r & 7) : c ^ ((r >> 1) & 3)) << 4); };

    // Everything that follows from the token position: the positions seen, where the new row goes.
    const uint32_t entry = warp * S + rank;        // of the cluster's warps: neighbouring tiles lie on different SMs
    int32_t pos;
    bool have_new;
    uint32_t sl, new_slot, n_tiles;
    auto place = [&](int32_t pos_now) {
        pos = pos_now;
        const int64_t slot64 = (int64_t)pos * a.slot_mul + a.slot_add;
        have_new = slot64 >= 0 && slot64 < (int64_t)a.max_seq;  // a full cache takes no new row
        sl = slot64 < 0 ? 0 : (uint32_t)min(slot64 + 1, (int64_t)a.max_seq);
        new_slot = have_new ? (uint32_t)slot64 : 0xFFFFFFFFu;
        n_tiles = (sl + FA_ROWS - 1) / FA_ROWS;
    };
    // a tile's rows into stage s; rows past the end are zero, the new token's row comes later
    auto fetch = [&](uint32_t t, uint32_t s) {
        if (t < n_tiles) {
            const uint32_t kt = tiles_at + s * 2 * C::TILE;
#pragma unroll
            for (uint32_t i = lane; i < FA_ROWS * PPR; i += 32) {
                const uint32_t r = i / PPR, c = i % PPR, p = t * FA_ROWS + r, at = kt + place_of(r, c);
                if (p >= sl) {
                    asm volatile("st.shared.v4.u32 [%0], {%2,%2,%2,%2};\nst.shared.v4.u32 [%1], {%2,%2,%2,%2};\n" ::"r"(at), "r"(at + C::TILE), "r"(0u) : "memory");
                } else if (p != new_slot) {
                    const size_t ro = row_of(p) + c * 8;
                    fa_cp16(at, kcb + ro);
                    fa_cp16(at + C::TILE, vcb + ro);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // A decode step's predecessor in the stream (the q/k/v projection) does not touch the cache, and the rows
    // below the new token's were written steps ago: with `early_cache` the first tiles are requested and the
    // rotation angles computed BEFORE the dependency wait, on the position as it reads now.  The position is
    // read again after the wait; should it have changed (the kernel that advances it had not finished yet),
    // the speculative tiles are dropped and everything is placed again.
    const volatile int32_t *pos_ptr = a.pos_dev;
    const bool early = a.early_cache;
    if (!early) pdl_wait();
    const int32_t pos_seen = *pos_ptr;
    place(pos_seen);
    fetch(entry, 0);
    fetch(entry + E, 1);
    float ca[VEC], sa[VEC];
    fa_rope_angles<VEC>(ca, sa, lane, (float)pos, a.inv_freq);
    if (early) {
        pdl_wait();
        const int32_t pos_now = *pos_ptr;
        if (pos_now != pos_seen) {                 // uniform in a warp only (others may have read the old position): nothing here waits for more
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            place(pos_now);
            fetch(entry, 0);
            fetch(entry + E, 1);
            fa_rope_angles<VEC>(ca, sa, lane, (float)pos, a.inv_freq);
        }
    }

    // ---- rotation: warp w prepares query heads w, w + W, ...; the last warp also the new token's k and v ----
    for (uint32_t hh = warp; hh < 8; hh += W) {
        float x[VEC];
        const uint16_t *q = a.q + (size_t)b * a.src_stride + (size_t)(h0 + hh) * HD + lane * VEC;
#pragma unroll
        for (int i = 0; i < VEC; i++) x[i] = hh < nhl ? fa_h2f(q[i]) : 0.0f;
        fa_rope_apply<VEC>(x, ca, sa, lane);
#pragma unroll
        for (int i = 0; i < VEC; i++) qs[hh * HD + lane * VEC + i] = fa_f2h(x[i]);
    }
    const uint32_t new_tile = new_slot / FA_ROWS;
    if (warp == W - 1) {
        float kn[VEC];
        const uint16_t *k = a.k + (size_t)b * a.src_stride + (size_t)kh * HD + lane * VEC;
        const uint16_t *v = a.v + (size_t)b * a.src_stride + (size_t)kh * HD + lane * VEC;
#pragma unroll
        for (int i = 0; i < VEC; i++) kn[i] = fa_h2f(k[i]);
        if (a.rope_k) fa_rope_apply<VEC>(kn, ca, sa, lane);
        const bool append = have_new && ht == 0 && rank == new_tile % S;
        const size_t new_off = append ? row_of(new_slot) : 0;
#pragma unroll
        for (int i = 0; i < VEC; i++) {
            const uint16_t kb = fa_f2h(kn[i]), vb = v[i];
            newk[lane * VEC + i] = kb;
            newv[lane * VEC + i] = vb;
            // KVCache::append: the first head tile of a group stores the row for all later steps
            if (append) {
                kcb[new_off + lane * VEC + i] = kb;
                vcb[new_off + lane * VEC + i] = vb;
            }
        }
    }
    __syncthreads();

    // ---- this warp's tiles ---------------------------------------------------------------------------
    const uint32_t mat = lane >> 3, hp = (lane & 3) * 2;  // the lane's heads: hp, hp + 1
    uint32_t qf[MT][2];                                   // q^T, 16 elements at a time
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const uint16_t *src = qs + (lane >> 2) * HD + i * 16 + hp;
        qf[i][0] = *reinterpret_cast<const uint32_t *>(src);
        qf[i][1] = *reinterpret_cast<const uint32_t *>(src + 8);
    }
    const float scale2 = 1.4426950408889634f / sqrtf((float)HD);
    float o[MT][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int c = 0; c < 4; c++) o[i][c] = 0.0f;
    uint32_t st = 0;
    for (uint32_t t = entry; t < n_tiles; t += E, st ^= 1) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        const uint32_t kt = tiles_at + st * 2 * C::TILE, vt = kt + C::TILE;
        if (have_new && t == new_tile)
            for (uint32_t c = lane; c < PPR; c += 32) {
                const uint4 kv = reinterpret_cast<const uint4 *>(newk)[c], vv = reinterpret_cast<const uint4 *>(newv)[c];
                const uint32_t at = kt + place_of(new_slot % FA_ROWS, c);
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(at), "r"(kv.x), "r"(kv.y), "r"(kv.z), "r"(kv.w) : "memory");
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(at + C::TILE), "r"(vv.x), "r"(vv.y), "r"(vv.z), "r"(vv.w) : "memory");
            }
        __syncwarp();
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < MT; i++) {
            uint32_t k4[4];
            fa_ldm(k4, kt + place_of(lane & 15, 2 * i + (lane >> 4)));
            fa_mma(i & 1 ? s2 : s, k4, qf[i][0], qf[i][1]);
        }
        const uint32_t p0 = t * FA_ROWS + (lane >> 2);
        float w[4];
#pragma unroll
        for (int c = 0; c < 4; c++) w[c] = p0 + (c >> 1) * 8 < sl ? (s[c] + s2[c]) * scale2 : -INFINITY;
        float f[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            float top = fmaxf(w[j], w[2 + j]);
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, x));
            top = fmaxf(top, m[j]);
            const float sub = top == -INFINITY ? 0.0f : top;  // nothing but scores of -inf so far: weights 0
            f[j] = exp2f(m[j] - sub);
            m[j] = top;
            w[j] = exp2f(w[j] - sub);
            w[2 + j] = exp2f(w[2 + j] - sub);
            l[j] = l[j] * f[j] + (w[j] + w[2 + j]);
        }
        uint32_t hi[2], lo[2];
        fa_split(w[0], w[1], hi[0], lo[0]);
        fa_split(w[2], w[3], hi[1], lo[1]);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            hi[j] = fa_transpose(hi[j]);
            lo[j] = fa_transpose(lo[j]);
        }
#pragma unroll
        for (int i = 0; i < MT; i++) {
            uint32_t v4[4];
            fa_ldm_t(v4, vt + place_of((lane & 7) + (mat >> 1) * 8, 2 * i + (mat & 1)));
#pragma unroll
            for (int c = 0; c < 4; c++) o[i][c] *= f[c & 1];
            fa_mma(o[i], v4, hi[0], hi[1]);
            fa_mma(o[i], v4, lo[0], lo[1]);
        }
        __syncwarp();                              // the whole warp is done with the stage
        fetch(t + 2 * E, st);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");

    // ---- merge: every warp that had a tile stores its part where it is finished ----------------------
    const uint32_t used = min(E, n_tiles), per = C::pieces(S);
    asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
    if (entry < used) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) l[j] += __shfl_xor_sync(0xFFFFFFFFu, l[j], x);
        for (uint32_t r = lane >> 2; r < S; r += 8) {
            *reinterpret_cast<float2 *>(cluster.map_shared_rank(mx_all + entry * 8 + hp, r)) = make_float2(m[0], m[1]);
            *reinterpret_cast<float2 *>(cluster.map_shared_rank(sum_all + entry * 8 + hp, r)) = make_float2(l[0], l[1]);
        }
#pragma unroll
        for (int i = 0; i < MT; i++) {
            const uint32_t owner = i / per;
            *reinterpret_cast<float4 *>(cluster.map_shared_rank(recv + ((size_t)(entry * per + (i - owner * per)) * 32 + lane) * 4, owner)) =
                make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
        }
    }
    cluster.sync();                                // nobody touches a peer's memory after this barrier
    for (uint32_t hh = warp; hh < 8; hh += W) {
        float top = -INFINITY, sum = 0.0f;
        for (uint32_t e = lane; e < used; e += 32) top = fmaxf(top, mx_all[e * 8 + hh]);
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, x));
        for (uint32_t e = lane; e < used; e += 32) {
            const float f = exp2f(mx_all[e * 8 + hh] - top);
            wgt[e * 8 + hh] = f;
            sum += sum_all[e * 8 + hh] * f;
        }
#pragma unroll
        for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, x);
        const float inv = 1.0f / (sum + 1e-10f);
        __syncwarp();
        for (uint32_t e = lane; e < used; e += 32) wgt[e * 8 + hh] *= inv * (1.0f / FA_PARTS);
    }
    __syncthreads();
    const uint32_t own = rank * per < (uint32_t)MT ? min(per, MT - rank * per) : 0;
    for (uint32_t t = threadIdx.x; t < own * 128; t += C::THREADS) {
        const uint32_t i = t >> 7, ln = (t >> 2) & 31, c = t & 3, hh = (ln & 3) * 2 + (c & 1);
        float v = 0.0f;
        for (uint32_t e = 0; e < used; e++) v += recv[(size_t)(e * per + i) * 128 + (t & 127)] * wgt[e * 8 + hh];
        if (hh < nhl) a.out[(size_t)b * a.nh * HD + (size_t)(h0 + hh) * HD + (rank * per + i) * 16 + (ln >> 2) + (c >> 1) * 8] = fa_f2h(v);
    }
}

bool attn_fused_eligible(const AttnArgs &a) {
    return !a.int8 && (a.hd == 32 || a.hd == 64 || a.hd == 128 || a.hd == 256) && a.pos_dev != nullptr &&
           a.nkv != 0 && a.nh % a.nkv == 0 && (a.seq_stride * 2) % 16 == 0 &&
           reinterpret_cast<uintptr_t>(a.k) % 16 == 0 && reinterpret_cast<uintptr_t>(a.v) % 16 == 0;
}

template <int HD>
static int launch_attn_fused_hd(prism_cuda_ctx *ctx, FusedAttnArgs &fa) {
    using C = FaCfg<HD>;
    const uint32_t g = fa.nh / fa.nkv;
    fa.gt = std::min(8u, g);
    if (ctx->attn_group > 0) fa.gt = std::min(fa.gt, (uint32_t)ctx->attn_group);
    const uint32_t clusters = fa.nkv * ((g + fa.gt - 1) / fa.gt) * fa.batch;
    static int resident16[PRISM_MAX_DEVICES] = {0};  // plus one; 0: not asked yet
    if (!resident16[ctx->device]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(attn_fused_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(C::smem(1), C::smem(FA_MAX_S))));
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(attn_fused_kernel<HD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        const int n = resident_clusters(attn_fused_kernel<HD>, FA_MAX_S, C::THREADS, C::smem(FA_MAX_S), FA_MAX_S);
        resident16[ctx->device] = 1 + n;
    }
    uint32_t S = attn_cluster_ctas((uint32_t)ctx->sm_count, clusters, fa.max_seq, C::WARPS * FA_ROWS, (uint32_t)resident16[ctx->device] - 1);
    if (ctx->attn_cluster == 1 || ctx->attn_cluster == 2 || ctx->attn_cluster == 4 || ctx->attn_cluster == 8)
        S = (uint32_t)ctx->attn_cluster;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters / fa.batch * S, fa.batch);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::smem(S);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 2 : 1;
    (void)cudaLaunchKernelEx(&cfg, attn_fused_kernel<HD>, fa);
    return after_launch(ctx, "attn_fused_kernel");
}

// The rotation frequencies base^(-2j/hd), j < hd/2, as the CPU path computes them (powf in fp32,
// cpu_fallback.rs:137), once per (head size, base) on the host and kept on the device.
int rope_table(prism_cuda_ctx *ctx, uint32_t hd, float base, const float **out) {
    for (auto *t : ctx->rope_tabs) {
        if (t->hd == hd && t->base == base) {
            *out = t->dev;
            return PRISM_OK;
        }
    }
    auto *t = new prism_cuda_ctx::RopeTab{hd, base, nullptr, {0}};
    cudaError_t e = cudaMalloc((void **)&t->dev, 128 * sizeof(float));
    if (e != cudaSuccess) {
        delete t;
        return cuda_fail(ctx, e, "cudaMalloc(rope table)");
    }
    for (uint32_t j = 0; j < hd / 2; j++) t->host[j] = powf(base, -2.0f * (float)j / (float)hd);
    ctx->rope_tabs.push_back(t);
    // the host copy lives as long as the context, so the asynchronous copy may read it after this returns
    PRISM_CUDA_TRY(ctx, cudaMemcpyAsync(t->dev, t->host, (hd / 2) * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
    *out = t->dev;
    return PRISM_OK;
}

// q_src/k_src/v_src: this step's projection rows (src_stride halfs apart); a.k / a.v: the cache.
int launch_attn_fused(prism_cuda_ctx *ctx, const AttnArgs &a, const uint16_t *k_src, const uint16_t *v_src,
                      uint32_t rope_k, float rope_base) {
    if (!attn_fused_eligible(a)) return fail(ctx, PRISM_E_ARG, "fused attention: fp16 cache and head_dim 32/64/128/256 only");
    FusedAttnArgs fa{};
    fa.q = a.q; fa.k = k_src; fa.v = v_src; fa.src_stride = a.q_stride;
    fa.kc = static_cast<uint16_t *>(const_cast<void *>(a.k));
    fa.vc = static_cast<uint16_t *>(const_cast<void *>(a.v));
    fa.out = a.out;
    fa.pos_dev = a.pos_dev; fa.slot_mul = a.slot_mul; fa.slot_add = a.slot_add;
    fa.nh = a.nh; fa.nkv = a.nkv; fa.batch = a.batch;
    fa.seq_stride = a.seq_stride; fa.max_seq = a.max_seq;
    fa.rope_k = rope_k;
    fa.page_tbl = a.page_tbl; fa.page_shift = a.page_shift; fa.tbl_stride = a.tbl_stride;
    fa.early_cache = a.early_cache;
    PRISM_TRY(rope_table(ctx, a.hd, rope_base, &fa.inv_freq));
    switch (a.hd) {
    case 32: return launch_attn_fused_hd<32>(ctx, fa);
    case 64: return launch_attn_fused_hd<64>(ctx, fa);
    case 128: return launch_attn_fused_hd<128>(ctx, fa);
    default: return launch_attn_fused_hd<256>(ctx, fa);
    }
}

}  // namespace prism
