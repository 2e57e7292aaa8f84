// Palettized linear for few tokens (1..32):  Y[t][r] = f16( sum_k f32(X[t][k]) * f32(W[r][k]) ), with the residual or the SwiGLU
// product on the way out -- lut_gemv_cpu per activation row, as the other kernels (src/lut/engine_impl.rs:1046-1053).
//
// The palettes live in registers.  A lane holds the 16 (or 4) entries of its four rows as bytes, low ones and high ones apart;
// four index nibbles are a byte-permute selector as they stand, so one PRMT picks four low bytes of eight entries, and two more
// interleave low and high bytes into half2.  Together 2.6 integer instructions a weight at 4 bits and 1.3 at 2 bits, and what
// comes out is an A fragment of mma.sync with rows and k where the instruction wants them: eight tokens share one product, up to
// 32 the same weights.  No tables to build, no TMEM, nothing handed between warps: a launch costs little beyond its bytes.
//
// k is permuted inside a step so that index loads are 16 bytes a lane: the four lanes of a row take a chunk (32 or 64 k) each,
// and X lies in shared memory in the order that the B fragments read it.
//
// A cluster of CTAs owns some rows and divides K; each CTA stages its part of X once.  Sums travel as stores into the CTA that
// owns eight rows, one cluster barrier later that adds them in the order of k: no scratch in global memory, no counters.
//
// Bound at 4 bits: the integer pipe (about 400 instructions per 4096 weights of a warp; 16 warps, since one alone issues every
// sixth cycle; 65 % active at 8 tokens of 18944 x 3584), from 24 tokens on mma.sync besides.  At 2 bits that pipe is 53 % active and the
// waits for X and at the cluster's end count as much.  Small linears are launch, the way of X into shared memory and the barrier.
// Measured at 4 bits with cold weights, the tcgen05 GEMM or batched GEMV before / this, 8 | 16 | 32 tokens, us: 3584 x 3584 13.0 /
// 8.4 | 15.7 / 9.2 | 15.7 / 11.7; 896 x 4864 11.2 / 5.5 | 26.6 / 5.8 | 26.5 / 7.8; gate and up of 18944 x 3584 39.3 / 30.4
// (2.2 TB/s) | 40.2 / 33.0; 3584 x 18944 26.5 / 22.9 | 26.6 / 25.1.  Where other kernels stay ahead: reg_plan.hpp.
#include "common.cuh"
#include "reg_plan.hpp"
#include "tensor_map.cuh"

namespace prism {

enum RegOut { REG_PLAIN = 0, REG_RESID = 1, REG_SWIGLU = 2 };

struct RegArgs {
    const uint8_t *idx, *idx2;   // one tensor, or gate and up
    const uint16_t *pal, *pal2;
    uint32_t n_hb, m, n_chunks, n_steps;
    uint32_t subs, ctas, rows, parts;
    uint32_t x_bytes;            // of shared memory before the received sums
    const uint16_t *x;
    uint32_t x_stride, batch, k;
    float norm_eps;              // >= 0 (one token): RMSNorm of x on the way in
    uint16_t *y;
    const uint16_t *resid;       // may be y
    uint32_t y_stride, mode, wide;
};

namespace {

__device__ __forceinline__ uint32_t rg_prmt(uint32_t a, uint32_t b, uint32_t s) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(s));
    return d;
}
__device__ __forceinline__ void rg_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 rg_ldg(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

template <int BITS>
struct RgPalette;
// Entries 0..7 and 8..15 are gathered with the low three bits of an index, the fourth chooses between them: a byte of that bit is
// the sign that PRMT spreads out of the word itself and of the word shifted by a nibble.
template <>
struct RgPalette<4> {
    static constexpr int WORD = 4;                       // half2 of an index word
    uint32_t lo[4], hi[4];
    __device__ __forceinline__ void load(const uint16_t *pal, uint32_t row) {
        const uint4 p = *reinterpret_cast<const uint4 *>(pal + (size_t)row * 16), q = *reinterpret_cast<const uint4 *>(pal + (size_t)row * 16 + 8);
        const uint32_t e[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            lo[i] = rg_prmt(e[2 * i], e[2 * i + 1], 0x6420);
            hi[i] = rg_prmt(e[2 * i], e[2 * i + 1], 0x7531);
        }
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 4; i++) lo[i] = hi[i] = 0;
    }
    // (k0,k1), (k2,k3), (k4,k5), (k6,k7)
    __device__ __forceinline__ void expand(uint32_t (&h)[4], uint32_t w) const {
        const uint32_t s = w & 0x77777777u, w4 = w * 16u;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t sel = i ? s >> 16 : s, m = rg_prmt(w, w4, i ? 0xBFAE : 0x9D8C);
            const uint32_t l = (rg_prmt(lo[0], lo[1], sel) & ~m) | (rg_prmt(lo[2], lo[3], sel) & m);
            const uint32_t u = (rg_prmt(hi[0], hi[1], sel) & ~m) | (rg_prmt(hi[2], hi[3], sel) & m);
            h[2 * i] = rg_prmt(l, u, 0x5140);
            h[2 * i + 1] = rg_prmt(l, u, 0x7362);
        }
    }
};
// Four entries are a register of low bytes and one of high bytes; the even and the odd indices of a word are nibble selectors after one
// AND.  (As bytes 2c and 2c + 1 of one register pair, selectors by multiplication: gate and up of 18944 x 3584 18.4 us at one token, 27.4 and
// 33.7 at 24 and 32; this way 18.6, 25.8, 31.2.)
template <>
struct RgPalette<2> {
    static constexpr int WORD = 8;
    uint32_t lo, hi;
    __device__ __forceinline__ void load(const uint16_t *pal, uint32_t row) {
        const uint2 p = *reinterpret_cast<const uint2 *>(pal + (size_t)row * 4);
        lo = rg_prmt(p.x, p.y, 0x6420);
        hi = rg_prmt(p.x, p.y, 0x7531);
    }
    __device__ __forceinline__ void clear() { lo = hi = 0; }
    // (k0,k2), (k4,k6), (k1,k3), (k5,k7), then the same of k8..k15
    __device__ __forceinline__ void expand(uint32_t (&h)[8], uint32_t w) const {
        const uint32_t s[2] = {w & 0x33333333u, (w >> 2) & 0x33333333u};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t sel = i & 2 ? rg_prmt(s[i & 1], 0, 0x4432) : s[i & 1];
            const uint32_t l = rg_prmt(lo, lo, sel), u = rg_prmt(hi, hi, sel);
            h[2 * i] = rg_prmt(l, u, 0x5140);
            h[2 * i + 1] = rg_prmt(l, u, 0x7362);
        }
    }
};

__device__ __forceinline__ uint32_t rg_word(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

}  // namespace

template <int BITS, int NT>
__global__ void __launch_bounds__(REG_WARPS * 32, 1) lut_gemm_reg_kernel(const RegArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int UNITS = BITS == 4 ? 4 : 8;             // 16-byte units of X per lane and step
    constexpr uint32_t KC = 8 * UNITS;                   // k of an index chunk
    constexpr int WORD = RgPalette<BITS>::WORD;
    pdl_launch_dependents();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");  // met below: the peers are there before anything is stored to them
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr uint32_t threads = REG_WARPS * 32, warps = REG_WARPS;
    const uint32_t g = lane >> 2, c = lane & 3;
    const uint32_t cluster = blockIdx.x / a.ctas, rank = blockIdx.x % a.ctas;
    const uint32_t s0 = a.n_steps * rank / a.ctas, s1 = a.n_steps * (rank + 1) / a.ctas;
    const uint32_t hb0 = cluster * a.rows, n_rows = min(a.rows, a.n_hb - hb0), jobs = n_rows * a.subs * a.parts;
    float *norm = reinterpret_cast<float *>(smem);       // one word a warp
    uint4 *const xs = reinterpret_cast<uint4 *>(smem + REG_NORM_BYTES);
    float *const recv = reinterpret_cast<float *>(smem + REG_NORM_BYTES + a.x_bytes);

    RgPalette<BITS> pal[4];
    uint4 cur[4], nxt[4];
    uint32_t p0 = 0, p1 = 0;                             // steps of the job
    const uint8_t *src = nullptr;
    auto load = [&](uint4 (&r)[4], uint32_t step) {
        if (4 * step + c < a.n_chunks) {
#pragma unroll
            for (int i = 0; i < 4; i++) r[i] = rg_ldg(src + (size_t)step * 2048 + i * 128);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) r[i] = make_uint4(0, 0, 0, 0);
        }
    };
    auto begin = [&](uint32_t job) {                     // indices and palettes: weights only
        const uint32_t part = job % a.parts, unit = job / a.parts, sub = unit % a.subs, hb = hb0 + unit / a.subs;
        p0 = s0 + (s1 - s0) * part / a.parts;
        p1 = s0 + (s1 - s0) * (part + 1) / a.parts;
        src = (sub ? a.idx2 : a.idx) + ((size_t)hb * a.n_chunks + c) * 512 + g * 16;
        if (p0 < p1) load(cur, p0);
        if (p0 + 1 < p1) load(nxt, p0 + 1);
#pragma unroll
        for (int i = 0; i < 4; i++) pal[i].load(sub ? a.pal2 : a.pal, hb * 32 + g + 8 * i);
    };
    if (warp < jobs) begin(warp);
    pdl_wait();

    // ---- X: this CTA's k, in the order of the B fragments; tokens and k that are not there are zero ------------
    float inv = 1.0f;
    if (a.norm_eps >= 0.0f) {  // the sum of squares of the whole row, in a fixed order (rms_norm_inplace, src/lut/cpu_fallback.rs:39-54)
        float ss = 0.0f;
        for (uint32_t i = tid; i < a.k / 8; i += threads) {
            const uint4 v = reinterpret_cast<const uint4 *>(a.x)[i];
            const __half2 *hp = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 f = __half22float2(hp[e]);
                ss += f.x * f.x + f.y * f.y;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
        if (lane == 0) norm[warp] = ss;
        __syncthreads();
        float tot = 0.0f;
        for (uint32_t w = 0; w < warps; w++) tot += norm[w];
        inv = 1.0f / sqrtf(tot / (float)a.k + a.norm_eps);
    }
    const uint32_t n_units = (s1 - s0) * UNITS * NT * 32;
    for (uint32_t u0 = tid; u0 < n_units; u0 += 4 * threads) {
        uint4 v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t u = u0 + e * threads, ch = u & 3, tok = (u / 32) % NT * 8 + (u >> 2 & 7), rest = u / (32 * NT);
            const uint32_t kk = ((s0 + rest / UNITS) * 4 + ch) * KC + rest % UNITS * 8;
            v[e] = make_uint4(0, 0, 0, 0);
            if (u < n_units && tok < a.batch && kk < a.k) v[e] = *reinterpret_cast<const uint4 *>(a.x + (size_t)tok * a.x_stride + kk);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const uint32_t u = u0 + e * threads;
            if (u >= n_units) break;
            uint4 w = v[e];
            if (a.norm_eps >= 0.0f) {
                __half2 *hp = reinterpret_cast<__half2 *>(&w);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 f = __half22float2(hp[i]);
                    hp[i] = __floats2half2_rn(f.x * inv, f.y * inv);
                }
            }
            if (BITS == 2) w = make_uint4(rg_prmt(w.x, w.y, 0x5410), rg_prmt(w.z, w.w, 0x5410), rg_prmt(w.x, w.y, 0x7632), rg_prmt(w.z, w.w, 0x7632));
            xs[u] = w;
        }
    }
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");

    // ---- jobs ----------------------------------------------------------------------------------------------
    const uint32_t recv_addr = (uint32_t)__cvta_generic_to_shared(recv), all = a.ctas * a.parts;
    for (uint32_t job = warp; job < jobs; job += warps) {
        if (job != warp) begin(job);
        float acc[2][NT][4];
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
            for (int n = 0; n < NT; n++) acc[t][n][0] = acc[t][n][1] = acc[t][n][2] = acc[t][n][3] = 0.0f;
        auto step_of = [&](uint4 (&r)[4], uint32_t step) {
            if (4 * step + 4 > a.n_chunks && 4 * step + c >= a.n_chunks) {  // no such chunk (last step of K): products of zeros
#pragma unroll
                for (int i = 0; i < 4; i++) pal[i].clear();
            }
            const uint4 *xb = xs + (size_t)(step - s0) * UNITS * NT * 32 + lane;
#pragma unroll
            for (int v = 0; v < 4; v++) {
                uint32_t h[4][WORD];
#pragma unroll
                for (int i = 0; i < 4; i++) pal[i].expand(h[i], rg_word(r[i], v));
#pragma unroll
                for (int e = 0; e < WORD / 4; e++)
#pragma unroll
                    for (int n = 0; n < NT; n++) {
                        const uint4 b = xb[((v * (WORD / 4) + e) * NT + n) * 32];
#pragma unroll
                        for (int t = 0; t < 2; t++) {
                            rg_mma(acc[t][n], h[2 * t][4 * e], h[2 * t + 1][4 * e], h[2 * t][4 * e + 1], h[2 * t + 1][4 * e + 1], b.x, b.y);
                            rg_mma(acc[t][n], h[2 * t][4 * e + 2], h[2 * t + 1][4 * e + 2], h[2 * t][4 * e + 3], h[2 * t + 1][4 * e + 3], b.z, b.w);
                        }
                    }
            }
        };
        for (uint32_t s = p0; s < p1; s += 2) {
            step_of(cur, s);
            if (s + 2 < p1) load(cur, s + 2);
            if (s + 1 < p1) {
                step_of(nxt, s + 1);
                if (s + 3 < p1) load(nxt, s + 3);
            }
        }
        // eight rows of a half-block are an octet; octet o of the cluster belongs to CTA o mod ctas
        const uint32_t part = job % a.parts, unit = job / a.parts, sub = unit % a.subs, o0 = unit / a.subs * 4;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t o = o0 + q, owner = o % a.ctas, slot = ((o / a.ctas) * a.subs + sub) * all + rank * a.parts + part;
            uint32_t dst;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(recv_addr + (slot * NT * 64 + c * 16 + g) * 4), "r"(owner));
#pragma unroll
            for (int n = 0; n < NT; n++) {
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + n * 256), "f"(acc[q / 2][n][q % 2 * 2]) : "memory");
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + n * 256 + 32), "f"(acc[q / 2][n][q % 2 * 2 + 1]) : "memory");
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");

    // ---- sums of this CTA's octets ----------------------------------------------------------------------------
    const uint32_t octets = n_rows * 4, mine = octets > rank ? (octets - rank + a.ctas - 1) / a.ctas : 0;
    for (uint32_t i = tid; i < mine * a.batch; i += threads) {
        const uint32_t l = i / a.batch, tok = i % a.batch, row = hb0 * 32 + (l * a.ctas + rank) * 8;
        if (row >= a.m) continue;
        float f[2][8];
#pragma unroll
        for (int s = 0; s < 2; s++) {
            if (s == 1 && a.subs == 1) break;
#pragma unroll
            for (int e = 0; e < 8; e++) f[s][e] = 0.0f;
            const float4 *p = reinterpret_cast<const float4 *>(recv + ((size_t)(l * a.subs + s) * all * NT * 8 + tok) * 8);
            for (uint32_t w = 0; w < all; w++, p += NT * 16) {
                const float4 u = p[0], v = p[1];
                f[s][0] += u.x; f[s][1] += u.y; f[s][2] += u.z; f[s][3] += u.w;
                f[s][4] += v.x; f[s][5] += v.y; f[s][6] += v.z; f[s][7] += v.w;
            }
        }
        uint16_t *y = a.y + (size_t)tok * a.y_stride + row;
        const bool whole = a.wide && row + 8 <= a.m;
        uint16_t old[8], out[8];
        if (a.mode == REG_RESID) {
            const uint16_t *res = a.resid + (size_t)tok * a.y_stride + row;
            if (whole) *reinterpret_cast<uint4 *>(old) = *reinterpret_cast<const uint4 *>(res);
            else
                for (int e = 0; e < 8; e++) old[e] = row + e < a.m ? res[e] : 0;
        }
#pragma unroll
        for (int e = 0; e < 8; e++) {
            __half h = __float2half_rn(f[0][e]);
            if (a.mode == REG_RESID) h = __float2half_rn(__half2float(h) + __half2float(__ushort_as_half(old[e])));
            if (a.mode == REG_SWIGLU) {
                const float gv = __half2float(h), uv = __half2float(__float2half_rn(f[1][e]));
                h = __float2half_rn(__half2float(__float2half_rn(gv / (1.0f + expf(-gv)))) * uv);
            }
            out[e] = __half_as_ushort(h);
        }
        if (whole) *reinterpret_cast<uint4 *>(y) = *reinterpret_cast<const uint4 *>(out);
        else
            for (int e = 0; e < 8; e++)
                if (row + e < a.m) y[e] = out[e];
    }
}

// ---- host side ---------------------------------------------------------------------------------
template <int BITS, int NT>
static int launch_reg(prism_cuda_ctx *ctx, RegArgs &a, const LutTensor &t, bool dry, RegPlan *plan) {
    static uint32_t resident[PRISM_MAX_DEVICES][4] = {{0}};
    uint32_t (&res)[4] = resident[ctx->device];
    if (!res[0]) {
        PRISM_CUDA_TRY(ctx, cudaFuncSetAttribute(lut_gemm_reg_kernel<BITS, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REG_MAX_SMEM));
        for (uint32_t i = 3; i > 0; i--) {
            const int n = resident_clusters(lut_gemm_reg_kernel<BITS, NT>, 1u << i, REG_WARPS * 32, REG_MAX_SMEM, (uint32_t)ctx->sm_count >> i << i);
            res[i] = n > 0 ? (uint32_t)n : 0;
        }
        res[0] = (uint32_t)ctx->sm_count;
    }
    if (dry) {
        *plan = reg_plan((t.m + 31) / 32, a.subs, t.n_chunks, BITS, a.batch, res);
        return PRISM_OK;
    }
    const RegPlan &p = *plan;
    a.ctas = p.ctas;
    a.rows = p.rows;
    a.parts = p.parts;
    a.x_bytes = (a.n_steps + p.ctas - 1) / p.ctas * (BITS == 4 ? 4 : 8) * NT * 512;
    launch_cluster_pdl(ctx, lut_gemm_reg_kernel<BITS, NT>, dim3(p.clusters * p.ctas), dim3(REG_WARPS * 32), p.smem, p.ctas, a);
    return after_launch(ctx, "lut_gemm_reg_kernel");
}

static int reg_dispatch(prism_cuda_ctx *ctx, RegArgs &a, const LutTensor &t, bool dry, RegPlan *plan) {
    const uint32_t nt = (a.batch + 7) / 8;
    if (t.bits == 4) {
        if (nt == 1) return launch_reg<4, 1>(ctx, a, t, dry, plan);
        if (nt == 2) return launch_reg<4, 2>(ctx, a, t, dry, plan);
        if (nt == 3) return launch_reg<4, 3>(ctx, a, t, dry, plan);
        return launch_reg<4, 4>(ctx, a, t, dry, plan);
    }
    if (nt == 1) return launch_reg<2, 1>(ctx, a, t, dry, plan);
    if (nt == 2) return launch_reg<2, 2>(ctx, a, t, dry, plan);
    if (nt == 3) return launch_reg<2, 3>(ctx, a, t, dry, plan);
    return launch_reg<2, 4>(ctx, a, t, dry, plan);
}

static RegArgs reg_args(GemvMode mode, const LutTensor &t, const LutTensor *t2, uint32_t batch) {
    RegArgs a{};
    a.idx = t.idx; a.pal = t.pal;
    if (mode == GEMV_SWIGLU && t2) { a.idx2 = t2->idx; a.pal2 = t2->pal; }
    a.subs = mode == GEMV_SWIGLU ? 2 : 1;
    a.n_hb = (t.m + 31) / 32; a.m = t.m; a.n_chunks = t.n_chunks; a.n_steps = (t.n_chunks + 3) / 4;
    a.batch = batch; a.k = t.k;
    a.mode = mode == GEMV_RESID ? REG_RESID : mode == GEMV_SWIGLU ? REG_SWIGLU : REG_PLAIN;
    return a;
}

static int reg_launch(prism_cuda_ctx *ctx, RegArgs &a, const LutTensor &t, RegPlan *plan, const uint16_t *x, uint32_t x_stride, uint16_t *y, uint32_t y_stride,
                      const uint16_t *resid, float norm_eps) {
    if ((reinterpret_cast<uintptr_t>(x) & 15) || x_stride % 8) return fail(ctx, PRISM_E_ARG, "gemm: activations must be 16-byte aligned");
    a.x = x; a.x_stride = x_stride;
    a.y = y; a.y_stride = y_stride; a.resid = resid;
    a.norm_eps = norm_eps;
    a.wide = y_stride % 8 == 0 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(resid)) & 15) == 0;
    return reg_dispatch(ctx, a, t, false, plan);
}

int gemm_few_tokens(prism_cuda_ctx *ctx, GemvMode mode, const LutTensor &t, const LutTensor *t2, const uint16_t *x, uint32_t x_stride, uint16_t *y,
                    uint32_t y_stride, const uint16_t *resid, uint32_t batch, float norm_eps, bool *takes) {
    *takes = false;
    if (ctx->gemv_variant != 1 || ctx->gemm_variant != 1 || ctx->batch_gemv_max) return PRISM_OK;  // the caller names the kernels
    if ((reinterpret_cast<uintptr_t>(x) & 15) || x_stride % 8) return PRISM_OK;
    if (mode != GEMV_PLAIN && mode != GEMV_RESID && mode != GEMV_SWIGLU) return PRISM_OK;
    if (batch == 0 || batch > REG_MAX_TOKENS || t.m == 0 || !((t.bits == 4 && t.k % 32 == 0 && t.k >= 32) || (t.bits == 2 && t.k % 64 == 0 && t.k >= 64))) return PRISM_OK;
    RegArgs a = reg_args(mode, t, t2, batch);
    if (batch < 8 && !reg_pays(t.m, t.k, t.bits, a.subs, batch, 0.0, 1e30)) return PRISM_OK;  // whatever the plan
    RegPlan plan;
    PRISM_TRY(reg_dispatch(ctx, a, t, true, &plan));
    if (!plan.ctas) return PRISM_OK;
    double gemm = 1e30;
    if (gemm_tc5_eligible(ctx, t, batch)) PRISM_TRY(gemm_tc5_cycles(ctx, t, batch, a.subs, &gemm));
    *takes = reg_pays(t.m, t.k, t.bits, a.subs, batch, plan.cycles, gemm);
    return *takes ? reg_launch(ctx, a, t, &plan, x, x_stride, y, y_stride, resid, norm_eps) : PRISM_OK;
}

int launch_gemm_reg(prism_cuda_ctx *ctx, GemvMode mode, const LutTensor &t, const LutTensor *t2, const uint16_t *x, uint32_t x_stride, uint16_t *y,
                    uint32_t y_stride, const uint16_t *resid, uint32_t batch, float norm_eps) {
    RegArgs a = reg_args(mode, t, t2, batch);
    RegPlan plan;
    PRISM_TRY(reg_dispatch(ctx, a, t, true, &plan));
    if (!plan.ctas) return fail(ctx, PRISM_E_ARG, "gemm: this shape does not fit the register-palette kernel");
    return reg_launch(ctx, a, t, &plan, x, x_stride, y, y_stride, resid, norm_eps);
}

}  // namespace prism
