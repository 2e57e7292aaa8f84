// Offline quantiser on the GPU, with exactly the operations, in exactly the order, of the reference's
// CPU quantiser wherever an order shows in the result, so the payload is bit-identical to it.
//
//   fit_palette      src/quantization/palette.rs:75-174   deterministic k-means++ seeding (first
//                    centroid = channel[n/2], golden-ratio threshold :177-182), <= max_iter Lloyd
//                    steps, early exit when the largest shift < 0.001, codebook sorted by |value|
//                    descending (stable)
//   encode_channel   src/quantization/palette.rs:189-217  nearest of the 16 entries, first wins on
//                    ties, element 2i in the low nibble
//   payload          src/lut/compiler.rs:50-61            all palettes as fp16, then all index rows
//
// Arithmetic uses the explicit round-to-nearest intrinsics: no multiply-add contraction (Rust never
// contracts a*b+c).  Distances, nearest entries and places are independent per element and are shared
// by the threads of a block; the sums that the CPU code carries from element to element stay one chain
// of additions in element order:
//  * the seeding's total: one warp walks the running minimum distances in shared memory, 4 per load.
//    Its running sum IS the sum the choice walks, so the value after every 32 elements is kept and only
//    the 32 elements in which the threshold is met are added again (the sum never falls: distances are
//    >= 0 and rounding is monotone);
//  * a Lloyd step's 16 sums: the elements are put in cluster order first (stable counting sort), then
//    16 lanes add their cluster's elements one after the other.
// Bound by those chains (4 cycles an element, 15 passes) and the instructions of the nearest-entry search.
// One block per row, so 14 rows of 3584 are at work on an SM at a time.
// 3584 x 3584 values: 1.08 ms, 25.9 with one thread per row.  Rows whose distances do not fit shared memory, and many short rows,
// still take one thread each.
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>

#include "common.cuh"

namespace prism {

constexpr int PQ_THREADS = 128;

__device__ __forceinline__ float pq_dist(float x, float c) {
    const float diff = __fsub_rn(x, c);
    return __fmul_rn(diff, diff);
}

// weighted_threshold (palette.rs:177-182)
__device__ __forceinline__ float pq_threshold(float total, uint32_t seed) {
    const double v = __dmul_rn((double)seed, 0.6180339887498949);
    const double frac = __dsub_rn(v, floor(v));
    return __fmul_rn(total, (float)frac);
}

__global__ void __launch_bounds__(PQ_THREADS) palettize_rows_kernel(const float *__restrict__ w, uint32_t dm,
                                                                    uint32_t dn, uint32_t k_req, uint32_t max_iter,
                                                                    uint8_t *__restrict__ payload) {
    const uint32_t r = blockIdx.x * PQ_THREADS + threadIdx.x;
    if (r >= dm) return;
    const float *ch = w + (size_t)r * dn;
    const uint32_t n = dn;
    float cb[16];
#pragma unroll
    for (int i = 0; i < 16; i++) cb[i] = 0.0f;
    uint32_t k = k_req > 16 ? 16 : k_req;
    if (k > n) k = n;

    // ---- seeding ----------------------------------------------------------------------------------
    uint32_t nc = 0;
    if (k > 0) cb[nc++] = ch[n / 2];
    for (uint32_t it = 1; it < k; it++) {
        // min_d[i] after this round = the smallest squared distance to centroids 0..nc-1
        float total = 0.0f;
        for (uint32_t i = 0; i < n; i++) {
            const float x = ch[i];
            float md = 3.40282347e+38f;
            for (uint32_t c = 0; c < nc; c++) {
                const float d = pq_dist(x, cb[c]);
                if (d < md) md = d;
            }
            total = __fadd_rn(total, md);
        }
        if (total <= 0.0f) {
            cb[nc] = ch[((size_t)nc * n / k) % n];
            nc++;
            continue;
        }
        const float target = pq_threshold(total, nc);
        float cum = 0.0f;
        uint32_t picked = 0;
        for (uint32_t i = 0; i < n; i++) {
            const float x = ch[i];
            float md = 3.40282347e+38f;
            for (uint32_t c = 0; c < nc; c++) {
                const float d = pq_dist(x, cb[c]);
                if (d < md) md = d;
            }
            cum = __fadd_rn(cum, md);
            if (cum >= target) {
                picked = i;
                break;
            }
        }
        cb[nc++] = ch[picked];
    }

    // ---- Lloyd steps --------------------------------------------------------------------------------
    for (uint32_t iter = 0; iter < max_iter && k > 0; iter++) {
        float sum[16];
        uint32_t cnt[16];
#pragma unroll
        for (int c = 0; c < 16; c++) {
            sum[c] = 0.0f;
            cnt[c] = 0;
        }
        for (uint32_t i = 0; i < n; i++) {
            const float x = ch[i];
            float best_d = 3.40282347e+38f;
            uint32_t best = 0;
            for (uint32_t c = 0; c < k; c++) {
                const float d = pq_dist(x, cb[c]);
                if (d < best_d) {
                    best_d = d;
                    best = c;
                }
            }
            sum[best] = __fadd_rn(sum[best], x);
            cnt[best]++;
        }
        float max_shift = 0.0f;
        for (uint32_t c = 0; c < k; c++) {
            if (cnt[c] > 0) {
                const float nv = __fdiv_rn(sum[c], (float)cnt[c]);
                const float shift = fabsf(__fsub_rn(cb[c], nv));
                if (shift > max_shift) max_shift = shift;
                cb[c] = nv;
            }
        }
        if (max_shift < 0.001f) break;
    }

    // ---- stable sort of the k centroids, |v| descending --------------------------------------------
    for (uint32_t i = 1; i < k; i++) {
        const float v = cb[i];
        uint32_t j = i;
        while (j > 0 && fabsf(cb[j - 1]) < fabsf(v)) {
            cb[j] = cb[j - 1];
            j--;
        }
        cb[j] = v;
    }

    // ---- encode against all 16 entries (unused ones are 0) and emit ---------------------------------
    uint8_t *pal = payload + (size_t)r * 32;
    uint8_t *idx = payload + (size_t)dm * 32 + (size_t)r * (dn / 2);
    uint8_t cur = 0;
    for (uint32_t i = 0; i < n; i++) {
        const float x = ch[i];
        uint32_t best = 0;
        float best_d = 3.40282347e+38f;
#pragma unroll
        for (uint32_t c = 0; c < 16; c++) {
            const float d = pq_dist(x, cb[c]);
            if (d < best_d) {
                best_d = d;
                best = c;
            }
        }
        if ((i & 1) == 0) {
            cur = (uint8_t)best;
            if (i + 1 == n) idx[i / 2] = cur;
        } else {
            idx[i / 2] = (uint8_t)(cur | (best << 4));
        }
    }
    // little-endian fp16 bit patterns; the palette of a row starts on a 32-byte boundary
    uint16_t *pal16 = reinterpret_cast<uint16_t *>(pal);
    for (int i = 0; i < 16; i++) pal16[i] = __half_as_ushort(__float2half_rn(cb[i]));
}

// ---- one block per row ---------------------------------------------------------------------------
constexpr int PB_THREADS = 128, PB_WARPS = PB_THREADS / 32;
constexpr float PB_FAR = 3.40282347e+38f;

// Distances (later: the elements in cluster order) padded to whole 32s, and the running sum after each 32.
__host__ __device__ constexpr size_t pb_smem_bytes(uint32_t n) { return (size_t)((n + 31) / 32) * (32 + 1) * 4; }
constexpr size_t PB_MAX_SMEM = 220 * 1024;

// Nearest entry, the first of equal ones; an entry that is NaN is never chosen.
__device__ __forceinline__ uint32_t pb_nearest(float x, const float (&cb)[16]) {
    float best_d = PB_FAR;
    uint32_t best = 0;
#pragma unroll
    for (uint32_t c = 0; c < 16; c++) {
        const float d = pq_dist(x, cb[c]);
        if (d < best_d) {
            best_d = d;
            best = c;
        }
    }
    return best;
}

__global__ void __launch_bounds__(PB_THREADS) palettize_block_kernel(const float *__restrict__ w, uint32_t dm, uint32_t n,
                                                                     uint32_t k_req, uint32_t max_iter, uint8_t *__restrict__ payload) {
    extern __shared__ __align__(16) float md[];
    __shared__ float cbs[16];
    __shared__ uint32_t cnt[PB_WARPS][16], off[PB_WARPS][16], first[17];
    __shared__ float max_shift;
    __shared__ uint32_t picked;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tiles = (n + 31) / 32;
    float *running = md + (size_t)tiles * 32;
    const size_t row = blockIdx.x;
    const float *ch = w + row * n;
    uint8_t *idx = payload + (size_t)dm * 32 + row * (n / 2);
    uint32_t k = k_req > 16 ? 16 : k_req;
    if (k > n) k = n;

    // ---- seeding ----------------------------------------------------------------------------------
    float last = ch[n / 2];  // the centroid chosen last
    if (tid < 16) cbs[tid] = __int_as_float(0x7fffffff);  // entries not chosen yet: NaN, never nearest
    __syncthreads();
    if (tid == 0) cbs[0] = last;
    for (uint32_t nc = 1; nc < k; nc++) {
#pragma unroll 4
        for (uint32_t i = tid; i < tiles * 32; i += PB_THREADS) {
            float m = 0.0f;  // padding adds +0 to a sum that is >= 0
            if (i < n) {
                m = nc == 1 ? PB_FAR : md[i];
                const float d = pq_dist(ch[i], last);
                if (d < m) m = d;
            }
            md[i] = m;
        }
        __syncthreads();
        if (warp == 0) {
            float sum = 0.0f;
            const float4 *m4 = reinterpret_cast<const float4 *>(md);
            for (uint32_t t = 0; t < tiles; t++) {
                float4 v[8];
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = m4[t * 8 + j];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    sum = __fadd_rn(sum, v[j].x);
                    sum = __fadd_rn(sum, v[j].y);
                    sum = __fadd_rn(sum, v[j].z);
                    sum = __fadd_rn(sum, v[j].w);
                }
                if (lane == 0) running[t] = sum;
            }
            __syncwarp();
            uint32_t at = (uint32_t)((size_t)nc * n / k % n);
            if (!(sum <= 0.0f)) {
                const float target = pq_threshold(sum, nc);
                at = 0;
                for (uint32_t t0 = 0; t0 < tiles; t0 += 32) {
                    const uint32_t met = __ballot_sync(0xFFFFFFFFu, t0 + lane < tiles && running[t0 + lane] >= target);
                    if (!met) continue;
                    const uint32_t t = t0 + __ffs(met) - 1;
                    float cum = t ? running[t - 1] : 0.0f;
                    uint32_t j = 0;
                    for (; j < 32; j++) {
                        cum = __fadd_rn(cum, md[t * 32 + j]);
                        if (cum >= target) break;
                    }
                    at = t * 32 + j;
                    break;
                }
            }
            if (lane == 0) {
                picked = at;
                cbs[nc] = ch[at];
            }
        }
        __syncthreads();
        last = ch[picked];
    }
    __syncthreads();

    // ---- Lloyd steps --------------------------------------------------------------------------------
    // a warp owns consecutive 32s; the choice of each element is kept in the row's index bytes
    const uint32_t per_warp = (tiles + PB_WARPS - 1) / PB_WARPS;
    const uint32_t t_lo = min(tiles, warp * per_warp), t_hi = min(tiles, t_lo + per_warp);
    float cb[16];
    for (uint32_t iter = 0; iter < max_iter; iter++) {
#pragma unroll
        for (int c = 0; c < 16; c++) cb[c] = cbs[c];
        if (lane < 16) cnt[warp][lane] = 0;
        __syncwarp();
#pragma unroll 2
        for (uint32_t t = t_lo; t < t_hi; t++) {
            const uint32_t i = t * 32 + lane;
            const uint32_t best = i < n ? pb_nearest(ch[i], cb) : 16;
            const uint32_t high = __shfl_down_sync(0xFFFFFFFFu, best, 1);
            if (!(lane & 1) && i < n) idx[i / 2] = (uint8_t)(best | (high << 4));  // n is even
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, best);
            if (best < 16 && lane == 31 - __clz(same)) cnt[warp][best] += __popc(same);
            __syncwarp();
        }
        __syncthreads();
        if (tid < 16) {
            uint32_t before = 0, own = 0;
            for (int v = 0; v < PB_WARPS; v++)
                for (uint32_t c = 0; c <= tid; c++) (c < tid ? before : own) += cnt[v][c];
            first[tid] = before;
            if (tid == 15) first[16] = before + own;
            for (int v = 0; v < PB_WARPS; v++) {
                off[v][tid] = before;
                before += cnt[v][tid];
            }
        }
        __syncthreads();
#pragma unroll 2
        for (uint32_t t = t_lo; t < t_hi; t++) {
            const uint32_t i = t * 32 + lane;
            const uint32_t best = i < n ? (idx[i / 2] >> (4 * (lane & 1))) & 15 : 16;
            const uint32_t same = __match_any_sync(0xFFFFFFFFu, best);
            if (best < 16) {
                const uint32_t rank = __popc(same & ((1u << lane) - 1));
                const uint32_t at = off[warp][best] + rank;
                md[at] = ch[i];
            }
            __syncwarp();
            if (best < 16 && lane == 31 - __clz(same)) off[warp][best] += __popc(same);
            __syncwarp();
        }
        __syncthreads();
        if (warp == 0) {
            float shift = 0.0f;
            if (lane < k) {
                const uint32_t a = first[lane], b = first[lane + 1];
                float sum = 0.0f;
                uint32_t i = a;
                for (; i + 8 <= b; i += 8) {
                    float v[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] = md[i + j];
#pragma unroll
                    for (int j = 0; j < 8; j++) sum = __fadd_rn(sum, v[j]);
                }
                for (; i < b; i++) sum = __fadd_rn(sum, md[i]);
                if (b > a) {
                    const float nv = __fdiv_rn(sum, (float)(b - a));
                    const float s = fabsf(__fsub_rn(cbs[lane], nv));
                    if (s > 0.0f) shift = s;
                    cbs[lane] = nv;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) shift = fmaxf(shift, __shfl_xor_sync(0xFFFFFFFFu, shift, o));
            if (lane == 0) max_shift = shift;
        }
        __syncthreads();
        if (max_shift < 0.001f) break;
    }

    // ---- stable sort of the k centroids, |v| descending; unused entries are 0 -----------------------
    if (tid == 0) {
        for (uint32_t i = k; i < 16; i++) cbs[i] = 0.0f;
        for (uint32_t i = 1; i < k; i++) {
            const float v = cbs[i];
            uint32_t j = i;
            while (j > 0 && fabsf(cbs[j - 1]) < fabsf(v)) {
                cbs[j] = cbs[j - 1];
                j--;
            }
            cbs[j] = v;
        }
    }
    __syncthreads();

    // ---- encode against all 16 entries and emit; the palette of a row starts on a 32-byte boundary --
#pragma unroll
    for (int c = 0; c < 16; c++) cb[c] = cbs[c];
#pragma unroll 2
    for (uint32_t i = tid; i < n / 2; i += PB_THREADS)
        idx[i] = (uint8_t)(pb_nearest(ch[2 * i], cb) | (pb_nearest(ch[2 * i + 1], cb) << 4));
    if (tid < 16)
        reinterpret_cast<uint16_t *>(payload + row * 32)[tid] = __half_as_ushort(__float2half_rn(cbs[tid]));
}

static cudaError_t palettize_rows(const float *w_dev, uint32_t dm, uint32_t dn, uint32_t k, uint32_t max_iter, uint8_t *payload_dev, cudaStream_t stream) {
    const size_t smem = pb_smem_bytes(dn);
    // Many short rows: a block pays some 15 ns of the GPU a row before its first element, a thread per row 14 us an element however
    // many rows there are up to the GPU's threads.  100000 rows of 16 / 64 / 128 values: blocks 1541 / 2059 / 2384 us, threads 165 /
    // 955 / 1836.
    const bool threads = dn <= 128 && dm >= 720u * dn;
    if (smem <= PB_MAX_SMEM && !threads) {
        if (smem > 48 * 1024) {
            const cudaError_t e = cudaFuncSetAttribute(palettize_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PB_MAX_SMEM);
            if (e != cudaSuccess) return e;
        }
        palettize_block_kernel<<<dm, PB_THREADS, smem, stream>>>(w_dev, dm, dn, k, max_iter, payload_dev);
    } else {
        palettize_rows_kernel<<<(dm + PQ_THREADS - 1) / PQ_THREADS, PQ_THREADS, 0, stream>>>(w_dev, dm, dn, k, max_iter, payload_dev);
    }
    return cudaGetLastError();
}

// ---- a matrix in host memory -----------------------------------------------------------------------
// A copy from pageable memory goes through the driver at 12 GB/s, one thread, also when several ask, and a copy into memory that was
// never touched at 2.  Here up to 4 threads carry a part of the rows each onto the GPU and their payload back, through two pinned
// slots of their own.  The slots (4 MB; in huge pages their first use takes 1.5 ms, through cudaHostAlloc 3 to 15) and device buffers of
// at most PZ_KEEP together stay with the context; another allocation that finds no memory takes the device buffers back (device_malloc).
// 3584 x 3584 values: 8.0 -> 3.4 ms (matrix 1.8, kernel 1.08, payload 0.5), a context's first call 9.9 -> 6.4; 896 x 896, one thread and
// kept device buffers: 1.13 -> 0.5 ms.
constexpr uint32_t PZ_WORKERS = 4;
constexpr size_t PZ_SLOT = 512 * 1024;                  // two of them a worker
constexpr size_t PZ_PAGE = 2 << 20;
constexpr size_t PZ_LEAST = 8 << 20;                    // bytes of a matrix from which it is shared: below, the slots' first use takes longer than they save
constexpr size_t PZ_KEEP = 64 << 20;                    // matrix and payload of 3584 x 3584 are 58

struct PalettizePool {
    uint8_t *pinned = nullptr;
    cudaEvent_t event[PZ_WORKERS][2] = {};
    void *dev[2] = {};                                   // matrix, payload
    size_t bytes[2] = {};
};
void palettize_pool_free(PalettizePool *p) {
    if (!p) return;
    for (auto &w : p->event)
        for (cudaEvent_t e : w)
            if (e) cudaEventDestroy(e);
    if (p->pinned) cudaHostUnregister(p->pinned);
    free(p->pinned);
    for (void *d : p->dev) cudaFree(d);
    delete p;
}

bool palettize_pool_trim(PalettizePool *p) {
    bool any = false;
    for (int i = 0; p && i < 2; i++) {
        any = any || p->dev[i];
        cudaFree(p->dev[i]);
        p->dev[i] = nullptr;
        p->bytes[i] = 0;
    }
    return any;
}

struct PalettizeJob {
    const float *w;
    uint32_t dm, dn, k, max_iter, workers;
    uint8_t *payload;
    PalettizePool *pool;
    int device;
    cudaStream_t stream;
    std::atomic<uint32_t> carried{0}, failed{0}, launched{0};  // shares on their way to the GPU; one of them failed; the kernel is in the stream
};
// Worker t's share; its copies take its two slots in turn, a slot is free again when its event has come.  Whoever has carried the
// last share launches the kernel.
static cudaError_t palettize_share(PalettizeJob &j, uint32_t t) {
    PalettizePool &p = *j.pool;
    uint8_t *slot[2] = {p.pinned + (size_t)t * 2 * PZ_SLOT, p.pinned + ((size_t)t * 2 + 1) * PZ_SLOT};
    uint8_t *w_dev = static_cast<uint8_t *>(p.dev[0]), *p_dev = static_cast<uint8_t *>(p.dev[1]);
    const size_t r0 = (size_t)j.dm * t / j.workers, r1 = (size_t)j.dm * (t + 1) / j.workers, row = (size_t)j.dn * 4;
    uint32_t turn = 0;
    cudaError_t e = cudaSetDevice(j.device);
    for (size_t at = r0 * row; at < r1 * row && e == cudaSuccess; at += PZ_SLOT, turn ^= 1) {
        const size_t n = std::min(r1 * row - at, PZ_SLOT);
        if ((e = cudaEventSynchronize(p.event[t][turn])) != cudaSuccess) break;
        memcpy(slot[turn], reinterpret_cast<const uint8_t *>(j.w) + at, n);
        e = cudaMemcpyAsync(w_dev + at, slot[turn], n, cudaMemcpyHostToDevice, j.stream);
        if (e == cudaSuccess) e = cudaEventRecord(p.event[t][turn], j.stream);
    }
    if (e != cudaSuccess) j.failed = 1;
    if (j.carried.fetch_add(1) + 1 == j.workers) {
        if (!j.failed && (e = palettize_rows(static_cast<const float *>(p.dev[0]), j.dm, j.dn, j.k, j.max_iter, p_dev, j.stream)) != cudaSuccess) j.failed = 1;
        j.launched = 1;
    }
    while (!j.launched) std::this_thread::yield();
    if (j.failed) return e;
    for (int s = 0; s < 2 && e == cudaSuccess; s++) e = cudaEventSynchronize(p.event[t][s]);
    const size_t part[2][2] = {{r0 * 32, r1 * 32}, {(size_t)j.dm * 32 + r0 * (j.dn / 2), (size_t)j.dm * 32 + r1 * (j.dn / 2)}};
    for (const auto &range : part) {
        size_t behind = range[0], behind_n = 0;          // what the other slot is receiving
        for (size_t at = range[0]; e == cudaSuccess && (at < range[1] || behind_n); turn ^= 1) {
            const size_t n = std::min(range[1] - at, PZ_SLOT);
            if (n) {
                e = cudaMemcpyAsync(slot[turn], p_dev + at, n, cudaMemcpyDeviceToHost, j.stream);
                if (e == cudaSuccess) e = cudaEventRecord(p.event[t][turn], j.stream);
            }
            if (behind_n && e == cudaSuccess && (e = cudaEventSynchronize(p.event[t][turn ^ 1])) == cudaSuccess) memcpy(j.payload + behind, slot[turn ^ 1], behind_n);
            behind = at;
            behind_n = n;
            at += n;
        }
    }
    return e;
}

static cudaError_t palettize_slots(PalettizePool &p) {
    cudaError_t e = cudaSuccess;
    if (!p.pinned) {
        const size_t bytes = 2 * PZ_WORKERS * PZ_SLOT;
        void *m = aligned_alloc(PZ_PAGE, bytes);
        if (!m) return cudaErrorMemoryAllocation;
        madvise(m, bytes, MADV_HUGEPAGE);                // a wish: without it registering takes longer
        memset(m, 0, bytes);
        if ((e = cudaHostRegister(m, bytes, cudaHostRegisterDefault)) != cudaSuccess) {
            free(m);
            return e;
        }
        p.pinned = static_cast<uint8_t *>(m);
    }
    for (auto &w : p.event)
        for (cudaEvent_t &v : w)
            if (!v && (e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming)) != cudaSuccess) return e;
    return e;
}
static cudaError_t palettize_device(PalettizePool &p, int i, size_t bytes) {
    if (p.bytes[i] >= bytes) return cudaSuccess;
    cudaFree(p.dev[i]);
    p.dev[i] = nullptr;
    p.bytes[i] = 0;
    const cudaError_t e = cudaMalloc(&p.dev[i], bytes);
    if (e == cudaSuccess) p.bytes[i] = bytes;
    else p.dev[i] = nullptr;
    return e;
}

}  // namespace prism

using namespace prism;

extern "C" int prism_cuda_palettize_dev(prism_cuda_ctx *ctx, const float *weights_dev, uint32_t dim_m, uint32_t dim_n,
                                        uint32_t k, uint32_t max_iter, uint8_t *payload_dev) {
    if (!ctx || !weights_dev || !payload_dev) return fail(ctx, PRISM_E_NULL, "null argument");
    if (dim_m == 0 || dim_n == 0 || dim_n % 2 != 0 || k == 0)
        return fail(ctx, PRISM_E_ARG, "palettize: dim_m, dim_n > 0, dim_n even, k >= 1");
    PRISM_CUDA_TRY(ctx, palettize_rows(weights_dev, dim_m, dim_n, k, max_iter, payload_dev, ctx->stream));
    ctx->launches++;
    return PRISM_OK;
}

extern "C" int prism_cuda_palettize(prism_cuda_ctx *ctx, const float *weights, uint32_t dim_m, uint32_t dim_n, uint32_t k,
                                    uint32_t max_iter, uint8_t *payload, size_t len) {
    if (!ctx || !weights || !payload) return fail(ctx, PRISM_E_NULL, "null argument");
    if (dim_m == 0 || dim_n == 0 || dim_n % 2 != 0 || k == 0)
        return fail(ctx, PRISM_E_ARG, "palettize: dim_m, dim_n > 0, dim_n even, k >= 1");
    const size_t need = (size_t)dim_m * 32 + (size_t)dim_m * (dim_n / 2);
    if (len != need) return fail(ctx, PRISM_E_ARG, "palettize: payload must hold dim_m*32 + dim_m*dim_n/2 bytes");
    PRISM_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    PRISM_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &capture));
    if (capture != cudaStreamCaptureStatusNone) return cuda_fail(ctx, cudaErrorStreamCaptureUnsupported, "palettize");
    const size_t w_bytes = (size_t)dim_m * dim_n * sizeof(float);
    const uint32_t most = std::min(PZ_WORKERS, std::max(1u, std::thread::hardware_concurrency()));
    uint32_t workers = w_bytes < PZ_LEAST ? 1 : std::min(most, dim_m);
    if (!ctx->palettize && !(ctx->palettize = new (std::nothrow) PalettizePool())) return fail(ctx, PRISM_E_CUDA, "palettize: out of host memory");
    PalettizePool &pool = *ctx->palettize;
    if (workers > 1 && palettize_slots(pool) != cudaSuccess) {  // no pinned memory to be had: one thread needs none
        (void)cudaGetLastError();
        workers = 1;
    }
    cudaError_t e = palettize_device(pool, 0, w_bytes);
    if (e == cudaSuccess) e = palettize_device(pool, 1, need);
    if (e == cudaSuccess && workers == 1) {
        e = cudaMemcpyAsync(pool.dev[0], weights, w_bytes, cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = palettize_rows(static_cast<const float *>(pool.dev[0]), dim_m, dim_n, k, max_iter, static_cast<uint8_t *>(pool.dev[1]), ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(payload, pool.dev[1], need, cudaMemcpyDeviceToHost, ctx->stream);
        const cudaError_t done = cudaStreamSynchronize(ctx->stream);
        if (e == cudaSuccess) e = done;
        if (e == cudaSuccess) ctx->launches++;
    } else if (e == cudaSuccess) {
        // as many shares as there are threads to be had for them: the shares wait for one another
        PalettizeJob job;
        job.w = weights; job.dm = dim_m; job.dn = dim_n; job.k = k; job.max_iter = max_iter;
        job.payload = payload; job.pool = &pool; job.device = ctx->device; job.stream = ctx->stream;
        cudaError_t results[PZ_WORKERS] = {};
        std::thread threads[PZ_WORKERS];
        std::atomic<uint32_t> go{0};                     // workers there are, once that is known
        uint32_t have = 1;
        try {
            for (; have < workers; have++)
                threads[have] = std::thread([&job, &results, &go](uint32_t t) {
                    while (!go) std::this_thread::yield();
                    results[t] = palettize_share(job, t);
                }, have);
        } catch (...) {
        }
        job.workers = have;
        go = have;
        results[0] = palettize_share(job, 0);
        for (std::thread &t : threads)
            if (t.joinable()) t.join();
        for (cudaError_t r : results)
            if (e == cudaSuccess) e = r;
        const cudaError_t done = cudaStreamSynchronize(ctx->stream);  // nothing of this call is left on the GPU, failed or not
        if (e == cudaSuccess) e = done;
        if (e == cudaSuccess) ctx->launches++;
    }
    if (pool.bytes[0] + pool.bytes[1] > PZ_KEEP || e != cudaSuccess) palettize_pool_trim(&pool);
    if (e == cudaSuccess) return PRISM_OK;
    (void)cudaGetLastError();
    return cuda_fail(ctx, e, "palettize");
}
