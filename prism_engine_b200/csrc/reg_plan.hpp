// How the register-palette GEMM (gemm_reg.cu) divides a linear; kept free of CUDA so that it can be checked on a host
// (tests/cpp/test_reg_plan.cpp).
#pragma once

#include <cstddef>
#include <cstdint>

namespace prism {

constexpr uint32_t REG_MAX_TOKENS = 32;
constexpr size_t REG_MAX_SMEM = 227 * 1024 - 1024;

// Asked only while the options that name other kernels are at their defaults.
// Whether that kernel takes less time than the ones beside it for `tensors` (2: gate and up) of m rows of k weights.  From 8 tokens
// on the other one is the tcgen05 GEMM and the two estimates are compared (`cycles` of reg_plan, `gemm_cycles` of gm_plan, each
// within some 12 % of the times; 1e30 where the GEMM does not take the shape).  On 40 cases of 2 and 4 bits and 8 to 32 tokens that
// picks the slower one where they are within 10 % of each other.  Below that the others are the batched GEMV, and for one token the
// pair-table and stream-K GEMV; measured, cold weights, other / this in us:
//  * one token: at 4 bits the pair tables are ahead wherever they are used (3584 x 3584 5.8 / 8.4, gate and up of 18944 x 3584
//    20.3 / 30.0), at 2 bits for single tensors (3584 x 18944 12.1 / 14.0, 19008 x 3584 11.2 / 15.6) and small gates and ups (two of
//    9472 x 3584 8.7 / 11.8, 68 million weights).  For larger ones it depends on how evenly this kernel's CTAs share the rows, so its estimate
//    meets one of the stream-K GEMV (6.1 us and 0.104 us a million weights, within 7 % on 14 shapes of 117 to 283 million; the bounds of 100
//    and 268 keep to where that was fitted): two of 18944 x 3584 21.5 / 18.3, 13824 x 5120 21.2 / 19.8, 23680 x 3584 24.7 / 24.1, but
//    19264 x 3584 21.8 / 23.7, 10240 x 8192 24.1 / 26.6, 28672 x 4096 30.6 / 33.4 (a share of nine half-blocks is 18 jobs: a second round of
//    the 16 warps for two);
//  * 2 bits, 2 to 7 tokens: ahead (18944 x 3584, two: 34.8 / 18.6 at 2, 84.2 / 19.1 at 6);
//  * short rows, little work: behind, since its clusters and the staging of X cost 2.6 us at least (2 bits, k < 1024 and fewer than nine
//    million weights x tokens: 320 x 192 1.9 / 2.9 at 12, 896 x 896 2.8 / 3.1 at 6, 960 x 320 3.1 / 3.8 at 24, but 1600 x 192 5.7 / 4.0 at
//    32; up to 8 tokens, since from 9 on the tcgen05 GEMM is beside it where it can be: 640 x 256 5.0 / 3.0 at 12; 4 bits, k < 512 and three million:
//    320 x 192 2.2 / 2.6 at 4, 3520 x 192 2.5 / 2.8 at 4, but 192 x 832 5.2 / 2.8 at 4);
//  * 4 bits, single tensors of 2^22 weights with more rows than k: behind at 2 tokens (5120 x 2048 5.5 / 6.4, 4864 x 896 3.9 / 4.5,
//    but 2048 x 5120 6.8 / 6.5), at 3 where they are four times as many (4864 x 896 4.3 / 4.5, but 5120 x 2048 6.7 / 6.4);
//  * 4 bits, up to 2^25 weights: ahead (3584 x 3584 9.6 / 8.3 at 4, 5120 x 2048, two: 12.0 / 10.6 at 2);
//  * 4 bits, more weights: behind at 2 tokens (8192 x 8192 15.1 / 18.8), at 3 and 4 for long rows (8192 x 29568 44.9 / 55.4, but
//    18944 x 3584, two: 36.9 / 30.1), ahead from 5 on (3584 x 18944 26.7 / 22.7 at 6).
inline bool reg_pays(uint64_t m, uint64_t k, uint32_t bits, uint32_t tensors, uint32_t tokens, double cycles, double gemm_cycles) {
    const uint64_t weights = m * k * tensors;
    if (bits == 2 && k < 1024 && tokens > 1 && tokens * weights < 9000000u && (tokens <= 8 || gemm_cycles >= 1e30)) return false;
    if (bits == 4 && k < 512 && tokens > 1 && tokens < 8 && tokens * weights < 3000000u) return false;
    if (tokens >= 8) return cycles < 0.95 * gemm_cycles;
    if (tokens <= 1) return bits == 2 && tensors == 2 && weights >= 100000000u && weights < 1u << 28 && cycles < 12000.0 + 204e-6 * (double)weights;
    if (bits == 4 && tokens <= 3 && tensors == 1 && weights >= 1u << 22 && m > (tokens == 2 ? k : 4 * k)) return false;
    return bits == 2 || weights < 1u << 25 || tokens > 4 || (tokens > 2 && k < 8192);
}

// A cluster of `ctas` CTAs owns `rows` half-blocks of 32 output rows; CTA r of it takes the r-th part of K for all of them, and
// cuts its part into `parts`: (half-block, tensor, part) is a job of one of its 16 warps.
struct RegPlan {
    uint32_t ctas = 0, rows = 0, parts = 0, clusters = 0;
    size_t smem = 0;
    double cycles = 1e30;
};
constexpr uint32_t REG_WARPS = 16;
constexpr uint32_t REG_NORM_BYTES = 256;  // shared memory before the activations

// n_hb half-blocks of 32 rows, subs tensors (2: gate and up), n_chunks 16-byte index chunks a row; resident[i]: clusters of 2^i
// CTAs that the GPU holds at once.
// Estimated cycles: a step, four chunks of 32 rows by one warp, keeps an SM sub-partition's integer pipe busy for `busy` and takes
// a warp that is alone there `chain`; the activations of a part come at 16 bytes a cycle; a job's sums cost 140 per eight tokens on
// their way, the cluster barrier 1000.  Fitted to all choices for 80 cases (20 shapes of 2 and 4 bits, 8 to 32 tokens, cold weights):
// the choice takes 1.1 % more than the best one on average, 12 % at most; scaled, the estimate is within 7 % (rms) of the times.
inline RegPlan reg_plan(uint32_t n_hb, uint32_t subs, uint32_t n_chunks, uint32_t bits, uint32_t tokens, const uint32_t (&resident)[4]) {
    RegPlan best;
    const uint32_t n_steps = (n_chunks + 3) / 4, nt = (tokens + 7) / 8, units = bits == 4 ? 4 : 8;
    const double more = nt - 1.0, busy = bits == 4 ? 800.0 + 66.0 * more : 1540.0 + 180.0 * more,
                 chain = bits == 4 ? 2900.0 + 340.0 * more : 3450.0 + 500.0 * more;
    for (uint32_t i = 0; i < 4; i++) {
        const uint32_t ctas = 1u << i;
        if (!resident[i] || ctas > n_steps) continue;
        const uint32_t rows = (n_hb + resident[i] - 1) / resident[i], span = (n_steps + ctas - 1) / ctas;
        for (uint32_t parts = 1; parts <= REG_WARPS && parts <= span; parts++) {
            const uint32_t jobs = rows * subs * parts;
            RegPlan p;
            p.ctas = ctas;
            p.rows = rows;
            p.parts = parts;
            p.clusters = (n_hb + rows - 1) / rows;
            const size_t x = (size_t)span * units * nt * 512, sums = (size_t)((rows * 4 + ctas - 1) / ctas) * subs * ctas * parts * nt * 256;
            p.smem = REG_NORM_BYTES + x + sums;
            if (p.smem > REG_MAX_SMEM) break;
            const double steps = (span + parts - 1) / parts, rounds = (jobs + REG_WARPS - 1) / REG_WARPS, last = jobs % REG_WARPS;
            const double per = jobs / REG_WARPS * (REG_WARPS / 4) + (uint32_t)(last + 3) / 4;  // jobs of the first sub-partition
            const double cost = x / 16.0 + (per * steps * busy > rounds * steps * chain ? per * steps * busy : rounds * steps * chain) + rounds * 150.0 +
                     (ctas > 1 ? 1000.0 : 0.0) + jobs * nt * 140.0;
            p.cycles = bits == 4 ? 0.93 * cost + 5500.0 - 800.0 * nt : 0.69 * cost + 4300.0 + 400.0 * nt;
            if (p.cycles < best.cycles) best = p;
        }
    }
    return best;
}

}  // namespace prism
