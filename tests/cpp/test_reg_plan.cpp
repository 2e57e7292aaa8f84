// Host-only check of reg_plan and reg_pays (prism_engine_b200/csrc/reg_plan.hpp): every part of every linear belongs to exactly one
// job, the shared memory holds what the kernel puts there, and the lines of the rule.
#include <cstdio>
#include <initializer_list>

#include "../../prism_engine_b200/csrc/reg_plan.hpp"

#define CHECK(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    const uint32_t gpus[3][4] = {{148, 74, 33, 15}, {148, 74, 0, 0}, {1, 1, 1, 1}};
    unsigned fits = 0;
    for (const auto &resident : gpus)
        for (uint32_t n_hb : {1u, 2u, 7u, 28u, 112u, 144u, 594u, 4752u})
            for (uint32_t chunks : {1u, 3u, 4u, 5u, 28u, 112u, 152u, 592u, 924u})
                for (uint32_t bits : {2u, 4u})
                    for (uint32_t subs = 1; subs <= 2; subs++)
                        for (uint32_t tokens : {1u, 8u, 9u, 24u, 32u}) {
                            const prism::RegPlan p = prism::reg_plan(n_hb, subs, chunks, bits, tokens, resident);
                            if (!p.ctas) continue;
                            fits++;
                            uint32_t i = 0;
                            while (1u << i < p.ctas) i++;
                            CHECK(1u << i == p.ctas && i < 4 && p.clusters <= resident[i] && p.parts >= 1);
                            CHECK((uint64_t)p.clusters * p.rows >= n_hb && (uint64_t)(p.clusters - 1) * p.rows < n_hb);  // no empty cluster
                            const uint32_t steps = (chunks + 3) / 4, nt = (tokens + 7) / 8;
                            uint32_t longest = 0;
                            for (uint32_t r = 0; r < p.ctas; r++) {
                                const uint32_t n = steps * (r + 1) / p.ctas - steps * r / p.ctas;
                                longest = n > longest ? n : longest;
                            }
                            const size_t x = (size_t)((steps + p.ctas - 1) / p.ctas) * (bits == 4 ? 4 : 8) * nt * 512;
                            CHECK((size_t)longest * (bits == 4 ? 4 : 8) * nt * 512 <= x);
                            // the last slot of the last octet of the owner that has most of them
                            const size_t slots = (size_t)((p.rows * 4 - 1) / p.ctas * subs + subs - 1) * p.ctas * p.parts + p.ctas * p.parts;
                            CHECK(prism::REG_NORM_BYTES + x + slots * nt * 256 <= p.smem && p.smem <= prism::REG_MAX_SMEM);
                        }
    CHECK(fits > 3000);
    using prism::reg_pays;
    auto pays = [](uint64_t m, uint64_t k, uint32_t bits, uint32_t tensors, uint32_t tokens) { return reg_pays(m, k, bits, tensors, tokens, 2, 1); };
    CHECK(pays(18944, 3584, 2, 2, 1) && !pays(29568, 8192, 2, 2, 1) && !pays(3584, 18944, 2, 1, 1) && !pays(18944, 3584, 4, 2, 1));
    CHECK(pays(3584, 18944, 2, 1, 2) && pays(8192, 29568, 2, 1, 7) && !pays(3584, 18944, 2, 1, 8) && !pays(3584, 3584, 4, 1, 8));
    CHECK(pays(3584, 3584, 4, 1, 2) && pays(3584, 3584, 4, 1, 7) && !pays(8192, 8192, 4, 1, 2));
    CHECK(pays(18944, 3584, 4, 2, 3) && !pays(8192, 29568, 4, 1, 4) && pays(8192, 29568, 4, 1, 5));
    CHECK(reg_pays(3584, 3584, 4, 1, 8, 94, 100) && !reg_pays(3584, 3584, 4, 1, 8, 96, 100) && reg_pays(3584, 3584, 4, 1, 32, 1e29, 1e30));
    CHECK(reg_pays(18944, 3584, 2, 2, 1, 38000, 1e30) && !reg_pays(19264, 3584, 2, 2, 1, 45800, 1e30) && !reg_pays(9472, 3584, 2, 2, 1, 24200, 1e30));
    CHECK(!reg_pays(896, 896, 2, 1, 6, 2, 1e30) && !reg_pays(192, 832, 2, 1, 32, 2, 1e30) && reg_pays(640, 256, 2, 1, 12, 94, 100) && !reg_pays(640, 256, 2, 1, 8, 94, 100));
    CHECK(reg_pays(1600, 192, 2, 1, 32, 2, 1e30) && !reg_pays(320, 192, 4, 1, 4, 2, 1e30) && reg_pays(192, 832, 4, 1, 4, 2, 1e30) && reg_pays(320, 192, 4, 1, 8, 2, 1e30));
    CHECK(!reg_pays(5120, 2048, 4, 1, 2, 2, 1e30) && reg_pays(2048, 5120, 4, 1, 2, 2, 1e30) && !reg_pays(4864, 896, 4, 1, 3, 2, 1e30) && reg_pays(5120, 2048, 4, 1, 3, 2, 1e30));
    printf("ok\n");
    return 0;
}
