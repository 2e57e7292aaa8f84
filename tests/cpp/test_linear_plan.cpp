// Host-only check of gemm_pays_at_8 (prism_engine_b200/csrc/linear_plan.hpp): both sides of each of its lines, and shapes that were
// measured on either side.
#include <cstdio>

#include "../../prism_engine_b200/csrc/linear_plan.hpp"

#define CHECK(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    auto pays = [](uint64_t m, uint64_t k, uint32_t bits, bool two) { return prism::gemm_pays_at_8(m, k, bits, two, 148); };
    // the GEMV is ahead
    CHECK(!pays(4608, 3584, 4, false) && !pays(3584, 3584, 4, false));             // fewer than 2^25 weights
    CHECK(!pays(2048, 18944, 4, false) && !pays(2048, 29568, 4, false) && !pays(2048, 8192, 2, true));
    CHECK(!pays(5120, 3584, 4, true) && !pays(8192, 4096, 4, true) && !pays(8192, 2048, 4, true));
    CHECK(!pays(8192, 4096, 4, false) && !pays(8192, 5120, 4, false));
    // the GEMM is
    CHECK(pays(18944, 3584, 4, true) && pays(29568, 8192, 4, true) && pays(3584, 18944, 4, false) && pays(8192, 29568, 4, false));
    CHECK(pays(8192, 8192, 4, false) && pays(10240, 8192, 4, false) && pays(10240, 2048, 4, true) && pays(6144, 8192, 4, false));
    CHECK(pays(5120, 3584, 2, true) && pays(8192, 4096, 2, false) && pays(3584, 5120, 2, true));
    // the lines
    CHECK(pays(4096, 8192, 4, false) && !pays(4096, 8191, 4, false));
    CHECK(pays(10240, 3584, 4, true) && !pays(10239, 3584, 4, true) && pays(3072, 16384, 4, false) && !pays(3071, 16384, 4, false));
    CHECK(!pays(7105, 8191, 4, false) && pays(7104, 8191, 4, false) && !pays(9472, 8191, 4, false) && pays(9473, 8191, 4, false));
    CHECK(pays(8192, 8192, 4, true) && !pays(8192, 8191, 4, true) && !pays(8191, 8192, 4, true));
    CHECK(pays(2048, 18432, 2, false) && !pays(2048, 18431, 2, false) && !pays(2047, 18944, 2, false));
    printf("ok\n");
    return 0;
}
