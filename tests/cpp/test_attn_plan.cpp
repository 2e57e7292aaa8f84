// Host-only check of attn_cluster_ctas (prism_engine_b200/csrc/attn_plan.hpp).
#include <cstdio>

#include "../../prism_engine_b200/csrc/attn_plan.hpp"

#define CHECK(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    using prism::attn_cluster_ctas;
    CHECK(attn_cluster_ctas(148, 4, 100, 128, 8) == 1 && attn_cluster_ctas(148, 4, 129, 128, 8) == 2);
    CHECK(attn_cluster_ctas(148, 4, 4096, 128, 8) == 16 && attn_cluster_ctas(148, 4, 4095, 128, 8) == 8);
    // GPUs that hold fewer clusters of 16 than the launch has, or none, keep 8
    CHECK(attn_cluster_ctas(148, 4, 4096, 128, 3) == 8 && attn_cluster_ctas(148, 1, 40960, 128, 0) == 8);
    CHECK(attn_cluster_ctas(148, 9, 8192, 128, 8) == 8 && attn_cluster_ctas(148, 8, 8192, 128, 8) == 16);
    // a CTA per SM at most
    CHECK(attn_cluster_ctas(148, 32, 8192, 128, 8) == 4 && attn_cluster_ctas(148, 200, 8192, 128, 8) == 1);
    printf("ok\n");
    return 0;
}
