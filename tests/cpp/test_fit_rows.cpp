// Host-only check of fit_rows (prism_engine_b200/csrc/scratch.hpp): the sizes it asks for when memory is short.
#include <cstdio>
#include <vector>

#include "../../prism_engine_b200/csrc/scratch.hpp"

#define CHECK(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); return 1; } } while (0)

static std::vector<unsigned> asked;
// Memory holds `room` rows.
static int run(unsigned &rows, unsigned least, unsigned room) {
    asked.clear();
    return prism::fit_rows(rows, least, [&](unsigned n) { asked.push_back(n); return n <= room ? 0 : 2; });
}

int main() {
    typedef std::vector<unsigned> V;
    unsigned rows = 2048;
    CHECK(run(rows, 61, 4096) == 0 && rows == 2048 && asked == V({2048}));
    rows = 2048;
    CHECK(run(rows, 512, 600) == 0 && rows == 512 && asked == V({2048, 1024, 512}));
    // short prompts of a batch: down to one of them, as many rows as one prompt needs
    rows = 2048;
    CHECK(run(rows, 61, 100) == 0 && rows == 64 && asked == V({2048, 1024, 512, 256, 128, 64}));
    rows = 2048;
    CHECK(run(rows, 61, 61) == 0 && rows == 61 && asked.back() == 61);
    rows = 2048;
    CHECK(run(rows, 61, 60) == 2 && rows == 61 && asked.back() == 61);
    rows = 100;
    CHECK(run(rows, 100, 60) == 2 && asked == V({100}));
    printf("ok\n");
    return 0;
}
