// Prints tree_pool_nodes(samples, nodes a sample, least) for every triple of arguments (host code only), then the
// largest pool.
#include <cstdio>
#include <cstdlib>

#include "rg_internal.cuh"

int main(int argc, char** argv) {
    for (int i = 1; i + 2 < argc; i += 3)
        std::printf("%zu\n", rg::tree_pool_nodes(std::strtoull(argv[i], nullptr, 10), std::strtoull(argv[i + 1], nullptr, 10),
                                                 std::strtoull(argv[i + 2], nullptr, 10)));
    std::printf("%u\n", (unsigned)rg::kTreePoolMax);
    return 0;
}
