// Frames of one work size through ChunkPlan, on the host: samples of given density (nodes a sample, by eighth of the
// frame), two chunks in flight at most.  Arguments: work lanes pool nominal frames d0 .. d7.  Prints a line a frame:
// chunks done, chunks that filled the pool, samples rendered, largest chunk.  Exit code 1: a chunk larger
// than the pool, a sample rendered twice, or no progress.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "tree_plan.h"

int main(int argc, char** argv) {
    if (argc < 14) return 2;
    auto num = [&](int i) { return (uint32_t)std::strtoul(argv[i], nullptr, 10); };
    const uint32_t work = num(1), lanes = num(2), pool = num(3), nominal = num(4), frames = num(5);
    double density[8];
    for (int i = 0; i < 8; ++i) density[i] = std::strtod(argv[6 + i], nullptr);
    std::vector<double> before(work + 1, 0.0);
    for (uint32_t i = 0; i < work; ++i) before[i + 1] = before[i] + density[(uint64_t)i * 8 / work];
    rg::TreeLoad load;
    for (uint32_t f = 0; f < frames; ++f) {
        rg::ChunkPlan plan(work, lanes, pool, nominal, std::move(load));
        std::vector<char> seen(work, 0);
        struct Lane {
            uint32_t base, n;
            bool busy;
        } lane[2] = {};
        uint32_t done = 0, full = 0, samples = 0, largest = 0;
        for (uint32_t l = 0; l < lanes; ++l) lane[l].busy = plan.next(lane[l].base, lane[l].n);
        for (uint32_t turn = 0; lane[0].busy || lane[1].busy; ++turn) {
            if (turn > 4 * work + 100) return 1;
            Lane& L = lane[turn % 2];
            if (!L.busy) continue;
            if (L.n == 0 || L.n > pool) return 1;
            largest = std::max(largest, L.n);
            const uint32_t nodes = (uint32_t)(before[L.base + L.n] - before[L.base]);
            if (nodes > pool && L.n > 1) {
                plan.filled(L.base, L.n);
                ++full;
            } else {
                plan.done(L.base, L.n, nodes);
                for (uint32_t i = L.base; i < L.base + L.n; ++i)
                    if (seen[i]++) return 1;
                samples += L.n;
                ++done;
            }
            L.busy = plan.next(L.base, L.n);
        }
        load = plan.load();
        std::printf("%u %u %u %u\n", done, full, samples, largest);
    }
    return 0;
}
