// Host rules of the fused plan, for a grid and the box widths in use:
//   plan_check <n0> <n1> <n2> <n3> <theta widths> <v widths> <y levels (mask)> <cells a window> <batched>
// Prints whether windows are read directly, and the words of a set's dilated copies.
//   plan_check shape <n0> <n1> <slices> <representatives a slice>
// Prints the threads, rows a part, parts and kernel of a launch.
#include <iostream>
#include <string>

#include "device_emulation.hpp"

using namespace gsc_b200;

int main(int argc, char** argv) {
    if (argc == 6 && std::string(argv[1]) == "shape") {
        GridInfo g{};
        g.n[0] = std::atoi(argv[2]);
        g.n[1] = std::atoi(argv[3]);
        g.W = (g.n[0] + kBits - 1) / kBits;
        const SliceShape s = slice_shape(g, std::atoi(argv[4]), std::atoi(argv[5]));
        std::cout << s.threads << " " << s.part_rows << " " << s.parts(g.n[1]) << " " << s.wide << "\n";
        return 0;
    }
    if (argc < 10) return 2;
    GridInfo g{};
    for (int d = 0; d < 4; ++d) g.n[d] = static_cast<uint32_t>(std::atoi(argv[1 + d]));
    g.W = (g.n[0] + kBits - 1) / kBits;
    g.sw = (g.n[1] * g.W + 3) & ~3u;
    g.slices = g.n[2] * g.n[3];
    PlanRecord pl{};
    pl.dil.nk = std::atoi(argv[5]);
    pl.dil.nl = std::atoi(argv[6]);
    pl.ylevels = std::atoi(argv[7]);
    pl.reps = g.slices;
    pl.rep_rows = pl.reps * std::strtoull(argv[8], nullptr, 10);
    std::cout << reads_windows_directly(g, pl, std::atoi(argv[9]) != 0) << " " << dilated_words(g, pl.dil, pl.ylevels) << "\n";
    return 0;
}
