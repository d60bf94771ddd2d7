// One fixpoint iteration of fused::slice_task on the CPU (device_emulation.hpp)
// over an instance drawn from a seed, against the same iteration state by
// state:
//   slice_check <order seed: 0 ascending, 1 descending, else shuffled> <seed>
//               <rows> <x cells> <inputs> <inputs a pass> <group: 32 = a warp>
//               <hits: 1 = no input of the first pass hits, all later do> <valid test> <rows a block>
// Prints the first difference and returns 1.
#include <random>

#include "device_emulation.hpp"

#include "gsc_fused_body.cuh"

using namespace gsc_b200;

namespace {

template <typename T>
std::vector<T> zeros(size_t n, T v = T{}) {
    return std::vector<T>(n, v);
}

struct Box {
    int x0, x1, y0, y1;   // offsets from the state's cell
    uint32_t z, nz, v, nv;
};

template <int W>
int check(int argc, char** argv) {
    const uint64_t order_seed = std::strtoull(argv[1], nullptr, 10), seed = std::strtoull(argv[2], nullptr, 10);
    const uint32_t n1 = std::atoi(argv[3]), n0 = std::atoi(argv[4]), M = std::atoi(argv[5]), pass = std::atoi(argv[6]);
    const uint32_t threads = std::atoi(argv[7]);
    const bool burst = argc > 8 && std::atoi(argv[8]) != 0, need_valid = argc > 9 && std::atoi(argv[9]) != 0;
    std::mt19937_64 rng(seed);
    const auto below = [&](uint32_t n) { return static_cast<uint32_t>(rng() % n); };

    GridInfo g{};
    g.n[0] = n0;
    g.n[1] = n1;
    g.n[2] = 4;
    g.n[3] = 2;
    g.W = W;
    g.sw = (n1 * W + 3) & ~3u;
    g.slices = 8;
    g.rows = static_cast<uint64_t>(n1) * g.slices;
    g.S = g.rows * n0;
    g.ma = M;
    g.mw = 1;
    g.M = M;
    g.K = 1;
    g.xy_planes = 1;
    const uint32_t words = g.slices * g.sw, W1 = (n1 + 31) / 32, slice = 5;

    // Sets: D', the valid set, the slice's active states.
    auto dp0 = zeros<uint4>(words / 4), dp1 = dp0, validb = dp0, active = dp0, reach = dp0;
    bword* D = reinterpret_cast<bword*>(dp0.data());
    bword* V = reinterpret_cast<bword*>(validb.data());
    bword* A = reinterpret_cast<bword*>(active.data());
    bword* R = reinterpret_cast<bword*>(reach.data());
    const auto word_of = [&](uint32_t s, uint32_t y, uint32_t x) { return s * g.sw + y * W + x / 32; };
    for (uint32_t s = 0; s < g.slices; ++s)
        for (uint32_t y = 0; y < n1; ++y)
            for (uint32_t x = 0; x < n0; ++x) {
                const bword bit = bword(1) << (x % 32);
                const bool d = burst ? x >= n0 / 2 : below(16) == 0;
                if (d) D[word_of(s, y, x)] |= bit;
                if (need_valid ? below(3) == 0 : true) V[word_of(s, y, x)] |= bit;
                if (s == slice && (burst ? x < n0 / 4 : below(2) == 0)) A[word_of(s, y, x)] |= bit;
            }
    dp1 = dp0;

    // Inputs: boxes of at most 8 x 3 cells over at most two theta and v cells
    // (theta wraps).
    std::vector<Box> box(M);
    std::vector<SliceRep> reps(static_cast<size_t>(g.slices) * M);
    auto needv = zeros<uint32_t>(static_cast<size_t>(g.slices) * M * W1, 0xFFFFFFFFu);
    for (uint32_t j = 0; j < M; ++j) {
        Box& b = box[j];
        if (burst) {
            b = j < pass ? Box{static_cast<int>(n0 / 2), static_cast<int>(n0 / 2), 0, 0, 1, 1, 1, 1} : Box{0, 0, 0, 0, 1, 1, 1, 1};
        } else {
            b.x0 = static_cast<int>(below(9)) - 4;
            b.x1 = b.x0 + static_cast<int>(below(8));
            b.y0 = static_cast<int>(below(3)) - 1;
            b.y1 = b.y0 + static_cast<int>(below(3));
            b.z = below(4);
            b.nz = 1 + below(2);
            b.v = below(2);
            b.nv = 1 + (b.v == 0 ? below(2) : 0u);
        }
        SliceRep r{};
        r.j = j;
        r.zw = pack16(b.z, b.nz);
        r.vw = pack16(b.v, b.nv) | (need_valid ? 0x80000000u : 0u);
        r.hx = static_cast<uint32_t>(b.x1 - b.x0 + 1) | ((static_cast<uint32_t>(b.x0) & 0xFFu) << 8) | kBoxX | kBoxY;
        r.hy = static_cast<uint32_t>(b.y1 - b.y0 + 1) | ((static_cast<uint32_t>(b.y0) & 0xFFu) << 8);
        const int x0 = std::max(0, -b.x0), x1 = std::min<int>(n0, static_cast<int>(n0) - b.x1);
        const int y0 = std::max(0, -b.y0), y1 = std::min<int>(n1, static_cast<int>(n1) - b.y1);
        r.xr = pack16(x0, std::max(x0, x1));
        r.yr = pack16(y0, std::max(0, y1 - y0));
        reps[static_cast<size_t>(slice) * M + j] = r;
    }
    auto nreps = zeros<uint32_t>(g.slices, M);
    auto controller = zeros<uint32_t>(g.S, kInvalid32), step = controller;
    auto rowlost = zeros<uint32_t>(2 * (g.slices * W1 + 1));
    auto stats = zeros<unsigned long long>(kStatsCols * 4);
    FixControl fc{};
    fc.max_iterations = 2;
    fc.stats_cap = 4;

    // The same iteration state by state.
    auto want = controller;
    auto wantA = active, wantD = dp0, wantR = reach;
    uint64_t hits = 0;
    for (uint32_t y = 0; y < n1; ++y)
        for (uint32_t x = 0; x < n0; ++x) {
            const bword bit = bword(1) << (x % 32);
            const uint32_t e = word_of(slice, y, x);
            if (!(A[e] & bit)) continue;
            for (uint32_t j = 0; j < M; ++j) {
                const Box& b = box[j];
                const int xa = static_cast<int>(x) + b.x0, xb = static_cast<int>(x) + b.x1;
                const int ya = static_cast<int>(y) + b.y0, yb = static_cast<int>(y) + b.y1;
                if (xa < 0 || ya < 0 || xb >= static_cast<int>(n0) || yb >= static_cast<int>(n1)) continue;
                bool blocked = false, has_valid = false;
                for (uint32_t v = b.v; v < b.v + b.nv; ++v)
                    for (uint32_t i = 0; i < b.nz; ++i)
                        for (int yy = ya; yy <= yb; ++yy)
                            for (int xx = xa; xx <= xb; ++xx) {
                                const uint32_t q = word_of((b.z + i) % g.n[2] + g.n[2] * v, yy, xx);
                                blocked |= (D[q] >> (xx % 32)) & 1u;
                                has_valid |= (V[q] >> (xx % 32)) & 1u;
                            }
                if (blocked || (need_valid && !has_valid)) continue;
                want[(static_cast<uint64_t>(slice) * n1 + y) * n0 + x] = j;
                reinterpret_cast<bword*>(wantA.data())[e] &= ~bit;
                reinterpret_cast<bword*>(wantR.data())[e] |= bit;
                reinterpret_cast<bword*>(wantD.data())[e] &= ~bit;
                ++hits;
                break;
            }
        }

    FusedFixArgs a{};
    a.validb = V;
    a.dp[0] = D;
    a.dp[1] = reinterpret_cast<bword*>(dp1.data());
    a.reach0 = R;
    a.active = A;
    a.controller = controller.data();
    a.reach_step = step.data();
    a.fc = &fc;
    a.stats = stats.data();
    a.reps = reps.data();
    a.nreps = nreps.data();
    a.pass = pass;
    a.direct = 1;
    a.shape.part_rows = argc > 10 ? std::atoi(argv[10]) : n1;
    a.rowlost = rowlost.data();
    a.rl_words = g.slices * W1 + 1;
    a.needv = needv.data();

    const size_t smem_words = 8ull * pass + g.sw + pass * W1 + 2 * W1 + kHitNotes * (W + 1) + (n1 + 1) / 2 + 4;
    auto smem = zeros<uint4>((smem_words + 3) / 4);
    uint32_t meta[3] = {};
    std::vector<uint32_t> order(threads);
    for (uint32_t i = 0; i < threads; ++i) order[i] = order_seed == 1 ? threads - 1 - i : i;
    std::mt19937_64 shuffle(order_seed);
    if (order_seed > 1) std::shuffle(order.begin(), order.end(), shuffle);
    bool ended = true;
    for (uint32_t part = 0; ended && part < a.shape.parts(n1); ++part) ended = emu::run_block(threads, order, [&] {
        if (threads == 32)
            fused::slice_task<W, 1, 1, true, false, false>(g, a, slice, 0, reinterpret_cast<bword*>(smem.data()), meta);
        else
            fused::slice_task<W, 1, 1, false, false, true>(g, a, slice, part, reinterpret_cast<bword*>(smem.data()), meta);
    });
    if (!ended) {
        std::printf("the threads wait for one another\n");
        return 1;
    }
    for (uint64_t s = 0; s < g.S; ++s)
        if (controller[s] != want[s]) {
            std::printf("state %llu: input %u, expected %u\n", static_cast<unsigned long long>(s), controller[s], want[s]);
            return 1;
        }
    const bool same = !std::memcmp(active.data(), wantA.data(), 4ull * words) &&
                      !std::memcmp(reach.data(), wantR.data(), 4ull * words) &&
                      !std::memcmp(dp1.data(), wantD.data(), 4ull * words);
    if (!same) {
        std::printf("the sets differ\n");
        return 1;
    }
    // The rows that lost a cell, and nothing past the last.
    for (uint32_t y = 0; y < 32 * W1; ++y) {
        bool lost = false;
        for (uint32_t w = 0; y < n1 && w < W; ++w)
            lost |= D[slice * g.sw + y * W + w] != reinterpret_cast<const bword*>(wantD.data())[slice * g.sw + y * W + w];
        if (((rowlost[a.rl_words + slice * W1 + y / 32] >> (y % 32)) & 1u) != lost) {
            std::printf("row %u is recorded wrongly\n", y);
            return 1;
        }
    }
    std::printf("ok %llu\n", static_cast<unsigned long long>(hits));
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    if (argc < 8) return 2;
    return std::atoi(argv[4]) <= 32 ? check<1>(argc, argv) : check<2>(argc, argv);
}
