// One block of the batched satisfaction kernel's task walk
// (fused::batch_slices) on the CPU (device_emulation.hpp) over a list of
// instances that have stopped and instances that run, in turn:
//   batch_check <order seed: 0 ascending, 1 descending, else shuffled> <threads> <warp tasks>
// A stopped instance's sets are left null.  Prints "ok" and the running
// instances' states, or what went wrong.
#include <memory>
#include <random>

#include "device_emulation.hpp"

#include "gsc_fused_body.cuh"

using namespace gsc_b200;

namespace {

// 32 x 8 cells in each of two slices, one input whose box is the state's own
// cell, every state active and D' empty: every state is satisfied by input 0.
struct Instance {
    InstanceDesc d{};
    FixControl fc{};
    std::vector<uint4> dp0, dp1, active, reach;
    std::vector<SliceRep> reps;
    std::vector<uint32_t> nreps, controller, step, rowlost;
    std::vector<unsigned long long> stats;
    explicit Instance(bool stopped) {
        GridInfo& g = d.g;
        g.n[0] = 32;
        g.n[1] = 8;
        g.n[2] = 2;
        g.n[3] = 1;
        g.W = 1;
        g.sw = 8;
        g.slices = 2;
        g.rows = 16;
        g.S = 512;
        g.ma = g.mw = g.M = g.K = g.xy_planes = 1;
        d.a.fc = &fc;
        if (stopped) {
            fc.stop = 1;
            return;
        }
        fc.max_iterations = 2;
        fc.stats_cap = 4;
        fc.candidate_count = 1;
        dp0.resize(4);
        dp1 = reach = dp0;
        active.assign(4, make_uint4(~0u, ~0u, ~0u, ~0u));
        SliceRep r{};
        r.zw = pack16(0, 1);
        r.vw = pack16(0, 1);
        r.hx = 1u | kBoxX | kBoxY;
        r.hy = 1u;
        r.xr = pack16(0, 32);
        r.yr = pack16(0, 8);
        reps.assign(2, r);
        nreps.assign(2, 1u);
        controller.assign(g.S, kInvalid32);
        step = controller;
        rowlost.assign(6, 0u);
        stats.assign(kStatsCols * 4, 0ull);
        FusedFixArgs& a = d.a;
        a.dp[0] = reinterpret_cast<bword*>(dp0.data());
        a.dp[1] = reinterpret_cast<bword*>(dp1.data());
        a.active = reinterpret_cast<bword*>(active.data());
        a.reach0 = reinterpret_cast<bword*>(reach.data());
        a.controller = controller.data();
        a.reach_step = step.data();
        a.stats = stats.data();
        a.reps = reps.data();
        a.nreps = nreps.data();
        a.pass = 1;
        a.direct = 1;
        a.rowlost = rowlost.data();
        a.rl_words = 3;
    }
};

}  // namespace

int main(int argc, char** argv) {
    if (argc < 4) return 2;
    const uint64_t seed = std::strtoull(argv[1], nullptr, 10);
    const uint32_t threads = std::atoi(argv[2]);
    const bool warp = std::atoi(argv[3]) != 0;
    std::vector<std::unique_ptr<Instance>> inst;
    for (int i = 0; i < 6; ++i) inst.push_back(std::make_unique<Instance>(i % 2 == 0));
    std::vector<InstanceDesc> descs;
    std::vector<uint32_t> slot, off{0};
    for (uint32_t i = 0; i < inst.size(); ++i) {
        descs.push_back(inst[i]->d);
        slot.push_back(i);
        off.push_back(off.back() + 2);
    }
    WorkList wl{};
    wl.slot = slot.data();
    wl.sat_off = off.data();
    wl.n = static_cast<uint32_t>(inst.size());
    const uint32_t task_words = (8 + 8 + 3 + kHitNotes * 2 + 4 + 7) & ~3u;
    std::vector<uint4> smem(task_words / 4 * (threads / 32));
    std::vector<InstanceDesc> sd(threads / 32);
    std::vector<uint32_t> meta(3 * (threads / 32));
    std::vector<uint32_t> order(threads);
    for (uint32_t i = 0; i < threads; ++i) order[i] = seed == 1 ? threads - 1 - i : i;
    std::mt19937_64 shuffle(seed);
    if (seed > 1) std::shuffle(order.begin(), order.end(), shuffle);
    const bool ended = emu::run_block(threads, order, [&] {
        bword* s = reinterpret_cast<bword*>(smem.data());
        const uint32_t grp = warp ? emu::cur / 32 : 0u, groups = warp ? threads / 32 : 1u;
        if (warp)
            fused::batch_slices<1, true>(descs.data(), wl, 0, wl.n, grp, groups, s + grp * task_words, sd[grp], &meta[3 * grp]);
        else
            fused::batch_slices<1, false>(descs.data(), wl, 0, wl.n, grp, groups, s, sd[grp], meta.data());
    });
    if (!ended) {
        std::printf("the threads wait for one another\n");
        return 1;
    }
    uint32_t states = 0;
    for (const auto& x : inst) {
        if (x->controller.empty()) continue;
        if (x->fc.iter != 1) {
            std::printf("an instance is at iteration %u\n", x->fc.iter);
            return 1;
        }
        for (uint32_t c : x->controller) states += c == 0;
    }
    std::printf("ok %u\n", states);
    return 0;
}
