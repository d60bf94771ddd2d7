// gsc_batch_kernels.cu -- the fused fixpoint over many instances at once.
//
// Each kernel is one launch over listed instances: blocks walk a task list
// (instance k owns tasks off[k] .. off[k+1]-1, found by a binary search) and
// run the same device bodies as the one-problem kernels
// (gsc_fused_body.cuh), so an instance computes the same bits alone and in a
// batch.  Instances that have stopped skip their tasks.  One iteration:
//   k_batch_dilate  (theta, v)-dilated D' of the running instances that read it;
//   k_batch_slice   one launch per row width, a task per slice of every running
//                   instance of that width; an instance's last task (ticket)
//                   applies its stop rules;
//   k_batch_status  one block: a copy of every instance's control record, the
//                   number still running, and the CUDA-graph loop condition.
// Instances big enough to fill the GPU alone run the one-problem kernels in
// the same step (launch_batch_step) and share only init and status.
#include "gsc_fused_body.cuh"

namespace gsc_b200 {

using namespace fused;

namespace {

__global__ void __launch_bounds__(256) k_batch_init(const InstanceDesc* __restrict__ descs, WorkList wl) {
    const uint32_t total = wl.ini_off[wl.n];
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const uint32_t k = find_task(wl.ini_off, wl.n, t);
        const InstanceDesc& d = descs[wl.slot[k]];
        const uint64_t b = static_cast<uint64_t>(t - wl.ini_off[k]) * wl.chunk;
        const uint64_t e_end = b + wl.chunk;
        const uint64_t wend = min(e_end, static_cast<uint64_t>(d.words));
        for (uint64_t e = b + threadIdx.x; e < wend; e += blockDim.x) init_word(d.a, e);
        const uint64_t send = min(e_end, d.g.S);
        for (uint64_t s = b + threadIdx.x; s < send; s += blockDim.x) init_state(d.a, d.cand, s);
        const uint64_t tend = min(e_end, static_cast<uint64_t>(kStatsCols) * d.stats_cap);
        for (uint64_t i = b + threadIdx.x; i < tend; i += blockDim.x) d.a.stats[i] = 0;
        if (t == wl.ini_off[k] && threadIdx.x == 0) init_control(d.a.fc, d.max_iterations, d.stats_cap, d.counts);
    }
}

__global__ void __launch_bounds__(256) k_batch_dilate(const InstanceDesc* __restrict__ descs, WorkList wl) {
    extern __shared__ __align__(16) bword smem[];
    const uint32_t total = wl.dil_off[wl.n];
    for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
        // Instances that read D' itself have no task: the last of equal offsets.
        const uint32_t k = find_task(wl.dil_off, wl.n, t);
        const InstanceDesc& d = descs[wl.slot[k]];
        if (d.a.fc->stop) continue;
        const uint32_t c = d.a.fc->iter;
        const uint32_t* lost = c > 0 ? d.a.rowlost + (c & 1) * d.a.rl_words : nullptr;
        dilate_tile(d.g, d.a.dp[c & 1], d.a.dzw, d.a.dil, d.a.tile, t - wl.dil_off[k], lost, smem);
        __syncthreads();
    }
}

// One launch per row width: the slices of the instances [kb, ke) of the list,
// whose rows have W words (batch_slices).  The dynamic shared memory holds the
// largest instance's staging, once per task group: every warp of the block
// (WARP) or the block.
template <int W, bool WARP>
__global__ void __launch_bounds__(256) k_batch_slice(const InstanceDesc* __restrict__ descs, WorkList wl, uint32_t kb,
                                                     uint32_t ke, uint32_t task_words) {
    extern __shared__ __align__(16) bword smem[];
    constexpr uint32_t kGroups = WARP ? 8u : 1u;
    __shared__ __align__(16) InstanceDesc sd[kGroups];
    __shared__ uint32_t s_meta[kGroups][3];
    const uint32_t grp = WARP ? (threadIdx.x >> 5) : 0u;
    const uint32_t ngrp = WARP ? (blockDim.x >> 5) : 1u;
    batch_slices<W, WARP>(descs, wl, kb, ke, blockIdx.x * ngrp + grp, gridDim.x * ngrp, smem + grp * task_words, sd[grp],
                          s_meta[grp]);
}

__global__ void __launch_bounds__(256) k_batch_status(const InstanceDesc* __restrict__ descs, WorkList wl,
                                                      cudaGraphConditionalHandle cond, int use_cond) {
    __shared__ uint32_t running;
    if (threadIdx.x == 0) running = 0;
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t k = threadIdx.x; k < wl.n; k += blockDim.x) {
        const FixControl* fc = descs[wl.slot[k]].a.fc;
        if (wl.status) wl.status[k] = *fc;
        mine += fc->stop ? 0u : 1u;
    }
    if (mine) atomicAdd(&running, mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (wl.running) *wl.running = running;
        if (use_cond) cudaGraphSetConditional(cond, running ? 1u : 0u);
    }
}

inline unsigned int grid_of(uint32_t tasks, uint32_t cap) {
    const uint32_t b = tasks < cap ? tasks : cap;
    return b ? b : 1u;
}

template <int W, bool WARP>
cudaError_t launch_slice_t(const InstanceDesc* descs, const WorkList& wl, const BatchClass& c, const BatchShape& sh,
                           cudaStream_t st) {
    const cudaError_t e = allow_smem(k_batch_slice<W, WARP>);
    if (e != cudaSuccess) return e;
    const uint32_t per_block = WARP ? sh.sat_threads / 32 : 1u;
    const uint32_t tasks = (c.tasks + per_block - 1) / per_block;
    const uint32_t blocks = sh.sat_blocks ? grid_of(tasks, sh.sat_blocks) : grid_of(tasks, 0xFFFFFFFFu);
    k_batch_slice<W, WARP><<<blocks, sh.sat_threads, per_block * c.smem, st>>>(
        descs, wl, c.begin, c.end, static_cast<uint32_t>(c.smem / sizeof(bword)));
    return cudaGetLastError();
}

template <int W>
cudaError_t launch_slice_w(const InstanceDesc* descs, const WorkList& wl, const BatchClass& c, const BatchShape& sh,
                           cudaStream_t st) {
    // Warp tasks whose staging does not fit one block run one task per block.
    return sh.warp && (sh.sat_threads / 32) * c.smem <= kFusedSmemOptIn
               ? launch_slice_t<W, true>(descs, wl, c, sh, st)
               : launch_slice_t<W, false>(descs, wl, c, sh, st);
}

}  // namespace

cudaError_t launch_batch_init(const InstanceDesc* descs, const WorkList& wl, const WorkTotals& tot, int sms,
                              cudaStream_t st) {
    if (tot.ini == 0) return cudaSuccess;
    k_batch_init<<<grid_of(tot.ini, 8u * sms), 256, 0, st>>>(descs, wl);
    return cudaGetLastError();
}

cudaError_t launch_batch_step(const InstanceDesc* descs, const WorkList& small, const WorkTotals& tot_small,
                              const BatchClass* classes, uint32_t nclasses, const WorkList& all,
                              const BigInstance* big, uint32_t nbig, const BatchShape& sh, int sms,
                              cudaGraphConditionalHandle cond, int use_cond, cudaStream_t st, uint32_t* launches) {
    if (sh.sat_threads < 32 || sh.sat_threads > 256 || sh.sat_threads % 32) return cudaErrorInvalidValue;
    uint32_t n = 0;
    cudaError_t e = cudaSuccess;
    // A stopped big instance's kernels return at once (they read its stop flag).
    for (uint32_t i = 0; e == cudaSuccess && i < nbig; ++i) e = launch_fused_iteration(big[i].g, big[i].a, st, &n);
    if (e == cudaSuccess && tot_small.dil) {
        e = allow_smem(k_batch_dilate);
        if (e != cudaSuccess) return e;
        k_batch_dilate<<<grid_of(tot_small.dil, 16u * sms), 256, tot_small.dil_smem, st>>>(descs, small);
        e = cudaGetLastError();
        ++n;
    }
    for (uint32_t i = 0; e == cudaSuccess && i < nclasses; ++i) {
        const BatchClass& c = classes[i];
        switch (c.W) {
            case 1: e = launch_slice_w<1>(descs, small, c, sh, st); break;
            case 2: e = launch_slice_w<2>(descs, small, c, sh, st); break;
            case 3: e = launch_slice_w<3>(descs, small, c, sh, st); break;
            case 4: e = launch_slice_w<4>(descs, small, c, sh, st); break;
            case 5: e = launch_slice_w<5>(descs, small, c, sh, st); break;
            case 6: e = launch_slice_w<6>(descs, small, c, sh, st); break;
            case 7: e = launch_slice_w<7>(descs, small, c, sh, st); break;
            default: e = launch_slice_w<8>(descs, small, c, sh, st); break;
        }
        ++n;
    }
    if (e == cudaSuccess) {
        k_batch_status<<<1, 256, 0, st>>>(descs, all, cond, use_cond);
        e = cudaGetLastError();
        ++n;
    }
    if (launches) *launches += n;
    return e;
}

}  // namespace gsc_b200
