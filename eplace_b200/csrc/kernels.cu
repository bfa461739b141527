// kernels.cu -- the launchers of the loop's kernels: each picks the working
// precision from KernelCtx::fp64 (loop.h).  Also the kernels that need none, the
// grids of the reductions, and the L1 / shared-memory split.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <utility>
#include <vector>

#include "loop.h"

namespace ep {

namespace {

// The accepted trial ends the step: the scalar side of k_update.
__global__ void k_bktrk_commit(DevScalars *__restrict__ S) {
    pdl_begin();
    if (S->done) return;
    S->iter += 1;
    S->lambda_pending = 1;
    if (S->stop_pending) {
        S->done = 1;
        if (S->stage == EP_STAGE_MGP) S->mgp_iterations = S->iter;
    }
}

// Scalars that a call sets before its kernels, in stream order (a read-back, a
// change on the host and a copy cost two synchronisations).
__global__ void k_set_scalars(DevScalars *__restrict__ S, ScalarSet what, double value) {
    pdl_begin();
    if (what == ScalarSet::kLambda) {
        S->lambda = value;
        return;
    }
    S->lambda0_mode = 1;  // the next evaluation is initialization()'s
    if (what == ScalarSet::kInitialize) {
        S->lambda = 0.0;
        S->status = 0;
        S->done = 0;
    }
}

}  // namespace

int launch_priority(bool high) {
    // the range is the same on every device; a function-local static is
    // initialised once even when engines are created on several threads
    static const int2 range = [] {
        int l = 0, h = 0;
        cudaDeviceGetStreamPriorityRange(&l, &h);
        return make_int2(l, h);
    }();
    return high ? range.y : range.x;
}

int prep_blocks(const Grid &g) { return std::min(blocks_for(g.nx * g.ny, kThreads), kSms * 8); }

int reduction_blocks(const DeviceNetlist &d, int which) {
    switch (which) {
        case 0: return d.n_block_nets + std::min(blocks_for(d.n_net_tasks - d.n_block_nets, kNetWarps), kNetBlocks);
        default: return big_blocks(d) + std::min(blocks_for(d.n_obj, kThreads), kCombineBlocks);
    }
}

void launch_scatter(const KernelCtx &c, const DeviceNetlist &d, ull *maps, const DevScalars *S, cudaStream_t st) {
    c.fp64 ? Loop<double>::scatter(c, d, maps, S, st) : Loop<float>::scatter(c, d, maps, S, st);
}

void launch_update_scatter(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g,
                           void *y_prev, void *g_prev, ull *maps, DevScalars *S, int *progress, cudaStream_t st) {
    c.fp64 ? Loop<double>::update_scatter(c, d, pos, x, g, y_prev, g_prev, maps, S, progress, st)
           : Loop<float>::update_scatter(c, d, pos, x, g, y_prev, g_prev, maps, S, progress, st);
}

void launch_prep(const KernelCtx &c, ull *node_q, ull *filler_q, const float2 *static_map, void *rho,
                 void *rho_bf16, float *node_f, float *filler_f, int zero_maps, DevScalars *S, cudaStream_t st) {
    c.fp64 ? Loop<double>::prep(c, node_q, filler_q, static_map, rho, rho_bf16, node_f, filler_f, zero_maps, S, st)
           : Loop<float>::prep(c, node_q, filler_q, static_map, rho, rho_bf16, node_f, filler_f, zero_maps, S, st);
}

void launch_wirelength(const KernelCtx &c, const DeviceNetlist &d, void *pin_grad, DevScalars *S, cudaStream_t st) {
    c.fp64 ? Loop<double>::wirelength(c, d, pin_grad, S, st) : Loop<float>::wirelength(c, d, pin_grad, S, st);
}

void launch_combine(const KernelCtx &c, const DeviceNetlist &d, const void *field, const void *pin_grad, void *g,
                    const void *g_prev, const void *y_prev, void *dump_gd, void *dump_gwl, int stepping, DevScalars *S,
                    cudaStream_t st) {
    c.fp64 ? Loop<double>::combine(c, d, field, pin_grad, g, g_prev, y_prev, dump_gd, dump_gwl, stepping, S, st)
           : Loop<float>::combine(c, d, field, pin_grad, g, g_prev, y_prev, dump_gd, dump_gwl, stepping, S, st);
}

void launch_update(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g, void *y_prev,
                   void *g_prev, DevScalars *S, int *progress, cudaStream_t st) {
    c.fp64 ? Loop<double>::update(c, d, pos, x, g, y_prev, g_prev, S, progress, st)
           : Loop<float>::update(c, d, pos, x, g, y_prev, g_prev, S, progress, st);
}

void launch_bktrk_move(const KernelCtx &c, const DeviceNetlist &d, const void *ysave, const void *g, const void *x,
                       void *pos, void *xtrial, const DevScalars *S, cudaStream_t st) {
    c.fp64 ? Loop<double>::bktrk_move(c, d, ysave, g, x, pos, xtrial, S, st)
           : Loop<float>::bktrk_move(c, d, ysave, g, x, pos, xtrial, S, st);
}

void launch_bktrk_commit(DevScalars *S, cudaStream_t st) { launch_k(k_bktrk_commit, 1, 1, 0, st, S); }

void launch_stage_begin(const KernelCtx &c, const DeviceNetlist &d, const void *pos, void *x, int step_cap,
                        DevScalars *S, int *progress, cudaStream_t st) {
    c.fp64 ? Loop<double>::stage_begin(d, pos, x, step_cap, S, progress, st)
           : Loop<float>::stage_begin(d, pos, x, step_cap, S, progress, st);
}

void launch_set_scalars(DevScalars *S, ScalarSet what, double value, cudaStream_t st) {
    launch_k(k_set_scalars, 1, 1, 0, st, S, what, value);
}

void launch_wrap_up(const KernelCtx &c, const DeviceNetlist &d, void *pos, const void *x, cudaStream_t st) {
    c.fp64 ? Loop<double>::wrap_up(c, d, pos, x, st) : Loop<float>::wrap_up(c, d, pos, x, st);
}

void launch_hpwl(const KernelCtx &c, const DeviceNetlist &d, int mode, DevScalars *S, cudaStream_t st) {
    c.fp64 ? Loop<double>::hpwl(c, d, mode, S, st) : Loop<float>::hpwl(c, d, mode, S, st);
}

int carveout_percent(size_t smem_bytes) {
    // shared-memory capacities of an sm_100 SM, KB; the driver maps a
    // preferred percentage of the largest to one of them, so ask for the
    // middle of the interval that rounds to the capacity wanted
    static const int kConfigs[] = {0, 8, 16, 32, 64, 100, 132, 164, 196, 228};
    const double kb = (double)smem_bytes / 1024.0;
    for (int i = 1; i < 10; i++)
        if (kConfigs[i] >= kb) return (int)std::ceil(50.0 * (kConfigs[i - 1] + kConfigs[i]) / 228.0);
    return 100;
}

// One L1/shared split, kLoopSmemBytes of shared memory, for every kernel of
// the loop: an SM whose split has to change between consecutive kernels must
// drain first, which costs the programmatic overlap of the launches (on the
// 200k-cell solve with the FFT Poisson path: 14.5 ms per solve with one split
// against 18.3 ms with the driver's choice per kernel).  64 KB holds the
// per-net and combine kernels' staging at full occupancy and leaves 192 KB of
// L1; smaller splits cost them occupancy, larger ones L1.
// Function attributes belong to the current device, and setting one loads the
// kernel: once per device for the kernels that every loop has, and for each
// precision and wirelength form once an engine has it.  (All forms of both
// precisions at once, in one file: 17.4 ms for the first engine of a process at
// 100 cells, 13.5 so.)
void set_loop_carveout(const KernelCtx &c) {
    static std::mutex mu;
    static std::vector<std::pair<int, int>> done;  // device, form (-1: the common kernels)
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    auto first = [&](int form) {
        if (std::find(done.begin(), done.end(), std::make_pair(dev, form)) != done.end()) return false;
        done.emplace_back(dev, form);
        return true;
    };
    std::lock_guard<std::mutex> lock(mu);
    const int carveout = carveout_percent(kLoopSmemBytes);
    auto set = [&](const std::vector<const void *> &fns) {
        for (const void *f : fns) cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, carveout);
    };
    const bool exact = c.exact_exp != 0, lse = c.lse != 0;
    if (first((c.fp64 ? 4 : 0) + (exact ? 2 : 0) + (lse ? 1 : 0)))
        set(c.fp64 ? Loop<double>::kernels(exact, lse) : Loop<float>::kernels(exact, lse));
    if (first(-1)) {
        set({(const void *)k_bktrk_commit, (const void *)k_set_scalars});
        set_sgemm_carveout(carveout);
    }
}

}  // namespace ep
