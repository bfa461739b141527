// loop.h -- the launchers of the loop's kernels (loop_kernels.cuh) in one working
// precision.  Each precision is instantiated in a file of its own
// (loop_f32.cu, loop_f64.cu): a file's device code is loaded as a whole when its
// first kernel is used, and a process seldom uses both.
#pragma once
#include <vector>

#include "engine.h"

namespace ep {

using ull = unsigned long long;

namespace {
constexpr int kThreads = 256;
constexpr int kSms = 148;
// Grids of the kernels that loop over their work and end in a grid sum: one
// block for each that an SM holds in FP32, so that a block's reduction and the
// wait for its slowest warp are paid once.  Fixed numbers, the same in FP64, so
// that the sums do not depend on anything else.
constexpr int kNetBlocks = kSms * 6, kCombineBlocks = kSms * 3;
inline int blocks_for(int n, int t) { return (n + t - 1) / t; }


// Blocks of the object kernels that take the kBig objects (object_unit).
inline int big_blocks(const DeviceNetlist &d) {
    return d.n_huge_objs + blocks_for(d.n_big_objs - d.n_huge_objs, kThreads / 32);
}
}  // namespace

// As the launch_* functions of engine.h, which pick the precision.
template <typename R>
struct Loop {
    static void scatter(const KernelCtx &c, const DeviceNetlist &d, ull *maps, const DevScalars *S, cudaStream_t st);
    static void update_scatter(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g,
                               void *y_prev, void *g_prev, ull *maps, DevScalars *S, int *progress, cudaStream_t st);
    static void prep(const KernelCtx &c, ull *node_q, ull *filler_q, const float2 *static_map, void *rho,
                     void *rho_bf16, float *node_f, float *filler_f, int zero_maps, DevScalars *S, cudaStream_t st);
    static void wirelength(const KernelCtx &c, const DeviceNetlist &d, void *pin_grad, DevScalars *S, cudaStream_t st);
    static void hpwl(const KernelCtx &c, const DeviceNetlist &d, int mode, DevScalars *S, cudaStream_t st);
    static void combine(const KernelCtx &c, const DeviceNetlist &d, const void *field, const void *pin_grad, void *g,
                        const void *g_prev, const void *y_prev, void *dump_gd, void *dump_gwl, int stepping,
                        DevScalars *S, cudaStream_t st);
    static void update(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g, void *y_prev,
                       void *g_prev, DevScalars *S, int *progress, cudaStream_t st);
    static void bktrk_move(const KernelCtx &c, const DeviceNetlist &d, const void *ysave, const void *g, const void *x,
                           void *pos, void *xtrial, const DevScalars *S, cudaStream_t st);
    static void stage_begin(const DeviceNetlist &d, const void *pos, void *x, int step_cap, DevScalars *S,
                            int *progress, cudaStream_t st);
    static void wrap_up(const KernelCtx &c, const DeviceNetlist &d, void *pos, const void *x, cudaStream_t st);
    // the kernels that a loop with this wirelength form launches
    static std::vector<const void *> kernels(bool exact_exp, bool lse);
};
extern template struct Loop<float>;
extern template struct Loop<double>;

}  // namespace ep
