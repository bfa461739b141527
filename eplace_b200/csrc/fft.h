// fft.h -- the plan of the fast-transform Poisson solve and its passes
// (fft_kernels.cuh) in one working precision, each instantiated in a file of its
// own (fft_f32.cu, fft_f64.cu; loop.h has the reason).
#pragma once
#include <string>
#include <vector>

#include "engine.h"

namespace ep {

constexpr int kMinLog = 3, kMaxLog = 11;  // log2 of the bins on an axis

struct FftPlan {
    int lognx = 0, logny = 0;
    int fp64 = 0;
    // twiddles, stage-major: stage s (half-size h = 2^s) holds e^{-i pi j / h},
    // j < h, at [h - 1 + j]; n - 1 entries per axis (vec2<R>)
    void *twx = nullptr, *twy = nullptr;
    // (cos, sin)(pi k / 2n), k <= n/2 (vec2<R>)
    void *qx = nullptr, *qy = nullptr;
    void *wx = nullptr, *wy = nullptr;  // frequency weights (R)
    double kscale = 0.0;                // 4 / (nx ny)
    void *T = nullptr;                  // [nx][ny] after the first pass (R)
    void *X = nullptr;                  // X1, X2: [2][nx][ny] (R)
    size_t smem_rows_fwd = 0, smem_cols = 0, smem_rows_inv = 0;
    int pairs_fwd = 1, rows_inv = 1, cols = 2;
};

template <typename R>
struct FftPasses {
    // the tables, the intermediates and the kernels' attributes; an ep_status
    static int init(FftPlan *f, int nx, int ny, const std::vector<double> &wx, const std::vector<double> &wy,
                    std::string &err);
    static void run(const FftPlan *f, int nx, int ny, const R *rho, vec2<R> *field, R *phi, const DevScalars *S,
                    cudaStream_t st);
};
extern template struct FftPasses<float>;
extern template struct FftPasses<double>;

}  // namespace ep
