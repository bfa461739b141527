// fft_f64.cu -- the fast-transform Poisson solve in FP64.
#include "fft_kernels.cuh"

namespace ep {
template struct FftPasses<double>;
}
