// fft_f32.cu -- the fast-transform Poisson solve in FP32.
#include "fft_kernels.cuh"

namespace ep {
template struct FftPasses<float>;
}
