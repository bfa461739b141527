// loop_f32.cu -- the loop's kernels in FP32 positions, field and wirelength terms.
#include "loop_kernels.cuh"

namespace ep {
template struct Loop<float>;
}
