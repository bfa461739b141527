// loop_f64.cu -- the loop's kernels in the plain FP64 form.
#include "loop_kernels.cuh"

namespace ep {
template struct Loop<double>;
}
