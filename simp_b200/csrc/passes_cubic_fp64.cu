// The tile passes of the cubic spline in FP64.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_cubic_fp64(int hs, int blocks) { return pass_form<double, SIMP_SKF_CUBIC>(hs, blocks); }

}  // namespace pass
}  // namespace simp
