// The tile passes of the cubic spline in mixed precision.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_cubic_mixed(int hs, int blocks) { return pass_form<float, SIMP_SKF_CUBIC>(hs, blocks); }

}  // namespace pass
}  // namespace simp
