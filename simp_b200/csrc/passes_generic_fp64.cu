// The tile passes of the kernel functions that are chosen at run time in FP64.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_generic_fp64(int hs, int blocks) { return pass_form<double, 0>(hs, blocks); }

}  // namespace pass
}  // namespace simp
