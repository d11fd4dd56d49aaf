// The tile passes of Wendland C6 in FP64.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_wendland_fp64(int hs, int blocks) { return pass_form<double, SIMP_SKF_WENDLAND_C6>(hs, blocks); }

}  // namespace pass
}  // namespace simp
