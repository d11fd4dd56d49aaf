// The tile passes of Wendland C6 in mixed precision.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_wendland_mixed(int hs, int blocks) { return pass_form<float, SIMP_SKF_WENDLAND_C6>(hs, blocks); }

}  // namespace pass
}  // namespace simp
