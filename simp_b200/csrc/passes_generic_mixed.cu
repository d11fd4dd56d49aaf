// The tile passes of the kernel functions that are chosen at run time in mixed precision.
#include "pass_kernels.cuh"

namespace simp {
namespace pass {

PassForm passes_generic_mixed(int hs, int blocks) { return pass_form<float, 0>(hs, blocks); }

}  // namespace pass
}  // namespace simp
