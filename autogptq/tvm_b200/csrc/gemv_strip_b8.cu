// The 8-bit instantiations of the decode GEMV (a translation unit of their own, to compile side by side).
#include "gemv_strip.cuh"

namespace b200gptq {
const void* gemv_strip_kernel_b8(int sub, int mode, int nt, int T, int warps, bool apart, bool split) {
    return strip_kernel_bits<8>(sub, mode, nt, T, warps, apart, split);
}
}  // namespace b200gptq
