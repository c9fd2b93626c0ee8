// Q1 hexahedra with every element in FP64, one thread per element (pxg_q1f64.h): the
// loads the fixed-point kernel (pxg_q1fx.cu) does not provide.
#include "pxg_q1f64.h"

namespace pxg
{
// NT threads per block, at least MINB blocks per SM (the register budget per thread:
// 128 x 1 -> 254 registers, 8 warps per SM; 64 x 6 -> 170 registers, 12 warps per SM)
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) kAssembleQ1F64(AsmArgs const __grid_constant__ a)
{
  int64_t const i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i0 >= a.nelem)
    return;
  elementF64(a, elemOf(a, i0));
}

void launchAssembleQ1F64(AsmArgs const & a, cudaStream_t s, int threads)
{
  if (a.nelem <= 0)
    return;
  // constant and sin sin sin loads, or none: the fixed-point kernel, 2.6 x faster at
  // 128^3; other analytic functions and projections evaluate doubles per point
  if (!a.rkind || (a.rkind == 1 && (a.fn == PXG_FN_CONST || a.fn == PXG_FN_SIN3)))
    launchAssembleQ1Fx(a, s, threads);
  else if (threads == 64)
    launchElemKernel(kAssembleQ1F64<64, 6>, (unsigned)((a.nelem + 63) / 64), 64, 0, s, a);
  else
    launchElemKernel(kAssembleQ1F64<128, 1>, (unsigned)((a.nelem + 127) / 128), 128, 0, s, a);
}

} // namespace pxg
