// wf_brick16.cu -- binary16 and bfloat16 instantiations of the one-shot brick
// step (wf_brick_impl.cuh); wf_brick.cu dispatches to them.
#include "wf_brick_impl.cuh"

namespace wf {

cudaError_t brick16_prepare(int prec) {
  return prec == kPrecF16 ? brick_prepare_t<false, __half>() : brick_prepare_t<false, __nv_bfloat16>();
}

cudaError_t brick16_launch(const BrickMaps &m, const BrickArgs &a, cudaStream_t s) {
  return a.g.prec == kPrecF16 ? brick_launch_t<false, __half>(m, a, s)
                              : brick_launch_t<false, __nv_bfloat16>(m, a, s);
}

}  // namespace wf
