// wf_brick.cu -- FP32-storage instantiations of the one-shot brick step
// (wf_brick_impl.cuh) and the dispatch of every storage type.
#include "wf_brick_impl.cuh"

namespace wf {

void brick_boxes(int prec, unsigned e_box[4], unsigned h_box[4]) {
  const unsigned pad = prec == kPrecF32 ? 4u : 8u;  // 16 bytes of x
  e_box[0] = kBrickX + 2 * pad; e_box[1] = kBrickY + 2; e_box[2] = kBrickZ + 2; e_box[3] = 3;
  h_box[0] = kBrickX + pad; h_box[1] = kBrickY + 1; h_box[2] = kBrickZ + 1; h_box[3] = 3;
}

cudaError_t brick_prepare(int prec, bool fma) {
  if (prec != kPrecF32) return fma ? cudaErrorInvalidValue : brick16_prepare(prec);
  return fma ? brick_prepare_t<true, float>() : brick_prepare_t<false, float>();
}

cudaError_t launch_brick(const BrickMaps &m, const BrickArgs &a, bool fma, cudaStream_t s) {
  if (a.g.prec != kPrecF32) return fma ? cudaErrorInvalidValue : brick16_launch(m, a, s);
  return fma ? brick_launch_t<true, float>(m, a, s) : brick_launch_t<false, float>(m, a, s);
}

cudaError_t brick_batch_prepare() {
  cudaError_t e = cudaFuncSetAttribute(k_brick_batch<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       BrickL<float>::BYTES);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_brick_batch<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              BrickL<float>::BYTES);
}

cudaError_t launch_brick_batch(const BrickScene *scenes, const int4 *items, int n_items, int parity,
                               bool xs, cudaStream_t s) {
  if (n_items <= 0) return cudaSuccess;
  if (xs)
    k_brick_batch<true><<<n_items, kBrickThreads, BrickL<float>::BYTES, s>>>(scenes, items, parity);
  else
    k_brick_batch<false><<<n_items, kBrickThreads, BrickL<float>::BYTES, s>>>(scenes, items, parity);
  return cudaGetLastError();
}

}  // namespace wf
