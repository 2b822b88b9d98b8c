// Test entry point of the refined reciprocals.
#include "common.cuh"
#include "reciprocals.cuh"

namespace bem {
namespace {

__global__ void reciprocals_kernel(int kind, int64_t n, const double* __restrict__ in, double* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (kind == 0) {
    out[i] = rsqrt_pos(in[i]);
    return;
  }
  const double2 a = make_double2(in[2 * i], in[2 * i + 1]);
  double2 r;
  if (kind == 1) {
    bool in_range;
    r = cinv_fast(a, in_range);
    if (!in_range) r = cinv(a);
  } else {
    const float2 f = gj_reciprocal((float)a.x, (float)a.y);
    r = make_double2(f.x, f.y);
  }
  out[2 * i] = r.x;
  out[2 * i + 1] = r.y;
}

}  // namespace
}  // namespace bem

extern "C" int bem_reciprocals(int kind, int64_t n, const double* in_dev, double* out_dev, void* stream) {
  using namespace bem;
  if (kind < 0 || kind > 2 || n <= 0 || !in_dev || !out_dev)
    return set_error(BEM_ERR_INVALID_ARGUMENT, "bem_reciprocals: bad arguments");
  reciprocals_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(kind, n, in_dev, out_dev);
  count_launches(1);
  BEM_CUDA_CHECK(cudaGetLastError());
  return BEM_OK;
}
