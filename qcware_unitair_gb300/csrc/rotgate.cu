// Rotation gates exp(-i a P) for a batch of angles, and the angles'
// gradient.  unitair stacks them from elementwise torch operations
// (src/unitair/gates/gates.py:6-91): about ten launches forward and twice as
// many backward for a few kilobytes.  Here each direction is one launch,
// bound by it.
#include "common.cuh"

namespace gbsv {

constexpr int RG_THREADS = 128;

template <typename R> struct RgMath;
template <> struct RgMath<float> {
  __device__ static float cos(float a) { return cosf(a); }
  __device__ static float sin(float a) { return sinf(a); }
};
template <> struct RgMath<double> {
  __device__ static double cos(double a) { return ::cos(a); }
  __device__ static double sin(double a) { return ::sin(a); }
};

// axis 0: [[c, -i s], [-i s, c]]; 1: [[c, -s], [s, c]]; 2: diag(c - i s,
// c + i s)
template <typename R>
__global__ void __launch_bounds__(RG_THREADS)
    rotation_gates_kernel(const R* angles, int64_t stride, int64_t count,
                          int axis, Cx<R>* out) {
  const int64_t i = (int64_t)blockIdx.x * RG_THREADS + threadIdx.x;
  if (i >= count) return;
  const R a = angles[i * stride];
  const R c = RgMath<R>::cos(a), s = RgMath<R>::sin(a);
  Cx<R> m[4];
  m[0].x = m[3].x = c;
  m[0].y = m[3].y = 0;
  m[1].x = m[1].y = m[2].x = m[2].y = 0;
  if (axis == 0) {
    m[1].y = m[2].y = -s;
  } else if (axis == 1) {
    m[1].x = -s;
    m[2].x = s;
  } else {
    m[0].y = -s;
    m[3].y = s;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) out[4 * i + j] = m[j];
}

// dL/da = Re sum_jk grad[j, k] conj(dm[j, k] / da)
template <typename R>
__global__ void __launch_bounds__(RG_THREADS)
    rotation_gates_grad_kernel(const R* angles, int64_t stride, int64_t count,
                               int axis, const Cx<R>* grad, R* out) {
  const int64_t i = (int64_t)blockIdx.x * RG_THREADS + threadIdx.x;
  if (i >= count) return;
  const R a = angles[i * stride];
  const R c = RgMath<R>::cos(a), s = RgMath<R>::sin(a);
  const Cx<R>* g = grad + 4 * i;
  const R diag = g[0].x + g[3].x;
  R off;
  if (axis == 0) off = -(g[1].y + g[2].y);
  else if (axis == 1) off = g[2].x - g[1].x;
  else off = g[3].y - g[0].y;
  out[i] = c * off - s * diag;
}

}  // namespace gbsv

using namespace gbsv;

static int rg_check(const void* angles, int dtype, int64_t stride,
                    int64_t count, int axis, const void* a, const void* b) {
  if (dtype != GBSV_C64 && dtype != GBSV_C128)
    return set_error(GBSV_ERR_INVALID_ARG, "gates must be complex");
  if (axis < 0 || axis > 2 || stride < 0 || count < 0 ||
      count > (int64_t)0x7fffffff * RG_THREADS)
    return set_error(GBSV_ERR_INVALID_ARG, "bad axis %d, stride or count",
                     axis);
  if (count > 0 && (!angles || !a || !b))
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  return GBSV_OK;
}

extern "C" int gbsv_rotation_gates(const void* angles, int dtype,
                                   int64_t stride, int64_t count, int axis,
                                   void* out, void* stream) {
  int rc = rg_check(angles, dtype, stride, count, axis, out, out);
  if (rc || count == 0) return rc;
  const unsigned grid = (unsigned)((count + RG_THREADS - 1) / RG_THREADS);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == GBSV_C64)
    rotation_gates_kernel<float><<<grid, RG_THREADS, 0, st>>>(
        static_cast<const float*>(angles), stride, count, axis,
        static_cast<float2*>(out));
  else
    rotation_gates_kernel<double><<<grid, RG_THREADS, 0, st>>>(
        static_cast<const double*>(angles), stride, count, axis,
        static_cast<double2*>(out));
  return after_launch("rotation_gates_kernel");
}

extern "C" int gbsv_rotation_gates_grad(const void* angles, int dtype,
                                        int64_t stride, int64_t count,
                                        int axis, const void* grad,
                                        void* grad_angles, void* stream) {
  int rc = rg_check(angles, dtype, stride, count, axis, grad, grad_angles);
  if (rc || count == 0) return rc;
  const unsigned grid = (unsigned)((count + RG_THREADS - 1) / RG_THREADS);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == GBSV_C64)
    rotation_gates_grad_kernel<float><<<grid, RG_THREADS, 0, st>>>(
        static_cast<const float*>(angles), stride, count, axis,
        static_cast<const float2*>(grad), static_cast<float*>(grad_angles));
  else
    rotation_gates_grad_kernel<double><<<grid, RG_THREADS, 0, st>>>(
        static_cast<const double*>(angles), stride, count, axis,
        static_cast<const double2*>(grad),
        static_cast<double*>(grad_angles));
  return after_launch("rotation_gates_grad_kernel");
}
