// The balls' scale of csrc/walk.cuh (one sample's and a pair's) beside sqrtf and the division, at the
// floats first, first + stride, ... (`count` of them, by their bits) of the square.
#include "walk.cuh"

namespace {

__device__ float by_norm(float square, float radius) {
  const float norm = sqrtf(square);
  return norm > radius ? radius / norm : 1.0f;
}

// `any`: of the unrolled solve, else of a solve, whose radii are usual.
__global__ void check(float radius, bool any, unsigned first, unsigned stride, unsigned count, unsigned long long* wrong) {
  const urb::Ball ball = any ? urb::Ball::any(radius) : urb::Ball(radius);
  unsigned long long mine = 0;
  for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    const float x = __uint_as_float(first + k * stride);
    // The other half: the square's neighbour, one within the ball, one far beyond it.
    const float others[3] = {__uint_as_float(first + k * stride + 1), 0.0f, 1e30f};
    const float y = others[k % 3];
    const urb::Pair got = urb::ball2(urb::pair(x, y), ball);
    const unsigned gx = __float_as_uint(urb::first(got)), gy = __float_as_uint(urb::second(got));
    mine += gx != __float_as_uint(by_norm(x, radius)) || gy != __float_as_uint(by_norm(y, radius)) ||
            __float_as_uint(urb::ball(x, ball)) != __float_as_uint(by_norm(x, radius));
  }
  if (mine != 0) atomicAdd(wrong, mine);
}

}  // namespace

// The number of them at which a scale differs, or -1 where the device failed.
extern "C" long long ball_check(float radius, int any, unsigned first, unsigned stride, unsigned count) {
  unsigned long long* wrong = nullptr;
  unsigned long long host = 0;
  if (cudaMalloc(&wrong, sizeof(host)) != cudaSuccess) return -1;
  bool good = cudaMemset(wrong, 0, sizeof(host)) == cudaSuccess;
  if (good) check<<<592, 256>>>(radius, any != 0, first, stride, count, wrong);
  good = good && cudaMemcpy(&host, wrong, sizeof(host), cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(wrong);
  return good ? static_cast<long long>(host) : -1;
}
