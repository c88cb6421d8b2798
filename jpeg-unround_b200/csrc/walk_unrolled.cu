// The unrolled solve's iteration as a walk (walk.cuh), of every picture of the problem at once: the
// dual step D_k and the primal step P_{k+1} in one pass, where they were a tile kernel and a block
// kernel (84 bytes a pixel and its intervals' 12 moved; now 72 and 12). The proximal maps' warps
// take each coefficient's interval and centre from the problem's arrays, a block row ahead, and
// t = tau m and r = 1 / (1 + t) from tables that the CTA makes for its picture. A step whose branches --
// clip, balls -- the adjoint takes again must not differ, so each value is made by the operations of the
// two kernels: outputs and checkpoints were equal to theirs bit for bit, from one block to 5 pictures of
// 40 x 1000, when it took their place (unrolled.cu's primal_kernel still makes P_1). The tests hold it to
// the FP64 reference.
//
// 16 pictures of 512 x 512, an iteration: 85 us (28 + 52 and the gap) -> 73 us.
#include "walk.cuh"

namespace urb {

namespace {

using Unrolled = Walk<true, 1, false, 1, 1, 0, true>;

// t and r of a picture's frequencies, plain and of flat blocks, at prox_slot(k).
struct ClipTable {
  float2 plain[64];
  float2 flat[64];
};

// A block row's constants at a lane (row m of its block), read ahead of their use.
struct ClipAhead {
  float4 lower[2], upper[2], centre[2];
  float middle;
  std::uint8_t flat;
};

__device__ __forceinline__ ClipAhead clip_ahead(const UnrolledWalk& P, int image, int j, int i, int lane) {
  const int across = P.step.dual.g.columns / 8, down = P.step.dual.g.rows / 8;
  const int jc = min(j, P.step.dual.g.columns - 1);
  const std::size_t block = (static_cast<std::size_t>(image) * down + i / 8) * across + jc / 8;
  const std::size_t at = block * 64 + (lane & 7) * 8;
  ClipAhead a;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    a.lower[h] = __ldg(reinterpret_cast<const float4*>(P.lower + at) + h);
    a.upper[h] = __ldg(reinterpret_cast<const float4*>(P.upper + at) + h);
    a.centre[h] = __ldg(reinterpret_cast<const float4*>(P.centre + at) + h);
  }
  a.middle = __ldg(P.middle + block);
  a.flat = __ldg(P.flat + block);
  return a;
}

// x~ of a block row at the lane's column, v down the column from the tile (prox_rows of walk.cuh
// with the unrolled solve's clip: zeta = clip((e + t c) r, a, b)).
template <int WIDTH>
__device__ __forceinline__ void clip_rows(float* tile, const ClipAhead& a, const ClipTable& table, float* next,
                                          int pitch, int lane, bool column_in) {
  const int m = lane & 7;
  float* const t = tile + lane / 8 * 8;
  auto entry = [&](int k, int n) -> float& { return t[k * WIDTH + (n ^ k)]; };
  float v[8], col[8], row[8], zeta[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = tile[r * WIDTH + lane] - a.middle;
  forward8(v, col);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) entry(k, m) = col[k];
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 8; ++u) row[u] = entry(m, u);
  forward8(row, zeta);
  const float2* factors = (a.flat != 0 ? table.flat : table.plain) + m * 8;
  auto of = [](const float4(&f)[2], int u) -> float {
    const float4 q = f[u >> 2];
    return (u & 3) == 0 ? q.x : (u & 3) == 1 ? q.y : (u & 3) == 2 ? q.z : q.w;
  };
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const float2 f = factors[u ^ m];  // t, r
    const float z = __fmul_rn(fmaf(f.x, of(a.centre, u), zeta[u]), f.y);
    zeta[u] = fminf(fmaxf(z, of(a.lower, u)), of(a.upper, u));
  }
  inverse8(zeta, row);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) entry(m, k) = row[k];
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) col[k] = entry(k, m);
  inverse8(col, v);
  if (column_in) {
#pragma unroll
    for (int r = 0; r < 8; ++r) next[static_cast<std::size_t>(r) * pitch] = v[r] + a.middle;
  }
}

__global__ void __launch_bounds__(walk_threads<1>(), 3)
    walk_unrolled_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ UnrolledWalk P) {
  using W = Unrolled::W;
  extern __shared__ __align__(128) float shared[];
  __shared__ __align__(8) WalkBarriers bars;
  __shared__ ClipTable table;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, image = blockIdx.z;
  const float tau = __ldg(P.tau + image);
  for (int n = tid; n < 128; n += walk_threads<1>()) {
    const int k = n & 63;
    const float t = __fmul_rn(tau, __ldg((n < 64 ? P.weight : P.flat_weight) + image * 64 + k));
    (n < 64 ? table.plain : table.flat)[prox_slot(k)] = make_float2(t, 1.0f / __fadd_rn(1.0f, t));
  }
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) barrier_init(&bars.full[s], 1);
    for (int s = 0; s < 2; ++s) {
      barrier_init(&bars.drained[s], kDual + 1);
      barrier_init(&bars.go[s], 3);
      barrier_init(&bars.luma[s], kDual);
      barrier_init(&bars.chroma[s], kDual);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const Geometry& g = P.step.dual.g;
  const int i0 = blockIdx.y * P.step.strip_rows, x0 = static_cast<int>(blockIdx.x) * W::WIDTH;
  const Unrolled walk{P.step,
                      shared,
                      x0,
                      i0,
                      min(i0 + P.step.strip_rows, g.rows),
                      image,
                      tau,
                      __ldg(P.sigma + image),
                      __ldg(P.alpha1 + image),
                      __ldg(P.alpha0 + image)};
  float* const next = P.step.next + (static_cast<std::size_t>(image) * g.rows + i0) * g.pitch + x0;
  bool good = true;
  int issued = 0;
  if (warp < kDual) {
    good = walk.dual_warp(bars, &failed, warp, lane);
  } else if (warp == kDual) {
    good = walk.copy_warp(&map, bars, &failed, lane, issued);
  } else {
    const int column = 32 * (warp - kDual - 1) + lane;
    auto let_go = [&](int band) {
      if (lane == 0) barrier_arrive(&bars.go[band & 1]);
    };
    let_go(0);
    ClipAhead ahead = clip_ahead(P, image, x0 + column, i0, lane);
    for (int i = i0, b = 0; i < walk.i1 && good; i += 8, ++b) {
      const ClipAhead now = ahead;
      if (i + 8 < walk.i1) ahead = clip_ahead(P, image, x0 + column, i + 8, lane);
      good = __all_sync(kAll, wait_unless(&bars.luma[b & 1], (b >> 1) & 1, &failed));
      if (!good) break;
      let_go(b + 1);
      clip_rows<W::WIDTH>(shared + W::LUMA + (b & 1) * kChunk * W::WIDTH + column - lane, now, table,
                          next + static_cast<std::size_t>(i - i0) * g.pitch + column, g.pitch, lane,
                          x0 + column < g.columns);
      __syncwarp();
    }
  }
  if (!good) {
    *static_cast<volatile int*>(&failed) = 1;
    // The strip's first x~ says so, and the next walk's x there, and every later x: the clip takes its
    // interval's end for a NaN, but the relaxation keeps it. unrolled.cu looks for it at a pass's end
    // (failed_kernel). An error word, told here, costs registers that the walk has not: 6.97 -> 7.16 ms of
    // 16 x 512 x 512, 100 iterations.
    if (lane == 0) *next = __int_as_float(0x7fc00000);
    for (int n = max(issued - kSlots, 0); n < issued; ++n) barrier_wait(&bars.full[n % kSlots], (n / kSlots) & 1);
  }
}

}  // namespace

cudaError_t launch_walk_unrolled(const CUtensorMap& map, const UnrolledWalk& p, cudaStream_t stream) {
  using W = Unrolled::W;
  constexpr std::size_t bytes = W::FLOATS * sizeof(float);
  static std::atomic<int> resident[64] = {};
  int device = 0;
  cudaGetDevice(&device);
  int ctas = resident[device & 63].load();
  if (ctas == 0) {
    cudaError_t e = cudaFuncSetAttribute(walk_unrolled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes));
    int per_sm = 0, sms = 0;
    if (e == cudaSuccess) {
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk_unrolled_kernel, walk_threads<1>(), bytes);
    }
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    ctas = std::max(1, per_sm * sms);
    resident[device & 63].store(ctas);
  }
  UnrolledWalk q = p;
  // As one picture of all the pictures' strips side by side.
  const Geometry& g = p.step.dual.g;
  Geometry all = g;
  const int strips = (g.columns + W::WIDTH - 1) / W::WIDTH;
  all.columns = strips * W::WIDTH * p.images;
  q.step.strip_rows = walk_rows(all, ctas, W::WIDTH, 8);
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(strips, (g.rows + q.step.strip_rows - 1) / q.step.strip_rows, p.images);
  config.blockDim = dim3(walk_threads<1>());
  config.dynamicSmemBytes = bytes;
  config.stream = stream;
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &early;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, walk_unrolled_kernel, map, q);
}

}  // namespace urb
