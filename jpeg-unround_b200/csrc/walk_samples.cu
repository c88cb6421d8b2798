// The iteration of pictures of rounded samples as a walk (walk.cuh): the dual step D_n and the primal
// step P_{n+1} in one pass, where they are the dual sweep and samples.cu's primal kernel (TGV: 72
// bytes and a 2-byte level a sample, against 68 and 18). In place of the block rows' proximal map a
// warp takes each sample of its column of a chunk to its interval: the levels looked up a chunk
// ahead, their intervals while the dual step makes the chunk's v. The canvas is the picture itself,
// of any rows and columns. The values are bit for bit those of the two launches.
//
// What bounds it: the dual step's warps, as the other walks. An iteration, in two launches and now:
// TGV of three channels 128x128 20.6 -> 4.5 us, 512x512 22.7 -> 12.1, 901x1203 63.0 -> 48.8,
// 1600x1600 126 -> 103; of one channel 512x512 18.5 -> 8.0, 1600x1600 47.2 -> 37.5; TV of three
// channels 512x512 16.5 -> 7.8, 901x1203 29.9 -> 24.4; of one channel 512x512 14.4 -> 4.1.
#include "walk.cuh"

namespace urb {

namespace {

struct SamplesWalk {
  IterationParams step;
  SamplesStep samples;
};

template <bool TGV, int C, bool COUPLED>
__global__ void __launch_bounds__(walk_threads<C>(), walk_ctas<TGV, C>())
    walk_samples_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ SamplesWalk P) {
  using W = WalkLayout<TGV, C, 1>;
  extern __shared__ __align__(128) float shared[];
  __shared__ __align__(8) WalkBarriers bars;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) barrier_init(&bars.full[s], 1);
    for (int s = 0; s < 2; ++s) {
      barrier_init(&bars.drained[s], kDual + 1);
      barrier_init(&bars.go[s], 1 + (C == 1 ? 2 : C));
      barrier_init(&bars.luma[s], kDual);
      barrier_init(&bars.chroma[s], kDual);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const Geometry& g = P.step.dual.g;
  const int i0 = blockIdx.y * P.step.strip_rows, x0 = static_cast<int>(blockIdx.x) * W::WIDTH;
  // Whole chunks: what lies past the last row is not written.
  const int i1 = min(i0 + P.step.strip_rows, (g.rows + kChunk - 1) / kChunk * kChunk);
  const Walk<TGV, C, COUPLED, 1, 1, 0, false, true> walk{P.step, shared, x0, i0, i1};
  bool good = true;
  int issued = 0;
  if (warp < kDual) {
    good = walk.dual_warp(bars, &failed, warp, lane);
  } else if (warp == kDual) {
    good = walk.copy_warp(&map, bars, &failed, lane, issued);
  } else {
    const int z = warp - kDual - 1, c = C == 1 ? 0 : z, column = (C == 1 ? 32 * z : 0) + lane, j = x0 + column;
    std::uint64_t* const full = c == 0 ? bars.luma : bars.chroma;
    const float* const tile = shared + (c == 0 ? W::LUMA : W::CHROMA + (c - 1) * kChunk * W::WIDTH) + column;
    const int stride = (c == 0 ? 1 : C - 1) * kChunk * W::WIDTH;
    const std::size_t plane = c * g.plane + min(j, g.columns - 1);
    auto let_go = [&](int band) {
      if (lane == 0) barrier_arrive(&bars.go[band & 1]);
    };
    auto look_up = [&](unsigned(&level)[kChunk], int i) {
#pragma unroll
      for (int r = 0; r < kChunk; ++r) {
        level[r] = __ldg(P.samples.levels + plane + static_cast<std::size_t>(min(i + r, g.rows - 1)) * g.pitch);
      }
    };
    let_go(0);
    unsigned ahead[kChunk];
    look_up(ahead, i0);
    for (int i = i0, b = 0; i < i1; i += kChunk, ++b) {
      float4 ends[kChunk];
#pragma unroll
      for (int r = 0; r < kChunk; ++r) ends[r] = __ldg(reinterpret_cast<const float4*>(P.samples.ends) + ahead[r]);
      if (i + kChunk < i1) look_up(ahead, i + kChunk);
      good = __all_sync(kAll, wait_unless(&full[b & 1], (b >> 1) & 1, &failed));
      if (!good) break;
      let_go(b + 1);
      float* const next = P.step.next + plane + static_cast<std::size_t>(i) * g.pitch;
#pragma unroll
      for (int r = 0; r < kChunk; ++r) {
        const float v = tile[(b & 1) * stride + r * W::WIDTH];
        const float x = __fmul_rn(fmaf(P.samples.t, ends[r].z, v), P.samples.r);
        if (j < g.columns && i + r < g.rows) {
          next[static_cast<std::size_t>(r) * g.pitch] = fminf(fmaxf(x, ends[r].x), ends[r].y);
        }
      }
      __syncwarp();
    }
  }
  if (!good) {
    *static_cast<volatile int*>(&failed) = 1;
    if (lane == 0 && P.step.dual.error != nullptr) atomicExch(P.step.dual.error, 1);
    for (int n = max(issued - kSlots, 0); n < issued; ++n) barrier_wait(&bars.full[n % kSlots], (n / kSlots) & 1);
  }
}

template <bool TGV, int C, bool COUPLED>
cudaError_t launch_samples(const CUtensorMap& map, SamplesWalk& p, cudaStream_t stream) {
  using W = WalkLayout<TGV, C, 1>;
  static std::atomic<int> resident[64] = {};
  return launch_strips(walk_samples_kernel<TGV, C, COUPLED>, walk_threads<C>(), W::FLOATS * sizeof(float), W::WIDTH,
                       kChunk, map, p, p.step, resident, stream);
}

}  // namespace

cudaError_t launch_walk_samples(const CUtensorMap& map, const DualParams& dual, const SamplesStep& samples, bool tgv,
                                bool coupled, cudaStream_t stream) {
  SamplesWalk p;
  p.step.dual = dual;
  p.step.next = samples.next;
  p.samples = samples;
  if (dual.g.channels == 1) {
    return tgv ? launch_samples<true, 1, false>(map, p, stream) : launch_samples<false, 1, false>(map, p, stream);
  }
  if (dual.g.channels != 3) return cudaErrorInvalidValue;
  if (tgv) return coupled ? launch_samples<true, 3, true>(map, p, stream) : launch_samples<true, 3, false>(map, p, stream);
  return coupled ? launch_samples<false, 3, true>(map, p, stream) : launch_samples<false, 3, false>(map, p, stream);
}

}  // namespace urb
