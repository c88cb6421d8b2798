// The walk (walk.cuh) of iterations that keep nothing; walk_duals.cu and walk_primal.cu have those
// that keep a record's values (files of their own, compiled beside one another).
#include "walk.cuh"

namespace urb {

bool make_walk_map(CUtensorMap& map, const float* planes, const Geometry& g, int count) {
  return make_box_map(map, planes, g, count, g.plane, 2, sweep_width(g.channels) + 2 * kHalo);
}

int walk_partials(const Geometry& g) {
  return 2 * ((g.columns + 63) / 64) * ((g.rows + kChunk - 1) / kChunk);
}

cudaError_t launch_walk(const CUtensorMap& map, const IterationParams& p, bool tgv, bool coupled, int cell_rows,
                        int cell_columns, WalkKeep keep, cudaStream_t stream, int* partials) {
  switch (keep) {
    case WalkKeep::primal: return launch_walk_primal(map, p, tgv, coupled, cell_rows, cell_columns, stream, partials);
    case WalkKeep::duals: return launch_walk_duals(map, p, tgv, coupled, cell_rows, cell_columns, stream);
    default: return launch_keep<0>(map, p, tgv, coupled, cell_rows, cell_columns, stream, nullptr);
  }
}

}  // namespace urb
