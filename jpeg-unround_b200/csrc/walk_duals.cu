// The walk (walk.cuh) of iterations whose dual step is kept for a record: the tilde duals.
#include "walk.cuh"

namespace urb {

cudaError_t launch_walk_duals(const CUtensorMap& map, const IterationParams& p, bool tgv, bool coupled, int cell_rows,
                              int cell_columns, cudaStream_t stream) {
  return launch_keep<2>(map, p, tgv, coupled, cell_rows, cell_columns, stream, nullptr);
}

}  // namespace urb
