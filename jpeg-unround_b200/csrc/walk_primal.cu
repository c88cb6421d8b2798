// The walk (walk.cuh) of iterations whose primal step is kept for a record: zeta, v, G's terms.
#include "walk.cuh"

namespace urb {

cudaError_t launch_walk_primal(const CUtensorMap& map, const IterationParams& p, bool tgv, bool coupled, int cell_rows,
                               int cell_columns, cudaStream_t stream, int* partials) {
  return launch_keep<1>(map, p, tgv, coupled, cell_rows, cell_columns, stream, partials);
}

}  // namespace urb
