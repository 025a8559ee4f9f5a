// nz_ufg.cu -- per-step records of bond percolation, one run per thread block.
#include "nz_group_rows.cuh"

namespace nz {

cudaError_t launch_uf_groups(const UfParams &p, bool given, bool span, cudaStream_t s) {
    if (p.n_runs <= 0) return cudaSuccess;
    return p.g.kind == NZ_GRAPH_TORUS2D ? group::launch_groups<true, false>(p, given, span, s)
                                        : group::launch_groups<false, false>(p, given, span, s);
}

}  // namespace nz
