// nz_lattice.cu -- site percolation on the grid, the chain and the torus, one
// run per thread block.
//
// An extension that the reference lists as to-do (percolate/__init__.py:68-78;
// percolate/percolate.py:210-211 rejects every model but 'bond'), writing the
// same per-step records, so the fused microcanonical reductions, the canonical
// convolution and every other consumer of records apply unchanged.
//
// Site percolation (Newman & Ziff, Phys. Rev. Lett. 85, 4104 (2000); Phys.
// Rev. E 64, 016706 (2001), Sec. II): step n occupies the n-th site of a
// permutation of the N sites -- a new cluster of one site -- and joins it to
// each occupied neighbour.  The statistics count occupied sites only (T_k over
// occupied clusters, so m1 = n - max; m0 = clusters - 1, or 0 while no site is
// occupied).  A caller-supplied index out of range or repeated occupies nothing.
#include "nz_group_rows.cuh"

namespace nz {

cudaError_t launch_site_groups(const UfParams &p, bool given, bool span, cudaStream_t s) {
    if (p.n_runs <= 0) return cudaSuccess;
    return p.g.kind == NZ_GRAPH_TORUS2D ? group::launch_groups<true, true>(p, given, span, s)
                                        : group::launch_groups<false, true>(p, given, span, s);
}

}  // namespace nz
