// mdg_nonbonded_batch.cu -- the whole-warp pair kernel for batches of systems:
// its candidate search calls the sweep code from one place (see
// scan_candidates_one in mdg_nonbonded_kernel.cuh).
#include "mdg_nonbonded_kernel.cuh"

namespace mdg {

cudaError_t launch_nb_batch(mdg_system *s, const NbArgs &a, int coul_tile, bool want_lj, bool sw,
                            int energy, int dump) {
    return dispatch_shape<false, true>(s, a, coul_tile, want_lj, sw, energy, dump);
}

}  // namespace mdg
