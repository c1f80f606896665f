// mdg_nonbonded_block.cu -- instantiations of the pair kernel's block form
// (several warps per work item; see mdg_nonbonded_kernel.cuh).
#include "mdg_nonbonded_kernel.cuh"

namespace mdg {

cudaError_t launch_nb_block(mdg_system *s, const NbArgs &a, int warps, bool want_lj, bool sw,
                            int energy, int dump) {
    const size_t smem = 2 * sizeof(float) * kPkChunk * nb_block_chunks(warps);
    const dim3 grid(a.n_items), block(32 * warps);
    auto go = [&](auto kernel) {
        kernel<<<grid, block, smem, s->stream>>>(a);
        return cudaGetLastError();
    };
    if (dump) return go(k_nonbonded_block<MDG_COUL_EWALD, true, false, false, true>);
    if (!want_lj)
        return energy ? go(k_nonbonded_block<MDG_COUL_EWALD, false, false, true, false>)
                      : go(k_nonbonded_block<MDG_COUL_EWALD, false, false, false, false>);
    if (sw)
        return energy ? go(k_nonbonded_block<MDG_COUL_EWALD, true, true, true, false>)
                      : go(k_nonbonded_block<MDG_COUL_EWALD, true, true, false, false>);
    return energy ? go(k_nonbonded_block<MDG_COUL_EWALD, true, false, true, false>)
                  : go(k_nonbonded_block<MDG_COUL_EWALD, true, false, false, false>);
}

}  // namespace mdg
