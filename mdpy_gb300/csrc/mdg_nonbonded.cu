// mdg_nonbonded.cu -- short-range nonbonded forces.
//
// Replaces, for the pair work:
//   CharmmNonbondedConstraint.cpu_kernel / cuda_kernel
//     (mdpy/constraint/charmm_nonbonded_constraint.py:64-181): LJ 12-6 with
//     Lorentz-Berthelot combination, 1-4 parameters for scaling_particles,
//     bonded_particles excluded, hard cutoff r <= rc;
//   ElectrostaticConstraint (mdpy/constraint/electrostatic_constraint.py:52-135):
//     bare Coulomb, all pairs, minimum image (kept as MDG_COUL_BARE for parity);
// and adds the Ewald real-space term k q_i q_j erfc(beta r)/r (MDG_COUL_EWALD),
// which mdpy v0.2.1 does not have, plus an optional CHARMM switch for LJ.
//
// Design (GB300): `split` (nb_default_parts) independent work items per 32-atom
// i-cluster I, a warp each (no block barrier: a warp that finishes early frees its
// slot); several warps each where items are few (the block form).
//   1. each warp walks its own interleaved batches of cluster bounding boxes
//      (a balanced half shell: the cluster pair {I, J} belongs to one of the
//      two by the parity of I + J) and takes every (J, periodic image) whose
//      box lies within rc of I's box -- __ballot_sync over 32 clusters at a
//      time, no candidate list and no block barrier;
//   2. for each candidate every lane tests one j atom against I's bounding
//      box, and the survivors are appended (warp ballot + popc, no atomics)
//      to a 64-entry per-warp ring buffer in shared memory, already shifted
//      to the right periodic image and with a 32-bit exclusion mask (which i
//      lanes must skip this j);
//   3. each full chunk of 32 j entries is swept against the warp's 32 i atoms
//      in 32 rotation steps: at step t lane l pairs its i atom with entry
//      (l+t) mod 32, keeps the i force in registers and passes the j force
//      accumulator to lane l-1 with one shuffle per component, so after the
//      sweep every lane owns one entry's complete j force.  No shared-memory
//      atomics, no per-pair reduction trees.
// Forces leave as int64 fixed point (scale 2^32) through 64-bit global
// atomics: the sum is independent of the order of arrival, so results are
// bit-reproducible run to run.  Pairs are never stored: the pair set is
// found afresh from the current coordinates on every evaluation, so no
// Verlet skin or rebuild criterion exists that could miss a pair.
#include <algorithm>

#include "mdg_nonbonded_kernel.cuh"

namespace mdg {

cudaError_t launch_nb_half(mdg_system *s, const NbArgs &a, int coul_tile, bool want_lj, bool sw,
                           int energy, int dump);  // mdg_nonbonded_half.cu
cudaError_t launch_nb_quarter(mdg_system *s, const NbArgs &a, int coul_tile, bool want_lj,
                              bool sw, int energy, int dump);  // mdg_nonbonded_quarter.cu

cudaError_t launch_nb_batch(mdg_system *s, const NbArgs &a, int coul_tile, bool want_lj, bool sw,
                            int energy, int dump);  // mdg_nonbonded_batch.cu
cudaError_t launch_nb_block(mdg_system *s, const NbArgs &a, int warps, bool want_lj, bool sw,
                            int energy, int dump);  // mdg_nonbonded_block.cu

namespace {

// Bare Coulomb over all pairs with the minimum image (parity path for
// ElectrostaticConstraint, electrostatic_constraint.py:52-79), forces on i
// only.  The force jumps where a separation passes half the box, so a
// trajectory of this mode hangs on the last bit: each i atom's sum is one FP32
// chain over the j atoms in cluster order, whatever the launch.  A block takes
// one i-cluster (a lane per i atom).  Eight warps work out four j atoms each of
// a j-cluster, (force / r, d) of their 32 pairs into shared memory, while a
// ninth adds the previous cluster's 32 pairs in order.  Bound by shared-memory
// and shuffle throughput (400 cycles a j-cluster) and one block barrier per
// j-cluster.  A thread per i atom that did it all kept 139 of 152 SMs idle on
// 2,700 atoms: 1053 -> 55 us (8,000 atoms: 3083 -> 223 us).  j atoms by uniform
// loads in place of the shuffles: 61 us.
constexpr int kBareProducers = 8;
constexpr int kBareThreads = 32 * (kBareProducers + 1);

// x rounded to the nearest integer (ties to even, as rintf) for |x| < 2^22;
// two adds instead of a conversion at a quarter of their rate.  Larger |x|
// only occurs for padding slots, which carry no charge.
__device__ __forceinline__ float rint_small(float x) {
    return __fsub_rn(__fadd_rn(x, 12582912.0f), 12582912.0f);
}

template <bool ENERGY>
__global__ void __launch_bounds__(kBareThreads) k_coulomb_bare(NbArgs a) {
    __shared__ float4 s_pair[2][kCluster][32];  // j atom, lane: force / r, d
    __shared__ float s_e[ENERGY ? 2 : 1][kCluster][32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x;
    const int ik = I * kCluster + lane;
    const float4 xi = a.xq[ik];
    // uncharged slots (padding has q = 0) contribute nothing
    if (!__any_sync(kFull, xi.w != 0.f)) return;  // the same in every warp
    const SysDev &sd = a.sys[a.cl_sys[I]];
    const float L[3] = {sd.L[0], sd.L[1], sd.L[2]};
    const float invL[3] = {sd.invL[0], sd.invL[1], sd.invL[2]};
    const int2 rI = a.prange[I];
    float fx = 0.f, fy = 0.f, fz = 0.f, e = 0.f;
    // each lane's atom of the j-clusters t .. t + 3, loaded three ahead: a tile
    // takes less time than a load from L2
    auto load = [&](int t) {
        return a.xq[(sd.cl_off + min(t, sd.cl_cap - 1)) * kCluster + lane];
    };
    float4 xl = load(0), x1 = load(1), x2 = load(2), x3 = xl;
    for (int t = 0; t <= sd.cl_cap; ++t) {
        if (w < kBareProducers && t < sd.cl_cap) {
            const int J = sd.cl_off + t, buf = t & 1;
            x3 = load(t + 3);
            // the i lanes that must skip this lane's j atom: itself, its 1-2 / 1-3 partners
            unsigned ml = J == I ? 1u << lane : 0u;
            if (rI.y >= J * kCluster && rI.x < (J + 1) * kCluster)
                for (int k = 0; k < a.pw; ++k) {
                    const int p = a.partners[(size_t)(J * kCluster + lane) * a.pw + k];
                    const int pi = p - I * kCluster;
                    if (p >= 0 && !(p & 0x40000000) && pi >= 0 && pi < kCluster) ml |= 1u << pi;
                }
#pragma unroll
            for (int u = 0; u < kCluster / kBareProducers; ++u) {
                const int j = w * (kCluster / kBareProducers) + u;
                const float4 xj = make_float4(__shfl_sync(kFull, xl.x, j), __shfl_sync(kFull, xl.y, j),
                                              __shfl_sync(kFull, xl.z, j), __shfl_sync(kFull, xl.w, j));
                const unsigned m = __shfl_sync(kFull, ml, j);
                float d[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float sc = d[k] * invL[k];
                    d[k] = (sc - rint_small(sc)) * L[k];
                }
                const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                const float rinv = rsqrtf(r2);
                const float qq = xi.w * xj.w;
                const float ev = qq * rinv;
                const float fr = ev * rinv * rinv;
                const bool skip = xj.w == 0.f || ((m >> lane) & 1u);
                s_pair[buf][j][lane] = skip ? make_float4(0.f, 0.f, 0.f, 0.f)
                                            : make_float4(fr, d[0], d[1], d[2]);
                if (ENERGY) s_e[buf][j][lane] = skip ? 0.f : ev;
            }
            xl = x1;
            x1 = x2;
            x2 = x3;
        } else if (w == kBareProducers && t > 0) {
            const int buf = (t - 1) & 1;
#pragma unroll 8
            for (int j = 0; j < kCluster; ++j) {
                const float4 v = s_pair[buf][j][lane];
                if (ENERGY) e += 0.5f * s_e[buf][j][lane];
                fx -= v.x * v.y;
                fy -= v.x * v.z;
                fz -= v.x * v.w;
            }
        }
        __syncthreads();
    }
    if (w != kBareProducers) return;
    if (xi.w != 0.f) {
        fix_red(&a.f[ik], to_fix(fx));
        fix_red(&a.f[a.n_pad + ik], to_fix(fy));
        fix_red(&a.f[2 * a.n_pad + ik], to_fix(fz));
    }
    if (ENERGY) {
        const double es = warp_sum_d(xi.w != 0.f ? (double)e : 0.0);
        if (lane == 0)
            fix_red((unsigned long long *)&a.energy[a.cl_sys[I] * kEnergySlots +
                                                    MDG_TERM_COUL_REAL],
                    to_fix_d(es));
    }
}

// ---- special pairs ---------------------------------------------------------
struct SpArgs {
    const double *__restrict__ x;
    const int *__restrict__ inv_perm;
    const float *__restrict__ charge;  // q * sqrt(k_e), atom order
    const float4 *__restrict__ lj;     // atom order
    const int2 *__restrict__ excl;
    const int2 *__restrict__ p14;
    const SysDev *__restrict__ sys;
    const int *__restrict__ atom_sys;
    int n_excl, n_14, n_pad;
    float rc, rc2, rs2, sw_inv_den, beta, ewald_fc;
    int do_excl, do_lj14, do_coul14;
    float excl_weight;  // weight of the excluded-pair reciprocal correction's force
    unsigned long long *f;
    unsigned long long *fx;  // where the excluded-pair correction's force goes
    long long *energy;
    int *dump;
    long long dump_cap;
    unsigned long long *dump_count;
};

// Excluded 1-2/1-3 pairs: -k q q erf(beta r)/r removes their share of the
// reciprocal sum (term COUL_RECIP).  1-4 pairs: LJ with the 1-4 parameters
// (charmm_nonbonded_constraint.py:92-97) and the real-space Coulomb term.
// ENERGY: only an evaluation that reports energies sums them (three FP64 warp
// sums a thread otherwise).
template <bool SWITCH, bool DUMP, bool ENERGY>
__global__ void k_special(SpArgs a) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    float e_lj = 0.f, e_cr = 0.f, e_rec = 0.f;
    int sid = -1;
    if (t < a.n_excl + a.n_14) {
        const bool is14 = t >= a.n_excl;
        const int2 pr = is14 ? a.p14[t - a.n_excl] : a.excl[t];
        const int i = pr.x, j = pr.y;
        sid = a.atom_sys[i];
        const SysDev &sd = a.sys[sid];
        float d[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = min_image(sd, a.x[3 * j + k], a.x[3 * i + k], k);
        const float r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        const float r = sqrtf(r2);
        const float qq = a.charge[i] * a.charge[j];
        float fr = 0.f;
        if (!is14) {
            if (a.do_excl) {
                const float br = a.beta * r;
                const float ef = erff(br);
                e_rec = -qq * ef / r;
                fr = a.excl_weight * qq * (a.ewald_fc * expf(-br * br) * r - ef) / (r2 * r);
            }
        } else if (DUMP) {
            // pair dump: the reference's own float32 pair test decides
            if (ref_within32(a.x, i, j, sd, a.rc)) {
                unsigned long long slot = atomicAdd(a.dump_count, 1ull);
                if ((long long)slot < a.dump_cap) {
                    a.dump[2 * slot] = min(i, j);
                    a.dump[2 * slot + 1] = max(i, j);
                }
            }
        } else if (r2 <= a.rc2) {
            if (a.do_lj14) {
                const float4 pi = a.lj[i], pj = a.lj[j];
                const float sig = pi.z + pj.z;
                const float s2 = sig * sig / r2;
                const float s6 = s2 * s2 * s2;
                const float c6 = pi.w * pj.w * s6;
                float elj = c6 * (s6 - 1.0f);
                float flj = c6 * (12.0f * s6 - 6.0f) / r2;
                if (SWITCH && r2 > a.rs2) {
                    const float u = a.rc2 - r2;
                    const float sw = u * u * (a.rc2 + 2.0f * r2 - 3.0f * a.rs2) * a.sw_inv_den;
                    const float dsw = 12.0f * u * (a.rs2 - r2) * a.sw_inv_den;
                    flj = flj * sw - elj * dsw;
                    elj *= sw;
                }
                e_lj = elj;
                fr += flj;
            }
            if (a.do_coul14) {
                const float br = a.beta * r;
                const float ec = erfcf(br);
                e_cr = qq * ec / r;
                fr += qq * (ec / r + a.ewald_fc * expf(-br * br)) / r2;
            }
        }
        if (!DUMP && fr != 0.f) {
            const int ki = a.inv_perm[i], kj = a.inv_perm[j];
            unsigned long long *ff = is14 ? a.f : a.fx;
            fix_red(&ff[kj], to_fix(fr * d[0]));
            fix_red(&ff[a.n_pad + kj], to_fix(fr * d[1]));
            fix_red(&ff[2 * a.n_pad + kj], to_fix(fr * d[2]));
            fix_red(&ff[ki], to_fix(-fr * d[0]));
            fix_red(&ff[a.n_pad + ki], to_fix(-fr * d[1]));
            fix_red(&ff[2 * a.n_pad + ki], to_fix(-fr * d[2]));
        }
    }
    if (DUMP || !ENERGY) return;
    // FP64 block sums: the exclusion term is a sum of O(10^5) terms of either
    // sign whose total largely cancels the self energy
    const double v[3] = {(double)e_lj, (double)e_cr, (double)e_rec};
    const int slot[3] = {MDG_TERM_LJ, MDG_TERM_COUL_REAL, MDG_TERM_COUL_RECIP};
    block_energy_add<3>(a.energy, sid, v, slot);
}

NbArgs make_args(mdg_system *s) {
    NbArgs a;
    a.xq = s->xq;
    a.prm = s->prm_sorted;
    a.partners = s->partners_sorted;
    a.pw = s->pw;
    a.prange = s->cluster_partner_range;
    a.bbox = s->bbox;
    a.n = s->n;
    a.n_pad = s->n_pad;
    a.n_clusters = s->n_clusters;
    a.sys = s->sys_dev;
    a.cl_sys = s->cl_sys;
    a.cl_col = s->cl_col;
    a.hbox = s->hbox;
    a.qbox = s->qbox;
    a.col_xy = s->col_xy;
    a.col_rank = s->cell_rank;
    a.col_cl_start = s->col_cl_start;
    a.col_ncl = s->col_ncl;
    a.overhang = s->overhang;
    a.rc = s->cutoff;
    a.rc2 = s->cutoff * s->cutoff;
    const double rs = s->rswitch > 0 ? s->rswitch : s->cutoff;
    a.rs2 = (float)(rs * rs);
    const double den = (double)a.rc2 - rs * rs;
    a.sw_inv_den = den > 0 ? (float)(1.0 / (den * den * den)) : 0.f;
    a.sw_um = den > 0 ? (float)(-1.0 / den) : 0.f;
    a.sw_uc = den > 0 ? (float)((double)a.rc2 / den) : 1.f;
    a.sw_g = den > 0 ? (float)(12.0 / den) : 0.f;
    a.beta = (float)s->beta;
    a.beta_p = kAsP * (float)s->beta;
    a.ewald_exp_c = (float)(s->beta * s->beta * 1.4426950408889634);
    a.ewald_fc = (float)(2.0 * s->beta / 1.7724538509055159);
    a.lj_on = s->lj_on;
    a.f = s->f;
    a.energy = s->energy;
    a.status = s->status;
    a.stats = s->stats;
    a.dump = s->dump_buf;
    a.dump_cap = s->dump_cap;
    a.dump_count = s->dump_count;
    a.perm = s->perm;
    a.x = s->x;
    a.rc_ref = s->cutoff;
    a.by_size = s->nb_split == 0 && s->coul_mode == MDG_COUL_EWALD;
    a.split = nb_parts(s);
    a.persistent = s->nb_persistent > 0;
    a.n_items = s->n_clusters * a.split;
    a.queue = s->nb_queue;
    // persistent form: one queue atomic per `grab` consecutive items, so
    // that a batch of ~10^5 items does not serialise on the counter; each
    // resident warp still sees about 16 grabs, which keeps the tail short
    a.grab = 1;
    if (s->nb_persistent_ctas > 0)
        a.grab = std::max(1, std::min(8, a.n_items / (16 * s->nb_persistent_ctas)));
    a.split_rings = s->nb_split_rings;
    return a;
}


}  // namespace

// work items per cluster: as set, or the most that any system's size calls for.
// LJ without Ewald: 4 at every size, which keeps the bits of its FP32 chains (bare
// Coulomb runs hang on them).  A Lennard-Jones fluid, us at 2 / 4 items: 2,700 atoms
// 37 / 30.5, 12k 30 / 25, 20k 33 / 32, 80k 81 / 79, but 130k 108 / 117, 300k 231 / 287.
int nb_parts(const mdg_system *s) {
    if (s->nb_split > 0) return s->nb_split;
    if (s->coul_mode != MDG_COUL_EWALD) return 4;
    int p = 1;
    for (const SysDev &d : s->sys_h) p = std::max(p, nb_default_parts(d.n_atoms));
    return p;
}

bool nb_parts_uniform(const mdg_system *s) {
    if (s->nb_split > 0 || s->coul_mode != MDG_COUL_EWALD) return true;
    const int p = nb_default_parts(s->sys_h[0].n_atoms);
    return std::all_of(s->sys_h.begin(), s->sys_h.end(),
                       [p](const SysDev &d) { return nb_default_parts(d.n_atoms) == p; });
}

cudaError_t launch_nonbonded(mdg_system *s, unsigned mask, int energy, int dump) {
    const bool want_lj = (mask & MDG_MASK(MDG_TERM_LJ)) && s->lj_on;
    const bool want_c = (mask & MDG_MASK(MDG_TERM_COUL_REAL)) && s->coul_mode != MDG_COUL_NONE;
    if (!want_lj && !want_c) return cudaSuccess;
    NbArgs a = make_args(s);
    a.lj_on = want_lj ? 1 : 0;
    if (dump) {
        // the pair dump searches a little beyond the cutoff and lets the
        // reference's float32 test (ref_within32) decide each candidate:
        // the packed float32 coordinates differ from the reference's by
        // rounding (~1e-5 A), far below this margin
        a.rc = s->cutoff + kDumpMargin;
        a.rc2 = a.rc * a.rc;
    }
    const bool sw = s->rswitch > 0 && s->rswitch < s->cutoff;
    cudaError_t err = cudaSuccess;
    const int coul_tile = (want_c && s->coul_mode == MDG_COUL_EWALD) ? MDG_COUL_EWALD : MDG_COUL_NONE;
    if (want_lj || coul_tile == MDG_COUL_EWALD) {
        // Ewald items of small systems, too few to fill the GPU, are taken by several
        // warps each (the sums are the same; those of LJ without Ewald are FP32
        // chains, which only one warp can add up in their order): the most that keep every item with
        // work resident (16 warps an SM at this kernel's registers; 4 warps less, as
        // the PME and bonded kernels beside it take room).  A cluster's parts walk
        // batches of 32 clusters, so a system of 64 to 96 has three parts with work.
        // A whole step, us at 1 / 2 / 3 / 4 / 8 warps: 279 items with work (2,700 atoms,
        // rc 12) 67 / 46 / 41 / 37 / 35, 408 (3,000, rc 9) 50 / 36 / 31 / 31 / 40, 536
        // (3,900, rc 9) 49 / 36 / 33 / 33 / 45, 576 (4,200, rc 12) 57 / 41 / 37 / 40 / 50,
        // 748 (5,400, rc 12) 80 / 56 / 52 / 55 / 65, 788 (5,700, rc 9) 50 / 38 / 45 / 48 / 57,
        // 1060 (7,800, rc 10) 50 / 42 / 53 / 54 / 72
        bool small = true;
        int work = 0;
        for (const SysDev &d : s->sys_h) {
            small = small && d.n_atoms < kNbBlockSystem;
            const int cl = (d.n_atoms + kCluster - 1) / kCluster + d.n_cols / 2;
            work += cl * std::min(a.split, (cl + 31) / 32);
        }
        const int warps = work <= 2 * s->n_sms        ? 8
                          : work <= 18 * s->n_sms / 5 ? 4
                          : work <= 5 * s->n_sms      ? 3
                          : work <= 8 * s->n_sms      ? 2
                                                      : 1;
        // (a pair dump takes the form that the system's forces take: it asks for LJ
        // alone, so the mode decides)
        const bool ewald = dump ? s->coul_mode == MDG_COUL_EWALD : coul_tile == MDG_COUL_EWALD;
        if (ewald && s->nb_half == 0 && !s->nb_persistent && small && warps > 1)
            err = launch_nb_block(s, a, warps, want_lj, sw, energy, dump);
        else
            err = s->nb_half == 2   ? launch_nb_quarter(s, a, coul_tile, want_lj, sw, energy, dump)
                  : s->nb_half == 1 ? launch_nb_half(s, a, coul_tile, want_lj, sw, energy, dump)
                  : s->n_sys > 1 || small
                      ? launch_nb_batch(s, a, coul_tile, want_lj, sw, energy, dump)
                      : dispatch_shape<false>(s, a, coul_tile, want_lj, sw, energy, dump);
        s->launches += 1;
        if (err != cudaSuccess) return err;
    }
    if (want_c && s->coul_mode == MDG_COUL_BARE && !dump) {
        if (energy) k_coulomb_bare<true><<<s->n_clusters, kBareThreads, 0, s->stream>>>(a);
        else k_coulomb_bare<false><<<s->n_clusters, kBareThreads, 0, s->stream>>>(a);
        s->launches += 1;
        err = cudaGetLastError();
    }
    return err;
}

cudaError_t launch_special(mdg_system *s, unsigned mask, int energy, int dump) {
    SpArgs a;
    a.x = s->x;
    a.inv_perm = s->inv_perm;
    a.charge = s->charge;
    a.lj = s->lj;
    a.excl = s->excl_pairs;
    a.p14 = s->pairs14;
    a.n_excl = s->n_excl;
    a.n_14 = s->n_14;
    a.n_pad = s->n_pad;
    a.sys = s->sys_dev;
    a.atom_sys = s->atom_sys;
    a.rc = s->cutoff;
    a.rc2 = s->cutoff * s->cutoff;
    const double rs = s->rswitch > 0 ? s->rswitch : s->cutoff;
    a.rs2 = (float)(rs * rs);
    const double den = (double)a.rc2 - rs * rs;
    a.sw_inv_den = den > 0 ? (float)(1.0 / (den * den * den)) : 0.f;
    a.beta = (float)s->beta;
    a.ewald_fc = (float)(2.0 * s->beta / 1.7724538509055159);
    a.do_excl = (mask & MDG_MASK(MDG_TERM_COUL_RECIP)) && s->pme.on && !dump;
    a.excl_weight = s->recip_weight;
    a.do_lj14 = (mask & MDG_MASK(MDG_TERM_LJ)) && s->lj_on;
    a.do_coul14 = (mask & MDG_MASK(MDG_TERM_COUL_REAL)) && s->coul_mode == MDG_COUL_EWALD;
    a.f = s->f;
    a.fx = s->slow_target ? s->slow_target : s->f;
    a.energy = s->energy;
    a.dump = s->dump_buf;
    a.dump_cap = s->dump_cap;
    a.dump_count = s->dump_count;
    if (!dump && !a.do_lj14 && !a.do_coul14) a.n_14 = 0;
    if (!a.do_excl) a.n_excl = 0;
    if (dump && !(a.do_lj14 || a.do_coul14)) a.n_14 = 0;
    const int total = a.n_excl + a.n_14;
    if (total == 0) return cudaSuccess;
    const bool sw = s->rswitch > 0 && s->rswitch < s->cutoff;
    const int tb = 256, nb = (total + tb - 1) / tb;
    if (dump)
        k_special<false, true, false><<<nb, tb, 0, s->stream>>>(a);
    else if (energy)
        sw ? k_special<true, false, true><<<nb, tb, 0, s->stream>>>(a)
           : k_special<false, false, true><<<nb, tb, 0, s->stream>>>(a);
    else
        sw ? k_special<true, false, false><<<nb, tb, 0, s->stream>>>(a)
           : k_special<false, false, false><<<nb, tb, 0, s->stream>>>(a);
    s->launches += 1;
    return cudaGetLastError();
}

}  // namespace mdg
