// The kernels of the fake CUDA runtime (fake_cuda.cpp).  Their mechanics are chosen so
// that a test can read off what ran: a step's first kick and its last add a half of
// the force (1 after an evaluation) to every velocity, so n whole steps add n;
// positions move by 1 a step.
#include <cstdlib>
#include <cstring>
#include <functional>

#include "../../mdpy_gb300/csrc/mdg_internal.cuh"

cudaError_t issue(const char *name, std::function<void()> op);  // fake_cuda.cpp

static void kick(mdg_system *s) {
    for (int i = 0; i < 3 * s->n; ++i) s->v[i] += 0.5 * (double)s->f[0];
}

extern "C" __attribute__((visibility("default"))) long long fake_device_step(mdg_system *s) {
    return (long long)*s->step_dev;
}

namespace mdg {

cudaError_t launch_reorder(mdg_system *) { return issue("reorder", [] {}); }
cudaError_t launch_pack(mdg_system *s) {
    return issue("pack", [=] { s->f[0] = 0; });
}
cudaError_t launch_nonbonded(mdg_system *s, unsigned, int energy, int) {
    return issue("nonbonded", [=] {
        s->f[0] += 1;
        if (energy) s->energy[MDG_TERM_LJ] += 1;
    });
}
int nb_parts(const mdg_system *) { return 4; }
bool nb_parts_uniform(const mdg_system *) { return true; }
cudaError_t launch_special(mdg_system *, unsigned, int, int) { return issue("special", [] {}); }
cudaError_t launch_pme(mdg_system *, int, int *) { return issue("pme", [] {}); }
cudaError_t launch_bonded(mdg_system *, unsigned, int) { return issue("bonded", [] {}); }
cudaError_t launch_move(mdg_system *s, bool post) {
    return issue("move", [=] {
        if (post) kick(s);
        kick(s);
        for (int i = 0; i < 3 * s->n; ++i) s->x[i] += 1.0;
    });
}
cudaError_t launch_count_step(mdg_system *s) {
    return issue("count_step", [=] { *s->step_dev += 1; });
}
cudaError_t launch_integrate_post(mdg_system *s, int) {
    return issue("post", [=] {
        kick(s);
        *s->step_dev += 1;
    });
}
cudaError_t launch_kinetic(mdg_system *s) {
    return issue("kinetic", [=] { s->energy[kSlotKinetic] = (long long)(s->v[0] * 4294967296.0); });
}
cudaError_t launch_forces_out(mdg_system *s) {
    return issue("forces_out", [=] {
        for (int i = 0; i < 3 * s->n; ++i) s->fout[i] = (double)s->f[0];
    });
}
cudaError_t launch_positions_out(mdg_system *s, double *out) {
    return issue("positions_out", [=] { memcpy(out, s->x, sizeof(double) * 3 * s->n); });
}
cudaError_t launch_same_positions(mdg_system *, const double *, int *) { return cudaSuccess; }
cudaError_t launch_noise(mdg_system *, uint64_t, float *) { return cudaSuccess; }
cudaError_t launch_sd_step(mdg_system *, double) { return cudaSuccess; }
int prepare_sort_grid(mdg_system *s) {
    s->n_pad = s->n;
    if (!s->f) s->f = (unsigned long long *)calloc(3 * (size_t)s->n, sizeof(unsigned long long));
    return MDG_OK;
}
int pme_setup(mdg_system *, const int *) { return MDG_OK; }
int upload_sys_table(mdg_system *) { return MDG_OK; }
void pme_free(mdg_system *) {}
cudaError_t noalloc_scratch(int, long long **) { return cudaErrorNotSupported; }
cudaError_t launch_kinetic_scratch(mdg_system *, long long *) { return cudaErrorNotSupported; }
int ls_configure(mdg_system *, float, float, int) { return MDG_ERR_INVALID; }
void ls_free(mdg_system *) {}
cudaError_t ls_side(mdg_system *, int) { return cudaSuccess; }
cudaError_t ls_after_join(mdg_system *, int) { return cudaSuccess; }
cudaError_t ls_refresh_weights(mdg_system *) { return cudaSuccess; }
cudaError_t ls_train(mdg_system *, float, int, double *) { return cudaSuccess; }
cudaError_t ls_predict(mdg_system *, int) { return cudaSuccess; }

}  // namespace mdg
