/*
 * Launches of the element reverse kernels (p = 1 and p = 2), in a translation unit of their own
 * that is compiled with contraction (build.py): nothing in them decides anything and nothing of
 * the forward step is recomputed for its bits, so products and sums may fuse.  The kernels are
 * bound by FP64 issue and dependency chains (128 registers, 16 warps per SM; one p = 1 launch
 * on 200k triangles took 69-77 us for 31 us of bytes).  With H^(-4/3) by rcbrt, the p = 2
 * kernel's output adjoint read twice instead of held over the area loop (spills 392 -> 232 B)
 * and roe_flux_rev's four divisions instead of eleven, backward runs: 30 steps on 5k triangles
 * 4.08 -> 3.80 ms, 20 steps on 200k 10.62 -> 10.04, the p = 2 calibration of eight basins 10.43 ->
 * 9.69.
 */
#include "dgr_internal.cuh"
#include "dgr_p2_adjoint.cuh"
#include "dgr_tlm.cuh"

using namespace dgr;

template <int MODE>
static void adj_element(dgr_ctx *c, const double *S, const int *wd, const double *Rbar, const double *bnode,
                        const int *barg, double *lamS, double *lamU, int u_acc, double *fbar, double *zvb, double *nbar,
                        const double *dt)
{
    launch_dep(k_adj_element<MODE>, blocks(c->ne, 128), 128, c->stream, mesh_dev(c), S, wd, Rbar, bnode, barg, lamS, lamU,
               u_acc, fbar, zvb, nbar, c->n_el, c->p.g, dt);
}

void launch_adj_element(dgr_ctx *c, int mode, const double *S, const int *wd, const double *Rbar, const double *bnode,
                        const int *barg, double *lamS, double *lamU, int u_acc, double *fbar, double *zvb, double *nbar,
                        const double *dt)
{
    switch (mode) {
    case MODE_STAGE1: adj_element<MODE_STAGE1>(c, S, wd, Rbar, bnode, barg, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    case MODE_STAGE2: adj_element<MODE_STAGE2>(c, S, wd, Rbar, bnode, barg, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    case MODE_RK3_2: adj_element<MODE_RK3_2>(c, S, wd, Rbar, bnode, barg, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    default: adj_element<MODE_RK3_3>(c, S, wd, Rbar, bnode, barg, lamS, lamU, u_acc, fbar, zvb, nbar, dt);
    }
}

template <int MODE>
static void p2_adj_element(dgr_ctx *c, const double *S, const double *lamO, double *lamS, double *lamU, int u_acc,
                           double *fbar, double *zvb, double *nbar, const double *dt)
{
    launch_dep(k_p2_adj_element<MODE>, blocks(c->ne, 128), 128, c->stream, c->p2ref, mesh_dev(c), c->p2g, S, lamO, lamS,
               lamU, u_acc, fbar, zvb, nbar, c->n_el, c->p.g, dt);
}

void launch_p2_adj_element(dgr_ctx *c, int mode, const double *S, const double *lamO, double *lamS, double *lamU,
                           int u_acc, double *fbar, double *zvb, double *nbar, const double *dt)
{
    switch (mode) {
    case MODE_STAGE1: p2_adj_element<MODE_STAGE1>(c, S, lamO, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    case MODE_STAGE2: p2_adj_element<MODE_STAGE2>(c, S, lamO, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    case MODE_RK3_2: p2_adj_element<MODE_RK3_2>(c, S, lamO, lamS, lamU, u_acc, fbar, zvb, nbar, dt); break;
    default: p2_adj_element<MODE_RK3_3>(c, S, lamO, lamS, lamU, u_acc, fbar, zvb, nbar, dt);
    }
}
