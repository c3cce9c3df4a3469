// Granular walls (tmps_wall.cuh), one thread per atom, added to the forces.
#include "tmps_common.cuh"
#include "tmps_wall.cuh"

using namespace tmps;
using namespace tmps_wall_law;

namespace {

constexpr int kBlock = 128;

__global__ void __launch_bounds__(kBlock) k_wall(tmps_atoms a, tmps_wall_params P, double dt, int upd,
                                                 double* __restrict__ shear, int32_t* __restrict__ touch_,
                                                 int nslots) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = a.n;
    if (i >= n) return;
    const int u = a.uid ? a.uid[i] : i;
    double sh[3] = {0.0, 0.0, 0.0};
    int touch = 0;
    if (P.history) {
        sh[0] = shear[u];
        sh[1] = shear[(size_t)nslots + u];
        sh[2] = shear[2 * (size_t)nslots + u];
        touch = touch_[u];
    }
    const double4 xr = ld4(a.xr, i), vm = ld4(a.vm, i), om = ld4(a.om, i);
    const double x[3] = {xr.x, xr.y, xr.z}, v[3] = {vm.x, vm.y, vm.z}, w[3] = {om.x, om.y, om.z};
    const double ri = xr.w, mi = vm.w;
    bool contact = false;
    double F[3] = {0, 0, 0}, T[3] = {0, 0, 0};
    contact = wall_force(P, dt, upd, x, ri, v, mi, w, sh, touch, F, T);
    if (contact) {
        for (int k = 0; k < 3; ++k) {
            a.f[(size_t)k * n + i] += F[k];
            a.torque[(size_t)k * n + i] += T[k];
        }
    } else {
        touch = 0;
        sh[0] = sh[1] = sh[2] = 0.0;
    }
    if (P.history) {
        shear[u] = sh[0];
        shear[(size_t)nslots + u] = sh[1];
        shear[2 * (size_t)nslots + u] = sh[2];
        touch_[u] = touch;
    }
}

}  // namespace

extern "C" int tmps_wall_gran(const tmps_atoms* a, const tmps_wall_params* p, double dt, int32_t history_update,
                              double* d_shear, int32_t* d_touch, int32_t nslots, void* stream) {
    if (!a || !p || a->n < 0) return TMPS_ERR_BAD_ARG;
    if (p->kind < 0 || p->kind > 1 || p->axis < 0 || p->axis > 2 || (p->side != -1 && p->side != 1))
        return TMPS_ERR_BAD_ARG;
    if (p->kind == 0 && (p->shear_axis < -1 || p->shear_axis > 2 || p->shear_axis == p->axis)) return TMPS_ERR_BAD_ARG;
    if (p->history && (!d_shear || !d_touch || nslots < a->n)) return TMPS_ERR_BAD_ARG;
    if (a->n == 0) return TMPS_OK;
    k_wall<<<grid_for(a->n, kBlock), kBlock, 0, (cudaStream_t)stream>>>(*a, *p, dt, history_update, d_shear,
                                                                          d_touch, nslots);
    note_launches(1);
    return cudaPeekAtLastError() == cudaSuccess ? TMPS_OK : TMPS_ERR_CUDA;
}
