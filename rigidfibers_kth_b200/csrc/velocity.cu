// velocity.cu - the velocities from their integrals (the sums over the sources
// are in pair_sum.cu) and K4 advection.
//
// Reference: fortran/coeffs_and_vels.f90:698-730 (local term, scaling),
// advect_fibers.f90:498-523; src/kernels/update_velocities.cu:101-191,
// update_fibers*.cu.
#include "rf_kernels.h"

namespace rf {

// Local term and final scaling (coeffs_and_vels.f90:698-705, 723-730).
// A CTA owns kFinFibers fibers: one thread per (fiber, value) adds that value's
// per-chunk partials in chunk order (consecutive threads read consecutive
// values), then one thread per fiber combines its six.
constexpr int kFinFibers = 32;
__global__ void __launch_bounds__(6 * kFinFibers) velocity_finish_kernel(int M, int t0, int t1, const double *ori,
                                                                         const Tables *tab, const double *part,
                                                                         int nchunks, const double *pv_x,
                                                                         const double *pw_x, double *V, double *W) {
    __shared__ double s_s[6 * kFinFibers];
    const int i0 = t0 + blockIdx.x * kFinFibers;
    if (i0 + (int)threadIdx.x / 6 < t1) {
        const double *p = part + (int64_t)i0 * 6 + threadIdx.x;
        double s = 0.0;
        for (int c = 0; c < nchunks; ++c) s += p[(int64_t)c * 6 * M];
        s_s[threadIdx.x] = s;
    }
    __syncthreads();
    const int i = i0 + threadIdx.x;
    if (threadIdx.x >= kFinFibers || i >= t1) return;
    const double *s = s_s + 6 * threadIdx.x;
    const double d = tab->d, e = tab->e;
    const double *t = ori + 3 * i;
    const double *F = tab->force;
    const double tdf = t[0] * F[0] + t[1] * F[1] + t[2] * F[2];
    if (pv_x) {
        // reuse path: partials already hold scaled l = 0 terms; add the panel products
        for (int a = 0; a < 3; ++a) {
            V[3 * i + a] = 0.5 * ((d + e) * F[a] + (d - e) * tdf * t[a]) / d + s[a] + pv_x[3 * i + a];
            W[3 * i + a] = s[3 + a] + pw_x[3 * i + a];
        }
        return;
    }
    const double tdi = t[0] * s[3] + t[1] * s[4] + t[2] * s[5];
    for (int a = 0; a < 3; ++a) {
        const double loc = 0.5 * ((d + e) * F[a] + (d - e) * tdf * t[a]);
        V[3 * i + a] = (loc + 0.5 * s[a]) / d;
        W[3 * i + a] = 1.5 * (s[3 + a] - tdi * t[a]) / d;
    }
}

cudaError_t launch_velocity_finish(int M, int t0, int t1, const double *ori, const Tables *tab, const double *part,
                                   int nchunks, double *V, double *W, cudaStream_t st) {
    velocity_finish_kernel<<<(t1 - t0 + kFinFibers - 1) / kFinFibers, 6 * kFinFibers, 0, st>>>(
        M, t0, t1, ori, tab, part, nchunks, nullptr, nullptr, V, W);
    return cudaGetLastError();
}

cudaError_t launch_velocity_reuse_finish(int M, const double *ori, const Tables *tab, const double *pv_x,
                                         const double *pw_x, const double *vpart, int nchunks, double *V,
                                         double *W, cudaStream_t st) {
    velocity_finish_kernel<<<(M + kFinFibers - 1) / kFinFibers, 6 * kFinFibers, 0, st>>>(
        M, 0, M, ori, tab, vpart, nchunks, pv_x, pw_x, V, W);
    return cudaGetLastError();
}

// Forward Euler (first step) or the second-order multistep
// x+ = 4/3 x - 1/3 x- + 2/3 dt (2 v - v-), then t <- t/|t|
// (advect_fibers.f90:498-523).
__global__ void advect_kernel(int M, double dt, int first, const double *Xp, const double *Xc,
                              const double *Tp, const double *Tc, const double *Vn, const double *Vo,
                              const double *Wn, const double *Wo, double *Xn, double *Tn) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    double tn[3];
    for (int a = 0; a < 3; ++a) {
        const int k = 3 * i + a;
        if (first) {
            Xn[k] = Xc[k] + dt * Vn[k];
            tn[a] = Tc[k] + dt * Wn[k];
        } else {
            Xn[k] = 4.0 / 3.0 * Xc[k] - 1.0 / 3.0 * Xp[k] + 2.0 / 3.0 * dt * (2.0 * Vn[k] - Vo[k]);
            tn[a] = 4.0 / 3.0 * Tc[k] - 1.0 / 3.0 * Tp[k] + 2.0 / 3.0 * dt * (2.0 * Wn[k] - Wo[k]);
        }
    }
    const double tm = sqrt(tn[0] * tn[0] + tn[1] * tn[1] + tn[2] * tn[2]);
    for (int a = 0; a < 3; ++a) Tn[3 * i + a] = tn[a] / tm;
}

cudaError_t launch_advect(int M, double dt, bool first, const double *Xp, const double *Xc, const double *Tp,
                          const double *Tc, const double *Vn, const double *Vo, const double *Wn,
                          const double *Wo, double *Xn, double *Tn, cudaStream_t st) {
    advect_kernel<<<(M + 127) / 128, 128, 0, st>>>(M, dt, first ? 1 : 0, Xp, Xc, Tp, Tc, Vn, Vo, Wn, Wo, Xn, Tn);
    return cudaGetLastError();
}

__global__ void normalize_kernel(int M, double *T) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    double *t = T + 3 * i;
    const double tm = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    t[0] /= tm;
    t[1] /= tm;
    t[2] /= tm;
}

cudaError_t launch_normalize(int M, double *T, cudaStream_t st) {
    normalize_kernel<<<(M + 127) / 128, 128, 0, st>>>(M, T);
    return cudaGetLastError();
}

}  // namespace rf
