// FP64 residual of the finite-difference system, the refinement step of FD
// plans created with HELM_FP32_REFINE: the solve runs in FP32 (FP32 spectrum,
// FP32 tridiagonal solves), the residual r = f - A_h u is formed here from the
// 7-point stencil in FP64 (HypreFDM/src/Helmholtz3D_MPI.cpp:387-403, x and y
// periodic, the Robin rows eliminated into the first and last z equations as
// the solve does), and an FP32 solve of A_h d = r is added to u.  The adjoint
// refines the same way with the transposed stencil.
#include <cuda_runtime.h>

#include "helm_device.cuh"
#include "helm_fd_refine.cuh"

namespace helm {

namespace {

// The z rows of A_h on the interior unknowns: diagonal dz = -2 cz1 (+ dfirst at
// k = 0, + dlast at k = Nz - 1), neighbours cz1, except A[0][1] = sfirst and
// A[Nz-1][Nz-2] = slast; forward data terms scale_l * gl at k = 0 and
// scale_r * gr at k = Nz - 1 on the right-hand side.
//
// A CTA takes RES_PER * 256 consecutive points of one x plane, RES_PER a thread,
// and a thread fetches all it reads before it computes.  Bound: instruction issue (77 %
// of the slots, for eight neighbours' addresses and the FP64 arithmetic a point; the
// 66 MB of 256 x 128 x 100 alone would take 10 us).  One point after another with 64-bit
// divisions for (i, j, k) took 34.5 us there, this 29 us; marching along x with the
// planes in registers (2 or 4 a thread) took 30 and 36 us: the registers cost more
// warps than the reads saved.
constexpr int RES_PER = 2;

__global__ void __launch_bounds__(256) fd_residual_kernel(FdResidualArgs a)
{
    pdl_enter();
    const int nz = a.Nz, plane = a.Ny * nz, i = blockIdx.y;
    const int o0 = blockIdx.x * (256 * RES_PER) + threadIdx.x;
    const double* v = a.v + (long long)i * plane;
    const double* vm = a.v + (long long)(i == 0 ? a.Nx - 1 : i - 1) * plane;
    const double* vp = a.v + (long long)(i == a.Nx - 1 ? 0 : i + 1) * plane;
    const double* rhs = a.rhs + (long long)i * plane;
    const double* sub = a.sub ? a.sub + (long long)i * plane : nullptr;
    double vc[RES_PER], x0[RES_PER], x1[RES_PER], y0[RES_PER], y1[RES_PER], z0[RES_PER], z1[RES_PER], f[RES_PER],
        g[RES_PER];
    int kk[RES_PER];
#pragma unroll
    for (int e = 0; e < RES_PER; ++e) {
        const int o = min(o0 + 256 * e, plane - 1);
        const int j = o / nz, k = o - j * nz;
        kk[e] = k;
        vc[e] = v[o];
        x0[e] = vm[o];
        x1[e] = vp[o];
        y0[e] = v[j == 0 ? o + plane - nz : o - nz];
        y1[e] = v[j == a.Ny - 1 ? o - (plane - nz) : o + nz];
        z0[e] = v[k > 0 ? o - 1 : o];
        z1[e] = v[k < nz - 1 ? o + 1 : o];
        f[e] = rhs[o];
        g[e] = sub ? sub[o] : 0.0;
    }
    const double cdiag = -2.0 * (a.cx1 + a.cy1 + a.cz1) - a.lam;
#pragma unroll
    for (int e = 0; e < RES_PER; ++e) {
        const int o = o0 + 256 * e, k = kk[e];
        if (o >= plane) break;
        double az = ((k == 0 ? a.dfirst : 0.0) + (k == nz - 1 ? a.dlast : 0.0)) * vc[e];
        if (k > 0) az += (a.transpose ? (k == 1 ? a.sfirst : a.cz1) : (k == nz - 1 ? a.slast : a.cz1)) * z0[e];
        if (k < nz - 1) az += (a.transpose ? (k == nz - 2 ? a.slast : a.cz1) : (k == 0 ? a.sfirst : a.cz1)) * z1[e];
        const double av = a.cx1 * (x0[e] + x1[e]) + a.cy1 * (y0[e] + y1[e]) + cdiag * vc[e] + az;
        double r = f[e] - g[e];
        const long long rj = (long long)i * a.Ny + o / nz;
        if (k == 0 && a.gl) r += a.scale_l * a.gl[rj];
        if (k == nz - 1 && a.gr) r += a.scale_r * a.gr[rj];
        a.r[(long long)i * plane + o] = (float)(r - av);
    }
}

}  // namespace

int launch_fd_residual(const FdResidualArgs& a, cudaStream_t s)
{
    const int per = 256 * RES_PER, plane = a.Ny * a.Nz;
    return (int)launch_k(fd_residual_kernel, dim3((plane + per - 1) / per, a.Nx), dim3(256), 0, s, a);
}

}  // namespace helm
