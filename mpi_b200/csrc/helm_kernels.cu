// CUDA kernels of the Helmholtz solve (sm_100a):
//   * rows_kernel -- the per-wavenumber collocation solves of every spectrum
//     row (ConstructFundamentalSolutions + LUSolve, NonPeriodic2D_MPI.cpp:176-223,
//     LU_Decomposition.cpp:78-108), the element-interface tridiagonal sweep with
//     the Robin ends (NonPeriodic2D_MPI.cpp:265-295, 414-424) and the combination
//     u = phi + zl ul + zr ur (:466-470), fused, one warp per complex row (the LU
//     method; fast-diagonalisation plans with several elements: helm_multi.cu).
#include <algorithm>
#include <type_traits>

#include "helm_device.cuh"
#include "helm_kernels.cuh"

namespace helm {

// ======================================================== row solves ==

constexpr int ROW_WARPS = 4;
constexpr int ROW_NSMAX = 64;  // max GLL elements per row handled by rows_kernel

__device__ __forceinline__ float shfl(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ double shfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
template <typename T> __device__ __forceinline__ T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// x <- (P A)^-1 P x with the combined column-major L\U factor F (unit lower L),
// dinv = 1/U_ii, perm = source row of each position.  Lane l owns rows l + 32 s.
template <typename TF, int NSLOT>
__device__ __forceinline__ void lu_core(const TF* F, int ld, const TF* dinv, const int* perm, int n, TF (&xr)[NSLOT],
                                        TF (&xi)[NSLOT], TF* scr, int lane)
{
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
        scr[lane + 32 * s] = xr[s];
        scr[32 * NSLOT + lane + 32 * s] = xi[s];
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
        const int i = lane + 32 * s;
        const int p = (i < n) ? perm[i] : i;
        xr[s] = scr[p];
        xi[s] = scr[32 * NSLOT + p];
    }
    __syncwarp();
    // forward substitution with the unit lower factor
#pragma unroll
    for (int ks = 0; ks < NSLOT; ++ks) {
        for (int kl = 0; kl < 32; ++kl) {
            const int k = ks * 32 + kl;
            if (k >= n - 1) break;
            const TF yr = shfl(xr[ks], kl), yi = shfl(xi[ks], kl);
            const TF* col = F + (size_t)k * ld;
#pragma unroll
            for (int s = ks; s < NSLOT; ++s) {
                if (s > ks || lane > kl) {
                    const TF f = col[lane + 32 * s];
                    xr[s] -= f * yr;
                    xi[s] -= f * yi;
                }
            }
        }
    }
    // back substitution with U, column by column
#pragma unroll
    for (int ks = NSLOT - 1; ks >= 0; --ks) {
        for (int kl = 31; kl >= 0; --kl) {
            const int k = ks * 32 + kl;
            if (k >= n) continue;
            const TF di = dinv[k];
            const TF yr = shfl(xr[ks], kl) * di, yi = shfl(xi[ks], kl) * di;
            if (lane == kl) { xr[ks] = yr; xi[ks] = yi; }
            const TF* col = F + (size_t)k * ld;
#pragma unroll
            for (int s = 0; s <= ks; ++s) {
                if (s < ks || lane < kl) {
                    const TF f = col[lane + 32 * s];
                    xr[s] -= f * yr;
                    xi[s] -= f * yi;
                }
            }
        }
    }
}

// x <- V diag(1/(lam - sigma)) V^-1 x (fast diagonalisation of the interior
// operator); vinvT / vT column-major with leading dimension ld.
template <typename TF, int NSLOT>
__device__ __forceinline__ void fdm_core(const TF* vinvT, const TF* vT, int ld, const TF* rdiag, int n,
                                         TF (&xr)[NSLOT], TF (&xi)[NSLOT], cplx_t<TF>* scr, int lane)
{
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) scr[lane + 32 * s] = mk(xr[s], xi[s]);
    __syncwarp();
    TF wr[NSLOT], wi[NSLOT];
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) { wr[s] = 0; wi[s] = 0; }
    for (int k = 0; k < n; ++k) {
        const cplx_t<TF> f = scr[k];
        const TF* col = vinvT + (size_t)k * ld;
#pragma unroll
        for (int s = 0; s < NSLOT; ++s) {
            const TF v = col[lane + 32 * s];
            wr[s] += v * f.x;
            wi[s] += v * f.y;
        }
    }
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
        const TF d = rdiag[lane + 32 * s];
        wr[s] *= d;
        wi[s] *= d;
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) scr[lane + 32 * s] = mk(wr[s], wi[s]);
    __syncwarp();
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) { xr[s] = 0; xi[s] = 0; }
    for (int k = 0; k < n; ++k) {
        const cplx_t<TF> w = scr[k];
        const TF* col = vT + (size_t)k * ld;
#pragma unroll
        for (int s = 0; s < NSLOT; ++s) {
            const TF v = col[lane + 32 * s];
            xr[s] += v * w.x;
            xi[s] += v * w.y;
        }
    }
    __syncwarp();
}

// Shared-memory layout of rows_kernel.
struct RowSmem {
    size_t mat, diag, perm, scr, d2, ns, total;
};
__host__ __device__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
template <typename TS, typename TF, int METHOD, bool REFINE>
__host__ __device__ inline RowSmem row_smem_layout(int n, int ld)
{
    RowSmem L{};
    size_t o = 0;
    L.mat = o;
    o += (size_t)(METHOD == 1 ? 1 : 2) * n * ld * sizeof(TF);
    o = align_up(o, 16);
    L.diag = o;                                   // LU: 1/U_ii ; FDM: 1/(lam - sigma) per warp
    o += (size_t)(METHOD == 1 ? 1 : ROW_WARPS) * ld * sizeof(TF);
    o = align_up(o, 16);
    L.perm = o;
    o += (size_t)ld * sizeof(int);
    o = align_up(o, 16);
    L.scr = o;  // per warp: 2 * ld values of the widest type, complex-interleaved
    o += (size_t)ROW_WARPS * ld * 2 * (sizeof(TS) > sizeof(TF) ? sizeof(TS) : sizeof(TF));
    o = align_up(o, 16);
    L.ns = o;   // per warp: Ns sweep scalars (rhs re/im, b, c, zl re/im)
    o += (size_t)ROW_WARPS * (ROW_NSMAX + 1) * 6 * sizeof(TS);
    o = align_up(o, 16);
    L.d2 = o;
    if (REFINE) o += (size_t)n * ld * sizeof(double);
    L.total = align_up(o, 16);
    return L;
}

template <typename TS, typename TF, int NSLOT, int METHOD, bool REFINE, bool ADJ = false>
__global__ void __launch_bounds__(ROW_WARPS * 32) rows_kernel(RowArgs a)
{
    pdl_enter();
    using CS = cplx_t<TS>;
    using CF = cplx_t<TF>;
    extern __shared__ __align__(16) unsigned char row_smem[];
    const int n = a.n, P = a.P, ld = a.ldf;
    const int Ns = METHOD == 2 ? 1 : a.Ns;  // FDM with several elements: multi_rows_kernel
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const RowSmem Lay = row_smem_layout<TS, TF, METHOD, REFINE>(n, ld);
    TF* sMat = reinterpret_cast<TF*>(row_smem + Lay.mat);
    TF* sDiag = reinterpret_cast<TF*>(row_smem + Lay.diag);
    int* sPerm = reinterpret_cast<int*>(row_smem + Lay.perm);
    unsigned char* scrRaw = row_smem + Lay.scr + (size_t)warp * ld * 2 * (sizeof(TS) > sizeof(TF) ? sizeof(TS) : sizeof(TF));
    TS* sNs = reinterpret_cast<TS*>(row_smem + Lay.ns) + (size_t)warp * (ROW_NSMAX + 1) * 6;
    double* sD2 = reinterpret_cast<double*>(row_smem + Lay.d2);

    // shared operator data: the FDM transforms once per CTA; refinement D2
    if (METHOD == 2) {
        const TF* vi = static_cast<const TF*>(a.vinvT);
        const TF* vv = static_cast<const TF*>(a.vT);
        for (int e = threadIdx.x; e < n * ld; e += blockDim.x) { sMat[e] = vi[e]; sMat[(size_t)n * ld + e] = vv[e]; }
    }
    if (REFINE)
        for (int e = threadIdx.x; e < n * ld; e += blockDim.x) sD2[e] = a.d2t[e];
    __syncthreads();

    const bool hom_active = a.hom != nullptr;
    CS* spec = static_cast<CS*>(a.spec);

    // one CTA per group (LU: its factor is staged once); FDM: grid-stride over groups
    for (int grp = blockIdx.x; grp < a.ngroups; grp += gridDim.x) {
        if (METHOD == 1) {
            __syncthreads();
            const TF* fsrc = static_cast<const TF*>(a.fac) + (size_t)grp * a.fac_stride;
            const TF* dsrc = static_cast<const TF*>(a.dinv) + (size_t)grp * ld;
            const uint8_t* psrc = a.perm + (size_t)grp * ld;
            for (int e = threadIdx.x; e < n * ld; e += blockDim.x) sMat[e] = fsrc[e];
            for (int e = threadIdx.x; e < ld; e += blockDim.x) { sDiag[e] = dsrc[e]; sPerm[e] = psrc[e]; }
            __syncthreads();
        }
        const double sig = a.sigma[grp];
        TF* rdiag = sDiag + (size_t)warp * ld;  // FDM: this warp's 1/(lam - sigma)
        if (METHOD == 2) {
            for (int j = lane; j < ld; j += 32) rdiag[j] = (j < n) ? (TF)(1.0 / (a.lam[j] - sig)) : (TF)0;
            __syncwarp();
        }
        const double* ul = hom_active ? a.hom + (size_t)grp * 2 * P : nullptr;
        const double* ur = hom_active ? ul + P : nullptr;
        double d0ul = 0, d0ur = 0, dNul = 0, dNur = 0;
        if (hom_active) {
            d0ul = a.homs[grp * 4 + 0]; d0ur = a.homs[grp * 4 + 1];
            dNul = a.homs[grp * 4 + 2]; dNur = a.homs[grp * 4 + 3];
        }
        // the interior collocation solve of one element (transposed in an
        // adjoint run), with the FP64-residual sweeps of a refined plan
        auto solve_interior = [&](const TS (&fr)[NSLOT], const TS (&fi)[NSLOT], TS (&xr)[NSLOT], TS (&xi)[NSLOT]) {
            TF yr[NSLOT], yi[NSLOT];
#pragma unroll
            for (int s = 0; s < NSLOT; ++s) { yr[s] = (TF)fr[s]; yi[s] = (TF)fi[s]; }
            if (METHOD == 1) lu_core<TF, NSLOT>(sMat, ld, sDiag, sPerm, n, yr, yi, reinterpret_cast<TF*>(scrRaw), lane);
            else fdm_core<TF, NSLOT>(sMat, sMat + (size_t)n * ld, ld, rdiag, n, yr, yi, reinterpret_cast<CF*>(scrRaw), lane);
#pragma unroll
            for (int s = 0; s < NSLOT; ++s) { xr[s] = (TS)yr[s]; xi[s] = (TS)yi[s]; }
            if (REFINE) {
                // FP64 residual r = f - (D2int x - sigma x), then a corrected FP32 solve
                CS* scr = reinterpret_cast<CS*>(scrRaw);
                for (int sw = 0; sw < a.sweeps; ++sw) {
                    __syncwarp();
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) scr[lane + 32 * s] = mk(xr[s], xi[s]);
                    __syncwarp();
                    TS rr_[NSLOT], ri_[NSLOT];
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        rr_[s] = fr[s] + (TS)sig * xr[s];
                        ri_[s] = fi[s] + (TS)sig * xi[s];
                    }
                    for (int k = 0; k < n; ++k) {
                        const CS xk = scr[k];
                        const double* col = sD2 + (size_t)k * ld;
#pragma unroll
                        for (int s = 0; s < NSLOT; ++s) {
                            const double d = col[lane + 32 * s];
                            rr_[s] -= d * xk.x;
                            ri_[s] -= d * xk.y;
                        }
                    }
                    __syncwarp();
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) { yr[s] = (TF)rr_[s]; yi[s] = (TF)ri_[s]; }
                    if (METHOD == 1) lu_core<TF, NSLOT>(sMat, ld, sDiag, sPerm, n, yr, yi, reinterpret_cast<TF*>(scrRaw), lane);
                    else fdm_core<TF, NSLOT>(sMat, sMat + (size_t)n * ld, ld, rdiag, n, yr, yi, reinterpret_cast<CF*>(scrRaw), lane);
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) { xr[s] += (TS)yr[s]; xi[s] += (TS)yi[s]; }
                }
            }
        };
        const int r0 = a.grp_start[grp], r1 = a.grp_start[grp + 1];
        for (int rr = r0 + warp; rr < r1; rr += ROW_WARPS) {
            const long long rowoff = (long long)a.grp_rows[rr] * P;
            TS pr = 0, pi = 0;                        // running d/dy of the previous element (Ns > 1)
            TS rhs_r = 0, rhs_i = 0, bprev = 0, cprev = 0;
            TS d0r = 0, d0i = 0, dNr = 0, dNi = 0;
            TS xr[NSLOT], xi[NSLOT];
            for (int jj = 0; jj < Ns; ++jj) {
                CS* row = spec + (long long)jj * a.elem_stride + rowoff;
                TS fr[NSLOT], fi[NSLOT];
#pragma unroll
                for (int s = 0; s < NSLOT; ++s) {
                    const int i = lane + 32 * s;
                    CS v = mk((TS)0, (TS)0);
                    if (i < n) v = row[1 + i];
                    fr[s] = v.x;
                    fi[s] = v.y;
                }
                // ---- collocation solve of the interior nodes ----
                solve_interior(fr, fi, xr, xi);
                if (ADJ) {
                    // transposed collocation system: boundary unknowns from the 2x2
                    // system, interior = psi + v0 pl + vN pr (one element)
                    TS a0r = 0, a0i = 0, aNr = 0, aNi = 0;
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) {
                            const TS c0 = (TS)a.d0[1 + i], cN = (TS)a.dN[1 + i];
                            a0r += c0 * xr[s]; a0i += c0 * xi[s];
                            aNr += cN * xr[s]; aNi += cN * xi[s];
                        }
                    }
                    a0r = warp_sum(a0r); a0i = warp_sum(a0i);
                    aNr = warp_sum(aNr); aNi = warp_sum(aNi);
                    const CS w0 = row[0], wN = row[P - 1];
                    const double* m = a.homs + grp * 4;
                    const TS m00 = (TS)m[0], m01 = (TS)m[1], m10 = (TS)m[2], m11 = (TS)m[3];
                    const TS q0r = w0.x - a0r, q0i = w0.y - a0i, qNr = wN.x - aNr, qNi = wN.y - aNi;
                    TS v0r, v0i, vNr, vNi;
                    if (a.periodic) {
                        // periodic: mu = (q0 + qN) / b with the forward b = (D0 - DN).(ul + ur)
                        const TS bb = (TS)((m[0] + m[1]) - (m[2] + m[3]));
                        v0r = (q0r + qNr) / bb; v0i = (q0i + qNi) / bb;
                        vNr = v0r; vNi = v0i;
                    } else {
                        const TS det = m00 * m11 - m01 * m10;
                        v0r = (m11 * q0r - m01 * qNr) / det; v0i = (m11 * q0i - m01 * qNi) / det;
                        vNr = (m00 * qNr - m10 * q0r) / det; vNi = (m00 * qNi - m10 * q0i) / det;
                    }
                    const double* pl = a.hom + (size_t)grp * 2 * P;
                    const double* pr_ = pl + P;
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) {
                            const TS l = (TS)pl[1 + i], r = (TS)pr_[1 + i];
                            row[1 + i] = mk(xr[s] + v0r * l + vNr * r, xi[s] + v0i * l + vNi * r);
                        }
                    }
                    if (lane == 0) { row[0] = mk(v0r, v0i); row[P - 1] = mk(vNr, vNi); }
                    continue;
                }
                if (!hom_active) {
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) row[1 + i] = mk(xr[s], xi[s]);
                    }
                    if (lane == 0) { row[0] = mk((TS)0, (TS)0); row[P - 1] = mk((TS)0, (TS)0); }
                    continue;
                }
                // ---- d/dy of the particular solution at both ends ----
                TS a0r = 0, a0i = 0, aNr = 0, aNi = 0;
#pragma unroll
                for (int s = 0; s < NSLOT; ++s) {
                    const int i = lane + 32 * s;
                    if (i < n) {
                        const TS c0 = (TS)a.d0[1 + i], cN = (TS)a.dN[1 + i];
                        a0r += c0 * xr[s]; a0i += c0 * xi[s];
                        aNr += cN * xr[s]; aNi += cN * xi[s];
                    }
                }
                d0r = warp_sum(a0r); d0i = warp_sum(a0i);
                dNr = warp_sum(aNr); dNi = warp_sum(aNi);
                if (a.periodic) {
                    // the cyclic sweep needs every element's end slopes first
                    if (Ns > 1) {
                        if (lane == 0) {
                            sNs[jj * 6 + 0] = d0r; sNs[jj * 6 + 1] = d0i;
                            sNs[jj * 6 + 2] = dNr; sNs[jj * 6 + 3] = dNi;
                        }
#pragma unroll
                        for (int s = 0; s < NSLOT; ++s) {
                            const int i = lane + 32 * s;
                            if (i < n) row[1 + i] = mk(xr[s], xi[s]);
                        }
                    }
                    continue;
                }
                // ---- forward sweep of the interface system ----
                TS bj, cj;
                if (jj == 0) {
                    bj = (TS)(-a.al * d0ul + a.bl);
                    cj = (TS)(-a.al * d0ur);
                    const CS gl = row[0];
                    rhs_r = gl.x + (TS)a.al * d0r;
                    rhs_i = gl.y + (TS)a.al * d0i;
                } else {
                    const TS q = (TS)dNul / bprev;
                    bj = (TS)dNur - (TS)d0ul - cprev * q;
                    cj = (TS)(-d0ur);
                    rhs_r = d0r - pr - rhs_r * q;
                    rhs_i = d0i - pi - rhs_i * q;
                }
                bprev = bj; cprev = cj; pr = dNr; pi = dNi;
                if (Ns > 1) {
                    if (lane == 0) {
                        sNs[jj * 6 + 0] = rhs_r; sNs[jj * 6 + 1] = rhs_i;
                        sNs[jj * 6 + 2] = bj;    sNs[jj * 6 + 3] = cj;
                    }
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {  // park phi of this element in place
                        const int i = lane + 32 * s;
                        if (i < n) row[1 + i] = mk(xr[s], xi[s]);
                    }
                }
            }
            if (ADJ || !hom_active) continue;
            if (a.periodic) {
                if (Ns == 1) {
                    // u(0) = u(L) = zeta, slopes equal (Periodic2D_MPI.cpp:262-266, 524-531)
                    const TS bb = (TS)((d0ul + d0ur) - (dNul + dNur));
                    const TS zr_ = (dNr - d0r) / bb, zi_ = (dNi - d0i) / bb;
                    CS* row = spec + rowoff;
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) {
                            const TS l = (TS)ul[1 + i], r = (TS)ur[1 + i];
                            row[1 + i] = mk(xr[s] + zr_ * l + zr_ * r, xi[s] + zi_ * l + zi_ * r);
                        }
                    }
                    if (lane == 0) { row[0] = mk(zr_, zi_); row[P - 1] = mk(zr_, zi_); }
                    continue;
                }
                // cyclic interface sweep with the rank-one correction (Periodic2D_MPI.cpp:
                // forward 268-293, backward 533-565): slot jj of sNs holds rhs0 (then
                // zeta_l) in [0, 1], b in [2], c in [3], rhs1 (then eta_l) in [4]
                __syncwarp();
                if (lane == 0) {
                    const TS D0ul = (TS)d0ul, D0ur = (TS)d0ur, DNul = (TS)dNul, DNur = (TS)dNur;
                    TS pNr = sNs[(Ns - 1) * 6 + 2], pNi = sNs[(Ns - 1) * 6 + 3];  // DN.phi of the element before
                    TS bp = 0, cp = 0, q0r = 0, q0i = 0, q1 = 0;
                    for (int jj = 0; jj < Ns; ++jj) {
                        const TS e0r = sNs[jj * 6 + 0], e0i = sNs[jj * 6 + 1];
                        const TS eNr = sNs[jj * 6 + 2], eNi = sNs[jj * 6 + 3];
                        TS bj, cj;
                        if (jj == 0) {
                            bj = DNur - DNul - D0ul;
                            cj = -D0ur;
                            q0r = e0r - pNr; q0i = e0i - pNi;
                            q1 = DNul;
                        } else {
                            q0r = e0r - pNr - (q0r / bp) * DNul;
                            q0i = e0i - pNi - (q0i / bp) * DNul;
                            if (jj < Ns - 1) {
                                bj = DNur - D0ul - (cp / bp) * DNul;
                                cj = -D0ur;
                                q1 = -(q1 / bp) * DNul;
                            } else {
                                bj = DNur - D0ul + D0ur - (cp / bp) * DNul;
                                cj = 0;
                                q1 = -D0ur - (q1 / bp) * DNul;
                            }
                        }
                        sNs[jj * 6 + 0] = q0r; sNs[jj * 6 + 1] = q0i;
                        sNs[jj * 6 + 2] = bj;  sNs[jj * 6 + 3] = cj;
                        sNs[jj * 6 + 4] = q1;
                        bp = bj; cp = cj; pNr = eNr; pNi = eNi;
                    }
                    // back sweep: zeta_r(jj) = zeta_l(jj + 1), eta likewise
                    TS zlr = q0r / bp, zli = q0i / bp, el = q1 / bp;
                    sNs[(Ns - 1) * 6 + 0] = zlr; sNs[(Ns - 1) * 6 + 1] = zli; sNs[(Ns - 1) * 6 + 4] = el;
                    const TS zlastr = zlr, zlasti = zli, elast = el;
                    for (int jj = Ns - 2; jj >= 0; --jj) {
                        const TS bj = sNs[jj * 6 + 2], cj = sNs[jj * 6 + 3];
                        zlr = (sNs[jj * 6 + 0] - cj * zlr) / bj;
                        zli = (sNs[jj * 6 + 1] - cj * zli) / bj;
                        el = (sNs[jj * 6 + 4] - cj * el) / bj;
                        sNs[jj * 6 + 0] = zlr; sNs[jj * 6 + 1] = zli; sNs[jj * 6 + 4] = el;
                    }
                    // alpha = -(zeta_l + zeta_r) / (1 + eta_l + eta_r) of the last element,
                    // whose right values are the first element's left ones
                    const TS den = (TS)1 + elast + el;
                    const TS alr = -(zlastr + zlr) / den, ali = -(zlasti + zli) / den;
                    for (int jj = 0; jj < Ns; ++jj) {
                        const TS e = sNs[jj * 6 + 4];
                        sNs[jj * 6 + 0] += alr * e;
                        sNs[jj * 6 + 1] += ali * e;
                    }
                }
                __syncwarp();
                for (int jj = 0; jj < Ns; ++jj) {
                    CS* row = spec + (long long)jj * a.elem_stride + rowoff;
                    const int jn = (jj + 1 == Ns) ? 0 : jj + 1;
                    const TS zl_r = sNs[jj * 6 + 0], zl_i = sNs[jj * 6 + 1];
                    const TS zrr = sNs[jn * 6 + 0], zri = sNs[jn * 6 + 1];
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) {
                            const CS x = row[1 + i];
                            const TS l = (TS)ul[1 + i], r = (TS)ur[1 + i];
                            row[1 + i] = mk(x.x + zl_r * l + zrr * r, x.y + zl_i * l + zri * r);
                        }
                    }
                    if (lane == 0) { row[0] = mk(zl_r, zl_i); row[P - 1] = mk(zrr, zri); }
                }
                __syncwarp();
                continue;
            }
            // ---- right end, back sweep, combination ----
            CS* lastrow = spec + (long long)(Ns - 1) * a.elem_stride + rowoff;
            const CS gr = lastrow[P - 1];
            const TS lb = (TS)(a.ar * dNul);
            const TS bR = (TS)(a.ar * dNur + a.br) - (cprev / bprev) * lb;
            const TS rRr = gr.x - (TS)a.ar * dNr - (rhs_r / bprev) * lb;
            const TS rRi = gr.y - (TS)a.ar * dNi - (rhs_i / bprev) * lb;
            TS zr_r = rRr / bR, zr_i = rRi / bR;
            if (Ns == 1) {
                const TS zl_r = (rhs_r - cprev * zr_r) / bprev, zl_i = (rhs_i - cprev * zr_i) / bprev;
                CS* row = spec + rowoff;
#pragma unroll
                for (int s = 0; s < NSLOT; ++s) {
                    const int i = lane + 32 * s;
                    if (i < n) {
                        const TS l = (TS)ul[1 + i], r = (TS)ur[1 + i];
                        row[1 + i] = mk(xr[s] + zl_r * l + zr_r * r, xi[s] + zl_i * l + zr_i * r);
                    }
                }
                if (lane == 0) { row[0] = mk(zl_r, zl_i); row[P - 1] = mk(zr_r, zr_i); }
            } else {
                __syncwarp();
                if (lane == 0) {
                    for (int jj = Ns - 1; jj >= 0; --jj) {
                        const TS rr_ = sNs[jj * 6 + 0], ri_ = sNs[jj * 6 + 1], bj = sNs[jj * 6 + 2], cj = sNs[jj * 6 + 3];
                        const TS zl_r = (rr_ - cj * zr_r) / bj, zl_i = (ri_ - cj * zr_i) / bj;
                        sNs[jj * 6 + 4] = zl_r; sNs[jj * 6 + 5] = zl_i;
                        sNs[(jj + 1) * 6 + 0] = zr_r; sNs[(jj + 1) * 6 + 1] = zr_i;  // zr of element jj
                        zr_r = zl_r; zr_i = zl_i;
                    }
                }
                __syncwarp();
                for (int jj = 0; jj < Ns; ++jj) {
                    CS* row = spec + (long long)jj * a.elem_stride + rowoff;
                    const TS zl_r = sNs[jj * 6 + 4], zl_i = sNs[jj * 6 + 5];
                    const TS zrr = sNs[(jj + 1) * 6 + 0], zri = sNs[(jj + 1) * 6 + 1];
#pragma unroll
                    for (int s = 0; s < NSLOT; ++s) {
                        const int i = lane + 32 * s;
                        if (i < n) {
                            const CS x = row[1 + i];
                            const TS l = (TS)ul[1 + i], r = (TS)ur[1 + i];
                            row[1 + i] = mk(x.x + zl_r * l + zrr * r, x.y + zl_i * l + zri * r);
                        }
                    }
                    if (lane == 0) { row[0] = mk(zl_r, zl_i); row[P - 1] = mk(zrr, zri); }
                }
                __syncwarp();
            }
        }
    }
}

template <typename TS, typename TF, int NSLOT, int METHOD, bool REFINE, bool ADJ = false>
static int run_rows(const RowArgs& a, cudaStream_t s)
{
    auto k = rows_kernel<TS, TF, NSLOT, METHOD, REFINE, ADJ>;
    const RowSmem L = row_smem_layout<TS, TF, METHOD, REFINE>(a.n, a.ldf);
    cudaError_t e = allow_smem(k, L.total, kMaxSmemPerBlock);
    if (e != cudaSuccess) return (int)e;
    int grid = a.ngroups;
    if (METHOD == 2) {
        static std::atomic<unsigned long long> memo{0};
        const long long resident = resident_ctas(k, ROW_WARPS * 32, L.total, memo);
        grid = (int)std::min<long long>(a.ngroups, resident);
    }
    if (grid <= 0) return 0;
    return (int)launch_k(k, dim3(grid), dim3(ROW_WARPS * 32), L.total, s, a);
}

template <int NSLOT>
static int rows_dispatch_prec(int method, int prec, const RowArgs& a, cudaStream_t s)
{
    if (method == 2 && a.Ns > 1) return (int)cudaErrorInvalidValue;  // launch_multi
    if (a.adjoint) {  // transposed solve: FDM
        if (method != 2) return (int)cudaErrorInvalidValue;
        if (prec == 0) return run_rows<double, double, NSLOT, 2, false, true>(a, s);
        if (prec == 1) return run_rows<float, float, NSLOT, 2, false, true>(a, s);
        return run_rows<double, float, NSLOT, 2, true, true>(a, s);
    }
    if (method == 1) {
        if (prec == 0) return run_rows<double, double, NSLOT, 1, false>(a, s);
        if (prec == 1) return run_rows<float, float, NSLOT, 1, false>(a, s);
        return run_rows<double, float, NSLOT, 1, true>(a, s);
    }
    if (prec == 0) return run_rows<double, double, NSLOT, 2, false>(a, s);
    if (prec == 1) return run_rows<float, float, NSLOT, 2, false>(a, s);
    return run_rows<double, float, NSLOT, 2, true>(a, s);
}

// Finite-difference variant (HypreFDM stencil, HelmholtzSolvers/HypreFDM/src/
// Helmholtz3D_MPI.cpp:387-403, periodic x and y turned into the modified
// wavenumbers mx, my): one Thomas solve along z per complex spectrum row, one
// thread per row.  The forward sweep writes the modified right-hand side in
// place and the elimination coefficients to `cprime`; the backward sweep reads
// both.  Consecutive threads take consecutive rows, so every step's loads fall
// on lines the previous step brought into L1.  That takes all of an SM's L1, so the
// kernel runs alone (launch_alone): with CTAs of the FFT passes before or after it
// resident, their shared memory is L1 that it lacks, and 32 x 32 x 600 points took
// 730 us instead of 287 (FP32, pipelined passes of 128 threads), 128 x 128 x 600 2400
// instead of 354 with the passes that the tuner picks.
template <typename T>
__global__ void __launch_bounds__(128) thomas_kernel(ThomasArgs a)
{
    using C = cplx_t<T>;
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nrows) return;
    const int Nz = a.Nz;
    const int kx = (int)(r / a.Ny), ky = (int)(r - (long long)kx * a.Ny);
    const double d = -2.0 * a.cz1 - a.lambda - a.mx[kx] - a.my[ky];
    C* x = static_cast<C*>(a.spec) + r * Nz;
    T* cp = static_cast<T*>(a.cprime) + r * Nz;
    const T cz = (T)a.cz1;
    // matrix entries of row k: sub a_k, diagonal b_k, super c_k (transposed: the
    // sub-diagonal of row k is the super-diagonal of row k-1 and vice versa)
    auto diag = [&](int k) -> T {
        double b = d;
        if (k == 0) b += a.d_first;
        if (k == Nz - 1) b += a.d_last;
        return (T)b;
    };
    auto sub = [&](int k) -> T {  // k >= 1
        if (!a.transpose) return (k == Nz - 1) ? (T)a.s_last : cz;
        return (k - 1 == 0) ? (T)a.s_first : cz;
    };
    auto sup = [&](int k) -> T {  // k <= Nz-2
        if (!a.transpose) return (k == 0) ? (T)a.s_first : cz;
        return (k + 1 == Nz - 1) ? (T)a.s_last : cz;
    };
    T cprev = 0;
    C dprev = mk((T)0, (T)0);
    for (int k = 0; k < Nz; ++k) {
        const T ak = (k > 0) ? sub(k) : (T)0;
        const T m = (T)1 / (diag(k) - ak * cprev);
        const T ck = (k < Nz - 1) ? sup(k) * m : (T)0;
        const C f = x[k];
        const C dk = mk((f.x - ak * dprev.x) * m, (f.y - ak * dprev.y) * m);
        x[k] = dk;
        cp[k] = ck;
        cprev = ck;
        dprev = dk;
    }
    C xn = dprev;
    for (int k = Nz - 2; k >= 0; --k) {
        const C dk = x[k];
        const T ck = cp[k];
        xn = mk(dk.x - ck * xn.x, dk.y - ck * xn.y);
        x[k] = xn;
    }
}

// The same tridiagonal solves, one warp per spectrum row (Nz <= 32 M).  Lane p
// owns rows z = p M .. p M + M - 1 (rows beyond Nz are identity rows).  The row
// is read once and written once, both coalesced through a per-warp shared
// buffer; no elimination coefficients go to memory:
//   1. each lane eliminates its interior rows (a Thomas solve of size M - 2
//      with three right-hand sides), leaving two equations that couple its
//      first and last unknowns to the neighbouring lanes' last and first ones;
//   2. the 64 reduced equations (a tridiagonal system in the order first_0,
//      last_0, first_1, ...) are solved by parallel cyclic reduction over warp
//      shuffles, six steps;
//   3. each lane recovers its interior unknowns from its first and last.
// The matrix is diagonally dominant (|diag| >= 2 cz1 + lambda + mx + my), so
// neither elimination pivots.
template <typename T>
struct TriEq {
    T a, b, c;
    cplx_t<T> d;
};

// Shuffles of a whole equation within segments of w lanes.
template <typename T>
__device__ __forceinline__ TriEq<T> tri_shfl_up(const TriEq<T>& e, int k, int w = 32)
{
    TriEq<T> o;
    o.a = __shfl_up_sync(0xffffffffu, e.a, k, w);
    o.b = __shfl_up_sync(0xffffffffu, e.b, k, w);
    o.c = __shfl_up_sync(0xffffffffu, e.c, k, w);
    o.d.x = __shfl_up_sync(0xffffffffu, e.d.x, k, w);
    o.d.y = __shfl_up_sync(0xffffffffu, e.d.y, k, w);
    return o;
}
template <typename T>
__device__ __forceinline__ TriEq<T> tri_shfl_down(const TriEq<T>& e, int k, int w = 32)
{
    TriEq<T> o;
    o.a = __shfl_down_sync(0xffffffffu, e.a, k, w);
    o.b = __shfl_down_sync(0xffffffffu, e.b, k, w);
    o.c = __shfl_down_sync(0xffffffffu, e.c, k, w);
    o.d.x = __shfl_down_sync(0xffffffffu, e.d.x, k, w);
    o.d.y = __shfl_down_sync(0xffffffffu, e.d.y, k, w);
    return o;
}
// One cyclic-reduction update of equation e with its neighbours lo (index - s)
// and hi (index + s), whose b fields hold the reciprocal of their diagonal.
template <typename T>
__device__ __forceinline__ TriEq<T> tri_reduce(const TriEq<T>& e, const TriEq<T>& lo, const TriEq<T>& hi)
{
    const T k1 = e.a * lo.b, k2 = e.c * hi.b;
    TriEq<T> o;
    o.a = -lo.a * k1;
    o.c = -hi.c * k2;
    o.b = e.b - lo.c * k1 - hi.a * k2;
    o.d = mk(e.d.x - lo.d.x * k1 - hi.d.x * k2, e.d.y - lo.d.y * k1 - hi.d.y * k2);
    return o;
}

constexpr int TRI_WARPS = 4;

// Copies row r of the spectrum into the lane-chunked buffer sb of LPR chunks
// of M (asynchronous, coalesced: step j moves elements 32 j .. 32 j + 31);
// elements >= Nz, and every element of a row past the end (live = false), read 0.
template <typename T, int M, int LPR>
__device__ __forceinline__ void tri_issue_row(const ThomasArgs& a, long long r, bool live, cplx_t<T>* sb, int lane)
{
    using C = cplx_t<T>;
    const C* x = static_cast<const C*>(a.spec) + (live ? r : 0) * a.Nz;
#pragma unroll
    for (int j = 0; j < (LPR * M + 31) / 32; ++j) {
        const int e = j * 32 + lane;
        const bool ok = live && e < a.Nz;
        cp_async_elem<sizeof(C)>(&sb[(e / M) * (M + 1) + e % M], ok ? (const void*)&x[e] : a.spec, ok);
    }
}

// LPR = 16: each half-warp solves its own row (two rows per warp, 16 chunks of
// M per row, cyclic reduction over 16-lane segments: one step and half the
// shuffles fewer per row than LPR = 32).
template <typename T, int M, int LPR = 32>
__global__ void __launch_bounds__(TRI_WARPS * 32, (M <= 8 ? 4 : (sizeof(T) == 8 ? 2 : 3))) thomas_warp_kernel(ThomasArgs a)
{
    pdl_enter();
    using C = cplx_t<T>;
    constexpr int RPW = 32 / LPR;            // rows per warp
    constexpr int RB = LPR * (M + 1);        // one row's buffer
    extern __shared__ __align__(16) unsigned char tri_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int li = lane % LPR, hrow = lane / LPR;  // lane within its row, row within the warp
    C* bufs = reinterpret_cast<C*>(tri_smem) + (size_t)warp * 2 * RPW * RB;
    const int Nz = a.Nz;
    const T cz = (T)a.cz1;
    const TriEq<T> ident{(T)0, (T)1, (T)0, mk((T)0, (T)0)};
    const long long stride = (long long)gridDim.x * TRI_WARPS * RPW;
    long long r0 = ((long long)blockIdx.x * TRI_WARPS + warp) * RPW;  // first row of the warp
    int cur = 0;
    if (r0 < a.nrows)
        for (int hh = 0; hh < RPW; ++hh) tri_issue_row<T, M, LPR>(a, r0 + hh, r0 + hh < a.nrows, bufs + hh * RB, lane);
    cp_async_commit();
    for (; r0 < a.nrows; r0 += stride, cur ^= 1) {
        C* sbw = bufs + (size_t)cur * RPW * RB;
        if (r0 + stride < a.nrows)
            for (int hh = 0; hh < RPW; ++hh)
                tri_issue_row<T, M, LPR>(a, r0 + stride + hh, r0 + stride + hh < a.nrows,
                                         bufs + (size_t)(cur ^ 1) * RPW * RB + hh * RB, lane);
        cp_async_commit();
        cp_async_wait_prev();
        __syncwarp();
        C* sb = sbw + hrow * RB;  // this lane's row
        const long long r = min(r0 + hrow, a.nrows - 1);  // rows past the end solve zeros, unstored
        const int kx = (int)(r / a.Ny), ky = (int)(r - (long long)kx * a.Ny);
        const double dg = -2.0 * a.cz1 - a.lambda - a.mx[kx] - a.my[ky];
        // the lane's chunk is read from the staging buffer where it is used
        // (no register copy: registers for the elimination's arrays)
        const C* dv = sb + li * (M + 1);
        // row k: sub (k >= 1), diagonal, super (k <= Nz - 2); transposed, the sub of
        // row k is the super of row k - 1 and the super of row k the sub of row k + 1.
        // Rows k >= Nz are identity rows.
        auto sub = [&](int k) -> T {
            if (k == 0 || k >= Nz) return (T)0;
            if (!a.transpose) return (k == Nz - 1) ? (T)a.s_last : cz;
            return (k == 1) ? (T)a.s_first : cz;
        };
        auto sup = [&](int k) -> T {
            if (k >= Nz - 1) return (T)0;
            if (!a.transpose) return (k == 0) ? (T)a.s_first : cz;
            return (k + 2 == Nz) ? (T)a.s_last : cz;
        };
        auto dia = [&](int k) -> T {
            if (k >= Nz) return (T)1;
            double b = dg;
            if (k == 0) b += a.d_first;
            if (k == Nz - 1) b += a.d_last;
            return (T)b;
        };
        const int k0 = li * M, last = Nz - 1 - k0;  // the last row's place in the chunk
        // ---- 1. eliminate the lane's interior rows ----
        TriEq<T> e0, e1;
        C y[M > 2 ? M - 2 : 1];
        T v[M > 2 ? M - 2 : 1], w[M > 2 ? M - 2 : 1];
        if constexpr (M == 2) {
            e0 = TriEq<T>{sub(k0), dia(k0), sup(k0), dv[0]};
            e1 = TriEq<T>{sub(k0 + 1), dia(k0 + 1), sup(k0 + 1), dv[1]};
        } else {
            constexpr int NI = M - 2;
            T cp[NI];
            // Rows k0 + 1 .. k0 + M - 2 (never the first): cz dg cz, but for the last
            // row and its neighbour, the identity rows past it, and row 1 of the
            // transposed matrix.  A warp whose lanes all lie inside takes the
            // constants as they stand: 1024 x 1024 modes of 256 points, FP64, 1029 ->
            // 880 us (transposed 958), 512 x 512 of 128 152 -> 124 us; chunks that
            // the row ends in, 256 x 128 of 100, FP32 21.4 -> 19.3 us.
            const T dgT = (T)dg, dlast = (T)(dg + a.d_last);
            const T sub1 = (a.transpose && k0 == 0) ? (T)a.s_first : cz;
            const T sublast = a.transpose ? cz : (T)a.s_last, suplast = a.transpose ? (T)a.s_last : cz;
            auto eliminate = [&](auto inside) {
                constexpr bool IN = decltype(inside)::value;
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    const int jj = j + 1;
                    T al = jj == 1 ? sub1 : cz, b = dgT, c = cz;
                    if (!IN) {
                        if (jj == last && !a.transpose) al = sublast;
                        al = jj > last ? (T)0 : al;
                        b = jj < last ? dgT : jj == last ? dlast : (T)1;
                        c = jj + 1 < last ? cz : jj + 1 == last ? suplast : (T)0;
                    }
                    const T m = (T)1 / ((j > 0) ? b - al * cp[j > 0 ? j - 1 : 0] : b);
                    cp[j] = (j < NI - 1) ? c * m : (T)0;
                    if (j == 0) {
                        y[0] = mk(dv[1].x * m, dv[1].y * m);
                        v[0] = al * m;
                        w[0] = NI == 1 ? c * m : (T)0;
                    } else {
                        const C yp = y[j > 0 ? j - 1 : 0];
                        y[j] = mk((dv[jj].x - al * yp.x) * m, (dv[jj].y - al * yp.y) * m);
                        v[j] = -(al * v[j > 0 ? j - 1 : 0]) * m;
                        w[j] = (j == NI - 1) ? c * m : (T)0;
                    }
                }
            };
            if (__all_sync(0xffffffffu, last >= M - (a.transpose ? 0 : 1))) eliminate(std::true_type{});
            else eliminate(std::false_type{});
#pragma unroll
            for (int j = NI - 2; j >= 0; --j) {
                y[j] = mk(y[j].x - cp[j] * y[j + 1].x, y[j].y - cp[j] * y[j + 1].y);
                v[j] -= cp[j] * v[j + 1];
                w[j] -= cp[j] * w[j + 1];
            }
            const T c0 = sup(k0), aM = sub(k0 + M - 1);
            e0 = TriEq<T>{sub(k0), dia(k0) - c0 * v[0], -c0 * w[0],
                          mk(dv[0].x - c0 * y[0].x, dv[0].y - c0 * y[0].y)};
            e1 = TriEq<T>{-aM * v[NI - 1], dia(k0 + M - 1) - aM * w[NI - 1], sup(k0 + M - 1),
                          mk(dv[M - 1].x - aM * y[NI - 1].x, dv[M - 1].y - aM * y[NI - 1].y)};
        }
        // ---- 2. cyclic reduction of the 2 LPR reduced equations (2 li, 2 li + 1) ----
        {
            // stride 1: e0's lower neighbour is lane - 1's e1, e1's upper one lane + 1's e0
            const TriEq<T> q0{e0.a, (T)1 / e0.b, e0.c, e0.d}, q1{e1.a, (T)1 / e1.b, e1.c, e1.d};
            TriEq<T> lo = tri_shfl_up(q1, 1, LPR), hi = tri_shfl_down(q0, 1, LPR);
            if (li == 0) lo = ident;
            if (li == LPR - 1) hi = ident;
            const TriEq<T> n0 = tri_reduce(e0, lo, q1);
            const TriEq<T> n1 = tri_reduce(e1, q0, hi);
            e0 = n0;
            e1 = n1;
        }
#pragma unroll
        for (int k = 1; k < LPR; k <<= 1) {  // strides 2, 4, .., 2 LPR of the reduced index
            const TriEq<T> q0{e0.a, (T)1 / e0.b, e0.c, e0.d}, q1{e1.a, (T)1 / e1.b, e1.c, e1.d};
            TriEq<T> l0 = tri_shfl_up(q0, k, LPR), h0 = tri_shfl_down(q0, k, LPR);
            TriEq<T> l1 = tri_shfl_up(q1, k, LPR), h1 = tri_shfl_down(q1, k, LPR);
            if (li < k) { l0 = ident; l1 = ident; }
            if (li + k > LPR - 1) { h0 = ident; h1 = ident; }
            const TriEq<T> n0 = tri_reduce(e0, l0, h0);
            const TriEq<T> n1 = tri_reduce(e1, l1, h1);
            e0 = n0;
            e1 = n1;
        }
        const C xs = mk(e0.d.x / e0.b, e0.d.y / e0.b);
        const C xe = mk(e1.d.x / e1.b, e1.d.y / e1.b);
        // ---- 3. interior unknowns, coalesced store ----
        __syncwarp();
        sb[li * (M + 1)] = xs;
        sb[li * (M + 1) + M - 1] = xe;
        if constexpr (M > 2) {
#pragma unroll
            for (int j = 0; j < M - 2; ++j)
                sb[li * (M + 1) + j + 1] =
                    mk(y[j].x - xs.x * v[j] - xe.x * w[j], y[j].y - xs.y * v[j] - xe.y * w[j]);
        }
        __syncwarp();
        for (int hh = 0; hh < RPW; ++hh) {
            if (r0 + hh >= a.nrows) break;
            C* x = static_cast<C*>(a.spec) + (r0 + hh) * Nz;
            const C* sr = sbw + hh * RB;
#pragma unroll
            for (int j = 0; j < (LPR * M + 31) / 32; ++j) {
                const int e = j * 32 + lane;
                if (e < Nz) x[e] = sr[(e / M) * (M + 1) + e % M];
            }
        }
        __syncwarp();  // the buffers are refilled by the copies issued in the next iteration
    }
    asm volatile("cp.async.wait_all;\n" ::);
}

template <typename T, int M, int LPR = 32>
static int run_thomas_warp(const ThomasArgs& a, cudaStream_t s)
{
    auto k = thomas_warp_kernel<T, M, LPR>;
    const size_t smem = (size_t)TRI_WARPS * 2 * (32 / LPR) * LPR * (M + 1) * sizeof(cplx_t<T>);
    cudaError_t e = allow_smem(k, smem);
    if (e != cudaSuccess) return (int)e;
    static std::atomic<unsigned long long> memo{0};
    const long long resident = resident_ctas(k, TRI_WARPS * 32, smem, memo);
    const long long rows_per_cta = (long long)TRI_WARPS * (32 / LPR);
    long long grid = (a.nrows + rows_per_cta - 1) / rows_per_cta;
    if (grid > resident) grid = resident;
    if (grid <= 0) return 0;
    return (int)launch_k(k, dim3((unsigned)grid), dim3(TRI_WARPS * 32), smem, s, a);
}

template <typename T>
static int thomas_dispatch(const ThomasArgs& a, cudaStream_t s)
{
    if (a.half) {  // a row per half-warp
        if (a.Nz <= 32) return run_thomas_warp<T, 2, 16>(a, s);
        if (a.Nz <= 64) return run_thomas_warp<T, 4, 16>(a, s);
        if (a.Nz <= 128) return run_thomas_warp<T, 8, 16>(a, s);
        if (a.Nz <= 256) return run_thomas_warp<T, 16, 16>(a, s);
    }
    if (a.Nz <= 64) return run_thomas_warp<T, 2>(a, s);
    if (a.Nz <= 128) return run_thomas_warp<T, 4>(a, s);
    if (a.Nz <= 256) return run_thomas_warp<T, 8>(a, s);
    if (a.Nz <= 512) return run_thomas_warp<T, 16>(a, s);
    const long long blocks = (a.nrows + 127) / 128;
    if (blocks <= 0) return 0;
    return (int)launch_alone(thomas_kernel<T>, dim3((unsigned)blocks), dim3(128), 0, s, a);
}

int launch_thomas(int prec, const ThomasArgs& a, cudaStream_t s)
{
    return prec == 1 ? thomas_dispatch<float>(a, s) : thomas_dispatch<double>(a, s);
}

size_t rows_smem_bytes(int method, int prec, int n, int ld)
{
    if (method == 1) {
        if (prec == 0) return row_smem_layout<double, double, 1, false>(n, ld).total;
        if (prec == 1) return row_smem_layout<float, float, 1, false>(n, ld).total;
        return row_smem_layout<double, float, 1, true>(n, ld).total;
    }
    if (prec == 0) return row_smem_layout<double, double, 2, false>(n, ld).total;
    if (prec == 1) return row_smem_layout<float, float, 2, false>(n, ld).total;
    return row_smem_layout<double, float, 2, true>(n, ld).total;
}

int launch_rows(int method, int prec, const RowArgs& a, cudaStream_t s)
{
    if (a.Ns > ROW_NSMAX) return (int)cudaErrorInvalidValue;
    switch ((a.n + 31) / 32) {
        case 1: return rows_dispatch_prec<1>(method, prec, a, s);
        case 2: return rows_dispatch_prec<2>(method, prec, a, s);
        case 3: return rows_dispatch_prec<3>(method, prec, a, s);
        case 4: return rows_dispatch_prec<4>(method, prec, a, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

}  // namespace helm
