// Row solves of plans with several GLL elements (Ns > 1), fast-diagonalisation
// method, sm_100a.
//
// Per spectrum row the reference solves the interior collocation system of every
// element (ConstructFundamentalSolutions + LUSolve, NonPeriodic2D_MPI.cpp:176-223),
// then a tridiagonal system for the Ns + 1 interface values whose right-hand side
// is the jump of the element solutions' end slopes (:265-295, 414-424), then
// combines u = phi + zl ul + zr ur (:466-470); the periodic solvers close the
// chain (Periodic2D_MPI.cpp:268-293, 533-565).  Only the interface system couples
// the elements, and its matrix depends on the shift alone.  So here one CTA owns a
// few whole rows, all their elements in shared memory, and runs
//   1. the interior solves of all its (row, element) vectors side by side:
//      phi = V diag(1 / (lam - sigma)) V^-1 f as two products on the FP64 tensor
//      cores (m8n8k4), four complex vectors per warp (elements of up to 34 points;
//      longer ones: all warps on each vector, multi_solve_wide); the first
//      product's results are the second one's A operand as they stand, the order
//      of its k index being put into the B fragments; the second product has two
//      more output rows, D0 V and DN V, which give the end slopes;
//   2. the interface sweep, one row per warp, real and imaginary part on a lane
//      each: the pivots come from the plan, so a step is one multiply-add;
//   3. the combination and one coalesced store.
// The adjoint runs the transposes in the order dots, sweep, solves.
//
// Bound: latency.  The vectors are short (8 interior points and 52 elements in the
// stock 2D problem, 4.3 MB in all), so what counts is that no step of one element
// waits for another element's.  One warp walking the elements of a row in turn
// (rows_kernel, which the LU method keeps) took 84.4 us for the 257 rows of 52 x 10
// points and 96.3 us for 1056 rows of 25 x 10 (periodic); this kernel 14.8 and
// 14.5 us (the stage between events, as are the other stage times in these files).
#include "helm_device.cuh"
#include "helm_kernels.cuh"
#include "helm_multi.cuh"

namespace helm {

namespace {

struct MultiSmem {
    size_t x, y, rec, piv, mul, z, sl, total;
};

// Elements of more than this many interior points take multi_solve_wide.
constexpr int MULTI_WARP_N = 32;
// Vectors of one round of multi_solve_wide: four m-tiles (four complex vectors
// each) share every B fragment that a warp loads.
constexpr int MULTI_WIDE = 16;

// Doubles between the rows of multi_solve_wide's intermediate (8 mod 16: the
// double2 reads of an A fragment, eight rows by four, touch every bank twice).
__host__ __device__ inline int multi_wide_stride(int n)
{
    const int kp = (n + 7) / 8 * 8;
    return kp & 8 ? kp : kp + 8;
}

template <typename TS>
__host__ __device__ inline MultiSmem multi_smem(int R, int Ns, int P, int n)
{
    MultiSmem L{};
    size_t o = 0;
    const size_t nv = (size_t)R * Ns, kp = (n + 7) / 8 * 8;
    L.x = o;
    o += (nv * P * 2 * sizeof(TS) + 15) / 16 * 16;
    L.y = o;                                     // first product's results (multi_solve_wide)
    if (n > MULTI_WARP_N) {
        const size_t v = nv < MULTI_WIDE ? (nv + 3) / 4 * 4 : MULTI_WIDE;
        o += v * 2 * multi_wide_stride(n) * sizeof(double);
    }
    L.rec = o;                                   // 1 / (lam - sigma) of each row
    o += R * kp * sizeof(double);
    L.z = o;                                     // right-hand sides, then interface values
    o += (size_t)R * (Ns + 1) * 2 * sizeof(double);
    L.sl = o;                                    // end slopes (forward) / end dots (adjoint) of each vector
    o += nv * 4 * sizeof(double);
    L.piv = o;                                   // reciprocal pivots
    o += (size_t)R * (Ns + 1) * sizeof(double);
    L.mul = o;                                   // elimination multipliers
    o += (size_t)R * (Ns + 1) * sizeof(double);
    L.total = o;
    return L;
}

// The interior solves of the four complex vectors v0 .. v0 + 3 by one warp.
// NT: n in tiles of 8 (upper bound, nt the actual count); SLOPES: the second
// product's rows n and n + 1 go to sl.
template <typename TS, int NT, bool SLOPES>
__device__ __forceinline__ void multi_solve4(const MultiArgs& a, TS* x, const double* rec, double* sl, int v0, int nv,
                                             int R, int lane)
{
    constexpr int NO = NT + (SLOPES ? 1 : 0);
    const int g = lane >> 2, q = lane & 3;
    const int n = a.n, nt = (n + 7) >> 3, kp = nt * 8;
    const int no = SLOPES ? (n + 9) >> 3 : nt;
    const int v = v0 + (g >> 1);
    const bool live = v < nv;
    TS* row = x + ((size_t)(live ? v : 0) * a.P + 1) * 2 + (g & 1);  // this lane's vector, real or imaginary part
    double c[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) c[t][0] = c[t][1] = 0.0;
    for (int kk = 0; kk < 2 * nt; ++kk) {
        const int k = 4 * kk + q;
        const double av = (live && k < n) ? (double)row[2 * k] : 0.0;
        const double* b = a.m1 + (size_t)kk * 32 + lane;
#pragma unroll
        for (int t = 0; t < NT; ++t)
            if (t < nt) dmma_8x8x4(c[t][0], c[t][1], av, __ldg(b + (size_t)t * 2 * nt * 32));
    }
    const double* rc = rec + (size_t)(live ? v % R : 0) * kp + 2 * q;
#pragma unroll
    for (int t = 0; t < NT; ++t)
        if (t < nt) {
            c[t][0] *= rc[8 * t];
            c[t][1] *= rc[8 * t + 1];
        }
    double o[NO][2];
#pragma unroll
    for (int t = 0; t < NO; ++t) o[t][0] = o[t][1] = 0.0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        if (t >= nt) break;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const double* b = a.m2 + (size_t)(2 * t + s) * 32 + lane;
#pragma unroll
            for (int i = 0; i < NO; ++i)
                if (i < no) dmma_8x8x4(o[i][0], o[i][1], c[t][s], __ldg(b + (size_t)i * 2 * nt * 32));
        }
    }
    __syncwarp();
    if (!live) return;
#pragma unroll
    for (int t = 0; t < NO; ++t)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int i = 8 * t + 2 * q + s;
            if (i < n) row[2 * i] = (TS)o[t][s];
            else if (SLOPES && i < n + 2) sl[(size_t)v * 4 + 2 * (i - n) + (g & 1)] = o[t][s];
        }
}

// The interior solves of all of a CTA's vectors by all of its warps, for elements of
// more than MULTI_WARP_N points: a warp takes one n-tile of a product (8 of the n
// columns) for MULTI_WIDE vectors at a time, so it carries 8 accumulators a lane
// whatever n is, every B fragment serves four m-tiles, and the few vectors of a short
// grid still occupy all warps.  The first product's results pass through y, the
// solutions go over the right-hand sides in x.  With whole-row accumulators
// (multi_solve4 at 8 and 16 tiles) these sizes spilled 250 bytes to 4.8 KB a thread
// and one warp walked 40 to 180 KB of fragments by itself: FP64 solves of 256 Fourier
// points by 2 x 67 took 53.5 us and by 6 x 103 113, walking the elements in turn 29.6
// and 71.6; with this 20.4 and 28.7.
template <typename TS, bool SLOPES>
__device__ __forceinline__ void multi_solve_wide(const MultiArgs& a, TS* x, const double* rec, double* sl, double* y,
                                                 int nv, int R, int lane, int warp, int nwarp)
{
    constexpr int G = MULTI_WIDE / 4;
    const int g = lane >> 2, q = lane & 3;
    const int n = a.n, nt = (n + 7) >> 3, kp = nt * 8, ys = multi_wide_stride(n);
    const int no = SLOPES ? (n + 9) >> 3 : nt;
    for (int c0 = 0; c0 < nv; c0 += MULTI_WIDE) {
        const int groups = min(G, (nv - c0 + 3) >> 2);
        // this lane's vector of each group, real or imaginary part (rows past the end: the first vector's, unused)
        const TS* row[G];
        bool live[G];
#pragma unroll
        for (int i = 0; i < G; ++i) {
            const int v = c0 + 4 * i + (g >> 1);
            live[i] = v < nv;
            row[i] = x + ((size_t)(live[i] ? v : 0) * a.P + 1) * 2 + (g & 1);
        }
        for (int t = warp; t < nt; t += nwarp) {
            const double* b = a.m1 + (size_t)t * 2 * nt * 32 + lane;
            double c[G][2];
#pragma unroll
            for (int i = 0; i < G; ++i) c[i][0] = c[i][1] = 0.0;
#pragma unroll 4
            for (int kk = 0; kk < 2 * nt; ++kk) {
                const double bv = __ldg(b + kk * 32);
                const int k = 4 * kk + q;
#pragma unroll
                for (int i = 0; i < G; ++i)
                    if (i < groups) dmma_8x8x4(c[i][0], c[i][1], (live[i] && k < n) ? (double)row[i][2 * k] : 0.0, bv);
            }
#pragma unroll
            for (int i = 0; i < G; ++i)
                if (i < groups) {
                    const double* rc = rec + (size_t)(live[i] ? (c0 + 4 * i + (g >> 1)) % R : 0) * kp + 8 * t + 2 * q;
                    *reinterpret_cast<double2*>(y + (size_t)(8 * i + g) * ys + 8 * t + 2 * q) =
                        make_double2(c[i][0] * rc[0], c[i][1] * rc[1]);
                }
        }
        __syncthreads();
        for (int t = warp; t < no; t += nwarp) {
            const double* b = a.m2 + (size_t)t * 2 * nt * 32 + lane;
            double o[G][2];
#pragma unroll
            for (int i = 0; i < G; ++i) o[i][0] = o[i][1] = 0.0;
#pragma unroll 2
            for (int kt = 0; kt < nt; ++kt) {
                const double b0 = __ldg(b + (size_t)kt * 64), b1 = __ldg(b + (size_t)kt * 64 + 32);
#pragma unroll
                for (int i = 0; i < G; ++i)
                    if (i < groups) {
                        const double2 av = *reinterpret_cast<const double2*>(y + (size_t)(8 * i + g) * ys + 8 * kt + 2 * q);
                        dmma_8x8x4(o[i][0], o[i][1], av.x, b0);
                        dmma_8x8x4(o[i][0], o[i][1], av.y, b1);
                    }
            }
#pragma unroll
            for (int i = 0; i < G; ++i) {
                if (!live[i]) continue;
                const int v = c0 + 4 * i + (g >> 1);
                TS* out = x + ((size_t)v * a.P + 1) * 2 + (g & 1);
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    const int j = 8 * t + 2 * q + s;
                    if (j < n) out[2 * j] = (TS)o[i][s];
                    else if (SLOPES && j < n + 2) sl[(size_t)v * 4 + 2 * (j - n) + (g & 1)] = o[i][s];
                }
            }
        }
        __syncthreads();  // y is overwritten by the next round
    }
}

// NT: tiles of 8 interior points a warp's accumulators hold (multi_solve4); 0: multi_solve_wide.
template <typename TS, int NT, bool ADJ>
__global__ void __launch_bounds__(256) multi_rows_kernel(MultiArgs a)
{
    extern __shared__ __align__(16) unsigned char multi_raw[];
    const int P = a.P, n = a.n, Ns = a.Ns, R = a.rows_per_cta, kp = (n + 7) / 8 * 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const MultiSmem L = multi_smem<TS>(R, Ns, P, n);
    TS* x = reinterpret_cast<TS*>(multi_raw + L.x);  // vector v = element * R + row
    double* y = reinterpret_cast<double*>(multi_raw + L.y);
    double* rec = reinterpret_cast<double*>(multi_raw + L.rec);
    double* z = reinterpret_cast<double*>(multi_raw + L.z);
    double* sl = reinterpret_cast<double*>(multi_raw + L.sl);
    double* piv = reinterpret_cast<double*>(multi_raw + L.piv);
    double* mul = reinterpret_cast<double*>(multi_raw + L.mul);
    const int r0 = blockIdx.x * R;
    const int nr = min(R, a.nrows - r0), nv = R * Ns, M = Ns + 1;
    const int itf = a.periodic ? 2 * M : M;

    // plan data, before the previous kernel's results are waited for
    for (int e = threadIdx.x; e < R * kp; e += blockDim.x) {
        const int r = e / kp, j = e - r * kp;
        rec[e] = (r < nr && j < n) ? 1.0 / (a.lam[j] - a.sigma[a.grp_of_row[r0 + r]]) : 0.0;
    }
    for (int e = threadIdx.x; e < R * M; e += blockDim.x) {
        const int r = e / M, j = e - r * M;
        double p = 0.0, m = 0.0;
        if (r < nr) {
            const int grp = a.grp_of_row[r0 + r];
            const double* f = a.itf + (size_t)grp * itf;
            p = f[j];
            // T[j][j-1] / b_{j-1}: the multiplier of the forward elimination
            if (j > 0) m = ((j == Ns && !a.periodic) ? a.ar : 1.0) * a.homs[grp * 4 + 2] * f[j - 1];
        }
        piv[e] = p;
        mul[e] = m;
    }
    pdl_enter();
    using C = cplx_t<TS>;
    C* spec = static_cast<C*>(a.spec) + (long long)r0 * P;
    C* xc = reinterpret_cast<C*>(x);
    const int seg = R * P, live = nr * P;  // one element's rows are one contiguous run
    for (int e = threadIdx.x; e < nv * P; e += blockDim.x) {
        const int j = e / seg, i = e - j * seg;
        const bool ok = i < live;
        cp_async_elem<sizeof(C)>(&xc[e], ok ? (const void*)&spec[(long long)j * a.elem_stride + i] : a.spec, ok);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();

    auto interior_solves = [&]() {
        if constexpr (NT == 0) {
            multi_solve_wide<TS, !ADJ>(a, x, rec, sl, y, nv, R, lane, warp, nwarp);
        } else {
            for (int v0 = 4 * warp; v0 < nv; v0 += 4 * nwarp)
                multi_solve4<TS, NT, !ADJ>(a, x, rec, sl, v0, nv, R, lane);
            __syncthreads();
        }
    };

    if constexpr (!ADJ) {
        interior_solves();
        for (int r = warp; r < nr; r += nwarp) {
            const int grp = a.grp_of_row[r0 + r];
            const double d0ur = a.homs[grp * 4 + 1];
            double* zr = z + (size_t)r * M * 2;
            const double* pv = piv + (size_t)r * M;
            const double* mv = mul + (size_t)r * M;
            // right-hand sides: jumps of the end slopes, the Robin data at the ends
            for (int e = lane; e < 2 * M; e += 32) {
                const int j = e >> 1, c = e & 1;
                double h;
                if (a.periodic) {
                    const int jp = j == 0 ? Ns - 1 : j - 1;
                    h = j < Ns ? sl[((size_t)j * R + r) * 4 + c] - sl[((size_t)jp * R + r) * 4 + 2 + c] : 0.0;
                } else if (j == 0) {
                    h = (double)x[((size_t)r * P) * 2 + c] + a.al * sl[(size_t)r * 4 + c];
                } else if (j == Ns) {
                    const size_t v = (size_t)(Ns - 1) * R + r;
                    h = (double)x[(v * P + P - 1) * 2 + c] - a.ar * sl[v * 4 + 2 + c];
                } else {
                    h = sl[((size_t)j * R + r) * 4 + c] - sl[((size_t)(j - 1) * R + r) * 4 + 2 + c];
                }
                zr[e] = h;
            }
            __syncwarp();
            if (lane < 2) {
                const int last = a.periodic ? Ns - 1 : Ns;
                double y = zr[lane];
#pragma unroll 4
                for (int j = 1; j <= last; ++j) {
                    y = zr[2 * j + lane] - mv[j] * y;
                    zr[2 * j + lane] = y;
                }
                y *= pv[last];
                zr[2 * last + lane] = y;
                // super-diagonal: -D0.ur, times alpha in the first row
#pragma unroll 4
                for (int j = last - 1; j >= 0; --j) {
                    const double c = ((j == 0 && !a.periodic) ? a.al : 1.0) * d0ur * pv[j];
                    y = zr[2 * j + lane] * pv[j] + c * y;
                    zr[2 * j + lane] = y;
                }
                if (a.periodic) {
                    // rank-one correction: zeta += alpha eta, the last element's right value the first one's left
                    const double* eta = a.itf + (size_t)grp * itf + M;
                    const double alpha = (zr[2 * (Ns - 1) + lane] + zr[lane]) * eta[Ns];
                    for (int j = 0; j < Ns; ++j) zr[2 * j + lane] += alpha * eta[j];
                    zr[2 * Ns + lane] = zr[lane];
                }
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nv * P; e += blockDim.x) {
            const int j = e / seg, i = e - j * seg;
            if (i >= live) continue;
            const int r = i / P, k = i - r * P;
            const double* h = a.hom + (size_t)a.grp_of_row[r0 + r] * 2 * P + k;
            const double* zz = z + ((size_t)r * M + j) * 2;
            const double l = h[0], rr = h[P];
            C u;
            if (k == 0) u = mk((TS)zz[0], (TS)zz[1]);
            else if (k == P - 1) u = mk((TS)zz[2], (TS)zz[3]);
            else
                u = mk((TS)((double)x[2 * (size_t)e] + zz[0] * l + zz[2] * rr),
                       (TS)((double)x[2 * (size_t)e + 1] + zz[1] * l + zz[3] * rr));
            spec[(long long)j * a.elem_stride + i] = u;
        }
    } else {
        // the transposed map (several elements, not periodic): zbar_j = ubar at the
        // nodes equal to z_j plus ubar . ul / ur of the adjacent elements
        for (int e = threadIdx.x; e < nv * 4; e += blockDim.x) {
            const int v = e >> 2, side = (e >> 1) & 1, c = e & 1, r = v % R;
            double s = 0.0;
            if (r < nr) {
                const double* h = a.hom + ((size_t)a.grp_of_row[r0 + r] * 2 + side) * P;
                const TS* u = x + (size_t)v * P * 2 + c;
                s = (double)u[side ? 2 * (P - 1) : 0];
#pragma unroll 4
                for (int k = 1; k <= n; ++k) s += h[k] * (double)u[2 * k];
            }
            sl[e] = s;
        }
        __syncthreads();
        for (int r = warp; r < nr; r += nwarp) {
            const int grp = a.grp_of_row[r0 + r];
            const double d0ur = a.homs[grp * 4 + 1];
            double* zr = z + (size_t)r * M * 2;
            const double* pv = piv + (size_t)r * M;
            const double* mv = mul + (size_t)r * M;
            for (int e = lane; e < 2 * M; e += 32) {
                const int j = e >> 1, c = e & 1;
                double h = 0.0;
                if (j < Ns) h = sl[((size_t)j * R + r) * 4 + c];
                if (j > 0) h += sl[((size_t)(j - 1) * R + r) * 4 + 2 + c];
                zr[e] = h;
            }
            __syncwarp();
            if (lane < 2) {
                // T = L U of the forward sweep: U^T y = zbar, then L^T w = y
                double y = zr[lane] * pv[0];
                zr[lane] = y;
#pragma unroll 4
                for (int j = 1; j <= Ns; ++j) {
                    const double c = (j == 1 ? a.al : 1.0) * d0ur * pv[j];
                    y = zr[2 * j + lane] * pv[j] + c * y;
                    zr[2 * j + lane] = y;
                }
#pragma unroll 4
                for (int j = Ns - 1; j >= 0; --j) {
                    y = zr[2 * j + lane] - mv[j + 1] * y;
                    zr[2 * j + lane] = y;
                }
            }
        }
        __syncthreads();
        // interior right-hand sides ubar + d0bar D0 + dNbar DN (in FP32 plans rounded once more)
        for (int e = threadIdx.x; e < nv * P; e += blockDim.x) {
            const int j = e / seg, i = e - j * seg;
            const int r = i / P, k = i - r * P;
            if (r >= nr || k == 0 || k == P - 1) continue;
            const double* w = z + ((size_t)r * M + j) * 2;
            const double c0 = (j == 0 ? a.al : 1.0) * a.d0[k], cN = (j == Ns - 1 ? -a.ar : -1.0) * a.dN[k];
            x[2 * (size_t)e] = (TS)((double)x[2 * (size_t)e] + w[0] * c0 + w[2] * cN);
            x[2 * (size_t)e + 1] = (TS)((double)x[2 * (size_t)e + 1] + w[1] * c0 + w[3] * cN);
        }
        __syncthreads();
        interior_solves();
        for (int e = threadIdx.x; e < nv * P; e += blockDim.x) {
            const int j = e / seg, i = e - j * seg;
            if (i >= live) continue;
            const int r = i / P, k = i - r * P;
            const double* w = z + ((size_t)r * M + j) * 2;
            C u = mk((TS)0, (TS)0);
            if (k == 0) { if (j == 0) u = mk((TS)w[0], (TS)w[1]); }
            else if (k == P - 1) { if (j == Ns - 1) u = mk((TS)w[2], (TS)w[3]); }
            else u = xc[e];
            spec[(long long)j * a.elem_stride + i] = u;
        }
    }
}

// The factors of the interface system of every shift (MultiArgs::itf), one shift a
// thread, when the plan is made.  Bound: the chain of Ns divisions.  On the host, with the
// copies of the result, they took 4.3 of the 12.6 ms in which a plan of 16641 shifts and 60
// elements is created, 9 of 22 ms if periodic.  (Each operation rounded by itself:
// fused ones would move the last bit.)
template <bool PERIODIC>
__global__ void __launch_bounds__(64) multi_interface_kernel(int ngroups, int Ns, const double* homs, double al,
                                                             double bl, double ar, double br, double* itf)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    auto mul = [](double x, double y) { return __dmul_rn(x, y); };
    auto add = [](double x, double y) { return __dadd_rn(x, y); };
    auto sub = [](double x, double y) { return __dsub_rn(x, y); };
    const double d0ul = homs[4 * g], d0ur = homs[4 * g + 1], dNul = homs[4 * g + 2], dNur = homs[4 * g + 3];
    if (!PERIODIC) {
        double* out = itf + (size_t)g * (Ns + 1);
        double c = mul(-al, d0ur), p = __drcp_rn(sub(bl, mul(al, d0ul)));
        out[0] = p;
        for (int j = 1; j < Ns; ++j) {
            p = __drcp_rn(sub(sub(dNur, d0ul), mul(c, mul(dNul, p))));
            out[j] = p;
            c = -d0ur;
        }
        out[Ns] = __drcp_rn(sub(add(mul(ar, dNur), br), mul(c, mul(mul(ar, dNul), p))));
        return;
    }
    // cyclic: first diagonal shifted, last one gains D0.ur; eta solves the same
    // system for the correction's right-hand side
    double* out = itf + (size_t)g * 2 * (Ns + 1);
    double* eta = out + Ns + 1;
    double p = __drcp_rn(sub(sub(dNur, dNul), d0ul)), e = dNul;
    out[0] = p;
    eta[0] = e;
    for (int j = 1; j < Ns; ++j) {
        const double m = mul(dNul, p);
        p = __drcp_rn(add(add(sub(dNur, d0ul), j == Ns - 1 ? d0ur : 0.0), mul(d0ur, m)));
        e = sub(j == Ns - 1 ? -d0ur : 0.0, mul(m, e));
        out[j] = p;
        eta[j] = e;
    }
    out[Ns] = 0.0;
    const double elast = e = mul(e, p);
    eta[Ns - 1] = e;
    for (int j = Ns - 2; j >= 0; --j) {
        e = mul(add(eta[j], mul(d0ur, e)), out[j]);
        eta[j] = e;
    }
    eta[Ns] = __ddiv_rn(-1.0, add(add(1.0, elast), e));
}

template <typename TS, int NT>
int run_multi(MultiArgs a, cudaStream_t s)
{
    auto k = a.adjoint ? multi_rows_kernel<TS, NT, true> : multi_rows_kernel<TS, NT, false>;
    int R = multi_rows_per_cta(a.nrows, a.Ns, a.sms);
    // three CTAs an SM by shared memory, two where all warps share each vector
    while (R > 1 && multi_smem<TS>(R, a.Ns, a.P, a.n).total > (NT == 0 ? 110 : 72) * 1024) --R;
    a.rows_per_cta = R;
    const size_t smem = multi_smem<TS>(R, a.Ns, a.P, a.n).total;
    if (smem > kMaxSmemPerBlock) return (int)cudaErrorInvalidValue;
    cudaError_t e = allow_smem(k, smem, kMaxSmemPerBlock);
    if (e != cudaSuccess) return (int)e;
    const int tasks = (R * a.Ns + 3) / 4;
    const int ctas = (a.nrows + R - 1) / R;
    // Beyond eight CTAs an SM in all, four warps each: more CTAs side by side hide
    // one another's barriers (4160 of 2 x 30 x 6 points 43 us, eight warps 53; but
    // 528 of 2 x 25 x 10 15.5 and 14.6).
    const int threads = (NT == 0 || (tasks >= 5 && ctas <= 8 * a.sms)) ? 256 : tasks >= 3 ? 128 : 64;
    return (int)launch_k(k, dim3(ctas), dim3(threads), smem, s, a);
}

template <typename TS>
int multi_dispatch(const MultiArgs& a, cudaStream_t s)
{
    const int nt = (a.n + 7) / 8;
    if (nt <= 1) return run_multi<TS, 1>(a, s);
    if (nt <= 2) return run_multi<TS, 2>(a, s);
    if (a.n <= MULTI_WARP_N) return run_multi<TS, 4>(a, s);
    return run_multi<TS, 0>(a, s);
}

}  // namespace

std::vector<double> multi_fragments1(int n, const double* M1)
{
    const int nt = (n + 7) / 8;
    std::vector<double> f(multi_fragment_doubles(n, n), 0.0);
    for (int t = 0; t < nt; ++t)
        for (int kk = 0; kk < 2 * nt; ++kk)
            for (int l = 0; l < 32; ++l) {
                const int j = 8 * t + (l >> 2), k = 4 * kk + (l & 3);
                if (j < n && k < n) f[((size_t)t * 2 * nt + kk) * 32 + l] = M1[(size_t)j * n + k];
            }
    return f;
}

std::vector<double> multi_fragments2(int n, int outs, const double* M2)
{
    const int nt = (n + 7) / 8, no = (outs + 7) / 8;
    std::vector<double> f(multi_fragment_doubles(n, outs), 0.0);
    for (int o = 0; o < no; ++o)
        for (int t = 0; t < nt; ++t)
            for (int s = 0; s < 2; ++s)
                for (int l = 0; l < 32; ++l) {
                    const int i = 8 * o + (l >> 2), j = 8 * t + 2 * (l & 3) + s;
                    if (i < outs && j < n) f[((size_t)o * 2 * nt + 2 * t + s) * 32 + l] = M2[(size_t)i * n + j];
                }
    return f;
}

int launch_multi_interface(int ngroups, int Ns, bool periodic, const double* homs, double al, double bl, double ar,
                           double br, double* out, cudaStream_t s)
{
    auto k = periodic ? multi_interface_kernel<true> : multi_interface_kernel<false>;
    return (int)launch_alone(k, dim3((ngroups + 63) / 64), dim3(64), 0, s, ngroups, Ns, homs, al, bl, ar, br, out);
}

int launch_multi(bool spec_double, MultiArgs a, cudaStream_t s)
{
    if (a.n < 1 || a.n > MULTI_NMAX || a.Ns < 2 || a.nrows < 1 || (a.adjoint && a.periodic))
        return (int)cudaErrorInvalidValue;
    return spec_double ? multi_dispatch<double>(a, s) : multi_dispatch<float>(a, s);
}

}  // namespace helm
