// Batched FFT passes along a strided (non-contiguous) axis, real-to-complex,
// complex-to-real, complex-to-complex, or a spectral derivative: one tile of
// columns per CTA with the whole transform length staged in shared memory,
// radix-8/16 Stockham passes in registers.  Replaces FourierTransformX / Y / XY
// (Fourier_Quadrature.cpp:516-609, 719-926, 1097-1155).  Instantiated once per
// precision (helm_fft_f64.cu, helm_fft_f32.cu, helm_fft_f32_f64.cu: FP32
// transforms of FP64 arrays); launch_fft (helm_fft.cu) picks among them.
#pragma once
#include "helm_device.cuh"
#include "helm_kernels.cuh"

namespace helm {

int launch_fft_f64(int L, int variant, int mode, int dir, const FftArgs& a, long long total_cols, cudaStream_t s);
int launch_fft_f32(int L, int variant, int mode, int dir, const FftArgs& a, long long total_cols, cudaStream_t s);
int launch_fft_f32_f64(int L, int variant, int mode, int dir, const FftArgs& a, long long total_cols, cudaStream_t s);

// The two neighbouring real columns of an R2C / C2R pair, or their two complex
// spectrum values, as one access (ld_pair, st_pair; FftArgs::pair says that the addresses allow
// it).  A thread that loads or stores the two separately leaves every other
// 8 or 16 bytes to the next instruction: each of the two touches all sectors of
// the row segment, and the stores reach L2 as partial sectors.  FP64 passes of
// length 1024 over 1024 x 256 columns (a floor of 0.66 ms of HBM traffic):
// real-to-complex 1.44 -> 1.13 ms, complex-to-real 1.71 -> 1.09 ms.  The choice
// between pair and single accesses is made once around each unrolled loop: made
// inside, every load waited for the one before.

template <typename T, int L, int THREADS, int SMALL>
struct FftShape {
    using RS = RadixV<L, SMALL>;
    static constexpr int R0 = RS::r0, R1 = RS::r1, R2 = RS::r2, NP = RS::n;
    static constexpr int TPC = L / R0;          // threads per column
    static constexpr int CT = THREADS / TPC;    // columns per tile
    static constexpr size_t smem = (size_t)L * CT * sizeof(cplx_t<T>);
};

template <int R, int DIR, typename T>
__device__ __forceinline__ void dft_sub(cplx_t<T>* v)
{
    cplx_t<T> w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = v[r];
    dft_reg<R, DIR, T>(w);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = w[r];
}

// One Stockham pass (radix R, NS = product of the earlier radices) reading
// shared memory: every thread loads, twiddles and transforms its R0/R items.
template <typename T, int L, int R, int NS, int DIR, int TPC, int CT, int R0, bool SW = false>
__device__ __forceinline__ void pass_from_smem(const cplx_t<T>* sm, const cplx_t<T>* tw, int tc, int cl,
                                               cplx_t<T> (&v)[R0])
{
    constexpr int IPT = R0 / R;
#pragma unroll
    for (int t = 0; t < IPT; ++t) {
        const int j = tc + t * TPC;
        const int jm = j % NS;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = j + r * (L / R);
            cplx_t<T> x = sm[(SW ? swizzle_row<R0>(row, CT * sizeof(cplx_t<T>)) : row) * CT + cl];
            if (NS > 1 && r > 0) {
                const cplx_t<T> w = tw[r * jm * (L / (NS * R))];
                x = (DIR < 0) ? cmul(x, w) : cmulc(x, w);
            }
            v[t * R + r] = x;
        }
        dft_sub<R, DIR, T>(&v[t * R]);
    }
}

// Output row of item (t, r) of a pass with radix R and NS.
template <int R, int NS, int TPC>
__device__ __forceinline__ int pass_out_row(int tc, int t, int r)
{
    const int j = tc + t * TPC;
    return (j / NS) * NS * R + (j % NS) + r * NS;
}

template <typename T, int L, int R, int NS, int TPC, int CT, int R0, bool SW = false>
__device__ __forceinline__ void pass_to_smem(cplx_t<T>* sm, int tc, int cl, const cplx_t<T> (&v)[R0])
{
#pragma unroll
    for (int t = 0; t < R0 / R; ++t)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = pass_out_row<R, NS, TPC>(tc, t, r);
            sm[(SW ? swizzle_row<R0>(row, CT * sizeof(cplx_t<T>)) : row) * CT + cl] = v[t * R + r];
        }
}

// The real outputs of one thread of a C2R pass: columns c0 (and c1 when has1)
// at the rows of its last-pass items v[t RL + r], scaled by sc.  In an adjoint
// pass (a.adj_mode) the GLL boundary slots also go to the boundary cotangents
// (first slot of batch a.gl_batch, last slot of batch a.gr_batch: the first and
// last GLL element) and acc gathers the lambda sum; the forward solution values
// it needs are loaded for a whole group of rows before any store of that group.
template <bool ADJ, typename T, typename TIO, int R0, int RL, int NSL, int TPC>
__device__ __forceinline__ void c2r_store(const FftArgs& a, TIO* out, long long out_base, int b, int tc, int c0,
                                          int c1, bool has1, const cplx_t<T> (&v)[R0], T sc, double& acc)
{
    const bool pair = (a.pair & 2) && has1;
    if constexpr (!ADJ) {
        if (pair) {
#pragma unroll
            for (int t = 0; t < R0 / RL; ++t) {
                TIO y0[RL], y1[RL];
                if (a.accumulate) {
#pragma unroll
                    for (int r = 0; r < RL; ++r)
                        ld_pair(out + (long long)pass_out_row<RL, NSL, TPC>(tc, t, r) * a.out_row + c0, y0[r], y1[r]);
                } else {
#pragma unroll
                    for (int r = 0; r < RL; ++r) y0[r] = y1[r] = (TIO)0;
                }
#pragma unroll
                for (int r = 0; r < RL; ++r)
                    st_pair(out + (long long)pass_out_row<RL, NSL, TPC>(tc, t, r) * a.out_row + c0,
                            y0[r] + (TIO)(v[t * RL + r].x * sc), y1[r] + (TIO)(v[t * RL + r].y * sc));
            }
            return;
        }
#pragma unroll
        for (int t = 0; t < R0 / RL; ++t)
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const long long row = pass_out_row<RL, NSL, TPC>(tc, t, r);
                TIO* o0 = out + row * a.out_row + c0;
                const TIO x0 = (TIO)(v[t * RL + r].x * sc), x1 = (TIO)(v[t * RL + r].y * sc);
                if (a.accumulate) {
                    *o0 += x0;
                    if (has1) o0[c1 - c0] += x1;
                } else {
                    *o0 = x0;
                    if (has1) o0[c1 - c0] = x1;
                }
            }
        return;
    } else {
    const int P = a.adj_P;
    const int k0 = c0 % P, j0 = c0 / P, k1 = c1 % P, j1 = c1 / P;
    const bool b0 = k0 == 0 || k0 == P - 1, b1 = k1 == 0 || k1 == P - 1;
    const bool zero0 = a.adj_mode == 1 && b0, zero1 = a.adj_mode == 1 && b1;
    double* const gbl = b == a.gl_batch ? a.gbar_l : nullptr;
    double* const gbr = b == a.gr_batch ? a.gbar_r : nullptr;
    const double* u = a.lam_u ? a.lam_u + out_base : nullptr;
    // in groups of GR rows: whatever a group reads is loaded before any of its stores
    constexpr int GR = RL < 4 ? RL : (sizeof(T) == 8 || RL < 8) ? 4 : 8;
#pragma unroll
    for (int g0 = 0; g0 < R0; g0 += GR) {
        const int t = g0 / RL, q0 = g0 % RL;
        double u0[GR], u1[GR];
        TIO y0[GR], y1[GR];
#pragma unroll
        for (int r = 0; r < GR; ++r) {
            u0[r] = u1[r] = 0.0;
            y0[r] = y1[r] = (TIO)0;
        }
        if (u) {
            if (pair) {
#pragma unroll
                for (int r = 0; r < GR; ++r)
                    ld_pair(&u[pass_out_row<RL, NSL, TPC>(tc, t, q0 + r) * a.out_row + c0], u0[r], u1[r]);
            } else {
#pragma unroll
                for (int r = 0; r < GR; ++r) {
                    const long long row = pass_out_row<RL, NSL, TPC>(tc, t, q0 + r);
                    u0[r] = zero0 ? 0.0 : u[row * a.out_row + c0];
                    u1[r] = (has1 && !zero1) ? u[row * a.out_row + c1] : 0.0;
                }
            }
        }
        if (a.accumulate) {
            if (pair) {
#pragma unroll
                for (int r = 0; r < GR; ++r)
                    ld_pair(&out[pass_out_row<RL, NSL, TPC>(tc, t, q0 + r) * a.out_row + c0], y0[r], y1[r]);
            } else {
#pragma unroll
                for (int r = 0; r < GR; ++r) {
                    const long long row = pass_out_row<RL, NSL, TPC>(tc, t, q0 + r);
                    y0[r] = out[row * a.out_row + c0];
                    y1[r] = has1 ? out[row * a.out_row + c1] : (TIO)0;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < GR; ++r) {
            const long long row = pass_out_row<RL, NSL, TPC>(tc, t, q0 + r);
            const double x0 = (double)(v[g0 + r].x * sc), x1 = (double)(v[g0 + r].y * sc);
            // (accumulate: a refinement sweep adds its correction to fbar and gbar)
            const TIO f0 = zero0 ? (TIO)0 : (TIO)(y0[r] + x0), f1 = zero1 ? (TIO)0 : (TIO)(y1[r] + x1);
            TIO* const o = &out[row * a.out_row + c0];
            if (pair) {
                st_pair(o, f0, f1);
            } else {
                o[0] = f0;
                if (has1) o[1] = f1;
            }
            if (!zero0) acc += x0 * u0[r];
            if (has1 && !zero1) acc += x1 * u1[r];
        }
        if (b0 || b1) {
            auto bound = [&](int k, int j, double x, long long row) {
                if (k == 0 && gbl) {
                    double* g = &gbl[row * a.bc_row + j];
                    *g = (a.accumulate ? *g : 0.0) + a.adj_scale_l * x;
                }
                if (k == P - 1 && gbr) {
                    double* g = &gbr[row * a.bc_row + j];
                    *g = (a.accumulate ? *g : 0.0) + a.adj_scale_r * x;
                }
            };
#pragma unroll
            for (int r = 0; r < GR; ++r) {
                const long long row = pass_out_row<RL, NSL, TPC>(tc, t, q0 + r);
                if (b0) bound(k0, j0, (double)(v[g0 + r].x * sc), row);
                if (b1 && has1) bound(k1, j1, (double)(v[g0 + r].y * sc), row);
            }
        }
    }
    }
}

// Adds every thread's acc into *a.lam_out (one atomic per CTA); all threads call.
__device__ __forceinline__ void c2r_lambda_sum(const FftArgs& a, double acc)
{
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += red[w];
        atomicAdd(a.lam_out, sum);
    }
}

// Spectral derivative: the spectrum Z = A + i B of two packed real columns times
// (i w K)^order, K = k below L/2 and K = k - L from there on (FirstDerivativeFourierX /
// SecondDerivativeFourierX, Fourier_Quadrature.cpp:1400-1407, 1630-1637).  The
// multiplier is Hermitian (its value at L - k is the conjugate of its value at k),
// so the product is the packed spectrum of the two derivatives.  At K = -L/2 the
// first derivative vanishes (the real part the reference keeps) and the second keeps
// -(w L/2)^2.
template <typename T, int L>
__device__ __forceinline__ cplx_t<T> deriv_mul_packed(int order, double w, int k, cplx_t<T> Z)
{
    const double K = (k < L / 2) ? (double)k : (double)(k - L);
    const double wk = w * K;
    if (order == 1) {
        const T m = (k == L / 2) ? (T)0 : (T)wk;
        return mk(-m * Z.y, m * Z.x);
    }
    const T m = (T)(-wk * wk);
    return mk(m * Z.x, m * Z.y);
}

// Whether the exchange after the first pass is swizzled (swizzle_row): FP64 lengths
// 1024 and 512 y passes 926 -> 890 us (1024 x 1024 x 256), x passes 141 / 135 -> 135 /
// 128 us (512 x 512 x 128), derivatives FP32 512 x 128 x 65 20.5 -> 18.6 us; not in FP64
// derivatives of length 512, whose two transforms it makes spill (32.8 -> 34.7 us).
template <typename T, int L, int MODE>
__host__ __device__ constexpr bool fft_swizzled()
{
    return !(MODE == FFT_DERIV && L == 512 && sizeof(T) == 8);
}

// Batch and column within it of column g < total; 64-bit division only where needed.
__device__ __forceinline__ void split_column(long long g, int ccols, long long total, int& b, int& c)
{
    if (total <= 0x7fffffff) {
        b = (int)((unsigned)g / (unsigned)ccols);
        c = (int)((unsigned)g - (unsigned)b * (unsigned)ccols);
    } else {
        b = (int)(g / ccols);
        c = (int)(g - (long long)b * ccols);
    }
}

// Warps an SM has room for: 24 (at most 85 registers a thread), or 16 where 16
// points of 8 bytes a thread, or an adjoint pass's operands, would spill at that.
template <typename T, typename TIO, int L, int MODE, int THREADS, int SMALL>
constexpr int fft_min_ctas()
{
    if (THREADS > 256) return 1;
    const bool many = MODE == FFT_C2R_ADJ || (RadixV<L, SMALL>::r0 > 8 && sizeof(TIO) == 8);
    return (many ? 512 : 768) / THREADS;
}

// MANY: complex passes of many tiles on 512 threads (length 512; FP32 1024 as well).  They have
// no pairs to keep in flight: given the registers of the bound above they hold half the
// warps, and gain only while the tiles are few.  Left to its own count the compiler
// takes 32 instead of 54 registers (FP32 length 512: 59.4 us a pass of 1024 x 512 x 64,
// 71.7 bounded) or 56 instead of 75 (FP64, 256 x 512 x 128: 58 and 86 us); two CTAs of length 1024
// FP32 need its exchange unswizzled (1024 x 1024 x 64: 125 us, 135 swizzled, 162 in one CTA).
template <typename T, int L, int MODE, int THREADS>
constexpr bool fft_has_many()
{
    return MODE == FFT_C2C && THREADS == 512 && (L == 512 || (L == 1024 && sizeof(T) == 4));
}

template <typename T, typename TIO, int L, int DIR, int MODE, int THREADS, int SMALL, bool MANY = false>
__global__ void __launch_bounds__(THREADS, (MANY ? (L == 512 ? 0 : 2) : fft_min_ctas<T, TIO, L, MODE, THREADS, SMALL>())) fft_kernel(FftArgs a, long long total_cols)
{
    using C = cplx_t<T>;
    using S = FftShape<T, L, THREADS, SMALL>;
    constexpr int R0 = S::R0, R1 = S::R1, R2 = S::R2, NP = S::NP, TPC = S::TPC, CT = S::CT;
    constexpr bool SW = fft_swizzled<T, L, MODE>() && !(MANY && L == 1024);
    extern __shared__ __align__(16) unsigned char fft_smem[];
    C* sm = reinterpret_cast<C*>(fft_smem);
    const C* tw = static_cast<const C*>(a.tw);

    const int tc = threadIdx.x / CT;
    const int cl = threadIdx.x - tc * CT;
    const long long g = (long long)blockIdx.x * CT + cl;
    const bool valid = g < total_cols;
    const int ccols = (MODE == FFT_C2C) ? a.ncols : (a.ncols + 1) >> 1;
    int b, c;
    split_column(valid ? g : 0, ccols, total_cols, b, c);
    const int c0 = 2 * c, c1 = 2 * c + 1;  // real columns of an R2C / C2R pair
    const bool has1 = c1 < a.ncols;
    const long long in_base = a.in_boff ? a.in_boff[b] : (long long)b * a.in_batch;
    const long long out_base = a.out_boff ? a.out_boff[b] : (long long)b * a.out_batch;
    // (the columns' addresses are plan data: worked out before the previous pass is waited for)
    pdl_enter();
    if (a.zero_out && blockIdx.x == 0 && threadIdx.x == 0) *a.zero_out = 0.0;

    C v[R0];
    // ---------------------------------------------------------- pass 0 --
    if constexpr (MODE == FFT_C2R || MODE == FFT_C2R_ADJ) {
        // Z_k = A_k + i B_k over the full length from the two half spectra
        const C* in = static_cast<const C*>(a.in) + in_base;
        auto put = [&](int k, C A, C B) {
            if (k == 0 || k == L / 2) { A.y = 0; B.y = 0; }
            sm[k * CT + cl] = mk(A.x - B.y, A.y + B.x);
            if (k != 0 && k != L / 2) sm[(L - k) * CT + cl] = mk(A.x + B.y, B.x - A.y);
        };
        // rows below L/2: all loads of a thread in flight at once
        constexpr int KPT = L / 2 / TPC;
        C A[KPT], B[KPT], Ah = mk((T)0, (T)0), Bh = mk((T)0, (T)0);
        const C* q = in + (long long)tc * a.in_row + c0;
        const C* qh = in + (long long)(L / 2) * a.in_row + c0;
        if (valid && has1 && (a.pair & 1)) {
#pragma unroll
            for (int j = 0; j < KPT; ++j) ld_pair(q + (long long)j * TPC * a.in_row, A[j], B[j]);
            if (tc == 0) ld_pair(qh, Ah, Bh);
        } else {
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                A[j] = valid ? q[(long long)j * TPC * a.in_row] : mk((T)0, (T)0);
                B[j] = (valid && has1) ? q[(long long)j * TPC * a.in_row + 1] : mk((T)0, (T)0);
            }
            if (tc == 0 && valid) {
                Ah = qh[0];
                if (has1) Bh = qh[1];
            }
        }
#pragma unroll
        for (int j = 0; j < KPT; ++j) put(tc + j * TPC, A[j], B[j]);
        if (tc == 0) put(L / 2, Ah, Bh);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R0; ++r) v[r] = sm[(tc + r * TPC) * CT + cl];
    } else if constexpr (MODE == FFT_DERIV) {
        const TIO* in = static_cast<const TIO*>(a.in) + in_base;
        if (valid && has1 && (a.pair & 1)) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                TIO x0, x1;
                ld_pair(&in[(tc + r * TPC) * a.in_row + c0], x0, x1);
                v[r] = mk((T)x0, (T)x1);
            }
        } else {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long row = tc + r * TPC;
                T x0 = 0, x1 = 0;
                if (valid) {
                    x0 = (T)in[row * a.in_row + c0];
                    if (has1) x1 = (T)in[row * a.in_row + c1];
                }
                v[r] = mk(x0, x1);
            }
        }
    } else if constexpr (MODE == FFT_R2C) {
        const TIO* in = static_cast<const TIO*>(a.in) + in_base;
        const TIO* sub = a.in_sub ? static_cast<const TIO*>(a.in_sub) + in_base : nullptr;
        int k0 = -1, k1 = -1, j0 = 0, j1 = 0;  // GLL slot of the two real columns
        if (a.P > 0) { k0 = c0 % a.P; j0 = c0 / a.P; k1 = c1 % a.P; j1 = c1 / a.P; }
        const bool bnd0 = a.P > 0 && (k0 == 0 || k0 == a.P - 1);
        const bool bnd1 = a.P > 0 && (k1 == 0 || k1 == a.P - 1);
        const double* s0 = (k0 == 0) ? (b == a.gl_batch ? a.gl : nullptr) : (b == a.gr_batch ? a.gr : nullptr);
        const double* s1 = (k1 == 0) ? (b == a.gl_batch ? a.gl : nullptr) : (b == a.gr_batch ? a.gr : nullptr);
        const bool pr = valid && has1 && (a.pair & 1);
        if (sub) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long o = (tc + r * TPC) * a.in_row + c0;
                TIO x0 = 0, x1 = 0, y0 = 0, y1 = 0;
                if (pr) {
                    ld_pair(&in[o], x0, x1);
                    ld_pair(&sub[o], y0, y1);
                } else if (valid) {
                    x0 = in[o];
                    y0 = sub[o];
                    if (has1) {
                        x1 = in[o + 1];
                        y1 = sub[o + 1];
                    }
                }
                v[r] = mk((T)((double)x0 - (double)y0), (T)((double)x1 - (double)y1));
            }
        } else if (pr) {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                TIO x0, x1;
                ld_pair(&in[(tc + r * TPC) * a.in_row + c0], x0, x1);
                v[r] = mk((T)x0, (T)x1);
            }
        } else {
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long o = (tc + r * TPC) * a.in_row + c0;
                v[r] = mk(valid ? (T)in[o] : (T)0, (valid && has1) ? (T)in[o + 1] : (T)0);
            }
        }
        // boundary slots: the data in place of the input, or added to it
        // (the input read again: held back it would cost every column its registers)
        auto bnd_value = [&](const double* g, int k, int j, int r, int c) -> T {
            const long long row = tc + r * TPC;
            double x = a.bc_add ? (double)in[row * a.in_row + c] : 0.0;
            if (g) x += (a.bc_add ? (k == 0 ? a.bc_scale_l : a.bc_scale_r) : 1.0) * g[row * a.bc_row + j];
            return (T)x;
        };
        if (bnd0 && valid)
#pragma unroll
            for (int r = 0; r < R0; ++r) v[r].x = bnd_value(s0, k0, j0, r, c0);
        if (bnd1 && valid && has1)
#pragma unroll
            for (int r = 0; r < R0; ++r) v[r].y = bnd_value(s1, k1, j1, r, c1);
    } else {
        const C* in = static_cast<const C*>(a.in) + in_base;
#pragma unroll
        for (int r = 0; r < R0; ++r) v[r] = valid ? in[(long long)(tc + r * TPC) * a.in_row + c] : mk((T)0, (T)0);
    }
    dft_reg<R0, DIR, T>(v);

    // --------------------------------------------------- later passes --
    if constexpr (NP >= 2) {
        if constexpr (MODE == FFT_C2R || MODE == FFT_C2R_ADJ) __syncthreads();  // pass 0 read shared memory
        pass_to_smem<T, L, R0, 1, TPC, CT, R0, SW>(sm, tc, cl, v);
        __syncthreads();
        pass_from_smem<T, L, R1, R0, DIR, TPC, CT, R0, SW>(sm, tw, tc, cl, v);
    }
    if constexpr (NP >= 3) {
        __syncthreads();
        pass_to_smem<T, L, R1, R0, TPC, CT, R0>(sm, tc, cl, v);
        __syncthreads();
        pass_from_smem<T, L, R2, R0 * R1, DIR, TPC, CT, R0>(sm, tw, tc, cl, v);
    }
    constexpr int RL = (NP == 1) ? R0 : (NP == 2 ? R1 : R2);   // radix of the last pass
    constexpr int NSL = L / RL;                                 // its NS

    // ---------------------------------------------------------- output --
    const T sc = (T)a.scale;
    if constexpr (MODE == FFT_DERIV) {
        // multiply in place, inverse transform, the two real output columns
#pragma unroll
        for (int t = 0; t < R0 / RL; ++t)
#pragma unroll
            for (int r = 0; r < RL; ++r)
                v[t * RL + r] = deriv_mul_packed<T, L>(a.deriv_order, a.deriv_w, pass_out_row<RL, NSL, TPC>(tc, t, r),
                                                       v[t * RL + r]);
        fft_inverse_mirror<T, L, TPC, R0, R1, R2, NP, SW>(sm, CT, tw, tc, cl, v);
        if (valid) {
            TIO* out = static_cast<TIO*>(a.out) + out_base;
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long row = tc + r * TPC;
                const TIO x0 = (TIO)(v[r].x * sc), x1 = (TIO)(v[r].y * sc);
                if ((a.pair & 2) && has1) {
                    st_pair(&out[row * a.out_row + c0], x0, x1);
                } else {
                    out[row * a.out_row + c0] = x0;
                    if (has1) out[row * a.out_row + c1] = x1;
                }
            }
        }
    } else if constexpr (MODE == FFT_C2C) {
        if (valid) {
            C* out = static_cast<C*>(a.out) + out_base;
#pragma unroll
            for (int t = 0; t < R0 / RL; ++t)
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const int row = pass_out_row<RL, NSL, TPC>(tc, t, r);
                    out[(long long)row * a.out_row + c] = cscale(v[t * RL + r], sc);
                }
        }
    } else if constexpr (MODE == FFT_C2R || MODE == FFT_C2R_ADJ) {
        double acc = 0.0;
        if (valid)
            c2r_store<MODE == FFT_C2R_ADJ, T, TIO, R0, RL, NSL, TPC>(a, static_cast<TIO*>(a.out) + out_base, out_base, b, tc, c0, c1, has1, v,
                                                sc, acc);
        if constexpr (MODE == FFT_C2R_ADJ)
            if (a.lam_out) c2r_lambda_sum(a, acc);
    } else {  // R2C: separate the two real columns' spectra, keep k = 0 .. L/2
        __syncthreads();
        pass_to_smem<T, L, RL, NSL, TPC, CT, R0>(sm, tc, cl, v);
        __syncthreads();
        if (valid) {
            C* out = static_cast<C*>(a.out) + out_base;
            const T h = (T)0.5 * sc;
            for (int k = tc; k <= L / 2; k += TPC) {
                const C Z = sm[k * CT + cl];
                const C Zm = sm[((L - k) & (L - 1)) * CT + cl];
                const C A = mk((Z.x + Zm.x) * h, (Z.y - Zm.y) * h), B = mk((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
                C* o = &out[(long long)k * a.out_row + c0];
                if ((a.pair & 2) && has1) {
                    st_pair(o, A, B);
                } else {
                    o[0] = A;
                    if (has1) o[1] = B;
                }
            }
        }
    }
}

// ------------------------------------------------ pipelined FFT pass --
// The same transforms as fft_kernel from a persistent grid: every CTA walks
// tiles blockIdx.x, blockIdx.x + gridDim.x, ... and copies the next tile's
// input into shared memory (cp.async, one copy per element) while it
// transforms the current one, so the loads of one tile overlap the butterflies
// and stores of the previous.  Two tile buffers per CTA; the buffer of the
// current tile doubles as the exchange buffer of its passes.


template <typename T, typename TIO, int L, int THREADS, int SMALL>
struct PipeShape {
    using S = FftShape<T, L, THREADS, SMALL>;
    // one tile buffer holds the staged input -- complex values (C2C), pairs of
    // real inputs (R2C), or the pairs A_k, B_k of rows k <= L/2 (C2R) -- and
    // then serves as the exchange buffer of the passes
    static constexpr size_t c2r = (size_t)(L + 2) * S::CT * 2 * sizeof(T);
    static constexpr size_t r2c = (size_t)L * S::CT * 2 * sizeof(TIO);
    static constexpr size_t exch = (size_t)L * S::CT * 2 * sizeof(T);
    static constexpr size_t big = c2r > r2c ? (c2r > exch ? c2r : exch) : (r2c > exch ? r2c : exch);
    static constexpr size_t buf = (big + 15) / 16 * 16;
    static constexpr size_t smem = 2 * buf;
};

// Issue the asynchronous copies of tile `tile` into `stage` (no commit).
template <typename T, typename TIO, int L, int MODE, int THREADS, int SMALL>
__device__ __forceinline__ void pipe_issue(const FftArgs& a, long long total_cols, long long tile,
                                           unsigned char* stage)
{
    using C = cplx_t<T>;
    using S = FftShape<T, L, THREADS, SMALL>;
    constexpr int R0 = S::R0, TPC = S::TPC, CT = S::CT;
    const int tc = threadIdx.x / CT;
    const int cl = threadIdx.x - tc * CT;
    const long long g = tile * CT + cl;
    const bool valid = g < total_cols;
    const int ccols = (MODE == FFT_C2C) ? a.ncols : (a.ncols + 1) >> 1;
    int b, c;
    split_column(valid ? g : 0, ccols, total_cols, b, c);
    const long long in_base = a.in_boff ? a.in_boff[b] : (long long)b * a.in_batch;
    if constexpr (MODE == FFT_C2C) {
        const C* in = static_cast<const C*>(a.in) + in_base;
        C* st = reinterpret_cast<C*>(stage);
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const long long row = tc + r * TPC;
            cp_async_elem<sizeof(C)>(&st[row * CT + cl], valid ? &in[row * a.in_row + c] : a.in, valid);
        }
    } else if constexpr (MODE == FFT_R2C || MODE == FFT_DERIV) {
        const TIO* in = static_cast<const TIO*>(a.in) + in_base;
        TIO* st = reinterpret_cast<TIO*>(stage);
        const int c0 = 2 * c, c1 = 2 * c + 1;
        const bool v1 = valid && c1 < a.ncols;
#pragma unroll
        for (int r = 0; r < R0; ++r) {
            const long long row = tc + r * TPC;
            if ((a.pair & 1) && v1) {
                cp_async_elem<2 * sizeof(TIO)>(&st[(row * CT + cl) * 2], &in[row * a.in_row + c0], true);
                continue;
            }
            cp_async_elem<sizeof(TIO)>(&st[(row * CT + cl) * 2], valid ? &in[row * a.in_row + c0] : a.in, valid);
            cp_async_elem<sizeof(TIO)>(&st[(row * CT + cl) * 2 + 1], v1 ? &in[row * a.in_row + c1] : a.in, v1);
        }
    } else {  // C2R: A_k, B_k for k = 0 .. L/2
        const C* in = static_cast<const C*>(a.in) + in_base;
        C* st = reinterpret_cast<C*>(stage);
        const int c0 = 2 * c, c1 = 2 * c + 1;
        const bool v1 = valid && c1 < a.ncols;
        for (int k = tc; k <= L / 2; k += TPC) {
            cp_async_elem<sizeof(C)>(&st[((long long)k * CT + cl) * 2], valid ? &in[(long long)k * a.in_row + c0] : a.in,
                                     valid);
            cp_async_elem<sizeof(C)>(&st[((long long)k * CT + cl) * 2 + 1],
                                     v1 ? &in[(long long)k * a.in_row + c1] : a.in, v1);
        }
    }
}

template <typename T, typename TIO, int L, int DIR, int MODE, int THREADS, int SMALL>
__global__ void __launch_bounds__(THREADS) fft_pipe_kernel(FftArgs a, long long total_cols, long long ntiles)
{
    pdl_enter();
    if (a.zero_out && blockIdx.x == 0 && threadIdx.x == 0) *a.zero_out = 0.0;
    using C = cplx_t<T>;
    using S = FftShape<T, L, THREADS, SMALL>;
    using PS = PipeShape<T, TIO, L, THREADS, SMALL>;
    constexpr int R0 = S::R0, R1 = S::R1, R2 = S::R2, NP = S::NP, TPC = S::TPC, CT = S::CT;
    constexpr bool SW = fft_swizzled<T, L, MODE>();
    extern __shared__ __align__(16) unsigned char fft_smem[];
    const C* tw = static_cast<const C*>(a.tw);
    const int tc = threadIdx.x / CT;
    const int cl = threadIdx.x - tc * CT;
    const int ccols = (MODE == FFT_C2C) ? a.ncols : (a.ncols + 1) >> 1;

    long long tile = blockIdx.x;
    int cur = 0;
    double lam_acc = 0.0;  // adjoint C2R: this thread's share of the lambda sum
    if (tile < ntiles) pipe_issue<T, TIO, L, MODE, THREADS, SMALL>(a, total_cols, tile, fft_smem);
    cp_async_commit();
    for (; tile < ntiles; tile += gridDim.x, cur ^= 1) {
        unsigned char* buf = fft_smem + (size_t)cur * PS::buf;
        const long long next = tile + gridDim.x;
        if (next < ntiles) pipe_issue<T, TIO, L, MODE, THREADS, SMALL>(a, total_cols, next, fft_smem + (size_t)(cur ^ 1) * PS::buf);
        cp_async_commit();
        cp_async_wait_prev();
        __syncthreads();

        C* sm = reinterpret_cast<C*>(buf);
        const long long g = tile * CT + cl;
        const bool valid = g < total_cols;
        int b, c;
        split_column(valid ? g : 0, ccols, total_cols, b, c);
        const int c0 = 2 * c, c1 = 2 * c + 1;
        const bool has1 = c1 < a.ncols;
        const long long out_base = a.out_boff ? a.out_boff[b] : (long long)b * a.out_batch;

        C v[R0];
        // ------------------------------------------------ pass 0 input --
        if constexpr (MODE == FFT_C2R || MODE == FFT_C2R_ADJ) {
            constexpr int KPT = (L / 2) / TPC + 1;  // half-spectrum rows per thread (upper bound)
            C A[KPT], B[KPT];
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const int k = tc + j * TPC;
                if (k <= L / 2) {
                    A[j] = sm[((size_t)k * CT + cl) * 2];
                    B[j] = sm[((size_t)k * CT + cl) * 2 + 1];
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < KPT; ++j) {
                const int k = tc + j * TPC;
                if (k <= L / 2) {
                    C Aj = A[j], Bj = B[j];
                    if (k == 0 || k == L / 2) { Aj.y = 0; Bj.y = 0; }
                    sm[k * CT + cl] = mk(Aj.x - Bj.y, Aj.y + Bj.x);
                    if (k != 0 && k != L / 2) sm[(L - k) * CT + cl] = mk(Aj.x + Bj.y, Bj.x - Aj.y);
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < R0; ++r) v[r] = sm[(tc + r * TPC) * CT + cl];
            __syncthreads();
        } else if constexpr (MODE == FFT_R2C || MODE == FFT_DERIV) {
            const TIO* st = reinterpret_cast<const TIO*>(buf);
            int k0 = -1, k1 = -1, j0 = 0, j1 = 0;
            if (a.P > 0) { k0 = c0 % a.P; j0 = c0 / a.P; k1 = c1 % a.P; j1 = c1 / a.P; }
            const bool bnd0 = a.P > 0 && (k0 == 0 || k0 == a.P - 1);
            const bool bnd1 = a.P > 0 && (k1 == 0 || k1 == a.P - 1);
            const double* s0 = (k0 == 0) ? (b == a.gl_batch ? a.gl : nullptr) : (b == a.gr_batch ? a.gr : nullptr);
            const double* s1 = (k1 == 0) ? (b == a.gl_batch ? a.gl : nullptr) : (b == a.gr_batch ? a.gr : nullptr);
#pragma unroll
            for (int r = 0; r < R0; ++r) {
                const long long row = tc + r * TPC;
                const TIO i0 = st[(row * CT + cl) * 2], i1 = st[(row * CT + cl) * 2 + 1];
                T x0 = (T)i0, x1 = (T)i1;
                if (bnd0) {
                    if (a.bc_add) {
                        double vv = (double)i0;
                        if (s0) vv += (k0 == 0 ? a.bc_scale_l : a.bc_scale_r) * s0[row * a.bc_row + j0];
                        x0 = (T)vv;
                    } else {
                        x0 = s0 ? (T)s0[row * a.bc_row + j0] : (T)0;
                    }
                }
                if (has1 && bnd1) {
                    if (a.bc_add) {
                        double vv = (double)i1;
                        if (s1) vv += (k1 == 0 ? a.bc_scale_l : a.bc_scale_r) * s1[row * a.bc_row + j1];
                        x1 = (T)vv;
                    } else {
                        x1 = s1 ? (T)s1[row * a.bc_row + j1] : (T)0;
                    }
                }
                if (!valid) { x0 = 0; x1 = 0; }
                v[r] = mk(x0, x1);
            }
            __syncthreads();  // the stage is the exchange buffer from here on
        } else {
#pragma unroll
            for (int r = 0; r < R0; ++r) v[r] = sm[(tc + r * TPC) * CT + cl];
            __syncthreads();
        }
        dft_reg<R0, DIR, T>(v);

        // ------------------------------------------------ later passes --
        if constexpr (NP >= 2) {
            pass_to_smem<T, L, R0, 1, TPC, CT, R0, SW>(sm, tc, cl, v);
            __syncthreads();
            pass_from_smem<T, L, R1, R0, DIR, TPC, CT, R0, SW>(sm, tw, tc, cl, v);
        }
        if constexpr (NP >= 3) {
            __syncthreads();
            pass_to_smem<T, L, R1, R0, TPC, CT, R0>(sm, tc, cl, v);
            __syncthreads();
            pass_from_smem<T, L, R2, R0 * R1, DIR, TPC, CT, R0>(sm, tw, tc, cl, v);
        }
        constexpr int RL = (NP == 1) ? R0 : (NP == 2 ? R1 : R2);
        constexpr int NSL = L / RL;

        // ------------------------------------------------------ output --
        const T sc = (T)a.scale;
        if constexpr (MODE == FFT_DERIV) {
            // multiply in place, inverse transform, the two real output columns
#pragma unroll
            for (int t = 0; t < R0 / RL; ++t)
#pragma unroll
                for (int r = 0; r < RL; ++r)
                    v[t * RL + r] = deriv_mul_packed<T, L>(a.deriv_order, a.deriv_w,
                                                           pass_out_row<RL, NSL, TPC>(tc, t, r), v[t * RL + r]);
            fft_inverse_mirror<T, L, TPC, R0, R1, R2, NP, SW>(sm, CT, tw, tc, cl, v);
            if (valid) {
                TIO* out = static_cast<TIO*>(a.out) + out_base;
#pragma unroll
                for (int r = 0; r < R0; ++r) {
                    const long long row = tc + r * TPC;
                    const TIO x0 = (TIO)(v[r].x * sc), x1 = (TIO)(v[r].y * sc);
                    if ((a.pair & 2) && has1) {
                        st_pair(&out[row * a.out_row + c0], x0, x1);
                    } else {
                        out[row * a.out_row + c0] = x0;
                        if (has1) out[row * a.out_row + c1] = x1;
                    }
                }
            }
        } else if constexpr (MODE == FFT_C2C) {
            if (valid) {
                C* out = static_cast<C*>(a.out) + out_base;
#pragma unroll
                for (int t = 0; t < R0 / RL; ++t)
#pragma unroll
                    for (int r = 0; r < RL; ++r) {
                        const int row = pass_out_row<RL, NSL, TPC>(tc, t, r);
                        out[(long long)row * a.out_row + c] = cscale(v[t * RL + r], sc);
                    }
            }
        } else if constexpr (MODE == FFT_C2R || MODE == FFT_C2R_ADJ) {
            if (valid)
                c2r_store<MODE == FFT_C2R_ADJ, T, TIO, R0, RL, NSL, TPC>(a, static_cast<TIO*>(a.out) + out_base, out_base, b, tc, c0, c1,
                                                    has1, v, sc, lam_acc);
        } else {
            __syncthreads();
            pass_to_smem<T, L, RL, NSL, TPC, CT, R0>(sm, tc, cl, v);
            __syncthreads();
            if (valid) {
                C* out = static_cast<C*>(a.out) + out_base;
                const T h = (T)0.5 * sc;
                for (int k = tc; k <= L / 2; k += TPC) {
                    const C Z = sm[k * CT + cl];
                    const C Zm = sm[((L - k) & (L - 1)) * CT + cl];
                    const C A = mk((Z.x + Zm.x) * h, (Z.y - Zm.y) * h), B = mk((Z.y + Zm.y) * h, (Zm.x - Z.x) * h);
                    C* o = &out[(long long)k * a.out_row + c0];
                    if ((a.pair & 2) && has1) {
                        st_pair(o, A, B);
                    } else {
                        o[0] = A;
                        if (has1) o[1] = B;
                    }
                }
            }
        }
        __syncthreads();  // this buffer is refilled two tiles later
    }
    asm volatile("cp.async.wait_all;\n" ::);
    if constexpr (MODE == FFT_C2R_ADJ)
        if (a.lam_out) c2r_lambda_sum(a, lam_acc);
}

template <typename T, typename TIO, int L, int DIR, int MODE, int THREADS, int SMALL>
static int run_fft_pipe(const FftArgs& a, long long total_cols, cudaStream_t s)
{
    using S = FftShape<T, L, THREADS, SMALL>;
    using PS = PipeShape<T, TIO, L, THREADS, SMALL>;
    auto k = fft_pipe_kernel<T, TIO, L, DIR, MODE, THREADS, SMALL>;
    if (PS::smem > kMaxSmemPerBlock) return (int)cudaErrorInvalidValue;
    cudaError_t e = allow_smem(k, PS::smem);
    if (e != cudaSuccess) return (int)e;
    const long long tiles = (total_cols + S::CT - 1) / S::CT;
    if (tiles <= 0) return 0;
    static std::atomic<unsigned long long> memo{0};
    long long grid = resident_ctas(k, THREADS, PS::smem, memo);
    if (grid > tiles) grid = tiles;
    return (int)launch_k(k, dim3((unsigned)grid), dim3(THREADS), PS::smem, s, a, total_cols, tiles);
}

template <typename T, typename TIO, int L, int DIR, int MODE, int THREADS, int SMALL>
static int run_fft(const FftArgs& a, long long total_cols, cudaStream_t s)
{
    using S = FftShape<T, L, THREADS, SMALL>;
    auto k = fft_kernel<T, TIO, L, DIR, MODE, THREADS, SMALL>;
    cudaError_t e = allow_smem(k, S::smem);
    if (e != cudaSuccess) return (int)e;
    const long long blocks = (total_cols + S::CT - 1) / S::CT;
    if (blocks <= 0) return 0;
    if constexpr (fft_has_many<T, L, MODE, THREADS>()) {
        // Beyond two waves of the bounded kernel: whole solves, bounded and this, 64 x 512 x 150 finite
        // differences FP32 (618 tiles) 73.4 and 69.6 us, 256 x 512 x 33 FP64 (532) 155.9 and 149.9, 1024 x
        // 512 x 64 FP32 461.7 and 438.0; below it the bounded one: 64 x 512 x 33 FP64 (136) 47.7 and 54.9,
        // 64 x 512 x 64 finite differences FP32 (264) 32.4 and 36.2
        static std::atomic<unsigned long long> memo{0};
        if (blocks > 2 * resident_ctas(k, THREADS, S::smem, memo)) {
            k = fft_kernel<T, TIO, L, DIR, MODE, THREADS, SMALL, true>;
            if ((e = allow_smem(k, S::smem)) != cudaSuccess) return (int)e;
        }
    }
    return (int)launch_k(k, dim3((unsigned)blocks), dim3(THREADS), S::smem, s, a, total_cols);
}

template <typename T, typename TIO, int L, int THREADS, int SMALL>
static int fft_dispatch_mode(int mode, int dir, const FftArgs& a, long long tc, cudaStream_t s, bool pipe)
{
    if (pipe) {
        if (mode == FFT_DERIV) return run_fft_pipe<T, TIO, L, -1, FFT_DERIV, THREADS, SMALL>(a, tc, s);
        if (mode == FFT_C2C)
            return dir < 0 ? run_fft_pipe<T, T, L, -1, FFT_C2C, THREADS, SMALL>(a, tc, s)
                           : run_fft_pipe<T, T, L, 1, FFT_C2C, THREADS, SMALL>(a, tc, s);
        if (mode == FFT_R2C) return run_fft_pipe<T, TIO, L, -1, FFT_R2C, THREADS, SMALL>(a, tc, s);
        if (mode == FFT_C2R_ADJ) {
            if constexpr (sizeof(TIO) == 8) return run_fft_pipe<T, TIO, L, 1, FFT_C2R_ADJ, THREADS, SMALL>(a, tc, s);
            return (int)cudaErrorInvalidValue;  // adjoint outputs are double
        }
        return run_fft_pipe<T, TIO, L, 1, FFT_C2R, THREADS, SMALL>(a, tc, s);
    }
    if (mode == FFT_C2C)
        return dir < 0 ? run_fft<T, T, L, -1, FFT_C2C, THREADS, SMALL>(a, tc, s)
                       : run_fft<T, T, L, 1, FFT_C2C, THREADS, SMALL>(a, tc, s);
    if (mode == FFT_R2C) return run_fft<T, TIO, L, -1, FFT_R2C, THREADS, SMALL>(a, tc, s);
    if (mode == FFT_DERIV) return run_fft<T, TIO, L, -1, FFT_DERIV, THREADS, SMALL>(a, tc, s);
    if (mode == FFT_C2R_ADJ) {
        if constexpr (sizeof(TIO) == 8) return run_fft<T, TIO, L, 1, FFT_C2R_ADJ, THREADS, SMALL>(a, tc, s);
        return (int)cudaErrorInvalidValue;
    }
    return run_fft<T, TIO, L, 1, FFT_C2R, THREADS, SMALL>(a, tc, s);
}

// Launch variants the autotuner chooses from: bit 0 -> 128-thread CTAs (half the
// columns per tile), bit 1 -> radix-8 schedule (lengths 128 and 256), bit 2 ->
// the persistent pipelined kernel, bit 3 -> 512-thread CTAs for lengths 512 and
// 1024 (twice the columns per tile: 128-byte runs of each row instead of 64 on
// the strided x pass); bits 3 and 0 together on an FP32 pass of length 1024:
// 1024-thread CTAs (16 column pairs, whole 128-byte lines of FP32 rows).
template <typename T, typename TIO, int L>
static int fft_dispatch_variant(int variant, int mode, int dir, const FftArgs& a, long long tc, cudaStream_t s)
{
    const bool small_cta = !(variant & 8) && (variant & 1) && (L / Radix<L>::r0 <= 128);
    const bool pipe = (variant & 4) != 0;
    if constexpr (L == 1024 && sizeof(T) == 4) {
        if ((variant & 9) == 9 && !pipe) return fft_dispatch_mode<T, TIO, L, 1024, 0>(mode, dir, a, tc, s, false);
    }
    if constexpr (L >= 512) {
        if (variant & 8) return fft_dispatch_mode<T, TIO, L, 512, 0>(mode, dir, a, tc, s, pipe);
    }
    if constexpr (has_small_radix<L>()) {
        if (variant & 2) {
            if (small_cta) return fft_dispatch_mode<T, TIO, L, 128, 1>(mode, dir, a, tc, s, pipe);
            return fft_dispatch_mode<T, TIO, L, 256, 1>(mode, dir, a, tc, s, pipe);
        }
    }
    if (small_cta) return fft_dispatch_mode<T, TIO, L, 128, 0>(mode, dir, a, tc, s, pipe);
    return fft_dispatch_mode<T, TIO, L, 256, 0>(mode, dir, a, tc, s, pipe);
}

template <typename T, typename TIO>
static int fft_dispatch_len(int L, int variant, int mode, int dir, const FftArgs& a, long long tc, cudaStream_t s)
{
    switch (L) {
        case 4: return fft_dispatch_variant<T, TIO, 4>(variant, mode, dir, a, tc, s);
        case 8: return fft_dispatch_variant<T, TIO, 8>(variant, mode, dir, a, tc, s);
        case 16: return fft_dispatch_variant<T, TIO, 16>(variant, mode, dir, a, tc, s);
        case 32: return fft_dispatch_variant<T, TIO, 32>(variant, mode, dir, a, tc, s);
        case 64: return fft_dispatch_variant<T, TIO, 64>(variant, mode, dir, a, tc, s);
        case 128: return fft_dispatch_variant<T, TIO, 128>(variant, mode, dir, a, tc, s);
        case 256: return fft_dispatch_variant<T, TIO, 256>(variant, mode, dir, a, tc, s);
        case 512: return fft_dispatch_variant<T, TIO, 512>(variant, mode, dir, a, tc, s);
        case 1024: return fft_dispatch_variant<T, TIO, 1024>(variant, mode, dir, a, tc, s);
        default: return (int)cudaErrorInvalidValue;
    }
}

}  // namespace helm
