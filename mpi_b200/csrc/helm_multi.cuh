// Row solves of plans with several GLL elements, fast-diagonalisation method
// (helm_multi.cu).
#pragma once
#include <cuda_runtime.h>
#include <vector>

namespace helm {

constexpr int MULTI_NMAX = 127;  // interior points per element the kernel covers

// One solve of every spectrum row: Ns element vectors of n interior values, the
// interface system that couples them, the combination.
struct MultiArgs {
    void* spec;               // complex [Ns][nrows][P] (elem_stride between elements)
    long long elem_stride;    // complex elements
    int P, n, Ns, nrows;
    int sms;                  // multiprocessors of the plan's device
    int rows_per_cta;         // set by launch_multi
    const int* grp_of_row;    // shift group of each spectrum row
    const double* m1;         // first transform, fragment order (multi_fragments)
    const double* m2;         // second transform; forward: with the two end-slope rows
    const double* lam;        // [n] eigenvalues of the interior operator
    const double* sigma;      // [groups]
    const double* hom;        // [groups][2][P] forward homogeneous solutions ul, ur
    const double* homs;       // [groups][4] their end slopes D0.ul, D0.ur, DN.ul, DN.ur
    // factors of the interface system (launch_multi_interface): [groups][Ns + 1] reciprocal
    // pivots; periodic: followed by the correction eta [Ns] and its weight
    const double* itf;
    const double* d0;         // [P] first and last row of D (adjoint)
    const double* dN;
    double al, ar;
    int periodic, adjoint;
};

// Doubles of one transform with `outs` output rows in fragment order.
inline size_t multi_fragment_doubles(int n, int outs)
{
    return (size_t)((n + 7) / 8) * 8 * ((outs + 7) / 8) * 8;
}
// Fragment order of the two transforms (m8n8k4 B operands): M1[j][k] (n x n)
// read in natural k order, M2[i][j] (outs x n) in the k order in which the first
// product leaves its results.
std::vector<double> multi_fragments1(int n, const double* M1);
std::vector<double> multi_fragments2(int n, int outs, const double* M2);

// Reciprocal pivots of the interface system of every shift (and the periodic
// correction) from the end slopes homs [groups][4]; out: multi_interface_doubles a shift.
inline int multi_interface_doubles(int Ns, bool periodic) { return (periodic ? 2 : 1) * (Ns + 1); }
int launch_multi_interface(int ngroups, int Ns, bool periodic, const double* homs, double al, double bl, double ar,
                           double br, double* out, cudaStream_t s);

// Rows per CTA before the shared memory bounds them: 64 vectors, two groups of four for
// each of eight warps, when the elements are few, while every SM still gets two CTAs.
// With 32 vectors a CTA's fixed costs (plan data, barriers, the sweep) weighed twice as
// much: 14.6 against 18.6 us (stage, between events) for 1056 rows of 25 x 10 points,
// 18.3 against 22.4 for 2112 of 6 x 20; 52 x 10 on 257 rows is the same 14.7.
inline int multi_rows_per_cta(int nrows, int Ns, int sms)
{
    const int r = 64 / Ns, most = (nrows + 2 * sms - 1) / (2 * sms), rows = r < most ? r : most;
    return rows < 1 ? 1 : rows;
}

// spec_double: the spectrum holds doubles (else floats); arithmetic is FP64.
int launch_multi(bool spec_double, MultiArgs a, cudaStream_t s);

}  // namespace helm
