// Launches a batched FFT pass in the precision of its arrays.
#include "helm_fft.cuh"

namespace helm {

// Whether the pairs of neighbouring columns 2 c, 2 c + 1 of every row start at a
// multiple of their size `bytes` (two elements).
static bool pairs_aligned(const void* p, size_t bytes, long long row, long long batch, int nbatch,
                          const long long* offs)
{
    return !offs && reinterpret_cast<uintptr_t>(p) % bytes == 0 && row % 2 == 0 && (nbatch <= 1 || batch % 2 == 0);
}

int launch_fft(int L, int mode, int dir, int t_double, int io_bytes, const FftArgs& args, long long total_cols,
               cudaStream_t s, int variant)
{
    FftArgs a = args;
    // rows of paired columns: the real side has io_bytes an element, the spectrum a complex value
    const size_t real2 = 2 * (size_t)(t_double ? 8 : io_bytes), cplx2 = 2 * (size_t)(t_double ? 16 : 8);
    a.pair = 0;
    if (mode != FFT_C2C) {
        const bool real_in = mode == FFT_R2C || mode == FFT_DERIV, real_out = mode != FFT_R2C;
        if (pairs_aligned(a.in, real_in ? real2 : cplx2, a.in_row, a.in_batch, a.nbatch, a.in_boff) &&
            (!a.in_sub || reinterpret_cast<uintptr_t>(a.in_sub) % real2 == 0))
            a.pair |= 1;
        if (pairs_aligned(a.out, real_out ? real2 : cplx2, a.out_row, a.out_batch, a.nbatch, a.out_boff) &&
            (!a.lam_u || reinterpret_cast<uintptr_t>(a.lam_u) % 16 == 0))
            a.pair |= 2;
    }
    if (t_double) return launch_fft_f64(L, variant, mode, dir, a, total_cols, s);
    if (io_bytes == 8) return launch_fft_f32_f64(L, variant, mode, dir, a, total_cols, s);
    return launch_fft_f32(L, variant, mode, dir, a, total_cols, s);
}

}  // namespace helm
