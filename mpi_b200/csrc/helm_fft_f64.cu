// Batched FFT passes: FP64 arrays and transforms.
#include "helm_fft.cuh"

namespace helm {

int launch_fft_f64(int L, int variant, int mode, int dir, const FftArgs& a, long long total_cols, cudaStream_t s)
{
    return fft_dispatch_len<double, double>(L, variant, mode, dir, a, total_cols, s);
}

}  // namespace helm
