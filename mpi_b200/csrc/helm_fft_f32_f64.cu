// Batched FFT passes: FP32 transforms of FP64 arrays.
#include "helm_fft.cuh"

namespace helm {

int launch_fft_f32_f64(int L, int variant, int mode, int dir, const FftArgs& a, long long total_cols, cudaStream_t s)
{
    return fft_dispatch_len<float, double>(L, variant, mode, dir, a, total_cols, s);
}

}  // namespace helm
