// FP32 instances of the mixed-radix passes (mixfft.cuh).
#include "mixfft.cuh"

namespace cyr {

namespace {
using Kernel = void (*)(MixParams<float2>);
Kernel kernel(MixForm form, bool row) {
  return form == kMixPlain   ? (row ? k_mix_fft<float2, false, kMixPlain> : k_mix_fft<float2, true, kMixPlain>)
         : form == kMixRader ? (row ? k_mix_fft<float2, false, kMixRader> : k_mix_fft<float2, true, kMixRader>)
                             : (row ? k_mix_fft<float2, false, kMixBluestein> : k_mix_fft<float2, true, kMixBluestein>);
}
}  // namespace

template <>
cudaError_t mix_launch<float2>(MixForm form, bool row, dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                               const MixParams<float2> &p) {
  kernel(form, row)<<<grid, threads, smem, st>>>(p);
  return cudaGetLastError();
}

template <>
const void *mix_kernel<float2>(MixForm form, bool row) {
  return reinterpret_cast<const void *>(kernel(form, row));
}

}  // namespace cyr
