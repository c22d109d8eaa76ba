// FP64 instances of the mixed-radix passes (mixfft.cuh).
#include "mixfft.cuh"

namespace cyr {

template <>
cudaError_t mix_launch<double2>(MixForm form, bool row, dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                               const MixParams<double2> &p) {
  auto kern = form == kMixPlain   ? (row ? k_mix_fft<double2, false, kMixPlain> : k_mix_fft<double2, true, kMixPlain>)
              : form == kMixRader ? (row ? k_mix_fft<double2, false, kMixRader> : k_mix_fft<double2, true, kMixRader>)
                                  : (row ? k_mix_fft<double2, false, kMixBluestein> : k_mix_fft<double2, true, kMixBluestein>);
  kern<<<grid, threads, smem, st>>>(p);
  return cudaGetLastError();
}

template <>
cudaError_t mix_attributes<double2>(int smem) {
  const void *kernels[] = {
      (const void *)k_mix_fft<double2, false, kMixPlain>,     (const void *)k_mix_fft<double2, true, kMixPlain>,
      (const void *)k_mix_fft<double2, false, kMixRader>,     (const void *)k_mix_fft<double2, true, kMixRader>,
      (const void *)k_mix_fft<double2, false, kMixBluestein>, (const void *)k_mix_fft<double2, true, kMixBluestein>,
  };
  for (const void *k : kernels) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace cyr
