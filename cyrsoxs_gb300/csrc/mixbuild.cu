// Field build fused with the x-row FFT for mixed-radix row lengths: a block builds
// the packed fields of a few rows into shared-memory lines and transforms them
// there with the stages of mixfft.cuh, so the packed volumes leave the chip once,
// already x-transformed (the separate build writes them and the row pass reads
// them back, 16 npk bytes per voxel).  Element x of a line is written straight to
// its slot in the row form's padded order.
// What bounds it: issue, as k_build_fields_rows; the morphology type and material
// count are one uniform branch per voxel around the unrolled field code.
// Measured, build + x, separate and fused: 240 x 240 x 90, 3 materials 268 -> 216 us;
// 450 x 450 x 75, 3 materials 1042 -> 782 us.  The rows of a block are chosen for full rounds of its
// 256 threads (two rows of 240: 292 us, three: 222); three blocks per SM (four, with smaller tiles: 249 us).
#include "mixfft.cuh"

namespace cyr {

// The block's lines (row r, packed volume j) at r npk + j, as the stages walk them.
struct BuildTile {
  const MixBuildParams &q;
  float2 *sm, *g;   // g: the first row's first element in volume 0
  size_t nvox;
  uint32_t lines;

  template <class F>
  __device__ __forceinline__ void each(const MixStage &st, F &&body) const {
    const uint32_t total = lines * st.nb;
    for (uint32_t t = threadIdx.x; t < total; t += blockDim.x) {
      const uint32_t l = mix_div(t, st.nb, st.nb_magic), r = mix_div(l, q.npk, q.npk_magic);
      body(g + size_t(l - r * q.npk) * nvox + size_t(r) * q.m.nx, sm + l * q.m.line_slots, t - l * st.nb, true);
    }
  }
  __device__ __forceinline__ uint32_t at(uint32_t s) const { return s; }
  __device__ __forceinline__ uint32_t jslot(uint32_t j) const {
    return q.m.pad ? j + mix_div(j, q.m.rs, q.m.rs_magic) : j;
  }
};

__global__ void __launch_bounds__(kMixThreads, 3) k_build_fields_mix(const __grid_constant__ MixBuildParams q) {
  extern __shared__ float2 bsm[];
  __shared__ float mean[kMaxFields];
  FieldParams f = q.f;
  field_group(f);
  field_means(f.mom, f.nmat, f.nsamp, mean);
  const MixParams<float2> &p = q.m;
  const uint32_t nx = p.nx, nrows = uint32_t((f.i1 - f.i0) / nx);
  BuildTile tile{q, bsm, nullptr, f.nvox, 0};
  for (uint32_t r0 = blockIdx.x * p.rows; r0 < nrows; r0 += gridDim.x * p.rows) {
    const uint32_t rows = min(p.rows, nrows - r0);
    const size_t base = f.i0 + size_t(r0) * nx;
    tile.g = f.out + base;
    tile.lines = rows * q.npk;
    __syncthreads();  // means ready; the previous rows' lines consumed
    for (uint32_t t = threadIdx.x; t < rows * nx; t += blockDim.x) {
      const uint32_t r = t / nx, x = t - r * nx;
      float w = 1.f;
      if (f.hann_x) {
        const size_t row = base / nx + r;
        w = f.hann_x[x] * (f.hann_y[row % f.ny] * f.hann_z[row / f.ny]);
      }
      float2 *s = bsm + r * q.npk * p.line_slots + __ldg(&q.slot[x]);
      auto put = [&](uint32_t j, float2 v) { s[j * p.line_slots] = v; };
      const size_t i = base + t;
      switch (q.form) {
#define CYR_FORM(m, n) \
  case 5 * m + n: voxel_fields<m, n>(f, i, w, mean, put); break;
        CYR_FORM(0, 1) CYR_FORM(0, 2) CYR_FORM(0, 3) CYR_FORM(0, 4)
        CYR_FORM(1, 0) CYR_FORM(1, 1) CYR_FORM(1, 2) CYR_FORM(1, 3) CYR_FORM(1, 4)
#undef CYR_FORM
        default: voxel_fields<0, 0>(f, i, w, mean, put);
      }
    }
    __syncthreads();
    // stage 1 in place, as the middle stages (block 0)
    mix_middle<float2, false>(p, tile, p.st[0], false);
    for (uint32_t s = 1; s + 1 < p.ns; ++s) {
      __syncthreads();
      mix_middle<float2, false>(p, tile, p.st[s], false);
    }
    __syncthreads();
    const MixStage &st = p.st[p.ns - 1];
    mix_radix(st.radix, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      tile.each(st, [&](float2 *g, float2 *s, uint32_t fb, bool) {
        const float2 *e = s + __ldg(&p.first[fb]);
        float2 v[R];
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = e[k];
        dft_reg<R>(v);
#pragma unroll
        for (int k = 0; k < R; ++k) g[fb + k * st.nb] = v[k];
      });
    });
  }
}

cudaError_t mix_build_launch(dim3 grid, size_t smem, cudaStream_t st, const MixBuildParams &p) {
  k_build_fields_mix<<<grid, kMixThreads, smem, st>>>(p);
  return cudaGetLastError();
}
const void *mix_build_kernel() { return reinterpret_cast<const void *>(k_build_fields_mix); }

}  // namespace cyr
