// The packed fields of one voxel (fields.cuh), shared by the build kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cyr {

constexpr int kMaxMaterials = 32;
constexpr int kMoments = 7;  // at most 8 (k_moments)

// Direction and fractions of one material at one voxel.
template <int MORPH>
__device__ __forceinline__ void director(float4 s, float &sx, float &sy, float &sz, float &pa, float &pui) {
  if (MORPH == 0) {  // Euler: s1 = (S, theta, psi, Vfrac), uniaxial.h:82-92
    float st, ct, sp, cp;
    sincosf(s.y, &st, &ct);
    sincosf(s.z, &sp, &cp);
    sx = cp * st;
    sy = sp * st;
    sz = ct;
    pa = s.w * s.x;
    pui = s.w - pa;
  } else {  // vector: s1 = (sx, sy, sz, phi_unaligned), uniaxial.h:207-216
    sx = s.x, sy = s.y, sz = s.z;
    pa = 1.f;
    pui = s.w;
  }
}

constexpr int kFieldsPerMaterial = 7;

// field 7 m + f of material m, and T last
__host__ __device__ constexpr uint32_t num_fields(uint32_t nmat) { return kFieldsPerMaterial * nmat + 1; }
__host__ __device__ constexpr uint32_t num_packed(uint32_t nmat) { return (num_fields(nmat) + 1) / 2; }

constexpr uint32_t kMaxFields = num_fields(kMaxMaterials);
constexpr uint32_t kMaxPacked = num_packed(kMaxMaterials);

// Field means from the per-material moments (k_moments over nsamp voxels), T
// last, computed by the calling block.  Any constant subtracted from a field
// changes only bin 0, which is replaced, so the means need only be close (a
// sample of rows from all over the volume, sample_row); they keep the FP32
// rounding of the transform proportional to the fluctuations.
__device__ __forceinline__ void field_means(const double *__restrict__ mom, uint32_t nmat, size_t nsamp,
                                            float *__restrict__ out) {
  const uint32_t nf = num_fields(nmat);
  for (uint32_t g = threadIdx.x; g < nf; g += blockDim.x) {
    double v = 0.0;
    if (g + 1 < nf) {
      v = mom[(g / kFieldsPerMaterial) * kMoments + g % kFieldsPerMaterial];
    } else {
      for (uint32_t m = 0; m < nmat; ++m) {
        const double *M = mom + m * kMoments;
        v += M[0] + M[1] + M[2] + M[6];
      }
    }
    out[g] = float(v / double(nsamp));
  }
}

struct FieldParams {
  const float4 *vox;     // [nmat][nvox] as the reference stores Voxel::s1
  // request group (blockIdx.y = request): its morphologies, and the strides of
  // its moments and packed volumes; null for a single request
  const float4 *const *vox_g;
  size_t mom_stride, out_stride;
  uint32_t nx, ny, nz, nmat;
  size_t nvox;
  const double *mom;     // [nmat][kMoments] moment sums over nsamp voxels
  size_t nsamp;
  size_t i0, i1;         // voxels built: [i0, i1) (whole z planes)
  const float *hann_x, *hann_y, *hann_z;  // null when no windowing
  float2 *out;           // [num_packed][nvox]: field 2j in .x, field 2j+1 in .y
};

// Selects request blockIdx.y of a request group.
__device__ __forceinline__ void field_group(FieldParams &p) {
  if (!p.vox_g) return;
  p.vox = p.vox_g[blockIdx.y];
  p.mom += size_t(blockIdx.y) * p.mom_stride;
  p.out += size_t(blockIdx.y) * p.out_stride;
}

// The packed fields of voxel i (window weight w), put(j, volume j's value) in order.  MT > 0: the material count is
// known at compile time, so every field's place, mean and parity are too; MT = 0: any count, four materials at a time.
template <int MORPH, int MT, class Put>
__device__ __forceinline__ void voxel_fields(const FieldParams &p, size_t i, float w, const float *mean, Put &&put) {
  float T = 0.f, pend = 0.f;
  uint32_t g = 0;
  // g is the same in every thread: the parity branches do not diverge
  auto emit = [&](float v) {
    v -= mean[g];
    if (g & 1u)
      put(g >> 1, make_float2(pend, v));
    else
      pend = v;
    ++g;
  };
  auto material = [&](float4 sv) {
    float sx, sy, sz, pa, pui;
    director<MORPH>(sv, sx, sy, sz, pa, pui);
    const float wa = w * pa;
    const float f0 = wa * sx * sx, f1 = wa * sy * sy, f2 = wa * sz * sz, f6 = w * pui;
    T += f0 + f1 + f2 + f6;
    emit(f0);
    emit(f1);
    emit(f2);
    emit(wa * sx * sy);
    emit(wa * sx * sz);
    emit(wa * sy * sz);
    emit(f6);
  };
  if constexpr (MT > 0) {
    float4 sv[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) sv[m] = __ldg(&p.vox[m * p.nvox + i]);
#pragma unroll
    for (int m = 0; m < MT; ++m) material(sv[m]);
  } else {
    for (uint32_t m0 = 0; m0 < p.nmat; m0 += 4) {
      float4 sv[4];  // the loads of up to 4 materials are issued before any is used
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (m0 + u < p.nmat) sv[u] = __ldg(&p.vox[(m0 + u) * p.nvox + i]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (m0 + u < p.nmat) material(sv[u]);
    }
  }
  emit(T);
  if (g & 1u) put(g >> 1, make_float2(pend, 0.f));
}

}  // namespace cyr
