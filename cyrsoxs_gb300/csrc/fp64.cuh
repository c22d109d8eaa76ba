// FP64 pipeline: the reference's scattering path with every amplitude in
// double, the drop-in for its -DDOUBLE_PRECISION build (include/Datatypes.h:
// 33-46) and the on-GPU FP64 check of the FP32 engine.
//
// The discrete decisions are made in float, exactly as the FP32 kernels make
// them (which pixel is NaN, which Ewald plane is read, which rotated pixel is
// written: ewald_geometry, warp_tap), so the NaN masks equal the FP32 path's.
// Every amplitude is double: the dielectric tensor from the optical constants
// (include/uniaxial.h:58-169 Euler, :184-292 vector), the Hanning window
// (src/cudaMain.cu:276-295), the 3D FFT (forward, unnormalised, double
// twiddles), the DC replacement (:123-176), the intensity |(k^2 I - Q Q^T) p|^2
// (include/cudaUtils.h:268-296), the plane interpolation, the bilinear blend of
// the rotation and detector warps, and the angle sum and mean (:877-909).
//
// Schedules.  Field spectra (k64_build_fields, k64_ewald_fields): the 7 M
// energy independent real fields of the morphology are transformed once, in
// pairs, and every energy and E angle is formed from them at the Ewald sample
// points, exact by linearity as in fields.cuh; GB300's FP64 rate is 1/64 of
// its FP32 rate, so the transforms' operations are what counts, and 3.5 M
// volumes per request replace 5 per energy (256 x 256 x 32, 2 materials, 3
// energies x 12 angles: 18.6 -> 2.57 ms, with the mixed-radix transforms of
// mixfft.cuh in the place of direct radix-8 sums; bound by the FP64 pipe).
// Per energy: LAB frame - the 5
// (6 with a tilted k) distinct entries of Nt are transformed once per energy
// and every E angle's p = Nt E / 4pi is formed at the sample points; MATERIAL
// frame - p = R^T Nt R x per angle, 3 transforms per angle, as the reference
// does.
#pragma once

#include "kernels.cuh"

namespace cyr {

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// Refractive indices of one energy, n = 1 - delta + i beta (include/PyClass/RefractiveIndex.h:101-106).
struct Mat64 {
  double2 npar[kMaxMaterials];
  double2 nper[kMaxMaterials];
};

struct Build64Params {
  const void *vox;          // [M][V] float4 (the FP32 path's input) or double4 (vox_fp64)
  uint32_t vox_fp64;
  uint32_t nx, ny, nz, nmat;
  size_t nvox;
  uint32_t morphology;      // 0 Euler, 1 vector
  uint32_t mode;            // 0: Nt entries xx xy xz yy yz [zz]; 1: p for E (R^T p in the MATERIAL frame)
  uint32_t nvol;
  uint32_t material_frame;
  double E[3];
  double R[9];              // row major
  const double *hann_x, *hann_y, *hann_z;  // null: no window
  double2 *out;             // [nvol][V]
};

__device__ __forceinline__ void load_s64(const Build64Params &p, uint32_t m, size_t i, double s[4]) {
  if (p.vox_fp64) {
    const double4_16a v = static_cast<const double4_16a *>(p.vox)[size_t(m) * p.nvox + i];
    s[0] = v.x, s[1] = v.y, s[2] = v.z, s[3] = v.w;
  } else {
    const float4 v = static_cast<const float4 *>(p.vox)[size_t(m) * p.nvox + i];
    s[0] = v.x, s[1] = v.y, s[2] = v.z, s[3] = v.w;
  }
}

// The six entries of Nr - phi I summed over materials, in the reference's form.
__device__ void nt64(const Build64Params &p, const Mat64 &mt, size_t i, double2 nt[6]) {
  for (int q = 0; q < 6; ++q) nt[q] = make_double2(0.0, 0.0);
  for (uint32_t m = 0; m < p.nmat; ++m) {
    double s[4];
    load_s64(p, m, i, s);
    const double2 np = mt.npar[m], nq = mt.nper[m];
    const double2 npar2 = zmul(np, np), nper2 = zmul(nq, nq);
    const double2 nsum = make_double2(np.x + 2.0 * nq.x, np.y + 2.0 * nq.y);
    const double2 nsum2 = zmul(nsum, nsum);
    double sx, sy, sz, phi_a, phi_ui, phi;
    if (p.morphology == 0) {  // Euler: (S, theta, psi, Vfrac)
      double st, ct, sp, cp;
      sincos(s[1], &st, &ct);
      sincos(s[2], &sp, &cp);
      sx = cp * st, sy = sp * st, sz = ct;
      phi_a = s[3] * s[0];
      phi_ui = s[3] - phi_a;
      phi = s[3];
    } else {  // vector: (sx, sy, sz, phi_unaligned), Vfrac = |s|^2 + phi_ui
      sx = s[0], sy = s[1], sz = s[2];
      phi_ui = s[3];
      phi = phi_ui + sx * sx + sy * sy + sz * sz;
      phi_a = 1.0;
    }
    const double2 iso = zscale(nsum2, phi_ui / 9.0);
    const double2 dn = zsub(npar2, nper2);
    const double sq[3] = {sx * sx, sy * sy, sz * sz};
    const int diag[3] = {0, 3, 5};
    for (int a = 0; a < 3; ++a) {
      const double2 t = zadd(zscale(npar2, sq[a]), zscale(nper2, sq[(a + 1) % 3] + sq[(a + 2) % 3]));
      nt[diag[a]] = zadd(nt[diag[a]], make_double2(phi_a * t.x + iso.x - phi, phi_a * t.y + iso.y));
    }
    nt[1] = zadd(nt[1], zscale(dn, phi_a * sx * sy));
    nt[2] = zadd(nt[2], zscale(dn, phi_a * sx * sz));
    nt[4] = zadd(nt[4], zscale(dn, phi_a * sy * sz));
  }
}

__global__ void __launch_bounds__(256) k64_build(Build64Params p, const Mat64 *__restrict__ mat) {
  const double inv4pi = 0.25 / 3.141592653589793238462643383279502884;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < p.nvox; i += size_t(gridDim.x) * blockDim.x) {
    double2 nt[6];
    nt64(p, *mat, i, nt);
    double w = 1.0;
    if (p.hann_x) {
      const uint32_t X = uint32_t(i % p.nx), Y = uint32_t((i / p.nx) % p.ny), Z = uint32_t(i / (size_t(p.nx) * p.ny));
      w = p.hann_x[X] * p.hann_y[Y] * p.hann_z[Z];
    }
    if (p.mode == 0) {
      for (uint32_t v = 0; v < p.nvol; ++v) p.out[size_t(v) * p.nvox + i] = zscale(nt[v], inv4pi * w);
      continue;
    }
    const double *E = p.E;
    double2 q[3];
    q[0] = zadd(zadd(zscale(nt[0], E[0]), zscale(nt[1], E[1])), zscale(nt[2], E[2]));
    q[1] = zadd(zadd(zscale(nt[1], E[0]), zscale(nt[3], E[1])), zscale(nt[4], E[2]));
    q[2] = zadd(zadd(zscale(nt[2], E[0]), zscale(nt[4], E[1])), zscale(nt[5], E[2]));
    for (int c = 0; c < 3; ++c) q[c] = zscale(q[c], inv4pi);
    if (p.material_frame) {  // p <- R^T p (rotate<true>, include/Rotation.h:371-394)
      double2 r[3];
      for (int a = 0; a < 3; ++a)
        r[a] = zadd(zadd(zscale(q[0], p.R[0 * 3 + a]), zscale(q[1], p.R[1 * 3 + a])), zscale(q[2], p.R[2 * 3 + a]));
      q[0] = r[0], q[1] = r[1], q[2] = r[2];
    }
    for (int c = 0; c < 3; ++c) p.out[size_t(c) * p.nvox + i] = zscale(q[c], w);
  }
}

// Bin 0 of each volume <- mean of its 6 (4 in 2D) periodic neighbours (src/cudaMain.cu:123-176).
__global__ void k64_dc(double2 *spec, uint32_t nvol, size_t vstride, uint32_t nx, uint32_t ny, uint32_t nz) {
  const uint32_t v = threadIdx.x;
  if (v >= nvol) return;
  double2 *V = spec + size_t(v) * vstride;
  const size_t P = size_t(nx) * ny;
  double2 s = zadd(zadd(V[1], V[nx]), zadd(V[nx - 1], V[size_t(ny - 1) * nx]));
  double cnt = 4.0;
  if (nz > 1) {
    s = zadd(s, zadd(V[P], V[size_t(nz - 1) * P]));
    cnt = 6.0;
  }
  V[0] = zscale(s, 1.0 / cnt);
}

// Weight of the second Ewald plane in double from the float plane position, as the reference's FP64 interpolation.
__device__ __forceinline__ double ewald_weight64(const EwaldGeom &g, uint32_t X, uint32_t Y, uint32_t Z0) {
  const float posx = __fadd_rn(g.start, __fmul_rn(float(X), g.dx));
  const float posy = __fadd_rn(g.start, __fmul_rn(float(Y), g.dy));
  const float ax = __fadd_rn(g.kx, posx), ay = __fadd_rn(g.ky, posy);
  const float val = __fsub_rn(__fsub_rn(__fmul_rn(g.kmag, g.kmag), __fmul_rn(ax, ax)), __fmul_rn(ay, ay));
  const float posz = __fadd_rn(-g.kz, __fsqrt_rn(val));
  return (double(posz) - (double(g.start) + double(__fmul_rn(float(Z0), g.dz)))) / double(g.dz);
}

// Ewald projection in double for every E angle: per detector pixel, the float
// geometry of ewald_geometry, the volumes gathered at the plane(s), per angle
// p_c = sum_b E_b vol[c][b], the intensity at each plane and the linear
// interpolation (1 - d) I0 + d I1 with d formed in double from the float
// plane position (include/uniaxial.h:876-947).  images[a][P] (double).
struct Ewald64Params {
  const double2 *spec;
  size_t vstride;
  uint32_t nbasis;
  uint32_t vol[3][3];
  EwaldGeom g;
  const float *qx, *qy, *qz;
  uint32_t nangles;
  const double *E;          // [nangles][nbasis] (MATERIAL frame: nbasis 1, coefficient 1)
  double *images;           // [nangles][P]
};

__global__ void __launch_bounds__(256) k64_ewald(Ewald64Params p) {
  const EwaldGeom &g = p.g;
  const size_t npix = size_t(g.nx) * g.ny;
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const uint32_t Y = uint32_t(t / g.nx), X = uint32_t(t % g.nx);
  uint32_t zs[2];
  float w1f;
  int nplanes;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (!ewald_geometry(g, X, Y, zs[0], zs[1], w1f, nplanes)) {
    for (uint32_t a = 0; a < p.nangles; ++a) p.images[size_t(a) * npix + t] = nan;
    return;
  }
  const double w1 = nplanes == 2 ? ewald_weight64(g, X, Y, zs[0]) : 0.0;
  const uint32_t ux = igor(X, g.nx), uy = igor(Y, g.ny);
  double2 P[2][3][3];
  double Q[2][3];
  for (int pl = 0; pl < nplanes; ++pl) {
    const uint32_t uz = g.twod ? 0u : igor(zs[pl], g.nz);
    const size_t idx = size_t(ux) + size_t(uy) * g.nx + size_t(uz) * g.nx * g.ny;
    for (uint32_t b = 0; b < p.nbasis; ++b)
      for (int c = 0; c < 3; ++c) P[pl][c][b] = p.spec[size_t(p.vol[c][b]) * p.vstride + idx];
    Q[pl][0] = double(g.kx) + double(p.qx[X]);
    Q[pl][1] = double(g.ky) + double(p.qy[Y]);
    Q[pl][2] = double(g.kz) + (g.twod ? 0.0 : double(p.qz[zs[pl]]));
  }
  const double d = double(g.kmag) * double(g.kmag);
  for (uint32_t a = 0; a < p.nangles; ++a) {
    const double *E = p.E + size_t(a) * p.nbasis;
    double I[2] = {0.0, 0.0};
    for (int pl = 0; pl < nplanes; ++pl) {
      double2 pc[3];
      for (int c = 0; c < 3; ++c) {
        pc[c] = make_double2(0.0, 0.0);
        for (uint32_t b = 0; b < p.nbasis; ++b) pc[c] = zadd(pc[c], zscale(P[pl][c][b], E[b]));
      }
      const double *q = Q[pl];
      const double2 qp = zadd(zadd(zscale(pc[0], q[0]), zscale(pc[1], q[1])), zscale(pc[2], q[2]));
      double r = 0.0;
      for (int c = 0; c < 3; ++c) {
        const double2 tt = zsub(zscale(pc[c], d), zscale(qp, q[c]));
        r += tt.x * tt.x + tt.y * tt.y;
      }
      I[pl] = r;
    }
    p.images[size_t(a) * npix + t] = nplanes == 2 ? (1.0 - w1) * I[0] + w1 * I[1] : I[0];
  }
}

// ---------------------------------------------------------------------------
// Field spectra in double.  Field 7 m + f of material m is w u_x^2, w u_y^2,
// w u_z^2, w u_x u_y, w u_x u_z, w u_y u_z, w phi_ui (f = 0..6; u = sqrt(phi_a) s,
// w the window), and with n^2 - 1 in the place of n^2 (the identity
// phi_a |s|^2 + phi_ui = phi)
//   Nt_ii = sum_m A u_i^2 + B (|u|^2 - u_i^2) + C phi_ui,  Nt_ij = sum_m D u_i u_j.
// Volume j holds fields 2 j and 2 j + 1 as real and imaginary part.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr uint32_t fields64_packed(uint32_t nmat) { return (7 * nmat + 1) / 2; }

// Contrasts over 4 pi of one energy: A = n_par^2 - 1, B = n_perp^2 - 1, C = ((n_par + 2 n_perp) / 3)^2 - 1, D = A - B.
struct Contrast64 {
  double2 A[kMaxMaterials], B[kMaxMaterials], C[kMaxMaterials], D[kMaxMaterials];
};

__global__ void __launch_bounds__(256) k64_build_fields(Build64Params p) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < p.nvox; i += size_t(gridDim.x) * blockDim.x) {
    double w = 1.0;
    if (p.hann_x) {
      const uint32_t X = uint32_t(i % p.nx), Y = uint32_t((i / p.nx) % p.ny), Z = uint32_t(i / (size_t(p.nx) * p.ny));
      w = p.hann_x[X] * p.hann_y[Y] * p.hann_z[Z];
    }
    double pend = 0.0;
    double2 *o = p.out + i;
    uint32_t g = 0;
    auto emit = [&](double v) {
      if (g & 1u)
        o[size_t(g >> 1) * p.nvox] = make_double2(pend, v);
      else
        pend = v;
      ++g;
    };
    for (uint32_t m = 0; m < p.nmat; ++m) {
      double s[4];
      load_s64(p, m, i, s);
      double sx, sy, sz, wa, wu;
      if (p.morphology == 0) {  // Euler: (S, theta, psi, Vfrac)
        double st, ct, sp, cp;
        sincos(s[1], &st, &ct);
        sincos(s[2], &sp, &cp);
        sx = cp * st, sy = sp * st, sz = ct;
        const double phi_a = s[3] * s[0];
        wa = w * phi_a;
        wu = w * (s[3] - phi_a);
      } else {  // vector: (sx, sy, sz, phi_unaligned)
        sx = s[0], sy = s[1], sz = s[2];
        wa = w;
        wu = w * s[3];
      }
      const double ax = wa * sx, ay = wa * sy;
      emit(ax * sx);
      emit(ay * sy);
      emit(wa * sz * sz);
      emit(ax * sy);
      emit(ax * sz);
      emit(ay * sz);
      emit(wu);
    }
    if (g & 1u) o[size_t(g >> 1) * p.nvox] = make_double2(pend, 0.0);
  }
}

struct FieldEwald64Params {
  const double2 *spec;      // [npk][V]
  uint32_t npk, nmat;
  size_t vstride;
  const Contrast64 *con;    // [ne]
  const float *kmag;        // [ne] wave numbers (float, as ewald_geometry takes them)
  uint32_t e0;              // the launch's first energy (blockIdx.y = energy - e0)
  float kvx, kvy, kvz;
  EwaldGeom g;              // kmag, kx, ky, kz filled per energy
  const float *qx, *qy, *qz;
  uint32_t nangles;
  const double *E;          // NB > 0: [nangles][NB]
  const double *map;        // NB = 0: [nangles][3][6]
  double *images;           // [batch][nangles][P]
};

// Ewald projection from the field spectra, for a batch of energies and every
// E angle.  NB = 2 or 3 (LAB frame): per plane the Gram matrix of the scattered
// basis fields, from which each angle takes NB (NB + 1) / 2 multiply-adds;
// NB = 0 (MATERIAL frame): p = map Nt per angle.
template <int NB>
__global__ void __launch_bounds__(128) k64_ewald_fields(FieldEwald64Params p) {
  const uint32_t e = p.e0 + blockIdx.y;
  EwaldGeom g = p.g;
  g.kmag = p.kmag[e];
  g.kx = __fmul_rn(g.kmag, p.kvx), g.ky = __fmul_rn(g.kmag, p.kvy), g.kz = __fmul_rn(g.kmag, p.kvz);
  const size_t npix = size_t(g.nx) * g.ny;
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const uint32_t Y = uint32_t(t / g.nx), X = uint32_t(t % g.nx);
  double *img = p.images + size_t(blockIdx.y) * p.nangles * npix + t;
  uint32_t zs[2];
  float w1f;
  int nplanes;
  if (!ewald_geometry(g, X, Y, zs[0], zs[1], w1f, nplanes)) {
    for (uint32_t a = 0; a < p.nangles; ++a) img[size_t(a) * npix] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const double w1 = nplanes == 2 ? ewald_weight64(g, X, Y, zs[0]) : 0.0;
  const uint32_t ux = igor(X, g.nx), uy = igor(Y, g.ny);
  const uint32_t mx = ux ? g.nx - ux : 0u, my = uy ? g.ny - uy : 0u;
  const Contrast64 &c = p.con[e];
  const double d = double(g.kmag) * double(g.kmag);
  constexpr int NG = NB * (NB + 1) / 2;
  double G[NG > 0 ? NG : 1] = {};
  double2 nt2[2][6];
  double Q2[2][3];
  for (int pl = 0; pl < nplanes; ++pl) {
    double2(&nt)[6] = nt2[NB == 0 ? pl : 0];
    double(&Q)[3] = Q2[NB == 0 ? pl : 0];
    const uint32_t uz = g.twod ? 0u : igor(zs[pl], g.nz), mz = uz ? g.nz - uz : 0u;
    const double2 *za = p.spec + (size_t(uz) * g.ny + uy) * g.nx + ux;
    const double2 *zb = p.spec + (size_t(mz) * g.ny + my) * g.nx + mx;
#pragma unroll
    for (int v = 0; v < 6; ++v) nt[v] = make_double2(0.0, 0.0);
    uint32_t m = 0, f = 0;  // the same in every thread
    auto mac = [](double2 &acc, double2 a, double2 b) {
      acc.x += a.x * b.x - a.y * b.y;
      acc.y += a.x * b.y + a.y * b.x;
    };
    auto add = [&](double2 F) {
      if (m >= p.nmat) return;
      if (f < 3 || f == 6) {
        mac(nt[0], f == 6 ? c.C[m] : f == 0 ? c.A[m] : c.B[m], F);
        mac(nt[3], f == 6 ? c.C[m] : f == 1 ? c.A[m] : c.B[m], F);
        if (NB != 2) mac(nt[5], f == 6 ? c.C[m] : f == 2 ? c.A[m] : c.B[m], F);
      } else if (f == 3) {
        mac(nt[1], c.D[m], F);
      } else if (f == 4) {
        mac(nt[2], c.D[m], F);
      } else {
        mac(nt[4], c.D[m], F);
      }
      if (++f == 7) f = 0, ++m;
    };
    for (uint32_t j = 0; j < p.npk; ++j) {
      const double2 a = __ldg(&za[size_t(j) * p.vstride]), b = __ldg(&zb[size_t(j) * p.vstride]);
      // F_2j = (Z(k) + conj Z(-k)) / 2, F_2j+1 = (Z(k) - conj Z(-k)) / 2i
      add(make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y)));
      add(make_double2(0.5 * (a.y + b.y), 0.5 * (b.x - a.x)));
    }
    Q[0] = double(g.kx) + double(p.qx[X]);
    Q[1] = double(g.ky) + double(p.qy[Y]);
    Q[2] = double(g.kz) + (g.twod ? 0.0 : double(p.qz[zs[pl]]));
    if constexpr (NB > 0) {
      const double w = nplanes == 2 ? (pl == 0 ? 1.0 - w1 : w1) : 1.0;
      double2 tt[NB][3];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const double2 p0 = nt[b], p1 = nt[b == 0 ? 1 : b == 1 ? 3 : 4], p2 = nt[b == 0 ? 2 : b == 1 ? 4 : 5];
        const double2 qp = zadd(zadd(zscale(p0, Q[0]), zscale(p1, Q[1])), zscale(p2, Q[2]));
        tt[b][0] = zsub(zscale(p0, d), zscale(qp, Q[0]));
        tt[b][1] = zsub(zscale(p1, d), zscale(qp, Q[1]));
        tt[b][2] = zsub(zscale(p2, d), zscale(qp, Q[2]));
      }
      int q = 0;
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int b2 = b; b2 < NB; ++b2) {
          double r = 0.0;
#pragma unroll
          for (int i = 0; i < 3; ++i) r += tt[b][i].x * tt[b2][i].x + tt[b][i].y * tt[b2][i].y;
          G[q++] += (b == b2 ? w : 2.0 * w) * r;
        }
    }
  }
  for (uint32_t a = 0; a < p.nangles; ++a) {
    double I = 0.0;
    if constexpr (NB > 0) {
      const double *E = p.E + size_t(a) * NB;
      int q = 0;
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int b2 = b; b2 < NB; ++b2) I += __ldg(&E[b]) * __ldg(&E[b2]) * G[q++];
    } else {
      const double *M = p.map + size_t(a) * 18;
      for (int pl = 0; pl < nplanes; ++pl) {
        double2 pc[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          pc[i] = make_double2(0.0, 0.0);
#pragma unroll
          for (int v = 0; v < 6; ++v) pc[i] = zadd(pc[i], zscale(nt2[pl][v], __ldg(&M[i * 6 + v])));
        }
        const double2 qp = zadd(zadd(zscale(pc[0], Q2[pl][0]), zscale(pc[1], Q2[pl][1])), zscale(pc[2], Q2[pl][2]));
        double r = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double2 s = zsub(zscale(pc[i], d), zscale(qp, Q2[pl][i]));
          r += s.x * s.x + s.y * s.y;
        }
        I += (nplanes == 2 ? (pl == 0 ? 1.0 - w1 : w1) : 1.0) * r;
      }
    }
    img[size_t(a) * npix] = I;
  }
}

// Bilinear blend in double at NPP's float sample position.
__device__ __forceinline__ bool warp_sample64(const double *__restrict__ src, int W, int H, const WarpCoef &c, int xd,
                                              int yd, double &out) {
  WarpTap tp;
  if (!warp_tap(W, H, c, xd, yd, tp)) return false;
  const double fx = tp.fx, fy = tp.fy;
  const double A = src[size_t(tp.y0) * W + tp.x0], B = src[size_t(tp.y0) * W + tp.x1];
  const double C = src[size_t(tp.y1) * W + tp.x0], D = src[size_t(tp.y1) * W + tp.x1];
  out = (1.0 - fy) * ((1.0 - fx) * A + fx * B) + fy * ((1.0 - fx) * C + fx * D);
  return true;
}

// Rotation of every angle's image (NaN prefill), mask, sum and mean in double
// (src/cudaMain.cu:830-909, include/uniaxial.h:958-992).
struct Rotate64Params {
  const double *images;     // [batch = blockIdx.y][nangles][P]
  const WarpCoef *coef;     // [nangles]
  int W, H;
  uint32_t nangles, rot_mask;
  double *avg;              // [batch][P]
};

__global__ void __launch_bounds__(256) k64_rotate_average(Rotate64Params p) {
  const size_t npix = size_t(p.W) * p.H;
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= npix) return;
  const int xd = int(t % p.W), yd = int(t / p.W);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  double sum = 0.0;
  uint32_t count = 0;
  for (uint32_t a = 0; a < p.nangles; ++a) {
    double v = nan;
    warp_sample64(p.images + (size_t(blockIdx.y) * p.nangles + a) * npix, p.W, p.H, p.coef[a], xd, yd, v);
    if (p.rot_mask) {
      if (isnan(v)) continue;
      ++count;
    }
    sum += v;
  }
  p.avg[size_t(blockIdx.y) * npix + t] = p.rot_mask ? (count == 0 ? 0.0 : sum / double(count)) : sum / double(p.nangles);
}

// Detector warp (src/cudaMain.cu:916-960): dst holds the prefill; written where the source falls inside.
__global__ void k64_warp(const double *__restrict__ src, double *__restrict__ dst, int W, int H, WarpCoef c,
                         double prefill, size_t dst_stride) {
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x, npix = size_t(W) * H;
  if (t >= npix) return;
  double v;
  if (!warp_sample64(src + blockIdx.y * npix, W, H, c, int(t % W), int(t / W), v)) v = prefill;
  dst[blockIdx.y * dst_stride + t] = v;
}

}  // namespace cyr
