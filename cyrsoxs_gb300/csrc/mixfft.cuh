// Forward FFT along one axis for every line length that is not a warp-FFT or
// per-thread power of two: mixed radices up to 16 on registers, and Bluestein
// transforms of any other length in one kernel.
//
// A line of M points is transformed in place by S decimation-in-frequency
// stages, M = R_1 ... R_S.  A thread takes one radix-R butterfly at a time on
// registers: it reads R points, transforms them, multiplies by the stage's
// twiddles and writes them back to the slots they came from, so the stages
// share one shared-memory buffer with one block barrier between them.  Stage
// 1 reads global memory and stage S writes it: a line of up to 256 points
// (two stages) meets shared memory once on the way in and once on the way
// out.  The digit-reversed order that an in-place transform leaves is undone
// by the addresses of the last stage's stores.
//
// What bounds it: DRAM, 16 bytes per point (read and write), up to two
// stages; the butterflies cost about 35 instructions a point, and three stages
// are bound by issue and shared memory as much as by DRAM.  The autosort
// Stockham pass that it replaces re-read shared memory once per radix-2..8
// stage with an integer division per butterfly and thread, and was bound by
// issue.  Measured, 11 volumes of 240 x 240 x 90 (135 us at the copy
// bandwidth): x 508 -> 157 us, y 510 -> 147, z 735 -> 154; 450 x 450 x 75
// (395 us): x 1882 -> 706, y 1912 -> 581, z 1921 -> 584.
//
// Column form (y and z lines): a block owns TX adjacent columns; a thread's
// column is threadIdx % TX, so global accesses are runs of TX points, shared
// accesses are free of bank conflicts for every radix and stride, and with
// TX = 32 the butterfly index, its divisions and its twiddles are the same in
// all lanes of a warp.  Row form (x lines): consecutive lanes take
// consecutive butterflies of a row.
//
// Lengths with a prime factor above 13 are convolutions of length M, made of
// the same stages: the forward transform leaves its digit-reversed order in
// shared memory, the last stage multiplies by the kernel's transform and at
// once begins the second transform, whose stages are the transposes of the
// first's, so that order is never undone.
//  * Rader (n prime, M = n - 1 with radices up to 16): with a generator g of
//    the residues mod n, X[g^-k] = x_0 + sum_q x[g^q] W_n^(g^(q - k)).
//  * Bluestein (any other n): with c_j = exp(-i pi j^2 / n),
//    X_k = c_k sum_j (x_j c_j) conj(c_{k-j}), a circular convolution of any
//    length M >= 2 n - 1.
// Measured, 8 volumes of 211 x 211 x 61 (51 us per axis at the copy
// bandwidth), all three axes: 2080 us as gather, FFT, product, FFT and scatter
// kernels over padded lines in memory, 364 us as one kernel per axis; 509
// (Bluestein, 1024 points): 1180 us per axis, bound by its eight stages.
//
// T = float2 for the FP32 engine, double2 for the FP64 pipeline.
#pragma once

#include <type_traits>
#include <utility>

#include "complex.cuh"
#include "fieldbuild.cuh"

namespace cyr {

template <class T>
using Real = decltype(T::x);

// cos(2 pi a / b) and sin(2 pi a / b) at compile time, by Taylor series on [0, pi / 4].
__host__ __device__ constexpr double taylor_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i <= 12; ++i) t *= -x * x / ((2 * i - 1) * (2 * i)), s += t;
  return s;
}
__host__ __device__ constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int i = 1; i <= 12; ++i) t *= -x * x / ((2 * i) * (2 * i + 1)), s += t;
  return s;
}
// octant reduction in integers: angle 2 pi a / b with 0 <= a < b
__host__ __device__ constexpr double cos_2pi(int a, int b) {
  a %= b;
  if (2 * a > b) a = b - a;                            // cos(-t) = cos t
  if (4 * a > b) return -cos_2pi(b - 2 * a, 2 * b);    // cos(pi - t) = -cos t
  return 8 * a <= b ? taylor_cos(6.283185307179586476925286766559 * a / b)
                    : taylor_sin(6.283185307179586476925286766559 * (b - 4 * a) / (4.0 * b));
}
__host__ __device__ constexpr double sin_2pi(int a, int b) { return cos_2pi((4 * a + 3 * b) % (4 * b), 4 * b); }  // sin t = cos(t - pi/2)

template <int N, class F, int... I>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
  static_for_impl<N>(f, std::make_integer_sequence<int, N>{});
}

// v * W_R^m, W_R = exp(-2 pi i / R), with m known at compile time.
template <int R, int M, class T>
__device__ __forceinline__ T mul_root(T v) {
  constexpr int m = M % R;
  using S = Real<T>;
  if constexpr (m == 0) return v;
  else if constexpr (4 * m == R) return T{v.y, -v.x};
  else if constexpr (2 * m == R) return T{-v.x, -v.y};
  else if constexpr (4 * m == 3 * R) return T{-v.y, v.x};
  else if constexpr (8 * m == R) {
    constexpr S h = S(cos_2pi(1, 8));
    return T{h * (v.x + v.y), h * (v.y - v.x)};
  } else if constexpr (8 * m == 3 * R) {
    constexpr S h = S(cos_2pi(1, 8));
    return T{h * (v.y - v.x), -h * (v.x + v.y)};
  } else {
    constexpr S c = S(cos_2pi(m, R)), s = S(sin_2pi(m, R));
    return T{v.x * c + v.y * s, v.y * c - v.x * s};
  }
}

// Radix-R transforms on registers, natural order in and out.
template <int R, class T>
__device__ __forceinline__ void dft_reg(T (&v)[R]);

// Odd prime R: X_k and X_{R-k} from the sums and differences of v_j and v_{R-j}.
template <int R, class T>
__device__ __forceinline__ void dft_prime(T (&v)[R]) {
  constexpr int H = (R - 1) / 2;
  using S = Real<T>;
  T s[H], d[H], x0 = v[0];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    s[j] = cadd(v[j + 1], v[R - 1 - j]);
    d[j] = csub(v[j + 1], v[R - 1 - j]);
    v[0] = cadd(v[0], s[j]);
  }
  static_for<H>([&](auto ki) {
    constexpr int k = decltype(ki)::value + 1;
    T a = x0, b{};
    static_for<H>([&](auto ji) {
      constexpr int j = decltype(ji)::value + 1;
      constexpr S c = S(cos_2pi(j * k, R)), sn = S(sin_2pi(j * k, R));
      a = cfma(c, s[j - 1], a);
      if constexpr (j == 1)
        b = T{sn * d[0].x, sn * d[0].y};
      else
        b = cfma(sn, d[j - 1], b);
    });
    v[k] = T{a.x + b.y, a.y - b.x};
    v[R - k] = T{a.x - b.y, a.y + b.x};
  });
}

// The k in [0, A B) with k = a mod A and k = b mod B.
__host__ __device__ constexpr int crt(int a, int A, int b, int B) {
  while (a % B != b) a += A;
  return a;
}

// R = A B with A and B coprime (Good-Thomas): no twiddles, the index maps are compile-time.
template <int A, int B, class T>
__device__ __forceinline__ void dft_coprime(T (&v)[A * B]) {
  constexpr int R = A * B;
  T w[R];
  static_for<B>([&](auto bi) {
    constexpr int b = decltype(bi)::value;
    T t[A];
    static_for<A>([&](auto ai) { t[decltype(ai)::value] = v[(B * decltype(ai)::value + A * b) % R]; });
    dft_reg<A>(t);
    static_for<A>([&](auto ai) { w[decltype(ai)::value * B + b] = t[decltype(ai)::value]; });
  });
  static_for<A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    T t[B];
    static_for<B>([&](auto bi) { t[decltype(bi)::value] = w[a * B + decltype(bi)::value]; });
    dft_reg<B>(t);
    static_for<B>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      constexpr int k = crt(a, A, b, B);
      v[k] = t[b];
    });
  });
}

// R = A B with twiddles W_R^(k1 b) between the two factors.
template <int A, int B, class T>
__device__ __forceinline__ void dft_composite(T (&v)[A * B]) {
  constexpr int R = A * B;
  T w[R];
  static_for<B>([&](auto bi) {
    constexpr int b = decltype(bi)::value;
    T t[A];
    static_for<A>([&](auto ai) { t[decltype(ai)::value] = v[decltype(ai)::value * B + b]; });
    dft_reg<A>(t);
    static_for<A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      w[a * B + b] = mul_root<R, a * b>(t[a]);
    });
  });
  static_for<A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    T t[B];
    static_for<B>([&](auto bi) { t[decltype(bi)::value] = w[a * B + decltype(bi)::value]; });
    dft_reg<B>(t);
    static_for<B>([&](auto bi) { v[a + A * decltype(bi)::value] = t[decltype(bi)::value]; });
  });
}

template <int R, class T>
__device__ __forceinline__ void dft_reg(T (&v)[R]) {
  if constexpr (R == 2) {
    const T a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const T t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
    const T t4{t3.y, -t3.x};
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t4);
    v[3] = csub(t1, t4);
  } else if constexpr (R == 3 || R == 5 || R == 7 || R == 11 || R == 13) {
    dft_prime<R>(v);
  } else if constexpr (R == 6) {
    dft_coprime<2, 3>(v);
  } else if constexpr (R == 8) {
    dft_composite<2, 4>(v);
  } else if constexpr (R == 9) {
    dft_composite<3, 3>(v);
  } else if constexpr (R == 10) {
    dft_coprime<2, 5>(v);
  } else if constexpr (R == 12) {
    dft_coprime<4, 3>(v);
  } else if constexpr (R == 14) {
    dft_coprime<2, 7>(v);
  } else if constexpr (R == 15) {
    dft_coprime<3, 5>(v);
  } else {
    static_assert(R == 16, "radix");
    dft_composite<4, 4>(v);
  }
}

// ---------------------------------------------------------------------------
// Plans.  Stage s works on blocks of L_s = M / (R_1 ... R_{s-1}) points: the
// butterfly (block, j), j < m = L_s / R_s, takes the points block L_s + j +
// q m.  `block` and `span` are L_s and m in shared-memory slots, with the row
// form's padding.
// ---------------------------------------------------------------------------
constexpr int kMixMaxStages = 8;
constexpr int kMixMaxRadix = 16;

struct MixStage {
  uint32_t radix;
  uint32_t nb;               // butterflies per line, M / radix
  uint32_t nb_magic;         // ceil(2^32 / nb): t / nb = umulhi(t, magic) for t nb < 2^32
  uint32_t m, m_magic;       // butterflies per block
  uint32_t block, span;
  uint32_t tw;               // this stage's twiddles W_L^(j k), k < radix rounded up to even: at tw + j (that) + k
                             // (column form), tw + k m + j (row form)
};

template <class T>
struct MixParams {
  T *data;
  uint32_t nx, ny;
  size_t vstride;            // elements between volumes (blockIdx.y)
  uint32_t nlines;           // row form: rows per volume; column form: columns per `other`
  size_t ostride;            // column form: elements between successive "others" (y pass: planes)
  uint32_t tiles;            // column form: tiles per `other`
  uint32_t estride;          // elements between the points of a line
  uint32_t lg_tx;            // column form: log2 of the columns per block
  uint32_t rows;             // row form: rows per block
  uint32_t n, M;             // line length; transform length (n, or the Bluestein padding)
  uint32_t ns;
  uint32_t line_slots;       // row form: slots per line
  uint32_t pad, rs, rs_magic;  // row form: pad = 1 adds one slot per rs points (rs = R_S even)
  MixStage st[kMixMaxStages];
  const T *tw;
  const uint32_t *first;     // [M / R_S]: slot of the block that holds frequencies fb + k M / R_S
  const T *chirp, *bhat;     // Bluestein: c_j (j < n); both convolutions: FFT_M(kernel) / M in frequency order
  const uint32_t *in, *out;  // Rader: g^q and g^-q mod n
};

enum MixForm : int { kMixPlain = 0, kMixBluestein = 1, kMixRader = 2 };

__device__ __forceinline__ uint32_t mix_div(uint32_t t, uint32_t d, uint32_t magic) {
  return d == 1 ? t : __umulhi(t, magic);
}

// v[k] *= W_L^(j k).  Column form: the lanes of a warp share j, and a
// butterfly's twiddles are contiguous (two per 16-byte load, one broadcast
// each).  Row form: the lanes hold consecutive j, and so do the tables.
template <int R, bool COL, class T>
__device__ __forceinline__ void mix_twiddle(T (&v)[R], const T *__restrict__ tw, uint32_t j, uint32_t m) {
  if constexpr (COL && sizeof(T) == 8) {
    const float4 *t4 = reinterpret_cast<const float4 *>(tw + j * ((R + 1) & ~1));
#pragma unroll
    for (int k = 0; k < R; k += 2) {
      const float4 w = __ldg(&t4[k / 2]);
      if (k) v[k] = cmul(v[k], T{w.x, w.y});
      if (k + 1 < R) v[k + 1] = cmul(v[k + 1], T{w.z, w.w});
    }
  } else {
#pragma unroll
    for (int k = 1; k < R; ++k) v[k] = cmul(v[k], __ldg(&tw[COL ? j * ((R + 1) & ~1) + k : k * m + j]));
  }
}

// f(integral_constant<int, R>) for the stage's radix.
template <class F>
__device__ __forceinline__ void mix_radix(uint32_t radix, F &&f) {
  switch (radix) {
#define CYR_MIX_R(r) \
  case r: f(std::integral_constant<int, r>{}); break;
    CYR_MIX_R(2) CYR_MIX_R(3) CYR_MIX_R(4) CYR_MIX_R(5) CYR_MIX_R(6) CYR_MIX_R(7) CYR_MIX_R(8) CYR_MIX_R(9)
    CYR_MIX_R(10) CYR_MIX_R(11) CYR_MIX_R(12) CYR_MIX_R(13) CYR_MIX_R(14) CYR_MIX_R(15) CYR_MIX_R(16)
#undef CYR_MIX_R
  }
}

// 256 threads at 64 registers: four blocks per SM, whose loads, stages and
// stores overlap (two blocks of 512 threads: 240-point z lines 174 us against 154 us).
constexpr int kMixThreads = 256;

// A block's lines, as the stage loops below see them.  COL: thread =
// (butterfly, column); the loop over butterflies is the same for every lane
// of a column group.  ROW: thread = (line, butterfly).
template <class T, bool COL>
struct MixTile {
  const MixParams<T> &p;
  T *sm;
  T *g;             // first point of the tile's first line
  uint32_t valid;   // lines of the tile that exist
  uint32_t lane;    // COL: this thread's column

  // body(line pointer in global memory, line's first slot, butterfly, whether the line exists)
  template <class F>
  __device__ __forceinline__ void each(const MixStage &st, F &&body) const {
    if constexpr (COL) {
      const uint32_t step = blockDim.x >> p.lg_tx;
      for (uint32_t b = threadIdx.x >> p.lg_tx; b < st.nb; b += step) body(g + lane, sm + lane, b, lane < valid);
    } else {
      const uint32_t total = valid * st.nb;
      for (uint32_t t = threadIdx.x; t < total; t += blockDim.x) {
        const uint32_t l = mix_div(t, st.nb, st.nb_magic);
        body(g + size_t(l) * p.nx, sm + size_t(l) * p.line_slots, t - l * st.nb, true);
      }
    }
  }
  // element offset of slot s
  __device__ __forceinline__ uint32_t at(uint32_t s) const { return COL ? s << p.lg_tx : s; }
  __device__ __forceinline__ uint32_t gat(uint32_t i) const { return COL ? i * p.estride : i; }
  // slot offset of butterfly j inside its block
  __device__ __forceinline__ uint32_t jslot(uint32_t j) const {
    return COL || !p.pad ? j : j + mix_div(j, p.rs, p.rs_magic);
  }
};

// A stage between the first and the last; inverse: its transpose, for the second transform of a convolution.
template <class T, bool COL, class Tile>
__device__ __forceinline__ void mix_middle(const MixParams<T> &p, const Tile &tile, const MixStage &st, bool inverse) {
  mix_radix(st.radix, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    tile.each(st, [&](T *, T *s, uint32_t b, bool) {
      const uint32_t blk = mix_div(b, st.m, st.m_magic), j = b - blk * st.m;
      T *e = s + tile.at(blk * st.block + tile.jslot(j));
      T v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = e[tile.at(q * st.span)];
      if (inverse) mix_twiddle<R, COL>(v, p.tw + st.tw, j, st.m);
      dft_reg<R>(v);
      if (!inverse) mix_twiddle<R, COL>(v, p.tw + st.tw, j, st.m);
#pragma unroll
      for (int k = 0; k < R; ++k) e[tile.at(k * st.span)] = v[k];
    });
  });
}

template <class T, bool COL, int FORM>
__global__ void __launch_bounds__(kMixThreads, sizeof(T) == 8 ? 4 : 2) k_mix_fft(const __grid_constant__ MixParams<T> p) {
  extern __shared__ unsigned char mix_smem[];
  MixTile<T, COL> tile{p, reinterpret_cast<T *>(mix_smem), nullptr, 0, 0};
  T *vol = p.data + size_t(blockIdx.y) * p.vstride;
  if constexpr (COL) {
    const uint32_t tx = 1u << p.lg_tx, other = blockIdx.x / p.tiles, c0 = (blockIdx.x % p.tiles) * tx;
    tile.g = vol + size_t(other) * p.ostride + c0;
    tile.valid = min(tx, p.nlines - c0);
    tile.lane = threadIdx.x & (tx - 1);
  } else {
    const uint32_t r0 = blockIdx.x * p.rows;
    tile.g = vol + size_t(r0) * p.nx;
    tile.valid = min(p.rows, p.nlines - r0);
  }
  // stage 1: global -> shared (a single-stage line goes straight back to global)
  {
    const MixStage &st = p.st[0];
    mix_radix(st.radix, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      tile.each(st, [&](T *g, T *s, uint32_t b, bool ok) {
        T v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const uint32_t i = b + q * st.m;
          v[q] = T{};
          if (FORM == kMixBluestein) {
            if (ok && i < p.n) v[q] = cmul(g[tile.gat(i)], __ldg(&p.chirp[i]));
          } else if (ok) {
            v[q] = g[tile.gat(FORM == kMixRader ? __ldg(&p.in[i]) : i)];
          }
        }
        dft_reg<R>(v);
        if (FORM == kMixPlain && p.ns == 1) {
          if (ok)
#pragma unroll
            for (int k = 0; k < R; ++k) g[tile.gat(uint32_t(k))] = v[k];
          return;
        }
        mix_twiddle<R, COL>(v, p.tw + st.tw, b, st.m);
        const uint32_t j = tile.jslot(b);
#pragma unroll
        for (int k = 0; k < R; ++k) s[tile.at(j + k * st.span)] = v[k];
      });
    });
  }
  if (FORM == kMixPlain && p.ns == 1) return;
  for (uint32_t s = 1; s + 1 < p.ns; ++s) {
    __syncthreads();
    mix_middle<T, COL>(p, tile, p.st[s], false);
  }
  __syncthreads();
  // last stage: blocks of R consecutive points, frequencies fb + k M / R
  {
    const MixStage &st = p.st[p.ns - 1];
    mix_radix(st.radix, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      tile.each(st, [&](T *g, T *s, uint32_t fb, bool ok) {
        T *e = s + tile.at(__ldg(&p.first[fb]));
        T v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = e[tile.at(uint32_t(q))];
        dft_reg<R>(v);
        if constexpr (FORM != kMixPlain) {
          // product with the chirp's transform, conjugated: the second (forward) transform then gives the conjugate
#pragma unroll
          for (int k = 0; k < R; ++k) {
            T w = cmul(v[k], __ldg(&p.bhat[fb + k * st.nb]));
            if (FORM == kMixRader && k == 0 && fb == 0 && ok) {
              // frequency 0: the sum of x_1 ... x_{n-1}; adding x_0 to its product adds x_0 to every output
              const T x0 = g[0];
              g[0] = cadd(x0, v[0]);
              w = cadd(w, x0);
            }
            v[k] = T{w.x, -w.y};
          }
          dft_reg<R>(v);
#pragma unroll
          for (int q = 0; q < R; ++q) e[tile.at(uint32_t(q))] = v[q];
        } else if (ok) {
#pragma unroll
          for (int k = 0; k < R; ++k) g[tile.gat(fb + k * st.nb)] = v[k];
        }
      });
    });
  }
  if constexpr (FORM != kMixPlain) {
    for (uint32_t s = p.ns - 2; s >= 1; --s) {
      __syncthreads();
      mix_middle<T, COL>(p, tile, p.st[s], true);
    }
    __syncthreads();
    const MixStage &st = p.st[0];
    mix_radix(st.radix, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      tile.each(st, [&](T *g, T *s, uint32_t b, bool ok) {
        const T *e = s + tile.at(tile.jslot(b));
        T v[R];
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = e[tile.at(k * st.span)];
        mix_twiddle<R, COL>(v, p.tw + st.tw, b, st.m);
        dft_reg<R>(v);
        if (ok)
#pragma unroll
          for (int q = 0; q < R; ++q) {
            const uint32_t i = b + q * st.m;
            if (FORM == kMixRader)
              g[tile.gat(__ldg(&p.out[i]))] = T{v[q].x, -v[q].y};
            else if (i < p.n)
              g[tile.gat(i)] = cmul(__ldg(&p.chirp[i]), T{v[q].x, -v[q].y});
          }
      });
    });
  }
}

// Field build fused with the x pass for the row lengths that k_mix_fft takes in two stages or more
// (mixbuild.cu): the general form of k_build_fields_rows.
struct MixBuildParams {
  FieldParams f;
  MixParams<float2> m;       // row form: tables and stages; rows = rows per block
  const uint32_t *slot;      // [nx]: shared-memory slot of element x of a line
  uint32_t npk, npk_magic;
  uint32_t form;             // 5 (morphology) + material count up to 4 (0: any)
};
cudaError_t mix_build_launch(dim3 grid, size_t smem, cudaStream_t st, const MixBuildParams &p);
const void *mix_build_kernel();

// The kernel instances live in translation units of their own (mixfft_f32.cu, mixfft_f64.cu).
template <class T>
cudaError_t mix_launch(MixForm form, bool row, dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                       const MixParams<T> &p);
template <class T>
const void *mix_kernel(MixForm form, bool row);

}  // namespace cyr
