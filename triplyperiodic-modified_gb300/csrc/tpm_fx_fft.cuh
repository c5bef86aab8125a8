// Pencil transforms of the FP64 path in 64-bit fixed point (tpm_fx.cuh), for
// pencils of at most kFxMaxPoints points; included by tpm_fft.cu.
//
// A block transforms npen = 2^lq pencils.  The first stage's inputs stay in
// registers while the block finds each pencil's largest exponent, and so do
// the last stage's outputs, so a two-stage plan (256 = 16 x 16 points)
// crosses shared memory once.  Between stages element t of pencil q lies at
// t * npen + q (consecutive lanes take consecutive pencils: no conflicts).
// The shift after the first stage is applied by the second one when it reads
// its inputs, which needs no barrier of its own.
#pragma once

#include "tpm_fx.cuh"

namespace tpm {
namespace {

// The longest pencil.  Up to it the error is below that of FP64 for every length and
// kind of data but a single mode, which FP64 transforms nearly exactly
// (tests/fx_check.cpp); for white data it is above for most lengths from 320 points
// (1.0 to 1.5 times) and twice that of FP64 from 675.
constexpr int kFxMaxPoints = 256;
constexpr int kFxThreads = 256;    // threads per block of the x passes
constexpr int kFxItems = 128;      // threads per block of the y and z passes at most
constexpr int kFxPens = 32;        // pencils per block at most

// scales of a block's pencils
struct FxScales {
  unsigned emax[kFxPens];      // largest exponent field
  unsigned units[2][kFxPens];  // sums of moduli (forward; inverse in the z pass)
};

__device__ __forceinline__ void fx_scales_clear(FxScales &sc) {
  if (threadIdx.x < kFxPens) {
    sc.emax[threadIdx.x] = kFxExpMin;
    sc.units[0][threadIdx.x] = sc.units[1][threadIdx.x] = 0;
  }
  __syncthreads();
}

// over the lanes of a warp that hold the same pencil (lane mod npen)
__device__ __forceinline__ unsigned fx_lanes_max(unsigned v, int lq) {
  for (int o = 1 << lq; o < 32; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ unsigned fx_lanes_sum(unsigned v, int lq) {
  for (int o = 1 << lq; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// First stage from global memory (load(q, t): a point as doubles): one item
// per thread, the launch gives (n / R) npen <= blockDim.x.
template <int R, int SIGN, typename Load>
__device__ __forceinline__ void fx_first(const FxPlan &pl, int lq, FxScales &sc, fx2 *out,
                                         Load &&load) {
  const int m = pl.n / R, q = threadIdx.x & ((1 << lq) - 1), i = threadIdx.x >> lq;
  const bool on = i < m;
  double2 raw[R];
  unsigned e = 0;
#pragma unroll
  for (int t = 0; t < R; ++t) raw[t] = on ? load(q, i + t * m) : make_double2(0, 0);
#pragma unroll
  for (int t = 0; t < R; ++t) e = max(e, max(fx_exp(raw[t].x), fx_exp(raw[t].y)));
  e = fx_lanes_max(e, lq);
  if ((threadIdx.x & 31) < (1 << lq)) atomicMax(&sc.emax[q], e);
  __syncthreads();
  e = sc.emax[q];
  fx2 v[R];
  unsigned part = 0;
#pragma unroll
  for (int t = 0; t < R; ++t) {
    v[t] = {fx_from(raw[t].x, e), fx_from(raw[t].y, e)};
    part += fx_part(v[t]);
  }
  const unsigned units = fx_lanes_sum(on ? fx_units(part) : 0u, lq);
  if ((threadIdx.x & 31) < (1 << lq)) atomicAdd(&sc.units[0][q], units);
  fx_dft<R, SIGN>(v);
  if (on) {
#pragma unroll
    for (int u = 0; u < R; ++u) out[((i * R + u) << lq) + q] = v[u];
  }
}

// First stage of rows staged in shared memory (their exponents known); `twice`
// leaves room for twice the sum of moduli
template <int R, int SIGN, typename Load>
__device__ __forceinline__ void fx_first_staged(const FxPlan &pl, int lq, FxScales &sc, fx2 *out,
                                                int twice, Load &&load) {
  const int m = pl.n / R, q = threadIdx.x & ((1 << lq) - 1);
  const unsigned e = sc.emax[q];
  unsigned units = 0;
  for (int idx = threadIdx.x; idx < (m << lq); idx += blockDim.x) {
    const int i = idx >> lq;
    fx2 v[R];
    unsigned part = 0;
#pragma unroll
    for (int t = 0; t < R; ++t) {
      v[t] = load(q, i + t * m, e);
      part += fx_part(v[t]);
    }
    units += fx_units(part);
    fx_dft<R, SIGN>(v);
#pragma unroll
    for (int u = 0; u < R; ++u) out[((i * R + u) << lq) + q] = v[u];
  }
  units = fx_lanes_sum(units << twice, lq);
  if ((threadIdx.x & 31) < (1 << lq)) atomicAdd(&sc.units[0][q], units);
}

// the inputs of one butterfly of a later stage, twiddled; `shift`: the second
// stage shifts them first
template <int R>
__device__ __forceinline__ void fx_inputs(const FxPlan &pl, const fx2 *a, int lq, int q, int i,
                                          int k, int p, bool second, const FxShift &shift,
                                          fx2 *v) {
  const int m = pl.n / R;
  const FxTw *tw = pl.tw + (p - 1) + k * (R - 1) - 1;
#pragma unroll
  for (int t = 0; t < R; ++t) {
    v[t] = a[((i + t * m) << lq) + q];
    if (second) v[t] = fx_shift(v[t], shift, t & 1);
  }
  if (k > 0) {  // (k = 0: by 1, exact)
#pragma unroll
    for (int t = 1; t < R; ++t) v[t] = fx_cmul(v[t], tw[t]);
  }
}

// A later stage of radix R: put(q, point, value)
template <int R, int SIGN, typename Put>
__device__ __forceinline__ void fx_stage(const FxPlan &pl, const fx2 *a, int lq, int s, int p,
                                         const unsigned *units, Put &&put) {
  // (units is null where the first stage's inputs were scaled)
  const int m = pl.n / R, q = threadIdx.x & ((1 << lq) - 1);
  const bool second = s == 1 && units;
  const FxShift shift = fx_shift_of(second ? fx_bits_over(units[q]) : 0);
  for (int idx = threadIdx.x; idx < (m << lq); idx += blockDim.x) {
    const int i = idx >> lq, ip = fdiv(i, pl.pmag[s]), k = i - ip * p;
    fx2 v[R];
    fx_inputs<R>(pl, a, lq, q, i, k, p, second, shift, v);
    fx_dft<R, SIGN>(v);
    const int j = ip * p * R + k;
#pragma unroll
    for (int u = 0; u < R; ++u) put(q, j + u * p, v[u]);
  }
}

#define TPM_FX_RADIX(R_, CALL)       \
  switch (R_) {                      \
    case 16: CALL(16); break;        \
    case 8: CALL(8); break;          \
    case 5: CALL(5); break;          \
    case 4: CALL(4); break;          \
    case 3: CALL(3); break;          \
    case 2: CALL(2); break;          \
    default: CALL(1); break;         \
  }

// Stages 1 .. nst - 1 from buffer a (b is the other one), the last one's
// outputs to put.  Starts and ends each stage but the last with a barrier.
template <int SIGN, typename Put>
__device__ __forceinline__ void fx_rest(const FxPlan &pl, fx2 *a, fx2 *b, int lq,
                                        const unsigned *units, Put &&put) {
  int p = pl.radix[0];
  for (int s = 1; s < pl.nst; ++s) {
    __syncthreads();
    const int R = pl.radix[s];
    if (s < pl.nst - 1) {
      auto mid = [&](int q, int t, fx2 v) { b[(t << lq) + q] = v; };
#define TPM_FX_CALL(N) fx_stage<N, SIGN>(pl, a, lq, s, p, units, mid)
      TPM_FX_RADIX(R, TPM_FX_CALL)
#undef TPM_FX_CALL
      fx2 *t = a;
      a = b;
      b = t;
    } else {
#define TPM_FX_CALL(N) fx_stage<N, SIGN>(pl, a, lq, s, p, units, put)
      TPM_FX_RADIX(R, TPM_FX_CALL)
#undef TPM_FX_CALL
    }
    p *= R;
  }
}

// the scale of pencil q after its transform, and `more` bits
__device__ __forceinline__ int fx_scale_of(const FxScales &sc, int q, int more) {
  return fx_scale(sc.emax[q], fx_bits_over(sc.units[0][q]) + more);
}

// ------------------------------------------------------------------ y passes
// (five blocks per SM: 128^3 22.8 us, with four 29.3; 256^3 116 us, with four 3 % more)
template <int SIGN>
__global__ void __launch_bounds__(kFxItems, 5)
k_fx_y(Grid g, FxPlan pl, double2 *__restrict__ spec, int lq, const int *__restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FxScales sc;
  fx2 *a = reinterpret_cast<fx2 *>(smem_raw), *b = a + (pl.n << lq);
  const int npen = 1 << lq, tiles = (g.nxh + npen - 1) >> lq;
  const int kz = blockIdx.x / tiles, kx0 = (blockIdx.x - kz * tiles) << lq;
  double2 *base = spec + (long long)kz * g.ny * g.sxh + kx0;
  auto load = [&](int q, int ky) {
    return kx0 + q < g.nxh ? base[ky * g.sxh + q] : make_double2(0, 0);
  };
  fx_scales_clear(sc);
#define TPM_FX_CALL(N) fx_first<N, SIGN>(pl, lq, sc, a, load)
  TPM_FX_RADIX(pl.radix[0], TPM_FX_CALL)
#undef TPM_FX_CALL
  fx_rest<SIGN>(pl, a, b, lq, sc.units[0], [&](int q, int ky, fx2 v) {
    if (kx0 + q < g.nxh) {
      const int k = fx_scale_of(sc, q, 0);
      base[ky * g.sxh + q] = make_double2(fx_to(v.x, k), fx_to(v.y, k));
    }
  });
}

// ------------------------------------------- z pass with the wave-number divide
// The table holds inv = 1/(ax + ay + az) of each mode as inv 2^(62 - e0) with
// 2^e0 above the pencil's largest (inv_e[ky nxh + kx] = e0), its low six bits
// a further right shift, so that a small reciprocal keeps 56 bits; the zero
// mode's is 1.  The inverse plan takes the forward one's radices in reverse,
// so the last forward butterfly of a thread leaves exactly the modes of an
// inverse first one: divide and inverse stage follow in registers, one item
// per thread.  The quotients' sum of moduli is known before that stage and
// scales them there (its plan's second stage shifts no more).
template <int R>
__device__ __forceinline__ void fx_z_middle(const FxPlan &pl, const fx2 *a, fx2 *out, int lq, int s,
                                            int p, FxScales &sc, const long long *inv,
                                            long long inv_step, bool in) {
  const int m = pl.n / R, q = threadIdx.x & ((1 << lq) - 1), i = threadIdx.x >> lq;
  const bool on = i < m;  // (the last stage's span is m: k = i)
  fx2 v[R];
  unsigned part = 0;
  if (on) {
    long long w[R];
#pragma unroll
    for (int u = 0; u < R; ++u) w[u] = in ? inv[(i + u * m) * inv_step + q] : 0;
    const FxShift shift = fx_shift_of(s == 1 ? fx_bits_over(sc.units[0][q]) : 0);
    fx_inputs<R>(pl, a, lq, q, i, i, p, s == 1, shift, v);
    fx_dft<R, -1>(v);
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const fxw f = fx_split(w[u]);
      const int d = (int)w[u] & 63;
      v[u] = {fx_mul(v[u].x, f) >> d, fx_mul(v[u].y, f) >> d};
      part += fx_part(v[u]);
    }
  }
  const unsigned units = fx_lanes_sum(on ? fx_units(part) : 0u, lq);
  if ((threadIdx.x & 31) < (1 << lq)) atomicAdd(&sc.units[1][q], units);
  __syncthreads();
  if (on) {
    const FxShift shift = fx_shift_of(fx_bits_over(sc.units[1][q]));
#pragma unroll
    for (int u = 0; u < R; ++u) v[u] = fx_shift(v[u], shift, u & 1);
    fx_dft<R, +1>(v);
#pragma unroll
    for (int u = 0; u < R; ++u) out[((i * R + u) << lq) + q] = v[u];
  }
}

__global__ void __launch_bounds__(kFxItems, 3)
k_fx_z_solve(Grid g, FxPlan pl, FxPlan pli, double2 *__restrict__ spec,
             const long long *__restrict__ inv, const int *__restrict__ inv_e, int lq,
             const int *__restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FxScales sc;
  fx2 *a = reinterpret_cast<fx2 *>(smem_raw), *b = a + (pl.n << lq);
  const int npen = 1 << lq, tiles = (g.nxh + npen - 1) >> lq;
  const int ky = blockIdx.x / tiles, kx0 = (blockIdx.x - ky * tiles) << lq;
  const long long plane = (long long)g.ny * g.sxh, iplane = (long long)g.ny * g.nxh;
  double2 *base = spec + (long long)ky * g.sxh + kx0;
  const long long *ib = inv + (long long)ky * g.nxh + kx0;
  const int myq = threadIdx.x & (npen - 1);
  const bool in = kx0 + myq < g.nxh;
  const int e0 = in ? inv_e[ky * g.nxh + kx0 + myq] : 0;
  auto load = [&](int q, int kz) { return in ? base[kz * plane + q] : make_double2(0, 0); };
  fx_scales_clear(sc);
#define TPM_FX_CALL(N) fx_first<N, -1>(pl, lq, sc, a, load)
  TPM_FX_RADIX(pl.radix[0], TPM_FX_CALL)
#undef TPM_FX_CALL
  int p = pl.radix[0];
  int s = 1;
  for (; s < pl.nst - 1; ++s) {
    __syncthreads();
    auto mid = [&](int q, int t, fx2 v) { b[(t << lq) + q] = v; };
#define TPM_FX_CALL(N) fx_stage<N, -1>(pl, a, lq, s, p, sc.units[0], mid)
    TPM_FX_RADIX(pl.radix[s], TPM_FX_CALL)
#undef TPM_FX_CALL
    fx2 *t = a;
    a = b;
    b = t;
    p *= pl.radix[s];
  }
  __syncthreads();
#define TPM_FX_CALL(N) fx_z_middle<N>(pl, a, b, lq, s, p, sc, ib, iplane, in)
  TPM_FX_RADIX(pl.radix[s], TPM_FX_CALL)
#undef TPM_FX_CALL
  fx_rest<+1>(pli, b, a, lq, nullptr, [&](int q, int kz, fx2 v) {
    if (in) {
      const int k = fx_scale_of(sc, q, 2 + e0 + fx_bits_over(sc.units[1][q]));
      base[kz * plane + q] = make_double2(fx_to(v.x, k), fx_to(v.y, k));
    }
  });
}

// that table
__global__ void k_fx_inv(Grid g, const double *__restrict__ ax, const double *__restrict__ ay,
                         const double *__restrict__ az, long long *__restrict__ inv,
                         int *__restrict__ inv_e) {
  const int total = g.nxh * g.ny;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < total; m += gridDim.x * blockDim.x) {
    const int ky = m / g.nxh, kx = m - ky * g.nxh;
    const double axy = ax[kx] + ay[ky];
    // az is smallest (zero) at kz = 0, next smallest at kz = 1
    double top = kx + ky > 0 ? 1.0 / (axy + az[0]) : 1.0;
    if (kx + ky == 0 && g.nz > 1) top = fmax(top, 1.0 / (axy + az[1]));
    const int e0 = (int)(fx_exp(top) >> 20) - 1022;
    for (int kz = blockIdx.y; kz < g.nz; kz += gridDim.y) {
      const double v = kx + ky + kz > 0 ? 1.0 / (axy + az[kz]) : 1.0;
      // v = f 2^e, f in [1/2, 1): f 2^62 with the low six bits for e0 - e
      const int e = (int)(fx_exp(v) >> 20) - 1022;
      const long long f = (long long)((fx_bits(v) & 0xfffffffffffffull) | 0x10000000000000ull) << 9;
      inv[(long long)kz * total + m] = f | (e0 - e < 63 ? e0 - e : 63);
    }
    if (blockIdx.y == 0) inv_e[m] = e0;
  }
}

// ------------------------------------------------------------------ x passes
// A warp per row (several warps per row when the block has more warps than
// rows): f(row, q, i) for i = 0 .. count - 1
template <typename F>
__device__ __forceinline__ void fx_rows(int npen, long long row0, long long nrows, int count,
                                        F &&f) {
  const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpr = nw > npen ? nw / npen : 1;  // warps per row
  for (int rw = w; rw < npen * wpr; rw += nw) {
    const int q = rw / wpr, part = rw - q * wpr;
    f(row0 + q, q, part * 32 + lane, wpr * 32, row0 + q < nrows, count);
  }
}

__host__ __device__ __forceinline__ int fx_row_pitch(int n) { return n | 1; }  // odd: no conflicts

// dynamic shared memory of the x passes: the staged rows (inverse: Nx/2 + 1
// modes each) and the other buffer
__host__ __device__ __forceinline__ int fx_x_smem(int n, int npen) {
  return npen * (fx_row_pitch(n + 1) + fx_row_pitch(n)) * 16;
}

// the transform of the staged rows: first stage from `load`, the result row by
// row (pitch sp) in the returned buffer
template <int SIGN, typename Load>
__device__ __forceinline__ fx2 *fx_row_transform(const FxPlan &pl, int lq, FxScales &sc, fx2 *s,
                                                 fx2 *a, int sp, Load &&load) {
#define TPM_FX_CALL(N) fx_first_staged<N, SIGN>(pl, lq, sc, a, SIGN < 0, load)
  TPM_FX_RADIX(pl.radix[0], TPM_FX_CALL)
#undef TPM_FX_CALL
  fx2 *z = (pl.nst & 1) ? a : s;  // the buffer the last stage does not read
  fx_rest<SIGN>(pl, a, s, lq, sc.units[0], [&](int q, int t, fx2 v) { z[q * sp + t] = v; });
  __syncthreads();
  return z;
}

// The x passes run three blocks of 256 threads per SM (at most 85 registers):
// with two, 16 warps left the waits for rows and barriers uncovered (256^3,
// inverse: 244 us; single cells 267, with two blocks 314; a fourth block spills, 285).
//
// forward x pass of the rows src(g, m), the cells 2 m and 2 m + 1 of row (j, k):
// real-to-complex
template <typename Src>
__global__ void __launch_bounds__(kFxThreads, 3)
k_fx_xfwd(Grid g, FxPlan pl, const FxTw *__restrict__ r2c, Src src, double2 *__restrict__ spec,
          int lq, unsigned nhmag, const int *__restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FxScales sc;
  const int npen = 1 << lq, M = pl.n, sp = fx_row_pitch(M);
  fx2 *s = reinterpret_cast<fx2 *>(smem_raw), *a = s + npen * fx_row_pitch(M + 1);
  const long long nrows = (long long)g.ny * g.nz, row0 = (long long)blockIdx.x << lq;
  fx_scales_clear(sc);
  fx_rows(npen, row0, nrows, M, [&](long long row, int q, int m, int step, bool in, int count) {
    double2 *out = reinterpret_cast<double2 *>(s + q * sp);
    unsigned e = 0;
    int j = 0, k = 0;
    if (in) row_jk(g, row, j, k);
    src.row(g, j, k);
    auto cells = [&](auto &&pair) {
      for (; m < count; m += step) {
        const double2 r = in ? pair(m) : make_double2(0, 0);
        out[m] = r;
        e = max(e, max(fx_exp(r.x), fx_exp(r.y)));
      }
    };
    if (src.wide)  // (the same for all rows)
      cells([&](int i) { return src.fp64_pair(g, i); });
    else
      cells([&](int i) { return src(g, i); });
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&sc.emax[q], e);
  });
  __syncthreads();
  const fx2 *z = fx_row_transform<-1>(pl, lq, sc, s, a, sp, [&](int q, int t, unsigned e) {
    const double2 v = reinterpret_cast<const double2 *>(s)[q * sp + t];
    return fx2{fx_from(v.x, e), fx_from(v.y, e)};
  });
  // 2 X[k] = Fe[k] + W^k Fo[k], Fe = Z[k] + conj Z[M-k], Fo = (Z[k] - conj Z[M-k]) / i
  for (int idx = threadIdx.x; idx < npen * g.nxh; idx += blockDim.x) {
    const int q = fdiv(idx, nhmag), kx = idx - q * g.nxh;
    const long long row = row0 + q;
    if (row >= nrows) continue;
    const fx2 Z = z[q * sp + (kx == M ? 0 : kx)];
    const fx2 Y = z[q * sp + (kx == 0 ? 0 : M - kx)];
    const fx2 fe = {Z.x + Y.x, Z.y - Y.y}, fo = {Z.y + Y.y, Y.x - Z.x};
    const fx2 x = kx == 0 ? fe + fo : fe + fx_cmul(fo, r2c[kx]);
    const int k = fx_scale_of(sc, q, -1);
    spec[row * g.sxh + kx] = make_double2(fx_to(x.x, k), fx_to(x.y, k));
  }
}

// inverse x pass: upd(c, values) for every pair of cells c, c + 1, the values the
// unscaled transform times wtot 2^(etot - 62)
template <typename Upd>
__global__ void __launch_bounds__(kFxThreads, 3)
k_fx_xinv(Grid g, FxPlan pl, const FxTw *__restrict__ c2r, const double2 *__restrict__ spec,
          Upd upd, fxw wtot, int etot, int lq, const int *__restrict__ skip) {
  if (skip && *skip) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FxScales sc;
  const int npen = 1 << lq, M = pl.n, sp = fx_row_pitch(M), sx = fx_row_pitch(M + 1);
  fx2 *s = reinterpret_cast<fx2 *>(smem_raw), *a = s + npen * sx;
  const long long nrows = (long long)g.ny * g.nz, row0 = (long long)blockIdx.x << lq;
  fx_scales_clear(sc);
  fx_rows(npen, row0, nrows, M + 1, [&](long long row, int q, int i, int step, bool in, int count) {
    double2 *out = reinterpret_cast<double2 *>(s) + q * sx;
    unsigned e = 0;
    for (; i < count; i += step) {
      const double2 v = in ? spec[row * g.sxh + i] : make_double2(0, 0);
      out[i] = v;
      e = max(e, max(fx_exp(v.x), fx_exp(v.y)));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&sc.emax[q], e);
  });
  __syncthreads();
  // Z[k] = (X[k] + conj X[M-k]) + i (X[k] - conj X[M-k]) W^-k, over 4
  const fx2 *z = fx_row_transform<+1>(pl, lq, sc, s, a, sp, [&](int q, int t, unsigned e) {
    const double2 xv = reinterpret_cast<const double2 *>(s)[q * sx + t];
    const double2 yv = reinterpret_cast<const double2 *>(s)[q * sx + M - t];
    const fx2 X = {fx_from(xv.x, e), fx_from(xv.y, e)};
    const fx2 Y = {fx_from(yv.x, e), -fx_from(yv.y, e)};
    const fx2 f = X + Y, d = fx_cmul4(X - Y, c2r[t]);
    return fx2{fx_quarter(f.x) - d.y, fx_quarter(f.y) + d.x};
  });
  upd.begin();
  fx_rows(npen, row0, nrows, M, [&](long long row, int q, int m, int step, bool in, int count) {
    if (!in) return;
    const int k = fx_scale_of(sc, q, 4 + etot);
    for (; m < count; m += step) {
      const fx2 f = z[q * sp + m];
      upd(row * g.nx + 2 * m,
          make_double2(fx_to(fx_mul(f.x, wtot), k), fx_to(fx_mul(f.y, wtot), k)));
    }
  });
  upd.end();
}

}  // namespace
}  // namespace tpm
