// zonal_fft.cuh -- real zonal FFTs of nlon = 2 H points (H = 32 .. 512) as half-length complex
// transforms split in two register steps, H = R1 R2.
//
// A row (one latitude of one column) is transformed by G = R2 threads of one warp.  With n = R2 a + b and
// k = k1 + R1 k2,
//   Z[k1 + R1 k2] = sum_b w_R2^(b k2) [ w_H^(b k1) sum_a w_R1^(a k1) z[R2 a + b] ]:
// thread b forms the inner sum over a of its R1 points in registers, the rows' threads exchange the R2 x R1
// results through shared memory once (a warp barrier, no block barrier inside the transform), and each
// forms R1 / R2 outer sums of R2 points.  The register transforms are radix-2 stages unrolled at compile
// time with the trivial twiddles left out; the factors w_H^(b k1) are a thread's own, loaded before the
// dependency wait.  A block holds CB columns of one latitude, so that the Fourier side is read and written
// in runs of CB consecutive columns, and walks column tiles.
// Why this split: radix-2 in shared memory spent a pass, a barrier and full complex products per stage (FP64
// T42L20 step: forward 35, inverse 66 us, bound by the FP64 pipe at 2300 FP64 instructions a row; 27 and 51
// us here at 1650 and the quotients); a warp per row spent 20 shuffles per pair of points (FP32 T42L20, 32 members: forward 76
// us with the load-store pipe 97 % busy, 405 instructions a row; 38 us here, 75); a row per thread needs 152
// registers at nlon 128 (inverse 90 us at 17 % of the warps; 76 us here).  Separate, conflict-free pitches
// for the exchange, and the next tile's coefficients loaded ahead, measured no better (76 and 80 us).
#pragma once
#include "jgcm_internal.cuh"
#include "transform_ops.cuh"

namespace jgcm {

__host__ __device__ constexpr int brev_c(int x, int bits) {
  int r = 0;
  for (int b = 0; b < bits; b++) r |= ((x >> b) & 1) << (bits - 1 - b);
  return r;
}
__host__ __device__ constexpr int log2_c(int x) { return x <= 1 ? 0 : 1 + log2_c(x / 2); }

// x e^(SIGN 2 pi i E / 32), E < 16 a compile-time constant once unrolled
template <typename T, int SIGN>
__device__ __forceinline__ void rot32(int E, T& x, T& y) {
  constexpr double C[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                           0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                           0.19509032201612826785, 0.0};
  const T a = x, b = y;
  if (E == 0) return;
  if (E == 8) {
    x = SIGN > 0 ? -b : b;
    y = SIGN > 0 ? a : -a;
  } else if (E == 4 || E == 12) {
    const T h = (T)C[4];
    const T p = SIGN > 0 ? a - b : a + b, q = SIGN > 0 ? a + b : b - a;  // (1 + SIGN i) (a + i b)
    if (E == 4) {
      x = p * h;
      y = q * h;
    } else {  // x SIGN i more
      x = (SIGN > 0 ? -q : q) * h;
      y = (SIGN > 0 ? p : -p) * h;
    }
  } else {
    const T c = (T)(E < 8 ? C[E & 7] : -C[(16 - E) & 15]), s = (T)SIGN * (T)(E < 8 ? C[8 - E] : C[E - 8]);
    x = a * c - b * s;
    y = a * s + b * c;
  }
}

// R points in registers, decimation in frequency: result k at index brev_c(k, log2 R)
template <typename T, int R, int SIGN>
__device__ __forceinline__ void fft_reg(T (&re)[R], T (&im)[R]) {
#pragma unroll
  for (int s = R / 2; s >= 1; s >>= 1) {
#pragma unroll
    for (int b = 0; b < R; b += 2 * s) {
#pragma unroll
      for (int j = 0; j < s; j++) {
        const int i0 = b + j, i1 = i0 + s;
        const T ar = re[i0], ai = im[i0], br = re[i1], bi = im[i1];
        re[i0] = ar + br;
        im[i0] = ai + bi;
        T dr = ar - br, di = ai - bi;
        rot32<T, SIGN>(j * (16 / s), dr, di);
        re[i1] = dr;
        im[i1] = di;
      }
    }
  }
}

template <int H>
struct FFTSplit {
  static constexpr int R1 = H == 32 || H == 64 ? 8 : H == 128 || H == 256 ? 16 : 32, R2 = H / R1;
  static constexpr int P = H + R1 + 1;  // row pitch in shared memory (odd: a run of columns meets no bank twice)
};

// The twiddles w_H^(SIGN b k1) of thread b, k1 >= 1, from the table of e^(2 pi i t / nlon), t < H
template <typename T, int H, int SIGN>
__device__ __forceinline__ void load_twiddles(const T* __restrict__ tw, int b, T (&c)[FFTSplit<H>::R1],
                                              T (&s)[FFTSplit<H>::R1]) {
#pragma unroll
  for (int k = 1; k < FFTSplit<H>::R1; k++) {
    const int t = 2 * b * k;  // < 2 H
    const V2<T> w = reinterpret_cast<const V2<T>*>(tw)[t & (H - 1)];
    const bool neg = t & H;
    c[k] = neg ? -w.x : w.x;
    s[k] = (SIGN > 0) == neg ? -w.y : w.y;
  }
}

// The row transform of thread b of a row: z[R2 a + b] in (re, im)[a] -> Z[k1 + R1 k2], k1 = b + R2 h, in
// (re, im)[h R2 + brev(k2)].  `row`: the row's shared memory, free for the exchange after the warp barrier.
template <typename T, int H, int SIGN>
__device__ __forceinline__ void fft_row(T (&re)[FFTSplit<H>::R1], T (&im)[FFTSplit<H>::R1], V2<T>* row, int b,
                                        const T (&c)[FFTSplit<H>::R1], const T (&s)[FFTSplit<H>::R1]) {
  constexpr int R1 = FFTSplit<H>::R1, R2 = FFTSplit<H>::R2, L1 = log2_c(R1);
  fft_reg<T, R1, SIGN>(re, im);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < R1; k++) {
    const T x = re[brev_c(k, L1)], y = im[brev_c(k, L1)];
    V2<T> v;
    v.x = k ? x * c[k] - y * s[k] : x;
    v.y = k ? x * s[k] + y * c[k] : y;
    row[k * (R2 + 1) + b] = v;
  }
  __syncwarp();
#pragma unroll
  for (int h = 0; h < R1 / R2; h++) {
    T x[R2], y[R2];
#pragma unroll
    for (int q = 0; q < R2; q++) {
      const V2<T> v = row[(b + R2 * h) * (R2 + 1) + q];
      x[q] = v.x;
      y[q] = v.y;
    }
    fft_reg<T, R2, SIGN>(x, y);
#pragma unroll
    for (int q = 0; q < R2; q++) {
      re[h * R2 + q] = x[q];
      im[h * R2 + q] = y[q];
    }
  }
}

// x / c with rc = 1 / c at hand.  FP32: the product, within an ulp of the quotient.  FP64: the product corrected by
// its residual, which the fused operation forms exactly (P. Markstein, IBM J. Res. Dev. 34, 1990): the quotient's own
// rounding (none of 2e8 random pairs differed; the product alone differs in 27 %).  A product that is not finite
// stays as it is.  T42L20's inverse 51 us, 47 with the bare product, 60 with divisions.
__device__ __forceinline__ float quotient(float x, float, float rc) { return x * rc; }
__device__ __forceinline__ double quotient(double x, double c, double rc) {
  const double q = x * rc, z = fma(fma(-q, c, x), rc, q);
  return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : z;
}

// The epilogue of a run of a row: x(λ_2i) = re[r], x(λ_2i+1) = im[r] for i = i0 + step r, the group's epilogue
// chosen once per run and each pair of longitudes stored as one 8- or 16-byte word.
template <typename T, int V>
__device__ __forceinline__ void ifft_store_row(const GridOutGroup& g, const Tables<T>& tb, int k, int j, int nlat,
                                               int nlon, const T (&re)[V], const T (&im)[V], int i0, int step) {
  using P = V2<T>;
  const size_t row = ((size_t)k * nlat + j) * nlon;
  P* dst = reinterpret_cast<P*>((T*)g.dst + row) + i0;
  auto put = [&](P* d, int r, T a, T b) {
    P v;
    v.x = a;
    v.y = b;
    d[step * r] = v;
  };
  switch (g.epi) {
    case EPI_NONE:
#pragma unroll
      for (int r = 0; r < V; r++) put(dst, r, re[r], im[r]);
      break;
    case EPI_DIVCOS: {
      const T c = tb.cosj[j], rc = (T)1 / c;
#pragma unroll
      for (int r = 0; r < V; r++) put(dst, r, quotient(re[r], c, rc), quotient(im[r], c, rc));
    } break;
    case EPI_EXP2: {
      const T sh = pick<T>(g.shift, g.shiftf), es = pick<T>(g.eshift, g.eshiftf);
      P* d2 = reinterpret_cast<P*>((T*)g.dst2 + row) + i0;
#pragma unroll
      for (int r = 0; r < V; r++) {
        put(dst, r, re[r] + sh, im[r] + sh);
        put(d2, r, exp(re[r]) * es, exp(im[r]) * es);
      }
    } break;
    case EPI_DIVCOS_MULPS: {  // level k of ps
      const T c = tb.cosj[j], rc = (T)1 / c;
      const P* ps = reinterpret_cast<const P*>((const T*)g.ps + row) + i0;
#pragma unroll
      for (int r = 0; r < V; r++) {
        const P q = ps[step * r];
        put(dst, r, quotient(re[r], c, rc) * q.x, quotient(im[r], c, rc) * q.y);
      }
    } break;
    case EPI_ADJ_G2S: {
      const auto sc = tb.wts[j] / (T)(2 * nlon);
#pragma unroll
      for (int r = 0; r < V; r++) put(dst, r, (T)(re[r] * sc), (T)(im[r] * sc));
    } break;
    case EPI_ANOM: {
      const T mean = ((const V2<T>*)g.ps)[k].x;
      P* d2 = reinterpret_cast<P*>((T*)g.dst2 + row) + i0;
#pragma unroll
      for (int r = 0; r < V; r++) {
        put(dst, r, re[r] + mean, im[r] + mean);
        put(d2, r, re[r], im[r]);
      }
    } break;
  }
}

// The pairs of grid values z[i] = (x(λ_2i), x(λ_2i+1)), i = i0 + step r, of row (k, j) under the group's
// prologue (fft_load), which is chosen once per row: a row's loads are all in flight together
template <typename T, int R>
__device__ __forceinline__ void fft_load_row(const FFTPlan& plan, const GridInGroup& g, int k, int j, int nlat, int nlon,
                                             T cj, T (&re)[R], T (&im)[R], int i0, int step) {
  using V = V2<T>;
  const size_t row = ((size_t)k * nlat + j) * nlon;
  auto at = [&](const void* p, int r) -> V { return (reinterpret_cast<const V*>((const T*)p + row) + i0)[step * r]; };
  auto put = [&](int r, T a, T b) {
    re[r] = a;
    im[r] = b;
  };
  switch (g.pro) {
    case PRO_NONE:
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V x = at(g.src, r);
        put(r, x.x, x.y);
      }
      break;
    case PRO_MULCOS:
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V x = at(g.src, r);
        put(r, x.x * cj, x.y * cj);
      }
      break;
    case PRO_FLUXU:
    case PRO_FLUXV: {
      const T f = ((const T*)plan.coriolis)[j], km = -pick<T>(plan.kappa_m, plan.kappa_mf);
      const bool fu = g.pro == PRO_FLUXU;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V u = at(g.src, r), v = at(g.s1, r), z = at(g.s2, r);
        const T a = z.x + f, b = z.y + f;
        put(r, fu ? (km * u.x + a * v.x) * cj : (km * v.x + (-a) * u.x) * cj,
            fu ? (km * u.y + b * v.y) * cj : (km * v.y + (-b) * u.y) * cj);
      }
    } break;
    case PRO_KIN:
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V u = at(g.src, r), v = at(g.s1, r);
        put(r, (T)0.5 * (u.x * u.x + v.x * v.x), (T)0.5 * (u.y * u.y + v.y * v.y));
      }
      break;
    case PRO_SWH: {
      const T kt = -pick<T>(plan.kappa_t, plan.kappa_tf);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const V h = at(g.src, r), u = at(g.s1, r), v = at(g.s2, r), dl = at(g.s3, r), dt = at(g.s4, r), dv = at(g.s5, r),
                he = at(g.s6, r);
        put(r, (kt * (h.x - he.x) - (u.x * dl.x + v.x * dt.x)) - h.x * dv.x,
            (kt * (h.y - he.y) - (u.y * dl.y + v.y * dt.y)) - h.y * dv.y);
      }
    } break;
  }
}

// Fourier -> grid.  grid (column tiles or fewer, nlat), CB R2 threads, CB P complex T of shared memory.
// With X the Hermitian spectrum (0 above N, Im X[0] dropped), D = X[m] - conj X[H-m] and w = e^(2 pi i m / nlon):
// Z[m] = (X[m] + conj X[H-m]) + i w D, and Z[H-m] is formed from the same sum and product.
// NB: blocks of 256 threads that the registers leave room for on an SM (0: the compiler's choice).
template <typename T, int H, int NB = 0>
__global__ void __launch_bounds__(256, NB) k_ifft_reg(const __grid_constant__ IFFTPlan plan, Tables<T> tb,
                                                  const V2<T>* __restrict__ F, int N, int nlat, int lcb, int ntiles) {
  using V = V2<T>;
  constexpr int R1 = FFTSplit<H>::R1, R2 = FFTSplit<H>::R2, P = FFTSplit<H>::P, L2 = log2_c(R2);
  extern __shared__ __align__(16) unsigned char smem[];
  const int CB = 1 << lcb, j = blockIdx.y, C = plan.C, b = threadIdx.x % R2, cc = threadIdx.x / R2;
  V* S = (V*)smem;  // [CB][P]
  T c1[R1], s1[R1];
  load_twiddles<T, H, 1>(tb.tw, b, c1, s1);
  pdl_wait();  // programmatic dependent launch: the predecessor's output is complete
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int cbase = tile << lcb;
    // the coefficient pairs m, H - m of column q, m = m0 + R2 it: PB pairs' loads are issued together
    constexpr int IT = (H / 2 + R2) / R2, PB = 5;
    const int q = threadIdx.x & (CB - 1), m0 = threadIdx.x >> lcb, cq = cbase + q;
    const V* Fq = F + (size_t)j * C + cq;
    const size_t mstride = (size_t)nlat * C;
    V* Sq = S + q * P;
#pragma unroll
    for (int ib = 0; ib < IT; ib += PB) {
      V xs[PB], ys[PB];
#pragma unroll
      for (int p = 0; p < PB; p++) {
        const int m = m0 + R2 * (ib + p);
        xs[p].x = xs[p].y = ys[p].x = ys[p].y = 0;
        if (ib + p < IT && cq < C && m <= H / 2) {
          if (m <= N) xs[p] = Fq[m * mstride];
          if (m >= 1 && H - m <= N) ys[p] = Fq[(H - m) * mstride];
          if (m == 0) xs[p].y = 0;  // only Re X[0] reaches the grid
        }
      }
#pragma unroll
      for (int p = 0; p < PB; p++) {
        const int m = m0 + R2 * (ib + p);
        if (ib + p >= IT || m > H / 2) continue;
        const V x = xs[p], y = ys[p], w = reinterpret_cast<const V*>(tb.tw)[m];
        const T er = x.x + y.x, ei = x.y - y.y, dr = x.x - y.x, di = x.y + y.y;
        const T orr = dr * w.x - di * w.y, oi = dr * w.y + di * w.x;
        V z;
        z.x = er - oi;
        z.y = ei + orr;
        Sq[m] = z;
        if (m >= 1 && m < H / 2) {
          z.x = er + oi;
          z.y = orr - ei;
          Sq[H - m] = z;
        }
      }
    }
    __syncthreads();
    V* row = S + cc * P;
    T re[R1], im[R1];
#pragma unroll
    for (int a = 0; a < R1; a++) {
      const V v = row[R2 * a + b];
      re[a] = v.x;
      im[a] = v.y;
    }
    fft_row<T, H, 1>(re, im, row, b, c1, s1);
    const int c = cbase + cc;
    if (c < C) {  // z[i] = x[2i] + i x[2i+1]
      int k;
      const GridOutGroup& g = group_of(plan.g, plan.ng, c, &k);
#pragma unroll
      for (int h = 0; h < R1 / R2; h++) {
        T x[R2], y[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) {
          x[q] = re[h * R2 + brev_c(q, L2)];
          y[q] = im[h * R2 + brev_c(q, L2)];
        }
        ifft_store_row<T, R2>(g, tb, k, j, nlat, 2 * H, x, y, b + R2 * h, R1);
      }
    }
    __syncthreads();  // the tile's shared memory is free for the next one
  }
}

// Grid -> Fourier: fft/nlon, modes 0..N.  PLAIN: every group of the plan reads its field as it is (PRO_NONE).
template <typename T, int H, bool PLAIN>
__global__ void __launch_bounds__(256) k_fft_reg(const __grid_constant__ FFTPlan plan, Tables<T> tb,
                                                 V2<T>* __restrict__ F, int N, int nlat, int lcb, int ntiles) {
  using V = V2<T>;
  constexpr int R1 = FFTSplit<H>::R1, R2 = FFTSplit<H>::R2, P = FFTSplit<H>::P, L2 = log2_c(R2), NLON = 2 * H;
  extern __shared__ __align__(16) unsigned char smem[];
  const int CB = 1 << lcb, j = blockIdx.y, C = plan.C, b = threadIdx.x % R2, cc = threadIdx.x / R2;
  V* S = (V*)smem;  // [CB][P]
  T c1[R1], s1[R1];
  load_twiddles<T, H, -1>(tb.tw, b, c1, s1);
  const T cj = tb.cosj[j];
  pdl_wait();  // programmatic dependent launch: the predecessor's output is complete
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int cbase = tile << lcb, c = cbase + cc;
    T re[R1], im[R1];
    if (c < C) {
      int k;
      const GridInGroup& g = group_of(plan.g, plan.ng, c, &k);
      if constexpr (PLAIN) {
        const V* src = reinterpret_cast<const V*>((const T*)g.src + ((size_t)k * nlat + j) * NLON) + b;
#pragma unroll
        for (int a = 0; a < R1; a++) {  // z[n] = x[2n] + i x[2n+1], n = R2 a + b
          const V v = src[R2 * a];
          re[a] = v.x;
          im[a] = v.y;
        }
      } else {
        fft_load_row<T, R1>(plan, g, k, j, nlat, NLON, cj, re, im, b, R2);
      }
    } else {
#pragma unroll
      for (int a = 0; a < R1; a++) re[a] = im[a] = 0;
    }
    V* row = S + cc * P;
    fft_row<T, H, -1>(re, im, row, b, c1, s1);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < R1 / R2; h++)
#pragma unroll
      for (int q = 0; q < R2; q++) {
        V v;
        v.x = re[h * R2 + brev_c(q, L2)];
        v.y = im[h * R2 + brev_c(q, L2)];
        row[b + R2 * h + R1 * q] = v;
      }
    __syncthreads();
    // X[m] = E[m] + e^(-2 pi i m / nlon) O[m], E = (Z[m] + conj Z[H-m])/2, O = (Z[m] - conj Z[H-m])/(2i)
    const T scale = (T)0.5 / (T)NLON;  // exact
    for (int i = threadIdx.x; i < (N + 1) << lcb; i += blockDim.x) {
      const int q = i & (CB - 1), m = i >> lcb;
      if (cbase + q >= C) continue;
      const V zm = S[q * P + m], zq = S[q * P + ((H - m) & (H - 1))];
      const V w = reinterpret_cast<const V*>(tb.tw)[m];
      const T er = zm.x + zq.x, ei = zm.y - zq.y;   // 2 E
      const T orr = zm.y + zq.y, oi = zq.x - zm.x;  // 2 O
      V o;
      o.x = (er + (w.x * orr + w.y * oi)) * scale;
      o.y = (ei + (w.x * oi - w.y * orr)) * scale;
      F[((size_t)m * nlat + j) * C + cbase + q] = o;
    }
    __syncthreads();  // the tile's shared memory is free for the next one
  }
}

}  // namespace jgcm
