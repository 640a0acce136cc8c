// transform_ops.cuh -- per-element pieces shared by the SIMT and the tensor-core Legendre
// kernels: the spectral prologues of the synthesis (the inputs built from neighbouring total
// wavenumbers) and the epilogues of the analysis (plain store, alpha operator, Laplacian of the
// energy, fused damping + leapfrog + Robert-Asselin filter, shallow-water implicit correction).
#pragma once
#include "jgcm_internal.cuh"

namespace jgcm {

template <typename T>
using V2 = typename C2<T>::t;

// Ampere-style asynchronous global -> shared copy of 16 bytes (both addresses 16-byte aligned):
// staged tables need no registers and every copy is in flight at once
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// four consecutive values in 16-byte loads and stores (the address is 16-byte aligned)
__device__ __forceinline__ void ld4(const float* p, float (&w)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&w)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
}

// np pairs of values converted along blockIdx.x, CAST_U pairs in flight per thread: every load and store
// instruction of a warp is one run of consecutive pairs (a store to host memory that leaves gaps in its
// sectors, four values per thread, ran at half the rate)
constexpr int CAST_U = 4;
template <typename A, typename B>
__device__ __forceinline__ void cast_pairs(const A* __restrict__ src, B* __restrict__ dst, size_t np) {
  const V2<A>* __restrict__ s = reinterpret_cast<const V2<A>*>(src);
  V2<B>* __restrict__ d = reinterpret_cast<V2<B>*>(dst);
  for (size_t t = (size_t)blockIdx.x * blockDim.x * CAST_U + threadIdx.x; t < np;
       t += (size_t)gridDim.x * blockDim.x * CAST_U) {
    V2<A> x[CAST_U];
#pragma unroll
    for (int u = 0; u < CAST_U; u++)
      if (t + (size_t)u * blockDim.x < np) x[u] = s[t + (size_t)u * blockDim.x];
#pragma unroll
    for (int u = 0; u < CAST_U; u++)
      if (t + (size_t)u * blockDim.x < np) {
        V2<B> y;
        y.x = (B)x[u].x;
        y.y = (B)x[u].y;
        d[t + (size_t)u * blockDim.x] = y;
      }
  }
}

// Spectra between the host layout [k][n][m] (FP64 pairs, m fastest) and the device layout [m][n][k]: one
// total wavenumber's 32 x 32 tile of the (k, m) matrix transposed through shared memory by 256 threads,
// both sides in runs of consecutive pairs.  Entries n < m are not read and become zero.
template <typename T>
__device__ __forceinline__ void spec_tile_h2d(const double2* __restrict__ src, V2<T>* __restrict__ dst, int N, int ns,
                                              int L, int m0, int n, int k0) {
  __shared__ V2<T> tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int q = ty; q < 32; q += 8) {
    const int k = k0 + q, m = m0 + tx;
    V2<T> v;
    v.x = v.y = 0;
    if (k < L && m <= N && m <= n) {
      const double2 x = src[((size_t)k * (ns + 1) + n) * (N + 1) + m];
      v.x = (T)x.x;
      v.y = (T)x.y;
    }
    tile[q][tx] = v;
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int m = m0 + q, k = k0 + tx;
    if (k < L && m <= N) dst[((size_t)m * (ns + 1) + n) * L + k] = tile[tx][q];
  }
}
template <typename T>
__device__ __forceinline__ void spec_tile_d2h(const V2<T>* __restrict__ src, double2* __restrict__ dst, int N, int ns,
                                              int L, int m0, int n, int k0) {
  __shared__ V2<T> tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int q = ty; q < 32; q += 8) {
    const int m = m0 + q, k = k0 + tx;
    if (k < L && m <= N) tile[tx][q] = src[((size_t)m * (ns + 1) + n) * L + k];
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int k = k0 + q, m = m0 + tx;
    if (k < L && m <= N) {
      const V2<T> v = tile[q][tx];
      dst[((size_t)k * (ns + 1) + n) * (N + 1) + m] = make_double2((double)v.x, (double)v.y);
    }
  }
}

template <typename G>
__device__ __forceinline__ const G& group_of(const G* g, int ng, int c, int* k) {
  int i = 0;
  for (; i < ng - 1; i++)
    if (c < g[i].col0 + g[i].L) break;
  *k = c - g[i].col0;
  return g[i];
}

// Fused spectral time stepping used by the G2S epilogues (Time_Integrator.jl:58-101).
template <typename T>
__device__ __forceinline__ void damp_leapfrog(const StepParams& sp, T d, T& dq, T qp, T& qc, T& qn) {
  const T r = pick<T>(sp.robert, sp.robertf);
  const int Dt = sp.dt;
  if (sp.init_step) {
    dq = (dq - qc * d) / ((T)1.0 + (T)Dt * d);
    qn = qc + (T)Dt * dq;
    qc = qc + r * ((T)-1.0 * qc + qn);
  } else {
    dq = (dq - qp * d) / ((T)1.0 + (T)(2 * Dt) * d);
    qc = qc + r * (qp - (T)2 * qc);
    qn = qp + (T)(2 * Dt) * dq;
    qc = qc + r * qn;
  }
}

template <typename T>
__device__ __forceinline__ void leapfrog_c(const StepParams& sp, T d, V2<T>& dq, V2<T> qp, V2<T>& qc, V2<T>& qn,
                                           bool damp) {
  if (!damp) d = 0;
  damp_leapfrog<T>(sp, d, dq.x, qp.x, qc.x, qn.x);
  damp_leapfrog<T>(sp, d, dq.y, qp.y, qc.y, qn.y);
}


// Input of the synthesis for total wavenumber n (>= m) of column k of group g: the field itself,
// cos(lat) x its gradient (Compute_Gradient_Cos!, Spectral_Spherical_Mesh.jl:655-692) or ucos / vcos
// from vorticity and divergence (Compute_Ucos_Vcos_From_Vor_Div!, :517-580; these fill row N+1).
// OP: the group's operator, S2G_ANY = looked up per call.  The tensor-core kernel looks it up: with a call of its
// own per operator it compiled to 40 registers instead of 48, fewer loads in flight (T85, 8 barotropic
// members, BF16x3: 18.4 -> 22.3 us).
constexpr int S2G_ANY = -1;
template <typename T, int OP = S2G_ANY>
__device__ __forceinline__ V2<T> s2g_input(const S2GGroup& g, const Tables<T>& tb, int m, int n, int ns, size_t mrow,
                                             int k) {
  using V = V2<T>;
  const int L = g.L, op = OP == S2G_ANY ? g.op : OP;
  const V* a = (const V*)g.a;
  V x;
  x.x = 0;
  x.y = 0;
  switch (op) {
    case S2G_PLAIN:
      x = a[(mrow + n) * L + k];
      if (m == 0 && n == 0) x.x = x.x - pick<T>(g.shift, g.shiftf);
      break;
    case S2G_ANOM:
      x = a[(mrow + n) * L + k];
      if (m == 0 && n == 0) x.x = 0;
      break;
    case S2G_ADJ_G2S:  // the synthesis weights every m >= 1 twice; the analysis never sees row N+1
      if (n < ns) {
        x = a[(mrow + n) * L + k];
        if (m > 0) {
          x.x = x.x * (T)0.5;
          x.y = x.y * (T)0.5;
        }
      }
      break;
    case S2G_DLAM: {  // coef_dlam .* (i h)
      T cf = tb.dlam[mrow + n];
      V h = a[(mrow + n) * L + k];
      x.x = cf * (-h.y);
      x.y = cf * h.x;
    } break;
    case S2G_DTH: {  // coef_dthp h_{n+1} + coef_dthm h_{n-1}
      if (n <= ns - 1) {
        T cp = tb.dthp[mrow + n];
        V h = a[(mrow + n + 1) * L + k];
        x.x = cp * h.x;
        x.y = cp * h.y;
      }
      if (n - 1 >= m) {
        T cm = tb.dthm[mrow + n];
        V h = a[(mrow + n - 1) * L + k];
        x.x = x.x + cm * h.x;
        x.y = x.y + cm * h.y;
      }
    } break;
    case S2G_UCOS:
    case S2G_VCOS: {
      // ucos = uvc (i div) - uvm vor_{n-1} - uvp vor_{n+1}
      // vcos = uvc (i vor) + uvm div_{n-1} + uvp div_{n+1}
      const V* vor = a;
      const V* dv = (const V*)g.b;
      const bool u = op == S2G_UCOS;
      const V* ic = u ? dv : vor;  // term multiplied by i*uvc
      const V* nb = u ? vor : dv;  // neighbour terms
      T sg = u ? (T)-1 : (T)1;
      T cc = tb.uvc[mrow + n];
      V z = ic[(mrow + n) * L + k];
      x.x = cc * (-z.y);
      x.y = cc * z.x;
      if (n - 1 >= m) {
        T cm = tb.uvm[mrow + n];
        V h = nb[(mrow + n - 1) * L + k];
        x.x = x.x + sg * (cm * h.x);
        x.y = x.y + sg * (cm * h.y);
      }
      if (n + 1 <= ns) {
        T cp = tb.uvp[mrow + n];
        V h = nb[(mrow + n + 1) * L + k];
        x.x = x.x + sg * (cp * h.x);
        x.y = x.y + sg * (cp * h.y);
      }
    } break;
  }
  return x;
}

// Rows n = m + r, r = r0, r0 + rstep, ... < K of one column into X[r * CT]; the group's operator is chosen
// once, so several rows' loads are in flight
template <typename T, int OP>
__device__ __forceinline__ void s2g_column_op(const S2GGroup& g, const Tables<T>& tb, int m, int ns, size_t mrow, int k,
                                              V2<T>* X, int CT, int r0, int rstep, int K) {
#pragma unroll 4
  for (int r = r0; r < K; r += rstep) X[r * CT] = s2g_input<T, OP>(g, tb, m, m + r, ns, mrow, k);
}
template <typename T>
__device__ __forceinline__ void s2g_column(const S2GGroup& g, const Tables<T>& tb, int m, int ns, size_t mrow, int k,
                                           V2<T>* X, int CT, int r0, int rstep, int K) {
  switch (g.op) {
    case S2G_PLAIN: s2g_column_op<T, S2G_PLAIN>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    case S2G_DLAM: s2g_column_op<T, S2G_DLAM>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    case S2G_DTH: s2g_column_op<T, S2G_DTH>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    case S2G_UCOS: s2g_column_op<T, S2G_UCOS>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    case S2G_VCOS: s2g_column_op<T, S2G_VCOS>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    case S2G_ADJ_G2S: s2g_column_op<T, S2G_ADJ_G2S>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
    default: s2g_column_op<T, S2G_ANOM>(g, tb, m, ns, mrow, k, X, CT, r0, rstep, K); break;
  }
}

// Analysis epilogue for output (m, n) of column k of group g (sidx = its MNK index) from the
// contraction results r0..r3 of the group's slots.
template <typename T>
__device__ __forceinline__ void g2s_store(const G2SPlan& plan, const SpecOutGroup& g, const Tables<T>& tb, size_t mrow,
                                          int n, size_t sidx, V2<T> r0, V2<T> r1, V2<T> r2, V2<T> r3) {
  using V = V2<T>;
  const T eig = tb.eig[mrow + n];
  switch (g.op) {
    case G2S_PLAIN:
    case G2S_ADJ_S2G:
      ((V*)g.dst)[sidx] = r0;
      break;
    case G2S_VOR:
      ((V*)g.dst)[sidx] = r0;
      break;
    case G2S_DIV: {
      V v = r0;
      if (g.colE >= 0) {  // - laplacian(G2S(E) + extra)
        V e = r2;
        if (g.extra) {
          V x = ((const V*)g.extra)[sidx];
          e.x = e.x + x.x;
          e.y = e.y + x.y;
        }
        v.x = v.x - eig * e.x;
        v.y = v.y - eig * e.y;
      }
      ((V*)g.dst)[sidx] = v;
    } break;
    case G2S_BARO: {  // Barotropic_Dynamics.jl:31-36: vorticity tendency, damping, leapfrog
      V dq = r0;
      V* qc = (V*)g.qc[0];
      const V* qp = (const V*)g.qp[0];
      V c0 = qc[sidx], p0 = qp[sidx], n0;
      T d = ((const T*)plan.sp.damping)[mrow + n];
      leapfrog_c<T>(plan.sp, d, dq, p0, c0, n0, true);
      qc[sidx] = c0;
      ((V*)g.dst)[sidx] = n0;
    } break;
    case G2S_SW: {  // Shallow_Water_Dynamics.jl:133-165
      // slots: 0 = du cos, 1 = dv cos, 2 = kinetic energy, 3 = dh
      V dvor = r0;
      V ddiv = r1;
      V kin = r2;
      V dh = r3;
      const V* hc_p = (const V*)g.qc[2];
      V hc = hc_p[sidx], hp = ((const V*)g.qp[2])[sidx];
      V dc = ((const V*)g.qc[1])[sidx], dp = ((const V*)g.qp[1])[sidx];
      // spe_energy = (kin + h_c) * eig ; ddiv -= spe_energy
      ddiv.x = ddiv.x - eig * (kin.x + hc.x);
      ddiv.y = ddiv.y - eig * (kin.y + hc.y);
      // Implicit_Correction! (SW) :25-54
      const T h0 = pick<T>(plan.sp.h0, plan.sp.h0f);
      const T Dt = plan.sp.init_step ? (T)plan.sp.dt : (T)(2 * plan.sp.dt);
      ddiv.x = ddiv.x + eig * (hc.x - hp.x);
      ddiv.y = ddiv.y + eig * (hc.y - hp.y);
      dh.x = dh.x + h0 * (dc.x - dp.x);
      dh.y = dh.y + h0 * (dc.y - dp.y);
      const T mu = pick<T>(plan.sp.implicit_coef, plan.sp.implicit_coeff) * Dt, mu2 = mu * mu;
      const T den = (T)1.0 - mu2 * eig * h0;
      ddiv.x = (ddiv.x - mu * eig * dh.x) / den;
      ddiv.y = (ddiv.y - mu * eig * dh.y) / den;
      dh.x = dh.x - mu * h0 * ddiv.x;
      dh.y = dh.y - mu * h0 * ddiv.y;
      const T d = ((const T*)plan.sp.damping)[mrow + n];
      V vc = ((V*)g.qc[0])[sidx], vp = ((const V*)g.qp[0])[sidx], vn, dn, hn;
      leapfrog_c<T>(plan.sp, d, dvor, vp, vc, vn, true);
      leapfrog_c<T>(plan.sp, d, ddiv, dp, dc, dn, true);
      leapfrog_c<T>(plan.sp, d, dh, hp, hc, hn, true);
      ((V*)g.qc[0])[sidx] = vc;
      ((V*)g.qc[1])[sidx] = dc;
      ((V*)g.qc[2])[sidx] = hc;
      ((V*)g.dst)[sidx] = vn;
      ((V*)g.dst2)[sidx] = dn;
      ((V*)g.dst3)[sidx] = hn;
    } break;
  }
}

}  // namespace jgcm
