// hs_transforms.cu -- the Held-Suarez step's Legendre analysis as one contraction per
// (zonal-wavenumber pair, level group, member).
//
// The general analysis kernel (k_g2s_legendre, transforms.cu) treats every output column on its
// own: a column tile per block, a group lookup and an input slot per column, the quadrature weights
// re-read for every column.  The Held-Suarez step always analyses the same four fields per level
// (δu cos, δv cos, the energy and δT, plus δ ln ps per member) into the same three outputs per level
// (the vorticity and divergence tendencies of the alpha operator, Vor_Div_From_Grid_UV! and
// Compute_Alpha_Operator!, Spectral_Spherical_Mesh.jl:349-459, with ∇² of the energy taken off the
// divergence, Spectral_Dynamics.jl:286-296, and the temperature tendency; Trans_Grid_To_Spherical!
// :221-293 for δ ln ps).  Here one thread owns one (m, n, level) and forms all of its outputs from
// the same weight rows (P w, the alpha operator's two rows) and the same folded inputs, so each
// weight load serves 12 multiply-adds instead of 2.  Blocks take the zonal wavenumbers in pairs
// (m, N - m), whose output counts K_m + K_{N-m} = N + 4 are the same for every pair, so the blocks
// carry equal work.  Sums run over the folded latitudes in order, four weights per load, as in the
// general kernel's one-lane form.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "jgcm_internal.cuh"
#include "transform_ops.cuh"

namespace jgcm {

namespace {

template <typename T>
struct HSAnaArgs {
  const V2<T>* F;                       // Fourier buffer [m][j][Cin]
  V2<T> *dvor, *ddiv, *dt, *dlnps;      // outputs, MNK: [m][n][L] (dlnps: [m][n][E])
  int Cin;                              // columns of the Fourier buffer
  int colU, colV, colE, colT, colP;     // base columns of δu cos, δv cos, energy, δT (L each), δ ln ps (E)
  int nd, L, E, N, ns, nlat, nh;
  int LG;                               // levels per block (the level nd of a member is δ ln ps)
};

// row pitch of the staged weight tables: one 16-byte pad per row, so that the rows read by the
// threads of a warp start in different shared-memory banks
template <typename T>
__host__ __device__ constexpr int wpitch(int nh) {
  return nh + 16 / (int)sizeof(T);
}

// Both values summed over the SP neighbouring lanes of an output, which take the same branches
template <int SP, typename T>
__device__ __forceinline__ void pair_sum(T& x, T& y) {
  const unsigned group = ((1u << SP) - 1) << (threadIdx.x & 31 & ~(SP - 1));
#pragma unroll
  for (int o = 1; o < SP; o <<= 1) {
    x += __shfl_xor_sync(group, x, o);
    y += __shfl_xor_sync(group, y, o);
  }
}

// grid (N/2 + 1 pairs, ceil((nd + 1) / LG) level groups, members), blockDim >= rows * LG * SP with rows the
// largest per-pair thread count (N + 4 for NP = 1).  SP = 2 (FP64, small launches): two
// neighbouring lanes share an output's latitudes in turns of four (hs_analysis_shape).
template <typename T, int NP, int SP>
__global__ void __launch_bounds__(256) k_hs_analysis(HSAnaArgs<T> a, Tables<T> tb) {
  using V = V2<T>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int N = a.N, ns = a.ns, nh = a.nh, LG = a.LG, nd = a.nd, nlat = a.nlat;
  const int m1 = blockIdx.x, m2 = N - m1, g = blockIdx.y, e = blockIdx.z;
  const int nm = m2 != m1 ? 2 : 1;
  const int K1 = ns + 1 - m1, K2 = nm == 2 ? ns + 1 - m2 : 0;
  const int wp = wpitch<T>(nh);
  // weights: slot s (m1, m2) holds [3][K_s][wp]: P w, the alpha operator's i-term and its B-term
  T* W = (T*)smem;
  const size_t wsz = (size_t)3 * (K1 + K2) * wp;
  // folded inputs [f][jh][parity][slot][level]: the lanes of a warp that read one latitude of one
  // field read neighbouring words
  V* X = (V*)(smem + ((wsz * sizeof(T) + 15) & ~(size_t)15));
  // 1. the weight rows n = m..ns of both m (constants): asynchronous 16-byte copies, issued before
  //    the dependency wait and waited for once
  {
    constexpr int ce = 16 / (int)sizeof(T);  // weights per chunk
    const int nchunk = nh / ce;
    for (int s = 0; s < nm; s++) {
      const int m = s ? m2 : m1, K = s ? K2 : K1;
      const size_t src = ((size_t)m * (ns + 1) + m) * nh;
      T* dst = W + (s ? (size_t)3 * K1 * wp : 0);
      for (int i = threadIdx.x; i < K * nchunk; i += blockDim.x) {
        const int r = i / nchunk, c = i - r * nchunk;
        const size_t to = (size_t)r * wp + c * ce, from = src + (size_t)i * ce;
        cp_async16(dst + to, tb.PW + from);
        cp_async16(dst + (size_t)K * wp + to, tb.CA + from);
        cp_async16(dst + (size_t)2 * K * wp + to, tb.CB + from);
      }
    }
    cp_async_commit();
  }
  pdl_wait();  // programmatic dependent launch: the forward FFT's coefficients are complete
  // 2. hemisphere folds of the block's input columns: thread (l, jh) loads its latitude pair of all
  //    fields of both m first (up to 16 loads in flight), then folds them; consecutive threads take
  //    consecutive levels, i.e. neighbouring columns of the Fourier buffer
  for (int item = threadIdx.x; item < LG * nh; item += blockDim.x) {
    const int jh = item / LG, l = item - jh * LG, lv = g * LG + l;
    V x[2][4], y[2][4];
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
      for (int f = 0; f < 4; f++) {
        x[s][f].x = x[s][f].y = y[s][f].x = y[s][f].y = 0;
        int col = -1;
        if (lv < nd)
          col = (f == 0 ? a.colU : f == 1 ? a.colV : f == 2 ? a.colE : a.colT) + e * nd + lv;
        else if (lv == nd && f == 3)
          col = a.colP + e;
        if (s < nm && col >= 0) {
          const int m = s ? m2 : m1;
          x[s][f] = a.F[((size_t)m * nlat + jh) * a.Cin + col];
          y[s][f] = a.F[((size_t)m * nlat + (nlat - 1 - jh)) * a.Cin + col];
        }
      }
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
      for (int f = 0; f < 4; f++) {
        if (s >= nm) continue;
        V sv, av;
        sv.x = x[s][f].x + y[s][f].x;
        sv.y = x[s][f].y + y[s][f].y;
        av.x = x[s][f].x - y[s][f].x;
        av.y = x[s][f].y - y[s][f].y;
        const size_t base = ((size_t)(f * nh + jh) * 2) * nm * LG + (size_t)s * LG + l;
        X[base] = sv;
        X[base + (size_t)nm * LG] = av;
      }
  }
  cp_async_wait_all();
  __syncthreads();
  // 3. one thread per (m, level) and NP total wavenumbers of one parity, n and n + 2 (NP = 2:
  //    each folded input loaded from shared memory serves both; rows r = 4 i + b, b < 2)
  const int h = threadIdx.x % SP;
  int q = threadIdx.x / SP / LG;
  const int l = threadIdx.x / SP - q * LG;
  const int Q1 = NP == 1 ? K1 : 2 * ((K1 + 3) / 4), Q2 = nm == 2 ? (NP == 1 ? K2 : 2 * ((K2 + 3) / 4)) : 0;
  if (q >= Q1 + Q2) return;
  const int s = q < Q1 ? 0 : 1;
  if (s) q -= Q1;
  const int m = s ? m2 : m1, K = s ? K2 : K1;
  const int r0 = NP == 1 ? q : 4 * (q >> 1) + (q & 1);
  if (r0 >= K) return;
  const int lv = g * LG + l;
  if (lv > nd) return;
  const bool even = (r0 & 1) == 0;  // P_n^m is symmetric about the equator for n - m even
  const T* wbase = W + (s ? (size_t)3 * K1 * wp : 0);
  const T* pw[NP];
  const T* ca[NP];
  const T* cb[NP];
  bool live[NP];
#pragma unroll
  for (int u = 0; u < NP; u++) {
    const int r = r0 + 2 * u;
    live[u] = r < K;
    const int rr = live[u] ? r : r0;  // a row past K reads row r0's weights and is not stored
    pw[u] = wbase + (size_t)rr * wp;
    ca[u] = wbase + ((size_t)K + rr) * wp;
    cb[u] = wbase + ((size_t)2 * K + rr) * wp;
  }
  // element (f, jh, parity) of this thread's column: X[((f nh + jh) 2 + par) nm LG + s LG + l]
  const size_t pstride = (size_t)nm * LG, jstride = 2 * pstride, fstride = (size_t)nh * jstride;
  const V* xcol = X + (size_t)s * LG + l;
  const size_t same = even ? 0 : pstride, other = even ? pstride : 0;
  const size_t mrow = (size_t)m * (ns + 1);
  if (lv == nd) {  // δ ln ps of member e: plain analysis
    const V* src = xcol + 3 * fstride + same;
    T sr[NP], si[NP];
#pragma unroll
    for (int u = 0; u < NP; u++) sr[u] = si[u] = 0;
    for (int jh = 4 * h; jh < nh; jh += 4 * SP) {
      T w[NP][4];
#pragma unroll
      for (int u = 0; u < NP; u++) ld4(pw[u] + jh, w[u]);
#pragma unroll
      for (int v = 0; v < 4; v++) {
        const V x = src[(size_t)(jh + v) * jstride];
#pragma unroll
        for (int u = 0; u < NP; u++) {
          sr[u] += x.x * w[u][v];
          si[u] += x.y * w[u][v];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < NP; u++) {
      const int n = m + r0 + 2 * u;
      pair_sum<SP>(sr[u], si[u]);
      if (!live[u] || h) continue;
      V o;
      o.x = n == ns ? (T)0 : sr[u] * (T)0.5;
      o.y = n == ns ? (T)0 : si[u] * (T)0.5;
      a.dlnps[(mrow + n) * a.E + e] = o;
    }
    return;
  }
  const V* us = xcol + same;                 // δu cos, parity of n - m
  const V* uo = xcol + other;                // δu cos, the other parity
  const V* vs = xcol + fstride + same;       // δv cos
  const V* vo = xcol + fstride + other;
  const V* es = xcol + 2 * fstride + same;   // energy
  const V* ts = xcol + 3 * fstride + same;   // δT
  // vorticity: alpha operator of (A = δv cos, B = δu cos), i Σ CA A - Σ CB B
  // divergence: alpha operator of (A = δu cos, B = δv cos), i Σ CA A + Σ CB B, less ∇² of the energy
  T var[NP], vai[NP], vbr[NP], vbi[NP], dar[NP], dai[NP], dbr[NP], dbi[NP], er[NP], ei[NP], tr[NP], ti[NP];
#pragma unroll
  for (int u = 0; u < NP; u++)
    var[u] = vai[u] = vbr[u] = vbi[u] = dar[u] = dai[u] = dbr[u] = dbi[u] = er[u] = ei[u] = tr[u] = ti[u] = 0;
  for (int jh = 4 * h; jh < nh; jh += 4 * SP) {
    T wP[NP][4], wA[NP][4], wB[NP][4];
#pragma unroll
    for (int u = 0; u < NP; u++) {
      ld4(pw[u] + jh, wP[u]);
      ld4(ca[u] + jh, wA[u]);
      ld4(cb[u] + jh, wB[u]);
    }
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const size_t o = (size_t)(jh + v) * jstride;
      const V xu = us[o], yv = vo[o], xv = vs[o], yu = uo[o], xe = es[o], xt = ts[o];
#pragma unroll
      for (int u = 0; u < NP; u++) {
        var[u] += (-xv.y) * wA[u][v];
        vai[u] += xv.x * wA[u][v];
        vbr[u] += yu.x * wB[u][v];
        vbi[u] += yu.y * wB[u][v];
        dar[u] += (-xu.y) * wA[u][v];
        dai[u] += xu.x * wA[u][v];
        dbr[u] += yv.x * wB[u][v];
        dbi[u] += yv.y * wB[u][v];
        er[u] += xe.x * wP[u][v];
        ei[u] += xe.y * wP[u][v];
        tr[u] += xt.x * wP[u][v];
        ti[u] += xt.y * wP[u][v];
      }
    }
  }
#pragma unroll
  for (int u = 0; u < NP; u++) {
    pair_sum<SP>(var[u], vai[u]);
    pair_sum<SP>(vbr[u], vbi[u]);
    pair_sum<SP>(dar[u], dai[u]);
    pair_sum<SP>(dbr[u], dbi[u]);
    pair_sum<SP>(er[u], ei[u]);
    pair_sum<SP>(tr[u], ti[u]);
    if (!live[u] || h) continue;
    const int n = m + r0 + 2 * u;
    V ov, od, ot;
    if (n == ns) {  // row N+1 of the analysis is zero (Trans_Grid_To_Spherical!, :288-291)
      ov.x = ov.y = od.x = od.y = ot.x = ot.y = 0;
    } else {
      const T eig = tb.eig[mrow + n];
      ov.x = var[u] + (T)-1 * vbr[u];
      ov.y = vai[u] + (T)-1 * vbi[u];
      od.x = dar[u] + dbr[u];
      od.y = dai[u] + dbi[u];
      od.x = od.x - eig * (er[u] * (T)0.5);
      od.y = od.y - eig * (ei[u] * (T)0.5);
      ot.x = tr[u] * (T)0.5;
      ot.y = ti[u] * (T)0.5;
    }
    const size_t sidx = (mrow + n) * a.L + (size_t)e * nd + lv;
    a.dvor[sidx] = ov;
    a.ddiv[sidx] = od;
    a.dt[sidx] = ot;
  }
}

template <typename T>
size_t hs_analysis_smem(const jgcm_mesh* m, int LG) {
  const int N = m->N, nh = m->nh;
  const size_t w = (size_t)3 * (N + 4) * wpitch<T>(nh) * sizeof(T);
  return ((w + 15) & ~(size_t)15) + (size_t)4 * nh * 2 * 2 * LG * sizeof(V2<T>);
}

PerDeviceOnce g_hs_ana_smem[2];

// The same analysis for launches of many columns, FP32: a block takes 32 consecutive columns (levels of
// all members in a row) of one m, a warp four rows n of one parity (n = m + 8 i + p + 2 u, u < 4), a lane one
// column.  Per latitude pair the lane reads its eight inputs (coalesced), folds them, and with the warp's 12
// weights (three broadcast loads) makes 48 multiply-adds; with two rows per thread and a weight row per load
// the shared-memory pipe was the bound (T42L20, 32 members: 68 % of its wavefronts at 22 % of the warps, 37 M
// instructions for 7.6 M multiply-adds, 70 us; 128 x T21L20 60 us).  The Fourier rows stream through a
// ring of AT_STAGES x AT_JC latitude pairs by asynchronous copies, and the weights are laid out for it once
// per mesh ([m][latitude][row group][table][u], hs_tables_build): 40 and 29 us; staged and folded in step,
// with a transposition of the weights per block, 50 and 41.  The columns of
// δ ln ps (one per member) are tiles of their own behind the levels', with the δT slot alone.  Same sums in
// the same order.  grid (level tiles + δ ln ps tiles, N + 1), 32 at_groups(ns + 1) threads.
constexpr int AT_ROWS = 4, AT_JC = 8, AT_STAGES = 3;
__host__ __device__ constexpr int at_groups(int K) { return 2 * ((K + 2 * AT_ROWS - 1) / (2 * AT_ROWS)); }
__host__ __device__ constexpr int at_pitch(int ns) { return at_groups(ns + 1) * 3 * AT_ROWS; }  // floats per latitude

__global__ void k_at_weights(Tables<float> tb, float* __restrict__ out, int N, int ns, int nh) {
  const int wp = at_pitch(ns);
  const size_t total = (size_t)(N + 1) * nh * wp;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    const int q = (int)(t % wp), jh = (int)(t / wp % nh), m = (int)(t / wp / nh);
    const int g = q / (3 * AT_ROWS), tbl = q / AT_ROWS % 3, u = q % AT_ROWS, n = m + 8 * (g >> 1) + (g & 1) + 2 * u;
    const float* from = tbl == 0 ? tb.PW : tbl == 1 ? tb.CA : tb.CB;
    out[t] = n <= ns ? from[((size_t)m * (ns + 1) + n) * nh + jh] : 0.f;
  }
}

// 8-byte asynchronous copy, or zeros when !live (the source address is valid either way)
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc, bool live) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gsrc), "r"(live ? 8 : 0) : "memory");
}

template <int NT, int NB>
__global__ void __launch_bounds__(NT, NB) k_hs_analysis_tiles(HSAnaArgs<float> a, Tables<float> tb,
                                                              const float* __restrict__ wt) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int ns = a.ns, nh = a.nh, nlat = a.nlat, m = blockIdx.y, K = ns + 1 - m, G = at_groups(K), wp = at_pitch(ns);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nt = (a.L + 31) / 32;
  const bool isp = (int)blockIdx.x >= nt;  // a tile of δ ln ps columns
  const int col = ((int)blockIdx.x - (isp ? nt : 0)) * 32 + lane;
  const bool live = col < (isp ? a.E : a.L);
  float* W = (float*)smem;                                         // [nh][wp]
  float2* X = (float2*)(smem + (size_t)nh * wp * sizeof(float));  // [stage][latitude][field][south, north][32]
  const size_t mrow = (size_t)m * (ns + 1);
  {
    const float* src = wt + (size_t)m * nh * wp;
    const int nc = G * 3;  // 16-byte chunks of a latitude's weights in use
    for (int i = threadIdx.x; i < nh * nc; i += blockDim.x) {
      const int jh = i / nc, c = i - jh * nc;
      cp_async16(W + (size_t)jh * wp + c * 4, src + (size_t)jh * wp + c * 4);
    }
  }
  pdl_wait();  // programmatic dependent launch: the forward FFT's coefficients are complete
  constexpr int SZ = AT_JC * 8 * 32;  // pairs per stage
  // the fields' columns follow one another (U, V, T, E, L apart); a δ ln ps tile has the third slot alone
  const unsigned C = a.Cin, fs = isp ? 0u : (unsigned)a.L;
  const unsigned o0 = (unsigned)m * nlat * C + (live ? (isp ? a.colP : a.colU) + col : 0);
  auto fetch = [&](int j0, int stage) {
    float2* dst = X + stage * SZ + warp * 32 + lane;
    for (int q = warp; q < 8 * AT_JC; q += nw, dst += nw * 32) {
      const unsigned f = q >> 1 & 3, jh = j0 + (q >> 3), j = q & 1 ? nlat - 1 - jh : jh;
      const bool on = live && (!isp || f == 2);
      cp_async8(dst, a.F + (o0 + j * C + (on ? f * fs : 0u)), on);
    }
  };
  const int nchunk = nh / AT_JC;
#pragma unroll
  for (int s = 0; s < AT_STAGES - 1; s++) {
    if (s < nchunk) fetch(s * AT_JC, s);
    cp_async_commit();  // (the first group holds the weights, too)
  }
  float var[AT_ROWS], vai[AT_ROWS], vbr[AT_ROWS], vbi[AT_ROWS], dar[AT_ROWS], dai[AT_ROWS], dbr[AT_ROWS], dbi[AT_ROWS],
      er[AT_ROWS], ei[AT_ROWS], tr[AT_ROWS], ti[AT_ROWS];
#pragma unroll
  for (int u = 0; u < AT_ROWS; u++)
    var[u] = vai[u] = vbr[u] = vbi[u] = dar[u] = dai[u] = dbr[u] = dbi[u] = er[u] = ei[u] = tr[u] = ti[u] = 0;
  // the hemisphere fold of a row's parity is south + sg north, the other parity's south - sg north (P_n^m is
  // symmetric about the equator for n - m even)
  const float sg = warp & 1 ? -1.f : 1.f;
  for (int c = 0; c < nchunk; c++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(AT_STAGES - 2) : "memory");
    __syncthreads();  // chunk c is staged, and every warp has read chunk c - 1
    if (c + AT_STAGES - 1 < nchunk) fetch((c + AT_STAGES - 1) * AT_JC, (c + AT_STAGES - 1) % AT_STAGES);
    cp_async_commit();
    if (warp < G) {
      const float* w = W + (size_t)c * AT_JC * wp + warp * 3 * AT_ROWS;
      const float2* x = X + (c % AT_STAGES) * SZ + lane;
#pragma unroll 2
      for (int jj = 0; jj < AT_JC; jj++) {
        float wP[4], wA[4], wB[4];
        ld4(w, wP);
        ld4(w + AT_ROWS, wA);
        ld4(w + 2 * AT_ROWS, wB);
        const float2 us = x[0], un = x[32], vs = x[64], vn = x[96], ts = x[128], tn = x[160], es = x[192], en = x[224];
        const float xux = fmaf(sg, un.x, us.x), xuy = fmaf(sg, un.y, us.y), yux = fmaf(-sg, un.x, us.x),
                    yuy = fmaf(-sg, un.y, us.y), xvx = fmaf(sg, vn.x, vs.x), xvy = fmaf(sg, vn.y, vs.y),
                    yvx = fmaf(-sg, vn.x, vs.x), yvy = fmaf(-sg, vn.y, vs.y), xex = fmaf(sg, en.x, es.x),
                    xey = fmaf(sg, en.y, es.y), xtx = fmaf(sg, tn.x, ts.x), xty = fmaf(sg, tn.y, ts.y);
#pragma unroll
        for (int u = 0; u < AT_ROWS; u++) {
          var[u] += (-xvy) * wA[u];
          vai[u] += xvx * wA[u];
          vbr[u] += yux * wB[u];
          vbi[u] += yuy * wB[u];
          dar[u] += (-xuy) * wA[u];
          dai[u] += xux * wA[u];
          dbr[u] += yvx * wB[u];
          dbi[u] += yvy * wB[u];
          er[u] += xex * wP[u];
          ei[u] += xey * wP[u];
          tr[u] += xtx * wP[u];
          ti[u] += xty * wP[u];
        }
        w += wp;
        x += 8 * 32;
      }
    }
  }
  if (warp >= G || !live) return;
#pragma unroll
  for (int u = 0; u < AT_ROWS; u++) {
    const int r = 8 * (warp >> 1) + (warp & 1) + 2 * u, n = m + r;
    if (r >= K) continue;
    const bool last = n == ns;  // row N+1 of the analysis is zero (Trans_Grid_To_Spherical!, :288-291)
    const float2 ot = last ? make_float2(0.f, 0.f) : make_float2(tr[u] * 0.5f, ti[u] * 0.5f);
    if (isp) {
      a.dlnps[(mrow + n) * a.E + col] = ot;
      continue;
    }
    float2 ov = make_float2(0.f, 0.f), od = ov;
    if (!last) {
      const float eig = tb.eig[mrow + n];
      ov.x = var[u] + -1.f * vbr[u];
      ov.y = vai[u] + -1.f * vbi[u];
      od.x = dar[u] + dbr[u];
      od.y = dai[u] + dbi[u];
      od.x = od.x - eig * (er[u] * 0.5f);
      od.y = od.y - eig * (ei[u] * 0.5f);
    }
    const size_t sidx = (mrow + n) * a.L + col;
    a.dvor[sidx] = ov;
    a.ddiv[sidx] = od;
    a.dt[sidx] = ot;
  }
}

size_t at_smem(const jgcm_mesh* m) {
  return (size_t)m->nh * at_pitch(m->ns) * sizeof(float) + (size_t)AT_STAGES * AT_JC * 8 * 32 * sizeof(float2);
}
// whether the tiled kernel serves this mesh
bool at_fits(const jgcm_mesh* m) {
  return m->nh % AT_JC == 0 && 32 * at_groups(m->ns + 1) <= 640 && at_smem(m) <= kSmemBudget;
}

}  // namespace

// total wavenumbers per thread: two of one parity for member ensembles (each folded input loaded
// from shared memory serves both: the analysis is shared-memory-bound at that scale), one otherwise
// (shorter chains for the latency-bound single member)
static int hs_analysis_np(const jgcm_mesh* m, int E) { return !is_fp64(m) && E >= 4 ? 2 : 1; }

// threads per level of a block: the largest row count of an m pair (rows r = 4 i + b, b < 2, for
// two rows per thread)
static int hs_analysis_rows(const jgcm_mesh* m, int np) {
  if (np == 1) return m->N + 4;
  int q = 0;
  for (int m1 = 0; m1 <= m->N / 2; m1++) {
    const int m2 = m->N - m1, K1 = m->ns + 1 - m1, K2 = m2 != m1 ? m->ns + 1 - m2 : 0;
    q = std::max(q, 2 * ((K1 + 3) / 4) + 2 * ((K2 + 3) / 4));
  }
  return q;
}

// Levels per block and lanes per output (SP) of the Held-Suarez analysis: the tuned number of levels when set
// (clamped to what a block of 256 threads holds); for FP32 ensembles as many as a block holds; else what makes the
// load of the busiest sub-partition least: rounds of blocks over the SMs x (a block's warps on one of its four
// sub-partitions / SP + half a unit for staging and folds), a block of δ ln ps alone not counted, the smaller block
// at a tie.  Measured in FP64 (levels x lanes; as many as a block holds first): T42L20 5x1 32.8 us, 4x1 28.7, 2x2 30.8,
// 3x1 43; T21L20 10x1 20.6, 2x1 16.4, 2x2 12.3; T31L20 7x1 30.8, 4x1 20.6, 3x2 18.5; 4 members of T42L20 5x1 100, 4x1 76,
// 2x2 83 (two rows per thread 117).  In FP32, a member's step: T42L20 5 levels 38.05 us, 4 37.6; T31L13 7 35.35, 2 33.7;
// T21L20 10 34.7, 2 33.8.
struct HSAnaShape {
  int LG, SP;
};
static HSAnaShape hs_analysis_shape(const jgcm_mesh* m, int nd, int E) {
  const int rows = hs_analysis_rows(m, hs_analysis_np(m, E)), lg_max = 256 / rows;
  if (m->hs_levels > 0) return {std::min(m->hs_levels, lg_max), 1};
  if (!is_fp64(m) && E >= 4) return {lg_max, 1};
  HSAnaShape best = {lg_max, 1};
  double least = 1e30;
  for (int sp = is_fp64(m) ? 2 : 1; sp >= 1; sp--)
    for (int lg = 1; lg <= std::min(256 / (rows * sp), nd + 1); lg++) {
      const long blocks = (long)(m->N / 2 + 1) * ((nd + lg - 1) / lg) * E;
      const int warps = (rows * lg * sp + 31) / 32;
      const double cost = (double)((blocks + m->sm_count - 1) / m->sm_count) * ((double)((warps + 3) / 4) / sp + 0.5);
      if (cost < least) {
        least = cost;
        best = {lg, sp};
      }
    }
  return best;
}

// The tiled kernel serves an FP32 launch of E members: from five blocks per four SMs on (T42L20, 4 members
// 15.5 -> 16.5 us, 8 members 23 -> 19, 16 members 38 -> 25, 4 members of T63L20 29.6 -> 27.4, one 14 -> 22)
static int at_tiles(int nd, int E) { return (nd * E + 31) / 32 + (E + 31) / 32; }
static bool at_pays(const jgcm_mesh* m, int nd, int E) {
  return (size_t)4 * at_tiles(nd, E) * (m->N + 1) >= (size_t)5 * m->sm_count;
}

// The tiled kernel's weights, built with the first Held-Suarez model that it serves (freed with the mesh)
int hs_tables_build(jgcm_mesh* m, int nd, int E) {
  if (m->d_at || is_fp64(m) || !at_fits(m) || !at_pays(m, nd, E)) return JGCM_OK;
  const size_t n = (size_t)(m->N + 1) * m->nh * at_pitch(m->ns);
  JG_CUDA(cudaMalloc(&m->d_at, n * sizeof(float)));
  k_at_weights<<<(int)std::min<size_t>((n + 255) / 256, 1184), 256, 0, m->stream>>>(tables<float>(m), m->d_at, m->N, m->ns, m->nh);
  JG_CUDA(cudaGetLastError());
  return JGCM_OK;
}

// The Held-Suarez analysis kernel serves this mesh: not tuned away (levels per block -1), SIMT
// Legendre path, weights in 16-byte rows, shared memory within the budget.
bool hs_analysis_fits(const jgcm_mesh* m, int nd, int E) {
  if (m->hs_levels < 0) return false;  // tuned to the general analysis kernel
  if (m->tc.on && !m->simt_legendre) return false;
  if (m->nh % 4 != 0) return false;  // weights four at a time (and rows of whole 16-byte chunks)
  const int LG = hs_analysis_shape(m, nd, E).LG;
  if (LG < 1) return false;
  const size_t sm = is_fp64(m) ? hs_analysis_smem<double>(m, LG) : hs_analysis_smem<float>(m, LG);
  return sm <= kSmemBudget;
}

// Forward FFT of the step's tendency groups (the FFT plan's columns: δu cos, δv cos, δT, energy
// at colU, colV, colT, colE with L columns each, δ ln ps at colP with E), then the analysis.
template <typename T>
int launch_hs_analysis(jgcm_mesh* m, const FFTPlan& fp, int colU, int colV, int colE, int colT, int colP, int nd,
                       int E, void* dvor, void* ddiv, void* dt, void* dlnps, cudaStream_t st, void* fbuf, int cap) {
  JG_ARG(hs_analysis_fits(m, nd, E), "the Held-Suarez analysis kernel does not fit this mesh");
  JG_TRY(launch_fft_only<T>(m, fp, st, fbuf, cap));
  const auto [LG, sp] = hs_analysis_shape(m, nd, E);
  const size_t sm = hs_analysis_smem<T>(m, LG);
  JG_TRY(g_hs_ana_smem[sizeof(T) == 8 ? 1 : 0].run([]() -> int {
    JG_CUDA(cudaFuncSetAttribute(k_hs_analysis<T, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    if constexpr (std::is_same<T, double>::value) {
      JG_CUDA(cudaFuncSetAttribute(k_hs_analysis<T, 1, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    } else {
      JG_CUDA(cudaFuncSetAttribute(k_hs_analysis<T, 2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
      JG_CUDA(cudaFuncSetAttribute(k_hs_analysis_tiles<384, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
      JG_CUDA(cudaFuncSetAttribute(k_hs_analysis_tiles<640, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget));
    }
    return JGCM_OK;
  }));
  HSAnaArgs<T> a;
  a.F = (const V2<T>*)(fbuf ? fbuf : m->d_fbuf);
  a.dvor = (V2<T>*)dvor;
  a.ddiv = (V2<T>*)ddiv;
  a.dt = (V2<T>*)dt;
  a.dlnps = (V2<T>*)dlnps;
  a.Cin = fp.C;
  a.colU = colU;
  a.colV = colV;
  a.colE = colE;
  a.colT = colT;
  a.colP = colP;
  a.nd = nd;
  a.L = nd * E;
  a.E = E;
  a.N = m->N;
  a.ns = m->ns;
  a.nlat = m->nlat;
  a.nh = m->nh;
  a.LG = LG;
  if constexpr (std::is_same<T, float>::value) {
    const int th = 32 * at_groups(m->ns + 1);
    // (the columns in the step's order, 32-bit offsets)
    if (m->d_at && m->hs_levels == 0 && at_pays(m, nd, E) && colV == colU + a.L && colT == colU + 2 * a.L &&
        colE == colU + 3 * a.L && (size_t)(m->N + 1) * m->nlat * fp.C < ((size_t)1 << 31)) {
      const dim3 gt(at_tiles(nd, E), m->N + 1);
      JG_CUDA(th <= 384 ? launch_pdl(k_hs_analysis_tiles<384, 2>, gt, th, at_smem(m), st, a, tables<float>(m), m->d_at)
                        : launch_pdl(k_hs_analysis_tiles<640, 1>, gt, th, at_smem(m), st, a, tables<float>(m), m->d_at));
      mark(st);
      JG_CUDA(cudaGetLastError());
      return JGCM_OK;
    }
  }
  const int np = hs_analysis_np(m, E);
  const int threads = (hs_analysis_rows(m, np) * LG * sp + 31) / 32 * 32;
  dim3 grid(m->N / 2 + 1, (nd + 1 + LG - 1) / LG, E);
  auto kernel = k_hs_analysis<T, 1, 1>;
  if constexpr (std::is_same<T, double>::value) {
    if (sp == 2) kernel = k_hs_analysis<T, 1, 2>;
  } else {
    if (np == 2) kernel = k_hs_analysis<T, 2, 1>;
  }
  JG_CUDA(launch_pdl(kernel, grid, threads, sm, st, a, tables<T>(m)));
  mark(st);
  JG_CUDA(cudaGetLastError());
  return JGCM_OK;
}

template int launch_hs_analysis<float>(jgcm_mesh*, const FFTPlan&, int, int, int, int, int, int, int, void*, void*,
                                       void*, void*, cudaStream_t, void*, int);
template int launch_hs_analysis<double>(jgcm_mesh*, const FFTPlan&, int, int, int, int, int, int, int, void*, void*,
                                        void*, void*, cudaStream_t, void*, int);

}  // namespace jgcm
