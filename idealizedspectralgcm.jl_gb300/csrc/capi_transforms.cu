// capi_transforms.cu -- host-pointer C ABI of the mesh-level operators (jgcm.h).
//
// Each call converts its FP64 host arrays (reference layout; read and written in place by the kernels
// where the device can, else through the mesh's staging buffer: host_in, host_out) to the device layout
// and precision, runs the transform kernels on the mesh stream and blocks until the results are on the
// host.  Grids of an FP64 mesh have the host's layout and type: its FFT kernels read and write them
// without a conversion.
#include <cstring>
#include <initializer_list>

#include "jgcm_internal.cuh"

using namespace jgcm;

namespace {

// every argument of a call, before anything is queued
int check_args(const jgcm_mesh* m, int nlev, std::initializer_list<const double*> arrays) {
  JG_ARG(m != nullptr, "mesh is NULL");
  JG_ARG(nlev == m->nd || nlev == 1, "third dimension must be nd=%d or 1 (got %d)", m->nd, nlev);
  for (const double* a : arrays) JG_ARG(a != nullptr, "an array of the call is NULL");
  return JGCM_OK;
}

double* slot(jgcm_mesh* m, int i) { return m->d_stage + (size_t)i * m->stage_slot; }

// input spectrum / grid `i` of a call as the kernels read it (device layout and precision)
int spec_in(jgcm_mesh* m, int i, const double* src, int nlev, const void** use) {
  const double* p;
  JG_TRY(host_in(m, src, 2 * spec_elems(m, nlev), slot(m, i), m->stream, &p));
  JG_TRY(spec_host_to_dev(m, p, m->d_spec[i], nlev, m->stream));
  *use = m->d_spec[i];
  return JGCM_OK;
}
// (copy: as a copy on the device on FP64 meshes, too, whose kernels otherwise read the host's array)
int grid_in(jgcm_mesh* m, int i, const double* src, int nlev, const void** use, bool copy = false) {
  const double* p;
  const size_t n = grid_elems(m, nlev);
  JG_TRY(host_in(m, src, n, slot(m, i), m->stream, &p));
  *use = p;
  if (is_fp64(m) && !copy) return JGCM_OK;
  JG_TRY(grid_host_to_dev(m, p, m->d_grid[i], n, m->stream));
  *use = m->d_grid[i];
  return JGCM_OK;
}
// output grid of a call, staged in slot `i`: where the kernels write it, and its way to the host
struct GridOut {
  double *dst, *use;
  void* dev;
};
int grid_out(jgcm_mesh* m, int i, double* dst, int nlev, GridOut* o) {
  o->dst = dst;
  JG_TRY(host_out(m, dst, grid_elems(m, nlev), slot(m, i), &o->use));
  o->dev = is_fp64(m) ? (void*)o->use : m->d_grid[i];
  return JGCM_OK;
}
int grid_done(jgcm_mesh* m, const GridOut& o, int nlev) {
  const size_t n = grid_elems(m, nlev);
  if (!is_fp64(m)) JG_TRY(grid_dev_to_host(m, o.dev, o.use, n, m->stream));
  return host_out_done(o.dst, o.use, n, m->stream);
}
// the device spectrum d_spec[i] to the host array dst (staged in slot i)
int spec_done(jgcm_mesh* m, int i, double* dst, int nlev) {
  double* p;
  const size_t n = 2 * spec_elems(m, nlev);
  JG_TRY(host_out(m, dst, n, slot(m, i), &p));
  JG_TRY(spec_dev_to_host(m, m->d_spec[i], p, nlev, m->stream));
  return host_out_done(dst, p, n, m->stream);
}
int finish(jgcm_mesh* m, HostCall& call) {
  JG_CUDA(cudaStreamSynchronize(m->stream));
  call.done = true;
  JG_CUDA(cudaGetLastError());
  if (m->tc.on) JG_TRY(tc_status(m));  // a tensor-core kernel whose bounded wait gave up
  return JGCM_OK;
}

template <typename T>
int s2g_run(jgcm_mesh* m, const S2GPlan& sp, const IFFTPlan& ip) {
  return launch_s2g<T>(m, sp, ip, m->stream);
}
int s2g(jgcm_mesh* m, const S2GPlan& sp, const IFFTPlan& ip) {
  return is_fp64(m) ? s2g_run<double>(m, sp, ip) : s2g_run<float>(m, sp, ip);
}
int g2s(jgcm_mesh* m, const FFTPlan& fp, const G2SPlan& gp) {
  return is_fp64(m) ? launch_g2s<double>(m, fp, gp, m->stream) : launch_g2s<float>(m, fp, gp, m->stream);
}

S2GGroup s2g_group(int op, const void* a, const void* b, int L, int col0) {
  S2GGroup g;
  memset(&g, 0, sizeof(g));
  g.op = op;
  g.a = a;
  g.b = b;
  g.L = L;
  g.col0 = col0;
  return g;
}
GridOutGroup out_group(int epi, void* dst, int L, int col0) {
  GridOutGroup g;
  memset(&g, 0, sizeof(g));
  g.epi = epi;
  g.dst = dst;
  g.L = L;
  g.col0 = col0;
  return g;
}
GridInGroup in_group(int pro, const void* src, int L, int col0) {
  GridInGroup g;
  memset(&g, 0, sizeof(g));
  g.pro = pro;
  g.src = src;
  g.L = L;
  g.col0 = col0;
  return g;
}
SpecOutGroup spec_group(int op, void* dst, int L, int col0, int colA, int colB, int colE) {
  SpecOutGroup g;
  memset(&g, 0, sizeof(g));
  g.op = op;
  g.dst = dst;
  g.L = L;
  g.col0 = col0;
  g.colA = colA;
  g.colB = colB;
  g.colE = colE;
  g.colH = -1;
  return g;
}

// spectral gradient -> two grid fields (device), used by compute_gradients / advection
int gradients_dev(jgcm_mesh* m, const void* d_spec, int nlev, void* d_gl, void* d_gt) {
  S2GPlan sp;
  memset(&sp, 0, sizeof(sp));
  sp.ng = 2;
  sp.C = 2 * nlev;
  sp.g[0] = s2g_group(S2G_DLAM, d_spec, nullptr, nlev, 0);
  sp.g[1] = s2g_group(S2G_DTH, d_spec, nullptr, nlev, nlev);
  IFFTPlan ip;
  memset(&ip, 0, sizeof(ip));
  ip.ng = 2;
  ip.C = 2 * nlev;
  ip.g[0] = out_group(EPI_DIVCOS, d_gl, nlev, 0);
  ip.g[1] = out_group(EPI_DIVCOS, d_gt, nlev, nlev);
  return s2g(m, sp, ip);
}

}  // namespace

namespace {
// one group of a synthesis / of an analysis: plan, kernels, host arrays
int synthesis(jgcm_mesh* m, int op, int epi, const double* spec, int nlev, double* grid) {
  JG_TRY(check_args(m, nlev, {spec, grid}));
  HostCall call(m->stream);
  const void* a;
  GridOut o;
  JG_TRY(spec_in(m, 0, spec, nlev, &a));
  JG_TRY(grid_out(m, 1, grid, nlev, &o));
  S2GPlan sp;
  memset(&sp, 0, sizeof(sp));
  sp.ng = 1;
  sp.C = nlev;
  sp.g[0] = s2g_group(op, a, nullptr, nlev, 0);
  IFFTPlan ip;
  memset(&ip, 0, sizeof(ip));
  ip.ng = 1;
  ip.C = nlev;
  ip.g[0] = out_group(epi, o.dev, nlev, 0);
  JG_TRY(s2g(m, sp, ip));
  JG_TRY(grid_done(m, o, nlev));
  return finish(m, call);
}
int analysis(jgcm_mesh* m, int op, const double* grid, int nlev, double* spec) {
  JG_TRY(check_args(m, nlev, {grid, spec}));
  HostCall call(m->stream);
  const void* x;
  JG_TRY(grid_in(m, 1, grid, nlev, &x));
  FFTPlan fp;
  memset(&fp, 0, sizeof(fp));
  fp.ng = 1;
  fp.C = nlev;
  fp.g[0] = in_group(PRO_NONE, x, nlev, 0);
  G2SPlan gp;
  memset(&gp, 0, sizeof(gp));
  gp.ng = 1;
  gp.C = nlev;
  gp.g[0] = spec_group(op, m->d_spec[0], nlev, 0, 0, -1, -1);
  gp.g[0].scale = m->nlon;
  JG_TRY(g2s(m, fp, gp));
  JG_TRY(spec_done(m, 0, spec, nlev));
  return finish(m, call);
}
}  // namespace

extern "C" int jgcm_trans_spherical_to_grid(jgcm_mesh* m, const double* snm, int nlev, double* pfield) {
  return synthesis(m, S2G_PLAIN, EPI_NONE, snm, nlev, pfield);
}

extern "C" int jgcm_trans_grid_to_spherical(jgcm_mesh* m, const double* pfield, int nlev, double* snm) {
  return analysis(m, G2S_PLAIN, pfield, nlev, snm);
}

// Adjoint of Trans_Spherical_To_Grid!: grid cotangent -> spectral cotangent (row N+1 included).
extern "C" int jgcm_trans_spherical_to_grid_adjoint(jgcm_mesh* m, const double* grid_bar, int nlev, double* spec_bar) {
  return analysis(m, G2S_ADJ_S2G, grid_bar, nlev, spec_bar);
}

// Adjoint of Trans_Grid_To_Spherical!: spectral cotangent (row N+1 ignored) -> grid cotangent.
extern "C" int jgcm_trans_grid_to_spherical_adjoint(jgcm_mesh* m, const double* spec_bar, int nlev, double* grid_bar) {
  return synthesis(m, S2G_ADJ_G2S, EPI_ADJ_G2S, spec_bar, nlev, grid_bar);
}

extern "C" int jgcm_trans_grid_to_fourier(jgcm_mesh* m, const double* pfield, int nlev, double* fourier) {
  JG_TRY(check_args(m, nlev, {pfield, fourier}));
  HostCall call(m->stream);
  const size_t nf = 2 * grid_elems(m, nlev);  // complex [nlev][nlat][nlon]: staging slots 1 and 2
  const void* x;
  double* f;
  // the kernel reads rows and writes modes at once: a field that lies in the output array is copied first (the
  // other calls write in place after everything has been read)
  const bool overlap = pfield < fourier + nf && fourier < pfield + nf / 2;
  JG_TRY(grid_in(m, 0, pfield, nlev, &x, overlap));
  JG_TRY(host_out(m, fourier, nf, slot(m, 1), &f));
  JG_TRY(fourier_full_to_host(m, x, nlev, f, m->stream));
  JG_TRY(host_out_done(fourier, f, nf, m->stream));
  return finish(m, call);
}

extern "C" int jgcm_vor_div_from_grid_uv(jgcm_mesh* m, const double* u, const double* v, int nlev, double* vor,
                                         double* div) {
  JG_TRY(check_args(m, nlev, {u, v, vor, div}));
  HostCall call(m->stream);
  const void *gu, *gv;
  JG_TRY(grid_in(m, 0, u, nlev, &gu));
  JG_TRY(grid_in(m, 1, v, nlev, &gv));
  FFTPlan fp;
  memset(&fp, 0, sizeof(fp));
  fp.ng = 2;
  fp.C = 2 * nlev;
  fp.g[0] = in_group(PRO_MULCOS, gu, nlev, 0);     // u cos
  fp.g[1] = in_group(PRO_MULCOS, gv, nlev, nlev);  // v cos
  G2SPlan gp;
  memset(&gp, 0, sizeof(gp));
  gp.ng = 2;
  gp.C = 2 * nlev;
  gp.g[0] = spec_group(G2S_VOR, m->d_spec[0], nlev, 0, nlev, 0, -1);     // A = v cos, B = u cos, sign -1
  gp.g[1] = spec_group(G2S_DIV, m->d_spec[1], nlev, nlev, 0, nlev, -1);  // A = u cos, B = v cos, sign +1
  JG_TRY(g2s(m, fp, gp));
  JG_TRY(spec_done(m, 0, vor, nlev));
  JG_TRY(spec_done(m, 1, div, nlev));
  return finish(m, call);
}

extern "C" int jgcm_uv_grid_from_vor_div(jgcm_mesh* m, const double* vor, const double* div, int nlev, double* u,
                                         double* v) {
  JG_TRY(check_args(m, nlev, {vor, div, u, v}));
  HostCall call(m->stream);
  const void *sv, *sd;
  GridOut ou, ov;
  JG_TRY(spec_in(m, 0, vor, nlev, &sv));
  JG_TRY(spec_in(m, 1, div, nlev, &sd));
  JG_TRY(grid_out(m, 2, u, nlev, &ou));
  JG_TRY(grid_out(m, 3, v, nlev, &ov));
  S2GPlan sp;
  memset(&sp, 0, sizeof(sp));
  sp.ng = 2;
  sp.C = 2 * nlev;
  sp.g[0] = s2g_group(S2G_UCOS, sv, sd, nlev, 0);
  sp.g[1] = s2g_group(S2G_VCOS, sv, sd, nlev, nlev);
  IFFTPlan ip;
  memset(&ip, 0, sizeof(ip));
  ip.ng = 2;
  ip.C = 2 * nlev;
  ip.g[0] = out_group(EPI_DIVCOS, ou.dev, nlev, 0);
  ip.g[1] = out_group(EPI_DIVCOS, ov.dev, nlev, nlev);
  JG_TRY(s2g(m, sp, ip));
  JG_TRY(grid_done(m, ou, nlev));
  JG_TRY(grid_done(m, ov, nlev));
  return finish(m, call);
}

extern "C" int jgcm_compute_gradients(jgcm_mesh* m, const double* hs, int nlev, double* gdl, double* gdt) {
  JG_TRY(check_args(m, nlev, {hs, gdl, gdt}));
  HostCall call(m->stream);
  const void* a;
  GridOut ol, ot;
  JG_TRY(spec_in(m, 0, hs, nlev, &a));
  JG_TRY(grid_out(m, 2, gdl, nlev, &ol));
  JG_TRY(grid_out(m, 3, gdt, nlev, &ot));
  JG_TRY(gradients_dev(m, a, nlev, ol.dev, ot.dev));
  JG_TRY(grid_done(m, ol, nlev));
  JG_TRY(grid_done(m, ot, nlev));
  return finish(m, call);
}

extern "C" int jgcm_add_horizontal_advection(jgcm_mesh* m, const double* hs, const double* u, const double* v,
                                             int nlev, double* dh) {
  JG_TRY(check_args(m, nlev, {hs, u, v, dh}));
  HostCall call(m->stream);
  const size_t ng = grid_elems(m, nlev);
  const void* a;
  const double *pu, *pv, *ph;
  JG_TRY(spec_in(m, 0, hs, nlev, &a));
  JG_TRY(gradients_dev(m, a, nlev, m->d_grid[0], m->d_grid[1]));
  JG_TRY(host_in(m, u, ng, slot(m, 1), m->stream, &pu));
  JG_TRY(host_in(m, v, ng, slot(m, 2), m->stream, &pv));
  JG_TRY(host_in(m, dh, ng, slot(m, 3), m->stream, &ph));
  double* out;
  JG_TRY(host_out(m, dh, ng, slot(m, 3), &out));
  JG_TRY(advection_update(m, m->d_grid[0], m->d_grid[1], pu, pv, ph, out, ng, m->stream));
  JG_TRY(host_out_done(dh, out, ng, m->stream));
  return finish(m, call);
}

extern "C" int jgcm_apply_laplacian(jgcm_mesh* m, double* spe, int nlev) {
  JG_TRY(check_args(m, nlev, {spe}));
  HostCall call(m->stream);
  const void* a;
  JG_TRY(spec_in(m, 0, spe, nlev, &a));
  JG_TRY(apply_laplacian(m, m->d_spec[0], nlev, m->stream));
  JG_TRY(spec_done(m, 0, spe, nlev));
  return finish(m, call);
}

extern "C" int jgcm_area_weighted_global_mean(jgcm_mesh* m, const double* grid, double* out) {
  JG_TRY(check_args(m, 1, {grid, out}));
  HostCall call(m->stream);
  const void* x;
  // copied: the one block of the sum would wait for the host link row by row (T42 66 us, T85 103; copied 35 and 48)
  JG_TRY(grid_in(m, 0, grid, 1, &x, true));
  JG_TRY(area_mean(m, x, m->d_red, m->stream));
  JG_CUDA(cudaMemcpyAsync(out, m->d_red, 8, cudaMemcpyDeviceToHost, m->stream));
  return finish(m, call);
}
