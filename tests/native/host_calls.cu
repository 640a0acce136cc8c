// The host-pointer entry points of capi_transforms.cu over stand-ins for everything they queue, for tests on the
// CPU: each stand-in records 'q' (work queued that may touch the caller's arrays) and can be told to fail; a
// stream synchronisation records 's'.  capi_transforms.cu launches no kernel itself, and the process that loads
// this sees no device.
#include "capi_transforms.cu"

#include <cstdio>

namespace {
std::string g_events;
int g_countdown;  // the stand-in call that fails, 1 = the next one; 0 = none

int queue() {
  if (g_countdown && --g_countdown == 0) return JGCM_E_CUDA;
  g_events += 'q';
  return JGCM_OK;
}
cudaError_t stub_error(cudaError_t e) { return e; }
}  // namespace

// the runtime calls that the entry points make themselves (linked with --wrap)
extern "C" cudaError_t __wrap_cudaStreamSynchronize(cudaStream_t) {
  g_events += 's';
  return stub_error(cudaSuccess);
}
extern "C" cudaError_t __wrap_cudaGetLastError() { return stub_error(cudaSuccess); }
extern "C" cudaError_t __wrap_cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) {
  return queue() == JGCM_OK ? cudaSuccess : cudaErrorInvalidValue;
}

namespace jgcm {
void set_error(const char*, ...) {}
int host_in(jgcm_mesh*, const double* src, size_t, double*, cudaStream_t, const double** use) {
  JG_ARG(src != nullptr, "input");
  *use = src;
  return JGCM_OK;
}
int host_out(jgcm_mesh*, double* dst, size_t, double*, double** use) {
  JG_ARG(dst != nullptr, "output");
  *use = dst;
  return JGCM_OK;
}
int host_out_done(double*, const double*, size_t, cudaStream_t) { return JGCM_OK; }
int spec_host_to_dev(jgcm_mesh*, const double*, void*, int, cudaStream_t) { return queue(); }
int spec_dev_to_host(jgcm_mesh*, const void*, double*, int, cudaStream_t) { return queue(); }
int grid_host_to_dev(jgcm_mesh*, const double*, void*, size_t, cudaStream_t) { return queue(); }
int grid_dev_to_host(jgcm_mesh*, const void*, double*, size_t, cudaStream_t) { return queue(); }
int fourier_full_to_host(jgcm_mesh*, const void*, int, double*, cudaStream_t) { return queue(); }
int apply_laplacian(jgcm_mesh*, void*, int, cudaStream_t) { return queue(); }
int advection_update(jgcm_mesh*, const void*, const void*, const double*, const double*, const double*, double*, size_t,
                     cudaStream_t) {
  return queue();
}
int area_mean(jgcm_mesh*, const void*, double*, cudaStream_t) { return queue(); }
int tc_status(jgcm_mesh*) { return JGCM_OK; }
template <typename T>
int launch_s2g(jgcm_mesh*, const S2GPlan&, const IFFTPlan&, cudaStream_t, void*, int) { return queue(); }
template <typename T>
int launch_g2s(jgcm_mesh*, const FFTPlan&, const G2SPlan&, cudaStream_t, void*, int) { return queue(); }
template int launch_s2g<float>(jgcm_mesh*, const S2GPlan&, const IFFTPlan&, cudaStream_t, void*, int);
template int launch_s2g<double>(jgcm_mesh*, const S2GPlan&, const IFFTPlan&, cudaStream_t, void*, int);
template int launch_g2s<float>(jgcm_mesh*, const FFTPlan&, const G2SPlan&, cudaStream_t, void*, int);
template int launch_g2s<double>(jgcm_mesh*, const FFTPlan&, const G2SPlan&, cudaStream_t, void*, int);
}  // namespace jgcm

extern "C" jgcm_mesh* stub_mesh(int precision) {
  jgcm_mesh* m = new jgcm_mesh();
  m->N = 5;
  m->ns = 6;
  m->nlat = 10;
  m->nlon = 16;
  m->nd = 3;
  m->precision = precision;
  return m;
}
extern "C" void stub_begin(int fail_at) {
  g_events.clear();
  g_countdown = fail_at;
}
extern "C" const char* stub_events() { return g_events.c_str(); }
