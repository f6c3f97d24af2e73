// C ABI of the design-variable maps (element fields are dense ex*ey*ez
// device arrays, coefficients dense n_coeff device arrays).
#include "rso_internal.cuh"
#include <cstring>

using namespace rso;

__global__ void k_f2d_n(const float* __restrict__ a, double* __restrict__ b, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (double)a[i];
}
__global__ void k_d2f_n(const double* __restrict__ a, float* __restrict__ b, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

static rso_status finish(rso_handle* h) {
  RSO_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  return RSO_OK;
}

// The maps read and write the caller's arrays directly.  An output (ne floats) may
// overlap an input, the shell mask too: the input (ne entries, or none) is then read
// from a copy in a scratch field.
template <typename T>
static rso_status apart(rso_handle* h, const T** in, const float* out, float* scratch) {
  const size_t ne = (size_t)h->L[0].ne;
  const char *a = (const char*)*in, *b = (const char*)out;
  if (!a || a >= b + sizeof(float) * ne || a + sizeof(T) * ne <= b) return RSO_OK;
  RSO_CHECK_CUDA(h, cudaMemcpyAsync(scratch, *in, sizeof(T) * ne, cudaMemcpyDeviceToDevice, h->stream));
  *in = reinterpret_cast<const T*>(scratch);
  return RSO_OK;
}

static rso_status sensitivity_api(rso_handle* h, const double* u, float* out, int energy) {
  if (!h || !u || !out) return RSO_ERR_INVALID_ARG;
  RSO_TRY(pad_nodes(h, 0, u, h->L[0].u64));
  RSO_TRY(zero_support(h, h->L[0].u64));
  RSO_TRY(sensitivity(h, h->L[0].u64, out, energy, true));
  return finish(h);
}

extern "C" rso_status rso_sensitivity(rso_handle* h, const double* u, float* sens) {
  return sensitivity_api(h, u, sens, 0);
}
extern "C" rso_status rso_element_energy(rso_handle* h, const double* u, float* en) {
  return sensitivity_api(h, u, en, 1);
}

extern "C" rso_status rso_heaviside(rso_handle* h, const float* in, double beta, const uint8_t* shell, float* out) {
  if (!h || !in || !out) return RSO_ERR_INVALID_ARG;
  RSO_TRY(apart(h, &in, out, h->e_a));
  RSO_TRY(apart(h, &shell, out, h->e_b));
  RSO_TRY(heaviside(h, in, beta, shell, out, true));
  return finish(h);
}

extern "C" rso_status rso_heaviside_chain(rso_handle* h, const float* rho, double beta, const float* gin, float* gout) {
  if (!h || !rho || !gin || !gout) return RSO_ERR_INVALID_ARG;
  RSO_TRY(apart(h, &rho, gout, h->e_a));
  RSO_TRY(apart(h, &gin, gout, h->e_b));
  RSO_TRY(heaviside_chain(h, rho, beta, gin, gout, true));
  return finish(h);
}

static rso_status filter_api(rso_handle* h, double R, const float* in, float* out, int adjoint) {
  if (!h || !in || !out || !(R > 0)) return RSO_ERR_INVALID_ARG;
  RSO_TRY(apart(h, &in, out, h->e_a));
  RSO_TRY(filter(h, R, in, out, adjoint, true));
  return finish(h);
}

extern "C" rso_status rso_filter(rso_handle* h, double R, const float* in, float* out) {
  return filter_api(h, R, in, out, 0);
}
extern "C" rso_status rso_density_filter(rso_handle* h, double R, const float* in, float* out) {
  return filter_api(h, R, in, out, 0);
}
extern "C" rso_status rso_density_filter_adjoint(rso_handle* h, double R, const float* in, float* out) {
  return filter_api(h, R, in, out, 1);
}

extern "C" rso_status rso_volume(rso_handle* h, const float* rho, double* vol) {
  if (!h || !rho || !vol) return RSO_ERR_INVALID_ARG;
  return volume(h, rho, vol, true);
}

extern "C" rso_status rso_spline_setup(rso_handle* h, int order, int px, int py, int pz, int* n_coeff) {
  if (!h) return RSO_ERR_INVALID_ARG;
  RSO_TRY(spline_setup(h, order, px, py, pz));
  if (n_coeff) *n_coeff = (int)h->sp.n_coeff;
  return finish(h);
}

extern "C" rso_status rso_spline_axis(rso_handle* h, int axis, int* idx, double* N, double* dN) {
  if (!h || axis < 0 || axis > 2 || !h->sp.order) return RSO_ERR_INVALID_ARG;
  const Spline& s = h->sp;
  if (idx) std::memcpy(idx, s.h_idx[axis].data(), sizeof(int) * s.h_idx[axis].size());
  if (N) std::memcpy(N, s.h_N[axis].data(), sizeof(double) * s.h_N[axis].size());
  if (dN) std::memcpy(dN, s.h_dN[axis].data(), sizeof(double) * s.h_dN[axis].size());
  return RSO_OK;
}

extern "C" rso_status rso_coeff2density(rso_handle* h, const float* coeff, const uint8_t* shell, float* rho_hat) {
  if (!h || !coeff || !rho_hat) return RSO_ERR_INVALID_ARG;
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  RSO_TRY(apart(h, &shell, rho_hat, h->e_a));
  RSO_TRY(coeff2density(h, coeff, shell, rho_hat, true));
  return finish(h);
}

extern "C" rso_status rso_density2coeff_adjoint(rso_handle* h, const float* g, const uint8_t* shell, float* dc) {
  if (!h || !g || !dc) return RSO_ERR_INVALID_ARG;
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  RSO_TRY(density2coeff(h, g, shell, h->coef_b, true));
  k_d2f_n<<<cdiv(h->sp.n_coeff, 256), 256, 0, h->stream>>>(h->coef_b, dc, h->sp.n_coeff); rso::note_launch();
  RSO_TRY(launch_check(h, "density2coeff"));
  return finish(h);
}

extern "C" rso_status rso_selfsupport(rso_handle* h, const float* coeff, double beta, int mode, double opt_angle,
                                      double default_angle, float* per, float* dc, double* value, double* count,
                                      double* dirsum) {
  if (!h || !coeff || mode < 0 || mode > 5) return RSO_ERR_INVALID_ARG;
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  k_f2d_n<<<cdiv(h->sp.n_coeff, 256), 256, 0, h->stream>>>(coeff, h->coef_a, h->sp.n_coeff); rso::note_launch();
  RSO_TRY(selfsupport(h, h->coef_a, beta, mode, opt_angle, default_angle, per, dc ? h->coef_b : nullptr, value, count,
                      dirsum));
  if (dc) { k_d2f_n<<<cdiv(h->sp.n_coeff, 256), 256, 0, h->stream>>>(h->coef_b, dc, h->sp.n_coeff); rso::note_launch(); }
  RSO_TRY(launch_check(h, "selfsupport"));
  return finish(h);
}
