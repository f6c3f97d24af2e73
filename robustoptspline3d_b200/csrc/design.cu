// Design-variable maps and their adjoints on the element grid:
// compliance sensitivity, Heaviside projection, sensitivity/density filter,
// B-spline density map (forward and race-free adjoint) and the self-support
// constraint with its analytic coefficient gradient.
//
// The B-spline maps are separable.  Element centres lie on the element grid,
// so the basis values depend on one coordinate each; they are tabulated per
// axis (span index, order values and first derivatives) and the adjoint
// dC/dc_ijk = sum_e g_e Nx_i(x_e) Ny_j(y_e) Nz_k(z_e) is evaluated as three
// successive one-axis contractions (a gather per output, no atomics), instead
// of the reference's racy per-element scatter (grid/Grid.cu:3797, 3908, 8220).
// The forward maps go through the same three contractions in reverse.
#include "rso_internal.cuh"
#include <cmath>
#include <algorithm>

namespace rso {

// Element fields come in two layouts, the padded one of the handle and the
// dense one of the public interface; every kernel here reads and writes either
// through a view, so that the public calls need no conversion passes (two or
// three of 99 us each per call at 256^3, as long as most maps themselves).
struct View {
  long long off, sz;
  int sy;
  __device__ __forceinline__ long long at(int x, int y, int z) const { return off + x + (long long)sy * y + sz * z; }
};
static View view_of(const Level& l, bool dense) {
  if (dense) return {0, (long long)l.ex * l.ey, l.ex};
  return {1 + (long long)l.qx * (1 + l.qy), (long long)l.qx * l.qy, l.qx};
}
// one thread per element: tiles of 32 x 8 of a plane, whose threads share their neighbours, or, where three sevenths of
// such tiles' threads would lie outside the box, the plane's elements one after another (a block of 256 x 1).  General
// filter, radius 6: 128^3 elements 3.0 ms in tiles, 3.3 in line; 1500 x 6 x 6 0.155 and 0.203; 33 x 40 x 41 0.279 and
// 0.261; 8 x 8 x 512 0.277 and 0.230; 4 x 16 x 512 0.416 and 0.229.  A launch has at most 65535 planes: the kernels
// step on.
static dim3 elem_block(const Level& l) {
  const long long tiles = (long long)cdiv(l.ex, 32) * cdiv(l.ey, 8) * 256;
  return 4 * tiles <= 7LL * l.ex * l.ey ? dim3(32, 8) : dim3(256, 1);
}
static dim3 elem_grid(const Level& l) {
  if (elem_block(l).y > 1) return dim3(cdiv(l.ex, 32), cdiv(l.ey, 8), std::min(l.ez, 65535));
  return dim3(cdiv((long long)l.ex * l.ey, 256), 1, std::min(l.ez, 65535));
}
// the thread's element of a plane; false outside the box
__device__ __forceinline__ bool elem_of(const Level& L, int& x, int& y) {
  unsigned i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (blockDim.y == 1) {  // in line
    j = i / (unsigned)L.ex;
    i -= j * (unsigned)L.ex;
  }
  x = (int)i, y = (int)j;
  return i < (unsigned)L.ex && j < (unsigned)L.ey;
}
// one thread per column of zc elements: long where the tiles of a plane alone
// give the GPU eight CTAs per SM, 4 at least (a plane is shared by two elements)
static dim3 column_grid(const Level& l, int zc) { return dim3(cdiv(l.ex, 32), cdiv(l.ey, 8), cdiv(l.ez, zc)); }
static int column_chunk(const Level& l) {
  int zc = 32;
  while (zc > 4 && (long long)cdiv(l.ex, 32) * cdiv(l.ey, 8) * cdiv(l.ez, zc) < 8 * 148) zc /= 2;
  return std::max(zc, cdiv(l.ez, 65535));
}
// FP64 powers by small whole exponents are products, as accurate as pow and a
// tenth of its instructions
__device__ __forceinline__ double power(double r, double p) {
  if (p == 1.0) return r;
  if (p == 2.0) return r * r;
  if (p == 3.0) return r * r * r;
  return pow(r, p);
}

// ---------------------------------------------------------------- sensitivity
// s_e = -p rho^(p-1) u_e^T K0 u_e (energy=0) or rho^p u_e^T K0 u_e (energy=1).
// In the sum/difference basis of the element's nodes, w = W u_e along each axis,
// K0 = W^T B W with the block structure of fine_op.cu, so the quadratic form is
// a sum over the eight blocks: about 120 operations where the 24 x 24 product
// takes 600.  256^3: 1887 us with the product (bound by the FP64 units), 382 with a
// thread marching along z, which transforms a node plane once for the elements on
// both sides but has too few loads in flight, 302 with a thread per element; 64^3
// 10.7 and 8.5.
// B.c in the order of cWp: A0 - B0, B0, A7 - B7, B7, P, Q, R, S.
struct WalshB { double c[8]; };
__global__ void __launch_bounds__(256) k_sensitivity(const Level L, const double* __restrict__ u,
                                                     const float* __restrict__ rho, const WalshB B, double p, int energy,
                                                     float* __restrict__ out, const View V) {
  int x, y;
  if (!elem_of(L, x, y)) return;
  for (int z = blockIdx.z; z < L.ez; z += gridDim.z) {
    const long long e = L.eidx(x, y, z), o = V.at(x, y, z);
    if (!L.emask[e]) { out[o] = 0.f; continue; }
    double w[8][3];  // modes (mx, my, mz) as bits, component
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double f[2][4];  // xy modes of the lower and upper face
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const double* q = u + L.nidx(x, y, z + b) + c * L.NP;
        const double a00 = q[0], a10 = q[1], a01 = q[L.px], a11 = q[L.px + 1];
        const double s0 = a00 + a10, d0 = a10 - a00, s1 = a01 + a11, d1 = a11 - a01;
        f[b][0] = s0 + s1; f[b][1] = d0 + d1; f[b][2] = s1 - s0; f[b][3] = d1 - d0;
      }
#pragma unroll
      for (int m = 0; m < 4; m++) { w[m][c] = f[0][m] + f[1][m]; w[m + 4][c] = f[1][m] - f[0][m]; }
    }
    auto full = [&](double i, double j, double k, double ab, double bb) {
      const double t = i + j + k;
      return ab * (i * i + j * j + k * k) + bb * (t * t);
    };
    auto pair = [&](double i, double j) { return B.c[4] * (i * i + j * j) + 2.0 * B.c[5] * (i * j); };
    auto both = [&](double i, double j, double k) { return B.c[6] * ((i + j) * (i + j)) + B.c[7] * (k * k); };
    double q = full(w[1][0], w[2][1], w[4][2], B.c[0], B.c[1]) + full(w[6][0], w[5][1], w[3][2], B.c[2], B.c[3]);
    q += pair(w[3][1], w[5][2]) + pair(w[3][0], w[6][2]) + pair(w[5][0], w[6][1]);
    q += both(w[2][0], w[1][1], w[7][2]) + both(w[4][0], w[1][2], w[7][1]) + both(w[4][1], w[2][2], w[7][0]);
    const double r = (double)rho[e];
    out[o] = energy ? (float)(power(r, p) * q) : (float)(-p * (p == 1.0 ? 1.0 : power(r, p - 1)) * q);
  }
}

rso_status sensitivity(rso_handle* h, const double* u_pad, float* sens, int energy, bool dense) {
  const Level& l = h->L[0];
  WalshB B;
  walsh_constants(h->K0, B.c);
  k_sensitivity<<<elem_grid(l), elem_block(l), 0, h->stream>>>(l, u_pad, h->rho, B, h->cfg.penal, energy, sens,
                                                               view_of(l, dense)); rso::note_launch();
  return launch_check(h, "sensitivity");
}

// ---------------------------------------------------------------- Heaviside
// in, gin and out share one layout and may be the same array; t0 = tanh(beta
// eta), den = t0 + tanh(beta (1 - eta)), the same for every element.  One
// exponential serves both maps: with E = exp(-2 |x|), tanh x = sign(x) (1 - E) /
// (1 + E) and its slope is 4 E / (1 + E)^2, without the cancellation of
// 1 - tanh^2 in the tails.  1 - E cancels towards x = 0, an error of 2e-16 in
// values of the size of beta / 2: below |beta| = 1e-3 (kStepSmall; 2e-13 there, an
// FP32 result's last bit is 6e-8) the step takes tanh, and divides by den, whose
// reciprocal may overflow.  (256^3: 122 us with tanh and a thread per
// element, bound by instructions and by each thread's two dependent loads, 70 so,
// a thread loading four elements of its column at once.)
// scale: 1 / den, for the chain beta / den; SMALL: den
constexpr double kStepSmall = 1e-3;
template <bool CHAIN, bool SMALL = false>
__global__ void __launch_bounds__(256) k_heaviside(const Level L, const float* in, double beta, double t0, double scale,
                                                   double rmin, const uint8_t* shell, const float* gin, float* out,
                                                   const View V, int zc) {
  const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
  if (x >= L.ex || y >= L.ey) return;
  const int z0 = blockIdx.z * zc, n = min(zc, L.ez - z0);
  const long long o0 = V.at(x, y, z0), qxy = (long long)L.qx * L.qy;
  const uint8_t* mask = L.emask + L.eidx(x, y, z0);
  const uint8_t* sh = shell ? shell + x + (long long)L.ex * (y + (long long)L.ey * z0) : nullptr;
  for (int z = 0; z < n; z += 4) {  // four elements' loads before any store (the arrays may be one)
    float a[4], g[4];
    bool on[4], one[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const bool ok = z + j < n;
      on[j] = ok && mask[(z + j) * qxy];
      a[j] = ok ? in[o0 + (z + j) * V.sz] : 0.f;
      if (CHAIN) g[j] = ok ? gin[o0 + (z + j) * V.sz] : 0.f;
      one[j] = !CHAIN && ok && sh && sh[(long long)(z + j) * L.ex * L.ey];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (z + j >= n) break;
      const double s = beta * ((double)a[j] - 0.5);
      double v;
      if constexpr (SMALL) {
        v = (t0 + tanh(s)) / scale;
      } else {
        const double E = exp(-2 * fabs(s)), q = __drcp_rn(1 + E);
        v = CHAIN ? (double)g[j] * (4 * E * q * q) * scale : (t0 + copysign((1 - E) * q, s)) * scale;
      }
      if (!CHAIN) {
        v = one[j] ? 1.0 : fmin(fmax(v, rmin), 1.0);
      }
      out[o0 + (z + j) * V.sz] = on[j] ? (float)v : 0.f;
    }
  }
}

rso_status heaviside(rso_handle* h, const float* in, double beta, const uint8_t* shell, float* out, bool dense) {
  const Level& l = h->L[0];
  const double t0 = std::tanh(beta * 0.5), den = t0 + std::tanh(beta * (1 - 0.5));
  const int zc = column_chunk(l);
  const bool small = std::fabs(beta) < kStepSmall;
  auto k = small ? k_heaviside<false, true> : k_heaviside<false>;
  k<<<column_grid(l, zc), dim3(32, 8), 0, h->stream>>>(l, in, beta, t0, small ? den : 1 / den, h->cfg.rho_min, shell,
                                                       nullptr, out, view_of(l, dense), zc); rso::note_launch();
  return launch_check(h, "heaviside");
}

rso_status heaviside_chain(rso_handle* h, const float* rho, double beta, const float* gin, float* gout, bool dense) {
  const Level& l = h->L[0];
  const double t0 = std::tanh(beta * 0.5), den = t0 + std::tanh(beta * (1 - 0.5));
  const int zc = column_chunk(l);
  k_heaviside<true><<<column_grid(l, zc), dim3(32, 8), 0, h->stream>>>(l, rho, beta, t0, beta / den, 0.0, nullptr, gin,
                                                                       gout, view_of(l, dense), zc); rso::note_launch();
  return launch_check(h, "heaviside_chain");
}

// ---------------------------------------------------------------- filter
// weights w(r) = 1 - 6r^2 + 8r^3 - 3r^4, r = |d|/R, |d|^2 <= R^2, reach int(R+0.5)
struct FOff { int dx, dy, dz; double w; };

// any radius: one thread per element over the tap table.  PADDED: in has the handle's
// layout, so that a tap's value and mask share one address; a dense input is copied
// there first from radius 5 on (515 taps: 128^3 elements, radius 8, 8.3 -> 6.7 ms a
// call with a second address a tap gone), not below 1 (one tap).
template <bool PADDED>
__global__ void k_filter(const Level L, const FOff* __restrict__ off, int noff, const float* __restrict__ in,
                         float* __restrict__ out, int mode, const float* __restrict__ wsum, const View V) {
  // mode 0: out = sum w in / sum w;  1: out = sum w (weight sums, padded);  2: out = sum w in/W_n (adjoint)
  int x, y;
  if (!elem_of(L, x, y)) return;
  for (int z = blockIdx.z; z < L.ez; z += gridDim.z) {
    const long long e = L.eidx(x, y, z), o = mode == 1 ? e : V.at(x, y, z);
    if (!L.emask[e]) { out[o] = 0.f; continue; }
    double gs = 0, ws = 0;
    for (int k = 0; k < noff; k++) {
      const int xx = x + off[k].dx, yy = y + off[k].dy, zz = z + off[k].dz;
      if (xx < 0 || yy < 0 || zz < 0 || xx >= L.ex || yy >= L.ey || zz >= L.ez) continue;
      const long long n = L.eidx(xx, yy, zz);
      if (!L.emask[n]) continue;
      const double w = off[k].w;
      ws += w;
      if (mode == 1) continue;
      const double v = (double)in[PADDED ? n : V.at(xx, yy, zz)];
      gs += mode == 0 ? w * v : w * v / (double)wsum[n];
    }
    out[o] = (float)(mode == 0 ? gs / ws : (mode == 1 ? ws : gs));
  }
}

// Radii from 1 to under 5.  A CTA of 32 x 8 threads marches along z through a
// tile of columns.  Each plane, with its halo of RZ elements, is staged once in
// shared memory as FP64 (so a value is converted once, not once per tap).  The
// weight depends on the three distances alone, so the neighbour columns at the
// same two in-plane distances (either way round) form a class: a thread adds up
// the four or eight columns of a class, and multiplies the sum once for each
// plane it reaches, into the 2 RZ + 1 outputs along z that it keeps in
// registers: 13 shared loads, 13 additions and 20 multiply-adds for the 33 taps
// of R = 2, the weights being kernel parameters.  A class or plane outside the
// radius is skipped, not multiplied by zero.  Where a staged plane is full
// (inside the box and all active) its part of the weight sum is known; else the
// mask is summed as the values are.  256^3, R = 2: 1007 us with a thread walking
// a tap table (loads and conversions), 464 with the columns' weights read from
// shared memory, 241 with the next plane's loads in flight during a plane's taps
// and 16 rows a CTA, 209 now: with 8 rows an SM has four barriers to wait at in
// turn instead of two, which is worth the wider halo, and a class is summed two
// by two instead of in a chain.
constexpr int FTX = 32, FTY = 8, kFiltRZ = 4;
constexpr int fclass(int a, int b) { return a >= b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a; }
constexpr int kFClasses = fclass(kFiltRZ, kFiltRZ) + 1;
struct FPlan {
  double w[kFClasses][kFiltRZ + 1];  // weight by class and |dz|
  double plane[kFiltRZ + 1];         // sum of a full plane's weights at |dz|
  int reach[kFClasses];              // the largest |dz| inside the radius, -1 if none is
};
// a staged plane's columns around p, class by class, into the outputs they reach
template <int RZ, typename T>
__device__ __forceinline__ void filter_taps(const FPlan& P, const T* p, double (&to)[2 * RZ + 1]) {
  constexpr int WX = FTX + 2 * RZ;
#pragma unroll
  for (int a = 0; a <= RZ; a++)
#pragma unroll
    for (int b = 0; b <= a; b++) {
      const int reach = P.reach[fclass(a, b)];
      if (reach < 0) continue;
      // the class's columns, two by two (FP32 for the mask: small whole numbers)
      T v[8];
      int n = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int sx = q & 1 ? 1 : -1, sy = q & 2 ? 1 : -1;
        if ((a == 0 && sx > 0) || (b == 0 && sy > 0)) continue;
        v[n++] = p[sy * b * WX + sx * a];
        if (a != b) v[n++] = p[sx * a * WX + sy * b];
      }
#pragma unroll
      for (int m = 1; m < 8; m *= 2)
#pragma unroll
        for (int i = 0; i + m < 8; i += 2 * m)
          if (i + m < n) v[i] += v[i + m];
      const T t = v[0];
      const double s = (double)t;
#pragma unroll
      for (int j = 0; j <= RZ; j++)
        if (j <= reach) {
          const double w = P.w[fclass(a, b)][j];
          to[RZ + j] = fma(w, s, to[RZ + j]);
          if (j > 0) to[RZ - j] = fma(w, s, to[RZ - j]);
        }
    }
}
template <int RZ, int MODE>
__global__ void __launch_bounds__(FTX* FTY) k_filter_tile(const Level L, const __grid_constant__ FPlan P,
                                                          const float* __restrict__ in, float* __restrict__ out,
                                                          const float* __restrict__ wsum, const View V, int zc) {
  constexpr int WX = FTX + 2 * RZ, WY = FTY + 2 * RZ, NW = WX * WY, NA = 2 * RZ + 1;
  __shared__ double sv[2][NW];  // values, zero where masked
  __shared__ float sm[2][NW];   // mask
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * FTX + tx;
  const int x0 = blockIdx.x * FTX, y0 = blockIdx.y * FTY, z0 = blockIdx.z * zc, z1 = min(z0 + zc, L.ez);
  const int x = x0 + tx, y = y0 + ty, c0 = (ty + RZ) * WX + tx + RZ;
  double acc[NA], wac[NA];
#pragma unroll
  for (int k = 0; k < NA; k++) acc[k] = wac[k] = 0;
  // this thread's window entries: their offsets in a plane of the fields, -1 outside the box
  constexpr int NK = (NW + FTX * FTY - 1) / (FTX * FTY);
  const long long qxy = (long long)L.qx * L.qy;
  long long eo[NK], vo[NK];
#pragma unroll
  for (int i = 0; i < NK; i++) {
    const int k = i * FTX * FTY + tid, wy = k / WX, wx = k - wy * WX, xx = x0 + wx - RZ, yy = y0 + wy - RZ;
    eo[i] = vo[i] = -1;
    if (k < NW && xx >= 0 && yy >= 0 && xx < L.ex && yy < L.ey) {
      eo[i] = L.eidx(xx, yy, 0);
      vo[i] = V.at(xx, yy, 0);
    }
  }
  float raw[NK], wgt[NK];
  bool on[NK];
  auto fetch = [&](int zp) {  // plane zp into registers
    const bool in_z = zp >= 0 && zp < L.ez;
#pragma unroll
    for (int i = 0; i < NK; i++) {
      const bool ok = in_z && eo[i] >= 0;
      on[i] = ok && L.emask[eo[i] + qxy * zp];
      raw[i] = MODE != 1 && ok ? in[vo[i] + V.sz * zp] : 0.f;
      wgt[i] = MODE == 2 && ok ? wsum[eo[i] + qxy * zp] : 1.f;
    }
  };
  fetch(z0 - RZ);
  // planes z0 - RZ .. z1 - 1 + RZ; after plane zp output zp - RZ is complete
  for (int zp = z0 - RZ; zp < z1 + RZ; zp++) {
    const int buf = (zp - z0 + RZ) & 1;
    bool full = true;
#pragma unroll
    for (int i = 0; i < NK; i++) {
      const int k = i * FTX * FTY + tid;
      if (k >= NW) break;
      double a = (double)raw[i];
      if (MODE == 2) a /= (double)wgt[i];
      sv[buf][k] = on[i] ? a : 0.0;
      sm[buf][k] = on[i] ? 1.f : 0.f;
      full = full && on[i];
    }
    full = __syncthreads_and(full) != 0;
    if (zp + 1 < z1 + RZ) fetch(zp + 1);  // in flight while this plane's taps are added
    if (MODE != 1) filter_taps<RZ>(P, sv[buf] + c0, acc);
    if (MODE != 2) {
      if (full) {
        wac[RZ] += P.plane[0];
#pragma unroll
        for (int j = 1; j <= RZ; j++) { wac[RZ + j] += P.plane[j]; wac[RZ - j] += P.plane[j]; }
      } else {
        filter_taps<RZ>(P, sm[buf] + c0, wac);
      }
    }
    // acc[k] belongs to output zp + k - RZ: acc[0] is complete
    const int z = zp - RZ;
    if (z >= z0 && x < L.ex && y < L.ey) {
      const long long e = L.eidx(x, y, z);
      const float r = (float)(MODE == 0 ? acc[0] / wac[0] : (MODE == 1 ? wac[0] : acc[0]));
      out[MODE == 1 ? e : V.at(x, y, z)] = L.emask[e] ? r : 0.f;
    }
#pragma unroll
    for (int k = 0; k + 1 < NA; k++) { acc[k] = acc[k + 1]; wac[k] = wac[k + 1]; }
    acc[NA - 1] = wac[NA - 1] = 0;
  }
}

static FPlan filter_plan(double R, int RZ) {
  FPlan P = {};
  const double R2 = R * R;
  for (int a = 0; a <= kFiltRZ; a++)
    for (int b = 0; b <= a; b++) {
      const int c = fclass(a, b), h2 = a * a + b * b;
      P.reach[c] = -1;
      for (int d = 0; d <= RZ && a <= RZ && h2 + d * d <= R2; d++) {
        const double r = std::sqrt((h2 + d * d) / R2), rr = r * r;
        P.reach[c] = d;
        P.w[c][d] = 1 - 6 * rr + 8 * rr * r - 3 * rr * rr;
        P.plane[d] += P.w[c][d] * ((a > 0 ? 2 : 1) * (b > 0 ? 2 : 1) * (a != b ? 2 : 1));
      }
    }
  return P;
}

template <int RZ>
static rso_status filter_tiles(rso_handle* h, double R, const float* in, float* out, int adjoint, const View& V) {
  const Level& l = h->L[0];
  const FPlan P = filter_plan(R, RZ);
  // planes per chunk: each chunk stages 2 RZ planes more than it writes, so
  // chunks are as long as the grid still has two CTAs per SM with them
  int zc = 32;
  while (zc > 8 && (long long)cdiv(l.ex, FTX) * cdiv(l.ey, FTY) * cdiv(l.ez, zc) < 2 * 148) zc /= 2;
  const dim3 g(cdiv(l.ex, FTX), cdiv(l.ey, FTY), cdiv(l.ez, zc)), b(FTX, FTY);
  if (!adjoint) {
    k_filter_tile<RZ, 0><<<g, b, 0, h->stream>>>(l, P, in, out, nullptr, V, zc); rso::note_launch();
  } else {
    float* W = h->e_d;
    k_filter_tile<RZ, 1><<<g, b, 0, h->stream>>>(l, P, nullptr, W, nullptr, V, zc); rso::note_launch();
    k_filter_tile<RZ, 2><<<g, b, 0, h->stream>>>(l, P, in, out, W, V, zc); rso::note_launch();
  }
  return launch_check(h, "filter");
}

rso_status filter(rso_handle* h, double R, const float* in, float* out, int adjoint, bool dense) {
  const Level& l = h->L[0];
  const View V = view_of(l, dense);
  if (R >= 1 && R < 2) return filter_tiles<1>(h, R, in, out, adjoint, V);
  if (R >= 2 && R < 3) return filter_tiles<2>(h, R, in, out, adjoint, V);
  if (R >= 3 && R < 4) return filter_tiles<3>(h, R, in, out, adjoint, V);
  if (R >= 4 && R < 5) return filter_tiles<4>(h, R, in, out, adjoint, V);
  std::vector<FOff> off;
  const int Ri = (int)(R + 0.5);
  const double R2 = R * R;
  for (int dx = -Ri; dx <= Ri; dx++)
    for (int dy = -Ri; dy <= Ri; dy++)
      for (int dz = -Ri; dz <= Ri; dz++) {
        const double r2 = dx * dx + dy * dy + dz * dz;
        if (r2 > R2) continue;
        const double r = std::sqrt(r2 / R2), rr = r * r;
        off.push_back({dx, dy, dz, 1 - 6 * rr + 8 * rr * r - 3 * rr * rr});
      }
  // the tap table is kept on the handle and rebuilt only when the radius changes
  if (!h->filt_taps || h->filt_radius != R) {
    h->filt_radius = -1.0;
    if ((long long)off.size() > h->filt_cap) {
      if (h->filt_taps) RSO_CHECK_CUDA(h, cudaFree(h->filt_taps));
      h->filt_taps = nullptr;
      h->filt_cap = 0;
      RSO_CHECK_CUDA(h, cudaMalloc(&h->filt_taps, sizeof(FOff) * off.size()));
      h->filt_cap = (long long)off.size();
    }
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(h->filt_taps, off.data(), sizeof(FOff) * off.size(), cudaMemcpyHostToDevice,
                                      h->stream));
    // the host table is a local vector: finish the copy before it goes away
    RSO_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
    h->filt_radius = R;
  }
  const FOff* d_off = static_cast<const FOff*>(h->filt_taps);
  const int n = (int)off.size();
  if (dense && n > 1) {
    RSO_TRY(pad_elems_f(h, in, h->e_b));
    in = h->e_b;
  }
  auto k = dense && n == 1 ? k_filter<false> : k_filter<true>;
  if (!adjoint) {
    k<<<elem_grid(l), elem_block(l), 0, h->stream>>>(l, d_off, n, in, out, 0, nullptr, V); rso::note_launch();
  } else {
    float* W = h->e_d;
    k<<<elem_grid(l), elem_block(l), 0, h->stream>>>(l, d_off, n, in, W, 1, nullptr, V); rso::note_launch();
    k<<<elem_grid(l), elem_block(l), 0, h->stream>>>(l, d_off, n, in, out, 2, W, V); rso::note_launch();
  }
  return launch_check(h, "filter");
}

// ---------------------------------------------------------------- volume
// Sum of the active elements: a warp per row, or per len elements of it (blockIdx.y).
// Bound by the loads in flight, so 256 elements' are written out: 23 us at 256^3, 29
// with the loop left to the compiler.
constexpr int kSumBlocks = 592;
__device__ __forceinline__ double warp_add(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__global__ void __launch_bounds__(256) k_sum_elems(const Level L, const float* __restrict__ a, const View V,
                                                   int len, double* __restrict__ part) {
  __shared__ double ws[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0;
  const int xa = blockIdx.y * len, xb = min(xa + len, L.ex);
  for (int r = blockIdx.x * 8 + warp; r < L.ey * L.ez; r += gridDim.x * 8) {
    const int z = r / L.ey, y = r - z * L.ey;
    const uint8_t* m = L.emask + L.eidx(0, y, z);
    const float* q = a + V.at(0, y, z);
    int x = xa + lane;
    for (; x + 224 < xb; x += 256) {
      float v[8];
      uint8_t k[8];
#pragma unroll
      for (int j = 0; j < 8; j++) { v[j] = q[x + 32 * j]; k[j] = m[x + 32 * j]; }
#pragma unroll
      for (int j = 0; j < 8; j++) s += k[j] ? (double)v[j] : 0.0;
    }
    for (; x < xb; x += 32) {
      const float v = q[x];
      s += m[x] ? (double)v : 0.0;
    }
  }
  s = warp_add(s);
  if (lane == 0) ws[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < 8; k++) t += ws[k];
    part[blockIdx.y * gridDim.x + blockIdx.x] = t;
  }
}
rso_status sum_elems(rso_handle* h, const float* a, bool dense, double* dev_out) {
  const Level& l = h->L[0];
  // rows past 256 elements are cut, at most kSumBlocks times: one warp's chain a row
  // took 6 % of an OC coefficient update on 1500 x 6 x 6
  const int len = 256 * cdiv(l.ex, 256 * kSumBlocks), cuts = cdiv(l.ex, len);
  const dim3 grid(std::min(std::max(1, kSumBlocks / cuts), cdiv((long long)l.ey * l.ez, 8)), cuts);
  k_sum_elems<<<grid, 256, 0, h->stream>>>(l, a, view_of(l, dense), len, h->red); rso::note_launch();
  RSO_TRY(launch_check(h, "sum_elems"));
  return reduce_partials(h, h->red, grid.x * grid.y, dev_out);
}

rso_status volume(rso_handle* h, const float* rho, double* vol, bool dense) {
  RSO_TRY(sum_elems(h, rho, dense, h->scal + 14));
  RSO_CHECK_CUDA(h, cudaMemcpyAsync(h->h_scal + 14, h->scal + 14, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  RSO_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  // Grid::volumeRatio divides by the GS-padded element count (grid/Grid.cu:5642-5650)
  *vol = h->h_scal[14] / (double)h->n_gs_elements;
  return RSO_OK;
}

// ---------------------------------------------------------------- spline set-up
// first-knot index i = (int)((pos - bmin)/step) + order in float (the
// reference's span computation, grid/Grid.cu:3477-3479) and Cox-de Boor
// values / first derivatives in double (Piegl-Tiller A2.2/A2.3, the
// recursion of SplineBasisX/SplineBasisDeriX grid/Grid.cu:427-857).
__global__ void k_spline_axis(int n, int order, int nb, float bmin, float step, const float* __restrict__ knots,
                              int* __restrict__ idx, double* __restrict__ N, double* __restrict__ dN) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  const float pos = (float)((double)((float)x * 1.0f) + 0.5);
  const int i = (int)__fdiv_rn(__fsub_rn(pos, bmin), step) + order;
  const bool inside = !(i < order || i > nb);
  idx[x] = inside ? i : -1;
  for (int j = 0; j < order; j++) { N[x * order + j] = 0; dN[x * order + j] = 0; }
  if (!inside) return;
  const int span = i - 1, p = order - 1;
  double ndu[6][6], left[6], right[6];
  ndu[0][0] = 1.0;
  const double u = (double)pos;
  for (int j = 1; j <= p; j++) {
    left[j] = u - (double)knots[span + 1 - j];
    right[j] = (double)knots[span + j] - u;
    double saved = 0.0;
    for (int r = 0; r < j; r++) {
      ndu[j][r] = right[r + 1] + left[j - r];
      const double temp = ndu[r][j - 1] / ndu[j][r];
      ndu[r][j] = saved + right[r + 1] * temp;
      saved = left[j - r] * temp;
    }
    ndu[j][j] = saved;
  }
  for (int j = 0; j <= p; j++) N[x * order + j] = ndu[j][p];
  for (int r = 0; r <= p; r++) {
    double d = 0;
    if (p >= 1) {
      if (r >= 1) d = ndu[r - 1][p - 1] / ndu[p][r - 1];
      if (r <= p - 1) d -= ndu[r][p - 1] / ndu[p][r];
      d *= p;
    }
    dN[x * order + r] = d;
  }
}

// de Boor value at an arbitrary coordinate (used by the orientation probe)
__device__ bool axis_basis(double u, int order, int nb, float bmin, float step, const float* knots, int* I,
                           double* N) {
  const float pf = (float)u;
  if (!knot_index(__fdiv_rn(__fsub_rn(pf, bmin), step), order, nb, I)) return false;
  const int span = *I - 1, p = order - 1;
  double left[6], right[6];
  N[0] = 1.0;
  for (int j = 1; j <= p; j++) {
    left[j] = u - (double)knots[span + 1 - j];
    right[j] = (double)knots[span + j] - u;
    double saved = 0;
    for (int r = 0; r < j; r++) {
      const double temp = N[r] / (right[r + 1] + left[j - r]);
      N[r] = saved + right[r + 1] * temp;
      saved = left[j - r] * temp;
    }
    N[j] = saved;
  }
  return true;
}

struct SplineDev {
  int order, nb0, nb1, nb2;
  float bmin0, bmin1, bmin2, step0, step1, step2;
  const float *k0, *k1, *k2;
  const int *i0, *i1, *i2;
  const double *N0, *N1, *N2, *D0, *D1, *D2;
  // x tables by function: tN, tD[q * ex + x] as N0, D0[x * order + q]; and the
  // values over each function's support, bN, bD[k * nb0 + a] at x = lo[a] + k
  const double *tN, *tD, *bN, *bD;
};

static SplineDev spline_dev(rso_handle* h, const float* knots_dev) {
  const Spline& s = h->sp;
  SplineDev d;
  d.order = s.order; d.nb0 = s.nb[0]; d.nb1 = s.nb[1]; d.nb2 = s.nb[2];
  d.bmin0 = s.bmin[0]; d.bmin1 = s.bmin[1]; d.bmin2 = s.bmin[2];
  d.step0 = s.step[0]; d.step1 = s.step[1]; d.step2 = s.step[2];
  d.k0 = knots_dev; d.k1 = knots_dev + s.knots[0].size(); d.k2 = d.k1 + s.knots[1].size();
  d.i0 = s.idx[0]; d.i1 = s.idx[1]; d.i2 = s.idx[2];
  d.N0 = s.N[0]; d.N1 = s.N[1]; d.N2 = s.N[2];
  d.D0 = s.dN[0]; d.D1 = s.dN[1]; d.D2 = s.dN[2];
  const long long no = (long long)s.order * h->L[0].ex, nb = (long long)s.nb[0] * s.sup;
  d.tN = s.xtab; d.tD = d.tN + no; d.bN = d.tD + no; d.bD = d.bN + nb;
  return d;
}

// ---------------------------------------------------------------- spline rows
// The tensor-product spline at the element centres is contracted one axis at a
// time: first z, R1[z][j][i] = sum_k c[k][j][i] B_k(z), then y,
// R2[z][y][i] = sum_j R1[z][j][i] B_j(y), a row of nb0 values per row of
// elements; an element then sums `order` of them along x, instead of order^3
// coefficients (the rows are nb0 / ex of the elements: 1/8 for 32 coefficients
// on 256).  D as well as N along z or y gives the rows of the derivatives.
// Rows outside the knots are zero.
template <typename C>
__global__ void __launch_bounds__(256) k_rows_z(SplineDev S, int ez, const C* __restrict__ c,
                                                double* __restrict__ rn, double* __restrict__ rd) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long pl = (long long)S.nb0 * S.nb1;
  if (t >= pl * ez) return;
  const int z = (int)(t / pl);
  const long long ij = t - pl * z;
  const int k0 = S.i2[z] - S.order;
  double n = 0, d = 0;
  if (k0 >= 0)
    for (int q = 0; q < S.order; q++) {
      const double v = (double)c[ij + (k0 + q) * pl];
      n += v * S.N2[z * S.order + q];
      if (rd) d += v * S.D2[z * S.order + q];
    }
  rn[t] = n;
  if (rd) rd[t] = d;
}
// rows NN from rn; with rd also DN (D along y) and ND (D along z), `comp` apart
__global__ void __launch_bounds__(256) k_rows_y(SplineDev S, int ey, int ez, const double* __restrict__ rn,
                                                const double* __restrict__ rd, double* __restrict__ out,
                                                long long comp) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= comp) return;
  const long long yz = t / S.nb0;
  const int i = (int)(t - yz * S.nb0), z = (int)(yz / ey), y = (int)(yz - (long long)z * ey);
  const int j0 = S.i1[y] - S.order;
  double nn = 0, dn = 0, nd = 0;
  if (j0 >= 0) {
    const long long base = i + (long long)S.nb0 * (j0 + (long long)S.nb1 * z);
    for (int q = 0; q < S.order; q++) {
      const double v = rn[base + (long long)q * S.nb0], N = S.N1[y * S.order + q];
      nn += v * N;
      if (rd) {
        dn += v * S.D1[y * S.order + q];
        nd += rd[base + (long long)q * S.nb0] * N;
      }
    }
  }
  out[t] = nn;
  if (rd) { out[t + comp] = dn; out[t + 2 * comp] = nd; }
}

// coefficients in double or float (whose conversion is exact: no pass of its own)
template <typename C>
static rso_status spline_rows(rso_handle* h, const SplineDev& S, const C* c, double* R, bool derivatives) {
  const Level& l = h->L[0];
  const long long nz = (long long)S.nb0 * S.nb1 * l.ez, comp = (long long)S.nb0 * l.ey * l.ez;
  double* rn = h->sp.work[1];
  double* rd = derivatives ? rn + nz : nullptr;
  k_rows_z<C><<<cdiv(nz, 256), 256, 0, h->stream>>>(S, l.ez, c, rn, rd); rso::note_launch();
  k_rows_y<<<cdiv(comp, 256), 256, 0, h->stream>>>(S, l.ey, l.ez, rn, rd, R, comp); rso::note_launch();
  return launch_check(h, "spline rows");
}

// ---------------------------------------------------------------- spline forward
// a thread keeps its x's basis values and walks along z (134 us at 256^3 with one
// element per thread, which loaded them each time: bound by those loads; 63 now)
template <int O>
__global__ void __launch_bounds__(256) k_coeff2density(const Level L, SplineDev S, const double* __restrict__ R,
                                                       double rmin, const uint8_t* __restrict__ shell,
                                                       float* __restrict__ out, const View V, int zc) {
  const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
  if (x >= L.ex || y >= L.ey) return;
  const int i = S.i0[x];
  const bool in_xy = i >= 0 && S.i1[y] >= 0;
  double N[O];
#pragma unroll
  for (int q = 0; q < O; q++) N[q] = S.tN[(long long)q * L.ex + x];
  const int z0 = blockIdx.z * zc, z1 = min(z0 + zc, L.ez);
  const long long rs = (long long)S.nb0 * L.ey, qxy = (long long)L.qx * L.qy;
  const double* row = R + (long long)S.nb0 * (y + (long long)L.ey * z0) + (in_xy ? i - O : 0);
  const uint8_t* mask = L.emask + L.eidx(x, y, z0);
  const uint8_t* sh = shell ? shell + x + (long long)L.ex * (y + (long long)L.ey * z0) : nullptr;
  out += V.at(x, y, z0);
#pragma unroll 4
  for (int z = 0; z < z1 - z0; z++) {
    double v = 0;
#pragma unroll
    for (int q = 0; q < O; q++) v += row[z * rs + q] * N[q];  // outside the knots: any row, not used
    if (!in_xy || S.i2[z0 + z] < 0) v = -0.2;
    v = fmin(fmax(v, rmin), 1.0);
    if (sh && sh[(long long)z * L.ex * L.ey]) v = 1.0;
    out[z * V.sz] = mask[z * qxy] ? (float)v : 0.f;
  }
}

template <typename C>
rso_status coeff2density(rso_handle* h, const C* c, const uint8_t* shell, float* out, bool dense) {
  const Level& l = h->L[0];
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  const SplineDev S = spline_dev(h, h->sp.knots_dev);
  RSO_TRY(spline_rows(h, S, c, h->sp.work[0], false));
  const int zc = column_chunk(l);
  const dim3 g = column_grid(l, zc), b(32, 8);
  const View V = view_of(l, dense);
  const double* R = h->sp.work[0];
  const double rmin = h->cfg.rho_min;
  if (S.order == 2) k_coeff2density<2><<<g, b, 0, h->stream>>>(l, S, R, rmin, shell, out, V, zc);
  else if (S.order == 3) k_coeff2density<3><<<g, b, 0, h->stream>>>(l, S, R, rmin, shell, out, V, zc);
  else if (S.order == 4) k_coeff2density<4><<<g, b, 0, h->stream>>>(l, S, R, rmin, shell, out, V, zc);
  else k_coeff2density<5><<<g, b, 0, h->stream>>>(l, S, R, rmin, shell, out, V, zc);
  rso::note_launch();
  return launch_check(h, "coeff2density");
}
template rso_status coeff2density<double>(rso_handle*, const double*, const uint8_t*, float*, bool);
template rso_status coeff2density<float>(rso_handle*, const float*, const uint8_t*, float*, bool);

// ---------------------------------------------------------------- separable adjoint
// Stage 1, x: a warp takes two rows of elements, kSeg elements at a time, their
// weights in shared memory, and a lane sums for its basis function over its
// support: G1[z][y][a] (+)= sum_x w(x) B_a(x).  Row reads are coalesced, every
// weight is read from memory once, and the function's values (bN, lanes side by
// side) serve both rows.  256^3, 32 coefficients: 202 us with a thread per
// (a, y, z) reading the fields directly, 205 with one row per warp and the values
// looked up through the span table, 88 now.
// Boxes with few rows cut them in chunks of x (XSplit), a warp each, which write
// sums of their own, `stride` apart; stage 2 adds up those a function's support meets.
constexpr int kSeg = 256, kAdjRows = 2, kAdjWarps = 4;
struct XSplit { int chunks, len; };
// Rows are cut where whole ones make fewer than four warps an SM, into pieces of 32
// elements at least, until there are eight an SM.  1500 x 6 x 6 elements, 32
// coefficients along x: adjoint 0.146 -> 0.057 ms a call, overhang constraint 0.644
// -> 0.125 (a thread an element or a sum, as before both: 0.100 and 0.317).
static XSplit x_split(const Level& l, int rows_per_warp, int seg) {
  const long long warps = cdiv((long long)l.ey * l.ez, rows_per_warp);
  int len = seg;
  if (warps >= 4 * 148) return {1, l.ex};
  while (len > 32 && warps * cdiv(l.ex, len) < 8 * 148) len /= 2;
  return l.ex <= len ? XSplit{1, l.ex} : XSplit{cdiv(l.ex, len), len};
}
__global__ void __launch_bounds__(32 * kAdjWarps) k_adj_x(const Level L, SplineDev S, const float* __restrict__ g,
                                                          const uint8_t* __restrict__ shell, const View V,
                                                          const int* __restrict__ lo, const int* __restrict__ hi,
                                                          int len, long long stride, double* __restrict__ G1) {
  __shared__ double w[kAdjWarps][kAdjRows][kSeg];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = L.ey * L.ez, r0 = (blockIdx.x * kAdjWarps + warp) * kAdjRows;
  if (r0 >= rows) return;
  const int x0 = blockIdx.y * len, x1 = min(x0 + len, L.ex);
  G1 += blockIdx.y * stride;
  for (int xa = x0; xa < x1; xa += kSeg) {
    const int xb = min(xa + kSeg, x1);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kAdjRows; j++) {
      const int r = r0 + j, z = r / L.ey, y = r - z * L.ey;
      const bool in = r < rows && S.i1[y] >= 0 && S.i2[z] >= 0;
      const uint8_t* m = L.emask + (in ? L.eidx(0, y, z) : 0);
      const float* q = g + (in ? V.at(0, y, z) : 0);
      const uint8_t* sh = shell && in ? shell + (long long)L.ex * r : nullptr;
#pragma unroll 4
      for (int x = xa + lane; x < xb; x += 32) {
        const float v = in ? q[x] : 0.f;
        w[warp][j][x - xa] = in && m[x] && !(sh && sh[x]) ? (double)v : 0.0;
      }
    }
    __syncwarp();
    for (int a = lane; a < S.nb0; a += 32) {
      const int l0 = lo[a], ka = max(l0, xa) - l0, kb = min(hi[a], xb - 1) - l0;
      double s[kAdjRows] = {};
#pragma unroll 4
      for (int k = ka; k <= kb; k++) {
        const double B = S.bN[(long long)k * S.nb0 + a];
#pragma unroll
        for (int j = 0; j < kAdjRows; j++) s[j] = fma(w[warp][j][l0 + k - xa], B, s[j]);
      }
#pragma unroll
      for (int j = 0; j < kAdjRows; j++)
        if (r0 + j < rows) {
          double* G = G1 + (long long)S.nb0 * (r0 + j) + a;
          *G = xa == x0 ? s[j] : *G + s[j];
        }
    }
  }
}
// Stage 2, y: G2[z][b][a] = sum_y G1[z][y][a] N_b(y) (+ Gd[z][y][a] D_b(y)); SPLIT: stage 1 in chunks of len
template <bool SPLIT>
__global__ void __launch_bounds__(256) k_adj_y(SplineDev S, int ey, int ez, const double* __restrict__ G1,
                                               const double* __restrict__ Gd, const int* __restrict__ lo,
                                               const int* __restrict__ hi, const int* __restrict__ xlo,
                                               const int* __restrict__ xhi, int len, long long stride,
                                               double* __restrict__ G2) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long pl = (long long)S.nb0 * S.nb1;
  if (t >= pl * ez) return;
  const int z = (int)(t / pl), ab = (int)(t - pl * z), b = ab / S.nb0, a = ab - b * S.nb0;
  const int c0 = SPLIT ? xlo[a] / len : 0, c1 = SPLIT ? xhi[a] / len : 0;
  auto stage1 = [&](const double* G, long long g) {
    double v = G[g + c0 * stride];
    if (SPLIT)
      for (int c = c0 + 1; c <= c1; c++) v += G[g + c * stride];
    return v;
  };
  double s = 0;
#pragma unroll 4
  for (int y = lo[b]; y <= hi[b]; y++) {
    const long long g = a + (long long)S.nb0 * (y + (long long)ey * z);
    const int k = y * S.order + b - S.i1[y] + S.order;
    s += stage1(G1, g) * S.N1[k];
    if (Gd) s += stage1(Gd, g) * S.D1[k];
  }
  G2[t] = s;
}
static void adj_y(rso_handle* h, const SplineDev& S, const XSplit& X, long long stride, const double* G1,
                  const double* Gd, double* G2) {
  const Level& l = h->L[0];
  const int *r0 = h->sp.ranges[0], *r1 = h->sp.ranges[1];
  auto k = X.chunks > 1 ? k_adj_y<true> : k_adj_y<false>;
  k<<<cdiv((long long)S.nb0 * S.nb1 * l.ez, 256), 256, 0, h->stream>>>(S, l.ey, l.ez, G1, Gd, r1, r1 + S.nb1, r0,
                                                                       r0 + S.nb0, X.len, stride, G2); rso::note_launch();
}
// Stage 3, z: dc[c][b][a] = scale (sum_z G2[z][b][a] N_c(z) (+ Gd[z][b][a] D_c(z))); scale from
// *count (its reciprocal, 0 for 0) when given.  The supports are a fifth of the box or
// more and there are few coefficients, so eight lanes share one and meet by shuffles.
__global__ void __launch_bounds__(256) k_adj_z(SplineDev S, const double* __restrict__ G2,
                                               const double* __restrict__ Gd, const int* __restrict__ lo,
                                               const int* __restrict__ hi, const double* __restrict__ count,
                                               double* __restrict__ dc) {
  const long long pl = (long long)S.nb0 * S.nb1, tot = pl * S.nb2;
  const long long t = blockIdx.x * 32LL + threadIdx.x;  // blockDim (32, 8)
  __shared__ double part[8][32];
  double s = 0;
  if (t < tot) {
    const int c = (int)(t / pl);
    const long long ab = t - pl * c;
    for (int z = lo[c] + threadIdx.y; z <= hi[c]; z += 8) {
      const int k = z * S.order + c - S.i2[z] + S.order;
      s += G2[ab + pl * z] * S.N2[k];
      if (Gd) s += Gd[ab + pl * z] * S.D2[k];
    }
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || t >= tot) return;
  for (int k = 1; k < 8; k++) s += part[k][threadIdx.x];
  const double scale = count ? (*count == 0 ? 0.0 : 1.0 / *count) : 1.0;
  dc[t] = scale * s;
}

rso_status density2coeff(rso_handle* h, const float* g, const uint8_t* shell, double* dc, bool dense) {
  const Level& l = h->L[0];
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  const SplineDev S = spline_dev(h, h->sp.knots_dev);
  double *G1 = h->sp.work[0], *G2 = h->sp.work[1];
  const int *r0 = h->sp.ranges[0], *r2 = h->sp.ranges[2];
  const long long rows = (long long)l.ey * l.ez, t3 = (long long)S.nb0 * S.nb1 * S.nb2, stride = S.nb0 * rows;
  const XSplit X = x_split(l, kAdjRows, kSeg);
  const dim3 grid(cdiv(rows, kAdjRows * kAdjWarps), X.chunks);
  k_adj_x<<<grid, 32 * kAdjWarps, 0, h->stream>>>(l, S, g, shell, view_of(l, dense), r0, r0 + S.nb0, X.len, stride, G1);
  rso::note_launch();
  adj_y(h, S, X, stride, G1, nullptr, G2);
  k_adj_z<<<cdiv(t3, 32), dim3(32, 8), 0, h->stream>>>(S, G2, nullptr, r2, r2 + S.nb2, nullptr, dc); rso::note_launch();
  return launch_check(h, "density2coeff");
}

// ---------------------------------------------------------------- self-support
// Grid.cu:123-190 penalty pieces
__device__ __forceinline__ double d_H(double s, double beta) {
  const double eta = 0.5;
  return (tanh(beta * eta) + tanh(beta * (s - eta))) / (tanh(beta * eta) + tanh(beta * (1 - eta)));
}

struct SSPar {
  int mode;
  double beta, cosang, mid, sc, fpara, na, ia;
};

// Sign of the orientation probe (grid/Grid.cu:7623-7714) by evaluating it: the
// spline 0.01 h along the gradient, through the Heaviside step
__device__ __noinline__ float probe_sign(const SplineDev& S, const double* __restrict__ c, double beta, int x, int y,
                                         int z, bool inside, double v, double g0, double g1, double g2) {
  const int o = S.order;
  const double pt[3] = {x + 0.5 + 0.01 * g0, y + 0.5 + 0.01 * g1, z + 0.5 + 0.01 * g2};
  int Ii[3];
  double Nb[3][6];
  bool ins = axis_basis(pt[0], o, S.nb0, S.bmin0, S.step0, S.k0, &Ii[0], Nb[0]);
  ins = ins && axis_basis(pt[1], o, S.nb1, S.bmin1, S.step1, S.k1, &Ii[1], Nb[1]);
  ins = ins && axis_basis(pt[2], o, S.nb2, S.bmin2, S.step2, S.k2, &Ii[2], Nb[2]);
  double vd = -0.1;
  if (ins) {
    vd = 0;
    for (int q = 0; q < o; q++)
      for (int b = 0; b < o; b++)
        for (int a = 0; a < o; a++)
          vd += c[(Ii[0] - o + a) + (long long)(Ii[1] - o + b) * S.nb0 + (long long)(Ii[2] - o + q) * S.nb0 * S.nb1] *
                Nb[0][a] * Nb[1][b] * Nb[2][q];
  }
  const double vv = inside ? v : -0.1;
  return d_H(vv, beta) - d_H(vd, beta) > 0 ? 1.f : -1.f;
}

// largest |c|; one CTA
__global__ void __launch_bounds__(1024) k_max_abs(long long n, const double* __restrict__ c, double* __restrict__ out) {
  __shared__ double sh[32];
  double m = 0;
#pragma unroll 8
  for (long long i = threadIdx.x; i < n; i += 1024) m = fmax(m, fabs(c[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 32; k++) m = fmax(m, sh[k]);
    *out = m;
  }
}

// The constraint on every element in one pass: value and gradient from the
// spline rows, the probe's sign, the penalty, and stage 1 (x) of the separable
// adjoint of its three weights.  A warp takes a row of elements, kSSSeg at a time.
//
// The probe walks t = 0.01 along the gradient g, so the spline there is at
// least v + t |g|^2 (1 - t H / 2), H a bound on its second derivatives: for
// order >= 3, |d2/dx2| <= 4 p (p - 1) M / s^2 and |d2/dxdy| <= 4 p^2 M / (s s')
// with M the largest coefficient, s the knot spacings and p = order - 1 (hcoef
// holds H / M).  Where that growth times the least slope of the step between the
// two values is far above the rounding of the two tanh, the probe's sign is
// known, -1, without evaluating it (64 coefficients, three basis recursions and
// six tanh: 3.4 of the 3.65 ms this stage took at 256^3; the whole pass takes 0.66); elsewhere probe_sign
// decides, as before.
//
// The penalty needs the sign `flip` that the sum of all probes gives.  It is
// taken as -1 (`direction` likewise), which the sum confirms in every design
// whose density grows along its gradient; the caller runs the pass again when
// it does not, without the probes (PROBE false), which cost most of it there.
struct SSOut { double *G1, *Gy, *Gz; float* per; double* part; };
constexpr int kSSRows = 4, kSSSeg = 128;
static int ss_blocks(const Level& l) { return cdiv((long long)l.ey * l.ez, kSSRows); }
template <int O, bool PROBE>
__global__ void __launch_bounds__(32 * kSSRows, 5) k_ss_rows(const Level L, SplineDev S, const double* __restrict__ c,
                                                             const double* __restrict__ R, long long comp, const SSPar P,
                                                             double flip, double direction,
                                                             const double* __restrict__ cmax, double hcoef, double smin,
                                                             const int* __restrict__ lo, const int* __restrict__ hi,
                                                             int len, SSOut Q, const View V) {
  __shared__ double w[kSSRows][4][kSSSeg];
  __shared__ double red[kSSRows][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = blockIdx.x * kSSRows + warp;
  double sper = 0;
  int ndir = 0, ndown = 0;  // probes with sign +1 less those with -1; downward faces
  if (r < L.ey * L.ez) {
    const int z = r / L.ey, y = r - z * L.ey;
    const long long gb = (long long)S.nb0 * r;
    const bool in_yz = S.i1[y] >= 0 && S.i2[z] >= 0;
    const double tH = 0.01 * hcoef * *cmax, least = 1e-11 * (1 + *cmax);
    const double rcos = 1 / P.cosang, rsc = 1 / P.sc;
    const uint8_t* mask = L.emask + L.eidx(0, y, z);
    const double *r0 = R + gb - O, *r1 = r0 + comp, *r2 = r1 + comp;
    float* per = Q.per ? Q.per + V.at(0, y, z) : nullptr;
    const int x0 = blockIdx.y * len, x1 = min(x0 + len, L.ex);
    Q.G1 += blockIdx.y * 3 * comp, Q.Gy += blockIdx.y * 3 * comp, Q.Gz += blockIdx.y * 3 * comp;
    for (int xa = x0; xa < x1; xa += kSSSeg) {
      const int xb = min(xa + kSSSeg, x1);
      __syncwarp();
      for (int x = xa + lane; x < xb; x += 32) {
        double wA = 0, wX = 0, wY = 0, wZ = 0;
        float val32 = 0.f;
        if (mask[x]) {
          const int I = S.i0[x];
          const bool inside = I >= 0 && in_yz;
          double f = 0, g0 = 0, g1 = 0, g2 = 0;
          if (inside) {
            const double *tn = S.tN + x, *td = S.tD + x;
#pragma unroll
            for (int q = 0; q < O; q++) {
              const double N = tn[q * L.ex], t = r0[I + q];
              f += t * N;
              g0 += t * td[q * L.ex];
              g1 += r1[I + q] * N;
              g2 += r2[I + q] * N;
            }
          }
          const double gg = g0 * g0 + g1 * g1 + g2 * g2;
          bool known = !PROBE;
          if (PROBE && O >= 3 && tH < 1.0 && inside) {
            const double grow = 0.01 * gg * (1 - 0.5 * tH);
            // sech^2(s) >= exp(-2 |s|), s up to beta (|v - 1/2| + what the probe may rise)
            const float slope = __expf((float)(-2 * P.beta * (fabs(f - 0.5) + 0.02 * gg)));
            known = (float)(P.beta * grow) * slope > 1e-12f && grow > least && 1e-4 * gg < smin * smin;
          }
          if (PROBE) ndir += known || probe_sign(S, c, P.beta, x, y, z, inside, f, g0, g1, g2) < 0.f ? -1 : 1;
          const bool dn = flip * g2 < 0;
          ndown += dn;
          const bool on = (P.mode % 2 == 1) || dn;
          // off: no penalty, and zero weights unless the direction is undefined
          if (on || !(gg > 0)) {
            const double rn = rsqrt(gg), n2 = flip * g2 * rn;  // n2: the unit normal's z
            const double inner = n2 * rcos;
            double val = 0, A = 0, B = 0;
            if (on) {
              const int m = P.mode;
              if (m <= 1) { val = pow(inner, P.fpara); B = P.fpara * pow(inner, P.fpara - 1); }
              else if (m <= 3) { val = inner >= 1 ? P.fpara * (inner - 1) * (inner - 1) : 0; B = inner >= 1 ? 2 * P.fpara * (inner - 1) : 0; }
              else {
                const double nd = exp(-P.na * (f - 0.5) * (f - 0.5));
                const double dnd = -2 * P.na * (f - 0.5) * nd;
                const double ex_ = exp(-(inner - P.mid) * rsc), q = __drcp_rn(1 + ex_);
                const double ov = 2 * q, dov = ov * q * rsc * ex_;
                const double in_ = inner > 1 ? P.ia * (inner - 1) + 1 : 1, din = inner > 1 ? P.ia : 1;
                val = nd * ov * in_; A = dnd * ov * in_; B = nd * dov * in_ + nd * ov * din;
              }
            }
            val32 = (float)val;
            if (inside) {
              // dinner = al*(N N dN) + be*(dN N N) + ga*(N dN N)  (see compute_spline_bg_selfsupp_constraint_dcoeff),
              // al = direction (nn - n2^2 / nn) / den, be = -direction n2 n0 / nn / den, den = nn^2 cosang
              const double k = B * (direction * rn * rcos), kt = -k * n2 * (flip * rn);
              wA = A; wZ = k * (1 - n2 * n2); wX = kt * g0; wY = kt * g1;
            }
          }
          sper += (double)val32;
        }
        if (per) per[x] = val32;
        w[warp][0][x - xa] = wA; w[warp][1][x - xa] = wX; w[warp][2][x - xa] = wY; w[warp][3][x - xa] = wZ;
      }
      __syncwarp();
      for (int a = lane; a < S.nb0; a += 32) {
        const int l0 = lo[a], ka = max(l0, xa) - l0, kb = in_yz ? min(hi[a], xb - 1) - l0 : -1;
        double s = 0, sy = 0, sz = 0;
        const double *bn = S.bN + a, *bd = S.bD + a;
#pragma unroll 2
        for (int k = ka; k <= kb; k++) {
          const double N = bn[(long long)k * S.nb0], D = bd[(long long)k * S.nb0];
          const int x = l0 + k - xa;
          s = fma(w[warp][0][x], N, fma(w[warp][1][x], D, s));
          sy = fma(w[warp][2][x], N, sy);
          sz = fma(w[warp][3][x], N, sz);
        }
        if (xa > x0 && kb < ka) continue;
        const bool first = xa == x0;
        Q.G1[gb + a] = first ? s : Q.G1[gb + a] + s;
        Q.Gy[gb + a] = first ? sy : Q.Gy[gb + a] + sy;
        Q.Gz[gb + a] = first ? sz : Q.Gz[gb + a] + sz;
      }
    }
  }
  sper = warp_add(sper);
  const double sdir = (double)__reduce_add_sync(0xffffffffu, ndir), sdown = (double)__reduce_add_sync(0xffffffffu, ndown);
  if (lane == 0) { red[warp][0] = sdir; red[warp][1] = sper; red[warp][2] = sdown; }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int k = 0; k < kSSRows; k++) t += red[k][threadIdx.x];
    Q.part[(threadIdx.x * (long long)gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = t;
  }
}
template <bool PROBE>
static auto ss_rows_of(int order) {
  return order == 2 ? k_ss_rows<2, PROBE> : order == 3 ? k_ss_rows<3, PROBE> : order == 4 ? k_ss_rows<4, PROBE>
                                                                                          : k_ss_rows<5, PROBE>;
}
static auto ss_rows(int order, bool probe) { return probe ? ss_rows_of<true>(order) : ss_rows_of<false>(order); }
// out[0..2] = the sums of probes, penalties and downward faces; out[3] the count the mean divides by
__global__ void __launch_bounds__(1024) k_ss_sums(const double* __restrict__ part, int n, int mode, double active,
                                                 double* __restrict__ out) {
  __shared__ double sh[32];
  double tot[3];
  for (int k = 0; k < 3; k++) {
    double s = 0;
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += 1024) s += part[(long long)k * n + i];
    s = warp_add(s);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    tot[k] = 0;
    for (int q = 0; q < 32; q++) tot[k] += sh[q];
  }
  if (threadIdx.x == 0) {
    out[0] = tot[0];
    out[1] = tot[1];
    out[2] = tot[2];
    out[3] = mode % 2 == 0 ? tot[2] : active;
  }
}

rso_status selfsupport(rso_handle* h, const double* c, double beta, int mode, double opt_angle, double default_angle,
                       float* per_dense, double* dc, double* value, double* count, double* dirsum) {
  const Level& l = h->L[0];
  if (!h->sp.order) { h->err = "spline not set up"; return RSO_ERR_STATE; }
  const SplineDev S = spline_dev(h, h->sp.knots_dev);
  SSPar P;
  P.mode = mode;
  P.beta = beta;
  P.cosang = std::cos(opt_angle);
  P.mid = std::cos(M_PI) / std::cos(default_angle);
  P.sc = (P.mid - 1) / std::log(1 / 0.004 - 1);
  P.fpara = mode <= 1 ? 8.0 : (mode <= 3 ? 10.0 : P.sc);  // p_norm, hfunction_c, adapt_sigmoid_c (grid/Grid.h:371-378)
  P.na = 200.0;
  P.ia = 15.0;
  const long long comp = (long long)S.nb0 * l.ey * l.ez, t2 = (long long)S.nb0 * S.nb1 * l.ez,
                  t3 = (long long)S.nb0 * S.nb1 * S.nb2;
  const XSplit X = x_split(l, 1, kSSSeg);
  const dim3 grid(ss_blocks(l), X.chunks);
  double* R = h->sp.work[2];
  double* sums = h->scal + 48;
  // H / M of the probe's bound
  const double p = S.order - 1, st[3] = {h->sp.step[0], h->sp.step[1], h->sp.step[2]};
  double hcoef = 0;
  for (int i = 0; i < 3; i++) {
    double row = 4 * p * (p - 1) / (st[i] * st[i]);
    for (int j = 0; j < 3; j++)
      if (j != i) row += 4 * p * p / (st[i] * st[j]);
    hcoef = std::max(hcoef, row);
  }
  double smin = st[0];
  for (int i = 0; i < 3; i++) smin = std::min(smin, std::min(st[i], -(double)h->sp.bmin[i]));
  k_max_abs<<<1, 1024, 0, h->stream>>>(h->sp.n_coeff, c, sums + 4); rso::note_launch();
  RSO_TRY(spline_rows(h, S, c, R, true));
  SSOut O;
  O.G1 = h->sp.work[0];
  O.Gy = O.G1 + comp;
  O.Gz = O.Gy + comp;
  O.per = per_dense;
  O.part = R + 3 * comp;
  double *G2 = h->sp.work[1], *G2z = G2 + t2;
  const int *r0 = h->sp.ranges[0], *r2 = h->sp.ranges[2];
  double flip = -1.0, direction = -1.0, ds = 0;
  for (int pass = 0; pass < 2; pass++) {
    auto rows = ss_rows(S.order, pass == 0);
    rows<<<grid, 32 * kSSRows, 0, h->stream>>>(l, S, c, R, comp, P, flip, direction, sums + 4, hcoef, smin, r0,
                                               r0 + S.nb0, X.len, O, view_of(l, true)); rso::note_launch();
    k_ss_sums<<<1, 1024, 0, h->stream>>>(O.part, (int)(grid.x * grid.y), mode, (double)l.n_active_e, sums); rso::note_launch();
    if (dc) {
      adj_y(h, S, X, 3 * comp, O.G1, O.Gy, G2);
      adj_y(h, S, X, 3 * comp, O.Gz, nullptr, G2z);
      k_adj_z<<<cdiv(t3, 32), dim3(32, 8), 0, h->stream>>>(S, G2, G2z, r2, r2 + S.nb2, sums + 3, dc); rso::note_launch();
    }
    RSO_TRY(launch_check(h, "selfsupport"));
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(h->h_scal + 48, sums, 4 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    RSO_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
    if (pass == 0) ds = h->h_scal[48];
    const double f = ds < 0 ? -1.0 : 1.0, d = ds > 0 ? 1.0 : -1.0;
    if (f == flip && d == direction) break;
    flip = f;
    direction = d;
  }
  const double sum = h->h_scal[49], cnt = h->h_scal[51];
  if (dirsum) *dirsum = ds;
  if (count) *count = cnt;
  double v = 0;
  if (cnt != 0) v = (mode <= 1) ? std::pow(sum / cnt, 1 / P.fpara) - 1 : sum / cnt;
  if (value) *value = v;
  return RSO_OK;
}

// knot series (grid/Grid.cpp:3307-3431, float arithmetic as the reference):
// the box [0, e] is enlarged by 2*e/(P+1) on both sides, step = (max-min)/(P+1),
// 'order' repeated end knots, n_basis = order + P.
rso_status spline_setup(rso_handle* h, int order, int px, int py, int pz) {
  if (order < 2 || order > 5 || px < 0 || py < 0 || pz < 0) return RSO_ERR_INVALID_ARG;
  Spline& s = h->sp;
  const Level& l = h->L[0];
  // not set up (order 0: the entry points refuse) until every buffer is there
  s.order = 0;
  auto drop = [](auto*& p) { cudaFree(p); p = nullptr; };
  for (int a = 0; a < 3; a++) {
    drop(s.idx[a]); drop(s.N[a]); drop(s.dN[a]); drop(s.ranges[a]);
  }
  drop(s.knots_dev);
  drop(s.xtab);
  for (auto& p : s.work) drop(p);
  drop(h->coef_a); drop(h->coef_b); drop(h->coef_c);
  drop(h->coef_df); drop(h->coef_dg);  // the design iteration makes them in the new size
  s.part[0] = px; s.part[1] = py; s.part[2] = pz;
  const int edim[3] = {l.ex, l.ey, l.ez};
  std::vector<float> allk;
  for (int a = 0; a < 3; a++) {
    const int P = s.part[a];
    s.nb[a] = order + P;
    float mn = 0.0f, mx = (float)edim[a];
    const float delta = mx - mn, scale_bound = 2.0f;
    mx += scale_bound * delta / (float)(P + 1);
    mn -= scale_bound * delta / (float)(P + 1);
    s.bmin[a] = mn; s.bmax[a] = mx;
    s.step[a] = (mx - mn) / (float)(P + 1);
    auto& K = s.knots[a];
    K.clear();
    float tmp = mn;
    for (int i = 0; i < order; i++) K.push_back(mn);
    for (int i = order; i < order + P; i++) { tmp += s.step[a]; K.push_back(tmp); }
    for (int i = order + P; i < 2 * order + P; i++) K.push_back(mx);
    allk.insert(allk.end(), K.begin(), K.end());
  }
  RSO_CHECK_CUDA(h, cudaMalloc(&s.knots_dev, sizeof(float) * allk.size()));
  RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.knots_dev, allk.data(), sizeof(float) * allk.size(), cudaMemcpyHostToDevice, h->stream));
  size_t koff = 0;
  for (int a = 0; a < 3; a++) {
    const int n = edim[a];
    RSO_CHECK_CUDA(h, cudaMalloc(&s.idx[a], sizeof(int) * n));
    RSO_CHECK_CUDA(h, cudaMalloc(&s.N[a], sizeof(double) * n * order));
    RSO_CHECK_CUDA(h, cudaMalloc(&s.dN[a], sizeof(double) * n * order));
    k_spline_axis<<<cdiv(n, 128), 128, 0, h->stream>>>(n, order, s.nb[a], s.bmin[a], s.step[a], s.knots_dev + koff,
                                                        s.idx[a], s.N[a], s.dN[a]); rso::note_launch();
    RSO_TRY(launch_check(h, "spline_axis"));
    koff += s.knots[a].size();
    s.h_idx[a].resize(n);
    s.h_N[a].resize((size_t)n * order);
    s.h_dN[a].resize((size_t)n * order);
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.h_idx[a].data(), s.idx[a], sizeof(int) * n, cudaMemcpyDeviceToHost, h->stream));
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.h_N[a].data(), s.N[a], sizeof(double) * n * order, cudaMemcpyDeviceToHost, h->stream));
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.h_dN[a].data(), s.dN[a], sizeof(double) * n * order, cudaMemcpyDeviceToHost, h->stream));
    RSO_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
    // support ranges of every basis function along this axis
    std::vector<int> rg(2 * s.nb[a]);
    for (int b = 0; b < s.nb[a]; b++) { rg[b] = 0; rg[s.nb[a] + b] = -1; }
    std::vector<bool> seen(s.nb[a], false);
    for (int x = 0; x < n; x++) {
      const int i = s.h_idx[a][x];
      if (i < 0) continue;
      for (int b = i - order; b < i; b++) {
        if (!seen[b]) { rg[b] = x; seen[b] = true; }
        rg[s.nb[a] + b] = x;
      }
    }
    if (a == 0) {
      // the x axis by function (see SplineDev); n and order values twice, then the supports'
      const int nb = s.nb[0];
      s.sup = 1;
      for (int b = 0; b < nb; b++) s.sup = std::max(s.sup, rg[nb + b] - rg[b] + 1);
      std::vector<double> tab(2 * ((size_t)n * order + (size_t)nb * s.sup), 0.0);
      double *tn = tab.data(), *td = tn + (size_t)n * order, *bn = td + (size_t)n * order, *bd = bn + (size_t)nb * s.sup;
      for (int x = 0; x < n; x++)
        for (int q = 0; q < order; q++) {
          const double N = s.h_N[0][(size_t)x * order + q], D = s.h_dN[0][(size_t)x * order + q];
          tn[(size_t)q * n + x] = N;
          td[(size_t)q * n + x] = D;
          if (s.h_idx[0][x] < 0) continue;
          const int b = s.h_idx[0][x] - order + q;
          bn[(size_t)(x - rg[b]) * nb + b] = N;
          bd[(size_t)(x - rg[b]) * nb + b] = D;
        }
      RSO_CHECK_CUDA(h, cudaMalloc(&s.xtab, sizeof(double) * tab.size()));
      RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.xtab, tab.data(), sizeof(double) * tab.size(), cudaMemcpyHostToDevice, h->stream));
    }
    RSO_CHECK_CUDA(h, cudaMalloc(&s.ranges[a], sizeof(int) * rg.size()));
    RSO_CHECK_CUDA(h, cudaMemcpyAsync(s.ranges[a], rg.data(), sizeof(int) * rg.size(), cudaMemcpyHostToDevice, h->stream));
  }
  s.n_coeff = (long long)s.nb[0] * s.nb[1] * s.nb[2];
  // work[0]: spline rows, or stage 1 of the adjoints (one or three weights, every chunk of x); work[1]: the
  // two arrays of the other stage; work[2]: the self-support constraint's rows of value and derivatives, and
  // its partial sums
  const size_t comp = (size_t)s.nb[0] * l.ey * l.ez;
  const size_t ca = x_split(l, kAdjRows, kSeg).chunks, cs = x_split(l, 1, kSSSeg).chunks;
  RSO_CHECK_CUDA(h, cudaMalloc(&s.work[0], sizeof(double) * std::max(ca, 3 * cs) * comp));
  RSO_CHECK_CUDA(h, cudaMalloc(&s.work[2], sizeof(double) * (3 * comp + 3 * cs * ss_blocks(l))));
  RSO_CHECK_CUDA(h, cudaMalloc(&s.work[1], sizeof(double) * 2 * (size_t)s.nb[0] * s.nb[1] * l.ez));
  RSO_CHECK_CUDA(h, cudaMalloc(&h->coef_a, sizeof(double) * s.n_coeff));
  RSO_CHECK_CUDA(h, cudaMalloc(&h->coef_b, sizeof(double) * s.n_coeff));
  RSO_CHECK_CUDA(h, cudaMalloc(&h->coef_c, sizeof(double) * s.n_coeff));
  s.order = order;
  return RSO_OK;
}

}  // namespace rso
