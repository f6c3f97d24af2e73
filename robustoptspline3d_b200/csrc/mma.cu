// Svanberg MMA (the reference's mma_t: optimization/mma_t.h:159-266,
// mma_t.cpp:18-118, mma_t.cu:15-909) in FP64 on the device.  An update is one
// cooperative kernel: the n-sized work (p/q, the reduced-system sums, the step
// bounds, the KKT residual of every line-search trial, the asymptotes) with
// deterministic grid-wide reductions, and the (m+1)^2 dual system with the
// m-sized bookkeeping, which every CTA carries out alike.
#include "rso_internal.cuh"
#include <cmath>
#include <algorithm>
#include <string>

constexpr int MMA_MAXM = 5;                       // constraints an update is built for
constexpr int MMA_BLOCKS = 256, MMA_THREADS = 256;  // set-up kernels
constexpr int MMA_UT = 512;                       // threads of a CTA of the update kernel
constexpr int MMA_RED = MMA_MAXM * MMA_MAXM + 2 * MMA_MAXM + 6;  // most values one reduction carries

struct rso_mma {
  int n = 0, m = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  double *x = nullptr, *xmin = nullptr, *xmax = nullptr, *L = nullptr, *U = nullptr, *alpha = nullptr,
         *beta = nullptr, *lastdx = nullptr, *xi = nullptr, *eta = nullptr, *curx = nullptr;
  double *P = nullptr, *Q = nullptr, *Dx = nullptr, *hdx = nullptr, *G = nullptr, *dx = nullptr, *dxi = nullptr,
         *deta = nullptr;
  double *part = nullptr, *res = nullptr, *h_res = nullptr;
  unsigned* bar = nullptr;  // the update kernel's grid barrier (gbar_sync)
  int ctas = 1;             // its CTAs, resident together: one per SM at most
  int stop_counter = 0;
};

namespace {

__global__ void k_reset(int n, double* x, const double* alpha, const double* beta, double* xi, double* eta) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double xv = 0.5 * (alpha[i] + beta[i]);
    x[i] = xv;
    xi[i] = fmax(1.0 / (xv - alpha[i]), 1.0);
    eta[i] = fmax(1.0 / (beta[i] - xv), 1.0);
  }
}

struct MmaArgs {
  int n;
  const double *df, *dg, *xmin, *xmax;
  double *x, *L, *U, *alpha, *beta, *lastdx, *xi, *eta, *curx, *P, *Q, *Dx, *hdx, *G, *dx, *dxi, *deta;
  double g[MMA_MAXM];
  double* part;   // [2][MMA_RED][CTAs]
  double* out;    // error, last step, sub-iterations, overflow, |dx|^2
  unsigned* bar;
};

// The m-sized state of the subproblem (a = 0, a0 = 1, c = 10, d = 1:
// optimization/mma_t.h:202-211), one copy per CTA, changed by thread 0 alone
template <int M>
struct Dual {
  double lam[M], lam_pq[M], y[M], mu[M], s[M], b[M];  // multipliers and slacks; lam_pq: those p and q were last formed with
  double dl[M], dy[M], dmu[M], ds[M], nl[M];          // search direction, and the trial's multipliers
  double z, zeta, dz, dzeta, eps, step, old_err, new_err, err, lasterr, damp;
  int stays, nsub, overflow, accepted, go;
};
constexpr double MMA_C = 10.0, MMA_D = 1.0, MMA_A0 = 1.0;

// Grid-wide sums (and maxima, bit r of mx) of R values per thread into
// res[0..R) of every CTA: shuffles and shared memory within a CTA, one partial
// per CTA in the buffer of this reduction's parity, a grid barrier, and every
// CTA adds the partials up in the same order.  False once a barrier wait has
// given up.
template <int R>
__device__ bool grid_reduce(double (&v)[R], unsigned long long mx, const MmaArgs& A, int& parity, unsigned& goal, double* res,
                            double (*sh)[MMA_UT / 32]) {
  static_assert(R <= MMA_RED && R <= 64, "a bit of the maxima mask and a slot per value");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < R; r++) {
    const bool m = (mx >> r) & 1ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double t = __shfl_down_sync(0xffffffffu, v[r], o);
      v[r] = m ? fmax(v[r], t) : v[r] + t;
    }
    if (lane == 0) sh[r][warp] = v[r];
  }
  __syncthreads();
  double* part = A.part + (long long)parity * MMA_RED * gridDim.x;
  parity ^= 1;
  if (threadIdx.x < R) {
    const int r = threadIdx.x;
    const bool m = (mx >> r) & 1ull;
    double acc = sh[r][0];
    for (int k = 1; k < MMA_UT / 32; k++) acc = m ? fmax(acc, sh[r][k]) : acc + sh[r][k];
    if (gridDim.x == 1) res[r] = acc;
    else part[(long long)r * gridDim.x + blockIdx.x] = acc;
  }
  if (gridDim.x == 1) {
    __syncthreads();
    return true;
  }
  if (!rso::gbar_sync(A.bar, goal, threadIdx.x, gridDim.x)) return false;
  for (int r = warp; r < R; r += MMA_UT / 32) {
    const bool m = (mx >> r) & 1ull;
    double acc = m ? -1e300 : 0.0;
    for (int k = lane; k < (int)gridDim.x; k += 32) {
      const double t = __ldcg(part + (long long)r * gridDim.x + k);
      acc = m ? fmax(acc, t) : acc + t;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double t = __shfl_down_sync(0xffffffffu, acc, o);
      acc = m ? fmax(acc, t) : acc + t;
    }
    if (lane == 0) res[r] = acc;
  }
  __syncthreads();
  return true;
}

// partial pivoting, as the host solve of earlier versions
template <int N>
__device__ void dense_solve(double (&A)[N][N], double (&b)[N], double (&x)[N]) {
  for (int k = 0; k < N; k++) {
    int piv = k;
    for (int i = k + 1; i < N; i++)
      if (fabs(A[i][k]) > fabs(A[piv][k])) piv = i;
    if (piv != k) {
      for (int j = 0; j < N; j++) { const double t = A[k][j]; A[k][j] = A[piv][j]; A[piv][j] = t; }
      const double t = b[k]; b[k] = b[piv]; b[piv] = t;
    }
    for (int i = k + 1; i < N; i++) {
      const double f = A[i][k] / A[k][k];
      for (int j = k; j < N; j++) A[i][j] -= f * A[k][j];
      b[i] -= f * b[k];
    }
  }
  for (int i = N - 1; i >= 0; i--) {
    double t = b[i];
    for (int j = i + 1; j < N; j++) t -= A[i][j] * x[j];
    x[i] = t / A[i][i];
  }
}

// 2-norm and inf-norm of the KKT residual (kkt_err, mma_t.cu:574-678): the n-sized sums q[0..2], the proxies
// gp and the n-sized maxima, and the m-sized rows
template <int M>
__device__ void kkt_norms(const Dual<M>& D, const double* q, const double* gp, const double* mx, const double* lam,
                          const double* y, double z, const double* mu, double zeta, const double* s, double damp,
                          double* e2, double* einf) {
  double sum = q[0] + q[1] + q[2], m = fmax(-10.0, fmax(mx[0], fmax(mx[1], mx[2])));
  auto acc = [&](double v) { sum += v * v; m = fmax(m, fabs(v)); };
  for (int j = 0; j < M; j++) acc(MMA_C + MMA_D * y[j] - lam[j] - mu[j]);
  acc(MMA_A0 - zeta);
  for (int j = 0; j < M; j++) acc((gp[j] - y[j] + s[j] - D.b[j]) / damp);
  for (int j = 0; j < M; j++) acc(mu[j] * y[j] - D.eps);
  acc(zeta * z - D.eps);
  for (int j = 0; j < M; j++) acc(lam[j] * s[j] - D.eps);
  *e2 = sqrt(sum);
  *einf = m;
}

// One update (mma_t::update) in one launch.  What bounds it is latency: some
// thirty Newton steps of three reductions each on a few hundred kilobytes that
// stay in L2.  As separate kernels with the dual system on the host an update of
// 32,768 variables took 6.7 ms, 2.7 of them in single-thread final sums and most
// of the rest in the 60 round trips.  A Newton step is three passes over the
// variables, each ending in a grid reduction: the system's sums together with
// the KKT residual at the current point (and the previous step taken), the
// direction with its step bounds, and the KKT residual of a trial: 1.08 ms with
// the copies of the design in and out.
template <int M>
__global__ void __launch_bounds__(MMA_UT, 1) k_mma_update(const __grid_constant__ MmaArgs A) {
  __shared__ double sh[MMA_RED][MMA_UT / 32];
  __shared__ double res[MMA_RED];
  __shared__ Dual<M> D;
  const int n = A.n, t0 = blockIdx.x * MMA_UT + threadIdx.x, ts = gridDim.x * MMA_UT;
  int parity = 0;
  unsigned goal = 0;
#define MMA_REDUCE(v, mx) \
  if (!grid_reduce(v, mx, A, parity, goal, res, sh)) return
  // init (mma_t.cu:69-106): p, q and the proxy offsets b at the current design; reset (mma_t.cu:702-713)
  {
    double v[M] = {};
    for (int i = t0; i < n; i += ts) {
      const double x = A.x[i], ux = A.U[i] - x, xl = x - A.L[i], raa = 1e-5 / (A.xmax[i] - A.xmin[i]);
      A.curx[i] = x;
#pragma unroll
      for (int j = 0; j <= M; j++) {
        const double d = j == 0 ? A.df[i] : A.dg[(long long)(j - 1) * n + i];
        const double pos = fmax(d, 0.0), neg = fmax(-d, 0.0);
        const double P = ux * ux * (1.001 * pos + 0.001 * neg + raa), Q = xl * xl * (0.001 * pos + 1.001 * neg + raa);
        A.P[(long long)j * n + i] = P;
        A.Q[(long long)j * n + i] = Q;
        if (j > 0) v[j - 1] += P / ux + Q / xl;
      }
      const double al = A.alpha[i], be = A.beta[i], xv = 0.5 * (al + be);
      A.x[i] = xv;
      A.xi[i] = fmax(1.0 / (xv - al), 1.0);
      A.eta[i] = fmax(1.0 / (be - xv), 1.0);
    }
    MMA_REDUCE(v, 0ull);
    if (threadIdx.x == 0) {
      for (int j = 0; j < M; j++) {
        D.b[j] = res[j] - A.g[j];
        D.y[j] = D.lam[j] = D.s[j] = 1;
        D.mu[j] = fmax(MMA_C / 2, 1.0);
        D.lam_pq[j] = 1;
      }
      D.z = D.zeta = 1;
      D.eps = 1;
      D.err = 1e30;
      D.lasterr = 0;
      D.step = 0;
      D.damp = 1;
      D.stays = D.nsub = D.overflow = D.accepted = 0;
      D.go = 1;
    }
    __syncthreads();
  }
  while (D.go) {
    // the accepted step taken; Newton system (solveLinearSystem, mma_t.cu:228-328) and KKT residual
    {
      constexpr int NS = M * M + 2 * M;
      double v[NS + 6] = {};
      const bool take = D.accepted != 0;
      const double step = D.step, eps = D.eps;
      for (int i = t0; i < n; i += ts) {
        double x = A.x[i], xi = A.xi[i], eta = A.eta[i];
        if (take) {
          x += step * A.dx[i]; xi += step * A.dxi[i]; eta += step * A.deta[i];
          A.x[i] = x; A.xi[i] = xi; A.eta[i] = eta;
        }
        const double ux = A.U[i] - x, xl = x - A.L[i], xa = x - A.alpha[i], bx = A.beta[i] - x;
        const double iu = 1 / ux, il = 1 / xl, iu2 = iu * iu, il2 = il * il;
        double p[M + 1], q[M + 1];
#pragma unroll
        for (int j = 0; j <= M; j++) { p[j] = A.P[(long long)j * n + i]; q[j] = A.Q[(long long)j * n + i]; }
        double pl = p[0], ql = q[0], pk = p[0], qk = q[0];
#pragma unroll
        for (int j = 0; j < M; j++) {
          pl += D.lam_pq[j] * p[j + 1]; ql += D.lam_pq[j] * q[j + 1];
          pk += D.lam[j] * p[j + 1]; qk += D.lam[j] * q[j + 1];
        }
        const double dxv = 2 * pl * iu2 * iu + 2 * ql * il2 * il + xi / xa + eta / bx;
        const double h = -(eps / xa - eps / bx - (pl * iu2 - ql * il2)), id = 1 / dxv;
        A.Dx[i] = id;
        A.hdx[i] = h;
        double g[M];
#pragma unroll
        for (int j = 0; j < M; j++) {
          g[j] = p[j + 1] * iu2 - q[j + 1] * il2;
          A.G[(long long)j * n + i] = g[j];
        }
        int r = 0;
#pragma unroll
        for (int j = 0; j < M; j++)
#pragma unroll
          for (int k = 0; k < M; k++) v[r++] += g[j] * (g[k] * id);
#pragma unroll
        for (int j = 0; j < M; j++) v[r++] += g[j] * (h * id);
#pragma unroll
        for (int j = 0; j < M; j++) v[r++] += p[j + 1] * iu + q[j + 1] * il;
        const double rex = pk * iu2 - qk * il2 - xi + eta, rxs = xi * xa - eps, ret = eta * bx - eps;
        v[NS] += rex * rex; v[NS + 1] += rxs * rxs; v[NS + 2] += ret * ret;
        v[NS + 3] = fmax(v[NS + 3], fabs(rex));
        v[NS + 4] = fmax(v[NS + 4], fabs(rxs));
        v[NS + 5] = fmax(v[NS + 5], fabs(ret));
      }
      MMA_REDUCE(v, 7ull << (NS + 3));
      if (threadIdx.x == 0) {
        const double *sg = res + M * M, *gp = res + M * M + M;
        double K[M + 1][M + 1], rhs[M + 1], sol[M + 1], hdy[M], Dy[M];
        for (int j = 0; j < M; j++) {
          Dy[j] = MMA_D + D.mu[j] / D.y[j];
          hdy[j] = -(D.lam[j] + D.eps / D.y[j] - MMA_C - MMA_D * D.y[j]);
          const double hdl = -(D.y[j] + D.b[j] - D.eps / D.lam[j] - gp[j]);
          for (int k = 0; k < M; k++) K[j][k] = res[j * M + k];
          K[j][j] += D.s[j] / D.lam[j] + 1 / Dy[j];
          K[j][M] = K[M][j] = 0;  // a = 0
          rhs[j] = hdl + hdy[j] / Dy[j] - sg[j];
        }
        K[M][M] = -D.zeta / D.z;
        rhs[M] = -(D.eps / D.z - MMA_A0);
        dense_solve<M + 1>(K, rhs, sol);
        D.dz = sol[M];
        for (int j = 0; j < M; j++) {
          D.dl[j] = sol[j];
          D.dy[j] = sol[j] / Dy[j] - hdy[j] / Dy[j];
          D.dmu[j] = D.eps / D.y[j] - D.dy[j] * D.mu[j] / D.y[j] - D.mu[j];
          D.ds[j] = D.eps / D.lam[j] - D.s[j] / D.lam[j] * sol[j] - D.s[j];
          D.lam_pq[j] = D.lam[j];
        }
        D.dzeta = D.eps / D.z - D.zeta - (D.zeta / D.z) * D.dz;
        double inf;
        kkt_norms<M>(D, res + NS, gp, res + NS + 3, D.lam, D.y, D.z, D.mu, D.zeta, D.s, 1.0, &D.old_err, &inf);
      }
      __syncthreads();
    }
    // search direction and step bounds
    {
      double v[4] = {-1e300, -1e300, -1e300, -1e300};
      const double cf = 0.99, eps = D.eps;
      for (int i = t0; i < n; i += ts) {
        const double id = A.Dx[i], x = A.x[i], xi = A.xi[i], eta = A.eta[i];
        double t = -A.hdx[i] * id;
#pragma unroll
        for (int j = 0; j < M; j++) t -= D.dl[j] * A.G[(long long)j * n + i] * id;
        const double ia = 1 / (x - A.alpha[i]), ib = 1 / (A.beta[i] - x);
        const double di = eps * ia - t * ia * xi - xi, de = eps * ib + eta * ib * t - eta;
        A.dx[i] = t; A.dxi[i] = di; A.deta[i] = de;
        v[0] = fmax(v[0], (-1 / cf) * (t * ia));
        v[1] = fmax(v[1], (1 / cf) * (t * ib));
        v[2] = fmax(v[2], (-1 / cf) * di / xi);
        v[3] = fmax(v[3], (-1 / cf) * de / eta);
      }
      MMA_REDUCE(v, 15ull);
      if (threadIdx.x == 0) {
        double t3 = fmax(res[2], res[3]);
        auto art = [&](double dv, double w) { t3 = fmax(t3, (-1 / cf) * dv / w); };
        for (int j = 0; j < M; j++) {
          art(D.dy[j], D.y[j]);
          art(D.dl[j], D.lam[j]);
          art(D.dmu[j], D.mu[j]);
          art(D.ds[j], D.s[j]);
        }
        art(D.dz, D.z);
        art(D.dzeta, D.zeta);
        D.step = 1 / fmax(fmax(res[0], res[1]), fmax(t3, 1.0));
        D.new_err = 1e30;
        D.err = 1e30;
        D.accepted = 0;
        for (int j = 0; j < M; j++) D.nl[j] = D.lam[j] + D.dl[j] * D.step;
      }
      __syncthreads();
    }
    // search_step (mma_t.cu:501-571)
    while (D.accepted == 0 && D.step > 1e-12 && D.new_err > D.old_err) {
      double v[3 + M + 3] = {};
      const double step = D.step, eps = D.eps;
      for (int i = t0; i < n; i += ts) {
        const double x = A.x[i] + step * A.dx[i], xi = A.xi[i] + step * A.dxi[i], eta = A.eta[i] + step * A.deta[i];
        const double iu = 1 / (A.U[i] - x), il = 1 / (x - A.L[i]);
        double pl = A.P[i], ql = A.Q[i];
#pragma unroll
        for (int j = 0; j < M; j++) {
          const double p = A.P[(long long)(j + 1) * n + i], q = A.Q[(long long)(j + 1) * n + i];
          pl += D.nl[j] * p; ql += D.nl[j] * q;
          v[3 + j] += p * iu + q * il;
        }
        const double rex = pl * iu * iu - ql * il * il - xi + eta;
        const double rxs = xi * (x - A.alpha[i]) - eps, ret = eta * (A.beta[i] - x) - eps;
        v[0] += rex * rex; v[1] += rxs * rxs; v[2] += ret * ret;
        v[3 + M] = fmax(v[3 + M], fabs(rex));
        v[4 + M] = fmax(v[4 + M], fabs(rxs));
        v[5 + M] = fmax(v[5 + M], fabs(ret));
      }
      MMA_REDUCE(v, 7ull << (3 + M));
      if (threadIdx.x == 0) {
        double ny[M], nmu[M], ns[M];
        for (int j = 0; j < M; j++) {
          ny[j] = D.y[j] + D.dy[j] * step; nmu[j] = D.mu[j] + D.dmu[j] * step; ns[j] = D.s[j] + D.ds[j] * step;
          D.lam_pq[j] = D.nl[j];  // the reference's kkt_err refreshes plambda/qlambda with the trial multipliers
        }
        const double nz = D.z + D.dz * step, nzeta = D.zeta + D.dzeta * step;
        kkt_norms<M>(D, res, res + 3, res + 3 + M, D.nl, ny, nz, nmu, nzeta, ns, D.damp, &D.new_err, &D.err);
        if (D.new_err < D.old_err) {
          for (int j = 0; j < M; j++) { D.lam[j] = D.nl[j]; D.y[j] = ny[j]; D.mu[j] = nmu[j]; D.s[j] = ns[j]; }
          D.z = nz;
          D.zeta = nzeta;
          D.accepted = 1;
        } else {
          D.step /= 2;
          for (int j = 0; j < M; j++) D.nl[j] = D.lam[j] + D.dl[j] * D.step;
        }
      }
      __syncthreads();
    }
    __syncthreads();  // every thread has read the loop's condition
    if (threadIdx.x == 0) {
      if ((D.err - D.lasterr) / D.err < 1e-5) D.stays++;
      else D.stays = 0;
      D.lasterr = D.err;
      if (D.stays > 6) { D.damp *= 10; D.stays = 0; }
      if (D.nsub++ > 80) {
        D.overflow = 1;
        D.go = 0;
      } else if (!(D.err > 0.9 * D.eps)) {  // the next barrier parameter
        D.eps *= 0.1;
        D.damp = 1;
        D.stays = 0;
        D.go = D.eps > 1e-6;
      }
    }
    __syncthreads();
  }
  // the last accepted step, adjust_asym (mma_t.cu:164-226) and |dx|^2
  {
    double v[1] = {};
    const bool take = D.accepted != 0;
    const double step = D.step;
    for (int i = t0; i < n; i += ts) {
      double xv = A.x[i];
      if (take) {
        xv += step * A.dx[i];
        A.x[i] = xv;
        A.xi[i] += step * A.dxi[i];
        A.eta[i] += step * A.deta[i];
      }
      const double d1 = xv - A.curx[i], d2 = A.lastdx[i], lo = A.xmin[i], hi = A.xmax[i], st = hi - lo;
      double gamma = 1;
      if (d1 * d2 > 0) gamma = 1.2;
      if (d1 * d2 < 0) gamma = 0.7;
      double nl = xv - gamma * (xv - d1 - A.L[i]);
      double nu = xv + gamma * (A.U[i] - xv + d1);
      nl = fmin(fmax(nl, xv - 10 * st), xv - 0.01 * st);
      nu = fmin(fmax(nu, xv + 0.01 * st), xv + 10 * st);
      A.L[i] = nl; A.U[i] = nu;
      A.alpha[i] = fmax(fmax(lo, nl + 0.1 * (xv - nl)), xv - 0.5 * st);
      A.beta[i] = fmin(fmin(hi, nu - 0.1 * (nu - xv)), xv + 0.5 * st);
      A.lastdx[i] = d1;
      v[0] += d1 * d1;
    }
    MMA_REDUCE(v, 0ull);
  }
#undef MMA_REDUCE
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.out[0] = D.err;
    A.out[1] = D.step;
    A.out[2] = D.nsub;
    A.out[3] = D.overflow;
    A.out[4] = res[0];
  }
  if (gridDim.x > 1) rso::gbar_exit(A.bar, threadIdx.x);
}

// clamp_asymptotes (mma_t.cu:747-761)
__global__ void k_clamp_asym(int n, const double* x, double* L, double* U, double* alpha, double* beta,
                             const double* xmin, const double* xmax) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double st = xmax[i] - xmin[i], xv = x[i];
    L[i] = fmin(fmax(L[i], xv - 10 * st), xv - 0.01 * st);
    U[i] = fmin(fmax(U[i], xv + 0.01 * st), xv + 10 * st);
    alpha[i] = fmax(xmin[i], fmax(L[i] + 0.1 * (xv - L[i]), xv - 0.5 * st));
    beta[i] = fmin(xmax[i], fmin(U[i] - 0.1 * (U[i] - xv), xv + 0.5 * st));
  }
}

#define MMA_CHECK(s, call)                                                         \
  do {                                                                             \
    cudaError_t _e = (call);                                                       \
    if (_e != cudaSuccess) { cudaGetLastError(); (s)->err = cudaGetErrorString(_e); return RSO_ERR_CUDA; } \
  } while (0)

}  // namespace

extern "C" rso_status rso_mma_create(int n, int m, const double* xmin, const double* xmax, rso_mma** out) {
  if (!out || n <= 0 || m < 1 || m > MMA_MAXM || !xmin || !xmax) return RSO_ERR_INVALID_ARG;
  rso_mma* s = new rso_mma();
  s->n = n; s->m = m;
  auto fail = [&](rso_status st) { rso_mma_destroy(s); cudaGetLastError(); return st; };
  if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(RSO_ERR_CUDA);
  double** vecs[] = {&s->x, &s->xmin, &s->xmax, &s->L, &s->U, &s->alpha, &s->beta, &s->lastdx, &s->xi, &s->eta,
                     &s->curx, &s->Dx, &s->hdx, &s->dx, &s->dxi, &s->deta};
  for (double** v : vecs)
    if (cudaMalloc(v, sizeof(double) * n) != cudaSuccess) return fail(RSO_ERR_OOM);
  if (cudaMalloc(&s->P, sizeof(double) * n * (m + 1)) != cudaSuccess) return fail(RSO_ERR_OOM);
  if (cudaMalloc(&s->Q, sizeof(double) * n * (m + 1)) != cudaSuccess) return fail(RSO_ERR_OOM);
  if (cudaMalloc(&s->G, sizeof(double) * n * m) != cudaSuccess) return fail(RSO_ERR_OOM);
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return fail(RSO_ERR_CUDA);
  s->ctas = (int)std::min<long long>(sms, rso::cdiv(n, MMA_UT));
  if (cudaMalloc(&s->part, sizeof(double) * 2 * MMA_RED * s->ctas) != cudaSuccess) return fail(RSO_ERR_OOM);
  if (cudaMalloc(&s->bar, sizeof(unsigned) * 4) != cudaSuccess) return fail(RSO_ERR_OOM);
  cudaMemsetAsync(s->bar, 0, sizeof(unsigned) * 4, s->stream);
  if (cudaMalloc(&s->res, sizeof(double) * 64) != cudaSuccess) return fail(RSO_ERR_OOM);
  if (cudaMallocHost(&s->h_res, sizeof(double) * 64) != cudaSuccess) return fail(RSO_ERR_OOM);
  // on the MMA's own stream: copies and fills on the default one may still be under way when they return
  cudaMemcpyAsync(s->xmin, xmin, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->xmax, xmax, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  // set_bound (mma_t.cu:809-819) and init_subproblem_variable (:797-807)
  cudaMemcpyAsync(s->alpha, xmin, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->beta, xmax, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->L, xmin, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(s->U, xmax, sizeof(double) * n, cudaMemcpyHostToDevice, s->stream);
  cudaMemsetAsync(s->lastdx, 0, sizeof(double) * n, s->stream);
  k_reset<<<MMA_BLOCKS, MMA_THREADS, 0, s->stream>>>(n, s->x, s->alpha, s->beta, s->xi, s->eta); rso::note_launch();
  k_clamp_asym<<<MMA_BLOCKS, MMA_THREADS, 0, s->stream>>>(n, s->x, s->L, s->U, s->alpha, s->beta, s->xmin, s->xmax); rso::note_launch();
  k_reset<<<MMA_BLOCKS, MMA_THREADS, 0, s->stream>>>(n, s->x, s->alpha, s->beta, s->xi, s->eta); rso::note_launch();
  if (cudaStreamSynchronize(s->stream) != cudaSuccess) return fail(RSO_ERR_CUDA);
  *out = s;
  return RSO_OK;
}

extern "C" rso_status rso_mma_set_x_dev(rso_mma* s, const double* x) {
  if (!s || !x) return RSO_ERR_INVALID_ARG;
  MMA_CHECK(s, cudaMemcpyAsync(s->x, x, sizeof(double) * s->n, cudaMemcpyDeviceToDevice, s->stream));
  k_clamp_asym<<<MMA_BLOCKS, MMA_THREADS, 0, s->stream>>>(s->n, s->x, s->L, s->U, s->alpha, s->beta, s->xmin, s->xmax); rso::note_launch();
  MMA_CHECK(s, cudaStreamSynchronize(s->stream));
  return RSO_OK;
}

extern "C" rso_status rso_mma_set_x(rso_mma* s, const double* x) {
  if (!s || !x) return RSO_ERR_INVALID_ARG;
  MMA_CHECK(s, cudaMemcpyAsync(s->x, x, sizeof(double) * s->n, cudaMemcpyHostToDevice, s->stream));
  k_clamp_asym<<<MMA_BLOCKS, MMA_THREADS, 0, s->stream>>>(s->n, s->x, s->L, s->U, s->alpha, s->beta, s->xmin, s->xmax); rso::note_launch();
  MMA_CHECK(s, cudaStreamSynchronize(s->stream));
  return RSO_OK;
}

extern "C" rso_status rso_mma_get(rso_mma* s, double* x, double* L, double* U, double* al, double* be) {
  if (!s) return RSO_ERR_INVALID_ARG;
  const size_t b = sizeof(double) * s->n;
  if (x) MMA_CHECK(s, cudaMemcpyAsync(x, s->x, b, cudaMemcpyDeviceToHost, s->stream));
  if (L) MMA_CHECK(s, cudaMemcpyAsync(L, s->L, b, cudaMemcpyDeviceToHost, s->stream));
  if (U) MMA_CHECK(s, cudaMemcpyAsync(U, s->U, b, cudaMemcpyDeviceToHost, s->stream));
  if (al) MMA_CHECK(s, cudaMemcpyAsync(al, s->alpha, b, cudaMemcpyDeviceToHost, s->stream));
  if (be) MMA_CHECK(s, cudaMemcpyAsync(be, s->beta, b, cudaMemcpyDeviceToHost, s->stream));
  MMA_CHECK(s, cudaStreamSynchronize(s->stream));
  return RSO_OK;
}

extern "C" const double* rso_mma_x_dev(rso_mma* s) { return s ? s->x : nullptr; }

// checkpoint of what an update carries to the next: x, the asymptotes L and
// U, the move limits alpha and beta, the previous step, the stop counter
extern "C" rso_status rso_mma_state_size(const rso_mma* s, long long* n_doubles) {
  if (!s || !n_doubles) return RSO_ERR_INVALID_ARG;
  *n_doubles = 6LL * s->n + 1;
  return RSO_OK;
}

extern "C" rso_status rso_mma_save(rso_mma* s, double* state_host) {
  if (!s || !state_host) return RSO_ERR_INVALID_ARG;
  const size_t b = sizeof(double) * s->n;
  const double* parts[6] = {s->x, s->L, s->U, s->alpha, s->beta, s->lastdx};
  for (int k = 0; k < 6; k++)
    MMA_CHECK(s, cudaMemcpyAsync(state_host + (size_t)k * s->n, parts[k], b, cudaMemcpyDeviceToHost, s->stream));
  MMA_CHECK(s, cudaStreamSynchronize(s->stream));
  state_host[6LL * s->n] = (double)s->stop_counter;
  return RSO_OK;
}

extern "C" rso_status rso_mma_load(rso_mma* s, const double* state_host) {
  if (!s || !state_host) return RSO_ERR_INVALID_ARG;
  const size_t b = sizeof(double) * s->n;
  double* parts[6] = {s->x, s->L, s->U, s->alpha, s->beta, s->lastdx};
  for (int k = 0; k < 6; k++)
    MMA_CHECK(s, cudaMemcpyAsync(parts[k], state_host + (size_t)k * s->n, b, cudaMemcpyHostToDevice, s->stream));
  MMA_CHECK(s, cudaStreamSynchronize(s->stream));
  s->stop_counter = (int)state_host[6LL * s->n];
  return RSO_OK;
}

extern "C" rso_status rso_mma_update(rso_mma* S, const double* df, const double* dg, const double* g, int* converged,
                                     double* info) {
  if (!S || !df || (!dg && S->m > 0) || !g) return RSO_ERR_INVALID_ARG;
  MmaArgs A;
  A.n = S->n;
  A.df = df; A.dg = dg; A.xmin = S->xmin; A.xmax = S->xmax;
  A.x = S->x; A.L = S->L; A.U = S->U; A.alpha = S->alpha; A.beta = S->beta; A.lastdx = S->lastdx;
  A.xi = S->xi; A.eta = S->eta; A.curx = S->curx; A.P = S->P; A.Q = S->Q; A.Dx = S->Dx; A.hdx = S->hdx; A.G = S->G;
  A.dx = S->dx; A.dxi = S->dxi; A.deta = S->deta;
  for (int j = 0; j < MMA_MAXM; j++) A.g[j] = j < S->m ? g[j] : 0.0;
  A.part = S->part; A.out = S->res; A.bar = S->bar;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(S->ctas);
  lc.blockDim = dim3(MMA_UT);
  lc.stream = S->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  lc.attrs = &at;
  lc.numAttrs = 1;
  void (*kernel)(MmaArgs) = S->m == 1   ? k_mma_update<1>
                            : S->m == 2 ? k_mma_update<2>
                            : S->m == 3 ? k_mma_update<3>
                            : S->m == 4 ? k_mma_update<4>
                                        : k_mma_update<5>;
  MMA_CHECK(S, cudaLaunchKernelEx(&lc, kernel, A)); rso::note_launch();
  // the result and the barrier's gave-up flag in one copy each, one synchronisation
  unsigned* flag = reinterpret_cast<unsigned*>(S->h_res + 8);
  MMA_CHECK(S, cudaMemcpyAsync(S->h_res, S->res, sizeof(double) * 5, cudaMemcpyDeviceToHost, S->stream));
  MMA_CHECK(S, cudaMemcpyAsync(flag, S->bar + 2, sizeof(unsigned), cudaMemcpyDeviceToHost, S->stream));
  MMA_CHECK(S, cudaStreamSynchronize(S->stream));
  if (*flag != 0) {
    MMA_CHECK(S, cudaMemsetAsync(S->bar, 0, sizeof(unsigned) * 4, S->stream));
    MMA_CHECK(S, cudaStreamSynchronize(S->stream));
    S->err = "a grid-barrier wait of the update kernel timed out";
    return RSO_ERR_CUDA;
  }
  if (std::sqrt(S->h_res[4]) < 1e-3) S->stop_counter++;
  if (info)
    for (int k = 0; k < 4; k++) info[k] = S->h_res[k];
  if (converged) *converged = S->stop_counter > 10 ? 1 : 0;
  return RSO_OK;
}

extern "C" void rso_mma_destroy(rso_mma* s) {
  if (!s) return;
  if (s->stream) cudaStreamSynchronize(s->stream);
  double* vecs[] = {s->x, s->xmin, s->xmax, s->L, s->U, s->alpha, s->beta, s->lastdx, s->xi, s->eta, s->curx,
                    s->Dx, s->hdx, s->dx, s->dxi, s->deta, s->P, s->Q, s->G, s->part, s->res};
  for (double* v : vecs) cudaFree(v);
  cudaFree(s->bar);
  if (s->h_res) cudaFreeHost(s->h_res);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
}

namespace rso {
double* mma_x(rso_mma* s) { return s->x; }
int mma_n(rso_mma* s) { return s->n; }
int mma_m(rso_mma* s) { return s->m; }
}  // namespace rso
