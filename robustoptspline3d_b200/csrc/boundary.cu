// Boundary-condition inputs of a mesh problem: shell elements, outward
// normals at points, region masks and region force fields.
//
// The reference builds them on the host with CGAL and Eigen:
//  - shell elements: HierarchyGrid::setSolidShellElement (grid/Grid.cpp:
//    253-322) walks every face's grown index box and asks the AABB tree for
//    the squared distance of each element centre to the mesh;
//  - normals: Grid::outwardNormal (grid/Grid.cpp:2838-2854), the closest
//    point of the mesh and its triangle's supporting-plane vector;
//  - regions and fields: the range and field classes of
//    boundary/BoundaryCondition.h, evaluated at node positions in
//    computeProjectionMatrix (grid/Grid.cpp:2694-2760).
// Here each is one FP64 kernel: a warp per face for the shell (an element
// in a face's index box within w of that face is within w of the mesh, and an
// element within w of the mesh lies in the index box of its nearest face, so
// the union over faces is the reference's set), a warp per point for the
// normals (the nearest face with the lowest index on a tie, found by a ring
// search over a uniform face grid, or by scanning all faces of small meshes),
// a warp per row of nodes or a thread per point for the regions and fields.  The file is compiled without
// multiply-add contraction so every product and sum rounds as in the host
// restatement the tests compare with.
#include "rso_internal.cuh"
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <new>
#include <thread>
#include <utility>
#include <vector>

namespace rso {
namespace {

struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 sub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ D3 cross(D3 a, D3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ D3 axpy(D3 a, double s, D3 d) { return {a.x + s * d.x, a.y + s * d.y, a.z + s * d.z}; }
__device__ __forceinline__ double qdiv(double n, double d) { return d != 0.0 ? n / d : 0.0; }
// Eigen normalized(): v / sqrt(|v|^2) when |v|^2 > 0, else v
__device__ __forceinline__ D3 unit(D3 v) {
  const double n = dot(v, v);
  if (!(n > 0.0)) return v;
  const double s = sqrt(n);
  return {v.x / s, v.y / s, v.z / s};
}

// Closest point of triangle (a, b, c) to p by Voronoi regions (Ericson,
// Real-Time Collision Detection, 5.1.5); degenerate edges give parameter 0.
__device__ D3 closest_on_triangle(D3 p, D3 a, D3 b, D3 c) {
  const D3 ab = sub(b, a), ac = sub(c, a), ap = sub(p, a);
  const double d1 = dot(ab, ap), d2 = dot(ac, ap);
  if (d1 <= 0.0 && d2 <= 0.0) return a;
  const D3 bp = sub(p, b);
  const double d3 = dot(ab, bp), d4 = dot(ac, bp);
  if (d3 >= 0.0 && d4 <= d3) return b;
  const double vc = d1 * d4 - d3 * d2;
  if (vc <= 0.0 && d1 >= 0.0 && d3 <= 0.0) return axpy(a, qdiv(d1, d1 - d3), ab);
  const D3 cp = sub(p, c);
  const double d5 = dot(ab, cp), d6 = dot(ac, cp);
  if (d6 >= 0.0 && d5 <= d6) return c;
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0.0 && d2 >= 0.0 && d6 <= 0.0) return axpy(a, qdiv(d2, d2 - d6), ac);
  const double va = d3 * d6 - d5 * d4;
  const double e43 = d4 - d3, e56 = d5 - d6;
  if (va <= 0.0 && e43 >= 0.0 && e56 >= 0.0) return axpy(b, qdiv(e43, e43 + e56), sub(c, b));
  const double den = va + vb + vc;
  const double v = qdiv(vb, den), w = qdiv(vc, den);
  return axpy(axpy(a, v, ab), w, ac);
}

__device__ __forceinline__ D3 vertex(const float* __restrict__ vtx, int i) {
  return {(double)vtx[3 * i], (double)vtx[3 * i + 1], (double)vtx[3 * i + 2]};
}

// Shell elements.  Every element of a byte array (rows of `pitch` bytes, a
// multiple of 8) is 0 (void), 1 (solid) or 2 (shell).  A warp takes a face: its
// lanes take rows of the face's grown index box, read eight elements at a time
// and compute distances for those still 1 only, since a face need not look at
// what another has marked (a stale 1 only costs the distance again, and every
// store to a byte stores the same 2).  Faces about the size of an element
// overlap in some hundred boxes, and nearly all of the FP64 work was there: one
// CTA a face testing every solid element took 3.2 ms for 262144 faces on 256^3
// elements, this 0.58 ms.  Faces whose box has more than kShellRows rows go to a
// list that a second launch works off by words of eight elements, its CTAs shared
// out over the list (one face after the other on the whole grid, a thread a row,
// left most threads idle: 277 ms for 40000 faces and w = 20 on 256^3, 12.6 so).
// Meshes of fewer faces than the GPU holds warps (kShellFew; on grids of under 32
// elements an edge, which all warps crowd on, kShellFewSmall) take one launch over
// all of them, a thread an element, the CTAs shared out likewise: no states and no
// list, whose three launches a coarse mesh does not earn back, and no lane walks a
// row alone.  A call, with its copies, so and by warps: 12 faces, 128^3, w = 3,
// 0.53 and 2.8 ms; 320 faces, 256^3, w = 10, 2.5 and 13.6 ms; 5120 faces, 128^3, w =
// 8, 1.01 and 0.93 ms, but 16^3, w = 3, 0.14 and 0.20 ms; 262144 faces, 256^3, w = 3,
// 5.6 and 4.3 ms.
constexpr int kShellRows = 2048, kShellFew = 148 * 24, kShellFewSmall = 8192, kShellCtas = 148 * 8;

struct ShellGrid {
  double b0[3], eh, w;
  int R, pitch;
};

// the index box of a face grown by the shell's width (all lanes of the warp together); 0 rows if it is empty
struct FaceBox {
  D3 a, b, c;
  double lo[3], hi[3];
  int lid[3], rid[3];
  double lim;  // squared distance to the face's bounding box from which an element is out
};

__device__ int face_box(const float* __restrict__ vtx, const int* __restrict__ faces, int f, const ShellGrid& G,
                        FaceBox* B) {
  const D3 a = vertex(vtx, faces[3 * f]), b = vertex(vtx, faces[3 * f + 1]), c = vertex(vtx, faces[3 * f + 2]);
  B->a = a, B->b = b, B->c = c;
  const double lo[3] = {fmin(fmin(a.x, b.x), c.x), fmin(fmin(a.y, b.y), c.y), fmin(fmin(a.z, b.z), c.z)};
  const double hi[3] = {fmax(fmax(a.x, b.x), c.x), fmax(fmax(a.y, b.y), c.y), fmax(fmax(a.z, b.z), c.z)};
  {  // lane j: the lower bound of axis j, lane 3 + j: its upper bound
    const int lane = threadIdx.x & 31, j = lane % 3;
    const bool up = lane >= 3;
    const double o = j == 0 ? G.b0[0] : (j == 1 ? G.b0[1] : G.b0[2]);
    const double l = j == 0 ? lo[0] : (j == 1 ? lo[1] : lo[2]), u = j == 0 ? hi[0] : (j == 1 ? hi[1] : hi[2]);
    double q = ((up ? u + G.w * 1.3 : l - G.w * 1.3) - o - 0.5 * G.eh) / G.eh;
    if (up) q += 1;
    // int conversion truncates; out-of-range quotients saturate before the clamp
    const int id = min(max((int)fmax(fmin(q, 2147483647.0), -2147483648.0), 0), G.R - 1);
    for (int k = 0; k < 3; k++) {
      B->lid[k] = __shfl_sync(0xffffffffu, id, k);
      B->rid[k] = __shfl_sync(0xffffffffu, id, 3 + k);
    }
  }
  double m2 = 0;  // (largest distance from an element of the box to a point of the face)^2
  for (int j = 0; j < 3; j++) {
    B->lo[j] = lo[j], B->hi[j] = hi[j];
    const double m = hi[j] - lo[j] + 1.3 * G.w + G.eh;
    m2 += m * m;
  }
  // Elements further than w from the face's bounding box need no distance if
  // the computed closest point lies on the face.  Rounding moves it off by at
  // most about 80 eps L^3 M^2 / |n|^2 (L the longest edge, M the distance, n
  // the face's normal: the barycentric sums cancel on slivers), so that is
  // kept below w / 1000 against the hundredth of w taken as margin; slivers
  // beyond it compute every distance.
  const D3 ab = sub(b, a), ac = sub(c, a), bc = sub(c, b), n = cross(ab, ac);
  const double l2 = fmax(dot(ab, ab), fmax(dot(ac, ac), dot(bc, bc)));
  const bool fit = dot(n, n) * G.w > 1e-10 * l2 * sqrt(l2) * m2;
  B->lim = fit ? 1.02 * G.w * G.w : INFINITY;
  const int nbx = B->rid[0] - B->lid[0], nby = B->rid[1] - B->lid[1], nbz = B->rid[2] - B->lid[2];
  return nbx > 0 && nby > 0 && nbz > 0 ? nby * nbz : 0;
}

__device__ __forceinline__ double outside(double x, double lo, double hi) {
  return x < lo ? lo - x : (x > hi ? x - hi : 0.0);
}

// row r of the box: its bytes and centre, and its distance^2 from the face's bounding box in y and z
struct ShellRow {
  uint8_t* row;
  double py, pz, ryz;
};
__device__ __forceinline__ ShellRow shell_row(const FaceBox& B, const ShellGrid& G, int r, uint8_t* state) {
  const int nby = B.rid[1] - B.lid[1], y = B.lid[1] + r % nby, z = B.lid[2] + r / nby;
  ShellRow W;
  W.row = state + ((size_t)z * G.R + y) * G.pitch;
  W.py = (y + 0.5) * G.eh + G.b0[1], W.pz = (z + 0.5) * G.eh + G.b0[2];
  const double oy = outside(W.py, B.lo[1], B.hi[1]), oz = outside(W.pz, B.lo[2], B.hi[2]);
  W.ryz = oy * oy + oz * oz;
  return W;
}
// its elements x8 .. x8 + 7 that lie in the box
__device__ __forceinline__ void shell_word(const FaceBox& B, const ShellGrid& G, const ShellRow& W, int x8) {
  const double sh2 = G.w * G.w;
  unsigned long long todo =
      __ldcg(reinterpret_cast<const unsigned long long*>(W.row + x8)) & 0x0101010101010101ull;
  if (x8 < B.lid[0]) todo &= ~0ull << (8 * (B.lid[0] - x8));
  if (x8 + 8 > B.rid[0]) todo &= ~0ull >> (8 * (x8 + 8 - B.rid[0]));
  for (; todo != 0; todo &= todo - 1) {
    const int x = x8 + (__ffsll((long long)todo) - 1) / 8;
    const D3 p = {(x + 0.5) * G.eh + G.b0[0], W.py, W.pz};
    const double ox = outside(p.x, B.lo[0], B.hi[0]);
    if (ox * ox + W.ryz > B.lim) continue;
    const D3 d = sub(p, closest_on_triangle(p, B.a, B.b, B.c));
    if (dot(d, d) < sh2) W.row[x] = 2;
  }
}

// A warp per face, in steps of `stride` (coprime to nf): neighbours in the list
// are neighbours in space, and in list order the warps at work together would
// all compute the distances of the same elements (1.29 ms; 0.75 ms in steps;
// 0.58 ms with the registers cut for six CTAs an SM).  `big` = {number, faces..}
// of those left to k_shell_big.
__global__ void __launch_bounds__(128, 6) k_shell(const float* __restrict__ vtx, const int* __restrict__ faces, int nf,
                                               int stride, ShellGrid G, uint8_t* state, int* __restrict__ big) {
  const long long wid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32;
  if (wid >= nf) return;
  const long long f = wid * stride % nf;
  FaceBox B;
  const int rows = face_box(vtx, faces, (int)f, G, &B), lane = threadIdx.x & 31;
  if (rows > kShellRows) {
    if (lane == 0) big[1 + atomicAdd(big, 1)] = (int)f;
    return;
  }
  for (int r = lane; r < rows; r += 32) {
    const ShellRow W = shell_row(B, G, r, state);
    if (W.ryz > B.lim) continue;
    for (int x8 = B.lid[0] & ~7; x8 < B.rid[0]; x8 += 8) shell_word(B, G, W, x8);
  }
}

// The grid's CTAs shared out over n faces: teams of `size` CTAs, this CTA being
// number `rank` of team `team`.  A team takes every teams-th face.
struct Team { int size, team, teams, rank; };
__device__ __forceinline__ Team team_of(int n, int least) {
  Team t;
  t.size = min(max((int)gridDim.x / max(n, 1), least), (int)gridDim.x);
  t.teams = gridDim.x / t.size;
  t.team = blockIdx.x / t.size;
  t.rank = blockIdx.x - t.team * t.size;
  return t;
}

// the listed faces, by words of eight elements
__global__ void __launch_bounds__(128) k_shell_big(const float* __restrict__ vtx, const int* __restrict__ faces,
                                                   ShellGrid G, uint8_t* state, const int* __restrict__ big) {
  const int nb = big[0];
  const Team T = team_of(nb, 8);
  if (T.team >= T.teams) return;
  for (int k = T.team; k < nb; k += T.teams) {
    FaceBox B;
    const int rows = face_box(vtx, faces, big[1 + k], G, &B);
    const int first = B.lid[0] & ~7;
    const unsigned nw = (B.rid[0] - first + 7) / 8;  // rows * nw <= 2048^3 / 8
    for (unsigned u = T.rank * 128 + threadIdx.x; u < rows * nw; u += T.size * 128) {
      const unsigned r = u / nw;
      const ShellRow W = shell_row(B, G, (int)r, state);
      if (!(W.ryz > B.lim)) shell_word(B, G, W, first + 8 * (int)(u - r * nw));
    }
  }
}

// all faces of a small mesh, by elements; an element that already is shell is left out (a stale byte
// only costs its distance again)
__global__ void __launch_bounds__(256) k_shell_few(const float* __restrict__ vtx, const int* __restrict__ faces, int nf,
                                                   ShellGrid G, const uint8_t* __restrict__ solid, uint8_t* shell) {
  const Team T = team_of(nf, 1);
  const double sh2 = G.w * G.w;
  if (T.team >= T.teams) return;
  for (int f = T.team; f < nf; f += T.teams) {
    FaceBox B;
    const int rows = face_box(vtx, faces, f, G, &B);
    const unsigned nbx = B.rid[0] - B.lid[0], nby = B.rid[1] - B.lid[1];
    if (rows == 0) continue;
    auto element = [&](unsigned x0, unsigned y0, unsigned z0) {
      const int x = B.lid[0] + (int)x0, y = B.lid[1] + (int)y0, z = B.lid[2] + (int)z0;
      const size_t e = ((size_t)z * G.R + y) * G.R + x;
      if (!solid[e] || shell[e]) return;
      const D3 p = {(x + 0.5) * G.eh + G.b0[0], (y + 0.5) * G.eh + G.b0[1], (z + 0.5) * G.eh + G.b0[2]};
      const double ox = outside(p.x, B.lo[0], B.hi[0]), oy = outside(p.y, B.lo[1], B.hi[1]),
                   oz = outside(p.z, B.lo[2], B.hi[2]);
      if (ox * ox + (oy * oy + oz * oz) > B.lim) return;
      const D3 d = sub(p, closest_on_triangle(p, B.a, B.b, B.c));
      if (dot(d, d) < sh2) shell[e] = 1;
    };
    const unsigned long long n = (unsigned long long)rows * nbx;
    const unsigned step = T.size * 256, start = T.rank * 256 + threadIdx.x;
    if (n < (1ull << 31)) {  // 32-bit divisions
      for (unsigned k = start; k < (unsigned)n; k += step) {
        const unsigned r = k / nbx, z = r / nby;
        element(k - r * nbx, r - z * nby, z);
      }
    } else {
      for (unsigned long long k = start; k < n; k += step) {
        const unsigned r = (unsigned)(k / nbx), z = r / nby;
        element((unsigned)(k - (unsigned long long)r * nbx), r - z * nby, z);
      }
    }
  }
}

// a warp per row: user's solid bytes (any non-zero is solid) to states, and states to shell bytes
template <bool IN>
__global__ void k_shell_bytes(uint8_t* __restrict__ user, uint8_t* __restrict__ state, int R, int pitch) {
  const int lane = threadIdx.x & 31;
  for (long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32; row < (long long)R * R;
       row += (long long)gridDim.x * blockDim.x / 32) {
    uint8_t *u = user + row * R, *s = state + row * pitch;
    if (IN)
      for (int x = lane; x < pitch; x += 32) s[x] = x < R && u[x] ? 1 : 0;
    else
      for (int x = lane; x < R; x += 32) u[x] = s[x] >> 1;
  }
}

constexpr int kNormalTile = 128;

// outwardNormal's rule for the closest point q of face bf to p: the supporting
// plane's vector (a - c) x (b - c) of CGAL's plane through three points when
// |q - p| < 1e-6, else (q - p) / |q - p| oriented along it
__device__ void emit_normal(const float* __restrict__ vtx, const int* __restrict__ faces, int bf, D3 bq, D3 p,
                            double* __restrict__ out) {
  const D3 ba = vertex(vtx, faces[3 * bf]), bb = vertex(vtx, faces[3 * bf + 1]), bc = vertex(vtx, faces[3 * bf + 2]);
  const D3 tn = cross(sub(ba, bc), sub(bb, bc));
  const D3 pq = sub(bq, p);
  double len = sqrt(dot(pq, pq));
  D3 n;
  if (len < 1e-6) {
    n = unit(tn);
  } else {
    if (dot(pq, tn) < 0.0) len = -len;
    n = {pq.x / len, pq.y / len, pq.z / len};
  }
  out[0] = n.x;
  out[1] = n.y;
  out[2] = n.z;
}

// one thread per point; faces staged through shared memory a tile at a time
__global__ void __launch_bounds__(kNormalTile) k_normals(const float* __restrict__ vtx, const int* __restrict__ faces,
                                                         int nf, const double* __restrict__ pts, int np,
                                                         double* __restrict__ nrm) {
  __shared__ double tri[kNormalTile][9];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  D3 p = {0.0, 0.0, 0.0};
  if (i < np) p = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
  double best = INFINITY;
  D3 bq = p;
  int bf = 0;  // face 0 when no distance compares (degenerate faces only)
  for (int t0 = 0; t0 < nf; t0 += kNormalTile) {
    __syncthreads();
    const int f = t0 + threadIdx.x;
    if (f < nf) {
      const D3 a = vertex(vtx, faces[3 * f]), b = vertex(vtx, faces[3 * f + 1]), c = vertex(vtx, faces[3 * f + 2]);
      tri[threadIdx.x][0] = a.x, tri[threadIdx.x][1] = a.y, tri[threadIdx.x][2] = a.z;
      tri[threadIdx.x][3] = b.x, tri[threadIdx.x][4] = b.y, tri[threadIdx.x][5] = b.z;
      tri[threadIdx.x][6] = c.x, tri[threadIdx.x][7] = c.y, tri[threadIdx.x][8] = c.z;
    }
    __syncthreads();
    const int nt = min(kNormalTile, nf - t0);
    if (i < np)
      for (int t = 0; t < nt; t++) {
        const double* q = tri[t];
        const D3 a = {q[0], q[1], q[2]}, b = {q[3], q[4], q[5]}, c = {q[6], q[7], q[8]};
        const D3 cq = closest_on_triangle(p, a, b, c);
        const D3 d = sub(cq, p);
        const double d2 = dot(d, d);
        if (d2 < best) {
          best = d2;
          bq = cq;
          bf = t0 + t;
        }
      }
  }
  if (i >= np) return;
  emit_normal(vtx, faces, bf, bq, p, nrm + 3 * i);
}

// A uniform grid over the mesh's bounding box: cell (x, y, z) lists the faces
// whose bounding box overlaps it (start[cell] .. start[cell + 1] in items).
struct FaceGrid {
  double lo[3], cs[3];
  int g[3];
  double slack;  // absolute slack on distances to cell boundaries (cell-index rounding)
  const int* start;
  const int* items;
};

__device__ __forceinline__ int cell_of(double x, double lo, double cs, int g) {
  const double q = floor((x - lo) / cs);
  return !(q >= 0.0) ? 0 : (q >= (double)g ? g - 1 : (int)q);
}

__device__ __forceinline__ void face_cells(const FaceGrid& G, D3 a, D3 b, D3 c, int* c0, int* c1) {
  const double lo[3] = {fmin(fmin(a.x, b.x), c.x), fmin(fmin(a.y, b.y), c.y), fmin(fmin(a.z, b.z), c.z)};
  const double hi[3] = {fmax(fmax(a.x, b.x), c.x), fmax(fmax(a.y, b.y), c.y), fmax(fmax(a.z, b.z), c.z)};
  for (int j = 0; j < 3; j++) {
    c0[j] = cell_of(lo[j], G.lo[j], G.cs[j], G.g[j]);
    c1[j] = cell_of(hi[j], G.lo[j], G.cs[j], G.g[j]);
  }
}

// FILL false: count the faces of every cell; true: write them (counts: the next item per cell)
template <bool FILL>
__global__ void k_bin_faces(const float* __restrict__ vtx, const int* __restrict__ faces, int nf, FaceGrid G,
                            int* __restrict__ counts, int* __restrict__ items) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  int c0[3], c1[3];
  face_cells(G, vertex(vtx, faces[3 * f]), vertex(vtx, faces[3 * f + 1]), vertex(vtx, faces[3 * f + 2]), c0, c1);
  for (int z = c0[2]; z <= c1[2]; z++)
    for (int y = c0[1]; y <= c1[1]; y++)
      for (int x = c0[0]; x <= c1[0]; x++) {
        const long long cell = x + (long long)G.g[0] * (y + (long long)G.g[1] * z);
        const int slot = atomicAdd(&counts[cell], 1);
        if (FILL) items[slot] = f;
      }
}

// One warp per point: cells in rings of growing Chebyshev radius around the
// point's cell, until no face outside the visited block can come as close as
// the best so far (the faces that could still tie or win lie within the
// bound); the best is the lexicographic minimum of (squared distance, face
// index), the brute-force scan's answer.  The cells of a row are consecutive,
// so a ring is a list of runs of items: each lane fetches one run's bounds, and
// all lanes share out the runs' faces.  Bound by the chain of distances of a
// point: a thread per point ran 128 CTAs with tens of FP64 distances one after
// the other (16384 points, 262144 faces: 1379 us), the warp takes 32 at once
// (177 us).
__global__ void __launch_bounds__(128) k_normals_grid(const float* __restrict__ vtx, const int* __restrict__ faces,
                                                      FaceGrid G, const double* __restrict__ pts, int np,
                                                      double* __restrict__ nrm) {
  const int i = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) / 32), lane = threadIdx.x & 31;
  if (i >= np) return;
  const D3 p = {pts[3 * (size_t)i], pts[3 * (size_t)i + 1], pts[3 * (size_t)i + 2]};
  const double pc[3] = {p.x, p.y, p.z};
  int c[3];
  for (int j = 0; j < 3; j++) c[j] = cell_of(pc[j], G.lo[j], G.cs[j], G.g[j]);
  double best = INFINITY;
  int bf = 0x7fffffff;
  const int rmax = max(G.g[0], max(G.g[1], G.g[2]));
  for (int r = 0; r <= rmax; r++) {
    const int z0 = max(c[2] - r, 0), z1 = min(c[2] + r, G.g[2] - 1);
    const int y0 = max(c[1] - r, 0), y1 = min(c[1] + r, G.g[1] - 1);
    const int x0 = max(c[0] - r, 0), x1 = min(c[0] + r, G.g[0] - 1);
    const int ny = y1 - y0 + 1, nrun = 2 * ny * (z1 - z0 + 1);
    for (int s0 = 0; s0 < nrun; s0 += 32) {
      // run s: row s / 2 of the block, whole on the ring's faces (s even), else its two end cells
      int from = 0, len = 0;
      if (s0 + lane < nrun) {
        const int side = (s0 + lane) & 1, y = y0 + ((s0 + lane) >> 1) % ny, z = z0 + ((s0 + lane) >> 1) / ny;
        const bool whole = z == c[2] - r || z == c[2] + r || y == c[1] - r || y == c[1] + r;
        const int xa = whole ? x0 : (side ? c[0] + r : c[0] - r), xb = whole ? x1 : xa;
        if ((!whole || !side) && xa >= 0 && xb < G.g[0]) {
          const long long row = (long long)G.g[0] * (y + (long long)G.g[1] * z);
          from = G.start[row + xa];
          len = G.start[row + xb + 1] - from;
        }
      }
      int end = len;  // inclusive prefix sum: the runs laid end to end
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      const int total = __shfl_sync(0xffffffffu, end, 31);
      for (int k0 = 0; k0 < total; k0 += 32) {
        const int k = k0 + lane;
        int run = 0;  // first run that ends after k
        for (int o = 16; o > 0; o >>= 1) {
          const int v = __shfl_sync(0xffffffffu, end, run + o - 1);
          if (v <= k) run += o;
        }
        const int re = __shfl_sync(0xffffffffu, end, run), rl = __shfl_sync(0xffffffffu, len, run);
        const int rf = __shfl_sync(0xffffffffu, from, run);
        if (k < total) {
          const int f = G.items[rf + (k - (re - rl))];
          const D3 d = sub(closest_on_triangle(p, vertex(vtx, faces[3 * f]), vertex(vtx, faces[3 * f + 1]),
                                               vertex(vtx, faces[3 * f + 2])), p);
          const double d2 = dot(d, d);
          if (d2 < best || (d2 == best && f < bf)) {
            best = d2;
            bf = f;
          }
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double d2 = __shfl_xor_sync(0xffffffffu, best, o);
      const int f = __shfl_xor_sync(0xffffffffu, bf, o);
      if (d2 < best || (d2 == best && f < bf)) {
        best = d2;
        bf = f;
      }
    }
    // lower bound on the distance from p to cells outside the block: the
    // nearest of the slabs of the grid beyond each block face
    const int b0[3] = {x0, y0, z0}, b1[3] = {x1, y1, z1};
    double bound = INFINITY;
    for (int a = 0; a < 3; a++)
      for (int side = 0; side < 2; side++) {
        if (side == 0 ? b0[a] == 0 : b1[a] == G.g[a] - 1) continue;
        double d2 = 0;
        for (int j = 0; j < 3; j++) {
          double lo = G.lo[j], hi = G.lo[j] + G.g[j] * G.cs[j];
          if (j == a) {
            if (side == 0) hi = G.lo[j] + b0[j] * G.cs[j];
            else lo = G.lo[j] + (b1[j] + 1) * G.cs[j];
          }
          const double e = pc[j] < lo ? lo - pc[j] : (pc[j] > hi ? pc[j] - hi : 0.0);
          d2 += e * e;
        }
        bound = fmin(bound, sqrt(d2));
      }
    if (bound == INFINITY) break;  // the block covers the grid
    const double bd = bound - G.slack;
    if (bd > 0.0 && best < bd * bd * (1.0 - 1e-12)) break;
  }
  if (lane != 0) return;
  D3 bq = p;  // face 0 when no distance compares (degenerate faces only)
  if (bf != 0x7fffffff)
    bq = closest_on_triangle(p, vertex(vtx, faces[3 * bf]), vertex(vtx, faces[3 * bf + 1]), vertex(vtx, faces[3 * bf + 2]));
  emit_normal(vtx, faces, bf == 0x7fffffff ? 0 : bf, bq, p, nrm + 3 * (size_t)i);
}

// Bounding box of the faces' vertices, {lo, hi} of each CTA (fminf and fmaxf
// pass over NaN).  On the host, three random reads a face through the whole
// list took 9 ms for 262144 faces.
__global__ void __launch_bounds__(256) k_face_bounds(const float* __restrict__ vtx, const int* __restrict__ faces,
                                                     long long nv, float* __restrict__ out) {
  float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < nv; k += gridDim.x * 256ll)
    for (int a = 0; a < 3; a++) {
      const float x = vtx[3 * (size_t)faces[k] + a];
      v[a] = fminf(v[a], x);
      v[3 + a] = fmaxf(v[3 + a], x);
    }
  __shared__ float part[8][6];
  for (int a = 0; a < 6; a++) {
    for (int o = 16; o > 0; o >>= 1) {
      const float x = __shfl_xor_sync(0xffffffffu, v[a], o);
      v[a] = a < 3 ? fminf(v[a], x) : fmaxf(v[a], x);
    }
    if ((threadIdx.x & 31) == 0) part[threadIdx.x / 32][a] = v[a];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    float x = part[0][threadIdx.x];
    for (int w = 1; w < 8; w++)
      x = threadIdx.x < 3 ? fminf(x, part[w][threadIdx.x]) : fmaxf(x, part[w][threadIdx.x]);
    out[6 * blockIdx.x + threadIdx.x] = x;
  }
}

// Exclusive scan of the cells' counts in two launches: the sums of 1024 cells,
// then every CTA adds up the sums before its own.  start saturates at
// INT32_MAX; the last CTA leaves the total.
__device__ __forceinline__ long long cta_sum(long long v, long long* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x / 32] = v;
  __syncthreads();
  v = 0;
  for (int w = 0; w < (int)blockDim.x / 32; w++) v += sh[w];
  __syncthreads();
  return v;
}

__global__ void __launch_bounds__(1024) k_cell_sums(const int* __restrict__ counts, long long ncell,
                                                    long long* __restrict__ sums) {
  __shared__ long long sh[32];
  const long long c = blockIdx.x * 1024ll + threadIdx.x;
  const long long s = cta_sum(c < ncell ? counts[c] : 0, sh);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

// the counts become cursors: the next item of every cell
__global__ void __launch_bounds__(1024) k_cell_start(int* __restrict__ counts, long long ncell,
                                                     const long long* __restrict__ sums, int* __restrict__ start,
                                                     long long* __restrict__ total) {
  __shared__ long long sh[32], wsum[32];
  long long base = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024) base += sums[b];
  base = cta_sum(base, sh);
  const long long c = blockIdx.x * 1024ll + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  const long long n = c < ncell ? counts[c] : 0;
  long long v = n;
  for (int o = 1; o < 32; o <<= 1) {
    const long long x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += x;
  }
  if (lane == 31) wsum[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; w++) base += wsum[w];
  if (c < ncell) {
    counts[c] = start[c] = (int)min(base + v - n, 0x7fffffffll);
    if (c == ncell - 1) {
      start[ncell] = (int)min(base + v, 0x7fffffffll);
      *total = base + v;
    }
  }
}

__device__ bool region_contains(const rso_region& r, D3 p) {
  const double* q = r.p;
  bool in = false;
  switch (r.kind) {
    case RSO_REGION_SPHERE: {
      const double dx = p.x - q[0], dy = p.y - q[1], dz = p.z - q[2];
      const double s = dx * dx + dy * dy + dz * dz, r2 = q[3] * q[3];
      in = s < r2 || (r.closed && (s - r2) < 1e-8);
      break;
    }
    case RSO_REGION_BOX: {
      const bool inner = q[0] < p.x && p.x < q[3] && q[1] < p.y && p.y < q[4] && q[2] < p.z && p.z < q[5];
      const bool closed_in = q[0] <= p.x && p.x <= q[3] && q[1] <= p.y && p.y <= q[4] && q[2] <= p.z && p.z <= q[5];
      in = inner || (r.closed && closed_in);
      break;
    }
    case RSO_REGION_HALFSPACE: {
      const double s = q[0] * p.x + q[1] * p.y + q[2] * p.z + q[3];
      in = s > 0.0 || (r.closed && s == 0.0);
      break;
    }
    case RSO_REGION_CYLINDER: {
      D3 z = {q[4], q[5], q[6]};
      const double height = sqrt(dot(z, z));
      z = {z.x / height, z.y / height, z.z / height};
      const D3 v = sub(p, D3{q[0], q[1], q[2]});
      const double proj = dot(v, z);
      if (proj > height || proj < 0.0) return false;
      const D3 cr = cross(v, z);
      return !(sqrt(dot(cr, cr)) >= q[3]);
    }
    default:
      return false;
  }
  return in != (r.complement != 0);
}

// 2^shift lanes per row of nodes: the row's y and z are divided out once, not per
// node (257^3 nodes: 113 -> 68 us); a warp, or as many lanes as a shorter row has
// nodes, up to the next power of two
__global__ void k_region_mask(const rso_region* __restrict__ regions, int nr, double ox, double oy, double oz,
                              double h, int nx, int ny, long long rows, int shift, uint8_t* __restrict__ mask) {
  const int lanes = 1 << shift;
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> shift; r < rows;
       r += (long long)gridDim.x * blockDim.x >> shift) {
    const int y = (int)(r % ny), z = (int)(r / ny);
    uint8_t* row = mask + r * nx;
    for (long long x = threadIdx.x & (lanes - 1); x < nx; x += lanes) {
      const D3 p = {ox + (int)x * h, oy + y * h, oz + z * h};
      bool in = false;
      for (int k = 0; k < nr; k++) in |= region_contains(regions[k], p);
      row[x] = in ? 1 : 0;
    }
  }
}

__device__ double field_norm(const rso_field& f, D3 p) {
  const double* q = f.norm_p;
  switch (f.norm_kind) {
    case RSO_FIELD_CONSTANT:
      return q[0];
    case RSO_FIELD_RADIAL: {
      const D3 d = sub(D3{q[0], q[1], q[2]}, p);
      const double radi = sqrt(dot(d, d));
      return q[3] * exp(-pow(radi, q[4] * 2));
    }
    case RSO_FIELD_TWIST: {
      const D3 s = {q[0], q[1], q[2]};
      const D3 ax = unit(sub(D3{q[3], q[4], q[5]}, s));
      const D3 cr = cross(sub(p, s), ax);
      return sqrt(dot(cr, cr)) * q[6];
    }
    default:
      return 0.0;
  }
}

__device__ D3 field_dir(const rso_field& f, D3 p) {
  const double* q = f.dir_p;
  switch (f.dir_kind) {
    case RSO_FIELD_CONSTANT:
      return unit(D3{q[0], q[1], q[2]});
    case RSO_FIELD_RADIAL:
      return unit(sub(D3{q[0], q[1], q[2]}, p));
    case RSO_FIELD_TWIST: {
      const D3 s = {q[0], q[1], q[2]};
      return unit(cross(sub(p, s), sub(D3{q[3], q[4], q[5]}, s)));
    }
    default:
      return {0.0, 0.0, 0.0};
  }
}

__global__ void k_region_field(const rso_field* __restrict__ fields, int nfld, const double* __restrict__ pts,
                               int np, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const D3 p = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
  D3 s = {0.0, 0.0, 0.0};
  for (int k = 0; k < nfld; k++) {
    if (!region_contains(fields[k].region, p)) continue;
    const double m = field_norm(fields[k], p);
    const D3 d = field_dir(fields[k], p);
    s = {s.x + m * d.x, s.y + m * d.y, s.z + m * d.z};
  }
  out[3 * i] = s.x;
  out[3 * i + 1] = s.y;
  out[3 * i + 2] = s.z;
}

constexpr int kCacheDevices = 64;
constexpr size_t kCacheCap = size_t(1) << 30;
struct BlockCache {
  std::mutex m;
  std::vector<std::pair<size_t, void*>> blocks[kCacheDevices];
  size_t held[kCacheDevices] = {};
};
BlockCache g_blocks;

}  // namespace

cudaError_t block_get(int dev, size_t bytes, void** p, size_t* cls) {
  size_t c = 256;
  while (c < bytes) c <<= 1;
  *cls = c;
  if (dev >= 0 && dev < kCacheDevices) {
    std::lock_guard<std::mutex> lk(g_blocks.m);
    auto& v = g_blocks.blocks[dev];
    for (size_t i = 0; i < v.size(); i++)
      if (v[i].first == c) {
        *p = v[i].second;
        g_blocks.held[dev] -= c;
        v.erase(v.begin() + i);
        return cudaSuccess;
      }
  }
  const cudaError_t e = cudaMalloc(p, c);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();  // the blocks of other sizes may be what is missing
  blocks_release(dev);
  return cudaMalloc(p, c);
}

// frees the cached blocks of a device, or of all (dev < 0)
void blocks_release(int dev) {
  for (int k = 0; k < kCacheDevices; k++) {
    if (dev >= 0 && k != dev) continue;
    std::vector<std::pair<size_t, void*>> v;
    {
      std::lock_guard<std::mutex> lk(g_blocks.m);
      v.swap(g_blocks.blocks[k]);
      g_blocks.held[k] = 0;
    }
    for (const auto& b : v) cudaFree(b.second);
  }
}

void block_put(int dev, size_t cls, void* p) {
  if (dev >= 0 && dev < kCacheDevices) {
    std::lock_guard<std::mutex> lk(g_blocks.m);
    if (g_blocks.held[dev] + cls <= kCacheCap) try {
        g_blocks.blocks[dev].push_back({cls, p});
        g_blocks.held[dev] += cls;
        return;
      } catch (const std::bad_alloc&) {  // no room in the list: freed
      }
  }
  cudaFree(p);
}

// Copies of tens of megabytes into ordinary host memory.  The driver's copy
// moves them through its own staging buffer on one core, which also takes the
// page faults of a destination that was never touched: 2.2 ms for 17 MB, where
// the transfer needs 0.3 ms (four 17 MB results of the mesh input, 19 -> 13 ms
// with the computations between them).  Here pieces go through a pinned ring, and a few
// threads carry them on to the destination, each piece's slot being refilled
// as soon as it is empty.  The ring (8 MB) is made on first use and kept until
// rso_release_mesh_memory; a call that finds it in use, or any failure to get threads or pinned memory,
// takes the driver's copy.  Starting the threads takes 0.1 to 0.4 ms, more or less
// from call to call, so copies below kRingLeast take the driver's too (region masks,
// medians of 25 calls: 5.3 MB 0.95 and 0.78 ms through the ring, 0.77 and 0.87 by
// the driver; 9.2 MB 1.00 and 1.23, 39.6 MB 2.5 and 8.9).
namespace {
constexpr size_t kPiece = size_t(1) << 20, kRingLeast = 8 * kPiece;
constexpr int kSlots = 8, kCarriers = 4;
struct HostRing {
  std::mutex m;
  char* slots = nullptr;
};
HostRing g_ring;

struct Carry {
  char* dst;
  const char* src;
  size_t n;
  int dev;
  cudaEvent_t landed[kSlots];
  std::atomic<int> failed{0};
  cudaError_t fetch(size_t piece) {  // piece into its slot, after everything before it on the default stream
    const int slot = (int)(piece % kSlots);
    const size_t o = piece * kPiece;
    cudaError_t e = cudaMemcpyAsync(g_ring.slots + slot * kPiece, src + o, std::min(kPiece, n - o),
                                    cudaMemcpyDeviceToHost, 0);
    if (e == cudaSuccess) e = cudaEventRecord(landed[slot], 0);
    return e;
  }
  // carrier t takes the pieces of slots t, t + kCarriers, ..: no other carrier touches them
  void run(int t, int carriers) {
    cudaError_t e = cudaSetDevice(dev);
    const size_t np = (n + kPiece - 1) / kPiece;
    for (size_t k = t; k < np && e == cudaSuccess; k++) {
      const int slot = (int)(k % kSlots);
      if (slot % carriers != t) continue;
      e = cudaEventSynchronize(landed[slot]);
      if (e != cudaSuccess) break;
      std::memcpy(dst + k * kPiece, g_ring.slots + slot * kPiece, std::min(kPiece, n - k * kPiece));
      if (k + kSlots < np) e = fetch(k + kSlots);
    }
    if (e != cudaSuccess) failed = (int)e;
  }
};
}  // namespace

// frees the ring, after the call that uses it
static void ring_release() {
  std::lock_guard<std::mutex> lk(g_ring.m);
  if (g_ring.slots) cudaFreeHost(g_ring.slots);
  g_ring.slots = nullptr;
}

cudaError_t copy_to_host(void* dst, const void* src, size_t n) {
  cudaPointerAttributes at{};
  std::unique_lock<std::mutex> lk(g_ring.m, std::defer_lock);
  if (n < kRingLeast || cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type != cudaMemoryTypeUnregistered ||
      !lk.try_lock() ||
      (!g_ring.slots && cudaHostAlloc((void**)&g_ring.slots, kSlots * kPiece, cudaHostAllocPortable) != cudaSuccess)) {
    cudaGetLastError();
    return cudaMemcpy(dst, src, n, cudaMemcpyDeviceToHost);
  }
  Carry c;
  c.dst = (char*)dst, c.src = (const char*)src, c.n = n;
  cudaError_t e = cudaGetDevice(&c.dev);
  int made = 0;
  for (; made < kSlots && e == cudaSuccess; made++) {
    e = cudaEventCreateWithFlags(&c.landed[made], cudaEventDisableTiming);
    if (e != cudaSuccess) break;
  }
  for (size_t k = 0; k < (size_t)kSlots && k * kPiece < n && e == cudaSuccess; k++) e = c.fetch(k);
  if (e == cudaSuccess) {
    std::thread helper[kCarriers - 1];
    int helpers = 0;
    try {  // std::thread throws when the system has no thread, or no memory, to give
      for (; helpers < kCarriers - 1; helpers++) helper[helpers] = std::thread(&Carry::run, &c, helpers + 1, kCarriers);
    } catch (...) {
    }
    c.run(0, kCarriers);
    for (int t = helpers + 1; t < kCarriers; t++) c.run(t, kCarriers);  // those without a thread of their own
    for (int t = 0; t < helpers; t++) helper[t].join();
    e = (cudaError_t)c.failed.load();
  }
  if (e != cudaSuccess) cudaStreamSynchronize(0);  // no copy into the ring outlives the call
  for (int i = 0; i < made; i++) cudaEventDestroy(c.landed[i]);
  return e;
}

namespace {

static_assert(sizeof(rso_region) == 80 && sizeof(rso_field) == 192, "rso_region / rso_field layout is part of the ABI");

bool faces_valid(const int* faces, int nf, int nv) {
  for (long long k = 0; k < 3LL * nf; k++)
    if (faces[k] < 0 || faces[k] >= nv) return false;
  return true;
}

bool regions_valid(const rso_region* r, int n) {
  for (int k = 0; k < n; k++)
    if (r[k].kind < RSO_REGION_SPHERE || r[k].kind > RSO_REGION_CYLINDER) return false;
  return true;
}

}  // namespace
}  // namespace rso

using namespace rso;

extern "C" rso_status rso_release_mesh_memory(void) {
  blocks_release(-1);
  ring_release();
  return RSO_OK;
}

extern "C" rso_status rso_shell_elements(const float* vertices_host, int n_vertices, const int* faces_host,
                                         int n_faces, const float* box_host, int resolution, double shell_width,
                                         const uint8_t* solid_host, uint8_t* shell_host) {
  if (!vertices_host || !faces_host || !box_host || !solid_host || !shell_host || n_vertices < 3 || n_faces < 1 ||
      resolution < 1 || resolution > 2048 || !(shell_width >= 0) || !faces_valid(faces_host, n_faces, n_vertices))
    return RSO_ERR_INVALID_ARG;
  const int R = resolution;
  const long long nvox = (long long)R * R * R;
  // element edge as the reference forms it: an FP32 difference over an FP32 quotient
  const double eh = (double)((box_host[3] - box_host[0]) / (float)R);
  const double wshell = shell_width * eh;
  Scratch s;
  const float* dv = s.upload(vertices_host, 3 * (size_t)n_vertices);
  const int* df = s.upload(faces_host, 3 * (size_t)n_faces);
  uint8_t* dsolid = s.upload(solid_host, (size_t)nvox);
  uint8_t* dshell = dsolid;  // many faces: the shell's bytes take the solid ones' place
  ShellGrid G{{box_host[0], box_host[1], box_host[2]}, eh, wshell, R, (R + 7) & ~7};
  if (n_faces < (R < 32 ? kShellFewSmall : kShellFew)) {
    dshell = s.alloc<uint8_t>((size_t)nvox);
    if (s.err == cudaSuccess) s.err = cudaMemset(dshell, 0, (size_t)nvox);
    if (s.err == cudaSuccess && wshell > 0) {
      k_shell_few<<<std::max(kShellCtas, n_faces), 256>>>(dv, df, n_faces, G, dsolid, dshell);
      note_launch();
      s.err = cudaGetLastError();
    }
    if (s.err == cudaSuccess) s.err = copy_to_host(shell_host, dshell, (size_t)nvox);
    return s.err == cudaSuccess ? RSO_OK : RSO_ERR_CUDA;
  }
  uint8_t* state = s.alloc<uint8_t>((size_t)R * R * G.pitch);
  int* big = s.alloc<int>(1 + (size_t)n_faces);
  if (s.err == cudaSuccess) s.err = cudaMemset(big, 0, sizeof(int));
  if (s.err == cudaSuccess) {
    const unsigned rows = (unsigned)std::min(((long long)R * R + 7) / 8, 148LL * 64);
    k_shell_bytes<true><<<rows, 256>>>(dshell, state, R, G.pitch);
    note_launch();
    if (wshell > 0) {
      int stride = (int)(0.618 * n_faces) + 1;
      while (std::gcd(stride, n_faces) != 1) stride++;
      k_shell<<<(unsigned)cdiv(n_faces, 4), 128>>>(dv, df, n_faces, stride, G, state, big);
      note_launch();
      k_shell_big<<<kShellCtas, 128>>>(dv, df, G, state, big);
      note_launch();
    }
    k_shell_bytes<false><<<rows, 256>>>(dshell, state, R, G.pitch);
    note_launch();
    s.err = cudaGetLastError();
  }
  if (s.err == cudaSuccess) s.err = copy_to_host(shell_host, dshell, (size_t)nvox);
  return s.err == cudaSuccess ? RSO_OK : RSO_ERR_CUDA;
}

extern "C" rso_status rso_mesh_normals(const float* vertices_host, int n_vertices, const int* faces_host, int n_faces,
                                       const double* points_host, int n_points, double* normals_host) {
  if (!vertices_host || !faces_host || n_vertices < 3 || n_faces < 1 || n_points < 0 ||
      (n_points > 0 && (!points_host || !normals_host)) || !faces_valid(faces_host, n_faces, n_vertices))
    return RSO_ERR_INVALID_ARG;
  if (n_points == 0) return RSO_OK;
  Scratch s;
  const float* dv = s.upload(vertices_host, 3 * (size_t)n_vertices);
  const int* df = s.upload(faces_host, 3 * (size_t)n_faces);
  const double* dp = s.upload(points_host, 3 * (size_t)n_points);
  double* dn = s.alloc<double>(3 * (size_t)n_points);
  // meshes of a few hundred faces or more: bin the faces on a uniform grid
  // of about two faces per cell and search rings of cells around each point
  bool grid = false;
  FaceGrid G{};
  if (s.err == cudaSuccess && n_faces >= 256) {
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    constexpr int kParts = 148;
    float part[6 * kParts];
    float* dpart = s.alloc<float>(6 * kParts);
    if (s.err == cudaSuccess) {
      k_face_bounds<<<kParts, 256>>>(dv, df, 3LL * n_faces, dpart);
      note_launch();
      s.err = cudaGetLastError();
    }
    if (s.err == cudaSuccess) s.err = cudaMemcpy(part, dpart, sizeof(part), cudaMemcpyDeviceToHost);
    for (int k = 0; k < kParts && s.err == cudaSuccess; k++)
      for (int a = 0; a < 3; a++) {
        lo[a] = std::fmin(lo[a], (double)part[6 * k + a]);
        hi[a] = std::fmax(hi[a], (double)part[6 * k + 3 + a]);
      }
    double ext[3], emax = 0, mag = 0;
    for (int a = 0; a < 3; a++) {
      ext[a] = hi[a] - lo[a];
      emax = std::fmax(emax, ext[a]);
      mag = std::fmax(mag, std::fmax(std::fabs(lo[a]), std::fabs(hi[a])));
    }
    if (s.err == cudaSuccess && emax > 0 && std::isfinite(emax) && std::isfinite(mag)) {
      const double target = std::min(std::max(n_faces / 2.0, 1.0), (double)(1 << 21));
      double vol = 1;
      for (int a = 0; a < 3; a++) vol *= std::fmax(ext[a], 1e-3 * emax);
      const double cs = std::cbrt(vol / target);
      long long ncell = 1;
      double csmin = INFINITY;
      for (int a = 0; a < 3; a++) {
        G.g[a] = (int)std::min(std::max(std::ceil(ext[a] / cs), 1.0), 1024.0);
        G.cs[a] = ext[a] > 0 ? ext[a] / G.g[a] : cs;
        G.lo[a] = lo[a];
        ncell *= G.g[a];
        csmin = std::fmin(csmin, G.cs[a]);
      }
      G.slack = 1e-9 * csmin + 1e-14 * mag;
      int* counts = s.alloc<int>((size_t)ncell);
      if (s.err == cudaSuccess) s.err = cudaMemset(counts, 0, sizeof(int) * ncell);
      if (s.err == cudaSuccess) {
        k_bin_faces<false><<<cdiv(n_faces, 256), 256>>>(dv, df, n_faces, G, counts, nullptr);
        note_launch();
        s.err = cudaGetLastError();
      }
      const int nsum = (int)cdiv(ncell, 1024);
      long long* sums = s.alloc<long long>((size_t)nsum + 1);  // + the total
      int* start = s.alloc<int>((size_t)ncell + 1);
      long long total = 0;
      if (s.err == cudaSuccess) {
        k_cell_sums<<<nsum, 1024>>>(counts, ncell, sums);
        note_launch();
        k_cell_start<<<nsum, 1024>>>(counts, ncell, sums, start, sums + nsum);
        note_launch();
        s.err = cudaMemcpy(&total, sums + nsum, sizeof(total), cudaMemcpyDeviceToHost);
      }
      if (s.err == cudaSuccess && total <= (1LL << 25)) {
        int* items = s.alloc<int>((size_t)std::max(total, 1LL));
        if (s.err == cudaSuccess) {
          G.start = start;
          G.items = items;
          k_bin_faces<true><<<cdiv(n_faces, 256), 256>>>(dv, df, n_faces, G, counts, items);
          note_launch();
          s.err = cudaGetLastError();
          grid = s.err == cudaSuccess;
        }
      }
    }
  }
  if (s.err == cudaSuccess && grid) {
    k_normals_grid<<<(unsigned)cdiv((long long)n_points, 4), 128>>>(dv, df, G, dp, n_points, dn);
    note_launch();
    s.err = cudaGetLastError();
  } else if (s.err == cudaSuccess) {
    k_normals<<<cdiv(n_points, kNormalTile), kNormalTile>>>(dv, df, n_faces, dp, n_points, dn);
    note_launch();
    s.err = cudaGetLastError();
  }
  if (s.err == cudaSuccess)
    s.err = cudaMemcpy(normals_host, dn, sizeof(double) * 3 * (size_t)n_points, cudaMemcpyDeviceToHost);
  return s.err == cudaSuccess ? RSO_OK : RSO_ERR_CUDA;
}

extern "C" rso_status rso_region_mask(const rso_region* regions_host, int n_regions, const double* origin_host,
                                      double h, int nx, int ny, int nz, uint8_t* mask_host) {
  if (n_regions < 0 || (n_regions > 0 && !regions_host) || !origin_host || !mask_host || nx < 1 || ny < 1 || nz < 1 ||
      !regions_valid(regions_host, n_regions))
    return RSO_ERR_INVALID_ARG;
  const long long nn = (long long)nx * ny * nz;
  Scratch s;
  const rso_region* dr = s.upload(regions_host, (size_t)n_regions);
  uint8_t* dm = s.alloc<uint8_t>((size_t)nn);
  if (s.err == cudaSuccess) {
    const long long rows = (long long)ny * nz;
    int shift = 0;
    while (shift < 5 && (1 << shift) < nx) shift++;
    const long long per = 256 >> shift;  // rows a CTA
    k_region_mask<<<(unsigned)std::min((rows + per - 1) / per, 148LL * 64), 256>>>(
        dr, n_regions, origin_host[0], origin_host[1], origin_host[2], h, nx, ny, rows, shift, dm);
    note_launch();
    s.err = cudaGetLastError();
  }
  if (s.err == cudaSuccess) s.err = copy_to_host(mask_host, dm, (size_t)nn);
  return s.err == cudaSuccess ? RSO_OK : RSO_ERR_CUDA;
}

extern "C" rso_status rso_region_field(const rso_field* fields_host, int n_fields, const double* points_host,
                                       int n_points, double* vectors_host) {
  if (n_fields < 0 || (n_fields > 0 && !fields_host) || n_points < 0 ||
      (n_points > 0 && (!points_host || !vectors_host)))
    return RSO_ERR_INVALID_ARG;
  for (int k = 0; k < n_fields; k++)
    if (!regions_valid(&fields_host[k].region, 1) || fields_host[k].norm_kind < 0 || fields_host[k].norm_kind > 2 ||
        fields_host[k].dir_kind < 0 || fields_host[k].dir_kind > 2)
      return RSO_ERR_INVALID_ARG;
  if (n_points == 0) return RSO_OK;
  Scratch s;
  const rso_field* df = s.upload(fields_host, (size_t)n_fields);
  const double* dp = s.upload(points_host, 3 * (size_t)n_points);
  double* dout = s.alloc<double>(3 * (size_t)n_points);
  if (s.err == cudaSuccess) {
    k_region_field<<<cdiv(n_points, 128), 128>>>(df, n_fields, dp, n_points, dout);
    note_launch();
    s.err = cudaGetLastError();
  }
  if (s.err == cudaSuccess)
    s.err = cudaMemcpy(vectors_host, dout, sizeof(double) * 3 * (size_t)n_points, cudaMemcpyDeviceToHost);
  return s.err == cudaSuccess ? RSO_OK : RSO_ERR_CUDA;
}
