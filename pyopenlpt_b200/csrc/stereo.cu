// Kernel family (b): stereo matching on the device.
//
// Reference: StereoMatch (src/srcSTB/StereoMatch.cpp): IDMap grid (:1413-1437),
// strip intersection (:1471-1570), point visit (:1572-1627), DFS build (:184-444),
// candidate enumeration (:449-498), back-projection (:1206-1227), quick
// triangulation gate (:1083-1141), camera selection (:1307-1411), check (:504-609).
//
// B200 mapping.
//  * Grid: one counting sort over the detections of all cameras (histogram -> scan ->
//    scatter), into cells of idmap_cell_px rows by a fraction of that in columns.  The
//    detections are renumbered by it: position G holds the coordinates, the line of sight
//    and the image lines on every camera of one detection, and a run of cells of one row is
//    a run of positions.  The paths carry positions; the candidates get the detections' ids
//    back at the end.
//  * Every detection's line of sight and its image line on every other camera are
//    computed once (same FP64 functions the reference calls on the fly, so the
//    values are bit-identical) and reused by every path that touches the point.
//  * The depth-first search over build cameras is expanded breadth-first: level k
//    holds all partial paths with k chosen cameras and the target camera of their
//    next choice.  enum_kernel finds the detections of the target camera inside the
//    path's strips that pass the back-projection test, tri_kernel applies the triangulation
//    gate to them.  Children are appended with atomics; the final candidate list is
//    sorted by ids, so append order never shows.
//  * 2D tests are decided in FP32 where the distance is clear of the tolerance by more
//    than FP32 can err, and by the reference's FP64 expressions elsewhere: the accepted set
//    is the FP64 one.
//  * The whole set of candidates (ids, e_check) is therefore identical to the
//    reference's.  Decisions that pass through acos/sin (only when the minimum
//    parallax is below 6 degrees) can differ by one ulp; those are the only
//    non-bit-exact inputs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "olpt_ctx.cuh"
#include "olpt_prune.h"
#include "olpt_scan.cuh"
#include "olpt_stereo.h"

namespace olpt {

struct SmView {
  int n_cam, m, n_active;
  int active[OLPT_MAX_CAM];
  int cell, sub;            // grid: rows of `cell` px, `sub` columns per `cell` px
  int rows[OLPT_MAX_CAM], cols[OLPT_MAX_CAM];  // in units of `cell`
  int cell_off[OLPT_MAX_CAM];                  // first cell of the camera in cstart
  int raw_off[OLPT_MAX_CAM + 1];               // detections of the cameras before it
  double Wd[OLPT_MAX_CAM], Hd[OLPT_MAX_CAM];
  const double* x[OLPT_MAX_CAM];               // the detections as found
  const double* y[OLPT_MAX_CAM];
  // by position G (camera c holds raw_off[c] .. raw_off[c + 1] - 1; detections outside the
  // image come last in their camera's range, in a cell of their own that no row reaches)
  const int* cstart;     // first position of every cell
  const int* pid;        // detection id in its camera's list
  const double2* xy;
  const float2* fxy;
  const double* los;     // x 6: line of sight
  const double* l2d;     // x n_cam x 6: image line on camera t (pt, unit, normalized unit)
  const float4* fl;      // x n_cam: (n, d) of that line, |n . p + d| = distance of p from it
  double tol2d, tol3d;
  float eps;             // FP32 error bound of a distance, without the part of |d|, for points
                         // in the image
  double tq[OLPT_MAX_CAM + 1];  // quick-gate tolerance of k lines without its angle factor
  double limit[6];
  // near-tolerance log (off when near_band == 0): 2D tests whose distance lies within
  // near_band px of tol2d are appended to near_rec
  double near_band;
  olpt_near_record* near_rec;
  unsigned long long* near_count;
  long long near_cap;
};

struct Path {
  int ids[OLPT_MAX_CAM];
  signed char cams[OLPT_MAX_CAM];
  int k;
  int target;
};

// A partial path of exactly N chosen points, as the level kernels pass it on: the
// chosen detection ids, their cameras packed 4 bits each (point i in bits 4i..4i+3)
// and the next camera.  16 bytes for N = 2 (the 30 M first-level children of a 2048^2
// frame) instead of the 48 of a full Path.
template <int N>
struct alignas(16) PathN {  // camera i in bits 4 i .. 4 i + 3 of cams
  int ids[N];
  unsigned cams;
  int target;
  __host__ __device__ int cam(int i) const { return (int)((cams >> (4 * i)) & 15u); }
};

namespace {

inline int nblk(int64_t n, int t = 256) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------- grid
__device__ __forceinline__ int cam_of(const SmView& v, int g) {
  int c = 0;
#pragma unroll
  for (int k = 1; k < OLPT_MAX_CAM; ++k)
    if (k < v.n_cam && g >= v.raw_off[k]) c = k;
  return c;
}

// Cell of every detection (IDMap::rebuild's cell, StereoMatch.cpp:1423-1437, cut into `sub`
// columns) and the cells' counts.
__global__ void bin_kernel(const __grid_constant__ SmView v, int n, int* key, int* counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cam_of(v, i), k = i - v.raw_off[c];
  const double x = v.x[c][k], y = v.y[c][k];
  const int cx = (int)floor(x / (double)v.cell), cy = (int)floor(y / (double)v.cell);
  int cell = v.rows[c] * v.cols[c] * v.sub;  // outside the image
  if (!(cx < 0 || cy < 0 || cx >= v.cols[c] || cy >= v.rows[c])) {
    const int f = (int)floor((x - (double)cx * v.cell) * v.sub / (double)v.cell);
    cell = (cy * v.cols[c] + cx) * v.sub + min(max(f, 0), v.sub - 1);
  }
  cell += v.cell_off[c];
  key[i] = cell;
  atomicAdd(&counts[cell], 1);
}

// Positions: the order inside a cell is arbitrary (no result depends on it).
__global__ void place_kernel(const __grid_constant__ SmView v, int n, const int* key, int* counts,
                             int* pid, double2* xy, float2* fxy) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cam_of(v, i), k = i - v.raw_off[c];
  const int g = v.cstart[key[i]] + atomicSub(&counts[key[i]], 1) - 1;
  const double x = v.x[c][k], y = v.y[c][k];
  pid[g] = k;
  xy[g] = make_double2(x, y);
  fxy[g] = make_float2((float)x, (float)y);
}

// ---------------------------------------------------------------- per-detection lines
// A polynomial camera with exponents 0..3 as a block's threads evaluate it: the terms'
// coefficients and, per term, the positions of its three factors in the thread's power list
// 1, x, x^2, x^3, 1, y, .. (one byte each), in shared memory.  The powers of a thread's point
// lie in shared memory too, one column a thread: indexed by the (uniform) positions they cost
// one load each, where an indexed local array went through memory.
constexpr int kLineThreads = 128;
struct PolyTab {
  double coef[6][OLPT_MAX_POLY];     // u, v, du/d0, du/d1, dv/d0, dv/d1
  uint32_t fac[6][OLPT_MAX_POLY];
  int same;                          // u and v share their monomials
  double pw[12][kLineThreads];
};

__device__ void load_poly(PolyTab& T, const CamDev& m) {
  const int n = m.n_coeff;
  if (threadIdx.x == 0) T.same = 1;
  __syncthreads();
  for (int i = threadIdx.x; i < 6 * n; i += blockDim.x) {
    const int q = i / n, k = i - q * n;
    const double* t = q == 0   ? m.ucoef + 4 * k
                      : q == 1 ? m.vcoef + 4 * k
                      : q == 2 ? m.ducoef + 4 * k
                      : q == 3 ? m.ducoef + 4 * (k + n)
                      : q == 4 ? m.dvcoef + 4 * k
                               : m.dvcoef + 4 * (k + n);
    T.coef[q][k] = t[0];
    uint32_t f = 0;
    for (int j = 0; j < 3; ++j) f |= (uint32_t)(4 * j + (int)t[1 + j]) << (8 * j);
    T.fac[q][k] = f;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x)
    if (T.fac[0][k] != T.fac[1][k] || T.fac[2][k] != T.fac[4][k] || T.fac[3][k] != T.fac[5][k])
      T.same = 0;
  __syncthreads();
}

__device__ __forceinline__ void set_powers(PolyTab& T, const double P[3]) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    T.pw[4 * j][threadIdx.x] = 1.0;
    T.pw[4 * j + 1][threadIdx.x] = P[j];
    T.pw[4 * j + 2][threadIdx.x] = poly_pow(P[j], 2.0);
    T.pw[4 * j + 3][threadIdx.x] = poly_pow(P[j], 3.0);
  }
}

// one term of polynomial q: coefficient times its three factors, in poly_project's order
__device__ __forceinline__ double term(const PolyTab& T, int q, int i) {
  const uint32_t f = T.fac[q][i];
  const int x = threadIdx.x;
  return T.coef[q][i] * T.pw[f & 255u][x] * T.pw[(f >> 8) & 255u][x] * T.pw[f >> 16][x];
}
// terms of two polynomials with the same monomial
__device__ __forceinline__ void term2(const PolyTab& T, int q, int r, int i, double& a, double& b) {
  const uint32_t f = T.fac[q][i];
  const int x = threadIdx.x;
  const double f0 = T.pw[f & 255u][x], f1 = T.pw[(f >> 8) & 255u][x], f2 = T.pw[f >> 16][x];
  a = T.coef[q][i] * f0 * f1 * f2;
  b = T.coef[r][i] * f0 * f1 * f2;
}

// poly_project at the point whose powers are set
__device__ __forceinline__ void project_set(const PolyTab& T, int n, double& u, double& v) {
  double su = 0, sv = 0;
  for (int i = 0; i < n; ++i) {
    double a, b;
    if (T.same) {
      term2(T, 0, 1, i, a, b);
    } else {
      a = term(T, 0, i);
      b = term(T, 1, i);
    }
    su += a;
    sv += b;
  }
  u = su;
  v = sv;
}

// poly_img_to_world on the table: the same operations in the same order
__device__ void newton_tab(PolyTab& T, const CamDev& m, double pu, double pv, double plane,
                           double P[3]) {
  P[0] = P[1] = P[2] = 0.5;
  const int rp = m.ref_plane, n = m.n_coeff;
  if (rp == 1) P[0] = plane;
  if (rp == 2) P[1] = plane;
  if (rp == 3) P[2] = plane;
  double err = 1.7976931348623157e308;
  int iter = 0;
  const bool same = T.same != 0;
  while (err > 1e-5 && iter < 50) {
    set_powers(T, P);
    double j00 = 0, j01 = 0, j10 = 0, j11 = 0, tu = 0, tv = 0;
    for (int i = 0; i < n; ++i) {
      double a, b, c, d, e, f;
      if (same) {
        term2(T, 2, 4, i, a, c);
        term2(T, 3, 5, i, b, d);
        term2(T, 0, 1, i, e, f);
      } else {
        a = term(T, 2, i);
        b = term(T, 3, i);
        c = term(T, 4, i);
        d = term(T, 5, i);
        e = term(T, 0, i);
        f = term(T, 1, i);
      }
      j00 += a;
      j01 += b;
      j10 += c;
      j11 += d;
      tu += e;
      tv += f;
    }
    double det = j00 * j11 - j01 * j10;
    if (fabs(det) < 1e-8) det = 1e-8;
    const double i00 = j11 / det, i01 = -j01 / det, i10 = -j10 / det, i11 = j00 / det;
    const double du = pu - tu, dv = pv - tv;
    const double dx = i00 * du + i01 * dv;
    const double dy = i10 * du + i11 * dv;
    if (rp == 1) {
      P[1] += dx;
      P[2] += dy;
    } else if (rp == 2) {
      P[0] += dx;
      P[2] += dy;
    } else {
      P[0] += dx;
      P[1] += dy;
    }
    err = sqrt(du * du + dv * dv);
    iter++;
  }
}

// Lines of sight: blockIdx.y = camera, two lanes per detection (a polynomial camera inverts
// two planes, one each).
__global__ void __launch_bounds__(kLineThreads) los_kernel(const __grid_constant__ SmView v,
                                                           const CamDev* cams, double* los) {
  __shared__ PolyTab T;
  const int c = blockIdx.y;
  const int n = v.raw_off[c + 1] - v.raw_off[c];
  if ((int64_t)blockIdx.x * (kLineThreads / 2) >= n) return;
  const CamDev& m = cams[c];
  const bool poly = m.type == CAM_POLYNOMIAL && m.pow3;
  if (poly) load_poly(T, m);
  const int k = blockIdx.x * (kLineThreads / 2) + (threadIdx.x >> 1), half = threadIdx.x & 1;
  const bool ok = k < n;
  const int g = v.raw_off[c] + (ok ? k : n - 1);
  const double2 p = v.xy[g];
  Line3 L;
  if (poly) {
    double P[3], Q[3];
    newton_tab(T, m, p.x, p.y, m.plane[half], P);
#pragma unroll
    for (int d = 0; d < 3; ++d) Q[d] = __shfl_xor_sync(0xffffffffu, P[d], 1);
    if (half) return;
    L.p[0] = P[0];
    L.p[1] = P[1];
    L.p[2] = P[2];
    unit_vector3(P, Q, L.u);
  } else {
    if (half) return;
    cam_los(m, p.x, p.y, L);
  }
  if (!ok) return;
  double* o = los + 6 * (int64_t)g;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    o[d] = L.p[d];
    o[3 + d] = L.u[d];
  }
}

// Image lines of every detection on camera t = blockIdx.y.
__global__ void __launch_bounds__(kLineThreads) lines_kernel(const __grid_constant__ SmView v,
                                                             const CamDev* cams, double* l2d,
                                                             float4* fl) {
  __shared__ PolyTab T;
  const int t = blockIdx.y;
  if (!v.active[t]) return;
  const CamDev& m = cams[t];
  const bool poly = m.type == CAM_POLYNOMIAL && m.pow3;
  if (poly) load_poly(T, m);
  const int g = blockIdx.x * kLineThreads + threadIdx.x;
  if (g >= v.raw_off[v.n_cam] || (g >= v.raw_off[t] && g < v.raw_off[t + 1])) return;
  const double* S = v.los + 6 * (int64_t)g;
  Line3 L;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    L.p[d] = S[d];
    L.u[d] = S[3 + d];
  }
  double o[4];
  if (poly) {  // los_to_line2d
    double ax, ay, bx, by;
    set_powers(T, L.p);
    project_set(T, m.n_coeff, ax, ay);
    const double B[3] = {L.p[0] + L.u[0], L.p[1] + L.u[1], L.p[2] + L.u[2]};
    set_powers(T, B);
    project_set(T, m.n_coeff, bx, by);
    const double dx = bx - ax, dy = by - ay;
    const double n = sqrt(dx * dx + dy * dy);
    o[0] = ax;
    o[1] = ay;
    o[2] = dx / n;
    o[3] = dy / n;
  } else {
    los_to_line2d(m, L, o);
  }
  double U0 = 1.0, U1 = 0.0;
  // IDMap::normalized (StereoMatch.cpp:1441-1451)
  const double n2 = o[2] * o[2] + o[3] * o[3];
  if (!(n2 <= 1e-24)) {
    const double inv = 1.0 / sqrt(n2);
    U0 = o[2] * inv;
    U1 = o[3] * inv;
  }
  const int64_t e = (int64_t)g * v.n_cam + t;
  double2* d = reinterpret_cast<double2*>(l2d + 6 * e);
  d[0] = make_double2(o[0], o[1]);
  d[1] = make_double2(o[2], o[3]);
  d[2] = make_double2(U0, U1);
  fl[e] = make_float4((float)-U1, (float)U0, (float)(U1 * o[0] - U0 * o[1]), 0.0f);
}

__device__ __forceinline__ void load_line3(const double* p, Line3& L) {
  L.p[0] = p[0];
  L.p[1] = p[1];
  L.p[2] = p[2];
  L.u[0] = p[3];
  L.u[1] = p[4];
  L.u[2] = p[5];
}

// StereoMatch::selectSecondCameraByLineLength segment length (StereoMatch.cpp:1309-1357)
__device__ double seg_len(const double* L, double W, double H) {
  const double px = L[0], py = L[1], ux = L[2], uy = L[3];
  double qx[4], qy[4];
  int n = 0;
  auto push_if = [&](double a, double b) {
    if (a >= 0.0 && a <= W && b >= 0.0 && b <= H) {
      qx[n] = a;
      qy[n] = b;
      ++n;
    }
  };
  if (fabs(ux) > 1e-12) {
    double t = (0.0 - px) / ux;
    push_if(0.0, py + t * uy);
    t = (W - 1 - px) / ux;
    push_if(W - 1, py + t * uy);
  }
  if (fabs(uy) > 1e-12) {
    double t = (0.0 - py) / uy;
    push_if(px + t * ux, 0.0);
    t = (H - 1 - py) / uy;
    push_if(px + t * ux, H - 1);
  }
  double ux2[4], uy2[4];
  int m = 0;
  for (int i = 0; i < n; ++i) {
    bool dup = false;
    for (int j = 0; j < m; ++j)
      if (fabs(ux2[j] - qx[i]) < 1e-9 && fabs(uy2[j] - qy[i]) < 1e-9) {
        dup = true;
        break;
      }
    if (!dup) {
      ux2[m] = qx[i];
      uy2[m] = qy[i];
      ++m;
    }
  }
  if (m < 2) return 0.0;
  const double dx = ux2[0] - ux2[1], dy = uy2[0] - uy2[1];
  return sqrt(dx * dx + dy * dy);
}

// seed level: one path per reference detection with its second build camera
__global__ void seed_kernel(const __grid_constant__ SmView v, int ref, PathN<1>* out, int* out_count,
                            int cap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + v.raw_off[ref];
  if (i >= v.raw_off[ref + 1]) return;
  int best = -1;
  double best_len = __longlong_as_double(0x7ff0000000000000LL);
  for (int cam = 0; cam < v.n_cam; ++cam) {
    if (!v.active[cam] || cam == ref) continue;
    const double L = seg_len(v.l2d + 6 * ((int64_t)i * v.n_cam + cam), v.Wd[cam], v.Hd[cam]);
    if (L < best_len - 1e-9) {
      best_len = L;
      best = cam;
    }
  }
  if (best < 0) return;
  int slot = atomicAdd(out_count, 1);
  if (slot >= cap) return;
  PathN<1> p;
  p.ids[0] = i;
  p.cams = (unsigned)ref;
  p.target = best;
  out[slot] = p;
}

// (I - n n^T) of one line of sight, in myMATH::triangulation's element order.
__device__ __forceinline__ void normal_terms(const double u[3], double t[9]) {
  const double nx = u[0], ny = u[1], nz = u[2];
  t[0] = 1 - nx * nx;
  t[1] = -nx * ny;
  t[2] = -nx * nz;
  t[3] = -nx * ny;
  t[4] = 1 - ny * ny;
  t[5] = -ny * nz;
  t[6] = -nx * nz;
  t[7] = -ny * nz;
  t[8] = 1 - nz * nz;
}

// Angle in degrees between two unit directions (StereoMatch.cpp:1077-1083).
__device__ __forceinline__ double pair_deg(const double a[3], const double b[3]) {
  double dot = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
  dot = fmax(-1.0, fmin(1.0, dot));
  return acos(dot) * 180.0 / M_PI;
}

// StereoMatch::calTriangulateTol (StereoMatch.cpp:1103-1126) from the min parallax.
__device__ __forceinline__ double quick_tol_from_deg(double min_deg, int k, int m, double tol3d) {
  const int kk = k > 2 ? k : 2;
  const int mm = m > 2 ? m : 2;
  const double alpha_depth = sqrt(double(mm) / double(kk));
  const double th = fmax(min_deg, 1.0);
  const double num = sin(6.0 * M_PI / 180.0);
  const double den = fmax(1e-6, sin(th * M_PI / 180.0));
  const double alpha_angle = fmax(1.0, fmin(2.0, num / den));
  return tol3d * alpha_depth * alpha_angle;
}

// One line's contribution to the triangulation error (myMATH.cpp:396-418);
// false where the reference throws (squared distance below -1e-8).
__device__ __forceinline__ bool line_error_term(const double X[3], const double p[3],
                                                const double u[3], double& e) {
  const double d0 = X[0] - p[0], d1 = X[1] - p[1], d2 = X[2] - p[2];
  const double nrm = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
  const double dt = d0 * u[0] + d1 * u[1] + d2 * u[2];
  double h = nrm * nrm - dt * dt;
  if (h < 0.0 && h >= -1e-8) {
    h = 0.0;
  } else if (h < -1e-8) {
    return false;
  } else {
    h = sqrt(h);
  }
  e += h * h;
  return true;
}

__device__ __forceinline__ double clamped_dot(const double a[3], const double b[3]) {
  const double dot = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
  return fmax(-1.0, fmin(1.0, dot));
}

// cos(6 deg): the quick-gate angle factor of calTriangulateTol is exactly 1 whenever
// the smallest pairwise parallax lies inside (6, 174) degrees.
constexpr double kCos6 = 0.99452189536827329;

// A path and the position of one of its candidates on the target camera: past all 2D tests,
// or (kEdge) so close to a tolerance that FP64 has to decide.
struct Pair {
  int path;
  unsigned g;
};
constexpr unsigned kEdge = 1u << 31;

// Slot in an append buffer for every active lane, one atomic per warp.
__device__ __forceinline__ int append_slot(int* counter) {
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(m));
  base = __shfl_sync(m, base, leader);
  return base + __popc(m & ((1u << lane) - 1u));
}

// Appends one near-tolerance 2D decision to the log (rare: only tests whose
// distance is within near_band px of the tolerance).
__device__ __noinline__ void near_append(const SmView& v, int kind, int k, int cam, int id,
                                         int other_cam, int other_id, double margin) {
  const unsigned long long slot = atomicAdd(v.near_count, 1ull);
  if ((long long)slot >= v.near_cap) return;
  olpt_near_record r;
  r.kind = kind;
  r.n_chosen = k;
  r.cam = cam;
  r.id = id;
  r.other_cam = other_cam;
  r.other_id = other_id;
  r.margin_px = margin;
  v.near_rec[slot] = r;
}

// The strip tests (IDMap::visitPointsInRowSpans) and back-projection tests
// (checkBackProjection, StereoMatch.cpp:1206-1227) of position g on camera t against a
// path's chosen points, in the reference's FP64 expressions; LOG: near-tolerance tests are
// recorded.
template <int K, bool LOG>
__device__ __noinline__ bool exact_2d(const SmView& v, const PathN<K>& P, int g) {
  const int t = P.target;
  const double tol2 = v.tol2d * v.tol2d;
  const double2 q = v.xy[g];
  bool ok = true;
  for (int i = 0; i < K; ++i) {
    const double* L = v.l2d + 6 * ((int64_t)P.ids[i] * v.n_cam + t);
    const double dx = q.x - L[0], dy = q.y - L[1];
    const double z = dy * L[4] - dx * L[5];
    ok = ok && !(z * z > tol2);
    if (LOG) {
      const double m = fabs(z) - v.tol2d;
      if (fabs(m) < v.near_band)
        near_append(v, 0, K, t, v.pid[g], P.cam(i), v.pid[P.ids[i]], m);
    }
  }
  for (int i = 0; i < K && ok; ++i) {
    const double* L = v.l2d + 6 * ((int64_t)g * v.n_cam + P.cam(i));
    const double2 c = v.xy[P.ids[i]];
    const double d0 = c.x - L[0], d1 = c.y - L[1];
    const double z = d1 * L[2] - d0 * L[3];
    ok = !(z * z > tol2);
    if (LOG) {
      const double m = fabs(z) - v.tol2d;
      if (fabs(m) < v.near_band)
        near_append(v, 1, K, t, v.pid[g], P.cam(i), v.pid[P.ids[i]], m);
    }
  }
  return ok;
}

// The search over the reference's cells, with every test in FP64: the cell ranges of
// IDMap::computeStripIntersection as a superset (row by row, cell centres within the strips
// widened by a cell's extent and 0.01 px).  For the near-tolerance log, which records the
// tests of exactly these visits, and for paths with an image line that is not finite.  Rows
// row0, row0 + step, ...
template <int K, bool LOG>
__device__ __noinline__ void visit_cells(const SmView& v, const PathN<K>& P, int pidx, int row0,
                                         int step, Pair* pairs, int* pair_count, int pair_cap) {
  const int t = P.target;
  const int rows = v.rows[t], cols = v.cols[t];
  const double hw = 0.5 * v.cell, tol_grow = v.tol2d + 1e-6;
  double n0[K], n1[K], dd[K], T[K];
  for (int i = 0; i < K; ++i) {
    const double* L = v.l2d + 6 * ((int64_t)P.ids[i] * v.n_cam + t);
    n0[i] = -L[5];
    n1[i] = L[4];
    dd[i] = -(n0[i] * L[0] + n1[i] * L[1]);
    T[i] = tol_grow + fabs(n0[i]) * hw + fabs(n1[i]) * hw;
  }
  int row_lo = 0, row_hi = rows - 1;
  if (K >= 2) {
    // cell-centre rows inside the y-extent of the first two strips' parallelogram
    const double det = n0[0] * n1[K > 1 ? 1 : 0] - n1[0] * n0[K > 1 ? 1 : 0];
    if (fabs(det) > 1e-9) {
      double ymin = 1e300, ymax = -1e300;
      for (int s0 = -1; s0 <= 1; s0 += 2)
        for (int s1 = -1; s1 <= 1; s1 += 2) {
          const int b = K > 1 ? 1 : 0;
          const double y = (n0[0] * (s1 * T[b] - dd[b]) - n0[b] * (s0 * T[0] - dd[0])) / det;
          ymin = fmin(ymin, y);
          ymax = fmax(ymax, y);
        }
      if (isfinite(ymin) && isfinite(ymax)) {
        const double lo = floor(ymin / v.cell - 0.5) - 1.0, hi = ceil(ymax / v.cell - 0.5) + 1.0;
        row_lo = (int)fmax(0.0, fmin((double)(rows - 1), lo));
        row_hi = (int)fmax(-1.0, fmin((double)(rows - 1), hi));
      }
    }
  }
  const float cellf = (float)v.cell, to_index = 1.0f / cellf;
  for (int cy = row_lo + row0; cy <= row_hi; cy += step) {
    int xmin = 0, xmax = cols - 1;
    const float yc = ((float)cy + 0.5f) * cellf;
    for (int i = 0; i < K; ++i) {
      const float C = fmaf((float)n1[i], yc, (float)dd[i]), Tf = (float)T[i] + 0.01f;
      if (fabs(n0[i]) < 1e-12) {
        if (fabsf(C) > Tf) {
          xmin = 1;
          xmax = 0;
        }
      } else {
        const float inv = 1.0f / (float)n0[i];
        float xl = (-Tf - C) * inv, xr = (Tf - C) * inv;
        if (xl > xr) {
          const float s_ = xl;
          xl = xr;
          xr = s_;
        }
        const int a = (int)ceilf(xl * to_index - 0.5f - 1e-3f);
        const int b = (int)floorf(xr * to_index - 0.5f + 1e-3f);
        xmin = max(xmin, max(a, 0));
        xmax = min(xmax, min(b, cols - 1));
      }
    }
    if (xmin > xmax) continue;
    const int base = v.cell_off[t] + cy * cols * v.sub;
    const int q1 = v.cstart[base + (xmax + 1) * v.sub];
    for (int q = v.cstart[base + xmin * v.sub]; q < q1; ++q)
      if (exact_2d<K, LOG>(v, P, q)) {
        const int slot = append_slot(pair_count);
        if (slot < pair_cap) pairs[slot] = Pair{pidx, (unsigned)q | kEdge};
      }
  }
}

// visit_cells for every path: a warp per path at level 1, else a thread.
template <int K>
__global__ void __launch_bounds__(256) enum_log_kernel(const __grid_constant__ SmView v,
                                                       const void* in_v, const int* n_ptr,
                                                       int in_cap, Pair* pairs, int* pair_count,
                                                       int pair_cap) {
  constexpr int L = K == 1 ? 32 : 1;
  const int n_in = *n_ptr;
  if (n_in > in_cap) return;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gt / L < n_in; gt += step)
    visit_cells<K, true>(v, static_cast<const PathN<K>*>(in_v)[gt / L], (int)(gt / L),
                         (int)(gt % L), L, pairs, pair_count, pair_cap);
}

// Expand one level, first half: the detections of the target camera inside the strips of a
// path's K chosen points.  Any search region that holds every point within tol2d of all lines
// gives the same set, because the tests decide; here it is, for each row of cells, the x range
// that the strips (widened by the FP32 error bound) cover over the row's height.  A lane takes
// four rows at a time (K >= 2: one path a lane, whose strips meet in a few rows; K = 1: one
// path a warp, its rows over the lanes), looks up their runs of positions together and walks
// them.  FP32 decides each distance; pairs whose distance is within the bound of the tolerance
// are marked for FP64.  Detections inside the strips collect in a buffer of the warp, from
// which 32 at a time take the back-projection test (its lines are gathers, and half of the
// detections fail it; tested by tri_kernel, after a trip through memory, these left half of
// its lanes idle: 419,000 detections on each of six cameras, 9.5 -> 7.9 ms a call); what
// passes collects in a second buffer, and one atomic serves up to 128.
constexpr int kHitBuf = 64;    // detections inside the strips; tested from 32 on
constexpr int kPairBuf = 160;  // pairs; flushed above 128

template <int K>
__global__ void __launch_bounds__(256, K <= 2 ? 4 : 3) enum_kernel(
    const __grid_constant__ SmView v, const void* in_v, const int* n_ptr, int in_cap, Pair* pairs,
    int* pair_count, int pair_cap) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kRowStep = K == 1 ? 32 : 1;
  const int n_in = *n_ptr;
  if (n_in > in_cap) return;  // paths are missing: the level before is repeated
  __shared__ Pair buf_s[8][kPairBuf];
  __shared__ uint2 hit_s[8][kHitBuf];  // (path's lane, position with its edge mark)
  const int lane = threadIdx.x & 31;
  Pair* buf = buf_s[threadIdx.x >> 5];
  uint2* hit = hit_s[threadIdx.x >> 5];
  const PathN<K>* in = static_cast<const PathN<K>*>(in_v);
  const float tol = (float)v.tol2d;
  int fill = 0, hits = 0;
  auto flush = [&] {
    int base = 0;
    if (lane == 0) base = atomicAdd(pair_count, fill);
    base = __shfl_sync(kFull, base, 0);
    __syncwarp();
    for (int i = lane; i < fill; i += 32)
      if (base + i < pair_cap) pairs[base + i] = buf[i];
    __syncwarp();
    fill = 0;
  };
  const int warps = gridDim.x * 8, w0 = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int n_chunk = K == 1 ? n_in : (n_in + 31) / 32;
  for (int ch = w0; ch < n_chunk; ch += warps) {
    const int pidx = K == 1 ? ch : ch * 32 + lane;
    const bool live = pidx < n_in;
    const PathN<K> P = in[live ? pidx : n_in - 1];
    const int t = P.target;
    float nx[K], ny[K], d[K], T[K], inv[K], r[K];
    bool finite = true;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const float4 L = v.fl[(int64_t)P.ids[i] * v.n_cam + t];
      nx[i] = L.x;
      ny[i] = L.y;
      d[i] = L.z;
      finite = finite && fabsf(L.x) + fabsf(L.y) + fabsf(L.z) < 1e30f;
      T[i] = tol + v.eps + 5e-7f * fabsf(L.z);
      inv[i] = fabsf(L.x) < 1e-6f ? 0.0f : 1.0f / L.x;
      r[i] = T[i] * fabsf(inv[i]);
    }
    const int rows = v.rows[t], colsf = v.cols[t] * v.sub;
    const float cellf = (float)v.cell, to_col = (float)v.sub / cellf;
    const float xmax = (float)v.cols[t] * cellf, pad = 0.005f + 1e-6f * xmax;
    int row_lo = 0, row_hi = live ? rows - 1 : -1;
    if (!finite) {
      if (live)
        visit_cells<K, false>(v, P, pidx, K == 1 ? lane : 0, kRowStep, pairs, pair_count, pair_cap);
      row_hi = -1;
    } else {
      // rows that the strips reach: the line's segment over the image's width (K = 1), the
      // y-extent of the first two strips' parallelogram
      float ymin = -1e30f, ymax = 1e30f;
      if (K == 1) {
        if (fabsf(ny[0]) >= 1e-6f) {
          const float in_ = 1.0f / ny[0];
          const float ya = -d[0] * in_, yb = -(d[0] + nx[0] * xmax) * in_;
          const float e = T[0] * fabsf(in_) + 0.05f + 1e-6f * (fabsf(ya) + fabsf(yb));
          ymin = fminf(ya, yb) - e;
          ymax = fmaxf(ya, yb) + e;
        }
      } else {
        constexpr int b = K > 1 ? 1 : 0;
        const float det = nx[0] * ny[b] - ny[0] * nx[b];
        if (fabsf(det) > 1e-4f) {
          const float id = 1.0f / det;
          const float c = (nx[b] * d[0] - nx[0] * d[b]) * id;
          const float e = (fabsf(nx[0]) * T[b] + fabsf(nx[b]) * T[0]) * fabsf(id) +
                          2.0f * v.eps * fabsf(id) + 0.01f;
          ymin = c - e;
          ymax = c + e;
        }
      }
      const float lo = floorf(ymin / cellf - 1e-3f), hi = floorf(ymax / cellf + 1e-3f);
      row_lo = (int)fminf(fmaxf(lo, 0.0f), (float)rows);
      row_hi = live ? (int)fmaxf(fminf(hi, (float)(rows - 1)), -1.0f) : -1;
    }
    // the first min(hits, 32) entries of the hit buffer through the back-projection test
    // (checkBackProjection, StereoMatch.cpp:1206-1227); the rest moves up
    auto test_hits = [&] {
      __syncwarp();
      const int n = min(hits, 32);
      const uint2 e = hit[lane < n ? lane : 0];
      const int o = (int)e.x;
      const int g = (int)(e.y & ~kEdge);
      bool ok = lane < n, edge = (e.y & kEdge) != 0;
      const unsigned cams = __shfl_sync(kFull, P.cams, o);
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const int id = __shfl_sync(kFull, P.ids[i], o);
        const float2 p = v.fxy[id];
        const float4 L = v.fl[(int64_t)g * v.n_cam + (int)((cams >> (4 * i)) & 15u)];
        const float z = fabsf(fmaf(L.x, p.x, fmaf(L.y, p.y, L.z)));
        float b = v.eps + 5e-7f * fabsf(L.z);
        // eps covers coordinates inside the image: a path's first point, which comes from the
        // list and not from the grid, may lie anywhere
        if (i == 0) b += 5e-7f * (fabsf(p.x) + fabsf(p.y));
        ok = ok && !(z > tol + b);
        edge = edge || !(z < tol - b);
      }
      const int path = __shfl_sync(kFull, pidx, o);
      const unsigned m = __ballot_sync(kFull, ok);
      if (ok)
        buf[fill + __popc(m & ((1u << lane) - 1u))] = Pair{path, (unsigned)g | (edge ? kEdge : 0u)};
      fill += __popc(m);
      const uint2 rest = hit[min(n + lane, kHitBuf - 1)];
      __syncwarp();
      if (n + lane < hits) hit[lane] = rest;
      hits -= n;
      if (fill > kPairBuf - 32) flush();
    };
    const int base = v.cell_off[t];
    const int n_row = max(0, row_hi - row_lo + 1);
    const int n_max = __reduce_max_sync(kFull, n_row);
    for (int j0 = 0; j0 < n_max; j0 += 4 * kRowStep) {
      int q0[4], end[4], total = 0;
      {
        int a[4], b[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int j = j0 + (K == 1 ? s * 32 + lane : s);
          a[s] = b[s] = 0;
          if (j < n_row) {
            const int cy = row_lo + j;
            const float y0 = (float)cy * cellf, y1 = y0 + cellf;
            float xl = 0.0f, xr = xmax;
#pragma unroll
            for (int i = 0; i < K; ++i) {
              if (inv[i] == 0.0f) continue;
              const float ca = -fmaf(ny[i], y0, d[i]) * inv[i];
              const float cb = -fmaf(ny[i], y1, d[i]) * inv[i];
              xl = fmaxf(xl, fminf(ca, cb) - r[i] - pad);
              xr = fminf(xr, fmaxf(ca, cb) + r[i] + pad);
            }
            const int fa = max(0, (int)floorf(xl * to_col - 0.01f));
            const int fb = min(colsf - 1, (int)floorf(xr * to_col + 0.01f));
            if (xl <= xr && fa <= fb) {
              a[s] = v.cstart[base + cy * colsf + fa];
              b[s] = v.cstart[base + cy * colsf + fb + 1];
            }
          }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          q0[s] = a[s] - total;
          total += b[s] - a[s];
          end[s] = total;
        }
      }
      const int most = __reduce_max_sync(kFull, total);
      for (int j = 0; j < most; ++j) {
        const int q = j + (j < end[0] ? q0[0] : j < end[1] ? q0[1] : j < end[2] ? q0[2] : q0[3]);
        bool ok = j < total, edge = false;
        if (ok) {
          const float2 p = v.fxy[q];
#pragma unroll
          for (int i = 0; i < K; ++i) {
            const float z = fabsf(fmaf(nx[i], p.x, fmaf(ny[i], p.y, d[i])));
            ok = ok && !(z > T[i]);
            edge = edge || !(z < 2.0f * tol - T[i]);
          }
        }
        const unsigned m = __ballot_sync(kFull, ok);
        if (m) {
          if (ok)
            hit[hits + __popc(m & ((1u << lane) - 1u))] =
                make_uint2(lane, (unsigned)q | (edge ? kEdge : 0u));
          hits += __popc(m);
          if (hits > kHitBuf - 32) test_hits();
        }
      }
    }
    while (hits) test_hits();  // before the lanes take other paths
  }
  if (fill) flush();
}

// Lines of sight of a path's chosen points and of a candidate (last).
template <int K>
struct Rays {
  double p[K + 1][3], u[K + 1][3];
};

// calTriangulateTol (StereoMatch.cpp:1103-1126) where the smallest parallax is near or below
// the 6-degree knee: the reference's acos / sin path.
template <int K>
__device__ __noinline__ double knee_tol(const SmView& v, const Rays<K>& r) {
  double min_deg = 180.0;
  for (int i = 0; i <= K; ++i)
    for (int j = i + 1; j <= K; ++j) min_deg = fmin(min_deg, pair_deg(r.u[i], r.u[j]));
  return quick_tol_from_deg(min_deg, K + 1, v.m, v.tol3d);
}

// TriangulationCheckWithTol (StereoMatch.cpp:1127-1141) with myMATH::triangulation's own
// operations: the lines summed in build order, the candidate last (myMATH.cpp:376-418).
template <int K>
__device__ __noinline__ bool gate_exact(const Rays<K>& r, double tq) {
  double M[9], b[3];
  for (int q = 0; q < 9; ++q) M[q] = 0.0;
  b[0] = b[1] = b[2] = 0.0;
  for (int i = 0; i <= K; ++i) {
    double tt[9];
    normal_terms(r.u[i], tt);
    for (int q = 0; q < 3; ++q)
      b[q] = b[q] + (tt[3 * q] * r.p[i][0] + tt[3 * q + 1] * r.p[i][1] + tt[3 * q + 2] * r.p[i][2]);
    for (int q = 0; q < 9; ++q) M[q] = M[q] + tt[q];
  }
  double Mi[9], X[3];
  gauss_inverse3(M, Mi);
  for (int q = 0; q < 3; ++q) X[q] = Mi[3 * q] * b[0] + Mi[3 * q + 1] * b[1] + Mi[3 * q + 2] * b[2];
  double e = 0.0;
  bool thrown = false;
  for (int i = 0; i <= K; ++i) thrown |= !line_error_term(X, r.p[i], r.u[i], e);
  if (thrown) return false;  // the reference's triangulation throws; the check fails
  return sqrt(e / (K + 1)) <= tq;
}

__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// The triangulation gate.  The sum E of the squared distances of the least-squares point to
// the lines is formed from the point o of line 0 nearest line 1: with v_i the perpendicular
// from o to line i, M = sum(I - u u^T) and b = sum v_i, E = sum |v_i|^2 - b M^-1 b.  The v_i
// are as small as the distances themselves, so nothing cancels, and it takes two divisions
// where the reference's elimination and square roots take 17 and 2 k.  The reference's own e
// is within a few ulp of |X - p|^2 per line of E; a value farther than a wide multiple of that
// from the limit decides as the reference does, any other goes through its operations, as do
// nearly parallel lines and points so far away that its distance could turn out negative
// enough to throw.
template <int K>
__device__ __forceinline__ bool gate(const SmView& v, const Rays<K>& r) {
  constexpr int k1 = K + 1;
  double maxdot = -2.0;
#pragma unroll
  for (int i = 0; i < k1; ++i)
#pragma unroll
    for (int j = i + 1; j < k1; ++j) maxdot = fmax(maxdot, clamped_dot(r.u[i], r.u[j]));
  // min parallax in (6 + 5e-7, 174 - 5e-7) deg: the angle factor is exactly 1
  const double tq =
      maxdot <= kCos6 - 1e-9 && maxdot >= -kCos6 + 1e-9 ? v.tq[k1] : knee_tol<K>(v, r);
  const double w[3] = {r.p[1][0] - r.p[0][0], r.p[1][1] - r.p[0][1], r.p[1][2] - r.p[0][2]};
  const double c = dot3(r.u[0], r.u[1]), s2 = 1.0 - c * c;
  const double t0 = (dot3(w, r.u[0]) - dot3(w, r.u[1]) * c) / s2;
  double o[3], R2 = t0 * t0;
#pragma unroll
  for (int d = 0; d < 3; ++d) o[d] = r.p[0][d] + t0 * r.u[0][d];
  double E, det = 1.0;
  if (K == 1) {
    const double q[3] = {r.p[1][0] - o[0], r.p[1][1] - o[1], r.p[1][2] - o[2]};
    const double a = dot3(q, r.u[1]);
    const double x[3] = {q[0] - a * r.u[1][0], q[1] - a * r.u[1][1], q[2] - a * r.u[1][2]};
    R2 = fmax(R2, dot3(q, q));
    E = 0.5 * dot3(x, x);  // the point halfway between the lines
  } else {
    double b[3] = {0, 0, 0}, S = 0.0;
    double mxx = k1, myy = k1, mzz = k1, mxy = 0, mxz = 0, myz = 0;
#pragma unroll
    for (int i = 0; i < k1; ++i) {
      const double* u = r.u[i];
      mxx -= u[0] * u[0];
      myy -= u[1] * u[1];
      mzz -= u[2] * u[2];
      mxy -= u[0] * u[1];
      mxz -= u[0] * u[2];
      myz -= u[1] * u[2];
      if (i == 0) continue;  // o lies on line 0
      const double q[3] = {r.p[i][0] - o[0], r.p[i][1] - o[1], r.p[i][2] - o[2]};
      const double a = dot3(q, u);
      R2 = fmax(R2, dot3(q, q));
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double x = q[d] - a * u[d];
        b[d] += x;
        S += x * x;
      }
    }
    const double cxx = myy * mzz - myz * myz, cxy = mxz * myz - mxy * mzz,
                 cxz = mxy * myz - mxz * myy;
    const double cyy = mxx * mzz - mxz * mxz, cyz = mxy * mxz - mxx * myz,
                 czz = mxx * myy - mxy * mxy;
    det = mxx * cxx + mxy * cxy + mxz * cxz;
    const double bMb = b[0] * (cxx * b[0] + 2.0 * (cxy * b[1] + cxz * b[2])) +
                       b[1] * (cyy * b[1] + 2.0 * cyz * b[2]) + czz * b[2] * b[2];
    E = S - bMb / det;
  }
  const double lim = k1 * (tq * tq);
  // R2 <= 4e6: the reference's squared distances are above -1e-8 (8 ulp of R2)
  const bool safe = s2 > 1e-3 && det > 1e-3 && R2 <= 4e6;
  const double band = 1e-6 * lim + k1 * 1e-14 * R2 + 1e-9 * E;
  if (safe && E > lim + band) return false;
  if (safe && E < lim - band) return true;
  return gate_exact<K>(r, tq);
}

// StereoMatch::selectNextCameraByMaxPairAngle (StereoMatch.cpp:1375-1411) in FP64.
template <int N>
__device__ __noinline__ int next_camera_exact(const SmView& v, const PathN<N>& ch) {
  int best = -1;
  double best_score = -1.0;
  for (int cam = 0; cam < v.n_cam; ++cam) {
    if (!v.active[cam]) continue;
    bool used = false;
    for (int i = 0; i < N; ++i) used |= (ch.cam(i) == cam);
    if (used) continue;
    double ux[N], uy[N];
    for (int i = 0; i < N; ++i) {
      const double* L = v.l2d + 6 * ((int64_t)ch.ids[i] * v.n_cam + cam);
      ux[i] = L[2];
      uy[i] = L[3];
    }
    double score = 0.0;
    for (int i = 0; i < N; ++i) {
      for (int j = i + 1; j < N; ++j) {
        const double s = fabs(ux[i] * uy[j] - uy[i] * ux[j]);
        if (s > score) score = s;
        if (score >= 1.0 - 1e-12) break;
      }
      if (score >= 1.0 - 1e-12) break;
    }
    if (score > best_score) {
      best_score = score;
      best = cam;
    }
  }
  return best;
}

// The same from the FP32 lines (their normals span the same angles): the largest score wins
// when it is clear of the others by far more than FP32 can err.
template <int N>
__device__ __forceinline__ int next_camera(const SmView& v, const PathN<N>& ch) {
  int best = -1, left = 0;
  float top = -1.0f, second = -1.0f;
  for (int cam = 0; cam < v.n_cam; ++cam) {
    bool used = !v.active[cam];
#pragma unroll
    for (int i = 0; i < N; ++i) used |= (ch.cam(i) == cam);
    if (used) continue;
    ++left;
    float2 n[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      n[i] = *reinterpret_cast<const float2*>(v.fl + (int64_t)ch.ids[i] * v.n_cam + cam);
    float score = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int j = i + 1; j < N; ++j)
        score = fmaxf(score, fabsf(n[i].x * n[j].y - n[i].y * n[j].x));
    if (score > top) {
      second = top;
      top = score;
      best = cam;
    } else if (score > second) {
      second = score;
    }
  }
  if (left <= 1 || top - second > 1e-5f) return best;
  return next_camera_exact<N>(v, ch);
}

// Expand one level, second half: one thread per (path, candidate) pair.  All 2D tests in FP64
// for the pairs that FP32 could not decide, the quick triangulation gate (computeMinParallaxDeg,
// calTriangulateTol, TriangulationCheckWithTol: StereoMatch.cpp:1072-1141), then the child path
// (terminal, or with its next target camera).  Bound by the gathers of the lines of sight and by
// L1 (70% busy at K = 1): the exact branches take rays and paths by address, so these lie in
// local memory, 336 to 624 B a thread.
template <int K>
__device__ __forceinline__ void tri_tile(const SmView& v, const void* in_v, const Pair* pairs,
                                         int n_pairs, int tile, void* out_v, int* out_count,
                                         int out_cap) {
  __shared__ int s_cnt[8], s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool last = K + 1 == v.m;
  const int64_t gi = tile * (int64_t)blockDim.x + threadIdx.x;
  PathN<K + 1> ch;
  bool ok = gi < n_pairs;
  if (ok) {
    const Pair pr = pairs[gi];
    const PathN<K> P = static_cast<const PathN<K>*>(in_v)[pr.path];
    const int g = (int)(pr.g & ~kEdge);
    if (pr.g & kEdge) ok = exact_2d<K, false>(v, P, g);
    if (ok) {
      Rays<K> r;
#pragma unroll
      for (int i = 0; i <= K; ++i) {
        const double2* S =
            reinterpret_cast<const double2*>(v.los + 6 * (int64_t)(i < K ? P.ids[i < K ? i : 0] : g));
        const double2 a = S[0], b = S[1], c = S[2];
        r.p[i][0] = a.x;
        r.p[i][1] = a.y;
        r.p[i][2] = b.x;
        r.u[i][0] = b.y;
        r.u[i][1] = c.x;
        r.u[i][2] = c.y;
      }
      ok = gate<K>(v, r);
    }
    if (ok) {
#pragma unroll
      for (int i = 0; i < K; ++i) ch.ids[i] = P.ids[i];
      ch.ids[K] = g;
      ch.cams = P.cams | ((unsigned)P.target << (4 * K));
      ch.target = -1;
      if (!last) {
        ch.target = K + 1 < OLPT_MAX_CAM ? next_camera<K + 1>(v, ch) : -1;
        ok = ch.target >= 0;
      }
    }
  }
  // one atomic a block
  const unsigned m = __ballot_sync(0xffffffffu, ok);
  if (lane == 0) s_cnt[warp] = __popc(m);
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < 8; ++w) {
      const int k = s_cnt[w];
      s_cnt[w] = t;
      t += k;
    }
    s_base = t ? atomicAdd(out_count, t) : 0;
  }
  __syncthreads();
  if (!ok) return;
  const int slot = s_base + s_cnt[warp] + __popc(m & ((1u << lane) - 1u));
  if (!last) {
    if (slot < out_cap) static_cast<PathN<K + 1>*>(out_v)[slot] = ch;
    return;
  }
  if (slot >= out_cap) return;
  Path full;
#pragma unroll
  for (int i = 0; i < OLPT_MAX_CAM; ++i) {
    full.ids[i] = i <= K ? ch.ids[i <= K ? i : 0] : 0;
    full.cams[i] = i <= K ? (signed char)ch.cam(i) : 0;
  }
  full.k = K + 1;
  full.target = -1;
  static_cast<Path*>(out_v)[slot] = full;
}

// LOOP: the blocks share the tiles of 256 pairs; else there is a block for each (the loop is 10%
// slower at the largest levels).
template <int K, bool LOOP>
__global__ void __launch_bounds__(256, K <= 2 ? 4 : K <= 4 ? 3 : 2) tri_kernel(
    const __grid_constant__ SmView v, const void* in_v, const Pair* pairs, const int* n_ptr,
    int pair_cap, void* out_v, int* out_count, int out_cap) {
  const int n_pairs = *n_ptr;
  if (n_pairs > pair_cap) return;  // pairs are missing: the level is repeated
  const int tiles = (int)((n_pairs + 255ll) / 256);
  int tile = blockIdx.x;
  if (tile >= tiles) return;
  for (;;) {
    tri_tile<K>(v, in_v, pairs, n_pairs, tile, out_v, out_count, out_cap);
    tile += gridDim.x;
    if (!LOOP || tile >= tiles) return;
    __syncthreads();  // the tile's counts are no longer read
  }
}

// StereoMatch::checkMatch, case "every active camera was used to build"
// (StereoMatch.cpp:520-540): triangulate in camera order, gate on tol_3d and limit.
__device__ __forceinline__ void check_path(const SmView& v, const Path& P, int* cand_ids,
                                           double* cand_e, double* cand_x, int* cand_count,
                                           int cap) {
  int ids[OLPT_MAX_CAM];
  for (int c = 0; c < v.n_cam; ++c) ids[c] = -1;
  for (int j = 0; j < P.k; ++j) ids[P.cams[j]] = P.ids[j];
  Line3 Ls[OLPT_MAX_CAM];
  const Line3* Lp[OLPT_MAX_CAM];
  int n = 0;
  for (int c = 0; c < v.n_cam; ++c) {
    if (ids[c] < 0) continue;
    load_line3(v.los + 6 * (int64_t)ids[c], Ls[n]);
    Lp[n] = &Ls[n];
    ++n;
  }
  double X[3], err;
  if (!triangulate<OLPT_MAX_CAM>(Lp, n, X, err)) return;  // the reference throws here
  if (err > v.tol3d) return;
  if (X[0] > v.limit[1] || X[0] < v.limit[0] || X[1] > v.limit[3] || X[1] < v.limit[2] ||
      X[2] > v.limit[5] || X[2] < v.limit[4])
    return;
  int slot = atomicAdd(cand_count, 1);
  if (slot >= cap) return;
  for (int c = 0; c < v.n_cam; ++c)
    cand_ids[(int64_t)slot * v.n_cam + c] = ids[c] < 0 ? -1 : v.pid[ids[c]];
  cand_e[slot] = err;
  cand_x[3 * slot] = X[0];
  cand_x[3 * slot + 1] = X[1];
  cand_x[3 * slot + 2] = X[2];
}

__global__ void check_kernel(const __grid_constant__ SmView v, const Path* term, const int* n_ptr,
                             int* cand_ids, double* cand_e, double* cand_x, int* cand_count,
                             int cap) {
  const int n = *n_ptr;
  if (n > cap) return;
  const int step = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
    check_path(v, term[i], cand_ids, cand_e, cand_x, cand_count, cap);
}

}  // namespace

// ---------------------------------------------------------------- host driver
// Steps 2-6 of pruneMatch on the candidates in ctx->prune.ids_s / e_s (M x n_cam, in
// the reference's order): the kept flags end in ctx->prune.sel (device, M bytes) and,
// when selected is given, on the host.  False when the comparator sorts must run on
// the host (prune_candidates) instead.
bool prune_select_device(olpt_ctx* ctx, const PruneView& pv, int M, int n_cam,
                         int64_t total_points, char* selected) {
  cudaStream_t s = ctx->stream;
  PruneWork& P = ctx->prune;
  prune_device(P, pv, M, n_cam, total_points, s);
  int cnt[PC_N];
  ReadBack rb(ctx);
  rb.add(cnt, P.counts.p, sizeof(cnt));
  rb.add(&P.n_sel, P.spos.as<int>() + M, sizeof(int));
  rb.finish();
  if (cnt[PC_FLAG]) return false;
  const int G = cnt[PC_BOTH];
  if (!cnt[PC_REPLACE]) {
    if (selected && M > 0) {
      OLPT_CUDA(cudaMemcpyAsync(selected, P.sel.p, (size_t)M, cudaMemcpyDeviceToHost, s));
      OLPT_CUDA(cudaStreamSynchronize(s));
    }
    return true;
  }
  // a replacement fires: the sequential greedy over pinned staging
  PhaseTimer pg(ctx->prof, PH_GREEDY_HOST);
  const size_t b_ord = (size_t)G * sizeof(int), b_pts = (size_t)G * n_cam * sizeof(int);
  const size_t b_dbl = (size_t)G * sizeof(double);
  P.pin.ensure(b_ord + b_pts + 2 * b_dbl + G + 64);
  char* hp = P.pin.as<char>();
  double* g_pct = reinterpret_cast<double*>(hp);
  double* g_e = reinterpret_cast<double*>(hp + b_dbl);
  int* order = reinterpret_cast<int*>(hp + 2 * b_dbl);
  int* g_pts = reinterpret_cast<int*>(hp + 2 * b_dbl + b_ord);
  uint8_t* g_cnt = reinterpret_cast<uint8_t*>(hp + 2 * b_dbl + b_ord + b_pts);
  if (G > 0) {
    OLPT_CUDA(cudaMemcpyAsync(order, P.val.p, b_ord, cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(g_pts, P.g_pts.p, b_pts, cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(g_cnt, P.g_cnt.p, (size_t)G, cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(g_pct, P.g_pct.p, b_dbl, cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(g_e, P.g_e.p, b_dbl, cudaMemcpyDeviceToHost, s));
  }
  OLPT_CUDA(cudaStreamSynchronize(s));
  std::vector<char> sel(G, 0);
  greedy_select(G, n_cam, g_pts, g_cnt, g_pct, g_e, total_points, sel.data());
  std::vector<char> flags(M, 0);
  for (int i = 0; i < G; ++i)
    if (sel[i]) flags[order[i]] = 1;
  if (M > 0) {
    OLPT_CUDA(cudaMemcpyAsync(P.sel.p, flags.data(), (size_t)M, cudaMemcpyHostToDevice, s));
    OLPT_CUDA(cudaStreamSynchronize(s));
  }
  if (selected) std::copy(flags.begin(), flags.end(), selected);
  count_selected(P, M, s);
  P.n_sel = 0;
  for (int i = 0; i < G; ++i) P.n_sel += sel[i] ? 1 : 0;
  return true;
}

void stereo_match_device(olpt_ctx* ctx, const SmParams& prm, StereoResult& res) {
  cudaStream_t s = ctx->stream;
  const int n_cam = ctx->n_cam;
  SmView v{};
  v.n_cam = n_cam;
  res.on_device = false;
  res.M = 0;
  int n_active = 0;
  for (int c = 0; c < n_cam; ++c) {
    v.active[c] = ctx->cams_h[c].is_active;
    n_active += v.active[c];
  }
  OLPT_REQUIRE(n_active >= 2, OLPT_ERR_INVALID_ARG, "preCheck: need at least 2 active cameras.");
  OLPT_REQUIRE(prm.match_cam_count >= 2 && prm.match_cam_count <= n_active, OLPT_ERR_INVALID_ARG,
               "preCheck: match_cam_count must be within [2," + std::to_string(n_active) + "].");
  v.n_active = n_active;
  v.m = std::min(std::max(2, prm.match_cam_count), n_active);
  OLPT_REQUIRE(v.m == n_active, OLPT_ERR_UNSUPPORTED,
               "match_cam_count below the number of active cameras: the reference aborts on this "
               "path (checkMatch leaves e_check NaN, StereoMatch.cpp:561-600 vs :129)");
  v.cell = std::max(1, prm.idmap_cell_px);
  v.tol2d = prm.tol_2d_px;
  v.tol3d = prm.tol_3d_mm;
  v.near_band = ctx->sm.near_band;
  if (v.near_band > 0.0) {
    v.near_rec = ctx->sm.near_rec.as<olpt_near_record>();
    v.near_count = ctx->sm.near_count.as<unsigned long long>();
    v.near_cap = ctx->sm.near_cap;
  }
  for (int q = 0; q < 6; ++q) v.limit[q] = prm.limit[q];

  StereoWork& W = ctx->sm;
  // reference camera: fewest detections among active (StereoMatch.cpp:70-85)
  int ref = -1;
  int64_t best = INT64_MAX;
  for (int c = 0; c < n_cam; ++c) {
    if (!v.active[c]) continue;
    if (ctx->det_counts_h[c] < best) {
      best = ctx->det_counts_h[c];
      ref = c;
    }
  }
  res.ref_cam = ref;

  // grid over the detections of all cameras
  int64_t total = 0;
  float max_side = 0.0f;
  int64_t cells = 0;
  for (int c = 0; c < n_cam; ++c) {
    const CamDev& cm = ctx->cams_h[c];
    v.raw_off[c] = (int)total;
    total += v.active[c] ? ctx->det_counts_h[c] : 0;
    v.x[c] = ctx->dets[c].x.as<double>();
    v.y[c] = ctx->dets[c].y.as<double>();
    v.Wd[c] = (double)cm.n_col;
    v.Hd[c] = (double)cm.n_row;
    v.rows[c] = std::max(1, cm.n_row / v.cell + (cm.n_row % v.cell ? 1 : 0));
    v.cols[c] = std::max(1, cm.n_col / v.cell + (cm.n_col % v.cell ? 1 : 0));
    max_side = std::max(max_side, (float)(v.rows[c] + v.cols[c]) * v.cell);
    cells += (int64_t)v.rows[c] * v.cols[c];
    if (v.active[c]) require_scan((int64_t)v.rows[c] * v.cols[c]);
  }
  OLPT_REQUIRE(total < (1ll << 30), OLPT_ERR_UNSUPPORTED, "stereo: too many detections");
  v.raw_off[n_cam] = (int)total;
  v.eps = 1e-6f * max_side;
  // calTriangulateTol (StereoMatch.cpp:1103-1126) with an angle factor of 1
  for (int k = 2; k <= OLPT_MAX_CAM; ++k)
    v.tq[k] = v.tol3d * std::sqrt(double(v.m > 2 ? v.m : 2) / double(k)) * 1.0;
  // columns of a pixel where the cells stay within a few million entries (a run of cells then
  // covers little more than its x range: 1.7 times fewer positions to test at 0.06
  // detections/px than with square cells of 4 px), else wider
  v.sub = v.cell;
  while (v.sub > 1 && cells * v.sub > (8ll << 20)) v.sub /= 2;
  int64_t n_cells = 0;
  for (int c = 0; c < n_cam; ++c) {
    v.cell_off[c] = (int)n_cells;
    if (v.active[c]) n_cells += (int64_t)v.rows[c] * v.cols[c] * v.sub + 1;
  }
  OLPT_REQUIRE(n_cells < (1ll << 30), OLPT_ERR_UNSUPPORTED, "stereo: too many grid cells");
  const int n = (int)total;
  W.cell_start.ensure((size_t)(n_cells + 1) * sizeof(int), s);
  W.cell_cnt.ensure((size_t)(n_cells + 1) * sizeof(int), s);
  W.cell_of.ensure((size_t)(n + 1) * sizeof(int), s);
  W.pid.ensure((size_t)(n + 1) * sizeof(int), s);
  W.xy.ensure((size_t)(n + 1) * sizeof(double2), s);
  W.fxy.ensure((size_t)(n + 1) * sizeof(float2), s);
  W.los.ensure((size_t)(n + 1) * 6 * sizeof(double), s);
  W.l2d.ensure((size_t)(n + 1) * n_cam * 6 * sizeof(double), s);
  W.fl.ensure((size_t)(n + 1) * n_cam * sizeof(float4), s);
  v.cstart = W.cell_start.as<int>();
  v.pid = W.pid.as<int>();
  v.xy = W.xy.as<double2>();
  v.fxy = W.fxy.as<float2>();
  v.los = W.los.as<double>();
  v.l2d = W.l2d.as<double>();
  v.fl = W.fl.as<float4>();
  OLPT_CUDA(cudaMemsetAsync(W.cell_cnt.p, 0, (size_t)n_cells * sizeof(int), s));
  if (n > 0)
    bin_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(v, n, W.cell_of.as<int>(), W.cell_cnt.as<int>());
  exclusive_scan(W.cell_cnt.as<int>(), (int)n_cells, W.cell_start.as<int>(), W.scan_tmp, s,
                 INT32_MAX);
  if (n > 0) {
    place_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(v, n, W.cell_of.as<int>(), W.cell_cnt.as<int>(),
                                                 W.pid.as<int>(), W.xy.as<double2>(),
                                                 W.fxy.as<float2>());
    int64_t most = 0;
    for (int c = 0; c < n_cam; ++c)
      most = std::max<int64_t>(most, v.raw_off[c + 1] - v.raw_off[c]);
    los_kernel<<<OLPT_G(dim3(nblk(most, kLineThreads / 2), n_cam)), kLineThreads, 0, s>>>(
        v, ctx->cams_d.as<CamDev>(), W.los.as<double>());
    lines_kernel<<<OLPT_G(dim3(nblk(n, kLineThreads), n_cam)), kLineThreads, 0, s>>>(
        v, ctx->cams_d.as<CamDev>(), W.l2d.as<double>(), W.fl.as<float4>());
  }
  OLPT_CUDA(cudaGetLastError());

  // Breadth-first expansion of the build DFS.  Counters: [0] the paths of level 1, [2l - 1] the
  // pairs of level l, [2l] its children (at the last level, the complete paths), [15] the
  // candidates.  The kernels read the counts on the device, and one whose input exceeds its
  // buffer does nothing, so that a level can be repeated over larger buffers.
  constexpr int kCand = 15;
  static_assert(2 * (OLPT_MAX_CAM - 1) < kCand, "stereo counters");
  W.counters.ensure(16 * sizeof(int), s);
  int* cnt = W.counters.as<int>();
  int h[16] = {0};
  const int64_t n_ref = v.raw_off[ref + 1] - v.raw_off[ref];
  const int cap_a = (int)std::max<int64_t>(n_ref, 1024);
  const int last = v.m - 1;
  // bytes of a partial path of k points
  auto rec = [&](int k) -> size_t {
    if (k >= v.m) return sizeof(Path);
    switch (k) {
      case 1: return sizeof(PathN<1>);
      case 2: return sizeof(PathN<2>);
      case 3: return sizeof(PathN<3>);
      case 4: return sizeof(PathN<4>);
      case 5: return sizeof(PathN<5>);
      case 6: return sizeof(PathN<6>);
      default: return sizeof(PathN<8>);
    }
  };
  // A look at the counts after every step lets the buffers and grids follow them, but leaves
  // the device idle for about 10 us.  Up to 16,384 seeds the levels are enqueued without one
  // (buffers of 16 paths and 8 pairs a seed or what earlier calls needed; 10,000 detections on
  // each of four cameras: 860 -> 745 us a call), over grids of those guesses or a full chip
  // (sized by buffers that a dense frame has grown, 300 detections on six cameras take 680 us
  // instead of the 395 on a fresh context).  The line, us a call with and without looks: 10,000
  // detections on four 1024^2 cameras 577 and 499, 16,000 732 and 653, 25,000 1,080 and 1,040,
  // 40,000 2,256 and 2,427; on six 2048^2 cameras 16,000 893 and 764, 40,000 1,396 and 1,278.
  bool look = v.near_band > 0.0 || n_ref > 16384;
  const int64_t path_guess = std::min<int64_t>(INT32_MAX, std::max<int64_t>(16 * n_ref, 4096));
  const int64_t pair_guess = std::min<int64_t>(INT32_MAX, std::max<int64_t>(8 * n_ref, 4096));
  const int64_t term_guess = std::max<int64_t>(4 * n_ref, 4096);
  // threads of a kernel whose count is not known: for the guess or a full chip, within the buffer
  auto at_once = [](int64_t cap, int64_t guess) {
    return std::min(cap, std::max<int64_t>(guess, 148 * 2048));
  };
  int pair_cap = (int)pair_guess;
  // buffers are grow-only: their capacity from earlier calls avoids a redo
  pair_cap = (int)std::max<int64_t>(pair_cap, (int64_t)(W.pairs.bytes / sizeof(Pair)) - 1);
  DevBuf* in_buf = &W.path_a;
  DevBuf* out_buf = &W.path_b;
  W.path_a.ensure(std::max(cap_a * rec(1), look ? 0 : (size_t)path_guess * rec(last)), s);
  if (!look) W.path_b.ensure((size_t)path_guess * rec(last), s);
  OLPT_CUDA(cudaMemsetAsync(cnt, 0, 16 * sizeof(int), s));
  if (n_ref > 0)
    seed_kernel<<<OLPT_G(nblk(n_ref)), 256, 0, s>>>(v, ref, W.path_a.as<PathN<1>>(), cnt, cap_a);
  OLPT_CUDA(cudaGetLastError());

  int in_cap = cap_a, out_cap = 0, cap_c = 0, level = 1;
  bool enumerate = true;
  auto check = [&] {
    W.cand_ids.ensure((size_t)cap_c * n_cam * sizeof(int), s);
    W.cand_e.ensure((size_t)cap_c * sizeof(double), s);
    W.cand_x.ensure((size_t)cap_c * 3 * sizeof(double), s);
    check_kernel<<<OLPT_G(std::min(nblk(look ? cap_c : at_once(cap_c, term_guess), 128), 148 * 64)), 128, 0, s>>>(
        v, W.term.as<Path>(), cnt + 2 * last, W.cand_ids.as<int>(), W.cand_e.as<double>(),
        W.cand_x.as<double>(), cnt + kCand, cap_c);
    OLPT_CUDA(cudaGetLastError());
  };
  auto read_counts = [&] {
    ReadBack rb(ctx);
    rb.add(h, cnt, sizeof(h));
    rb.finish();
  };
  int caps_pair[OLPT_MAX_CAM + 1], caps_out[OLPT_MAX_CAM + 1];
  while (n_ref > 0) {
    const bool log = v.near_band > 0.0;
    if (enumerate) {
      W.pairs.ensure((size_t)pair_cap * sizeof(Pair), s);
      auto kern = log ? enum_log_kernel<1> : enum_kernel<1>;
      switch (level) {
        case 1: break;
        case 2: kern = log ? enum_log_kernel<2> : enum_kernel<2>; break;
        case 3: kern = log ? enum_log_kernel<3> : enum_kernel<3>; break;
        case 4: kern = log ? enum_log_kernel<4> : enum_kernel<4>; break;
        case 5: kern = log ? enum_log_kernel<5> : enum_kernel<5>; break;
        case 6: kern = log ? enum_log_kernel<6> : enum_kernel<6>; break;
        default: kern = log ? enum_log_kernel<7> : enum_kernel<7>; break;
      }
      // so many blocks that a warp slot gets several chunks of the larger levels, which vary
      const int64_t work =
          level == 1 ? 32 * (int64_t)in_cap : look ? h[2 * level - 2] : at_once(in_cap, path_guess);
      const int pid = ctx->prof.begin(PROF_STEREO, s);
      kern<<<OLPT_G((int)std::min<int64_t>(nblk(work), 148 * 32)), 256, 0, s>>>(
          v, in_buf->p, cnt + 2 * level - 2, in_cap, W.pairs.as<Pair>(), cnt + 2 * level - 1,
          pair_cap);
      ctx->prof.end(PROF_STEREO, pid, s, 0.0);
      OLPT_CUDA(cudaGetLastError());
    }
    if (look) read_counts();
    // the triangulation gate and the children
    DevBuf* dst = level == last ? &W.term : out_buf;
    const int64_t guess =
        level == last ? term_guess
        : !look || level == 1 ? path_guess
                              : std::max<int64_t>(4 * (int64_t)h[2 * level - 2], 4096);
    out_cap = (int)std::min<int64_t>(
        INT32_MAX, std::max<int64_t>({(int64_t)out_cap, guess,
                                      (int64_t)(dst->bytes / rec(level + 1)) - 1}));
    dst->ensure((size_t)out_cap * rec(level + 1), s);
    auto kern = look ? tri_kernel<1, false> : tri_kernel<1, true>;
    switch (level) {
      case 1: break;
      case 2: kern = look ? tri_kernel<2, false> : tri_kernel<2, true>; break;
      case 3: kern = look ? tri_kernel<3, false> : tri_kernel<3, true>; break;
      case 4: kern = look ? tri_kernel<4, false> : tri_kernel<4, true>; break;
      case 5: kern = look ? tri_kernel<5, false> : tri_kernel<5, true>; break;
      case 6: kern = look ? tri_kernel<6, false> : tri_kernel<6, true>; break;
      default: kern = look ? tri_kernel<7, false> : tri_kernel<7, true>; break;
    }
    const int pid = ctx->prof.begin(PROF_STEREO, s);
    const int tiles = nblk(look ? std::min(h[2 * level - 1], pair_cap) : at_once(pair_cap, pair_guess));
    kern<<<OLPT_G(std::max(tiles, 1)), 256, 0, s>>>(
        v, in_buf->p, W.pairs.as<Pair>(), cnt + 2 * level - 1, pair_cap, dst->p, cnt + 2 * level,
        out_cap);
    ctx->prof.end(PROF_STEREO, pid, s, 0.0);
    OLPT_CUDA(cudaGetLastError());
    caps_pair[level] = pair_cap;
    caps_out[level] = out_cap;
    const bool done = level == last;
    if (done) {
      cap_c = out_cap;
      if (!look) check();
    }
    if (done || look) {
      read_counts();
      // the first level whose pairs or children did not fit: the levels after it did nothing
      int bad = look ? level : 1;
      while (bad <= level && h[2 * bad - 1] <= caps_pair[bad] && h[2 * bad] <= caps_out[bad]) ++bad;
      if (bad <= level) {
        look = true;  // from here on the buffers follow the counts
        if ((level - bad) & 1) std::swap(in_buf, out_buf);
        level = bad;
        in_cap = bad == 1 ? cap_a : caps_out[bad - 1];
        enumerate = h[2 * bad - 1] > caps_pair[bad];
        const int from = enumerate ? 2 * bad - 1 : 2 * bad;
        const int cap = (int)std::min<int64_t>(INT32_MAX, h[from] + (int64_t)h[from] / 4 + 1024);
        if (enumerate) pair_cap = cap;
        out_cap = enumerate ? 0 : cap;
        OLPT_CUDA(cudaMemsetAsync(cnt + from, 0, (16 - from) * sizeof(int), s));
        continue;
      }
      if (!done && h[2 * level] == 0) break;  // no children; the counts after it are 0
    }
    if (done) {
      if (look) {
        cap_c = std::max(h[2 * last], 1);
        check();
        read_counts();
      }
      break;
    }
    in_cap = out_cap;
    out_cap = 0;
    enumerate = true;
    std::swap(in_buf, out_buf);
    ++level;
  }
  const int M = h[kCand];
  res.n_cam = n_cam;
  PhaseTimer pt(ctx->prof, PH_PRUNE);
  std::vector<int> counts(n_cam);
  std::vector<int> active(n_cam);
  PruneView pv{};
  int64_t total_points = 0;
  int max_count = 0;
  for (int c = 0; c < n_cam; ++c) {
    counts[c] = (int)ctx->det_counts_h[c];
    active[c] = v.active[c];
    pv.active[c] = v.active[c];
    pv.count[c] = counts[c];
    pv.offset[c] = (int)total_points;
    total_points += counts[c];
    max_count = std::max(max_count, counts[c]);
  }
  res.M = M;
  PruneWork& P = ctx->prune;
  auto download = [&](const void* ids, const void* e, const void* X) {
    res.ids.resize((size_t)M * n_cam);
    res.e.resize(M);
    res.X.resize((size_t)M * 3);
    if (M == 0) return;
    OLPT_CUDA(cudaMemcpyAsync(res.ids.data(), ids, (size_t)M * n_cam * sizeof(int),
                              cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(res.e.data(), e, (size_t)M * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(res.X.data(), X, (size_t)M * 3 * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
  };
  // candidate order, prune and greedy on the device
  if (sort_candidates_device(P, W.cand_ids.as<int>(), W.cand_e.as<double>(),
                             W.cand_x.as<double>(), M, n_cam, max_count - 1, s)) {
    if (prune_select_device(ctx, pv, M, n_cam, total_points, nullptr)) {
      res.ids.clear();
      res.e.clear();
      res.X.clear();
      res.selected.clear();
      res.on_device = true;  // downloaded on demand (stereo_result_to_host)
      return;
    }
    download(P.ids_s.p, P.e_s.p, P.X_s.p);
    OLPT_CUDA(cudaStreamSynchronize(s));
  } else {
    download(W.cand_ids.p, W.cand_e.p, W.cand_x.p);
    OLPT_CUDA(cudaStreamSynchronize(s));
    sort_candidates(res);
  }
  prune_candidates(res, counts, active);
}

// The selected candidates' points and (when asked for) ids, in candidate order.
__global__ void sel_gather_kernel(const uint8_t* sel, const int* pos, int M, const double* X,
                                  double* out, const int* ids, int n, int* out_ids) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M || !sel[i]) return;
  const int64_t k = pos[i], j = i;
  if (out) {
    out[3 * k] = X[3 * j];
    out[3 * k + 1] = X[3 * j + 1];
    out[3 * k + 2] = X[3 * j + 2];
  }
  if (out_ids)
    for (int c = 0; c < n; ++c) out_ids[k * n + c] = ids[j * n + c];
}

// The matches of a result that is still on the device: gathered there (a tenth of the
// candidates), so that the others need not come over.
void stereo_matches(olpt_ctx* ctx, const StereoResult& r, int* ids, double* xyz) {
  cudaStream_t s = ctx->stream;
  PruneWork& P = ctx->prune;
  const int M = (int)r.M, n = r.n_cam;
  const size_t k = (size_t)P.n_sel, b_xyz = k * 3 * sizeof(double), b_ids = k * n * sizeof(int);
  if (k == 0 || (!ids && !xyz)) return;
  ctx->scratch.ensure(b_xyz + b_ids, s);
  double* dx = ctx->scratch.as<double>();
  int* di = reinterpret_cast<int*>(ctx->scratch.as<char>() + b_xyz);
  sel_gather_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(P.sel.as<uint8_t>(), P.spos.as<int>(), M,
                                                   P.X_s.as<double>(), xyz ? dx : nullptr,
                                                   P.ids_s.as<int>(), n, ids ? di : nullptr);
  OLPT_CUDA(cudaGetLastError());
  ReadBack rb(ctx);
  if (ids) rb.add(ids, di, b_ids);
  if (xyz) rb.add(xyz, dx, b_xyz);
  rb.finish();
}

void stereo_result_to_host(olpt_ctx* ctx, StereoResult& r) {
  if (!r.on_device) return;
  cudaStream_t s = ctx->stream;
  PruneWork& P = ctx->prune;
  const int64_t M = r.M;
  const int n = r.n_cam;
  r.ids.resize((size_t)M * n);
  r.e.resize(M);
  r.X.resize((size_t)M * 3);
  r.selected.resize(M);
  if (M > 0) {
    OLPT_CUDA(cudaMemcpyAsync(r.ids.data(), P.ids_s.p, (size_t)M * n * sizeof(int),
                              cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(r.e.data(), P.e_s.p, (size_t)M * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(r.X.data(), P.X_s.p, (size_t)M * 3 * sizeof(double),
                              cudaMemcpyDeviceToHost, s));
    OLPT_CUDA(cudaMemcpyAsync(r.selected.data(), P.sel.p, (size_t)M, cudaMemcpyDeviceToHost, s));
  }
  OLPT_CUDA(cudaStreamSynchronize(s));
  r.on_device = false;
}

int64_t stereo_objects(olpt_ctx* ctx, const StereoResult& r) {
  cudaStream_t s = ctx->stream;
  int64_t n = 0;
  if (r.on_device) {
    PruneWork& P = ctx->prune;
    const int M = (int)r.M;
    n = P.n_sel;
    ctx->obj.ensure(std::max<int64_t>(n, 1), ctx->n_cam, s);
    ctx->obj.n = n;
    if (n > 0)
      sel_gather_kernel<<<OLPT_G(nblk(M)), 256, 0, s>>>(P.sel.as<uint8_t>(), P.spos.as<int>(), M,
                                                       P.X_s.as<double>(), ctx->obj.xyz.as<double>(),
                                                       nullptr, 0, nullptr);
    OLPT_CUDA(cudaGetLastError());
    return n;
  }
  std::vector<double> xyz;
  for (size_t j = 0; j < r.selected.size(); ++j)
    if (r.selected[j]) xyz.insert(xyz.end(), &r.X[3 * j], &r.X[3 * j] + 3);
  n = (int64_t)(xyz.size() / 3);
  ctx->obj.ensure(std::max<int64_t>(n, 1), ctx->n_cam, s);
  ctx->obj.n = n;
  if (n > 0) {
    OLPT_CUDA(cudaMemcpyAsync(ctx->obj.xyz.p, xyz.data(), xyz.size() * sizeof(double),
                              cudaMemcpyHostToDevice, s));
    OLPT_CUDA(cudaStreamSynchronize(s));  // xyz is a local host buffer
  }
  return n;
}

}  // namespace olpt
