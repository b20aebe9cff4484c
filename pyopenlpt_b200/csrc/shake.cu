// Kernel family (c): Shake -- residual image, per-particle line search, score,
// repeated and ghost flags.
//
// Reference: Shake::runShake (src/srcSTB/Shake.cpp:36-163), calResidueImage (:165-244),
// calROIBound (:246-277), buildROIInfo (:279-328), shakeOneObject (:409-665),
// calObjectScore (:668-782), markRepeatedObj (:785-823), TracerShakeStrategy
// gaussIntensity / project2DInt / calShakeResidue (:901-1045).
//
// B200 mapping, per shake iteration:
//  1. splat: one thread per (object, camera) projects the object (FP64) and evaluates
//     the OTF there; the warp then raises every pixel of its 32 windows in a projection
//     plane to the window's Gaussian by atomic maxima (max-fusion does not depend on
//     order, and non-negative floats order as integers).
//  2. residual: one streaming pass writes residual = image - projection and sets the
//     projection plane back to 0.
//  3. shake: a group of 8 lanes (32 for few objects) per particle stages its 8x8
//     augmented ROI of every camera in shared memory, then runs the reference's
//     axis-wise line search.  Projections spread (trial point, camera) pairs over the
//     group's lanes, residues the pixels; a warp carries four particles, so the scalar
//     control flow is issued once for four.
// Precision: Real = float is the production path (residual, OTF Gaussian and MSE in
// FP32); Real = double is the parity path, which also sums every camera's squared
// error in the reference's row-major order so that only exp() rounding differs.
// Projections, polyfit and all decisions stay in FP64 in both.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "olpt_ctx.cuh"
#include "olpt_shake_dev.cuh"
#include "olpt_otf.cuh"
#include "olpt_scan.cuh"
#include "olpt_shake.h"

namespace olpt {

constexpr size_t kShakeSmemMax = 200 * 1024;  // shared memory of a shake block

namespace {

inline int nblk(int64_t n, int t = 256) { return (int)((n + t - 1) / t); }

// ---------------------------------------------------------------- 1. splat
__device__ __forceinline__ void raise_to(float* p, float v) {
  atomicMax(reinterpret_cast<unsigned int*>(p), __float_as_uint(v));
}
__device__ __forceinline__ void raise_to(double* p, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)__double_as_longlong(v));
}

// Bound by the FP64 geometry of the pairs and, per window, about 60 instructions on 16 lanes
// (a window's row is one 16-byte run of one sector for the atomics).  Replaces a pass over the
// objects, the counting sort of the pairs by 32x32 image tile (five launches) and a kernel in
// which four tiles each recomputed a pair's window and Gaussian per pixel: 120,000 objects on
// six 2048^2 cameras, the whole residual took 620 us and takes 270 us (cold caches).
template <typename Real>
__global__ void __launch_bounds__(256) splat_kernel(const __grid_constant__ ShakeView v,
                                                    const double* xyz, int64_t n, double* uv,
                                                    Real* otfp, const uint8_t* flags,
                                                    int all_cams, int per_warp) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warp = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32;
  const int64_t pair = lane < per_warp ? warp * per_warp + lane : n * v.n_cam;
  double u = 0.0, w = 0.0;
  Real o[5] = {0, 0, 0, 0, 0};
  Rect r{1, 0, 1, 0};
  int c = 0;
  if (pair < n * v.n_cam) {
    const int64_t obj = pair / v.n_cam;
    c = (int)(pair - obj * v.n_cam);
    const CamDev& cm = v.cams[c];
    const double X = xyz[3 * obj], Y = xyz[3 * obj + 1], Z = xyz[3 * obj + 2];
    cam_project(cm, X, Y, Z, u, w);
    uv[2 * pair] = u;
    uv[2 * pair + 1] = w;
    double q[5];
    otf_param(v.otf, c, X, Y, Z, q);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      o[k] = (Real)q[k];
      otfp[5 * pair + k] = o[k];
    }
    if (!(flags && flags[obj] != 0) && (all_cams || cm.is_active))
      r = roi_bound(cm.n_row, cm.n_col, u, w, v.r_px, v.r_px);
  }
  const bool some = r.rmax > r.rmin && r.cmax > r.cmin;
  unsigned todo = __ballot_sync(kFull, some);
  const int sub = lane & 15;
  // two windows at a time, 16 lanes each
  while (todo) {
    const int a = __ffs(todo) - 1;
    todo &= todo - 1;
    const int b = todo ? __ffs(todo) - 1 : -1;
    if (todo) todo &= todo - 1;
    const bool on = lane < 16 || b >= 0;
    const int src = lane < 16 || b < 0 ? a : b;
    const double uu = __shfl_sync(kFull, u, src), ww = __shfl_sync(kFull, w, src);
    Real q[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) q[k] = __shfl_sync(kFull, o[k], src);
    const int r0 = __shfl_sync(kFull, r.rmin, src), r1 = __shfl_sync(kFull, r.rmax, src);
    const int c0 = __shfl_sync(kFull, r.cmin, src), c1 = __shfl_sync(kFull, r.cmax, src);
    const int cc = __shfl_sync(kFull, c, src);
    if (!on) continue;
    const int wd = c1 - c0, area = wd * (r1 - r0);
    Real* plane = reinterpret_cast<Real*>(v.proj[cc].p);
    const int64_t pitch = v.proj[cc].pitch / (int64_t)sizeof(Real);
    for (int k = sub; k < area; k += 16) {
      const int dr = k / wd, row = r0 + dr, col = c0 + k - dr * wd;
      const Real g = gauss<Real>(col, row, uu, ww, q);
      if (g > (Real)0) raise_to(plane + row * pitch + col, g);
    }
  }
}

// ---------------------------------------------------------------- 2. residual
// residual = o where nothing projects, else min(o, o - p), clamped at 0 on request
template <typename Real>
__device__ __forceinline__ Real subtract(Real o, Real p, int clamp) {
  if (!(p > (Real)0)) return o;
  Real val = o - p;
  if (val > o) val = o;
  return clamp && val < (Real)0 ? (Real)0 : val;
}

// Streaming: four pixels a thread, 4-byte to 32-byte loads by type.  The projection planes
// are read and, where something projected, set back to 0 for the next pass.
template <typename Real, typename T>
__device__ __forceinline__ void residual_row4(const T* src, Real* proj, Real* dst, int col, int W,
                                              int clamp) {
  struct alignas(4 * sizeof(T) > 16 ? 16 : 4 * sizeof(T)) Quad {
    T v[4];
  };
  struct alignas(16) QuadR {
    Real v[4];
  };
  if (col + 4 <= W) {
    const Quad o = *reinterpret_cast<const Quad*>(src + col);
    const QuadR p = *reinterpret_cast<const QuadR*>(proj + col);
    QuadR r;
    bool any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      r.v[k] = subtract<Real>((Real)o.v[k], p.v[k], clamp);
      any |= p.v[k] != (Real)0;
    }
    *reinterpret_cast<QuadR*>(dst + col) = r;
    if (any) *reinterpret_cast<QuadR*>(proj + col) = QuadR{{0, 0, 0, 0}};
  } else {
    for (int k = col; k < W; ++k) {
      dst[k] = subtract<Real>((Real)src[k], proj[k], clamp);
      proj[k] = (Real)0;
    }
  }
}

template <typename Real>
__global__ void __launch_bounds__(256) residual_kernel(const __grid_constant__ ShakeView v,
                                                       int clamp, int all_cams) {
  const int cam = blockIdx.z;
  const CamDev& cm = v.cams[cam];
  if (!(all_cams || cm.is_active)) return;
  const PlaneView& s = v.orig[cam];
  const int col = 4 * (blockIdx.x * blockDim.x + threadIdx.x), row = blockIdx.y;
  if (row >= s.H || col >= s.W) return;
  Real* proj = reinterpret_cast<Real*>(v.proj[cam].p + row * v.proj[cam].pitch);
  Real* dst = reinterpret_cast<Real*>(v.res[cam].p + row * v.res[cam].pitch);
  const unsigned char* src = s.p + row * s.pitch;
  switch (s.dtype) {
    case OLPT_U8:
      residual_row4<Real>(src, proj, dst, col, s.W, clamp);
      break;
    case OLPT_U16:
      residual_row4<Real>(reinterpret_cast<const uint16_t*>(src), proj, dst, col, s.W, clamp);
      break;
    case OLPT_F32:
      residual_row4<Real>(reinterpret_cast<const float*>(src), proj, dst, col, s.W, clamp);
      break;
    default:
      residual_row4<Real>(reinterpret_cast<const double*>(src), proj, dst, col, s.W, clamp);
  }
}

// ---------------------------------------------------------------- 3. shake
// Camera parameters of a block in shared memory, [value][camera] so that the lanes of a
// group, each on its own camera, read neighbouring words.  Polynomial terms keep their
// coefficients as they are and their exponents (all 0..3, CamDev::pow3) as byte offsets of the
// factors in the point's power list (CamSmem::expo).
constexpr int kCamVals = 28;  // R 9, T 3, fx fy cx cy, distortion 12

struct Strided {
  const double* p;
  __device__ __forceinline__ double operator[](int i) const { return p[8 * i]; }
};

struct CamTab {  // one camera's column of the block's table
  Strided R, T, dist;
  double fx, fy, cx, cy;
  int is_distorted, n_dist;
};

struct CamSmem {
  int4* meta;      // 8: kind (project_tab), terms, distorted, distortion coefficients
  double* val;     // kCamVals x 8
  double* coef;    // 2 n_poly x 8: u, v coefficient of every term
  uint2* expo;     // n_poly x 8: byte offsets (one byte each for x, y, z) of the u term's and
                   // the v term's factors in the point's power list [3][4]
};

__device__ __forceinline__ CamSmem cam_smem(unsigned char* base, int n_poly) {
  CamSmem s;
  s.meta = reinterpret_cast<int4*>(base);
  s.val = reinterpret_cast<double*>(base + 8 * sizeof(int4));
  s.coef = s.val + kCamVals * 8;
  s.expo = reinterpret_cast<uint2*>(s.coef + 2 * n_poly * 8);
  return s;
}
size_t cam_smem_bytes(int n_poly) {
  return 8 * sizeof(int4) + (size_t)kCamVals * 64 + (size_t)n_poly * (2 * 64 + 64);
}

// The block's threads copy the cameras' parameters (the exponents are small integers
// stored as doubles) into the table.
__device__ void load_cams(const ShakeView& v, const CamSmem& s) {
  if ((int)threadIdx.x < v.n_cam) {
    const CamDev& m = v.cams[threadIdx.x];
    s.meta[threadIdx.x] = make_int4(m.type == CAM_PINHOLE ? 0 : m.pow3 ? 1 : 2, m.n_coeff,
                                    m.is_distorted, m.n_dist);
  }
  for (int i = threadIdx.x; i < kCamVals * 8; i += blockDim.x) {
    const int c = i & 7, k = i >> 3;
    double x = 0.0;
    if (c < v.n_cam) {
      const CamDev& m = v.cams[c];
      x = k < 9 ? m.R[k] : k < 12 ? m.T[k - 9] : k == 12 ? m.fx : k == 13 ? m.fy
          : k == 14 ? m.cx : k == 15 ? m.cy : m.dist[k - 16];
    }
    s.val[i] = x;
  }
  for (int i = threadIdx.x; i < v.n_poly * 8; i += blockDim.x) {
    const int c = i & 7, k = i >> 3;
    double cu = 0.0, cv = 0.0;
    uint2 e = make_uint2(0, 0);
    if (c < v.n_cam && v.cams[c].type == CAM_POLYNOMIAL && v.cams[c].pow3 &&
        k < v.cams[c].n_coeff) {
      const CamDev& m = v.cams[c];
      cu = m.ucoef[4 * k];
      cv = m.vcoef[4 * k];
      for (int j = 0; j < 3; ++j) {
        e.x |= (uint32_t)(8 * (4 * j + (int)m.ucoef[4 * k + 1 + j])) << (8 * j);
        e.y |= (uint32_t)(8 * (4 * j + (int)m.vcoef[4 * k + 1 + j])) << (8 * j);
      }
    }
    s.coef[(2 * k) * 8 + c] = cu;
    s.coef[(2 * k + 1) * 8 + c] = cv;
    s.expo[i] = e;
  }
}

// Polynomials with other exponents: out of line, so that pow() stays out of the kernel's
// instruction footprint.
__device__ __noinline__ double2 project_general(const CamDev* c, double X, double Y, double Z) {
  double u, w;
  poly_project(*c, X, Y, Z, u, w);
  return make_double2(u, w);
}

// cam_project with the parameters of the block's table (same operations, same order);
// kind: 0 pinhole, 1 polynomial with exponents 0..3 (pw: the point's powers, poly_powers),
// 2 any other polynomial (from the camera itself).
__device__ __forceinline__ void project_tab(const ShakeView& v, const CamSmem& cs,
                                            const double* pw, int c, double X, double Y, double Z,
                                            double& u, double& w) {
  const int4 meta = cs.meta[c];
  const int kind = meta.x, n_coeff = meta.y;
  if (kind == 0) {
    CamTab t;
    const double* b = cs.val + c;
    t.R.p = b;
    t.T.p = b + 9 * 8;
    t.dist.p = b + 16 * 8;
    t.fx = b[12 * 8];
    t.fy = b[13 * 8];
    t.cx = b[14 * 8];
    t.cy = b[15 * 8];
    t.is_distorted = meta.z;
    t.n_dist = meta.w;
    pinhole_project(t, X, Y, Z, u, w);
  } else if (kind == 1) {
    double su = 0, sv = 0;
    const double* cf = cs.coef + c;
    const uint2* ex = cs.expo + c;
    const char* pb = reinterpret_cast<const char*>(pw);
    auto power = [&](uint32_t off) { return *reinterpret_cast<const double*>(pb + off); };
#pragma unroll 2
    for (int i = 0; i < n_coeff; ++i) {
      double uu = cf[16 * i], vv = cf[16 * i + 8];
      const uint2 e = ex[8 * i];
      const double fx = power(e.x & 255u), fy = power((e.x >> 8) & 255u), fz = power(e.x >> 16);
      uu = uu * fx * fy * fz;
      if (e.x == e.y)  // u and v share the term's monomial, as in a full polynomial
        vv = vv * fx * fy * fz;
      else
        vv = vv * power(e.y & 255u) * power((e.y >> 8) & 255u) * power(e.y >> 16);
      su += uu;
      sv += vv;
    }
    u = su;
    w = sv;
  } else {
    const double2 p = project_general(v.cams + c, X, Y, Z);
    u = p.x;
    w = p.y;
  }
}

// A group of LPO lanes works on one object (32 / LPO objects a warp); its arrays in
// shared memory.  j: trial slot, c: camera.
template <typename Real>
struct Obj {
  Real* aug;       // n_cam x roi_area: augmented ROIs
  double* dd;      // n_cam x (roi_area + 1): squared differences (FP64 ordered sums)
  double2* uv;     // [j][c] projection
  Real* otf;       // [j][c][5]
  uint32_t* win;   // [j][c] rows (bits 0..15) and columns (16..31) of the ROI in the window
  int4* roi;       // [c] rmin, rmax, cmin, cmax
  Real* ey;        // [8] row factors of the camera and point at work
  double* pw;      // [j][3][4] powers of the points' coordinates (polynomial cameras)
};

template <typename Real>
__device__ __forceinline__ Obj<Real> obj_smem(const ShakeView& v, unsigned char* b) {
  Obj<Real> s;
  s.aug = reinterpret_cast<Real*>(b);
  s.dd = reinterpret_cast<double*>(b + v.off_dd);
  s.uv = reinterpret_cast<double2*>(b + v.off_uv);
  s.roi = reinterpret_cast<int4*>(b + v.off_roi);
  s.ey = reinterpret_cast<Real*>(b + v.off_ey);
  s.otf = reinterpret_cast<Real*>(b + v.off_otf);
  s.win = reinterpret_cast<uint32_t*>(b + v.off_win);
  s.pw = reinterpret_cast<double*>(b + v.off_pw);
  return s;
}

// The projection window's rows / columns [lo, hi) within 16 ROI rows / columns from r0.
__device__ __forceinline__ uint32_t span16(int lo, int hi, int r0) {
  const int a = max(0, min(16, lo - r0)), b = max(0, min(16, hi - r0));
  return b > a ? ((1u << b) - 1u) & ~((1u << a) - 1u) : 0u;
}

// Projection, OTF and window of point (X, Y, Z) on camera c into slot (j, c).
template <typename Real, int NC>
__device__ __forceinline__ void eval_slot(const ShakeView& v, const CamSmem& cs, Obj<Real>& S,
                                          int j, int c, double X, double Y, double Z) {
  double u, w;
  project_tab(v, cs, S.pw + 12 * j, c, X, Y, Z, u, w);
  S.uv[j * NC + c] = make_double2(u, w);
  double q[5];
  otf_param(v.otf, c, X, Y, Z, q);
  Real* o = S.otf + 5 * (j * NC + c);
#pragma unroll
  for (int k = 0; k < 5; ++k) o[k] = (Real)q[k];
  const int4 R = S.roi[c];
  // TracerShakeStrategy::calShakeResidue's window (Shake.cpp:951-1045)
  const uint32_t rows =
      span16((int)floor(w - v.r_px), min(R.y, (int)ceil(w + v.r_px + 1)), R.x);
  const uint32_t cols = span16((int)floor(u - v.r_px), (int)ceil(u + v.r_px + 1), R.z);
  S.win[j * NC + c] = rows | (cols << 16);
}

template <typename Real>
__device__ __forceinline__ Real positive(Real x) {
  if constexpr (sizeof(Real) == 4) return fmaxf(x, 0.0f);  // NaN gives 0 too
  return x > (Real)0 ? x : (Real)0;
}

// gauss() in two steps: per ROI column and row a factor, per pixel the rest.  With every
// OTF angle +0 (cos 1, sin +0) the factors are the exponent's terms b dx^2 and c dy^2, else
// the offsets dx and dy.  Outside the window the factor is NaN, which gauss()'s comparison
// turns into an intensity of 0.  The int -> double -> float conversions then run once per
// column and row instead of once per pixel.
template <typename Real>
__device__ __forceinline__ Real axis_factor(bool separable, int at, double centre, Real coef,
                                            bool in) {
  const Real d = (Real)((double)at - centre);
  const Real f = separable ? coef * d * d : d;
  return in ? f : (Real)__longlong_as_double(0x7ff8000000000000LL);
}

template <typename Real, bool SEP>
__device__ __forceinline__ Real pixel_gauss(Real fx, Real fy, const Real* o) {
  if (SEP) return positive(o[0] * exp(-(fx + fy)));
  const Real xx = fx * o[3] + fy * o[4];
  const Real yy = -fx * o[4] + fy * o[3];
  return positive(o[0] * exp(-(o[1] * xx * xx + o[2] * yy * yy)));
}

// the row factors that a lane needs: rows g / 8 + LPO / 8 i of the 8 at ey
template <typename Real, int LPO>
__device__ __forceinline__ void row_factors(const Real* ey, int g, Real (&fy)[64 / LPO]) {
  if constexpr (LPO == 8) {
    constexpr int N = 16 / sizeof(Real);
#pragma unroll
    for (int q = 0; q < 8 / N; ++q) {
      const uint4 x = reinterpret_cast<const uint4*>(ey)[q];
      const Real* r = reinterpret_cast<const Real*>(&x);
#pragma unroll
      for (int k = 0; k < N; ++k) fy[q * N + k] = r[k];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 64 / LPO; ++i) fy[i] = ey[(g >> 3) + (LPO / 8) * i];
  }
}

// calShakeResidue (Shake.cpp:951-1045) for the points in the geometry slots 0 .. nj - 1
// (nj = 1 or 3) against the staged ROIs, for the warp's 32 / LPO objects at once.  Summation
// order: the squares of camera c's pixels p are summed over p = q - c area, + 32, ... for
// each of 32 partial sums q, and those in a butterfly (q ^ 16, ^ 8, .. ^ 1).  A lane holds
// the partial sums q = lane, lane + LPO, ...; the butterfly's first steps run in the lane,
// the rest over the group.  FP64: the squares of every camera are summed in row-major order.
// One copy of the code for every camera and point (the loops stay rolled): the kernel is
// bound by instruction fetch once its code outgrows the instruction caches.
template <typename Real, int NC, int LPO>
__device__ __forceinline__ void residue(const ShakeView& v, Obj<Real>& S, int nj, double f[3]) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int NA = 32 / LPO;  // partial sums a lane
  const int g = threadIdx.x & (LPO - 1);
  const int area = v.roi_area;
  const bool sep = v.otf.alpha_zero != 0;
  double cost[3] = {0.0, 0.0, 0.0};
  int used = 0;
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    const int4 R = S.roi[c];
    const int h = R.y - R.x, w = R.w - R.z;
    const bool some = h > 0 && w > 0;
    used += some ? 1 : 0;
    // the lanes' sums for point j -> the camera's mean
    auto add = [&](int j, Real s) {
#pragma unroll
      for (int o = LPO / 2; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
      if (some) {
        const double t = w * h == 64 ? (double)s * 0.015625 : (double)s / (double)(w * h);
        if (j == 0)
          cost[0] += t;
        else if (j == 1)
          cost[1] += t;
        else
          cost[2] += t;
      }
    };
    if (area == 64 && __all_sync(kFull, w == 8 || !some)) {
      // an ROI of 8 columns: the lane's pixels lie in one column, rows g / 8 + LPO / 8 i
      const int col = g & 7;
      Real m[64 / LPO];
#pragma unroll
      for (int i = 0; i < 64 / LPO; ++i)
        m[i] = (g >> 3) + (LPO / 8) * i < h ? S.aug[c * area + LPO * i + g] : (Real)0;
#pragma unroll 1
      for (int j = 0; j < nj; ++j) {
        const int e = j * NC + c;
        Real part[NA];
#pragma unroll
        for (int k = 0; k < NA; ++k) part[k] = (Real)0;
        const double2 uw = S.uv[e];
        Real o[5], fy[64 / LPO];
#pragma unroll
        for (int k = 0; k < 5; ++k) o[k] = S.otf[5 * e + k];
        const uint32_t win = S.win[e];
        const Real fx = axis_factor<Real>(sep, R.z + col, uw.x, o[1], (win >> (16 + col)) & 1u);
        if (g < 8)
          S.ey[g] = axis_factor<Real>(sep, R.x + g, uw.y, o[2], (win >> g) & 1u);
        __syncwarp();
        row_factors<Real, LPO>(S.ey, g, fy);
        // rows past a clipped ROI hold 0 and lie outside the window: their squares are 0
        auto pixels = [&](auto separable) {
#pragma unroll
          for (int i = 0; i < 64 / LPO; ++i) {
            const Real d = m[i] - pixel_gauss<Real, decltype(separable)::value>(fx, fy[i], o);
            if (sizeof(Real) == 8)
              S.dd[e * (area + 1) + LPO * i + g] = d * d;
            else
              part[i % NA] += d * d;
          }
        };
        if (sep)
          pixels(std::true_type{});
        else
          pixels(std::false_type{});
        __syncwarp();
        if (sizeof(Real) == 4) {
#pragma unroll
          for (int o = NA / 2; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < o; ++k) part[k] += part[k + o];
          add(j, part[0]);
        }
      }
      continue;
    }
    // an ROI of another size: a pixel's place and value serve the points together (20,000 objects
    // on four cameras, 32 lanes, ROIs of 256 pixels: 1,297 -> 1,199 us against one point after
    // the other)
    Real part[3][NA];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int k = 0; k < NA; ++k) part[j][k] = (Real)0;
    if (some) {
      int first = g;
      if (sizeof(Real) == 4) {
        first = (g - c * area) % LPO;
        if (first < 0) first += LPO;
      }
      const int n = w * h;
      int k = 0;
#pragma unroll 1
      for (int p = first; p < n; p += LPO, k = (k + 1) % NA) {
        const int pr = p / w, pc = p - pr * w;
        const Real m = S.aug[c * area + p];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if (j >= nj) break;
          const int e = j * NC + c;
          const uint32_t win = S.win[e];
          Real pred = (Real)0;
          if ((win >> pr) & (win >> (16 + pc)) & 1u) {
            const double2 uw = S.uv[e];
            pred = gauss<Real>(R.z + pc, R.x + pr, uw.x, uw.y, S.otf + 5 * e);
          }
          const Real d = m - pred;
          if (sizeof(Real) == 8) {
            S.dd[e * (area + 1) + p] = d * d;
          } else {
#pragma unroll
            for (int q = 0; q < NA; ++q)
              if (q == k) part[j][q] += d * d;
          }
        }
      }
    }
    if (sizeof(Real) == 4) {
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int o = NA / 2; o > 0; o >>= 1)
#pragma unroll
          for (int k = 0; k < o; ++k) part[j][k] += part[j][k + o];
#pragma unroll 1
      for (int j = 0; j < nj; ++j) add(j, j == 0 ? part[0][0] : j == 1 ? part[1][0] : part[2][0]);
    }
  }
  if (sizeof(Real) == 8) {
    // one lane per (point, camera): its squares in row-major order
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t * LPO < nj * NC; ++t) {
      const int e = t * LPO + g;
      double mse = 0.0;
      if (e < nj * NC) {
        const int4 R = S.roi[e % NC];
        const int h = R.y - R.x, w = R.w - R.z;
        const int n = h > 0 && w > 0 ? w * h : 0;
        const double* d = S.dd + e * (area + 1);
        double sse = 0.0;
        for (int i = 0; i < n; ++i) sse += d[i];
        mse = n > 0 ? sse / (double)n : 0.0;
        S.dd[e * (area + 1)] = mse;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c < NC; ++c) {
      const int4 R = S.roi[c];
      if (R.y > R.x && R.w > R.z)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (j < nj) cost[j] += S.dd[(j * NC + c) * (area + 1)];
    }
    __syncwarp();
  }
  // lane j divides cost j
  const double q = (g == 0 ? cost[0] : g == 1 ? cost[1] : cost[2]) / (double)used;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double x = __shfl_sync(kFull, q, j, LPO);
    f[j] = used > 1 ? x : __longlong_as_double(0x7ff0000000000000LL);
  }
}

// (X^T X)^-1 X^T for a parabola through x[0..n): myMATH::polyfit order 2
// (myMATH.cpp:490-534) with the reference's operation order, n = 3 or 4.
__host__ __device__ inline void parabola_matrix(const double* x, int n, double B[3][4]) {
  double X[4][3];
  for (int i = 0; i < n; ++i) {
    X[i][0] = 1.0;
    X[i][1] = x[i];
    X[i][2] = x[i] * x[i];
  }
  double A[9];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) {
      double s = 0;
      for (int i = 0; i < n; ++i) s += X[i][r] * X[i][c];
      A[3 * r + c] = s;
    }
  double Ai[9];
  gauss_inverse3(A, Ai);
  for (int r = 0; r < 3; ++r)
    for (int i = 0; i < n; ++i) {
      double s = 0;
      for (int k = 0; k < 3; ++k) s += Ai[3 * r + k] * X[i][k];
      B[r][i] = s;
    }
}

// linear and quadratic coefficients of the parabola through four points (out of line: only
// an extended line search needs it)
__device__ __noinline__ double2 fit4(double delta, double x4, double y0, double y1, double y2,
                                     double y3) {
  const double x[4] = {-delta, 0.0, delta, x4}, y[4] = {y0, y1, y2, y3};
  double B[3][4];
  parabola_matrix(x, 4, B);
  double c1 = 0, c2 = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    c1 += B[1][i] * y[i];
    c2 += B[2][i] * y[i];
  }
  return make_double2(c1, c2);
}

__device__ __forceinline__ bool in_roi(const int4& R, double u, double w) {
  return R.z <= u && u < R.w && R.x <= w && w < R.y;
}

// The median of the group's values (lanes with `has`), as sorting them would give it; 0
// without any.
template <int LPO>
__device__ __forceinline__ double group_median(double x, bool has) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31, g = lane & (LPO - 1), base = lane - g;
  const unsigned all = (LPO == 32 ? kFull : ((1u << (LPO & 31)) - 1u)) << base;
  const unsigned m = __ballot_sync(kFull, has) & all;
  const int n = __popc(m);
  int rank = 0;
#pragma unroll
  for (int k = 0; k < OLPT_MAX_CAM; ++k) {
    const double y = __shfl_sync(kFull, x, k, LPO);
    if (((m >> base) >> k) & 1u) rank += (y < x || (y == x && k < g)) ? 1 : 0;
  }
  const int mid = n / 2;
  const unsigned bm = __ballot_sync(kFull, has && rank == mid) & all;
  const unsigned bl = __ballot_sync(kFull, has && rank == mid - 1) & all;
  const double hi = __shfl_sync(kFull, x, bm ? __ffs(bm) - 1 : lane);
  const double lo = __shfl_sync(kFull, x, bl ? __ffs(bl) - 1 : lane);
  if (n == 0) return 0.0;
  return (n & 1) == 0 ? 0.5 * (hi + lo) : hi;
}

// A group of LPO lanes per object, 32 / LPO objects a warp.  Bound by instruction issue (the
// line search's scalar FP64 code, 12 to 15 projections and about 70 ROI passes per object) and
// by its fetch.  One warp per object issued all scalar code for a single object, converted
// every pixel's coordinates from integer over double to float, and held one copy of the
// evaluation per use (7.6 of 11.6 cycles between issues went to instruction fetch).  Here
// four objects share the scalar code, the conversions run per ROI row and column, and one
// copy of the evaluation serves every step, entered by the block's warps together.
// 120,000 objects on six polynomial cameras: 1.9 ms a launch, 49 to 59% of the issue slots (9.0
// ms and 50% with one warp per object); every sum keeps its order, so results are unchanged.
// Four resident blocks an SM (128 registers a thread); built for five (102 registers), 8,000
// objects take 126 us instead of 115, 32,000 of six cameras 767 instead of 694.
template <typename Real, int NC, int LPO>
__global__ void __launch_bounds__(128, 4) shake_kernel(const __grid_constant__ ShakeView v,
                                                       int64_t n, double* xyz, double* uv,
                                                       const Real* otfp, double* score,
                                                       double delta, const uint8_t* active,
                                                       double* resid_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int OPW = 32 / LPO;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane & (LPO - 1), gi = lane / LPO;
  const CamSmem cs = cam_smem(smem_raw, v.n_poly);
  load_cams(v, cs);
  __syncthreads();
  const int64_t o_raw = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * OPW + gi;
  const bool live = o_raw < n && !(active && !active[o_raw]);
  const bool idle = !__any_sync(kFull, live);
  // a group without an object of its own repeats another's and stores nothing
  const int64_t o = o_raw < n ? o_raw : n - 1;
  Obj<Real> S = obj_smem<Real>(v, smem_raw + v.cam_bytes +
                                      v.obj_stride * (size_t)(warp * OPW + gi));
  const int area = v.roi_area;
  const bool sep = v.otf.alpha_zero != 0;
  double P[3] = {xyz[3 * o], xyz[3 * o + 1], xyz[3 * o + 2]};
  const double* uvo = uv + o * NC * 2;

  // ---- buildROIInfo (Shake.cpp:279-328): lane c sets up camera c
  if (g < NC) {
    Rect R{0, 0, 0, 0};  // default-constructed PixelRange for skipped cameras
    const CamDev& m = v.cams[g];
    uint32_t win = 0;
    if (m.is_active) {
      const double u = uvo[2 * g], w = uvo[2 * g + 1];
      R = roi_bound(m.n_row, m.n_col, u, w, v.r_px * v.ratio, v.r_px * v.ratio);
      const Rect pr = roi_bound(m.n_row, m.n_col, u, w, v.r_px, v.r_px);
      win = span16(pr.rmin, pr.rmax, R.rmin) | (span16(pr.cmin, pr.cmax, R.cmin) << 16);
      if (rect_empty(R)) R = Rect{1, 0, 1, 0};
    }
    S.roi[g] = make_int4(R.rmin, R.rmax, R.cmin, R.cmax);
    S.win[g] = win;
  }
  __syncwarp();
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    const int4 R = S.roi[c];
    const int h = R.y - R.x, w = R.w - R.z;
    const bool some = h > 0 && w > 0;
    const double u = uvo[2 * c], vv = uvo[2 * c + 1];
    const Real* res = reinterpret_cast<const Real*>(v.res[c].p);
    const int64_t rp = v.res[c].pitch / (int64_t)sizeof(Real);
    const Real* q5 = otfp + (o * NC + c) * 5;
    if (area == 64 && __all_sync(kFull, w == 8 || !some)) {
      const int col = g & 7;
      const uint32_t win = S.win[c];
      Real q[5], a[64 / LPO], fy[64 / LPO];
#pragma unroll
      for (int k = 0; k < 5; ++k) q[k] = q5[k];
      const Real fx = axis_factor<Real>(sep, R.z + col, u, q[1], (win >> (16 + col)) & 1u);
      if (g < 8) S.ey[g] = axis_factor<Real>(sep, R.x + g, vv, q[2], (win >> g) & 1u);
#pragma unroll
      for (int i = 0; i < 64 / LPO; ++i) {
        const int row = (g >> 3) + (LPO / 8) * i;
        a[i] = some && row < h ? res[(int64_t)(R.x + row) * rp + R.z + col] : (Real)0;
      }
      __syncwarp();
      row_factors<Real, LPO>(S.ey, g, fy);
#pragma unroll
      for (int i = 0; i < 64 / LPO; ++i) {
        const int row = (g >> 3) + (LPO / 8) * i;
        const Real p = sep ? pixel_gauss<Real, true>(fx, fy[i], q)
                           : pixel_gauss<Real, false>(fx, fy[i], q);
        if (some && row < h) S.aug[c * area + LPO * i + g] = positive(a[i] + p);
      }
      __syncwarp();
    } else if (some) {
      const CamDev& m = v.cams[c];
      const Rect pr = roi_bound(m.n_row, m.n_col, u, vv, v.r_px, v.r_px);
      for (int pix = g; pix < w * h; pix += LPO) {
        const int row = R.x + pix / w, col = R.z + pix % w;
        Real a = res[(int64_t)row * rp + col];
        if (row >= pr.rmin && row < pr.rmax && col >= pr.cmin && col < pr.cmax)
          a += gauss<Real>(col, row, u, vv, q5);
        S.aug[c * area + pix] = positive(a);
      }
    }
  }
  __syncwarp();
  const int4 my_roi = S.roi[g < NC ? g : 0];  // camera g's, for the group votes

  // ---- shakeOneObject (Shake.cpp:409-665), one axis after the other.  Step 0 evaluates the
  // three trial points -delta, 0, +delta (slots 0, 1, 2), step 1 a point further along a
  // monotone axis, step 2 the minimum of the parabola through them (slot 0 each); the last
  // round projects the final position.  The steps share one copy of the evaluation.
  double f_final = 0.0;
  double tmp[3] = {P[0], P[1], P[2]};  // the reference's trial position: not reset per axis
  double x0 = 0.0, fL = 0.0, f0 = 0.0, fR = 0.0, f4 = 0.0, dx4 = 0.0, bf = 0.0, bx = 0.0;
  double kappa = 0.0, last = 0.0;
  bool skip_expand = false, allow_xhat = true, mono = false, four = false;
  int s = 0;
#pragma unroll 1
  for (int it = 0; it <= 9; ++it) {
    // the block's warps start every step together, so that they fetch its code together
    __syncthreads();
    if (idle) continue;
    const int ax = it / 3, step = it - 3 * ax;
    bool go = true;     // this group evaluates a point in this round
    double step_x = 0;  // its offset from x0
    int nj = 1;
    if (it == 9) {
      // the final position
    } else if (step == 0) {
      x0 = ax == 0 ? P[0] : ax == 1 ? P[1] : P[2];
      nj = 3;
    } else if (step == 1) {
      four = false;
      go = !skip_expand && mono;
      if (!__any_sync(kFull, go)) continue;
      const int gc = g < NC ? g : 0;
      const double2 p0 = S.uv[gc], p1 = S.uv[NC + gc], p2 = S.uv[2 * NC + gc];
      double J = 0.0, M = 0.0;
      const bool hasJ = g < NC && in_roi(my_roi, p0.x, p0.y) && in_roi(my_roi, p2.x, p2.y);
      const bool hasM = g < NC && in_roi(my_roi, p1.x, p1.y);
      if (hasJ) J = hypot(p2.x - p0.x, p2.y - p0.y) / fmax(2.0 * delta, 1e-12);
      if (hasM)
        M = fmin(fmin(p1.x - my_roi.z, my_roi.w - 1.0 - p1.x),
                 fmin(p1.y - my_roi.x, my_roi.y - 1.0 - p1.y));
      const double Jx = group_median<LPO>(J, hasJ);
      const double mpx = group_median<LPO>(M, hasM);
      const double Delta_roi = (Jx > 0.0 && mpx > 0.0) ? (0.5 * mpx / Jx) : 0.0;
      double Delta_try = 0.0;
      if (kappa > 0.0) {
        const double x3 = delta * (fL - fR) / (2.0 * kappa);
        if (fabs(x3) > delta) {
          s = (x3 > 0.0 ? +1 : -1);
          if (Jx > 0.0 && fabs(x3) > (1.0 / Jx))
            Delta_try = 1.0 / Jx;
          else
            Delta_try = 1.15 * fabs(x3);
        }
      }
      if (Delta_try <= 0.0 && Jx > 0.0) Delta_try = 1.0 / Jx;
      const double Dp = (Delta_try > 0.0 && Delta_roi > 0.0) ? fmin(Delta_try, Delta_roi) : 0.0;
      go = go && Dp > 0.0;
      step_x = dx4 = (s >= 0 ? +Dp : -Dp);
    } else {
      double c1 = 0.0, c2 = 0.0;
      const double y[3] = {fL, f0, fR};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        c1 += v.fit3[0][i] * y[i];
        c2 += v.fit3[1][i] * y[i];
      }
      if (four) {
        const double2 c = fit4(delta, dx4, fL, f0, fR, f4);
        c1 = c.x;
        c2 = c.y;
      }
      go = allow_xhat && c2 > 0.0;
      if (go) {
        step_x = -c1 / (2.0 * c2);
        double xmin = fmin(fmin(-delta, 0.0), delta), xmax = fmax(fmax(-delta, 0.0), delta);
        if (four) {
          xmin = fmin(xmin, dx4);
          xmax = fmax(xmax, dx4);
        }
        go = step_x >= xmin && step_x <= xmax;
      }
    }
    if (it == 9 || step == 0 || __any_sync(kFull, go)) {
      if (step != 0 && go) last = x0 + step_x;
      __syncwarp();
      auto trial = [&](int j) {
        return nj == 1 ? last : x0 + (j == 0 ? -delta : j == 1 ? 0.0 : delta);
      };
      if (v.n_poly > 0) {  // the powers of the points' coordinates, one list for all cameras
#pragma unroll 1
        for (int t = g; t < 3 * nj; t += LPO) {
          const int j = t / 3, k = t - 3 * j;
          const double q = trial(j);
          const double x = it == 9 ? (k == 0 ? P[0] : k == 1 ? P[1] : P[2])
                           : k == ax ? q
                                     : (k == 0 ? tmp[0] : k == 1 ? tmp[1] : tmp[2]);
          double* p = S.pw + 12 * j + 4 * k;
          p[0] = 1.0;
          p[1] = x;
          p[2] = poly_pow(x, 2.0);
          p[3] = poly_pow(x, 3.0);
        }
        __syncwarp();
      }
#pragma unroll 1
      for (int t = g; t < nj * NC; t += LPO) {
        const int j = nj == 1 ? 0 : t / NC, c = t - j * NC;
        const double q = trial(j);
        eval_slot<Real, NC>(v, cs, S, j, c, it == 9 ? P[0] : ax == 0 ? q : tmp[0],
                            it == 9 ? P[1] : ax == 1 ? q : tmp[1],
                            it == 9 ? P[2] : ax == 2 ? q : tmp[2]);
      }
      __syncwarp();
      if (it == 9) break;
      if (step != 0) {  // a point outside any camera's ROI is not taken
        const double2 p = S.uv[g < NC ? g : 0];
        const unsigned ob = __ballot_sync(kFull, g < NC && !in_roi(my_roi, p.x, p.y));
        go = go &&
             ((ob >> (lane - g)) & (LPO == 32 ? kFull : (1u << (LPO & 31)) - 1u)) == 0u;
      }
      if (__any_sync(kFull, go)) {
        double f[3];
        residue<Real, NC, LPO>(v, S, nj, f);
        if (step == 0) {
          fL = f[0];
          f0 = f[1];
          fR = f[2];
        } else if (go) {
          if (step == 1) {
            four = true;
            f4 = f[0];
          }
          if (f[0] < bf) {
            bf = f[0];
            bx = x0 + step_x;
          }
        }
      }
    }
    if (step == 0) {
      last = x0 + delta;  // the axis position as left by the last evaluation
      const double tol = 1e-3 * fmax(1.0, f0);
      const bool mono_dec = (fL > f0 + tol) && (f0 > fR + tol);
      const bool mono_inc = (fR > f0 + tol) && (f0 > fL + tol);
      mono = mono_dec || mono_inc;
      s = mono_dec ? +1 : (mono_inc ? -1 : 0);
      kappa = (fL - 2.0 * f0 + fR);
      const double grad = (fR - fL) / fmax(2.0 * delta, 1e-12);
      skip_expand = false;
      allow_xhat = true;
      if (kappa > 0.0) {
        const double x3 = delta * (fL - fR) / (2.0 * kappa);
        if (fabs(x3) <= 0.95 * delta) {
          const double a = kappa / (delta * delta + 1e-12);
          const double rho_pred = (grad * grad) / (2.0 * a * fmax(f0, 1.0));
          skip_expand = true;
          if (rho_pred < 8e-4) allow_xhat = false;
        }
      }
      // best of the three trials (the first of equal ones)
      bf = fL;
      bx = x0 + -delta;
      if (f0 < bf) {
        bf = f0;
        bx = x0;
      }
      if (fR < bf) {
        bf = fR;
        bx = x0 + delta;
      }
    } else if (step == 2) {
      if (ax == 0) {
        P[0] = bx;
        tmp[0] = last;
      } else if (ax == 1) {
        P[1] = bx;
        tmp[1] = last;
      } else {
        P[2] = bx;
        tmp[2] = last;
      }
      f_final = bf;  // after the last axis: the residue at the final position
    }
  }

  if (idle) return;

  // ---- final projection + calObjectScore (Shake.cpp:668-782): lane c scores camera c
  double pk = 0.0, nu = 0.0, de = 0.0;
  bool use = false;
  if (g < NC) {
    const CamDev& m = v.cams[g];
    const double2 p = S.uv[g];
    if (m.is_active) {
      const Rect R = roi_bound(m.n_row, m.n_col, p.x, p.y, v.r_px, v.r_px);
      use = !rect_empty(R);
      if (use) {
        // peak over the rect, sums of max(0, meas) and of the predictions, row-major
        const int4 Q = my_roi;
        const bool qv = Q.y > Q.x && Q.w > Q.z;
        const Real* res = reinterpret_cast<const Real*>(v.res[g].p);
        const int64_t rp = v.res[g].pitch / (int64_t)sizeof(Real);
        const int qw = Q.w - Q.z;
        Real o[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) o[k] = S.otf[5 * g + k];
        // the column factors of up to four columns are kept over the rows
        const bool four = R.cmax - R.cmin <= 4;
        Real fx[4];
        if (four)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            fx[k] = axis_factor<Real>(sep, R.cmin + k, p.x, o[1], true);
        auto add = [&](int r, int cc, Real gv) {
          const bool inq = qv && r >= Q.x && r < Q.y && cc >= Q.z && cc < Q.w;
          const double val = inq ? (double)S.aug[g * area + (r - Q.x) * qw + (cc - Q.z)]
                                 : (double)res[(int64_t)r * rp + cc];
          if (val > pk) pk = val;
          nu += fmax(0.0, val);
          de += (double)gv;
        };
#pragma unroll 1
        for (int r = R.rmin; r < R.rmax; ++r) {
          const Real fy = axis_factor<Real>(sep, r, p.y, o[2], true);
          if (four) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (R.cmin + k < R.cmax)
                add(r, R.cmin + k,
                    sep ? pixel_gauss<Real, true>(fx[k], fy, o)
                        : pixel_gauss<Real, false>(fx[k], fy, o));
          } else {
#pragma unroll 1
            for (int cc = R.cmin; cc < R.cmax; ++cc) {
              const Real f1 = axis_factor<Real>(sep, cc, p.x, o[1], true);
              add(r, cc, sep ? pixel_gauss<Real, true>(f1, fy, o)
                             : pixel_gauss<Real, false>(f1, fy, o));
            }
          }
        }
      }
    }
  }
  int n_used = 0, max_id = -1;
  double max_v = -__longlong_as_double(0x7ff0000000000000LL);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const bool uc = __shfl_sync(kFull, use ? 1 : 0, c, LPO) != 0;
    const double pc = __shfl_sync(kFull, pk, c, LPO);
    if (!uc) continue;
    ++n_used;
    if (pc > max_v) {
      max_v = pc;
      max_id = c;
    }
  }
  double tn = 0.0, td = 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const bool uc = __shfl_sync(kFull, use ? 1 : 0, c, LPO) != 0;
    const double nc = __shfl_sync(kFull, nu, c, LPO), dc = __shfl_sync(kFull, de, c, LPO);
    if (!uc || (n_used > 2 && c == max_id)) continue;  // without the brightest camera
    tn += nc;
    td += dc;
  }
  double sc = 1e-12;
  if (n_used >= 2) {
    double ratio = (td > 1e-12) ? (tn / td) : 1.0;
    ratio = fmax(2.0 / 3.0, fmin(1.5, ratio));
    sc = sqrt(ratio);
  }
  if (!live) return;
  if (g == 0) {
    xyz[3 * o] = P[0];
    xyz[3 * o + 1] = P[1];
    xyz[3 * o + 2] = P[2];
    score[o] *= sc;
    if (resid_out) resid_out[o] = f_final;
  }
  if (g < NC) {
    const double2 p = S.uv[g];
    uv[(o * NC + g) * 2] = p.x;
    uv[(o * NC + g) * 2 + 1] = p.y;
  }
}

// ---------------------------------------------------------------- repeated / ghost
__global__ void hash_key_kernel(const double* xyz, int n, double cell, int n_buckets, int* key) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long cx = (long long)floor(xyz[3 * i] / cell);
  const long long cy = (long long)floor(xyz[3 * i + 1] / cell);
  const long long cz = (long long)floor(xyz[3 * i + 2] / cell);
  unsigned long long h = (unsigned long long)(cx * 73856093LL) ^ (unsigned long long)(cy * 19349663LL) ^
                         (unsigned long long)(cz * 83492791LL);
  key[i] = (int)(h % (unsigned long long)n_buckets);
}

// number of neighbours j != i with squared distance < r2 (nanoflann radius test)
__global__ void neighbour_kernel(const double* xyz, int n, double cell, int n_buckets,
                                 const int* start, const int* items, double r2, int* has_nb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double X = xyz[3 * i], Y = xyz[3 * i + 1], Z = xyz[3 * i + 2];
  const long long cx = (long long)floor(X / cell), cy = (long long)floor(Y / cell),
                  cz = (long long)floor(Z / cell);
  int cnt = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        unsigned long long h = (unsigned long long)((cx + dx) * 73856093LL) ^
                               (unsigned long long)((cy + dy) * 19349663LL) ^
                               (unsigned long long)((cz + dz) * 83492791LL);
        const int b = (int)(h % (unsigned long long)n_buckets);
        for (int q = start[b]; q < start[b + 1]; ++q) {
          const int j = items[q];
          if (j == i) continue;
          const double ddx = xyz[3 * j] - X, ddy = xyz[3 * j + 1] - Y, ddz = xyz[3 * j + 2] - Z;
          const double d2 = ddx * ddx + ddy * ddy + ddz * ddz;
          if (d2 < r2) ++cnt;
        }
      }
  has_nb[i] = cnt > 0 ? 1 : 0;
}

// Greedy in index order (Shake.cpp:802-822): an object that is not itself marked
// marks every neighbour within the radius.  Only objects with neighbours do work.
// `list` holds, in ascending order, the objects that have any neighbour (list_n[0]
// of them); objects without neighbours mark nothing, so skipping them keeps the
// greedy identical.
__global__ void repeat_greedy_kernel(const double* xyz, int n, double cell, int n_buckets,
                                     const int* start, const int* items, double r2,
                                     const int* list, const int* list_n, uint8_t* rep) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int m = list_n[0];
  for (int q0 = 0; q0 < m; ++q0) {
    const int i = list[q0];
    if (i >= n - 1 || rep[i]) continue;
    const double X = xyz[3 * i], Y = xyz[3 * i + 1], Z = xyz[3 * i + 2];
    const long long cx = (long long)floor(X / cell), cy = (long long)floor(Y / cell),
                    cz = (long long)floor(Z / cell);
    for (int dz = -1; dz <= 1; ++dz)
      for (int dy = -1; dy <= 1; ++dy)
        for (int dx = -1; dx <= 1; ++dx) {
          unsigned long long h = (unsigned long long)((cx + dx) * 73856093LL) ^
                                 (unsigned long long)((cy + dy) * 19349663LL) ^
                                 (unsigned long long)((cz + dz) * 83492791LL);
          const int b = (int)(h % (unsigned long long)n_buckets);
          for (int q = start[b]; q < start[b + 1]; ++q) {
            const int j = items[q];
            if (j == i) continue;
            const double ddx = xyz[3 * j] - X, ddy = xyz[3 * j + 1] - Y, ddz = xyz[3 * j + 2] - Z;
            if (ddx * ddx + ddy * ddy + ddz * ddz < r2) rep[j] = 1;
          }
        }
  }
}

// Shake.cpp:118-136: the ghost rule against the mean score of the non-repeated
// objects, which the reference sums in index order.  The flags are first decided with
// a tree-summed mean; a score within the bound by which the sequential and the tree
// sum can differ (|S_seq - S_tree| <= 2 n 2^-53 sum|x|) of the threshold marks the
// result ambiguous, and only then does ghost_kernel redo the sequential sum.
constexpr int kScoreBlocks = 296;

__global__ void score_partial_kernel(const double* score, const uint8_t* rep, int n,
                                     double* part) {
  __shared__ double s1[256], s2[256], s3[256];
  double a = 0.0, b = 0.0, c = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (!rep[i]) {
      a += score[i];
      b += fabs(score[i]);
      c += 1.0;
    }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = b;
  s3[threadIdx.x] = c;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) {
      s1[threadIdx.x] += s1[threadIdx.x + k];
      s2[threadIdx.x] += s2[threadIdx.x + k];
      s3[threadIdx.x] += s3[threadIdx.x + k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = s1[0];
    part[3 * blockIdx.x + 1] = s2[0];
    part[3 * blockIdx.x + 2] = s3[0];
  }
}

__global__ void ghost_flag_kernel(const double* score, const uint8_t* rep, int n, double thred,
                                  const double* part, int nb, uint8_t* flags, int* amb) {
  __shared__ double st[3];
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int b = 0; b < nb; ++b) t += part[3 * b + threadIdx.x];
    st[threadIdx.x] = t;
  }
  __syncthreads();
  const double cnt = st[2];
  const double m = cnt > 0 ? st[0] / cnt : 0.0;
  const double thr = m * thred;
  const double e = cnt > 0 ? (2.0 * (double)n * 1.1102230246251565e-16 * st[1]) / cnt : 0.0;
  const double band = 2.0 * (e * fabs(thred) + fabs(thr) * 4.5e-16);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double sc = score[i];
  uint8_t f = rep[i] ? 2 : 0;
  if (sc == 0.0 || sc < thr - band) {
    f |= 1;
  } else if (!(sc >= thr + band)) {
    atomicOr(amb, 1);
    if (sc < thr) f |= 1;
  }
  flags[i] = f;
}

__global__ void ghost_kernel(const double* score, const uint8_t* rep, int n, double thred,
                             uint8_t* flags, const int* amb) {
  if (!*amb) return;
  __shared__ double s_mean;
  if (threadIdx.x < 32) {
    // warp 0 streams the scores in; lane 0 adds them strictly in index order
    const int lane = threadIdx.x;
    double sum = 0.0;
    long long cnt = 0;
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      const bool valid = i < n && !rep[i];
      const double x = valid ? score[i] : 0.0;
      const unsigned ball = __ballot_sync(0xffffffffu, valid);
#pragma unroll 4
      for (int j = 0; j < 32; ++j) {
        const double y = __shfl_sync(0xffffffffu, x, j);
        if (lane == 0 && (ball >> j) & 1u) sum += y;
      }
      cnt += __popc(ball);
    }
    if (lane == 0) s_mean = cnt ? sum / (double)cnt : 0.0;
  }
  __syncthreads();
  const double m = s_mean;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    uint8_t f = rep[i] ? 2 : 0;
    if (score[i] < m * thred || score[i] == 0.0) f |= 1;
    flags[i] = f;
  }
}

// has_nb[i] is 0 or 1 after neighbour_kernel; pos = exclusive scan of it
__global__ void compact_kernel(const int* flag, const int* pos, int n, int* list) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && flag[i]) list[pos[i]] = i;
}

__global__ void fill_kernel(double* p, int64_t n, double v) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

}  // namespace

// ---------------------------------------------------------------- host drivers
// ---------------------------------------------------------------- learned shake
// correction in units of scale (mm); keep = not a ghost by the network's logit
__global__ void learned_apply_kernel(double* xyz, const float* o, int64_t n, double scale,
                                     float ghost_logit, int* keep) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* oi = o + 4 * i;
  const bool fin = isfinite(oi[0]) && isfinite(oi[1]) && isfinite(oi[2]) && isfinite(oi[3]);
  if (fin)
    for (int d = 0; d < 3; ++d) xyz[3 * i + d] += (double)oi[d] * scale;
  keep[i] = (fin && oi[3] <= ghost_logit) ? 1 : 0;
}

__global__ void compact_xyz_kernel(const int* keep, const int* pos, int64_t n, const double* a,
                                   double* a_out, const double* b, double* b_out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || !keep[i]) return;
  const int64_t k = pos[i];
  for (int d = 0; d < 3; ++d) {
    a_out[3 * k + d] = a[3 * i + d];
    b_out[3 * k + d] = b[3 * i + d];
  }
}

// objects whose residue after the refinement, divided by the mean squared OTF
// amplitude over the active cameras, exceeds thr (or is not finite) restart the
// full shake from their stereo position
template <typename Real>
__global__ void fallback_kernel(const double* res, const Real* otfp, const CamDev* cams, int C,
                                int64_t n, double thr, uint8_t* act, double* xyz,
                                const double* start, double* score, int* count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a2 = 0.0;
  int k = 0;
  for (int c = 0; c < C; ++c) {
    if (!cams[c].is_active) continue;
    const double a = (double)otfp[(i * C + c) * 5];
    a2 += a * a;
    ++k;
  }
  a2 = k > 0 ? a2 / k : 1.0;
  const double r = res[i] / (a2 > 1e-12 ? a2 : 1e-12);
  const bool fb = !(r <= thr);
  act[i] = fb ? 1 : 0;
  if (fb) {
    for (int d = 0; d < 3; ++d) xyz[3 * i + d] = start[3 * i + d];
    score[i] = 1.0;
    atomicAdd(count, 1);
  }
}

// refined objects carry a score over refine_loops iterations: bring it to the
// n_shake_loop scale of the plain schedule
__global__ void score_scale_kernel(double* score, const uint8_t* act, int64_t n, double expo) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n || act[i]) return;
  score[i] = pow(score[i], expo);
}

static ShakeView make_view(olpt_ctx* ctx, const ShakeParams& sp) {
  ShakeView v{};
  v.n_cam = ctx->n_cam;
  v.cams = ctx->cams_d.as<CamDev>();
  v.otf = otf_view(ctx);
  v.r_px = sp.radius_obj;
  v.ratio = (double)sp.ratio_augimg;
  const int side = (int)std::lround(2.0 * sp.radius_obj * sp.ratio_augimg);
  OLPT_REQUIRE(side >= 1 && side <= 16, OLPT_ERR_UNSUPPORTED,
               "augmented ROI side round(2 * radius_obj * ratio_augimg) must be in [1, 16]");
  v.roi_area = side * side;
  const int win = (int)std::lround(2.0 * sp.radius_obj);
  OLPT_REQUIRE(win >= 1 && win < 32, OLPT_ERR_UNSUPPORTED,
               "projection window round(2 * radius_obj) must be below 32 px");
  for (int c = 0; c < ctx->n_cam; ++c) {
    const CamDev& cm = ctx->cams_h[c];
    const ImagePlane& im = ctx->img[c];
    OLPT_REQUIRE(im.buf.p, OLPT_ERR_INVALID_ARG, "no image for camera");
    OLPT_REQUIRE(im.H == cm.n_row && im.W == cm.n_col, OLPT_ERR_INVALID_ARG,
                 "image size differs from the camera's n_row x n_col");
    v.orig[c] = PlaneView{im.buf.as<unsigned char>(), im.pitch, im.H, im.W, im.dtype};
  }
  for (int c = 0; c < ctx->n_cam; ++c) {
    const CamDev& cm = ctx->cams_h[c];
    if (cm.type == CAM_POLYNOMIAL && cm.pow3) v.n_poly = std::max(v.n_poly, cm.n_coeff);
  }
  v.cam_bytes = (cam_smem_bytes(v.n_poly) + 127) / 128 * 128;
  return v;
}

static void ensure_residual_planes(olpt_ctx* ctx, ShakeView& v, bool fp64) {
  const int dt = fp64 ? OLPT_F64 : OLPT_F32;
  const int esz = fp64 ? 8 : 4;
  for (int c = 0; c < ctx->n_cam; ++c) {
    ImagePlane& r = ctx->resid[c];
    const CamDev& cm = ctx->cams_h[c];
    const int64_t pitch = ((int64_t)cm.n_col * esz + 15) / 16 * 16;
    r.buf.ensure((size_t)pitch * cm.n_row + 64, ctx->stream);
    r.dtype = dt;
    r.H = cm.n_row;
    r.W = cm.n_col;
    r.pitch = pitch;
    v.res[c] = PlaneView{r.buf.as<unsigned char>(), r.pitch, r.H, r.W, dt};
  }
}

// Projection planes: zero between passes (the residual kernel leaves them so); allocated and
// zeroed when the geometry or the type changes, or when a pass did not get to its end.
static void ensure_projection_planes(olpt_ctx* ctx, ShakeView& v, bool fp64) {
  ShakeWork& W = ctx->shk;
  const int esz = fp64 ? 8 : 4;
  int64_t need = 0;
  for (int c = 0; c < ctx->n_cam; ++c) need += v.res[c].pitch * v.res[c].H;
  bool same = W.proj_clean && W.proj_esz == esz && W.proj_bytes == need;
  W.proj.ensure((size_t)need + 64, ctx->stream);
  if (!same || W.proj.p != W.proj_at)
    OLPT_CUDA(cudaMemsetAsync(W.proj.p, 0, (size_t)need, ctx->stream));
  W.proj_at = W.proj.p;
  W.proj_esz = esz;
  W.proj_bytes = need;
  int64_t off = 0;
  for (int c = 0; c < ctx->n_cam; ++c) {
    v.proj[c] = v.res[c];
    v.proj[c].p = W.proj.as<unsigned char>() + off;
    off += v.res[c].pitch * v.res[c].H;
  }
}

template <typename Real>
static void residual_pass(olpt_ctx* ctx, ShakeView& v, const uint8_t* flags, int all_cams,
                          int clamp) {
  cudaStream_t s = ctx->stream;
  ShakeWork& W = ctx->shk;
  const int64_t n = ctx->obj.n;
  const int C = ctx->n_cam;
  W.otfp.ensure((n * C + 1) * 5 * sizeof(Real), s);
  ensure_projection_planes(ctx, v, sizeof(Real) == 8);
  W.proj_clean = false;
  // 32 pairs a warp where that gives the SMs 16 warps each, else so few (down to 2) that it does:
  // a warp takes its windows one after the other (up to 9,000 objects on four cameras: 21 -> 12
  // us a launch; above 75,000 pairs the rule gives 32 and nothing changes)
  int per_warp = 32;
  while (per_warp > 2 && n * C < (int64_t)per_warp * 148 * 16) per_warp /= 2;
  if (n > 0)
    splat_kernel<Real><<<OLPT_G(nblk(n * C, 8 * per_warp)), 256, 0, s>>>(
        v, ctx->obj.xyz.as<double>(), n, ctx->obj.uv.as<double>(), W.otfp.as<Real>(), flags,
        all_cams, per_warp);
  OLPT_CUDA(cudaGetLastError());
  // algorithmic bytes: read the image, write the residual, for every computed camera
  double bytes = 0;
  int rows = 1, cols = 1;
  for (int c = 0; c < C; ++c) {
    rows = std::max(rows, v.orig[c].H);
    cols = std::max(cols, v.orig[c].W);
    if (!(all_cams || ctx->cams_h[c].is_active)) continue;
    const int d = v.orig[c].dtype;
    const int esz = d == OLPT_U8 ? 1 : d == OLPT_U16 ? 2 : d == OLPT_F32 ? 4 : 8;
    bytes += (double)v.orig[c].H * v.orig[c].W * (esz + sizeof(Real));
  }
  const int pid = ctx->prof.begin(PROF_RESIDUAL, s);
  const int t = ctx->tune.residual_threads;
  for (int y = 0; y < rows; y += 65535) {
    // one grid row per image row (a second launch past the grid's 65,535 rows)
    ShakeView part = v;
    if (y > 0)
      for (int c = 0; c < C; ++c) {
        for (PlaneView* p : {&part.orig[c], &part.proj[c], &part.res[c]}) {
          p->p += (int64_t)y * p->pitch;
          p->H = std::max(0, p->H - y);
        }
      }
    const dim3 grid((unsigned)nblk((cols + 3) / 4, t), (unsigned)std::min(rows - y, 65535), C);
    residual_kernel<Real><<<OLPT_G(grid), t, 0, s>>>(part, clamp, all_cams);
  }
  ctx->prof.end(PROF_RESIDUAL, pid, s, bytes);
  OLPT_CUDA(cudaGetLastError());
  W.proj_clean = true;
}

// Shared memory of one object's arrays (struct Obj).  The stride between the objects of a
// warp is the groups' share of the 32 banks, so that their equal offsets do not collide.
static void shake_layout(ShakeView& v, int lpo, bool fp64) {
  const size_t rsz = fp64 ? 8 : 4;
  auto up = [](size_t x) { return (x + 15) / 16 * 16; };
  size_t off = up((size_t)v.n_cam * v.roi_area * rsz);
  v.off_dd = off;
  if (fp64) off = up(off + 3 * (size_t)v.n_cam * (v.roi_area + 1) * 8);
  v.off_uv = off;
  off += 3 * (size_t)v.n_cam * 16;
  v.off_roi = off;
  off += (size_t)v.n_cam * 16;
  v.off_ey = off;
  off += 3 * 8 * rsz;
  v.off_otf = off;
  off += 3 * (size_t)v.n_cam * 5 * rsz;
  v.off_win = off;
  off = up(off + 3 * (size_t)v.n_cam * 4);
  v.off_pw = off;
  if (v.n_poly > 0) off += 3 * 12 * 8;
  const size_t share = std::min<size_t>((size_t)lpo * rsz, 64) % 128;
  while (off % 128 != share) off += 16;
  v.obj_stride = off;
}

template <typename Real, int NC, int LPO>
static void launch_shake(int warps, cudaStream_t s, const ShakeView& v, int64_t n, double* xyz,
                         double* uv, const Real* otfp, double* score, double delta,
                         const uint8_t* active, double* resid_out) {
  const size_t per_warp = v.obj_stride * (32 / LPO);
  while (warps > 1 && v.cam_bytes + per_warp * warps > kShakeSmemMax) warps /= 2;
  const size_t smem = v.cam_bytes + per_warp * warps;
  allow_smem<shake_kernel<Real, NC, LPO>>(smem);
  shake_kernel<Real, NC, LPO><<<OLPT_G(nblk(n, warps * (32 / LPO))), 32 * warps, smem, s>>>(
      v, n, xyz, uv, otfp, score, delta, active, resid_out);
}

// Lanes per object.  FP32, ROIs of up to 64 pixels: 8 once a wave of one-object warps (148 SMs x
// 16) no longer holds the objects, else 32 -- a lone object finishes sooner with more lanes.
// Measured per launch (4 pinhole cameras): 2,000 objects 77 us with 8 lanes, 75 us with 32;
// 3,500: 84 and 148 us; 20,000: 257 and 544 us.  Larger ROIs take their lanes through the pixels
// either way, so 8 lanes pay from the third wave on, and only where four blocks (what the
// registers allow) also find their ROIs' shared memory: 20,000 objects, ROIs of 100 pixels 759 and
// 827 us, of 196 (three blocks) 1,277 and 1,097, of 256 on eight cameras (one block) 7,139 and
// 1,989.  FP64: 32 always; its squared differences take 3 x 8 B per ROI pixel, so shared memory
// holds too few 8-lane groups (32,000 objects: 1,879 us with 8, 1,382 with 32).
constexpr int64_t kWaveObjects = 148 * 16;
constexpr size_t kSmSmem = 228 * 1024;  // of an SM, 1 KB a block reserved

template <typename Real, int NC>
static void launch_shake_nc(int warps, cudaStream_t s, ShakeView& v, int64_t n, double* xyz,
                            double* uv, const Real* otfp, double* score, double delta,
                            const uint8_t* active, double* resid_out) {
  if constexpr (sizeof(Real) == 4) {
    shake_layout(v, 8, false);
    const bool eight = v.roi_area <= 64
                           ? n > kWaveObjects && v.cam_bytes + 4 * v.obj_stride <= kShakeSmemMax
                           : n > 2 * kWaveObjects &&
                                 4 * (v.cam_bytes + 16 * v.obj_stride + 1024) <= kSmSmem;
    if (eight) {
      launch_shake<Real, NC, 8>(warps, s, v, n, xyz, uv, otfp, score, delta, active,
                                      resid_out);
      return;
    }
  }
  shake_layout(v, 32, sizeof(Real) == 8);
  launch_shake<Real, NC, 32>(warps, s, v, n, xyz, uv, otfp, score, delta, active,
                                   resid_out);
}

template <typename Real>
static void launch_shake_cams(int warps, cudaStream_t s, ShakeView& v, int64_t n, double* xyz,
                              double* uv, const Real* otfp, double* score, double delta,
                              const uint8_t* active, double* resid_out) {
  switch (v.n_cam) {
    case 2: launch_shake_nc<Real, 2>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    case 3: launch_shake_nc<Real, 3>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    case 4: launch_shake_nc<Real, 4>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    case 5: launch_shake_nc<Real, 5>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    case 6: launch_shake_nc<Real, 6>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    case 7: launch_shake_nc<Real, 7>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
    default: launch_shake_nc<Real, 8>(warps, s, v, n, xyz, uv, otfp, score, delta, active, resid_out); break;
  }
}

// n_loop shake iterations from the width delta (halved per iteration, clamped at the
// minimum); objects with active[o] == 0 stay fixed but still enter the residual
template <typename Real>
static void shake_iterations(olpt_ctx* ctx, const ShakeParams& sp, ShakeView& v, int n_loop,
                             double delta, const uint8_t* active, double* resid_out) {
  cudaStream_t s = ctx->stream;
  const int64_t n = ctx->obj.n;
  const int C = ctx->n_cam;
  ShakeWork& W = ctx->shk;
  double dmin = sp.shakewidth_min;
  dmin = (dmin > 0) ? dmin : sp.shake_width / 20;
  const int warps_per_blk = ctx->tune.shake_warps_per_block;  // 1, 2 or 4 (bound: 128 threads)

  for (int it = 0; it < n_loop; ++it) {
    residual_pass<Real>(ctx, v, nullptr, 0, 0);
    // algorithmic bytes: the augmented ROI of every active camera plus the object
    // state (xyz, projections, OTF parameters, score) read and written once
    int n_act = 0;
    for (int c = 0; c < C; ++c) n_act += ctx->cams_h[c].is_active;
    const double bytes = (double)n * (n_act * v.roi_area * (double)sizeof(Real) +
                                      2.0 * (3 * 8 + C * 2 * 8 + 8) + C * 5.0 * sizeof(Real));
    const int pid = ctx->prof.begin(PROF_SHAKE, s);
    const double x3[3] = {-delta, 0.0, delta};
    double B[3][4];
    parabola_matrix(x3, 3, B);
    for (int r = 0; r < 2; ++r)
      for (int i = 0; i < 3; ++i) v.fit3[r][i] = B[r + 1][i];
    if (n > 0)
      launch_shake_cams<Real>(warps_per_blk, s, v, n, ctx->obj.xyz.as<double>(),
                              ctx->obj.uv.as<double>(), W.otfp.as<Real>(),
                              ctx->obj.score.as<double>(), delta, active, resid_out);
    ctx->prof.end(PROF_SHAKE, pid, s, bytes);
    OLPT_CUDA(cudaGetLastError());
    delta *= 0.5;
    if (delta < dmin) delta = dmin;
  }
}

// Shake::runShake (Shake.cpp:103-136): repeated objects (greedy over the tol_3d
// neighbourhood) and ghosts (score below thred_ghost x mean score)
static void shake_flags(olpt_ctx* ctx, const ShakeParams& sp) {
  cudaStream_t s = ctx->stream;
  const int64_t n = ctx->obj.n;
  ShakeWork& W = ctx->shk;
  W.rep.ensure(n + 16, s);
  OLPT_CUDA(cudaMemsetAsync(W.rep.p, 0, n + 16, s));
  if (n > 0) {
    const double cell = std::max(sp.tol_3d_mm, 1e-9);
    const int nb = (int)std::max<int64_t>(1024, 2 * n);
    W.hkey.ensure((n + 1) * sizeof(int), s);
    W.has_nb.ensure((n + 1) * sizeof(int), s);
    hash_key_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.xyz.as<double>(), (int)n, cell, nb,
                                             W.hkey.as<int>());
    W.hash.build(W.hkey.as<int>(), (int)n, nb, s);
    const double r2 = sp.tol_3d_mm * sp.tol_3d_mm;
    neighbour_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.xyz.as<double>(), (int)n, cell, nb,
                                              W.hash.start.as<int>(), W.hash.items.as<int>(), r2,
                                              W.has_nb.as<int>());
    // ascending list of the objects that have neighbours (order-preserving compaction)
    W.nb_pos.ensure((n + 1) * sizeof(int), s);
    W.nb_list.ensure((n + 1) * sizeof(int), s);
    exclusive_scan(W.has_nb.as<int>(), (int)n, W.nb_pos.as<int>(), W.scan_tmp, s);
    compact_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(W.has_nb.as<int>(), W.nb_pos.as<int>(), (int)n,
                                                  W.nb_list.as<int>());
    repeat_greedy_kernel<<<OLPT_G(1), 32, 0, s>>>(ctx->obj.xyz.as<double>(), (int)n, cell, nb,
                                          W.hash.start.as<int>(), W.hash.items.as<int>(), r2,
                                          W.nb_list.as<int>(), W.nb_pos.as<int>() + n,
                                          W.rep.as<uint8_t>());
    const int sb = std::max(1, std::min(kScoreBlocks, nblk(n)));
    W.gpart.ensure((size_t)sb * 3 * sizeof(double) + sizeof(int) + 64, s);
    int* amb = reinterpret_cast<int*>(W.gpart.as<double>() + 3 * sb);
    OLPT_CUDA(cudaMemsetAsync(amb, 0, sizeof(int), s));
    score_partial_kernel<<<OLPT_G(sb), 256, 0, s>>>(ctx->obj.score.as<double>(),
                                                    W.rep.as<uint8_t>(), (int)n,
                                                    W.gpart.as<double>());
    ghost_flag_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.score.as<double>(),
                                                      W.rep.as<uint8_t>(), (int)n, sp.thred_ghost,
                                                      W.gpart.as<double>(), sb,
                                                      ctx->obj.flags.as<uint8_t>(), amb);
    ghost_kernel<<<OLPT_G(1), 1024, 0, s>>>(ctx->obj.score.as<double>(), W.rep.as<uint8_t>(), (int)n,
                                    sp.thred_ghost, ctx->obj.flags.as<uint8_t>(), amb);
    OLPT_CUDA(cudaGetLastError());
  }
}

template <typename Real>
static void shake_impl(olpt_ctx* ctx, const ShakeParams& sp) {
  const bool fp64 = sizeof(Real) == 8;
  cudaStream_t s = ctx->stream;
  ShakeView v = make_view(ctx, sp);
  ensure_residual_planes(ctx, v, fp64);
  const int64_t n = ctx->obj.n;
  ctx->obj.ensure(std::max<int64_t>(n, 1), ctx->n_cam, s);
  if (n > 0) fill_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.score.as<double>(), n, 1.0);
  shake_iterations<Real>(ctx, sp, v, sp.n_shake_loop, sp.shake_width, nullptr, nullptr);
  shake_flags(ctx, sp);
}

template <typename Real>
static void learned_impl(olpt_ctx* ctx, const ShakeParams& sp) {
  const bool fp64 = sizeof(Real) == 8;
  cudaStream_t s = ctx->stream;
  MlpWork& M = ctx->mlp;
  const LearnedParams& lp = M.lp;
  ShakeView v = make_view(ctx, sp);
  ensure_residual_planes(ctx, v, fp64);
  int64_t n = ctx->obj.n;
  const int C = ctx->n_cam;
  if (n > 0) {
    // 1. residual with every candidate at its stereo position, features, network
    residual_pass<Real>(ctx, v, nullptr, 0, 0);
    M.x.ensure((size_t)n * M.dims.in_pad * 2, s);
    mlp_features_device(ctx, sp, M.x.as<__nv_bfloat16>(), nullptr);
    M.o.ensure((size_t)n * kMlpOut * 4, s);
    mlp_infer_device(ctx, nullptr, M.x.as<__nv_bfloat16>(), n, M.o.as<float>());
    // 2. correction, and the network's ghosts leave before any shaking
    M.keep.ensure((size_t)(n + 1) * sizeof(int), s);
    M.pos.ensure((size_t)(n + 1) * sizeof(int), s);
    M.start_xyz.ensure((size_t)n * 3 * sizeof(double), s);
    OLPT_CUDA(cudaMemcpyAsync(M.start_xyz.p, ctx->obj.xyz.p, (size_t)n * 3 * sizeof(double),
                              cudaMemcpyDeviceToDevice, s));
    learned_apply_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.xyz.as<double>(), M.o.as<float>(),
                                                        n, lp.out_scale_mm, (float)lp.ghost_logit,
                                                        M.keep.as<int>());
    exclusive_scan(M.keep.as<int>(), (int)n, M.pos.as<int>(), ctx->shk.scan_tmp, s);
    const int kept = read_back(ctx, M.pos.as<int>() + n);
    // compacted copies (through the scratch pair act / nres, then back)
    M.act.ensure((size_t)(n + 1) * 3 * sizeof(double), s);
    M.nres.ensure((size_t)(n + 1) * 3 * sizeof(double), s);
    compact_xyz_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(
        M.keep.as<int>(), M.pos.as<int>(), n, ctx->obj.xyz.as<double>(), M.act.as<double>(),
        M.start_xyz.as<double>(), M.nres.as<double>());
    OLPT_CUDA(cudaGetLastError());
    n = kept;
    ctx->obj.n = n;
    if (n > 0) {
      OLPT_CUDA(cudaMemcpyAsync(ctx->obj.xyz.p, M.act.p, (size_t)n * 3 * sizeof(double),
                                cudaMemcpyDeviceToDevice, s));
      OLPT_CUDA(cudaMemcpyAsync(M.start_xyz.p, M.nres.p, (size_t)n * 3 * sizeof(double),
                                cudaMemcpyDeviceToDevice, s));
    }
  }
  ctx->obj.ensure(std::max<int64_t>(n, 1), C, s);
  if (n > 0) {
    // 3. short plain refinement from the corrected positions
    fill_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(ctx->obj.score.as<double>(), n, 1.0);
    M.nres.ensure((size_t)(n + 1) * sizeof(double), s);
    shake_iterations<Real>(ctx, sp, v, lp.refine_loops, lp.refine_width_mm, nullptr,
                           M.nres.as<double>());
    // 4. fallback: the full plain shake for objects whose residue stays high
    M.act.ensure((size_t)n + 16, s);
    M.fb.ensure(16, s);
    int* cnt = M.fb.as<int>();
    OLPT_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int), s));
    fallback_kernel<Real><<<OLPT_G(nblk(n)), 256, 0, s>>>(
        M.nres.as<double>(), ctx->shk.otfp.as<Real>(), ctx->cams_d.as<CamDev>(), C, n,
        lp.fallback_residual, M.act.as<uint8_t>(), ctx->obj.xyz.as<double>(),
        M.start_xyz.as<double>(), ctx->obj.score.as<double>(), cnt);
    OLPT_CUDA(cudaGetLastError());
    const int n_fb = read_back(ctx, cnt);
    M.n_fallback += n_fb;
    M.n_learned += n;
    if (n_fb > 0)
      shake_iterations<Real>(ctx, sp, v, sp.n_shake_loop, sp.shake_width, M.act.as<uint8_t>(),
                             nullptr);
    if (lp.refine_loops > 0 && lp.refine_loops != sp.n_shake_loop)
      score_scale_kernel<<<OLPT_G(nblk(n)), 256, 0, s>>>(
          ctx->obj.score.as<double>(), M.act.as<uint8_t>(), n,
          (double)sp.n_shake_loop / (double)lp.refine_loops);
    OLPT_CUDA(cudaGetLastError());
  }
  shake_flags(ctx, sp);
}

void residual_all_device(olpt_ctx* ctx, const ShakeParams& sp) {
  const bool fp64 = sp.precision == 1;
  ShakeView v = make_view(ctx, sp);
  ensure_residual_planes(ctx, v, fp64);
  if (fp64)
    residual_pass<double>(ctx, v, nullptr, 0, 0);
  else
    residual_pass<float>(ctx, v, nullptr, 0, 0);
}

void learned_shake_device(olpt_ctx* ctx, const ShakeParams& sp) {
  OLPT_REQUIRE(ctx->mlp.ready, OLPT_ERR_INVALID_ARG, "learned shake: network not initialised");
  OLPT_REQUIRE(ctx->n_cam == ctx->mlp.dims.cams, OLPT_ERR_UNSUPPORTED,
               "learned shake: the network was built for " + std::to_string(ctx->mlp.dims.cams) +
                   " cameras, the rig has " + std::to_string(ctx->n_cam));
  if (sp.precision == 1)
    learned_impl<double>(ctx, sp);
  else
    learned_impl<float>(ctx, sp);
}

void shake_device(olpt_ctx* ctx, const ShakeParams& sp) {
  OLPT_REQUIRE(ctx->n_cam >= 2, OLPT_ERR_INVALID_ARG, "shake needs at least 2 cameras");
  if (sp.precision == 1)
    shake_impl<double>(ctx, sp);
  else
    shake_impl<float>(ctx, sp);
}

// Shake::calResidualImage (output_ipr = true): every camera, clamped at 0, objects
// flagged Ghost/Repeated skipped when use_flags.  The result replaces the current
// images when make_current.
void residual_device(olpt_ctx* ctx, const ShakeParams& sp, bool use_flags, bool make_current) {
  const bool fp64 = sp.precision == 1;
  ShakeView v = make_view(ctx, sp);
  ensure_residual_planes(ctx, v, fp64);
  const uint8_t* fl = use_flags ? ctx->obj.flags.as<uint8_t>() : nullptr;
  if (fp64)
    residual_pass<double>(ctx, v, fl, 1, 1);
  else
    residual_pass<float>(ctx, v, fl, 1, 1);
  if (make_current)
    for (int c = 0; c < ctx->n_cam; ++c) std::swap(ctx->img[c], ctx->resid[c]);
}

}  // namespace olpt
