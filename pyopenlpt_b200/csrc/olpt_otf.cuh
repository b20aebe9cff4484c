// OTF table lookup on the device: OTF::getOTFParam (src/srcSTB/OTF.cpp:273-338)
// with myMATH::linspace grid nodes (myMATH.cpp:9-33) and myMATH::triLinearInterp
// (myMATH.cpp:131-214), evaluated in FP64 in the reference's operation order.
#pragma once
#include "olpt_device.cuh"

namespace olpt {

struct OtfView {
  int nx, ny, nz, n_grid, n_cam;
  double bmin[3], bmax[3], d[3];
  double inv_d[3];  // 1 / d
  // [n_cam][n_grid][4]: a, b, c, alpha of a node side by side, so that the two nodes of a
  // cell along z are one run of 64 bytes
  const double* table;
  // every alpha entry is +0.0: the interpolated angle is then +0.0 and its cosine and
  // sine are exactly 1 and +0 (the reference's values), so they are not evaluated
  int alpha_zero;
};

__device__ __forceinline__ double otf_lerp8(const double* v, double xd, double yd, double zd) {
  // v: c000, c100, c101, c001, c010, c110, c111, c011 (OTF.cpp:312-317 order)
  double c00 = v[0] * (1 - xd) + v[1] * xd;
  double c01 = v[3] * (1 - xd) + v[2] * xd;
  double c10 = v[4] * (1 - xd) + v[5] * xd;
  double c11 = v[7] * (1 - xd) + v[6] * xd;
  double c0 = c00 * (1 - yd) + c10 * yd;
  double c1 = c01 * (1 - yd) + c11 * yd;
  return c0 * (1 - zd) + c1 * zd;
}

// out: a, b, c, cos(alpha), sin(alpha)
__device__ __forceinline__ void otf_param(const OtfView& o, int cam, double X, double Y, double Z,
                                          double out[5]) {
  const double P[3] = {X, Y, Z};
  const int n[3] = {o.nx, o.ny, o.nz};
  double p[3], lo[3], hi[3];
  int id[3];
  for (int k = 0; k < 3; ++k) {
    p[k] = fmin(fmax(P[k], o.bmin[k]), o.bmax[k]);
    const double off = p[k] - o.bmin[k];
    // the cell floor(off / d): off * (1 / d) is within a few ulp of the quotient, so only a
    // product next to an integer needs the division
    double q = off * o.inv_d[k];
    if (!(fabs(q - rint(q)) > 1e-9 * (1.0 + fabs(q)))) q = off / o.d[k];
    int i = (int)floor(q);
    i = i < 0 ? 0 : i;
    i = i > n[k] - 2 ? n[k] - 2 : i;
    id[k] = i;
    lo[k] = o.bmin[k] + o.d[k] * i;  // d = (bmax - bmin) / (n - 1): the nodes' spacing
    hi[k] = o.bmin[k] + o.d[k] * (i + 1);
  }
  double t[3];
  for (int k = 0; k < 3; ++k) {
    double v = (p[k] - lo[k]) / (hi[k] - lo[k]);
    t[k] = fmax(0.0, fmin(1.0, v));
  }
  // corners in the order of otf_lerp8 (OTF.cpp:312-317)
  const int nyz = o.ny * o.nz;
  const double* base =
      o.table + 4 * ((int64_t)cam * o.n_grid + (id[0] * nyz + id[1] * o.nz + id[2]));
  double c[4][8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    // c000, c100, c101, c001, c010, c110, c111, c011
    constexpr int X[8] = {0, 1, 1, 0, 0, 1, 1, 0}, Y[8] = {0, 0, 0, 0, 1, 1, 1, 1},
                  Z[8] = {0, 0, 1, 1, 0, 0, 1, 1};
    const double2* n2 =
        reinterpret_cast<const double2*>(base + 4 * (X[k] * nyz + Y[k] * o.nz + Z[k]));
    const double2 ab = n2[0], ca = n2[1];
    c[0][k] = ab.x;
    c[1][k] = ab.y;
    c[2][k] = ca.x;
    c[3][k] = ca.y;
  }
  double res[4];
#pragma unroll
  for (int q = 0; q < 3; ++q) res[q] = otf_lerp8(c[q], t[0], t[1], t[2]);
  if (!o.alpha_zero) res[3] = otf_lerp8(c[3], t[0], t[1], t[2]);
  out[0] = res[0];
  out[1] = res[1];
  out[2] = res[2];
  if (o.alpha_zero) {
    out[3] = 1.0;
    out[4] = 0.0;
  } else {
    out[3] = cos(res[3]);
    out[4] = sin(res[3]);
  }
}

}  // namespace olpt
