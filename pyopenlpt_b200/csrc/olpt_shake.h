// Shake: parameter block, kernel views and device workspace (shake.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include "olpt_otf.cuh"

namespace olpt {

struct ShakeParams {
  double shake_width;
  double shakewidth_min;
  int n_shake_loop;
  double thred_ghost;
  int ratio_augimg;
  double radius_obj;
  double tol_3d_mm;
  int precision;  // 0 = FP32 residual / OTF / line-search sums, 1 = FP64
};

struct PlaneView {
  unsigned char* p;
  int64_t pitch;  // bytes
  int H, W;
  int dtype;
};

struct ShakeView {
  int n_cam;
  const CamDev* cams;
  OtfView otf;
  double r_px, ratio;
  int roi_area;          // augmented ROI pixels (side^2)
  PlaneView orig[OLPT_MAX_CAM];  // current images (u8/u16/f32/f64)
  PlaneView res[OLPT_MAX_CAM];   // residual planes (Real)
  PlaneView proj[OLPT_MAX_CAM];  // projection planes (Real), 0 outside a pass
  int n_poly;            // most terms of a polynomial camera with exponents 0..3
  double fit3[2][3];     // linear and quadratic rows of the three-point parabola fit
  // shared memory of the shake kernel: the cameras' table, then the objects' arrays
  size_t cam_bytes, obj_stride, off_dd, off_uv, off_roi, off_ey, off_otf, off_win, off_pw;
};

}  // namespace olpt
