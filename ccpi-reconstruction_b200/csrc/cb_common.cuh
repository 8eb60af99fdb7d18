// Definitions shared by the cone-beam projector translation units.
#pragma once

#include "common.cuh"

namespace ccpi {

__device__ __forceinline__ double cb_dmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double cb_dmin(double a, double b) { return (b < a) ? b : a; }
// std::min(a, b) as the reference evaluates it: (b < a) ? b : a.  Every
// call passes b = a ray's exit alpha, which is never NaN and never -0, and
// for such b the NaN-propagating hardware minimum returns the same value for
// every a (NaN a gives NaN, +-0 a with b > 0 gives a), in one instruction
// instead of a compare and a select.
__device__ __forceinline__ float fmin_ref(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Floats of a slice-plane table in shared memory (nz + 1 entries, rounded up
// to 4).
__host__ __device__ inline int cb_vz_floats(int nz) { return (nz + 1 + 3) & ~3; }

// Detector columns [hmin, hmax] whose rays can cross voxel column
// [x0,xn) x [y0,yn) at angle a (c2D.cpp:831-895): the projections of its
// four corners.
__device__ __forceinline__ void cb_column_hrange(const Geom &g, int a, double x0, double xn,
                                                 double y0, double yn, int &hmin, int &hmax) {
  const double c = g.cosA[a], s = g.sinA[a];
  const double p1x = g.p1x[a], p1y = g.p1y[a];
  const double dx0 = x0 - p1x, dy0 = y0 - p1y, dxn = xn - p1x, dyn = yn - p1y;
  const double cx0 = c * x0 - g.src[0], cxn = c * xn - g.src[0];
  const double sy0 = s * y0, syn = s * yn;
  double y00, y01, y10, y11;
  if (fabs(s) > fabs(c)) {
    const double il = g.cl / s;
    y00 = (c - dx0 / (sy0 + cx0)) * il;
    y01 = (c - dx0 / (syn + cx0)) * il;
    y10 = (c - dxn / (sy0 + cxn)) * il;
    y11 = (c - dxn / (syn + cxn)) * il;
  } else {
    const double il = g.cl / c;
    y00 = (-s + dy0 / (cx0 + sy0)) * il;
    y01 = (-s + dyn / (cx0 + syn)) * il;
    y10 = (-s + dy0 / (cxn + sy0)) * il;
    y11 = (-s + dyn / (cxn + syn)) * il;
  }
  const int h00 = int(floor(y00 * g.cipix + g.chpix0));
  const int h01 = int(floor(y01 * g.cipix + g.chpix0));
  const int h10 = int(floor(y10 * g.cipix + g.chpix0));
  const int h11 = int(floor(y11 * g.cipix + g.chpix0));
  hmin = max(min(min(h00, h01), min(h10, h11)), 0);
  hmax = min(max(max(h00, h01), max(h10, h11)), g.nh - 1);
}

// Rays (angle a, columns h) crossing voxel column [x0,xn) x [y0,yn), with
// their entry/exit alphas (bproject_ah, c2D.cpp:831-936).  Calls f(h, a0, a1).
template <class F>
__device__ void cb_column_rays(const Geom &g, int a, double x0, double xn, double y0,
                               double yn, F &&f) {
  const double eps = double(kEps);
  const double c = g.cosA[a], s = g.sinA[a];
  const double p1x = g.p1x[a], p1y = g.p1y[a];
  const double dx0 = x0 - p1x, dy0 = y0 - p1y, dxn = xn - p1x, dyn = yn - p1y;
  int hmin, hmax;
  cb_column_hrange(g, a, x0, xn, y0, yn, hmin, hmax);
  for (int h = hmin; h <= hmax; h++) {
    const double p2x = g.cdx[a] - s * g.hpix[h];
    const double p2y = g.sdx[a] + c * g.hpix[h];
    const double ddx = p2x - p1x, ddy = p2y - p1y;
    if (fabs(ddx) < eps || fabs(ddy) < eps)
      continue; // rejected by the reference ("Ooops", c2D.cpp:909-912)
    const double idx = 1.0 / ddx, idy = 1.0 / ddy;
    const double ax0 = dx0 * idx, ay0 = dy0 * idy, axn = dxn * idx, ayn = dyn * idy;
    const double amin =
        cb_dmax(cb_dmax(cb_dmin(ax0, axn), cb_dmin(ay0, ayn)), 0.0);
    const double amax =
        cb_dmin(cb_dmin(cb_dmax(ax0, axn), cb_dmax(ay0, ayn)), 1.0);
    if (amin < amax - eps)
      f(h, float(amin), float(amax));
  }
}

} // namespace ccpi
