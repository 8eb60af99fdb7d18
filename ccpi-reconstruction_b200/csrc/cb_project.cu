// Cone-beam projectors for sm_100a.
//
// Forward (cone_beam::f2D, Core/src/c2D.cpp:469-625): ray-driven.  One warp
// owns one ray (angle a, detector column h).  The warp walks the ray's xy
// Siddon path once in voxel-normalised coordinates (c2D.cpp:193-467, FP64
// geometry, alphas rounded to float exactly as the reference stores them)
// and stages the (alpha, column) list in its own slice of shared memory.
// The lanes then own detector rows v and replay the list: each xy segment is
// split across at most two z slices with the reference's float arithmetic
// and its three row regimes (all-inside, lower edge, upper edge;
// c2D.cpp:17-191), and the row is finally scaled by the source-pixel
// distance.  Per row the additions happen in the reference's order with
// unfused float operations, so the result matches the reference bit for bit.
//
// Backward (cone_beam::b2D, c2D.cpp:948-1119): the ray-driven scatter, whose
// additions into a voxel have no fixed order (two forms, see below), and the
// plan's table of every voxel column's band.  The gathers in the reference's
// order, bit for bit, are in cb_back.cu.
#include <algorithm>

#include "cb_common.cuh"
#include "kernels.h"

namespace ccpi {
namespace {

__device__ __forceinline__ float lds_f(unsigned a) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}

__device__ __forceinline__ double dmax(double a, double b) { return cb_dmax(a, b); }
__device__ __forceinline__ double dmin(double a, double b) { return cb_dmin(a, b); }

// xy walk of ray p1 -> p2 over the whole volume; writes alphas[0..n-1] and
// cells[0..n-2] (x*ny + y, or -1) with lane 0; returns n (0 if missed).
__device__ int cb_walk(const Geom &g, double p1x, double p1y, double p2x, double p2y,
                       float *alphas, int *cells, int cap) {
  const double eps = double(kEps);
  const int nx = g.nx, ny = g.ny;
  const bool w = (threadIdx.x & 31) == 0;
  const double q1x = (p1x - g.origin[0]) / g.size[0];
  const double q1y = (p1y - g.origin[1]) / g.size[1];
  const double q2x = (p2x - g.origin[0]) / g.size[0];
  const double q2y = (p2y - g.origin[1]) / g.size[1];
  const double ddx = q2x - q1x, ddy = q2y - q1y;
  const double idx = 1.0 / ddx, idy = 1.0 / ddy;
  int n = 0;
  if (fabs(ddx) < eps) {
    if (fabs(ddy) < eps)
      return 0;
    const int i = int(floor(q1x));
    if (i < 0 || i >= nx)
      return 0;
    if (ddy < 0.0) {
      if (w)
        alphas[0] = float((double(ny) - q1y) * idy);
      for (int j = ny - 1; j >= 0; j--) {
        if (w) {
          alphas[ny - j] = float((double(j) - q1y) * idy);
          cells[ny - 1 - j] = i * ny + j;
        }
      }
    } else {
      if (w)
        alphas[0] = float((0.0 - q1y) * idy);
      for (int j = 0; j < ny; j++) {
        if (w) {
          alphas[j + 1] = float((double(j + 1) - q1y) * idy);
          cells[j] = i * ny + j;
        }
      }
    }
    return ny + 1;
  }
  if (fabs(ddy) < eps) {
    const int j = int(floor(q1y));
    if (j < 0 || j >= ny)
      return 0;
    if (ddx < 0.0) {
      if (w)
        alphas[0] = float((double(nx) - q1x) * idx);
      for (int i = nx - 1; i >= 0; i--) {
        if (w) {
          alphas[nx - i] = float((double(i) - q1x) * idx);
          cells[nx - 1 - i] = i * ny + j;
        }
      }
    } else {
      if (w)
        alphas[0] = float((0.0 - q1x) * idx);
      for (int i = 0; i < nx; i++) {
        if (w) {
          alphas[i + 1] = float((double(i + 1) - q1x) * idx);
          cells[i] = i * ny + j;
        }
      }
    }
    return nx + 1;
  }
  const double ax0 = (0.0 - q1x) * idx, ay0 = (0.0 - q1y) * idy;
  const double axn = (double(nx) - q1x) * idx, ayn = (double(ny) - q1y) * idy;
  const double amin = dmax(dmax(dmin(ax0, axn), dmin(ay0, ayn)), 0.0);
  const double amax = dmin(dmin(dmax(ax0, axn), dmax(ay0, ayn)), 1.0);
  if (!(amin < amax - eps))
    return 0;
  const int sx = ddx > 0.0 ? 1 : -1, sy = ddy > 0.0 ? 1 : -1;
  int x = 0, y = 0;
  const bool x_face_first = !(sx > 0 && sy < 0);
  const double axe = sx > 0 ? ax0 : axn, aye = sy > 0 ? ay0 : ayn;
  auto cx = [&]() { return int(floor(q1x + amin * ddx)); };
  auto cy = [&]() { return int(floor(q1y + amin * ddy)); };
  if (x_face_first) {
    if (amin == axe) {
      x = sx > 0 ? 0 : nx - 1;
      y = (sx < 0 && sy < 0 && amin == ayn) ? ny - 1 : cy();
    } else if (amin == aye) {
      x = cx();
      y = sy > 0 ? 0 : ny - 1;
    }
  } else {
    if (amin == aye) {
      x = cx();
      y = ny - 1;
    } else if (amin == axe) {
      x = 0;
      y = cy();
    }
  }
  if (w)
    alphas[0] = float(amin);
  n = 1;
  while ((sx > 0 ? x < nx : x >= 0) && (sy > 0 ? y < ny : y >= 0) && n < cap) {
    const double nxa = (double(sx > 0 ? x + 1 : x) - q1x) * idx;
    const double nya = (double(sy > 0 ? y + 1 : y) - q1y) * idy;
    const int cell = (x >= 0 && x < nx && y >= 0 && y < ny) ? x * ny + y : -1;
    double an;
    if (nxa < nya - eps) {
      an = nxa;
      x += sx;
    } else if (nya < nxa - eps) {
      an = nya;
      y += sy;
    } else {
      an = dmax(nxa, nya);
      x += sx;
      y += sy;
    }
    if (w) {
      cells[n - 1] = cell;
      alphas[n] = float(an);
    }
    n++;
  }
  return n;
}

template <int EPI>
__device__ __forceinline__ float cb_fp_epi(float acc, i64 idx, const Epi &e, double &ssq) {
  if (EPI == EPI_NORM) {
    ssq += double(acc) * double(acc);
    return acc;
  } else if (EPI == EPI_SIRT) {
    return __fmul_rn(__fadd_rn(-acc, e.b[idx]), e.w[idx]);
  } else if (EPI == EPI_MLEM) {
    const float q = (acc != 0.0f) ? __fdiv_rn(e.b[idx], acc) : 0.0f;
    return (q < 0.0f) ? 0.0f : q;
  }
  return acc;
}

constexpr int kFpWarps = 4;

// Row regimes of a walked ray (c2D.cpp:45-99), evaluated warp-parallel:
// cells [1, ncom) have every row's slice and its neighbour inside the
// column; rows [min_v_all, max_v_all] stay inside it for every cell.
__device__ __forceinline__ void cb_row_regimes(const Geom &g, const float *alphas, int n,
                                               int lane, int &ncom, int &min_v_all,
                                               int &max_v_all) {
  const int nzm1 = g.nz - 1, mid = g.mid;
  const float pzbz = g.pzbz, inv_dz = g.inv_dz;
  ncom = 0;
  min_v_all = mid;
  max_v_all = mid - 1;
  if (n < 2)
    return;
  int min_xy_all = n, max_xy_all = n;
  const float dz0 = g.dz[0], dzl = g.dz[g.nv - 1];
  bool got_lo = false, got_hi = false;
  for (int m0 = 1; m0 < n && !(got_lo && got_hi); m0 += 32) {
    const int m = m0 + lane;
    int klo = 1, khi = nzm1 - 1;
    if (m < n) {
      const float av = __fmul_rn(alphas[m - 1], inv_dz);
      klo = int(floorf(__fadd_rn(pzbz, __fmul_rn(av, dz0))));
      khi = int(floorf(__fadd_rn(pzbz, __fmul_rn(av, dzl))));
    }
    if (!got_lo) {
      const unsigned b = __ballot_sync(0xffffffffu, m < n && klo <= 0);
      if (b) {
        const int src = __ffs(b) - 1;
        const int k = __shfl_sync(0xffffffffu, klo, src);
        min_xy_all = (k == 0) ? m0 + src : 0;
        got_lo = true;
      }
    }
    if (!got_hi) {
      const unsigned b = __ballot_sync(0xffffffffu, m < n && khi >= nzm1);
      if (b) {
        const int src = __ffs(b) - 1;
        const int k = __shfl_sync(0xffffffffu, khi, src);
        max_xy_all = (k == nzm1) ? m0 + src : 0;
        got_hi = true;
      }
    }
  }
  ncom = min(min_xy_all, max_xy_all);
  const float avl = __fmul_rn(alphas[n - 2], inv_dz);
  for (int v0 = 0; v0 < mid; v0 += 32) {
    const int v = v0 + lane;
    const bool ok = v < mid && int(floorf(__fadd_rn(pzbz, __fmul_rn(avl, g.dz[v])))) > 0;
    const unsigned b = __ballot_sync(0xffffffffu, ok);
    if (b) {
      min_v_all = v0 + __ffs(b) - 1;
      break;
    }
  }
  for (int v1 = g.nv - 1; v1 >= mid; v1 -= 32) {
    const int v = v1 - lane;
    const bool ok = v >= mid && int(floorf(__fadd_rn(pzbz, __fmul_rn(avl, g.dz[v])))) < nzm1;
    const unsigned b = __ballot_sync(0xffffffffu, ok);
    if (b) {
      max_v_all = v1 - (__ffs(b) - 1);
      break;
    }
  }
}

// How a pass of 32 * RPL rows lies to the source: all below, all above, or
// the first half of each lane's rows below and the second above.
enum Side { BELOW = 0, ABOVE = 1, HALVES = 2 };

// One pass over cells [1, m1), where every row's slice k and the neighbour
// on the far side of the plane it may cross lie inside the column.  Rows q
// and q + 1 of a lane go as packed pairs: per row the reference's unfused
// float operations (c2D.cpp:99-145), in its order.  int(x) is the low bits of
// 2^23 + x rounded toward zero (1 <= x).  Where the pass lies to the source is
// a template argument, so the neighbour is an immediate offset.
//
// Bound: instruction issue.  Scalar sums and conversions, and the neighbour's
// address formed per row, took 306 ms at 512^3 / 720 angles / 768^2; packed
// sums (mul2_nz), int(x) by addition and immediate offsets 260 ms; addresses
// as multiply-adds by a 4 the compiler cannot turn into shifts, which puts
// them on the FMA pipe instead of the ALU, 232 ms.
__device__ __forceinline__ const float *at_wide(unsigned k, unsigned four, const char *c) {
  const float *r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(k), "r"(four), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned at_smem(unsigned k, unsigned four, unsigned c) {
  unsigned r;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(k), "r"(four), "r"(c));
  return r;
}
template <int RPL, int SIDE>
__device__ __forceinline__ void cb_fp_cells(const Geom &g, const float *alphas, const int *cells,
                                            int m1, const float *vol, const float *svz,
                                            const float2 (&dz2)[RPL / 2],
                                            const float2 (&iz2)[RPL / 2],
                                            float2 (&acc2)[RPL / 2]) {
  constexpr unsigned kMagic = 0x4b000000u; // bits of 2^23
  const float2 nz = make_float2(g.neg0, g.neg0);
  const float2 pz = make_float2(g.pzbz, g.pzbz), big = make_float2(8388608.0f, 8388608.0f);
  const unsigned vz = unsigned(__cvta_generic_to_shared(svz)) - 4 * kMagic;
  for (int m = 1; m < m1; m++) {
    const int cell = cells[m - 1];
    if (cell < 0)
      continue;
    const float a0 = alphas[m - 1], a1 = alphas[m];
    const char *col = reinterpret_cast<const char *>(vol + i64(cell) * g.nz) - 4ll * kMagic;
    const float av = __fmul_rn(a0, g.inv_dz);
    const float2 av2 = make_float2(av, av), a02 = make_float2(a0, a0), a12 = make_float2(a1, a1);
#pragma unroll
    for (int q = 0; q < RPL; q += 2) {
      const float2 x = add2_rn(pz, mul2_nz(av2, dz2[q / 2], nz));
      const float2 b = add2_rz(x, big);
      const unsigned k0 = __float_as_uint(b.x), k1 = __float_as_uint(b.y);
      const int d0 = SIDE == BELOW || (SIDE == HALVES && q < RPL / 2) ? -1 : 1;
      const int d1 = SIDE == BELOW || (SIDE == HALVES && q + 1 < RPL / 2) ? -1 : 1;
      const float2 pl = mul2_rn(make_float2(lds_f(at_smem(k0, g.four, vz) + (d0 < 0 ? 0 : 4)),
                                            lds_f(at_smem(k1, g.four, vz) + (d1 < 0 ? 0 : 4))),
                                iz2[q / 2]);
      const float2 mz = make_float2(fmin_ref(pl.x, a1), fmin_ref(pl.y, a1));
      const float2 lo = sub2_rn(mz, a02), hi = sub2_rn(a12, mz);
      const float *c0 = at_wide(k0, g.four, col), *c1 = at_wide(k1, g.four, col);
      const float2 pk = mul2_nz(make_float2(__ldg(c0), __ldg(c1)), lo, nz);
      const float2 pn = mul2_nz(make_float2(__ldg(c0 + d0), __ldg(c1 + d1)), hi, nz);
      acc2[q / 2] = add2_rn(acc2[q / 2], add2_rn(pk, pn));
    }
  }
}

// cb_fp_cells for up to 32 rows, one per lane; side: the lane's side of the
// source (-1 below, 1 above).  With two rows per lane half of them were idle
// (512^2 x 8 from 16 rows, 60 angles: 7.9 ms; with one 6.5 ms).
__device__ __forceinline__ float cb_fp_cells_one(const Geom &g, const float *alphas,
                                                 const int *cells, int m1, const float *vol,
                                                 const float *svz, float dz, float iz, int side) {
  constexpr unsigned kMagic = 0x4b000000u; // bits of 2^23
  const unsigned vz =
      unsigned(__cvta_generic_to_shared(svz)) - 4 * kMagic + (side < 0 ? 0 : 4);
  float acc = 0.0f;
  for (int m = 1; m < m1; m++) {
    const int cell = cells[m - 1];
    if (cell < 0)
      continue;
    const float a0 = alphas[m - 1], a1 = alphas[m];
    const char *col = reinterpret_cast<const char *>(vol + i64(cell) * g.nz) - 4ll * kMagic;
    const float x = __fadd_rn(g.pzbz, __fmul_rn(__fmul_rn(a0, g.inv_dz), dz));
    const unsigned k = __float_as_uint(__fadd_rz(x, 8388608.0f));
    const float mz = fmin_ref(__fmul_rn(lds_f(at_smem(k, g.four, vz)), iz), a1);
    const float *c = at_wide(k, g.four, col);
    acc = __fadd_rn(acc, __fadd_rn(__fmul_rn(__ldg(c), __fsub_rn(mz, a0)),
                                   __fmul_rn(__ldg(c + side), __fsub_rn(a1, mz))));
  }
  return acc;
}

// RPL = detector rows per lane per pass.  The np passes of 32 * RPL rows start
// at row v0 <= 0, such that the first row above the source begins a pass or
// the second half of one; rows outside [0, nv) act as a row at the source
// height and are not stored.  BATCH: nb
// volumes (one after another) share each ray's walk and row regimes
// (EPI_STORE only).  Without it the item loop runs once and compiles away: a
// run-time loop costs the single-volume form 10 % at 512^3.
template <int EPI, int RPL, bool BATCH>
__global__ void __launch_bounds__(kFpWarps * 32)
    cb_fp_kernel(Geom g, const float *__restrict__ vol0, float *__restrict__ pix0, Epi e,
                 const int2 *__restrict__ hrange, int cap, int nb, int v0, int np) {
  extern __shared__ unsigned char smem_raw[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *svz = reinterpret_cast<float *>(smem_raw);
  float *alphas = svz + cb_vz_floats(g.nz) + size_t(wib) * 2 * cap;
  int *cells = reinterpret_cast<int *>(alphas + cap);
  for (int i = threadIdx.x; i <= g.nz; i += blockDim.x)
    svz[i] = g.vz[i];
  __syncthreads();
  const int nrays = g.na * g.nh;
  const int nzm1 = g.nz - 1, mid = g.mid;
  const float pzbz = g.pzbz, pzbz1 = g.pzbz1, inv_dz = g.inv_dz;
  double ssq = 0.0;
  for (int ray = blockIdx.x * kFpWarps + wib; ray < nrays; ray += gridDim.x * kFpWarps) {
    const int a = ray / g.nh, h = ray - a * g.nh;
    const int2 hr = hrange[a];
    int n = 0;
    if (h >= hr.x && h <= hr.y) {
      const double c = g.cosA[a], s = g.sinA[a];
      const double p2x = c * g.detx - s * g.hpix[h];
      const double p2y = s * g.detx + c * g.hpix[h];
      n = cb_walk(g, g.p1x[a], g.p1y[a], p2x, p2y, alphas, cells, cap);
    }
    __syncwarp();
    int ncom, min_v_all, max_v_all;
    cb_row_regimes(g, alphas, n, lane, ncom, min_v_all, max_v_all);
    // Rows, RPL per lane per pass.  Cells [1, mfast) have every row inside
    // the slab (c2D.cpp:99-145); the rest take the edge rules (:146-190).
    const int mfast = min(ncom, n);
    for (int b = 0; b < (BATCH ? nb : 1); b++) {
    // batch item b: its volume and its sinogram
    const float *__restrict__ vol = vol0 + i64(b) * g.nx * g.ny * g.nz;
    float *__restrict__ pix = pix0 + i64(b) * g.na * g.nh * g.nv;
    for (int vb = v0; vb < v0 + np * 32 * RPL; vb += 32 * RPL) {
      float acc[RPL], dzv[RPL], izv[RPL];
      bool vok[RPL], below[RPL];
#pragma unroll
      for (int q = 0; q < RPL; q++) {
        const int v = vb + q * 32 + lane;
        acc[q] = 0.0f;
        vok[q] = v >= 0 && v < g.nv;
        below[q] = v < mid;
        dzv[q] = vok[q] ? g.dz[v] : 0.0f;
        izv[q] = vok[q] ? g.iz[v] : 0.0f;
      }
      // In [1, mfast) the regime search has shown that the lowest row's
      // slice index is >= 1 and the highest row's < nz - 1 (c2D.cpp:45-99),
      // so every row's k and its neighbour k -/+ 1 are inside the column.
      if constexpr (RPL == 1) {
        acc[0] = cb_fp_cells_one(g, alphas, cells, mfast, vol, svz, dzv[0], izv[0],
                                 below[0] ? -1 : 1);
      } else {
      float2 acc2[RPL / 2], dz2[RPL / 2], iz2[RPL / 2];
#pragma unroll
      for (int q = 0; q < RPL; q += 2) {
        acc2[q / 2] = make_float2(0.0f, 0.0f);
        dz2[q / 2] = make_float2(dzv[q], dzv[q + 1]);
        iz2[q / 2] = make_float2(izv[q], izv[q + 1]);
      }
#define CB_FP_CELLS(S)                                                                     \
  cb_fp_cells<RPL, S>(g, alphas, cells, mfast, vol, svz, dz2, iz2, acc2)
      if (vb + 32 * RPL <= mid)
        CB_FP_CELLS(BELOW);
      else if (vb >= mid)
        CB_FP_CELLS(ABOVE);
      else // vb + 16 * RPL == mid
        CB_FP_CELLS(HALVES);
#undef CB_FP_CELLS
#pragma unroll
      for (int q = 0; q < RPL; q++)
        acc[q] = (q & 1) ? acc2[q / 2].y : acc2[q / 2].x;
      }
      for (int m = max(mfast, 1); m < n; m++) {
        const float a0 = alphas[m - 1], a1 = alphas[m];
        const int cell = cells[m - 1];
        if (cell < 0)
          continue;
        const float *col = vol + i64(cell) * g.nz;
        const float av = __fmul_rn(a0, inv_dz);
#pragma unroll
        for (int q = 0; q < RPL; q++) {
          const int v = vb + q * 32 + lane;
          if (!vok[q])
            continue;
          if (v >= min_v_all && v <= max_v_all) {
            const int k = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[q])));
            const int kn = below[q] ? k - 1 : k + 1;
            if (unsigned(k) > unsigned(nzm1) || unsigned(kn) > unsigned(nzm1))
              continue;
            const float mz = fmin_ref(__fmul_rn(svz[below[q] ? k : k + 1], izv[q]), a1);
            acc[q] = __fadd_rn(acc[q], __fadd_rn(__fmul_rn(__ldg(col + k), __fsub_rn(mz, a0)),
                                                 __fmul_rn(__ldg(col + kn), __fsub_rn(a1, mz))));
          } else if (ncom >= 1) {
            if (v < min_v_all) {
              const int k = int(__fadd_rn(pzbz1, __fmul_rn(av, dzv[q]))) - 1;
              if (k > 0 && k <= nzm1) {
                const float mz = fmin_ref(__fmul_rn(svz[k], izv[q]), a1);
                acc[q] = __fadd_rn(acc[q],
                                   __fadd_rn(__fmul_rn(__ldg(col + k), __fsub_rn(mz, a0)),
                                             __fmul_rn(__ldg(col + k - 1), __fsub_rn(a1, mz))));
              } else if (k == 0) {
                const float mz = fmin_ref(__fmul_rn(svz[0], izv[q]), a1);
                acc[q] = __fadd_rn(acc[q], __fmul_rn(__ldg(col), __fsub_rn(mz, a0)));
              }
            } else {
              const int k = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[q])));
              if (k < nzm1 && k >= 0) {
                const float mz = fmin_ref(__fmul_rn(svz[k + 1], izv[q]), a1);
                acc[q] = __fadd_rn(acc[q],
                                   __fadd_rn(__fmul_rn(__ldg(col + k), __fsub_rn(mz, a0)),
                                             __fmul_rn(__ldg(col + k + 1), __fsub_rn(a1, mz))));
              } else if (k == nzm1) {
                const float mz = fmin_ref(__fmul_rn(svz[g.nz], izv[q]), a1);
                acc[q] = __fadd_rn(acc[q], __fmul_rn(__ldg(col + nzm1), __fsub_rn(mz, a0)));
              }
            }
          }
        }
      }
      const i64 rbase = i64(ray) * g.nv;
#pragma unroll
      for (int q = 0; q < RPL; q++) {
        const int v = vb + q * 32 + lane;
        if (v >= 0 && v < g.nv) {
          const float dcv = g.dconv[i64(h) * g.nv + v];
          const float out = cb_fp_epi<EPI>(__fmul_rn(acc[q], dcv), rbase + v, e, ssq);
          // the SIRT / MLEM residual is the back projector's input: with
          // e.pre it is stored times d_conv (the reference's dpixels)
          pix[rbase + v] = ((EPI == EPI_SIRT || EPI == EPI_MLEM) && e.pre) ? __fmul_rn(out, dcv) : out;
        }
      }
    }
    } // batch items
    __syncwarp();
  }
  if (EPI == EPI_NORM) {
    __shared__ double red[kFpWarps];
    const double t = cta_sum<kFpWarps>(ssq, red);
    if (threadIdx.x == 0)
      e.partials[blockIdx.x] = t;
  }
}

// ---- backward, ray-driven scatter (the transpose of cb_fp_kernel)
//
// One warp per ray (angle a, detector column h), as in the forward
// projector, with the same walk.  The reference's back projector is not the
// exact transpose of its forward projector: it drops rays parallel to an
// axis and picks each row's slice rule from a band kept per voxel column
// (c2D.cpp:657-750), where the forward projector keeps one per ray.  So
// per (cell, row) this kernel takes the back projector's rule, from the
// plan's column band table: slice k, neighbour and weights (mz - a0,
// a1 - mz), and the row's value p = pix * d_conv times each weight goes to
// the two voxels, with float atomics.  The order of the additions into a
// voxel is not fixed: the result equals the reference's b2D to float
// rounding, not bit for bit (cb_back.cu has that form).  Detector columns are
// taken as even: off their even spacing b2D drops rays that its range of a
// voxel column misses, which this does not.  `vol` must be zero on entry; PRE:
// `pix` is already scaled by d_conv.
//
// Bound: instruction issue (82 % of the slots at 256^3), the L2 at 54 % of its
// throughput with the atomics.  Rows in lane-consecutive
// pairs, packed, and no atomic for a weight of zero: 512^3 501 -> 320 ms,
// 256^3 30.9 -> 20.6 ms.  Without the test for zero weights 586 ms; with a
// lane's pairs next to each other, so that an atomic instruction's slices
// spread over more sectors, 405 ms (4 rows per lane) and 513 ms (6).
//
// (A form with lanes on rows 32 apart and a warp segmented reduction per
// target was measured slower on every geometry: 1250 against 1012 ms at
// 512^3, 69 against 58 ms at 256^3.)

// An address computed in asm has lost its state space: name it here.
__device__ __forceinline__ void red_add(const float *p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// One cell whose rows of this pass all lie in the column's band, with every
// slice k and its neighbour inside the column (cb_row_regimes).  Rows j and
// j + 1 as packed pairs; a pair on one slice adds its two sums, in row order,
// and a weight of zero (the row does not cross the plane) adds nothing.  IDLE:
// many rows lie outside the detector, and their sums add nothing either.
template <int RPL, int SIDE, bool IDLE>
__device__ __forceinline__ void cb_scatter_cell(const Geom &g, float a0, float a1, float *vcol,
                                                unsigned vz, int side, const float (&dzv)[RPL],
                                                const float (&izv)[RPL], const float (&p)[RPL]) {
  constexpr unsigned kMagic = 0x4b000000u; // bits of 2^23
  const float2 nz = make_float2(g.neg0, g.neg0);
  const float2 pz = make_float2(g.pzbz, g.pzbz), big = make_float2(8388608.0f, 8388608.0f);
  const char *col = reinterpret_cast<const char *>(vcol) - 4ll * kMagic;
  const float av = __fmul_rn(a0, g.inv_dz);
  // a lane's side of the source in the group of rows that holds it
  const char *ncol = col + 4 * side;
  const unsigned vzm = vz - 4 * kMagic, vzs = vzm + (side < 0 ? 0 : 4);
  // D: the neighbour's step, 0 for the lane's own
  auto add = [&](unsigned k, int D, float s1, float s2) {
    const float *c = at_wide(k, g.four, col);
    if (!IDLE || s1 != 0.0f)
      red_add(c, s1);
    if (s2 != 0.0f)
      red_add(D == 0 ? at_wide(k, g.four, ncol) : c + D, s2);
  };
#pragma unroll
  for (int j = 0; j < RPL; j += 2) {
    // rows 32 j .. 32 j + n of the pass
    const int n = j + 1 < RPL ? 64 : 32;
    const int D = SIDE == BELOW ? -1 : SIDE == ABOVE ? 1 : 32 * j + n <= 16 * RPL ? -1
                  : 32 * j >= 16 * RPL ? 1 : 0;
    const unsigned za = D == 0 ? vzs : D < 0 ? vzm : vzm + 4;
    if (n == 64) {
      const float2 x =
          add2_rn(pz, mul2_nz(make_float2(av, av), make_float2(dzv[j], dzv[j + 1]), nz));
      const float2 b = add2_rz(x, big);
      const unsigned k0 = __float_as_uint(b.x), k1 = __float_as_uint(b.y);
      const float2 pl = mul2_rn(
          make_float2(lds_f(at_smem(k0, g.four, za)), lds_f(at_smem(k1, g.four, za))),
          make_float2(izv[j], izv[j + 1]));
      const float2 mz = make_float2(fmin_ref(pl.x, a1), fmin_ref(pl.y, a1));
      const float2 pp = make_float2(p[j], p[j + 1]);
      const float2 s1 = mul2_rn(pp, sub2_rn(mz, make_float2(a0, a0)));
      const float2 s2 = mul2_rn(pp, sub2_rn(make_float2(a1, a1), mz));
      const bool same = k0 == k1;
      add(k0, D, same ? __fadd_rn(s1.x, s1.y) : s1.x, same ? __fadd_rn(s2.x, s2.y) : s2.x);
      if (!same)
        add(k1, D, s1.y, s2.y);
    } else {
      const float x = __fadd_rn(g.pzbz, __fmul_rn(av, dzv[j]));
      const unsigned k = __float_as_uint(__fadd_rz(x, 8388608.0f));
      const float mz = fmin_ref(__fmul_rn(lds_f(at_smem(k, g.four, za)), izv[j]), a1);
      add(k, D, __fmul_rn(p[j], __fsub_rn(mz, a0)), __fmul_rn(p[j], __fsub_rn(a1, mz)));
    }
  }
}

// Row j of a lane in a pass of 32 * RPL rows: pairs of consecutive rows, a
// pair of every lane before the next pair, so that one instruction's atomics
// fall on consecutive slices.
template <int RPL> __device__ __forceinline__ int cb_scatter_row(int j, int lane) {
  return (j | 1) < RPL ? 32 * (j & ~1) + 2 * lane + (j & 1) : 32 * j + lane;
}
// The walk of ray (a, h) as the back projector takes it: no ray parallel to an
// axis (c2D.cpp:909-912), with its own differences.
__device__ __forceinline__ int cb_scatter_walk(const Geom &g, int a, int h,
                                               const int2 *__restrict__ hrange, float *alphas,
                                               int *cells, int cap) {
  const int2 hr = hrange[a];
  if (h < hr.x || h > hr.y)
    return 0;
  const double c = g.cosA[a], s = g.sinA[a];
  const double bdx = (g.cdx[a] - s * g.hpix[h]) - g.p1x[a];
  const double bdy = (g.sdx[a] + c * g.hpix[h]) - g.p1y[a];
  if (fabs(bdx) < double(kEps) || fabs(bdy) < double(kEps))
    return 0;
  const double p2x = c * g.detx - s * g.hpix[h];
  const double p2y = s * g.detx + c * g.hpix[h];
  return cb_walk(g, g.p1x[a], g.p1y[a], p2x, p2y, alphas, cells, cap);
}

template <int RPL, bool PRE>
__global__ void __launch_bounds__(kFpWarps * 32, 8)
    cb_bp_scatter(Geom g, const float *__restrict__ pix, float *__restrict__ vol,
                  const int2 *__restrict__ hrange, int cap, int v0, int np) {
  extern __shared__ unsigned char smem_raw[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *svz = reinterpret_cast<float *>(smem_raw);
  float *alphas = svz + cb_vz_floats(g.nz) + size_t(wib) * 2 * cap;
  int *cells = reinterpret_cast<int *>(alphas + cap);
  for (int i = threadIdx.x; i <= g.nz; i += blockDim.x)
    svz[i] = g.vz[i];
  __syncthreads();
  const int nrays = g.na * g.nh;
  const int nz = g.nz, nzm1 = g.nz - 1, mid = g.mid;
  const float pzbz = g.pzbz, pzbz1 = g.pzbz1, inv_dz = g.inv_dz;
  const unsigned vz = unsigned(__cvta_generic_to_shared(svz));
  // The lane's side of the source in the 64 rows (one row per lane: 32) that
  // hold row 16 * RPL, where a pass with the source in its middle has it.
  const int side = lane < (RPL == 1 ? 16 : 16 * RPL % 64 / 2) ? -1 : 1;
  for (int ray = blockIdx.x * kFpWarps + wib; ray < nrays; ray += gridDim.x * kFpWarps) {
    const int h = ray % g.nh;
    const int n = cb_scatter_walk(g, ray / g.nh, h, hrange, alphas, cells, cap);
    __syncwarp();
    int ncom, min_v_all, max_v_all;
    cb_row_regimes(g, alphas, n, lane, ncom, min_v_all, max_v_all);
    const int mfast = min(ncom, n);
    const i64 rbase = i64(ray) * g.nv;
    for (int vb = v0; n >= 2 && vb < v0 + np * 32 * RPL; vb += 32 * RPL) {
      float p[RPL], dzv[RPL], izv[RPL];
      bool vok[RPL], below[RPL];
#pragma unroll
      for (int j = 0; j < RPL; j++) {
        const int v = vb + cb_scatter_row<RPL>(j, lane);
        vok[j] = v >= 0 && v < g.nv;
        below[j] = v < mid;
        dzv[j] = vok[j] ? g.dz[v] : 0.0f;
        izv[j] = vok[j] ? g.iz[v] : 0.0f;
        const float y = vok[j] ? __ldg(pix + rbase + v) : 0.0f;
        p[j] = (PRE || !vok[j]) ? y : __fmul_rn(y, g.dconv[i64(h) * g.nv + v]);
      }
      const int r0 = max(vb, 0), r1 = min(vb + 32 * RPL, g.nv); // the pass's rows
      // with more than a sixteenth of its rows outside the detector a pass
      // tests every sum for zero (288 rows in a pass of 320: 8.5 against
      // 9.3 ms; 256^3 with every row inside: 22.5 against 20.6 ms)
      const bool idle = r1 - r0 < 30 * RPL;
      // the crossed column's band, loaded one cell ahead
      int2 band_next = cells[0] >= 0 ? g.colband[cells[0]] : make_int2(0, 0);
      for (int m = 1; m < n; m++) {
        const int cell = cells[m - 1];
        const int2 band = band_next;
        if (m + 1 < n && cells[m] >= 0)
          band_next = g.colband[cells[m]];
        if (cell < 0)
          continue;
        const float a0 = alphas[m - 1], a1 = alphas[m];
        float *col = vol + i64(cell) * nz;
        if (m < mfast && r0 >= band.x && r1 <= band.y) {
#define CB_SC_CELL(S)                                                                      \
  (idle ? cb_scatter_cell<RPL, S, true>(g, a0, a1, col, vz, side, dzv, izv, p)                \
        : cb_scatter_cell<RPL, S, false>(g, a0, a1, col, vz, side, dzv, izv, p))
          if (vb + 32 * RPL <= mid)
            CB_SC_CELL(BELOW);
          else if (vb >= mid)
            CB_SC_CELL(ABOVE);
          else // vb + 16 * RPL == mid
            CB_SC_CELL(HALVES);
#undef CB_SC_CELL
          continue;
        }
        const float av = __fmul_rn(a0, inv_dz);
        int ck = -1, ckn = -1, ckey = -1; // the lane's current run
        float q1 = 0.0f, q2 = 0.0f;
        // one row's run logic: a run of rows with the same slice and side
        // sums its two products in registers; when the slice changes the
        // run's two sums go to its slice and neighbour
        auto run = [&](int k, int kn, bool up, float s1, float s2) {
          const int key = k >= 0 ? 2 * k + (up ? 1 : 0) : -1;
          if (key != ckey) {
            if (ck >= 0) {
              atomicAdd(col + ck, q1);
              if (ckn >= 0)
                atomicAdd(col + ckn, q2);
            }
            ck = k;
            ckn = kn;
            ckey = key;
            q1 = 0.0f;
            q2 = 0.0f;
          }
          if (k >= 0) {
            q1 = __fadd_rn(q1, s1);
            q2 = __fadd_rn(q2, s2);
          }
        };
#pragma unroll
        for (int j = 0; j < RPL; j++) {
          const int v = vb + cb_scatter_row<RPL>(j, lane);
          // the back projector's rule for this row (c2D.cpp:680-750): a
          // band row feeds its slice k and the neighbour on the source's
          // side (k - 1 below the source, k + 1 above), a row below the
          // band k and k - 1, a row above it k and k + 1
          int k = -1, kn = -1;
          bool up = false;
          float w1 = 0.0f, w2 = 0.0f;
          if (vok[j]) {
            if (v >= band.x && v < band.y) {
              const int kk = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[j])));
              const int kkn = below[j] ? kk - 1 : kk + 1;
              if (unsigned(kk) <= unsigned(nzm1) && unsigned(kkn) <= unsigned(nzm1)) {
                const float mz = fmin_ref(__fmul_rn(svz[below[j] ? kk : kk + 1], izv[j]), a1);
                k = kk;
                kn = kkn;
                up = !below[j];
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              }
            } else if (v < band.x) {
              const int kk = int(__fadd_rn(pzbz1, __fmul_rn(av, dzv[j]))) - 1;
              if (kk > 0 && kk <= nzm1) {
                const float mz = fmin_ref(__fmul_rn(svz[kk], izv[j]), a1);
                k = kk;
                kn = kk - 1;
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              } else if (kk == 0) {
                k = 0;
                w1 = __fsub_rn(fmin_ref(__fmul_rn(svz[0], izv[j]), a1), a0);
              }
            } else {
              const int kk = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[j])));
              up = true;
              if (kk < nzm1 && kk >= 0) {
                const float mz = fmin_ref(__fmul_rn(svz[kk + 1], izv[j]), a1);
                k = kk;
                kn = kk + 1;
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              } else if (kk == nzm1) {
                k = nzm1;
                w1 = __fsub_rn(fmin_ref(__fmul_rn(svz[nz], izv[j]), a1), a0);
              }
            }
          }
          run(k, kn, up, __fmul_rn(p[j], w1), __fmul_rn(p[j], w2));
        }
        if (ck >= 0) {
          atomicAdd(col + ck, q1);
          if (ckn >= 0)
            atomicAdd(col + ckn, q2);
        }
      }
    }
    __syncwarp();
  }
}

// The form for detectors that reach past the volume's ends: passes of 32 * R
// rows, each taken whole where its own rows lie in the band and the column, so
// that the rows near the source's height need no general rule for the sake of
// those at the detector's edges.  R consecutive rows per lane, whose sums for
// a slice join before the atomic.  The form above takes a cell whole only if
// every row is inside: 20 to 40 % slower here (see cb_scatter_edge).
template <int R, bool PRE>
__global__ void __launch_bounds__(kFpWarps * 32, 8)
    cb_bp_scatter_edge(Geom g, const float *__restrict__ pix, float *__restrict__ vol,
                       const int2 *__restrict__ hrange, int cap) {
  extern __shared__ unsigned char smem_raw[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *svz = reinterpret_cast<float *>(smem_raw);
  float *alphas = svz + cb_vz_floats(g.nz) + size_t(wib) * 2 * cap;
  int *cells = reinterpret_cast<int *>(alphas + cap);
  for (int i = threadIdx.x; i <= g.nz; i += blockDim.x)
    svz[i] = g.vz[i];
  __syncthreads();
  const int nrays = g.na * g.nh;
  const int nz = g.nz, nzm1 = g.nz - 1, mid = g.mid;
  const float pzbz = g.pzbz, pzbz1 = g.pzbz1, inv_dz = g.inv_dz;
  for (int ray = blockIdx.x * kFpWarps + wib; ray < nrays; ray += gridDim.x * kFpWarps) {
    const int h = ray % g.nh;
    const int n = cb_scatter_walk(g, ray / g.nh, h, hrange, alphas, cells, cap);
    __syncwarp();
    const i64 rbase = i64(ray) * g.nv;
    for (int vb = 0; n >= 2 && vb < g.nv; vb += 32 * R) {
      float p[R], dzv[R], izv[R];
      // per row, fixed by its side of the source: the neighbour's step, the
      // slice plane the weights use (k or k + 1) and the lowest slice whose
      // neighbour stays inside the column
      int dk[R], off[R], klo[R];
      bool vok[R];
#pragma unroll
      for (int j = 0; j < R; j++) {
        const int v = vb + lane * R + j;
        vok[j] = v < g.nv;
        dk[j] = v < mid ? -1 : 1;
        off[j] = v < mid ? 0 : 1;
        klo[j] = v < mid ? 1 : 0;
        dzv[j] = vok[j] ? g.dz[v] : 0.0f;
        izv[j] = vok[j] ? g.iz[v] : 0.0f;
        const float y = vok[j] ? __ldg(pix + rbase + v) : 0.0f;
        p[j] = (PRE || !vok[j]) ? y : __fmul_rn(y, g.dconv[i64(h) * g.nv + v]);
      }
      // the crossed column's band, loaded one cell ahead
      int2 band_next = cells[0] >= 0 ? g.colband[cells[0]] : make_int2(0, 0);
      for (int m = 1; m < n; m++) {
        const int cell = cells[m - 1];
        const int2 band = band_next;
        if (m + 1 < n && cells[m] >= 0)
          band_next = g.colband[cells[m]];
        if (cell < 0)
          continue;
        const float a0 = alphas[m - 1], a1 = alphas[m];
        const float av = __fmul_rn(a0, inv_dz);
        float *col = vol + i64(cell) * nz;
        if (vb + 32 * R <= band.y && vb >= band.x && vb + 32 * R <= g.nv) {
          // every row of the pass valid and inside the column's band (the
          // test is the same for the whole warp): the band rule alone
#pragma unroll
          for (int j = 0; j < R; j += 2) {
            const int i = j + 1 < R ? j + 1 : j; // the odd row is its own pair
            const float2 kz = mul2_rn(make_float2(av, av), make_float2(dzv[j], dzv[i]));
            const int k0 = int(__fadd_rn(pzbz, kz.x)), k1 = int(__fadd_rn(pzbz, kz.y));
            // k and its neighbour k -/+ 1 inside [0, nz - 1]: one range test
            // (a one-slice column holds no neighbour)
            const bool ok0 = nzm1 > 0 && unsigned(k0 - klo[j]) <= unsigned(nzm1 - 1);
            const bool ok1 = i > j && nzm1 > 0 && unsigned(k1 - klo[i]) <= unsigned(nzm1 - 1);
            const float z0 = ok0 ? svz[k0 + off[j]] : 0.0f;
            const float z1 = ok1 ? svz[k1 + off[i]] : 0.0f;
            const float2 pl = mul2_rn(make_float2(z0, z1), make_float2(izv[j], izv[i]));
            const float2 mz = make_float2(fmin_ref(pl.x, a1), fmin_ref(pl.y, a1));
            const float2 pp = make_float2(p[j], p[i]);
            const float2 s1 = mul2_rn(pp, sub2_rn(mz, make_float2(a0, a0)));
            const float2 s2 = mul2_rn(pp, sub2_rn(make_float2(a1, a1), mz));
            // one pair of atomics when both rows share slice and side
            const bool same = ok0 && ok1 && k0 == k1 && dk[j] == dk[i];
            if (ok0) {
              atomicAdd(col + k0, same ? __fadd_rn(s1.x, s1.y) : s1.x);
              atomicAdd(col + k0 + dk[j], same ? __fadd_rn(s2.x, s2.y) : s2.x);
            }
            if (ok1 && !same) {
              atomicAdd(col + k1, s1.y);
              atomicAdd(col + k1 + dk[i], s2.y);
            }
          }
          continue;
        }
        int ck = -1, ckn = -1, ckey = -1; // the lane's current run
        float q1 = 0.0f, q2 = 0.0f;
        // one row's run logic: a run of rows with the same slice and side
        // sums its two products in registers; when the slice changes the
        // run's two sums go to its slice and neighbour
        auto run = [&](int k, int kn, bool up, float s1, float s2) {
          const int key = k >= 0 ? 2 * k + (up ? 1 : 0) : -1;
          if (key != ckey) {
            if (ck >= 0) {
              atomicAdd(col + ck, q1);
              if (ckn >= 0)
                atomicAdd(col + ckn, q2);
            }
            ck = k;
            ckn = kn;
            ckey = key;
            q1 = 0.0f;
            q2 = 0.0f;
          }
          if (k >= 0) {
            q1 = __fadd_rn(q1, s1);
            q2 = __fadd_rn(q2, s2);
          }
        };
#pragma unroll
        for (int j = 0; j < R; j++) {
          const int v = vb + lane * R + j;
          // the back projector's rule for this row (c2D.cpp:680-750): a
          // band row feeds its slice k and the neighbour on the source's
          // side (k - 1 below the source, k + 1 above), a row below the
          // band k and k - 1, a row above it k and k + 1
          int k = -1, kn = -1;
          bool up = false;
          float w1 = 0.0f, w2 = 0.0f;
          if (vok[j]) {
            if (v >= band.x && v < band.y) {
              const int kk = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[j])));
              const int kkn = v < mid ? kk - 1 : kk + 1;
              if (unsigned(kk) <= unsigned(nzm1) && unsigned(kkn) <= unsigned(nzm1)) {
                const float mz = fmin_ref(__fmul_rn(svz[v < mid ? kk : kk + 1], izv[j]), a1);
                k = kk;
                kn = kkn;
                up = v >= mid;
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              }
            } else if (v < band.x) {
              const int kk = int(__fadd_rn(pzbz1, __fmul_rn(av, dzv[j]))) - 1;
              if (kk > 0 && kk <= nzm1) {
                const float mz = fmin_ref(__fmul_rn(svz[kk], izv[j]), a1);
                k = kk;
                kn = kk - 1;
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              } else if (kk == 0) {
                k = 0;
                w1 = __fsub_rn(fmin_ref(__fmul_rn(svz[0], izv[j]), a1), a0);
              }
            } else {
              const int kk = int(__fadd_rn(pzbz, __fmul_rn(av, dzv[j])));
              up = true;
              if (kk < nzm1 && kk >= 0) {
                const float mz = fmin_ref(__fmul_rn(svz[kk + 1], izv[j]), a1);
                k = kk;
                kn = kk + 1;
                w1 = __fsub_rn(mz, a0);
                w2 = __fsub_rn(a1, mz);
              } else if (kk == nzm1) {
                k = nzm1;
                w1 = __fsub_rn(fmin_ref(__fmul_rn(svz[nz], izv[j]), a1), a0);
              }
            }
          }
          run(k, kn, up, __fmul_rn(p[j], w1), __fmul_rn(p[j], w2));
        }
        if (ck >= 0) {
          atomicAdd(col + ck, q1);
          if (ckn >= 0)
            atomicAdd(col + ckn, q2);
        }
      }
    }
    __syncwarp();
  }
}

// ---- backward
// Band rows [lo, hi) of a ray entering a column at a0: rows whose slice and
// its neighbour stay inside the column (c2D.cpp:664-668).
__device__ __forceinline__ int cb_band_lo(const Geom &g, float a0) {
  return int(ceilf(__fadd_rn(g.pzdeps, __fdiv_rn(g.z1, a0))));
}
__device__ __forceinline__ int cb_band_hi(const Geom &g, float a0) {
  return int(floorf(__fadd_rn(g.pzdv, __fdiv_rn(g.znm, a0))));
}

// The back projector's band of every voxel column (c2D.cpp:657-676): the
// rows inside the band of every ray that crosses the column.  One warp per
// column, lanes over the angles; geometry only, built once per plan.
constexpr int kBandWarps = 8;
__global__ void __launch_bounds__(kBandWarps * 32) cb_column_band_kernel(Geom g, int2 *band) {
  const int col = blockIdx.x * kBandWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (col >= g.nx * g.ny)
    return; // the whole warp
  const int i = col / g.ny, j = col - i * g.ny;
  const double x0 = g.origin[0] + double(i) * g.size[0];
  const double xn = g.origin[0] + double(i + 1) * g.size[0];
  const double y0 = g.origin[1] + double(j) * g.size[1];
  const double yn = g.origin[1] + double(j + 1) * g.size[1];
  int lo = 0, hi = g.nv;
  for (int a = lane; a < g.na; a += 32)
    cb_column_rays(g, a, x0, xn, y0, yn, [&](int, float a0, float) {
      lo = max(lo, cb_band_lo(g, a0));
      hi = min(hi, cb_band_hi(g, a0));
    });
  lo = __reduce_max_sync(0xffffffffu, lo);
  hi = __reduce_min_sync(0xffffffffu, hi);
  if (lane == 0)
    band[col] = make_int2(lo, hi);
}

} // namespace

size_t cb_fp_smem(const Geom &g) {
  return (size_t(cb_vz_floats(g.nz)) + size_t(kFpWarps) * 2 * size_t(g.nx + g.ny + 2)) *
         sizeof(float);
}

namespace {
// Passes over the rows with r rows per lane: aligned to the first row above
// the source (see cb_fp_kernel,
// cb_bp_scatter).
struct RowPasses {
  int rpl, v0, np;
};
RowPasses row_passes(const Geom &g, int r) {
  RowPasses p;
  p.rpl = r;
  p.v0 = g.mid - ((g.mid + 16 * r - 1) / (16 * r)) * 16 * r;
  p.np = (g.nv - p.v0 + 32 * r - 1) / (32 * r);
  return p;
}
// Rows per lane of the scatter: as for the forward projector, with a pass's
// reading of the cell and its band worth two rows per lane.  512^3 with 768
// rows: 476 ms with 2 rows per lane, 401 with 3, 364 with 4, 326 with 6,
// 320 with 8; 288 rows 8.5 ms with 10, 9.6 with two passes of 6.
RowPasses cb_scatter_rows(const Geom &g) {
  RowPasses best = row_passes(g, 1);
  for (int r : {2, 3, 4, 6, 8, 10}) {
    const RowPasses p = row_passes(g, r);
    if (p.np * (p.rpl + 2) <= best.np * (best.rpl + 2))
      best = p;
  }
  return best;
}
} // namespace

namespace {
// The edge form serves detectors whose outermost rows are past the volume's
// ends in more than an eighth of its depth.  First form over edge form: 151^3
// from 230 rows 0.65 of the time with every row inside, 0.94 at a tenth of the
// depth, 1.11 at a sixth, 1.3 at a half; 256^3 from 384 0.63, 0.84, 1.04, 1.27.
// Three rows per lane (65 to 96 rows) stay with the first: 64^3 from 96 0.85 at
// a half.
bool cb_scatter_edge(const Geom &g) {
  return g.row_edge > 0.12f && cb_scatter_rows(g).rpl != 3;
}
// Rows per lane of the edge form: the least idle rows.
int cb_edge_rows(const Geom &g) {
  auto idle = [&](int r) { return (g.nv + 32 * r - 1) / (32 * r) * 32 * r - g.nv; };
  int best = 2;
  for (int r : {3, 1})
    if (idle(r) < idle(best))
      best = r;
  return best;
}
} // namespace

int cb_backward_scatter(const Geom &g, const float *pix, float *vol, int pre,
                        const int2 *hrange, int grid, cudaStream_t st) {
  if (cudaMemsetAsync(vol, 0, size_t(g.nx) * g.ny * g.nz * sizeof(float), st) != cudaSuccess)
    return 2;
  const size_t smem = cb_fp_smem(g);
  const int cap = g.nx + g.ny + 2;
  if (cb_scatter_edge(g)) {
#define CB_SC_EDGE(R)                                                                      \
  (pre ? cb_bp_scatter_edge<R, true><<<grid, kFpWarps * 32, smem, st>>>(g, pix, vol, hrange, cap) \
       : cb_bp_scatter_edge<R, false><<<grid, kFpWarps * 32, smem, st>>>(g, pix, vol, hrange, cap))
    switch (cb_edge_rows(g)) {
    case 1:
      CB_SC_EDGE(1);
      break;
    case 2:
      CB_SC_EDGE(2);
      break;
    default:
      CB_SC_EDGE(3);
    }
#undef CB_SC_EDGE
    return 0;
  }
  const RowPasses p = cb_scatter_rows(g);
#define CB_SC_GO(R)                                                                        \
  (pre ? cb_bp_scatter<R, true><<<grid, kFpWarps * 32, smem, st>>>(g, pix, vol, hrange, cap,   \
                                                                   p.v0, p.np)              \
       : cb_bp_scatter<R, false><<<grid, kFpWarps * 32, smem, st>>>(g, pix, vol, hrange, cap,  \
                                                                    p.v0, p.np))
  switch (p.rpl) {
  case 1:
    CB_SC_GO(1);
    break;
  case 2:
    CB_SC_GO(2);
    break;
  case 3:
    CB_SC_GO(3);
    break;
  case 4:
    CB_SC_GO(4);
    break;
  case 6:
    CB_SC_GO(6);
    break;
  case 8:
    CB_SC_GO(8);
    break;
  default:
    CB_SC_GO(10);
  }
#undef CB_SC_GO
  return 0;
}

int cb_column_bands(const Geom &g, int2 *band, cudaStream_t st) {
  const int ncol = g.nx * g.ny;
  cb_column_band_kernel<<<(ncol + kBandWarps - 1) / kBandWarps, kBandWarps * 32, 0, st>>>(g, band);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 2;
}

namespace {
// Rows per lane: the fewest instructions per cell, where a pass costs about
// one more row per lane for reading the cell.
RowPasses cb_fp_rows(const Geom &g) {
  if (g.tune_rpl >= 2 && g.tune_rpl <= 12 && g.tune_rpl % 2 == 0)
    return row_passes(g, g.tune_rpl);
  if (row_passes(g, 1).np == 1)
    return row_passes(g, 1);
  RowPasses best = row_passes(g, 2);
  for (int r = 4; r <= 12; r += 2) {
    const RowPasses p = row_passes(g, r);
    if (p.np * (p.rpl + 1) <= best.np * (best.rpl + 1))
      best = p;
  }
  return best;
}

} // namespace
int cb_fp_rows_per_lane(const Geom &g) { return cb_fp_rows(g).rpl; }
namespace {

template <int EPI>
void launch_cb_fp(const Geom &g, const float *vol, float *pix, const Epi &e, const int2 *hrange,
                  int grid, cudaStream_t st, int nb) {
  const size_t smem = cb_fp_smem(g);
  const int cap = g.nx + g.ny + 2;
  const RowPasses p = cb_fp_rows(g);
#define CB_FP_GO(R, B)                                                                     \
  cb_fp_kernel<EPI, R, B><<<grid, kFpWarps * 32, smem, st>>>(g, vol, pix, e, hrange, cap, nb,  \
                                                             p.v0, p.np)
#define CB_FP_RPL(B)                                                                       \
  (p.rpl == 1   ? CB_FP_GO(1, B)                                                            \
   : p.rpl == 2 ? CB_FP_GO(2, B)                                                            \
   : p.rpl == 4 ? CB_FP_GO(4, B)                                                            \
   : p.rpl == 6 ? CB_FP_GO(6, B)                                                            \
   : p.rpl == 8 ? CB_FP_GO(8, B)                                                            \
   : p.rpl == 10 ? CB_FP_GO(10, B)                                                          \
                 : CB_FP_GO(12, B))
  if constexpr (EPI == EPI_STORE) {
    if (nb > 1) {
      CB_FP_RPL(true);
      return;
    }
  }
  CB_FP_RPL(false);
#undef CB_FP_RPL
#undef CB_FP_GO
}
} // namespace

int cb_prepare(const Geom &g) {
  // the limit is the function's, not the plan's: the largest any plan uses
  const int fp = 200 * 1024;
#define CB_FP_ALL(R)                                                                       \
  (const void *)cb_fp_kernel<EPI_STORE, R, false>, (const void *)cb_fp_kernel<EPI_NORM, R, false>, \
      (const void *)cb_fp_kernel<EPI_SIRT, R, false>,                                       \
      (const void *)cb_fp_kernel<EPI_MLEM, R, false>, (const void *)cb_fp_kernel<EPI_STORE, R, true>
  const void *fps[] = {CB_FP_ALL(1), CB_FP_ALL(2), CB_FP_ALL(4), CB_FP_ALL(6), CB_FP_ALL(8), CB_FP_ALL(10), CB_FP_ALL(12),
                       (const void *)cb_bp_scatter_edge<1, false>,
                       (const void *)cb_bp_scatter_edge<1, true>,
                       (const void *)cb_bp_scatter_edge<2, false>,
                       (const void *)cb_bp_scatter_edge<2, true>,
                       (const void *)cb_bp_scatter_edge<3, false>,
                       (const void *)cb_bp_scatter_edge<3, true>,
                       (const void *)cb_bp_scatter<1, false>,
                       (const void *)cb_bp_scatter<1, true>,
                       (const void *)cb_bp_scatter<2, false>,
                       (const void *)cb_bp_scatter<2, true>,
                       (const void *)cb_bp_scatter<3, false>,
                       (const void *)cb_bp_scatter<3, true>,
                       (const void *)cb_bp_scatter<4, false>,
                       (const void *)cb_bp_scatter<4, true>,
                       (const void *)cb_bp_scatter<6, false>,
                       (const void *)cb_bp_scatter<6, true>,
                       (const void *)cb_bp_scatter<8, false>,
                       (const void *)cb_bp_scatter<8, true>,
                       (const void *)cb_bp_scatter<10, false>,
                       (const void *)cb_bp_scatter<10, true>};
#undef CB_FP_ALL
  for (const void *f : fps)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, fp) != cudaSuccess)
      return 1;
  return cb_bp_prepare(g);
}

int cb_forward(const Geom &g, const float *vol, float *pix, int mode, const Epi &e,
               const int2 *hrange, int grid, cudaStream_t st, int nb) {
  switch (mode) {
  case EPI_STORE:
    launch_cb_fp<EPI_STORE>(g, vol, pix, e, hrange, grid, st, nb);
    break;
  case EPI_NORM:
    launch_cb_fp<EPI_NORM>(g, vol, pix, e, hrange, grid, st, nb);
    break;
  case EPI_SIRT:
    launch_cb_fp<EPI_SIRT>(g, vol, pix, e, hrange, grid, st, nb);
    break;
  case EPI_MLEM:
    launch_cb_fp<EPI_MLEM>(g, vol, pix, e, hrange, grid, st, nb);
    break;
  default:
    return 1;
  }
  return 0;
}

} // namespace ccpi
