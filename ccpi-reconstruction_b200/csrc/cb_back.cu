// Cone-beam back projector for sm_100a (cone_beam::b2D,
// Core/src/c2D.cpp:948-1119), a gather in the reference's summation order.
//
// cone_beam::calc_ah_z (c2D.cpp:640-751) adds, for every voxel of a column,
// first the band rows of every ray (list order: angle, then detector
// column; rows ascending), each row v feeding its slice k(v) with
// p (mz - a0) and the neighbour on the far side of the plane it may cross
// (k - 1 below the source, k + 1 above it) with p (a1 - mz); then the edge
// rows of every ray (below the band descending, above it ascending).
//
// cb_bp_tile: one lane owns one voxel column, a warp 8 x 4 columns, a CTA a
// tile of such warps and one chunk of slices.  For each angle the CTA stages
// the patch of detector columns and rows that its tile and chunk can see
// (times d_conv unless the producer already scaled it) in shared memory;
// then every lane takes its column's rays in turn.  All lanes step through
// the detector rows together: k(v) only rises with v, so a lane keeps the
// sums of the two slices that the current row feeds in registers and swaps
// one of them with its accumulators in shared memory ([slice][lane], no bank
// conflicts) when its slice changes.  Each voxel's additions are the
// reference's, in its order, with the same unfused roundings: the result is
// the reference's bit for bit.
//
// Bound: instruction issue (63 % issue slots busy at 256^3, where the row
// loop takes half of a central tile's time, the copies and barriers a
// quarter, ray set-up the rest).  Against one CTA per column with the rows
// over its threads (now cb_bp_column, for few columns), whose rows went
// through shared memory to the voxels: 512^3 1245 -> 625 ms, 256^3 98.6 ->
// 55 ms, 128^3 9.97 -> 7.3 ms.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "cb_common.cuh"
#include "kernels.h"

namespace ccpi {
namespace {

constexpr int kTileX = 8, kTileY = 4;     // lanes of a warp over the columns
constexpr int kMaxWarps = 8;              // warps of a CTA
constexpr int kMaxRaysPerAngle = 24;      // rays per (column, angle), an error beyond
constexpr int kGuardLo = 3, kGuardHi = 3; // accumulator rows below / above the chunk
constexpr int kRow = 128;                 // bytes of a slice's accumulators of a warp
constexpr int kMaxGroup = 8;              // angles staged together, parts of a chunk

struct TileShape {
  int wx, wy;    // warps of a CTA along x and y
  int zc;        // slices per chunk
  int ntx, nty, nzc;
  int rcap, cap; // staged rows, staged patch floats
};

// Accumulator rows of a chunk: slices Z0 - kGuardLo .. Z0 + zc + kGuardHi - 1.
__host__ __device__ inline int acc_rows(int zc) { return zc + kGuardLo + kGuardHi; }

size_t tile_smem(const TileShape &t) {
  return sizeof(float) * (size_t(t.wx) * t.wy * acc_rows(t.zc) * 32 +
                          ((2 * acc_rows(t.zc) + 3) & ~3) + size_t(2) * t.rcap + t.cap);
}

enum RowMode { LOWER = 0, UPPER = 1, EDGE_LO = 2, EDGE_UP = 3 };
constexpr bool mode_up(int mode) { return mode == UPPER || mode == EDGE_UP; }

// Shared memory by 32-bit address.  The accumulators are only touched
// through these, in program order; everything else the row loops read is
// loaded freely around them.
__device__ __forceinline__ float lds(unsigned a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
// A table entry, which no store changes while rows are added.
__device__ __forceinline__ float ldt(unsigned a) {
  float v;
  asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts(unsigned a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v));
}

// Slice index k of a row is int(x) (edge rows below the band: int(x) - 1):
// k >= K exactly when x >= enter(K), truncation toward zero included.
__device__ __forceinline__ float enter(int K) {
  return K >= 1 ? float(K) : __int_as_float(__float_as_int(float(K - 1)) - 1);
}

template <int MODE>
__device__ __forceinline__ float row_x(const Geom &g, float av, float dz) {
  return __fadd_rn(MODE == EDGE_LO ? g.pzbz1 : g.pzbz, __fmul_rn(av, dz));
}

// First row v of [lo, hi) with x(v) >= T (x rises with v), hi if none.
// slack = 0: exactly, by testing x around the estimate for evenly spaced
// rows; slack = +-1 (evenly spaced rows only): that row or up to two
// before (-1) / after (+1) it, without a look at the rows.
template <int MODE>
__device__ __forceinline__ int first_row(const Geom &g, float inv_av, float av, float T, int lo,
                                         int hi, int slack) {
  const float e =
      ((T - (MODE == EDGE_LO ? g.pzbz1 : g.pzbz)) * inv_av - g.dz0) * g.inv_pitch + float(slack);
  int v = int(ceilf(fminf(fmaxf(e, float(lo)), float(hi))));
  if (slack == 0) {
    while (v > lo && row_x<MODE>(g, av, __ldg(g.dz + v - 1)) >= T)
      v--;
    while (v < hi && row_x<MODE>(g, av, __ldg(g.dz + v)) < T)
      v++;
  }
  return v;
}

// One column's running state along the rows of one ray: slice k's sum A,
// its neighbour's sum B (k + 1 above the source, k - 1 below) and the plane
// between them.
struct Run {
  float a0, a1, av;
  float A, B, zc;
  unsigned ap; // accumulator of slice k
  unsigned zp; // table entry of slice k: {plane k, plane k + 1}
};

// The slice changes by one: the sum that no later row of this ray reaches
// goes back to shared memory, the next one comes in.
template <int MODE> __device__ __forceinline__ void next_slice(Run &L) {
  if (mode_up(MODE)) {
    sts(L.ap, L.A);
    L.A = L.B;
    L.ap += kRow;
    L.zp += 8;
    L.B = lds(L.ap + kRow);
    L.zc = lds(L.zp + 4);
  } else if (MODE == LOWER) {
    sts(L.ap - kRow, L.B);
    L.B = L.A;
    L.ap += kRow;
    L.zp += 8;
    L.A = lds(L.ap);
    L.zc = lds(L.zp);
  } else {
    sts(L.ap, L.A);
    L.A = L.B;
    L.ap -= kRow;
    L.zp -= 8;
    L.B = lds(L.ap - kRow);
    L.zc = lds(L.zp);
  }
}

// Both contributions of one row (c2D.cpp:694-711).
__device__ __forceinline__ void add_row(Run &L, float iz, float p) {
  const float mz = fmin_ref(__fmul_rn(L.zc, iz), L.a1);
  L.A = __fadd_rn(L.A, __fmul_rn(p, __fsub_rn(mz, L.a0)));
  L.B = __fadd_rn(L.B, __fmul_rn(p, __fsub_rn(L.a1, mz)));
}

// Where the fast row loop finds its operands.
struct Fast {
  unsigned kb;   // slot of slice int(x): bits of (2^23 + x, toward zero) - kb,
  unsigned top;  // at most top (also for slices below the first slot: the
                 // difference wraps); top and its neighbour are guards
  unsigned acc;  // this lane's accumulator in slot 0
  unsigned zt;   // table entry of slot 0 (+ 4 for the upper plane)
  unsigned n;    // slices of this part of the chunk: slots 2 .. 1 + n
  const float2 *tab; // indexed by the row
};

// Rows [R0, R1) of a warp none of whose columns has to skip one, all x >= 0.
// Everything that does not depend on the running sums (slice, plane, both
// contributions, the next slice's sum) is formed for four rows at a time, so
// that the only chain from row to row is a move and an add.  JUMP: a row may
// be more than one slice past the row before it.  MASK (with JUMP): slots 0,
// 1 and past 1 + F.n are other parts' accumulators, not guards: nothing is
// added to them (+0 changes no sum: none is ever -0).
template <int MODE, bool JUMP, bool MASK>
__device__ __forceinline__ void rows_fast(const Geom &g, Run &L, int R0, int R1, const Fast &F,
                                          const float *pp) {
  const float pz = g.pzbz;
  auto rows = [&](int v, auto count) {
    constexpr int N = decltype(count)::value;
    float c1[N], c2[N], nx[N], ax[N];
    unsigned ad[N];
#pragma unroll
    for (int u = 0; u < N; u++) {
      const float2 t = F.tab[v + u];
      const float x = __fadd_rn(pz, __fmul_rn(L.av, t.x));
      const unsigned slot = min(__float_as_uint(__fadd_rz(x, 8388608.0f)) - F.kb, F.top);
      ad[u] = F.acc + slot * kRow;
      // the sum that enters with this row's slice: no earlier row of the
      // ray has touched it
      nx[u] = lds(ad[u] + (MODE == UPPER ? kRow : 0));
      if (JUMP)
        ax[u] = lds(ad[u] - (MODE == UPPER ? 0 : kRow));
      const float p = pp[v + u];
      const float mz = fmin_ref(__fmul_rn(ldt(F.zt + slot * 8), t.y), L.a1);
      c1[u] = __fmul_rn(p, __fsub_rn(mz, L.a0));
      c2[u] = __fmul_rn(p, __fsub_rn(L.a1, mz));
      if (MASK) {
        c1[u] = slot - 2 < F.n ? c1[u] : 0.0f;
        c2[u] = slot - (MODE == UPPER ? 1 : 3) < F.n ? c2[u] : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < N; u++) {
      // a new slice: the sum that no later row reaches goes back, the
      // neighbour's becomes the slice's own (below the source the slice's
      // becomes the neighbour's), the next one comes in; predicated rather
      // than a branch, since some lane has a new slice at nearly every row
      if (!JUMP) {
        if (MODE == UPPER)
          asm volatile("{ .reg .pred p;\n\t"
                       "setp.ne.u32 p, %2, %3;\n\t"
                       "@p st.shared.f32 [%2], %0;\n\t"
                       "@p mov.f32 %0, %1;\n\t"
                       "@p mov.f32 %1, %4;\n\t}"
                       : "+f"(L.A), "+f"(L.B)
                       : "r"(L.ap), "r"(ad[u]), "f"(nx[u]));
        else
          asm volatile("{ .reg .pred p;\n\t"
                       "setp.ne.u32 p, %2, %3;\n\t"
                       "@p st.shared.f32 [%2+%5], %1;\n\t"
                       "@p mov.f32 %1, %0;\n\t"
                       "@p mov.f32 %0, %4;\n\t}"
                       : "+f"(L.A), "+f"(L.B)
                       : "r"(L.ap), "r"(ad[u]), "f"(nx[u]), "n"(-kRow));
      } else if (ad[u] != L.ap) {
        const bool one = ad[u] == L.ap + kRow;
        if (MODE == UPPER) {
          sts(L.ap, L.A);
          if (!one)
            sts(L.ap + kRow, L.B);
          L.A = one ? L.B : ax[u];
          L.B = nx[u];
        } else {
          sts(L.ap - kRow, L.B);
          if (!one)
            sts(L.ap, L.A);
          L.B = one ? L.A : ax[u];
          L.A = nx[u];
        }
      }
      L.ap = ad[u];
      L.A = __fadd_rn(L.A, c1[u]);
      L.B = __fadd_rn(L.B, c2[u]);
    }
  };
  int v = R0;
  for (; v + 4 <= R1; v += 4)
    rows(v, std::integral_constant<int, 4>());
  for (; v < R1; v++)
    rows(v, std::integral_constant<int, 1>());
}

// Rows [R0, R1) of one column with every case handled: it adds only its rows
// [lo, hi) and only to slices [Z0, Z1), slices may change by any number, k is
// the current slice kept within [kmin, kmax].  tab / pp (staged) or the
// sinogram itself.
template <int MODE, bool GLOBAL>
__device__ __forceinline__ void rows_any(const Geom &g, Run &L, int R0, int R1, int lo, int hi,
                                         int Z0, int Z1, int k, int kmin, int kmax, bool on,
                                         const float2 *tab,
                                         const float *pp, const float *dp) {
  for (int n = 0; n < R1 - R0; n++) {
    const int v = MODE == EDGE_LO ? R1 - 1 - n : R0 + n;
    const float dz = GLOBAL ? __ldg(g.dz + v) : tab[v].x;
    const float iz = GLOBAL ? __ldg(g.iz + v) : tab[v].y;
    float p = GLOBAL ? __ldg(pp + v) : pp[v];
    if (GLOBAL && dp)
      p = __fmul_rn(p, __ldg(dp + v));
    const float x = row_x<MODE>(g, L.av, dz);
    if (MODE == EDGE_LO) {
      while (on && k > kmin && x < enter(k + 1)) {
        next_slice<MODE>(L);
        k--;
      }
    } else {
      while (on && k < kmax && x >= enter(k + 1)) {
        next_slice<MODE>(L);
        k++;
      }
    }
    if (v >= lo && v < hi) {
      const float A = L.A, B = L.B;
      add_row(L, iz, p);
      const int kn = mode_up(MODE) ? k + 1 : k - 1;
      L.A = (k >= Z0 && k < Z1) ? L.A : A;
      L.B = (kn >= Z0 && kn < Z1) ? L.B : B;
    }
  }
}

// What a CTA can see of one projection, staged or not.
struct Window {
  int w0, w1, H0, H1; // rows [w0, w1), detector columns [H0, H1]
  int stride;         // floats per staged column
  int rofs, pofs;     // its rows in the table, its patch
  __device__ int rows() const { return w1 - w0; }
  __device__ int floats() const { return (H1 - H0 + 1) * stride; }
};

// The rows of one mode of one ray per lane (ok: the lane's column has one).
// acc, ztab: this lane's accumulator and the table entry of slice Zc -
// kGuardLo, Zc the chunk's first slice; [Z0, Z1) the chunk (whole) or a part.
template <int MODE>
__device__ __forceinline__ void
ray_rows(const Geom &g, const Window &W, bool fits, int a, int h, float a0, float a1, bool ok,
         int min_v, int max_v, int Zc, int Z0, int Z1, bool whole, unsigned acc, unsigned ztab,
         const float2 *tab, const float *patch, const float *pix, const float *dconv) {
  const int slack = g.even_rows ? 1 : 0;
  Run L;
  L.a0 = a0;
  L.a1 = a1;
  L.av = ok ? __fmul_rn(a0, g.inv_dz) : 0.0f;
  // the column's rows [lo, hi) of this mode; those that feed the chunk's
  // slices lie in [r0, r1)
  const int lo = MODE == LOWER ? min_v : MODE == UPPER ? max(g.mid, min_v)
                 : MODE == EDGE_LO ? 0 : max(max_v, 0);
  const int hi = MODE == LOWER ? min(g.mid, max_v) : MODE == UPPER ? max_v
                 : MODE == EDGE_LO ? min(min_v, g.nv) : g.nv;
  int r0 = hi, r1 = hi;
  if (ok && lo < hi) {
    // LOWER: slices Z0 .. Z1 (Z1's rows feed Z1 - 1); UPPER: Z0 - 1 ..
    // Z1 - 1, where band rows below slice 0 count as slice -1; EDGE_LO has
    // k = int(x) - 1
    const float ia = __fdividef(1.0f, L.av);
    const float Ta = enter(mode_up(MODE) ? Z0 - 1 : MODE == EDGE_LO ? Z0 + 1 : Z0);
    const float Tb = enter(mode_up(MODE) ? Z1 : MODE == EDGE_LO ? Z1 + 2 : Z1 + 1);
    r0 = (MODE == UPPER && Z0 == 0) ? lo : first_row<MODE>(g, ia, L.av, Ta, lo, hi, -slack);
    r1 = first_row<MODE>(g, ia, L.av, Tb, r0, hi, slack);
  }
  const bool on = ok && r0 < r1;
  if (!__any_sync(0xffffffffu, on))
    return;
  const int R0 = __reduce_min_sync(0xffffffffu, on ? r0 : INT_MAX);
  const int R1 = __reduce_max_sync(0xffffffffu, on ? r1 : 0);
  // a lane without rows stays on one slice (av = 0) and stores nothing
  L.av = on ? L.av : 0.0f;
  const float x = row_x<MODE>(g, L.av, __ldg(g.dz + (MODE == EDGE_LO ? R1 - 1 : R0)));
  const bool staged =
      __all_sync(0xffffffffu, fits && R0 >= W.w0 && R1 <= W.w1 && !(on && (h < W.H0 || h > W.H1)));
  // the fast loop: no lane skips a row, int(x) by adding 2^23
  const bool fast = (MODE == LOWER || MODE == UPPER) && staged &&
                    !__any_sync(0xffffffffu, on && (R0 < lo || R1 > hi || x < 0.0f));
  // slices next to the chunk act on guard accumulators that nothing reads;
  // next to a part of the chunk (whole is false) the loops add nothing
  const int kmin = (MODE == UPPER && Z0 == 0) ? -1 : mode_up(MODE) ? Z0 - 2 : Z0 - 1;
  const int kmax = mode_up(MODE) ? Z1 : Z1 + 1;
  const int k = on ? min(max(int(x) - (MODE == EDGE_LO ? 1 : 0), kmin), kmax) : Zc;
  // slot 0: slice Z0 - 2 (its lower neighbour is a guard or another part's),
  // top: Z1 + 1
  const int below = Z0 - Zc + kGuardLo - 2;
  Fast F;
  F.kb = 0x4b000000u + unsigned(Z0 - 2);
  F.top = unsigned(Z1 - Z0 + 3);
  F.n = unsigned(Z1 - Z0);
  F.acc = acc + below * kRow;
  F.zt = ztab + below * 8 + (mode_up(MODE) ? 4 : 0);
  F.tab = tab + W.rofs - W.w0;
  const unsigned slot =
      fast ? below + min(__float_as_uint(__fadd_rz(x, 8388608.0f)) - F.kb, F.top)
           : unsigned(k - Zc + kGuardLo);
  L.ap = acc + slot * kRow;
  L.zp = ztab + slot * 8;
  L.A = lds(L.ap);
  L.B = lds(mode_up(MODE) ? L.ap + kRow : L.ap - kRow);
  const float *pp = patch + W.pofs + (min(max(h, W.H0), W.H1) - W.H0) * W.stride - W.w0;
  if (fast) {
    if (!whole)
      rows_fast<MODE, true, true>(g, L, R0, R1, F, pp);
    else if (__any_sync(0xffffffffu, on && !(__fmul_rn(L.av, g.pitch_max) < 0.98f)))
      rows_fast<MODE, true, false>(g, L, R0, R1, F, pp);
    else
      rows_fast<MODE, false, false>(g, L, R0, R1, F, pp);
  } else {
    L.zc = lds(mode_up(MODE) ? L.zp + 4 : L.zp);
    const int l = on ? lo : 0, u = on ? hi : 0, hc = on ? h : 0;
    if (staged)
      rows_any<MODE, false>(g, L, R0, R1, l, u, Z0, Z1, k, kmin, kmax, on, F.tab, pp, nullptr);
    else
      rows_any<MODE, true>(g, L, R0, R1, l, u, Z0, Z1, k, kmin, kmax, on, nullptr,
                           pix + (i64(a) * g.nh + hc) * g.nv,
                           dconv ? dconv + i64(hc) * g.nv : nullptr);
  }
  if (on) {
    sts(L.ap, L.A);
    sts(mode_up(MODE) ? L.ap + kRow : L.ap - kRow, L.B);
  }
}

// Detector columns [hl, hh] that the square of edges ex, ey with corner
// (t, u) (axial distance from the source and offset along the detector, at
// angle cos, sin) projects to; the smallest axial distance and the largest.
__device__ __forceinline__ void project_square(float t, float u, float cf, float sf, float ex,
                                               float ey, float hscale, float hofs, float &hl,
                                               float &hh, float &tl, float &th) {
  hl = INFINITY;
  hh = -INFINITY;
  tl = INFINITY;
  th = -INFINITY;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float ox = (q & 1) ? ex : 0.0f, oy = (q & 2) ? ey : 0.0f;
    const float tq = t + cf * ox + sf * oy, uq = u - sf * ox + cf * oy;
    const float hq = __fdividef(uq, tq) * hscale + hofs;
    tl = fminf(tl, tq);
    th = fmaxf(th, tq);
    hl = fminf(hl, hq);
    hh = fmaxf(hh, hq);
  }
}

// The window of slices [Z0, Z1) of a tile of cx x cy columns at angle a: the
// detector columns between the projections of its corners, and the rows
// whose slices, over the tile's alphas, can lie in [Z0 - 1, Z1].
__device__ Window tile_window(const Geom &g, int a, int tx0, int ty0, int cx, int cy, int Z0,
                              int Z1) {
  const double c = g.cosA[a], s = g.sinA[a];
  const double X0 = g.origin[0] + double(tx0) * g.size[0];
  const double Y0 = g.origin[1] + double(ty0) * g.size[1];
  const float clf = float(g.cl), hmargin = 0.02f + 4e-6f * float(g.nh);
  float hl, hh, tl, th;
  project_square(float(c * X0 + s * Y0 - g.src[0]), float(c * Y0 - s * X0 - g.src[1]), float(c),
                 float(s), float(cx * g.size[0]), float(cy * g.size[1]), float(g.cl * g.cipix),
                 float(g.chpix0), hl, hh, tl, th);
  Window W;
  W.H0 = 0;
  W.H1 = g.nh - 1;
  W.w0 = 0;
  W.w1 = g.nv;
  if (tl > 1e-3f * clf) {
    W.H0 = int(fminf(fmaxf(floorf(hl - hmargin), 0.0f), float(g.nh - 1)));
    W.H1 = int(fminf(fmaxf(ceilf(hh + hmargin), 0.0f), float(g.nh - 1)));
    const float al = tl / clf * g.inv_dz, ah = th / clf * g.inv_dz;
    const float zl = float(Z0 - 2) - g.pzbz, zh = float(Z1 + 2) - g.pzbz;
    const float dl = zl / (zl < 0.0f ? al : ah), dh = zh / (zh < 0.0f ? ah : al);
    const float vl = floorf((dl - g.dz0) * g.inv_pitch) - 3.0f;
    const float vh = ceilf((dh - g.dz0) * g.inv_pitch) + 4.0f;
    W.w0 = int(fminf(fmaxf(vl, 0.0f), float(g.nv)));
    W.w1 = max(W.w0, int(fminf(fmaxf(vh, 0.0f), float(g.nv))));
  }
  W.stride = (W.w1 - W.w0) | 1; // odd: distinct columns, distinct banks
  W.rofs = W.pofs = 0;
  return W;
}

template <int EPI>
__global__ void __launch_bounds__(kMaxWarps * 32, 2)
    cb_bp_tile(Geom g, const float *__restrict__ pix0, float *__restrict__ vol0, Epi e, int *err,
               TileShape t) {
  extern __shared__ float4 smem4[];
  __shared__ Window swin[kMaxGroup];
  float *smem = reinterpret_cast<float *>(smem4);
  const int nw = t.wx * t.wy, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int arows = acc_rows(t.zc);
  float2 *zt = reinterpret_cast<float2 *>(smem4); // per slot its slice's {plane k, plane k + 1}
  float *wacc = smem + ((2 * arows + 3) & ~3) + wib * arows * 32;
  float2 *tab = reinterpret_cast<float2 *>(smem + ((2 * arows + 3) & ~3) + nw * arows * 32);
  float *patch = reinterpret_cast<float *>(tab + t.rcap);
  const unsigned acc = unsigned(__cvta_generic_to_shared(wacc + lane));
  const unsigned ztab = unsigned(__cvta_generic_to_shared(zt));
  const int chunk = blockIdx.x % t.nzc, tile = blockIdx.x / t.nzc;
  const int cx = t.wx * kTileX, cy = t.wy * kTileY;
  const int tx0 = (tile / t.nty) * cx, ty0 = (tile % t.nty) * cy;
  const int Z0 = chunk * t.zc, Z1 = min(Z0 + t.zc, g.nz);
  const int i = tx0 + (wib % t.wx) * kTileX + (lane & (kTileX - 1));
  const int j = ty0 + (wib / t.wx) * kTileY + lane / kTileX;
  const float *pix = pix0 + i64(blockIdx.y) * g.na * g.nh * g.nv;
  float *vol = vol0 + i64(blockIdx.y) * g.nx * g.ny * g.nz;
  const float *dconv = e.pre ? nullptr : g.dconv;

  for (int r = lane; r < arows * 32; r += 32)
    wacc[r] = 0.0f;
  for (int r = threadIdx.x; r < arows; r += blockDim.x) {
    const int k = Z0 - kGuardLo + r;
    zt[r] = make_float2(g.vz[min(max(k, 0), g.nz)], g.vz[min(max(k + 1, 0), g.nz)]);
  }

  // the column's square and its band rows (c2D.cpp:657-676)
  const double x0 = g.origin[0] + double(i) * g.size[0];
  const double xn = g.origin[0] + double(i + 1) * g.size[0];
  const double y0 = g.origin[1] + double(j) * g.size[1];
  const double yn = g.origin[1] + double(j + 1) * g.size[1];
  const int col = (i < g.nx && j < g.ny) ? i * g.ny + j : -1;
  const int2 band = col >= 0 ? g.colband[col] : make_int2(0, 0);
  const float bx = float(g.size[0]), by = float(g.size[1]);
  const float clf = float(g.cl), hscale = float(g.cl * g.cipix), hofs = float(g.chpix0);
  // A column's candidate rays.  The float projections hl, hh of its corners
  // are within hround (columns) of the reference's doubles, whose range is
  // floor(min) .. floor(max) of the columns' even spacing (cb_column_hrange).
  // With every column within 0.01 of that spacing (even_cols) a ray hmargin
  // below hl misses the voxel column, and one below hh - hround is in the
  // range; one between that and hh + hmargin is put to the reference's own
  // range if it crosses.  Other detectors take that range for every column.
  const float hround = 4e-6f * float(g.nh), hmargin = 0.02f + hround;
  const double eps = double(kEps);
  const int kb = int(g.pzbz); // every row above the source has k >= kb, every other k <= kb

  // one projection's window: its patch and its rows' tables.  The copies are
  // asynchronous: every load of the group is in flight at once.
  auto stage = [&](const Window &W, int a, int rofs, int pofs) {
    const int R = W.rows();
    for (int q = W.H0 + wib; q <= W.H1; q += nw) {
      const float *src = pix + (i64(a) * g.nh + q) * g.nv + W.w0;
      const unsigned dst = unsigned(__cvta_generic_to_shared(patch)) +
                           4 * (pofs + (q - W.H0) * W.stride);
#pragma unroll 4
      for (int r = lane; r < R; r += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * r), "l"(src + r));
    }
    for (int r = threadIdx.x; r < R; r += blockDim.x)
      tab[rofs + r] = make_float2(__ldg(g.dz + W.w0 + r), __ldg(g.iz + W.w0 + r));
  };
  // d_conv, on the elements this thread copied itself
  auto scale = [&](const Window &W, int pofs) {
    const int R = W.rows();
    for (int q = W.H0 + wib; q <= W.H1; q += nw) {
      const float *dsc = g.dconv + i64(q) * g.nv + W.w0;
      float *dst = patch + pofs + (q - W.H0) * W.stride;
#pragma unroll 4
      for (int r = lane; r < R; r += 32)
        dst[r] = __fmul_rn(dst[r], __ldg(dsc + r));
    }
  };
  auto staged = [&] { asm volatile("cp.async.wait_all;" ::: "memory"); };

  for (int pass = 0; pass < 2; pass++) {
    const bool has =
        col >= 0 && (pass == 0 ? band.y > band.x : (band.x > 0 || band.y < g.nv));
    if (!__syncthreads_or(has))
      continue;
    int group = 0;
    for (int ag = 0; ag < g.na; ag += group) {
      // ---- what the tile and chunk can see of the next projections (one
      // thread each), and how many of them fit the staging area
      const int ahead = min(kMaxGroup, g.na - ag);
      if (int(threadIdx.x) < ahead)
        swin[threadIdx.x] = tile_window(g, ag + threadIdx.x, tx0, ty0, cx, cy, Z0, Z1);
      __syncthreads();
      int rows = 0, floats = 0, items = 0;
      for (; items < ahead; items++) {
        const Window W = swin[items];
        if (rows + W.rows() > t.rcap || floats + W.floats() > t.cap)
          break;
        rows += W.rows();
        floats += W.floats();
      }
      // one that is too large alone is taken in parts of the chunk; one
      // that no split makes fit is read from the sinogram itself
      int parts = 1;
      bool fits = items > 0;
      for (int p = 2; !fits && p <= kMaxGroup; p *= 2) {
        const int sz = (t.zc + p - 1) / p;
        __syncthreads();
        if (int(threadIdx.x) < p)
          swin[threadIdx.x] = tile_window(g, ag, tx0, ty0, cx, cy, Z0 + threadIdx.x * sz,
                                          min(Z0 + int(threadIdx.x + 1) * sz, Z1));
        __syncthreads();
        fits = true;
        for (int q = 0; q < p; q++)
          fits = fits && swin[q].rows() <= t.rcap && swin[q].floats() <= t.cap;
        parts = p;
      }
      group = max(items, 1);
      if (items == 0)
        items = fits ? parts : 1;
      const bool whole = items == group && fits;
      rows = floats = 0;
      for (int q = 0; whole && q < items; q++) {
        stage(swin[q], ag + q, rows, floats);
        rows += swin[q].rows();
        floats += swin[q].floats();
      }
      if (whole) {
        staged();
        floats = 0;
        for (int q = 0; dconv && q < items; q++) {
          scale(swin[q], floats);
          floats += swin[q].floats();
        }
        __syncthreads();
      }
      rows = floats = 0;
      for (int q = 0; q < items; q++) {
        const int a = whole ? ag + q : ag;
        int Zs = Z0, Ze = Z1;
        Window W = swin[q];
        if (whole) {
          W.rofs = rows;
          W.pofs = floats;
          rows += W.rows();
          floats += W.floats();
        } else if (fits) {
          const int sz = (t.zc + parts - 1) / parts;
          Zs = Z0 + q * sz;
          Ze = min(Zs + sz, Z1);
          if (Zs >= Ze)
            break;
          __syncthreads();
          stage(W, a, 0, 0);
          staged();
          if (dconv)
            scale(W, 0);
          __syncthreads();
          W.rofs = W.pofs = 0;
        }
        const double c = g.cosA[a], s = g.sinA[a];
        const double p1x = g.p1x[a], p1y = g.p1y[a];
        // ---- the column's candidate rays; the exact tests below decide
        int hA = 0, cnt = 0, rays = 0;
        float hin = INFINITY; // candidates up to here are in the reference's range
        if (has) {
          float hl, hh, tl, th;
          project_square(float(c * x0 + s * y0 - g.src[0]), float(c * y0 - s * x0 - g.src[1]),
                         float(c), float(s), bx, by, hscale, hofs, hl, hh, tl, th);
          int hB;
          if (g.even_cols && tl > 1e-3f * clf) {
            hin = hh - hround;
            hA = int(fminf(fmaxf(ceilf(hl - hmargin), 0.0f), float(g.nh)));
            hB = int(fmaxf(fminf(floorf(hh + hmargin), float(g.nh - 1)), -1.0f));
          } else {
            // uneven columns, or beside the source
            cb_column_hrange(g, a, x0, xn, y0, yn, hA, hB);
          }
          cnt = max(hB - hA + 1, 0);
        }
        const int slots = __reduce_max_sync(0xffffffffu, cnt);
        double2 next = g.inv[i64(a) * g.nh + min(hA, g.nh - 1)];
        for (int n = 0; n < slots; n++) {
          const int h = min(hA + n, g.nh - 1);
          // entry and exit alphas (bproject_ah, c2D.cpp:896-936)
          const double2 inv = next;
          next = g.inv[i64(a) * g.nh + min(h + 1, g.nh - 1)];
          float a0 = 0.0f, a1 = 0.0f;
          bool ok = n < cnt && inv.x != 0.0;
          if (ok) {
            const double ax0 = (x0 - p1x) * inv.x, ay0 = (y0 - p1y) * inv.y;
            const double axn = (xn - p1x) * inv.x, ayn = (yn - p1y) * inv.y;
            const double amin = cb_dmax(cb_dmax(cb_dmin(ax0, axn), cb_dmin(ay0, ayn)), 0.0);
            const double amax = cb_dmin(cb_dmin(cb_dmax(ax0, axn), cb_dmax(ay0, ayn)), 1.0);
            ok = amin < amax - eps;
            a0 = float(amin);
            a1 = float(amax);
            if (ok && (float(h) > hin || fmax(fabs(inv.x), fabs(inv.y)) * g.cl > 1e6)) {
              // at the range's end, or nearly parallel to an axis, where
              // rounding may pass a ray that misses the column
              int hmin, hmax;
              cb_column_hrange(g, a, x0, xn, y0, yn, hmin, hmax);
              ok = h >= hmin && h <= hmax;
            }
            if (ok && ++rays > kMaxRaysPerAngle) {
              ok = false;
              atomicExch(err, 2);
            }
          }
          if (!__any_sync(0xffffffffu, ok))
            continue;
#define CB_ROWS(M)                                                                         \
  ray_rows<M>(g, W, fits, a, h, a0, a1, ok, band.x, band.y, Z0, Zs, Ze, whole, acc, ztab,    \
              tab, patch, pix, dconv)
          if (pass == 0) {
            if (Zs <= kb)
              CB_ROWS(LOWER);
            if (Ze > kb)
              CB_ROWS(UPPER);
          } else {
            CB_ROWS(EDGE_LO);
            CB_ROWS(EDGE_UP);
          }
#undef CB_ROWS
        }
      }
      __syncthreads(); // before the next patches
    }
  }

  // ---- store: lanes over the slices of one column after the other
  double ssq = 0.0;
  for (int q = 0; q < 32; q++) {
    const int cq = __shfl_sync(0xffffffffu, col, q);
    if (cq < 0)
      continue;
    const i64 base = i64(cq) * g.nz;
    for (int K = Z0 + lane; K < Z1; K += 32) {
      const float v = wacc[(K - Z0 + kGuardLo) * 32 + q];
      float o = v;
      if (EPI == EPI_NORM) {
        ssq += double(v) * double(v);
      } else if (EPI == EPI_SIRT) {
        const float w = __fadd_rn(e.x[base + K], __fmul_rn(1.0f, __fmul_rn(v, e.w[base + K])));
        o = (w < 0.0f) ? 0.0f : w;
      } else if (EPI == EPI_MLEM) {
        const float w = __fmul_rn(e.x[base + K], __fmul_rn(e.w[base + K], v));
        o = (w < 0.0f) ? 0.0f : w;
      }
      vol[base + K] = o;
    }
  }
  if (EPI == EPI_NORM) {
    __shared__ double red[kMaxWarps];
    for (int o = 16; o > 0; o >>= 1)
      ssq += __shfl_down_sync(0xffffffffu, ssq, o);
    if (lane == 0)
      red[wib] = ssq;
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0;
      for (int w = 0; w < nw; w++)
        sum += red[w];
      e.partials[blockIdx.x] = sum;
    }
  }
}

__global__ void cb_ray_spans_kernel(Geom g, double2 *inv) {
  const i64 n = i64(g.na) * g.nh;
  for (i64 r = blockIdx.x * i64(blockDim.x) + threadIdx.x; r < n; r += i64(gridDim.x) * blockDim.x) {
    const int a = int(r / g.nh), h = int(r - i64(a) * g.nh);
    const double ddx = (g.cdx[a] - g.sinA[a] * g.hpix[h]) - g.p1x[a];
    const double ddy = (g.sdx[a] + g.cosA[a] * g.hpix[h]) - g.p1y[a];
    const bool none = fabs(ddx) < double(kEps) || fabs(ddy) < double(kEps);
    inv[r] = none ? make_double2(0.0, 0.0) : make_double2(1.0 / ddx, 1.0 / ddy);
  }
}

// ---- few columns: one CTA per column
//
// Too few columns to give every SM a tile of them: one CTA owns one column
// and each thread up to four of its voxels and rows.  Rays are staged per angle chunk.  For a
// stage of ST rays each thread loads its band rows (RMAX per ray, all loads in
// flight together), forms every row's two contributions and records, for
// every slice K, the first band row whose index reaches K (k is monotone in
// the row).  Each voxel thread then adds, per ray, exactly the contributions
// that go to its voxel, in the reference's order.
constexpr int kGaChunk = 64;
constexpr int kGaRays = kMaxRaysPerAngle; // slots per angle
constexpr int kGaStage = 3;    // rays per stage when the kernel multiplies by d_conv itself
constexpr int kGaStagePre = 4; // rays per stage on a sinogram already scaled by d_conv

__host__ __device__ inline int round4(int n) { return (n + 3) & ~3; }

// Shared-memory layout of cb_bp_column (offsets in 4-byte words) for
// `st` rays per stage.
struct GaLayout {
  int vz, dz, iz, seg_h, seg_a0, seg_a1, cnt, off, map, fr, prow, drow, total;
  __host__ __device__ GaLayout(int nz, int nv, int st) {
    vz = 0;
    dz = vz + cb_vz_floats(nz);
    iz = dz + round4(nv);
    seg_h = iz + round4(nv);
    seg_a0 = seg_h + kGaChunk * kGaRays;
    seg_a1 = seg_a0 + kGaChunk * kGaRays;
    cnt = seg_a1 + kGaChunk * kGaRays;
    off = cnt + round4(kGaChunk + 1);
    map = off + round4(kGaChunk + 1);
    fr = map + kGaChunk * kGaRays;
    prow = fr + st * round4(nz + 2);
    drow = prow + st * round4(nv);
    total = drow + st * round4(nv);
  }
};

// Stage the rays of angles [ac, ac + nac) in list order: slots per angle,
// then a prefix over angles and a flat map.  Returns the ray count.  Each
// slot holds the ray's detector column h and its entry and exit alphas.
__device__ int cb_ga_stage_rays(const Geom &g, int ac, int nac, double x0, double xn, double y0,
                                double yn, int *seg_h, float *seg_a0, float *seg_a1, int *cnt,
                                int *off, int *map, int *ovf) {
  const int tid = threadIdx.x;
  if (tid < nac) {
    int c = 0;
    cb_column_rays(g, ac + tid, x0, xn, y0, yn, [&](int h, float a0, float a1) {
      if (c < kGaRays) {
        const int idx = tid * kGaRays + c;
        seg_h[idx] = h;
        seg_a0[idx] = a0;
        seg_a1[idx] = a1;
      }
      c++;
    });
    if (c > kGaRays) {
      *ovf = 1;
      c = kGaRays;
    }
    cnt[tid] = c;
  }
  __syncthreads();
  if (tid == 0) {
    int acc = 0;
    for (int t = 0; t < nac; t++) {
      off[t] = acc;
      acc += cnt[t];
    }
    off[nac] = acc;
  }
  __syncthreads();
  if (tid < nac)
    for (int c = 0; c < cnt[tid]; c++)
      map[off[tid] + c] = tid * kGaRays + c;
  __syncthreads();
  return off[nac];
}

// First-row table: row v of slice k follows row v - 1 of slice kp, so v is
// the first band row of the slices kp + 1 .. k (entries 0 .. nz + 1 kept).
__device__ __forceinline__ void cb_ga_mark(int *f, int kp, int k, int v, int nz) {
  if (k == kp + 1 && k >= 0 && k <= nz + 1) {
    f[k] = v; // the usual step: one slice per row change
    return;
  }
  for (int K = max(kp + 1, 0); K <= min(k, nz + 1); K++)
    f[K] = v;
}

// PRE: the sinogram is already scaled by d_conv (the reference's dpixels,
// c2D.cpp:1096-1117), so a staged row is one load and no multiply.  ST rays
// per stage.  T threads, each with NZT voxels and RMAX rows.  blockIdx.y: the
// sinogram of a batch.
template <int EPI, int T, int NZT, int RMAX, bool PRE, int ST>
__global__ void __launch_bounds__(T, NZT == 1 ? 1024 / T : NZT == 2 ? 3 : 2)
    cb_bp_column(Geom g, const float *__restrict__ pix0, float *__restrict__ vol0, Epi e,
                 int *err) {
  extern __shared__ unsigned char smem_raw[];
  int *W = reinterpret_cast<int *>(smem_raw);
  const int nz = g.nz, nv = g.nv, nzm1 = nz - 1, mid = g.mid;
  const GaLayout L(nz, nv, ST);
  float *svz = reinterpret_cast<float *>(W + L.vz);
  float *sdz = reinterpret_cast<float *>(W + L.dz);
  float *siz = reinterpret_cast<float *>(W + L.iz);
  int *seg_h = W + L.seg_h;
  float *seg_a0 = reinterpret_cast<float *>(W + L.seg_a0);
  float *seg_a1 = reinterpret_cast<float *>(W + L.seg_a1);
  int *cnt = W + L.cnt, *off = W + L.off, *map = W + L.map, *fr = W + L.fr;
  float *prow = reinterpret_cast<float *>(W + L.prow); // staged pixel rows
  float *drow = reinterpret_cast<float *>(W + L.drow); // their d_conv rows
  const int frs = round4(nz + 2), prs = round4(nv);
  __shared__ int s_minv, s_maxv, s_ovf;
  __shared__ int s_kf[ST], s_kl[ST]; // slices of a staged ray's first/last band row
  // the column's square; kept in shared memory so that its FP64 corners
  // hold no registers through the row and voxel phases
  __shared__ double s_box[4];
  const int tid = threadIdx.x;
  const int col = int(blockIdx.x);
  const int i = col / g.ny, j = col - (col / g.ny) * g.ny;
  for (int t = tid; t <= nz; t += blockDim.x)
    svz[t] = g.vz[t];
  for (int t = tid; t < nv; t += blockDim.x) {
    sdz[t] = g.dz[t];
    siz[t] = g.iz[t];
  }
  if (tid == 0) {
    // band limits over every ray of the column (c2D.cpp:657-676), from
    // the plan's table
    const int2 b = g.colband[col];
    s_minv = b.x;
    s_maxv = b.y;
    s_ovf = 0;
    s_box[0] = g.origin[0] + double(i) * g.size[0];
    s_box[1] = g.origin[0] + double(i + 1) * g.size[0];
    s_box[2] = g.origin[1] + double(j) * g.size[1];
    s_box[3] = g.origin[1] + double(j + 1) * g.size[1];
  }
  __syncthreads();
  const int min_v = s_minv, max_v = s_maxv;
  const int nb = max_v - min_v;
  const int lo_end = min(mid, max_v);         // lower band rows [min_v, lo_end)
  const int up_begin = max(mid, min_v);       // upper band rows [up_begin, max_v)
  const float pzbz = g.pzbz, pzbz1 = g.pzbz1, inv_dz = g.inv_dz;
  // this thread's band rows v = min_v + tid + r * 256 are the same for every
  // ray: their z tables stay in registers (sd: delta_z of v, sp: of v - 1,
  // si: inv_delz of v)
  float rsd[RMAX], rsp[RMAX], rsi[RMAX];
#pragma unroll
  for (int r = 0; r < RMAX; r++) {
    const int v = min_v + tid + r * T;
    const bool in = v < max_v;
    rsd[r] = in ? sdz[v] : 0.0f;
    rsp[r] = (in && v > min_v) ? sdz[v - 1] : 0.0f;
    rsi[r] = in ? siz[v] : 0.0f;
  }
  const float sd_first = nb > 0 ? sdz[min_v] : 0.0f, sd_last = nb > 0 ? sdz[max_v - 1] : 0.0f;
  double ssq = 0.0;
  const float *__restrict__ pix = pix0 + i64(blockIdx.y) * g.na * g.nh * nv;
  float *__restrict__ vol = vol0 + i64(blockIdx.y) * g.nx * g.ny * nz;
  float acc[NZT]; // this thread's voxels tid + z * T
#pragma unroll
  for (int z = 0; z < NZT; z++)
    acc[z] = 0.0f;

  // ---- band rows of every ray (c2D.cpp:680-713)
  for (int ac = 0; nb > 0 && ac < g.na; ac += kGaChunk) {
    const int nac = min(kGaChunk, g.na - ac);
    const int nseg = cb_ga_stage_rays(g, ac, nac, s_box[0], s_box[1], s_box[2], s_box[3], seg_h,
                                      seg_a0, seg_a1, cnt, off, map, &s_ovf);
    for (int s0 = 0; s0 < nseg; s0 += ST) {
      const int ns = min(ST, nseg - s0);
      // 1) this thread's band rows v = min_v + tid + r * 256 of every staged
      //    ray: pixel values (times d_conv unless pre-scaled), all loads
      //    issued together
      float pv[ST][RMAX], dv[PRE ? 1 : ST][RMAX];
#pragma unroll
      for (int s = 0; s < ST; s++) {
        const int m = map[s0 + (s < ns ? s : 0)];
        const int h = seg_h[m];
        const float *prw = pix + (i64(ac + m / kGaRays) * g.nh + h) * nv;
#pragma unroll
        for (int r = 0; r < RMAX; r++) {
          const int v = min_v + tid + r * T;
          const bool ok = s < ns && v < max_v;
          pv[s][r] = ok ? __ldg(prw + v) : 0.0f;
        }
        if (!PRE) {
          const float *drw = g.dconv + i64(h) * nv;
#pragma unroll
          for (int r = 0; r < RMAX; r++) {
            const int v = min_v + tid + r * T;
            dv[PRE ? 0 : s][r] = (s < ns && v < max_v) ? __ldg(drw + v) : 0.0f;
          }
        }
      }
      // 2) per ray: the first band row of every slice index (the whole
      //    table: below the first row's slice min_v, above the last row's
      //    max_v) and each row's two contributions as the reference forms
      //    them (c2D.cpp:694-711): c1 = p (mz - a0) goes to slice k, c2 =
      //    p (a1 - mz) to k - 1 below the source row, to k + 1 from it on
#pragma unroll
      for (int s = 0; s < ST; s++) {
        if (s >= ns)
          break;
        const int m = map[s0 + s];
        const float a0 = seg_a0[m], a1 = seg_a1[m];
        const float av = __fmul_rn(a0, inv_dz);
        int *f = fr + s * frs;
        const int kf = int(__fadd_rn(pzbz, __fmul_rn(av, sd_first)));
        const int kl = int(__fadd_rn(pzbz, __fmul_rn(av, sd_last)));
        // only voxels kf - 1 .. kl + 1 receive rows of this ray, and they
        // read entries kf - 2 .. kl + 3: the band rows' transitions write
        // (kf, kl], six threads write the ends
        if (tid < 6) {
          const int K = tid < 3 ? kf - tid : kl + tid - 2;
          if (K >= 0 && K <= nz + 1)
            f[K] = tid < 3 ? min_v : max_v;
        }
        if (tid == 0) {
          s_kf[s] = kf;
          s_kl[s] = kl;
        }
        float *c1 = prow + s * prs, *c2 = drow + s * prs;
        const float2 av2 = make_float2(av, av), a02 = make_float2(a0, a0),
                     a12 = make_float2(a1, a1);
#pragma unroll
        for (int r = 0; r < RMAX; r++) {
          if (r + 1 < RMAX && (r & 1) == 0) {
            // rows r and r + 1 as packed pairs: the same unfused float
            // operations per row, two rows per multiply and subtract
            const int v0 = min_v + tid + r * T, v1 = v0 + T;
            const float2 kk = mul2_rn(av2, make_float2(rsd[r], rsd[r + 1]));
            const float2 kq = mul2_rn(av2, make_float2(rsp[r], rsp[r + 1]));
            const int k0 = int(__fadd_rn(pzbz, kk.x)), k1 = int(__fadd_rn(pzbz, kk.y));
            if (v0 < max_v && v0 > min_v)
              cb_ga_mark(f, int(__fadd_rn(pzbz, kq.x)), k0, v0, nz);
            if (v1 < max_v)
              cb_ga_mark(f, int(__fadd_rn(pzbz, kq.y)), k1, v1, nz);
            const int kz0 = min(max(v0 < mid ? k0 : k0 + 1, 0), nz);
            const int kz1 = min(max(v1 < mid ? k1 : k1 + 1, 0), nz);
            const float2 pl =
                mul2_rn(make_float2(svz[kz0], svz[kz1]), make_float2(rsi[r], rsi[r + 1]));
            const float2 mz = make_float2(fmin_ref(pl.x, a1), fmin_ref(pl.y, a1));
            const float2 p = PRE ? make_float2(pv[s][r], pv[s][r + 1])
                                 : mul2_rn(make_float2(pv[s][r], pv[s][r + 1]),
                                           make_float2(dv[PRE ? 0 : s][r], dv[PRE ? 0 : s][r + 1]));
            const float2 w1 = mul2_rn(p, sub2_rn(mz, a02)), w2 = mul2_rn(p, sub2_rn(a12, mz));
            if (v0 < max_v) {
              c1[v0] = w1.x;
              c2[v0] = w2.x;
            }
            if (v1 < max_v) {
              c1[v1] = w1.y;
              c2[v1] = w2.y;
            }
            continue;
          }
          if (r & 1)
            continue; // done with its pair
          const int v = min_v + tid + r * T;
          if (v < max_v) {
            const int k = int(__fadd_rn(pzbz, __fmul_rn(av, rsd[r])));
            if (v > min_v)
              cb_ga_mark(f, int(__fadd_rn(pzbz, __fmul_rn(av, rsp[r]))), k, v, nz);
            const int kz = min(max(v < mid ? k : k + 1, 0), nz);
            const float mz = fmin_ref(__fmul_rn(svz[kz], rsi[r]), a1);
            const float p = PRE ? pv[s][r] : __fmul_rn(pv[s][r], dv[PRE ? 0 : s][r]);
            c1[v] = __fmul_rn(p, __fsub_rn(mz, a0));
            c2[v] = __fmul_rn(p, __fsub_rn(a1, mz));
          }
        }
      }
      __syncthreads();
      // 3) each voxel adds its rows' contributions in the reference's order
      for (int s = 0; s < ns; s++) {
        const int *f = fr + s * frs;
        const float *c1 = prow + s * prs, *c2 = drow + s * prs;
        const int klo = s_kf[s] - 1, khi = s_kl[s] + 1;
#pragma unroll
        for (int z = 0; z < NZT; z++) {
          const int K = tid + z * T;
          if (K >= nz || K < klo || K > khi)
            continue; // no row of this ray feeds voxel K
          const int fm = K >= 1 ? f[K - 1] : min_v, f0 = f[K], f1 = f[K + 1];
          float t = acc[z];
          // below the source row: rows of slice K give c1, then rows of
          // slice K + 1 give c2 (their neighbour k - 1 == K)
          for (int v = f0, ve = min(f[K + 2], lo_end); v < ve; v++)
            t = __fadd_rn(t, (v < f1 ? c1 : c2)[v]);
          // from the source row on: rows of slice K - 1 give c2 (their
          // neighbour k + 1 == K), then rows of slice K give c1
          for (int v = max(fm, up_begin), ve = min(f1, max_v); v < ve; v++)
            t = __fadd_rn(t, (v < f0 ? c2 : c1)[v]);
          acc[z] = t;
        }
      }
      __syncthreads();
    }
  }

  // ---- edge rows of every ray (c2D.cpp:715-750)
  if (min_v > 0 || max_v < nv) {
    for (int ac = 0; ac < g.na; ac += kGaChunk) {
      const int nac = min(kGaChunk, g.na - ac);
      const int nseg = cb_ga_stage_rays(g, ac, nac, s_box[0], s_box[1], s_box[2], s_box[3],
                                        seg_h, seg_a0, seg_a1, cnt, off, map, &s_ovf);
      for (int s = 0; s < nseg; s++) {
        const int m = map[s];
        const int h = seg_h[m];
        const float a0 = seg_a0[m], a1 = seg_a1[m];
        const float av = __fmul_rn(a0, inv_dz);
        const float *prw = pix + (i64(ac + m / kGaRays) * g.nh + h) * nv;
        const float *drw = g.dconv + i64(h) * nv;
#pragma unroll
        for (int z = 0; z < NZT; z++) {
          const int K = tid + z * T;
          if (K >= nz)
            continue;
          for (int v = min(min_v, nv) - 1; v >= 0; v--) {
            const int k = int(__fadd_rn(pzbz1, __fmul_rn(av, sdz[v]))) - 1;
            if (k < K)
              break; // k only falls as v falls (and k < 0 ends the reference's loop)
            if (k > K + 1)
              continue;
            const float p = PRE ? __ldg(prw + v) : __fmul_rn(__ldg(prw + v), __ldg(drw + v));
            if (k > 0) {
              const float mz = fmin_ref(__fmul_rn(svz[k], siz[v]), a1);
              acc[z] = __fadd_rn(acc[z], __fmul_rn(p, k == K ? __fsub_rn(mz, a0)
                                                             : __fsub_rn(a1, mz)));
            } else if (K == 0) {
              const float mz = fmin_ref(__fmul_rn(svz[0], siz[v]), a1);
              acc[z] = __fadd_rn(acc[z], __fmul_rn(p, __fsub_rn(mz, a0)));
            }
          }
          for (int v = max(max_v, 0); v < nv; v++) {
            const int k = int(__fadd_rn(pzbz, __fmul_rn(av, sdz[v])));
            if (k > K || k > nzm1)
              break; // k only rises with v (and k > nz - 1 ends the reference's loop)
            if (k < K - 1)
              continue;
            const float p = PRE ? __ldg(prw + v) : __fmul_rn(__ldg(prw + v), __ldg(drw + v));
            const float mz = fmin_ref(__fmul_rn(svz[k + 1], siz[v]), a1);
            if (k == K)
              acc[z] = __fadd_rn(acc[z], __fmul_rn(p, __fsub_rn(mz, a0)));
            else if (k < nzm1)
              acc[z] = __fadd_rn(acc[z], __fmul_rn(p, __fsub_rn(a1, mz)));
          }
        }
      }
      __syncthreads();
    }
  }
  const i64 base = i64(col) * nz;
#pragma unroll
  for (int z = 0; z < NZT; z++) {
    const int K = tid + z * T;
    if (K >= nz)
      break;
    const float v = acc[z];
    float o = v;
    if (EPI == EPI_NORM) {
      ssq += double(v) * double(v);
    } else if (EPI == EPI_SIRT) {
      const float t = __fadd_rn(e.x[base + K], __fmul_rn(1.0f, __fmul_rn(v, e.w[base + K])));
      o = (t < 0.0f) ? 0.0f : t;
    } else if (EPI == EPI_MLEM) {
      const float t = __fmul_rn(e.x[base + K], __fmul_rn(e.w[base + K], v));
      o = (t < 0.0f) ? 0.0f : t;
    }
    vol[base + K] = o;
  }
  if (tid == 0 && s_ovf)
    atomicExch(err, 2);
  if (EPI == EPI_NORM) {
    __shared__ double red[T / 32];
    const double t = cta_sum<T / 32>(ssq, red);
    if (threadIdx.x == 0)
      e.partials[blockIdx.x] = t;
  }
}

// Which kernel: a CTA per column costs its columns' rays and rows; the tiles'
// time is flat until there are columns enough for every SM.  Column / tile
// kernel, cubes with the 512^3 benchmark's proportions, 90 angles: 48^3 0.41 /
// 0.80 ms, 64^3 0.84 / 1.45, 80^3 1.70 / 2.16, 96^3 3.47 / 2.62; with two rays
// and two rows per voxel the tiles win from 64^3 (0.55 / 0.41 ms, 24 angles).
// On few columns the tiles lose at any height and row count: 32^2 x 512 from
// 768 rows 388 / 457 us, x 64 from 520 600 / 1190, 40^2 x 512 from 256 355 /
// 364, but 40^2 x 900 from 450 586 / 489.
bool small_volume(const Geom &g) {
  const i64 columns = i64(g.nx) * g.ny, voxels = columns * g.nz;
  return g.nz <= 1024 && g.nv <= 1024 &&
         ((voxels <= (1 << 19) && g.nz <= 256 && g.nv <= 512) ||
          (columns <= 1600 && voxels <= (1 << 20)));
}

size_t small_smem(const Geom &g) {
  return size_t(GaLayout(g.nz, g.nv, std::max(kGaStage, kGaStagePre)).total) * 4;
}

// Chunk height; warps per CTA.  Tall chunks spend less on ray set-up and
// on rows that straddle two chunks; small problems need short chunks to reach
// every SM.  Eight warps share a patch; CTAs of two or four reach more SMs but
// copy more, so that they pay only with 32 slices (128^3 / 180 angles 7.2 ms with
// four, 7.9 with eight) or where a voxel sees so many rays that few angles'
// patches fit (64^2 x 256 with 25 rays per voxel 3.5 / 4.1 ms; with 6 rays 1.30
// / 1.17; 8 slices, 96^3: 1.82 / 1.32).  32 slices, 8 warps and 17,000 patch floats
// make two CTAs per SM (36 KB of accumulators, 4 KB of row tables and 66 KB
// of patch each); 512^3: 625 ms, 660 ms with 24 slices, 831 ms with 16 slices
// and three CTAs, 676 ms with one CTA of 16 warps.
TileShape tile_shape(const Geom &g) {
  TileShape t;
  const i64 warps = i64((g.nx + kTileX - 1) / kTileX) * ((g.ny + kTileY - 1) / kTileY);
  t.zc = 32;
  while (t.zc > 8 && warps * ((g.nz + t.zc - 1) / t.zc) < i64(148) * 12)
    t.zc /= 2;
  t.nzc = (g.nz + t.zc - 1) / t.zc;
  t.wx = 2;
  t.wy = 4;
  // detector columns and rows per voxel on the axis
  const double mag = std::abs(g.cl / g.src[0]);
  const bool dense = g.size[0] * mag * g.cipix * g.size[2] * mag * g.inv_pitch > 20.0;
  while ((t.zc == 32 || (t.zc == 16 && dense)) && t.wy > 1 &&
         warps * t.nzc < i64(296) * t.wx * t.wy)
    t.wy /= 2;
  t.rcap = 512;
  t.cap = 17000;
  t.ntx = (g.nx + t.wx * kTileX - 1) / (t.wx * kTileX);
  t.nty = (g.ny + t.wy * kTileY - 1) / (t.wy * kTileY);
  return t;
}

// The column kernel's instance for a plan's slices and rows; its threads.
typedef void (*ColumnKernel)(Geom, const float *, float *, Epi, int *);
int column_threads(const Geom &g) { return g.nz <= 128 && g.nv <= 256 ? 128 : 256; }
template <int EPI, bool PRE> ColumnKernel column_kernel(const Geom &g) {
  constexpr int ST = PRE ? kGaStagePre : kGaStage;
#define CB_COLUMN_ROWS(Z)                                                                  \
  (g.nv <= 256   ? cb_bp_column<EPI, 256, Z, 1, PRE, ST>                                    \
   : g.nv <= 512 ? cb_bp_column<EPI, 256, Z, 2, PRE, ST>                                    \
   : g.nv <= 768 ? cb_bp_column<EPI, 256, Z, 3, PRE, ST>                                    \
                 : cb_bp_column<EPI, 256, Z, 4, PRE, ST>)
  if (column_threads(g) == 128)
    return g.nv <= 128 ? cb_bp_column<EPI, 128, 1, 1, PRE, ST>
                       : cb_bp_column<EPI, 128, 1, 2, PRE, ST>;
  return g.nz <= 256 ? CB_COLUMN_ROWS(1) : g.nz <= 512 ? CB_COLUMN_ROWS(2) : CB_COLUMN_ROWS(4);
#undef CB_COLUMN_ROWS
}

template <int EPI>
void launch_bp(const Geom &g, const float *pix, float *vol, const Epi &e, int *err,
               cudaStream_t st, int nbatch) {
  const i64 nin = i64(g.na) * g.nh * g.nv, nout = i64(g.nx) * g.ny * g.nz;
  const TileShape t = tile_shape(g);
  for (int b = 0; b < nbatch; b += 65535) {
    const unsigned ny = std::min(nbatch - b, 65535);
    if (small_volume(g))
      (e.pre ? column_kernel<EPI, true>(g) : column_kernel<EPI, false>(g))
          <<<dim3(g.nx * g.ny, ny), column_threads(g), small_smem(g), st>>>(
              g, pix + b * nin, vol + b * nout, e, err);
    else
      cb_bp_tile<EPI><<<dim3(t.ntx * t.nty * t.nzc, ny), t.wx * t.wy * 32, tile_smem(t), st>>>(
          g, pix + b * nin, vol + b * nout, e, err, t);
  }
}

// out[a][h][v] = in[a][h][v] * d_conv[h][v]: the reference's dpixels
// (c2D.cpp:1096-1117), the same float products the back projector would
// form row by row.
__global__ void cb_prescale_kernel(const float *__restrict__ in, float *__restrict__ out,
                                   const float *__restrict__ dconv, i64 per_angle, i64 n) {
  for (i64 i = blockIdx.x * i64(blockDim.x) + threadIdx.x; i < n;
       i += i64(gridDim.x) * blockDim.x)
    out[i] = __fmul_rn(in[i], dconv[i % per_angle]);
}

} // namespace

int cb_bp_parts(const Geom &g) {
  const TileShape t = tile_shape(g);
  return small_volume(g) ? g.nx * g.ny : t.ntx * t.nty * t.nzc;
}

int cb_bp_prepare(const Geom &g) {
  // the limit is the function's, not the plan's: the largest any plan uses
  bool ok = true;
  auto allow = [&](const void *f) {
    ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    220 * 1024) == cudaSuccess;
  };
#define CB_BP_ALLOW(E)                                                                     \
  if (small_volume(g)) {                                                                    \
    allow((const void *)column_kernel<E, false>(g));                                        \
    allow((const void *)column_kernel<E, true>(g));                                         \
  } else                                                                                    \
    allow((const void *)cb_bp_tile<E>);
  CB_BP_ALLOW(EPI_STORE)
  CB_BP_ALLOW(EPI_NORM)
  CB_BP_ALLOW(EPI_SIRT)
  CB_BP_ALLOW(EPI_MLEM)
#undef CB_BP_ALLOW
  return ok ? 0 : 1;
}

int cb_ray_spans(const Geom &g, double2 *inv, cudaStream_t st) {
  const i64 n = i64(g.na) * g.nh;
  cb_ray_spans_kernel<<<int(std::min<i64>((n + 255) / 256, i64(sm_count()) * 8)), 256, 0, st>>>(
      g, inv);
  return cudaPeekAtLastError() == cudaSuccess ? 0 : 2;
}

void cb_prescale(const Geom &g, const float *in, float *out, cudaStream_t st) {
  const i64 per = i64(g.nh) * g.nv, n = i64(g.na) * per;
  const i64 blocks = std::min<i64>((n + 255) / 256, i64(sm_count()) * 8);
  cb_prescale_kernel<<<int(std::max<i64>(blocks, 1)), 256, 0, st>>>(in, out, g.dconv, per, n);
}

int cb_backward(const Geom &g, const float *pix, float *vol, int mode, const Epi &e,
                int *err, cudaStream_t st, int nbatch) {
  switch (mode) {
  case EPI_STORE:
    launch_bp<EPI_STORE>(g, pix, vol, e, err, st, nbatch);
    break;
  case EPI_NORM:
    launch_bp<EPI_NORM>(g, pix, vol, e, err, st, nbatch);
    break;
  case EPI_SIRT:
    launch_bp<EPI_SIRT>(g, pix, vol, e, err, st, nbatch);
    break;
  case EPI_MLEM:
    launch_bp<EPI_MLEM>(g, pix, vol, e, err, st, nbatch);
    break;
  default:
    return 1;
  }
  return 0;
}

} // namespace ccpi
