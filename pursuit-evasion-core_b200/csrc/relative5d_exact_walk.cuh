// Exact relative 5D stage arithmetic for a thread that owns 4 consecutive x
// cells and walks the headings: the operations of relative5d_exact.cuh's
// cell_update (native_relative.cpp:38-67, :124-172) with every quotient and
// every ENO selection computed once per edge or node instead of once per
// cell that uses it.  Shared by the single-grid kernel
// (relative5d_tiled_exact.cu) and the batched one
// (relative5d_batch_tiled_exact.cu); both are compiled with -fmad=false.
//
// Why the results keep the bits of cell_update:
//   * with c2(j) = ((s[j+1] - 2 s[j]) + s[j-1]) / h^2, the reference's l2 of
//     node j is c2(j-1) and its r2 is c2(j+1), operation for operation, so
//     the selection of edge (j, j+1) -- "fabs(c2(j)) < fabs(c2(j+1)) ? c2(j)
//     : c2(j+1)" -- is both the high side of j and the low side of j+1, and
//     the missing outer node next to an end is c2 of the inner one;
//   * -2 s[j] is exact, so fma(-2, s[j], s[j+1]) rounds like the difference;
//   * a quotient by a spacing is RN(1/h) times the dividend with one FMA
//     correction (div_rn.cuh's method).  Differences of float32 values are
//     zero or at least 2^-149, so nothing underflows; the sign of a zero
//     quotient may differ from the division's, which no result depends on
//     (H enters as H < 0 ? H : 0);
//   * a dividend that is infinite or NaN gives a NaN quotient here.  Where the
//     reference's quotient would be infinite and matter, the NaN reaches H:
//     such a cell (and any cell whose update is not finite) is recomputed by
//     cell_update itself.  An infinite value that the ENO selection discards
//     is discarded here too, since a comparison with NaN is false and the
//     selection then takes its second operand, as it does for an infinite
//     first one; a NaN second operand reaches H.
#pragma once
#include <cfloat>

#include "relative5d_exact.cuh"

namespace pe {
namespace exact {

// One axis' spacing: h, h*h, .5*h and the reciprocals (rounded to nearest).
struct AxisStep {
  double h, rh, hh, rhh, half;
};

inline __host__ __device__ AxisStep axis_step(double h, double rh, double rhh) {
  return AxisStep{h, rh, h * h, rhh, .5 * h};
}

__device__ __forceinline__ double quot(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}
__device__ __forceinline__ double quot1(double a, const AxisStep &s) {
  return quot(a, s.h, s.rh);
}
__device__ __forceinline__ double quot2(double p, double v, double m, const AxisStep &s) {
  return quot(fma(-2.0, v, p) + m, s.hh, s.rhh);
}
// half a spacing times the smaller second difference, ties to the second
__device__ __forceinline__ double edge_term(double a, double b, const AxisStep &s) {
  double r;  // written out so that no integer sign masking is generated
  asm("{\n .reg .pred p;\n .reg .f64 ua, ub;\n abs.f64 ua, %1;\n abs.f64 ub, %2;\n"
      " setp.lt.f64 p, ua, ub;\n selp.f64 %0, %1, %2, p;\n}"
      : "=d"(r)
      : "d"(a), "d"(b));
  return s.half * r;
}

__device__ __forceinline__ float f4_get(const float4 &v, int i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

// Slopes of one cell along y or a speed axis from its five values; GENERAL
// applies the end rules (pos uniform or per lane).
template <int ORDER, bool GENERAL>
__device__ __forceinline__ Slopes axis_slopes(float m2, float m1, double v, float p1, float p2,
                                              int pos, int n, const AxisStep &s) {
  const double vm = m1, vp = p1;
  const double dl = quot1(v - vm, s), dh = quot1(vp - v, s);
  Slopes r{dl, dh};
  if (ORDER == 2) {
    const double c2 = quot2(vp, v, vm, s);
    double l2 = quot2(v, vm, (double)m2, s), r2 = quot2((double)p2, vp, v, s);
    if (GENERAL) {
      if (pos < 2) l2 = c2;
      if (pos + 2 >= n) r2 = c2;
    }
    r.lo = dl + edge_term(l2, c2, s);
    r.hi = dh - edge_term(c2, r2, s);
  }
  if (GENERAL) {
    if (pos == 0) r.lo = r.hi = dh;
    if (pos == n - 1) r.lo = r.hi = dl;
  }
  return r;
}

// Heading differences carried from one heading to the next: LO = low slope
// of heading k, D = quotient of edge (k, k+1), C2 = second quotient at k.
template <int ORDER>
struct HeadingCarry {
  double LO[4], D[4], C2[4];

  __device__ __forceinline__ void start(const float4 &m2, const float4 &m1, const float4 &v0,
                                        const float4 &p1, const AxisStep &s) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const double vm = f4_get(m1, i), v = f4_get(v0, i), vp = f4_get(p1, i);
      const double dl = quot1(v - vm, s);
      D[i] = quot1(vp - v, s);
      LO[i] = dl;
      C2[i] = 0;
      if (ORDER == 2) {
        C2[i] = quot2(vp, v, vm, s);
        LO[i] = dl + edge_term(quot2(v, vm, (double)f4_get(m2, i), s), C2[i], s);
      }
    }
  }

  // Slopes of heading k of cell i from V(k), V(k+1), V(k+2); moves on to k+1.
  __device__ __forceinline__ Slopes next(int i, double v, float vn, float vnew,
                                         const AxisStep &s) {
    Slopes r;
    const double a = vn, b = vnew;
    r.lo = LO[i];
    if (ORDER == 2) {
      const double c2n = quot2(b, a, v, s);
      const double e = edge_term(C2[i], c2n, s);
      r.hi = D[i] - e;
      LO[i] = D[i] + e;
      C2[i] = c2n;
    } else {
      r.hi = D[i];
      LO[i] = D[i];
    }
    D[i] = quot1(b - a, s);
    return r;
  }
};

// Constants of an item (uniform over its threads; may lie in shared memory).
struct ItemCoef {
  double vp, ve, wp, we, acc_p, acc_e, dt;
  int iv, nvp, ie, nve, nx;
  bool v_general, e_general;

  __device__ __forceinline__ void set(const Rel5Grid &g, int iv_, int ie_, double dt_) {
    iv = iv_;
    nvp = g.nvp;
    ie = ie_;
    nve = g.nve;
    nx = g.nx;
    v_general = iv < 2 || iv + 2 >= g.nvp;
    e_general = ie < 2 || ie + 2 >= g.nve;
    vp = g.vp_lo + iv * g.dvp;
    ve = g.ve_lo + ie * g.dve;
    wp = fabs(vp) * g.curv_p;
    we = fabs(ve) * g.curv_e;
    acc_p = g.acc_p;
    acc_e = g.acc_e;
    dt = dt_;
  }
};

// A thread's row: its y, and whether its warp takes the general y rules.
struct RowCoef {
  double y;
  int iy;
  bool general;
};

struct AxisSteps {
  AxisStep x, psi, v, e;
};

// The 4 cells' Hamiltonian plus dissipation at heading k.  w: the row window
// x0-2 .. x0+5 (C the cells); ycol the chunk's column in the own rows (rows
// iy-2 .. iy+2 ystride apart), nb in the speed-neighbour rows (vE-2, -1, +1, +2,
// vP-2 .. nbstride apart); VN, VNEW headings k+1, k+2.  XR = nx mod 4 places the
// x end rules at compile time, `kend` and `iend` saying whether nodes nx-2 and
// nx-1 lie in this chunk; XR = -1 takes their cells from `kcell` and `icell`
// (outside 0..3 where the chunk does not hold them).
template <int ORDER, int XR>
__device__ __forceinline__ void walk_hamiltonian(
    const float2 &xl, const float4 &C, const float2 &xr, const float4 &VN, const float4 &VNEW,
    const float *ycol, int ystride, const float *nb, int nbstride, bool first, bool kend,
    bool iend, int kcell, int icell, const double *xs, double cs, double sn, const ItemCoef &q,
    const RowCoef &row, const AxisSteps &st,
    HeadingCarry<ORDER> &carry, double H[4]) {
  const double bx = q.ve * cs - q.vp, by = q.ve * sn;
  double gx[4], gy[4], diss[4];
  {
    const double w[8] = {xl.x, xl.y, C.x, C.y, C.z, C.w, xr.x, xr.y};
    double D[5], E[5];
#pragma unroll
    for (int i = 0; i < 5; i++) D[i] = quot1(w[i + 2] - w[i + 1], st.x);
    if (ORDER == 2) {
      double c2[6];
#pragma unroll
      for (int i = 0; i < 6; i++) c2[i] = quot2(w[i + 2], w[i + 1], w[i], st.x);
      c2[1] = first ? c2[2] : c2[1];
#pragma unroll
      for (int i = 3; i >= 0; i--)
        if (XR < 0 || i == ((XR + 2) & 3)) c2[i + 2] = (XR < 0 ? kcell == i : kend) ? c2[i + 1] : c2[i + 2];
#pragma unroll
      for (int i = 0; i < 5; i++) E[i] = edge_term(c2[i], c2[i + 1], st.x);
    }
    const double ax = fabs(bx) + q.wp * fabs(row.y);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      double lo = ORDER == 2 ? D[i] + E[i] : D[i];
      double hi = ORDER == 2 ? D[i + 1] - E[i + 1] : D[i + 1];
      if (i == 0) {
        lo = first ? D[1] : lo;
        hi = first ? D[1] : hi;
      }
      if (XR < 0 || i == ((XR + 3) & 3)) {
        const bool at_end = XR < 0 ? icell == i : iend;
        lo = at_end ? D[i] : lo;
        hi = at_end ? D[i] : hi;
      }
      gx[i] = .5 * (lo + hi);
      diss[i] = ax * (hi - lo);
    }
  }
  const double aby = fabs(by);
  {
    const float4 m2 = *reinterpret_cast<const float4 *>(ycol - 2 * ystride);
    const float4 m1 = *reinterpret_cast<const float4 *>(ycol - ystride);
    const float4 p1 = *reinterpret_cast<const float4 *>(ycol + ystride);
    const float4 p2 = *reinterpret_cast<const float4 *>(ycol + 2 * ystride);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const double v = f4_get(C, i);
      const Slopes s =
          row.general ? axis_slopes<ORDER, true>(f4_get(m2, i), f4_get(m1, i), v, f4_get(p1, i),
                                                 f4_get(p2, i), row.iy, q.nx, st.x)
                      : axis_slopes<ORDER, false>(f4_get(m2, i), f4_get(m1, i), v,
                                                  f4_get(p1, i), f4_get(p2, i), row.iy, q.nx, st.x);
      gy[i] = .5 * (s.lo + s.hi);
      diss[i] = diss[i] + (aby + q.wp * fabs(xs[i])) * (s.hi - s.lo);
    }
  }
  const double ap = q.wp + q.we;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const Slopes s = carry.next(i, (double)f4_get(C, i), f4_get(VN, i), f4_get(VNEW, i), st.psi);
    const double gp = .5 * (s.lo + s.hi);
    diss[i] = diss[i] + ap * (s.hi - s.lo);
    H[i] = bx * gx[i] + by * gy[i] - q.wp * fabs(row.y * gx[i] - xs[i] * gy[i] - gp) +
           q.we * fabs(gp);
  }
  double je[4];  // the evader axis' jump: its slopes come first in the dissipation's
                 // neighbour order but its terms are added last
  {
    const float4 m2 = *reinterpret_cast<const float4 *>(nb + 4 * nbstride);
    const float4 m1 = *reinterpret_cast<const float4 *>(nb + 5 * nbstride);
    const float4 p1 = *reinterpret_cast<const float4 *>(nb + 6 * nbstride);
    const float4 p2 = *reinterpret_cast<const float4 *>(nb + 7 * nbstride);
    if (!q.v_general) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const Slopes s =
            axis_slopes<ORDER, false>(f4_get(m2, i), f4_get(m1, i), (double)f4_get(C, i),
                                      f4_get(p1, i), f4_get(p2, i), q.iv, q.nvp, st.v);
        // inside the speed range min(-a g, a g) = -(a |g|)
        H[i] = H[i] - q.acc_p * fabs(.5 * (s.lo + s.hi));
        diss[i] = diss[i] + q.acc_p * (s.hi - s.lo);
      }
    } else {
      const double pl = q.iv == 0 ? 0 : -q.acc_p, ph = q.iv == q.nvp - 1 ? 0 : q.acc_p;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const Slopes s =
            axis_slopes<ORDER, true>(f4_get(m2, i), f4_get(m1, i), (double)f4_get(C, i),
                                     f4_get(p1, i), f4_get(p2, i), q.iv, q.nvp, st.v);
        const double gv = .5 * (s.lo + s.hi);
        const double a = pl * gv, b = ph * gv;
        H[i] = H[i] + (b < a ? b : a);
        diss[i] = diss[i] + q.acc_p * (s.hi - s.lo);
      }
    }
  }
  {
    const float4 m2 = *reinterpret_cast<const float4 *>(nb);
    const float4 m1 = *reinterpret_cast<const float4 *>(nb + nbstride);
    const float4 p1 = *reinterpret_cast<const float4 *>(nb + 2 * nbstride);
    const float4 p2 = *reinterpret_cast<const float4 *>(nb + 3 * nbstride);
    if (!q.e_general) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const Slopes s =
            axis_slopes<ORDER, false>(f4_get(m2, i), f4_get(m1, i), (double)f4_get(C, i),
                                      f4_get(p1, i), f4_get(p2, i), q.ie, q.nve, st.e);
        H[i] = H[i] + q.acc_e * fabs(.5 * (s.lo + s.hi));
        je[i] = s.hi - s.lo;
      }
    } else {
      const double el = q.ie == 0 ? 0 : -q.acc_e, eh = q.ie == q.nve - 1 ? 0 : q.acc_e;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const Slopes s =
            axis_slopes<ORDER, true>(f4_get(m2, i), f4_get(m1, i), (double)f4_get(C, i),
                                     f4_get(p1, i), f4_get(p2, i), q.ie, q.nve, st.e);
        const double ge = .5 * (s.lo + s.hi);
        const double a = el * ge, b = eh * ge;
        H[i] = H[i] + (a < b ? b : a);
        je[i] = s.hi - s.lo;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) H[i] = H[i] + .5 * (diss[i] + q.acc_e * je[i]);
}

// Largest |change| and increase of a thread's cells, in double.  A float
// screen (rounding is monotonic, so |change| can only exceed the maximum
// where the rounded |change| reaches its rounded value) keeps the double
// comparison off the common path.
struct ChangeMax {
  double abs_max = 0, up_max = 0;
  float screen = 1.4e-45f;

  __device__ __forceinline__ void add(const float prev[4], const float now[4]) {
    const float d0 = now[0] - prev[0], d1 = now[1] - prev[1];
    const float d2 = now[2] - prev[2], d3 = now[3] - prev[3];
    const float m = fmaxf(fmaxf(fabsf(d0), fabsf(d1)), fmaxf(fabsf(d2), fabsf(d3)));
    if (m >= screen) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const double c = (double)now[i] - (double)prev[i];
        abs_max = fmax(abs_max, fabs(c));
        up_max = fmax(up_max, c);
      }
      screen = m;
    } else if (fmaxf(fmaxf(d0, d1), fmaxf(d2, d3)) > 0.f) {
#pragma unroll
      for (int i = 0; i < 4; i++) up_max = fmax(up_max, (double)now[i] - (double)prev[i]);
    }
  }
};

// cell_update of one cell out of line: the cells whose fast evaluation met a
// value that is not finite.
template <int ORDER, int BLEND>
__device__ __noinline__ bool slow_cell(const Rel5Grid &g, const Rel5Stage &s, int ix, int iy,
                                       int ip, int iv, int ie, int64_t j, double *change_abs,
                                       double *change_up) {
  double ca = 0, cu = 0;
  bool bad = false;
  cell_update<ORDER, BLEND, float>(g, s, ix, iy, ip, iv, ie, j, ca, cu, bad);
  *change_abs = fmax(*change_abs, ca);
  *change_up = fmax(*change_up, cu);
  return bad;
}

// The update of the 4 cells from H: RK2 average, exit, first crossing,
// change and store.  `valid`: cells inside the row (the row padding after
// them is stored as 0).  Returns true when an update is not finite.
template <int ORDER, int BLEND>
__device__ __forceinline__ bool walk_update(const Rel5Grid &g, const Rel5Stage &s, int x0,
                                            int ip, int64_t j, int valid, const ItemCoef &q,
                                            const RowCoef &row, const double *xs, const float4 &C,
                                            const float4 &P, const double H[4],
                                            ChangeMax &change) {
  float now[4], prev[4];
  bool redo = false;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double old = f4_get(C, i);
    prev[i] = BLEND ? f4_get(P, i) : f4_get(C, i);
    double value = old + q.dt * (H[i] < 0. ? H[i] : 0.);
    if (BLEND) value = .5 * ((double)prev[i] + value);
    now[i] = (float)value;
    const bool ok = fabs(H[i]) <= DBL_MAX && fabsf(now[i]) <= FLT_MAX;
    redo |= !ok && i < valid;
  }
  if (s.exit_r2 > 0) {
    const double yy = row.y * row.y;
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (xs[i] * xs[i] + yy > s.exit_r2) now[i] = prev[i] = (float)s.exit_r;
  }
  bool bad = false;
  if (redo) {  // every cell of the chunk, in the general form
    double ca = change.abs_max, cu = change.up_max;  // (the members stay in registers)
    for (int i = 0; i < valid; i++)
      bad |= slow_cell<ORDER, BLEND>(g, s, x0 + i, row.iy, ip, q.iv, q.ie, j + i, &ca, &cu);
    change.abs_max = ca;
    change.up_max = cu;
    return bad;
  }
#pragma unroll
  for (int i = 1; i < 4; i++)  // row padding stays 0 (valid >= 1)
    if (i >= valid) now[i] = prev[i] = 0.f;
  if (BLEND || ORDER == 1) {
    change.add(prev, now);
    // first crossing of zero: prev > 0 >= now (an exit cell never arrives)
    bool crossed = false;
#pragma unroll
    for (int i = 0; i < 4; i++) crossed |= prev[i] > 0.f && now[i] <= 0.f;
    if (crossed) {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (prev[i] > 0.f && now[i] <= 0.f && isnan(s.arrival[j + i])) {
          const double pv = prev[i];
          s.arrival[j + i] = (float)(s.t + s.dt * pv / (pv - (double)now[i]));
        }
    }
  }
  *reinterpret_cast<float4 *>(s.dst + j) = make_float4(now[0], now[1], now[2], now[3]);
  return bad;
}

}  // namespace exact
}  // namespace pe
