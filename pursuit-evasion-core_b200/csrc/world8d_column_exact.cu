// Dense 8D ENO/Lax-Friedrichs stage in the reference's operation order
// (native_world.cpp:32-74 slopes, :261-314 stage), bit for bit the
// thread-per-cell kernel of world8d_stage.cuh, by pursuer poses: the passes of
// the fast column kernel (world8d_fast.cu) with the exact arithmetic.
// Compiled with -fmad=false.
//
// A persistent CTA takes the evader block of one pursuer pose (xP, yP, thP,
// vP), staged in shared memory with two ghost rows on each side of xE and yE.
// Per group of vE columns:
//   A (a thread per cell): the four pursuer axes from the same cell of the 16
//     neighbouring blocks, the loads of the next two cells issued first; four
//     partial sums per cell to shared memory (flow terms, dissipation, heading
//     term, acceleration term: the reference adds them at different places);
//   B (a thread per vE column): the four evader axes from the padded block,
//     the vE quotients and selections once per edge and node of the column;
//     H + dissipation back to shared memory;
//   C (a thread per cell): update, RK2 average, tube, avoid floor, arrival.
// Position tests and index splits are per pose or column instead of per cell,
// and quotients by the spacings are the reciprocal product with one FMA
// correction without div_rn.cuh's range checks:
//   * underflow cannot occur while the field holds no nonzero value below
//     2^-70 (its differences are zero or at least 2^-93, and a residual is a
//     multiple of 2^-140 or more).  Every stage records whether its output
//     does; a launch whose input does runs the thread-per-cell arithmetic;
//   * overflow, infinities and NaN end in a total that is not finite; such a
//     cell is recomputed by the thread-per-cell arithmetic;
//   * the sign of a zero quotient may differ, and no sum depends on it (H and
//     the dissipation start from +0).
// Bound by instruction issue (64 % of the slots, 620 instructions per cell; 16
// warps per SM).  RK2 step of 11x9x7x7 (58 M cells) 7.73 -> 3.24 ms, of 9x8x7x7
// 2.79 -> 1.12 ms; it is the faster one down to the smallest grid (5x4x3x3: 35
// -> 31 us).  The x and y axes of a cell share their spacing and go through
// packed FP32 together (7 % of the step).
#include "launch_shape.cuh"
#include "world8d_column.cuh"
#include "world8d_stage.cuh"

namespace pe {
namespace {

constexpr int kT = 256;                     // threads
constexpr size_t kPerSm = 227 * 1024;       // shared memory of one SM's CTAs
constexpr int kBatch = 4;                   // cells of pass C loaded together

struct AxisQ {
  float h, rh, hh, rhh, half;
};

struct ColExactArgs {
  World8Grid g;
  World8Stage s;
  AxisQ axis[4];  // position, pursuer speed, heading, evader speed
  int inner, outer, ncols, group;
  Divisor dnh, dn;
};

__device__ __forceinline__ float quot(float a, float b, float r) {
  const float q = a * r;
  return fmaf(fmaf(-q, b, a), r, q);
}
__device__ __forceinline__ float quot1(float a, const AxisQ &x) { return quot(a, x.h, x.rh); }
// second difference quotient of m, v, p: ((p - 2 v) + m) / h^2, 2 v exact
__device__ __forceinline__ float quot2(float p, float v, float m, const AxisQ &x) {
  return quot(fmaf(-2.f, v, p) + m, x.hh, x.rhh);
}
// The smaller second quotient, ties to the first: one compare on the
// magnitudes and one select, written out so that no integer sign masking is
// generated.
__device__ __forceinline__ float smaller(float a, float b) {
  float r;
  asm("{\n .reg .pred p;\n .reg .f32 ua, ub;\n abs.f32 ua, %1;\n abs.f32 ub, %2;\n"
      " setp.le.f32 p, ua, ub;\n selp.f32 %0, %1, %2, p;\n}"
      : "=f"(r)
      : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float edge_term(float a, float b, const AxisQ &x) {
  return x.half * smaller(a, b);
}

// Value m nodes beyond an end (a: end node, b: the node next to it).
__device__ __forceinline__ float ghost_of(float a, float b, float m) {
  return a + m * fabsf(b - a) * ((a > 0) - (a < 0));
}

// Slopes of an interior (or ghost-extended) node.
template <int ORDER>
__device__ __forceinline__ void node_slopes(float m2, float m1, float f, float p1, float p2,
                                            const AxisQ &x, float &lo, float &hi) {
  lo = quot1(f - m1, x);
  hi = quot1(p1 - f, x);
  if (ORDER == 2) {
    const float dc = quot2(p1, f, m1, x);
    lo += edge_term(quot2(f, m1, m2, x), dc, x);
    hi -= edge_term(dc, quot2(p2, p1, f, x), x);
  }
}

// The same for two axes at once in packed FP32 (each element rounds as the
// scalar operation): x and y, or heading and pursuer speed, of one cell.
struct AxisQ2 {
  float2 nh, rh, nhh, rhh, half;  // -h and -h * h
};

__device__ __forceinline__ AxisQ2 pair_of(const AxisQ &a, const AxisQ &b) {
  return AxisQ2{make_float2(-a.h, -b.h), make_float2(a.rh, b.rh), make_float2(-a.hh, -b.hh),
                make_float2(a.rhh, b.rhh), make_float2(a.half, b.half)};
}
// Packed operations.  A packed product that goes into a packed sum is rounded
// once, in one fused operation, even with -fmad=false and as PTX's .rn forms:
// the only such product (edge_pair's) is taken element by element.
__device__ __forceinline__ uint64_t bits2(float2 a) {
  return (uint64_t)__float_as_uint(a.y) << 32 | __float_as_uint(a.x);
}
__device__ __forceinline__ float2 value2(uint64_t b) {
  return make_float2(__uint_as_float((uint32_t)b), __uint_as_float((uint32_t)(b >> 32)));
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)));
  return value2(r);
}
__device__ __forceinline__ float2 plus2(float2 a, float2 b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(a)), "l"(bits2(b)));
  return value2(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
  return value2(r);
}
__device__ __forceinline__ float2 two(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 minus(float2 a, float2 b) { return fma2(b, two(-1.f), a); }
__device__ __forceinline__ float2 quot_pair(float2 a, float2 nb, float2 r) {
  const float2 q = mul2(a, r);
  return fma2(fma2(q, nb, a), r, q);
}
__device__ __forceinline__ float2 quot2_pair(float2 p, float2 v, float2 m, const AxisQ2 &x) {
  return quot_pair(plus2(fma2(v, two(-2.f), p), m), x.nhh, x.rhh);
}
__device__ __forceinline__ float2 edge_pair(float2 a, float2 b, const AxisQ2 &x) {
  return make_float2(__fmul_rn(x.half.x, smaller(a.x, b.x)),
                     __fmul_rn(x.half.y, smaller(a.y, b.y)));
}
template <int ORDER>
__device__ __forceinline__ void node_slopes_pair(float2 m2, float2 m1, float2 f, float2 p1,
                                                 float2 p2, const AxisQ2 &x, float2 &lo,
                                                 float2 &hi) {
  lo = quot_pair(minus(f, m1), x.nh, x.rh);
  hi = quot_pair(minus(p1, f), x.nh, x.rh);
  if (ORDER == 2) {
    const float2 dc = quot2_pair(p1, f, m1, x);
    lo = plus2(lo, edge_pair(quot2_pair(f, m1, m2, x), dc, x));
    hi = minus(hi, edge_pair(dc, quot2_pair(p2, p1, f, x), x));
  }
}

// Ends of a non-periodic axis: ghosts from the clamped window.
__device__ __forceinline__ void extend(float &m2, float &m1, float f, float &p1, float &p2,
                                       int pos, int n) {
  if (pos == 0) {
    m1 = ghost_of(f, p1, 1.f);
    m2 = ghost_of(f, p1, 2.f);
  } else if (pos == 1) {
    m2 = ghost_of(m1, f, 1.f);
  }
  if (pos == n - 1) {
    p1 = ghost_of(f, m1, 1.f);
    p2 = ghost_of(f, m1, 2.f);
  } else if (pos == n - 2) {
    p2 = ghost_of(p1, f, 1.f);
  }
}

struct CellFlags {
  float change;
  bool bad, tiny;
};

// One cell in the thread-per-cell arithmetic, out of line.
__device__ __noinline__ CellFlags general_cell(const World8Grid &g, const World8Stage &s, int o,
                                               int inner, int e) {
  CellFlags f{0.f, false, false};
  w8::stage_cell<false>(g, s, o, inner, e, f.change, f.bad, f.tiny);
  return f;
}

template <int ORDER, int NE, int SKIND>
__global__ void __launch_bounds__(kT, 2)
    world8_column_exact_kernel(const __grid_constant__ ColExactArgs a) {
  extern __shared__ __align__(16) float sm[];
  __shared__ float warp_max[kT / 32];
  const World8Grid &g = a.g;
  const World8Stage &s = a.s;
  const int inner = a.inner, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nwarps = kT / 32;
  const int n = g.n, nh = g.nh;
  const int rowlen = nh * NE;
  const int sy = rowlen, sx = (n + 4) * rowlen;
  const int cells = a.group * NE;  // of one column group
  float *pad = sm;                 // [n+4][n+4][nh][NE]
  float *flow = sm + (n + 4) * sx, *diss = flow + cells, *turn = diss + cells,
        *accel = turn + cells;
  const AxisQ2 xy = pair_of(a.axis[0], a.axis[0]);
  float change_max = 0.f;
  bool bad = false, tiny = false;

  if (*s.src_tiny) {  // the input needs the range-checked quotients
    for (int o = blockIdx.x; o < a.outer; o += gridDim.x)
      for (int e = tid; e < inner; e += kT) {
        const CellFlags f = general_cell(g, s, o, inner, e);
        change_max = fmaxf(change_max, f.change);
        bad |= f.bad;
        tiny |= f.tiny;
      }
  } else {
    auto stage_block = [&](int o) {
      const float *src = s.src + (int64_t)o * inner;
      for (int r = warp; r < n * n; r += nwarps) {
        const int q4 = r / n, q5 = r - q4 * n;
        float *dst = pad + (q4 + 2) * sx + (q5 + 2) * sy;
        const float *row = src + r * rowlen;
        for (int j = lane; j < rowlen; j += 32) cp_async4(dst + j, row + j);
      }
    };
    // ghost rows: side 0-3 xE = -2, -1, n, n+1 at yE = idx; 4-7 along yE
    auto fill_ghosts = [&]() {
      for (int gr = warp; gr < 8 * n; gr += nwarps) {
        const int side = gr / n, idx = gr - side * n;
        const int q = side & 3;
        const int pos = q < 2 ? q - 2 : n - 2 + q;
        const float m = q == 0 || q == 3 ? 2.f : 1.f;
        const int end = q < 2 ? 0 : n - 1, next = q < 2 ? 1 : n - 2;
        const int along = side < 4 ? sx : sy, across = side < 4 ? sy : sx;
        const float *row_a = pad + (end + 2) * along + (idx + 2) * across;
        const float *row_b = pad + (next + 2) * along + (idx + 2) * across;
        float *row_g = pad + (pos + 2) * along + (idx + 2) * across;
        for (int j = lane; j < rowlen; j += 32) row_g[j] = ghost_of(row_a[j], row_b[j], m);
      }
    };

    if ((int)blockIdx.x < a.outer) stage_block(blockIdx.x);
    cp_async_commit();
    for (int o = blockIdx.x; o < a.outer; o += gridDim.x) {
      int qp[4];
      {
        int rest = o;
        qp[3] = rest % g.shape[3];
        rest /= g.shape[3];
        qp[2] = rest % g.shape[2];
        rest /= g.shape[2];
        qp[1] = rest % g.shape[1];
        qp[0] = rest / g.shape[1];
      }
      const float vp = __ldg(s.pv + qp[3]);
      const float palo = qp[3] == 0 ? 0 : -g.ap, pahi = qp[3] == g.np - 1 ? 0 : g.ap;
      const float fpx = vp * __ldg(s.cs + qp[2]), fpy = vp * __ldg(s.sn + qp[2]);
      const float wp = fabsf(vp) * g.kp;
      float avoid = -INFINITY;
      if (g.avoid_mode == 1) {
        const float ax = fabsf(__ldg(s.x + qp[0])), ay = fabsf(__ldg(s.x + qp[1]));
        avoid = (ax < ay ? ay : ax) - g.arena + 1e-6f;
      } else if (g.avoid_mode == 2) {
        avoid = -__ldg(s.p_clear + (qp[0] * g.n + qp[1]) * g.nh + qp[2]) + 1e-6f;
      }
      int poff[4][4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        int om2, om1, op1, op2;
        window_offsets(qp[k], g.shape[k], 1, k == 2, om2, om1, op1, op2);
        const int st = (int)g.stride[k];
        poff[k][0] = om2 * st;
        poff[k][1] = om1 * st;
        poff[k][2] = op1 * st;
        poff[k][3] = op2 * st;
      }
      const bool x_end = qp[0] < 2 || qp[0] + 2 >= n, y_end = qp[1] < 2 || qp[1] + 2 >= n;
      const bool v_end = qp[3] < 2 || qp[3] + 2 >= g.np;
      const int64_t j0 = (int64_t)o * inner;
      const float *__restrict__ src_o = s.src + j0;

      for (int c0 = 0; c0 < a.ncols; c0 += a.group) {
        const int c1 = min(a.ncols, c0 + a.group);
        const int e0 = c0 * NE, count = (c1 - c0) * NE;
        // ---- A
        auto load_cell = [&](int e, float (&buf)[17]) {
          // (block base, the same for the whole CTA) + 32-bit cell offset
          const uint32_t at = (uint32_t)(e0 + min(e, count - 1));
          buf[16] = __ldg(src_o + at);
#pragma unroll
          for (int k = 0; k < 4; k++)
#pragma unroll
            for (int m = 0; m < 4; m++) buf[4 * k + m] = __ldg(src_o + poff[k][m] + at);
        };
        auto pursuer_cell = [&](int e, float (&b)[17]) {
          const float f = b[16];
          float lo, hi;
          if (x_end) extend(b[0], b[1], f, b[2], b[3], qp[0], n);
          if (y_end) extend(b[4], b[5], f, b[6], b[7], qp[1], n);
          float2 xylo, xyhi;
          node_slopes_pair<ORDER>(make_float2(b[0], b[4]), make_float2(b[1], b[5]), two(f),
                                  make_float2(b[2], b[6]), make_float2(b[3], b[7]), xy, xylo,
                                  xyhi);
          const float2 gxy = mul2(two(.5f), plus2(xylo, xyhi));
          const float2 jxy = minus(xyhi, xylo);
          float Hs = 0.f + fpx * gxy.x;
          float ds = 0.f + .5f * fabsf(fpx) * jxy.x;
          Hs += fpy * gxy.y;
          ds += .5f * fabsf(fpy) * jxy.y;
          node_slopes<ORDER>(b[8], b[9], f, b[10], b[11], a.axis[2], lo, hi);
          const float g2 = .5f * (lo + hi);
          ds += .5f * wp * (hi - lo);
          if (SKIND == kExtrapolated) {
            if (v_end) extend(b[12], b[13], f, b[14], b[15], qp[3], g.np);
            node_slopes<ORDER>(b[12], b[13], f, b[14], b[15], a.axis[1], lo, hi);
          } else if (!v_end) {
            node_slopes<ORDER>(b[12], b[13], f, b[14], b[15], a.axis[1], lo, hi);
          } else {  // one-sided at the ends, the centred quotient next to them
            const float dl = quot1(f - b[13], a.axis[1]), dh = quot1(b[14] - f, a.axis[1]);
            lo = dl;
            hi = dh;
            if (ORDER == 2) {
              const float dc = quot2(b[14], f, b[13], a.axis[1]);
              const float l2 = qp[3] < 2 ? dc : quot2(f, b[13], b[12], a.axis[1]);
              const float r2 = qp[3] + 2 >= g.np ? dc : quot2(b[15], b[14], f, a.axis[1]);
              lo += edge_term(l2, dc, a.axis[1]);
              hi -= edge_term(dc, r2, a.axis[1]);
            }
            if (qp[3] == 0) lo = hi = dh;
            if (qp[3] == g.np - 1) lo = hi = dl;
          }
          const float g3 = .5f * (lo + hi);
          ds += .5f * g.ap * (hi - lo);
          const float p_lo = palo * g3, p_hi = pahi * g3;
          flow[e] = Hs;
          diss[e] = ds;
          turn[e] = -wp * fabsf(g2);
          accel[e] = p_hi < p_lo ? p_hi : p_lo;
        };
        {
          float bufA[17], bufB[17];
          if (tid < count) load_cell(tid, bufA);
          for (int e = tid; e < count; e += 2 * kT) {
            if (e + kT < count) load_cell(e + kT, bufB);
            pursuer_cell(e, bufA);
            if (e + kT >= count) break;
            if (e + 2 * kT < count) load_cell(e + 2 * kT, bufA);
            pursuer_cell(e + kT, bufB);
          }
        }
        if (c0 == 0) {
          cp_async_wait_all();
          __syncthreads();  // the block is in place
          fill_ghosts();
        }
        __syncthreads();  // ghosts and pursuer parts are in place
        // ---- B
        for (int c = c0 + tid; c < c1; c += kT) {
          int q6, q5;
          const int r = split(c, a.dnh, q6);
          const int q4 = split(r, a.dn, q5);
          const float *col = pad + (q4 + 2) * sx + (q5 + 2) * sy + q6 * NE;
          int om2, om1, op1, op2;
          window_offsets(q6, nh, NE, true, om2, om1, op1, op2);
          const float cs6 = __ldg(s.cs + q6), sn6 = __ldg(s.sn + q6);
          const int at = (c - c0) * NE;
          float vc[NE];
#pragma unroll
          for (int i = 0; i < NE; i++) vc[i] = col[i];
          // vE: quotient and selection of every edge (i, i+1), -1 <= i < NE
          // (inward: ends one-sided, the missing outer quotient is the inner)
          float lo7[NE], hi7[NE];
          {
            const AxisQ &x = a.axis[3];
            float w[NE + 4];
#pragma unroll
            for (int i = 0; i < NE; i++) w[i + 2] = vc[i];
            if (SKIND == kExtrapolated) {
              w[0] = ghost_of(vc[0], vc[1], 2.f);
              w[1] = ghost_of(vc[0], vc[1], 1.f);
              w[NE + 2] = ghost_of(vc[NE - 1], vc[NE - 2], 1.f);
              w[NE + 3] = ghost_of(vc[NE - 1], vc[NE - 2], 2.f);
            }
            constexpr int E0 = SKIND == kExtrapolated ? 0 : 1;  // first, last edge used:
            constexpr int E1 = SKIND == kExtrapolated ? NE : NE - 1;  // edge i: (i-1, i)
            float D[NE + 1], E[NE + 1], c2[NE + 2];  // c2[i + 1]: node i
#pragma unroll
            for (int i = E0; i <= E1; i++) D[i] = quot1(w[i + 2] - w[i + 1], x);
            if (ORDER == 2) {
#pragma unroll
              for (int i = -1; i <= NE; i++)
                if (SKIND == kExtrapolated || (i >= 1 && i <= NE - 2))
                  c2[i + 1] = quot2(w[i + 3], w[i + 2], w[i + 1], x);
              if (SKIND != kExtrapolated) {
                c2[1] = c2[2];
                c2[NE] = c2[NE - 1];
              }
#pragma unroll
              for (int i = E0; i <= E1; i++) E[i] = edge_term(c2[i], c2[i + 1], x);
            }
#pragma unroll
            for (int i = 0; i < NE; i++) {
              const bool first = SKIND != kExtrapolated && i == 0;
              const bool last = SKIND != kExtrapolated && i == NE - 1;
              const int el = first ? 1 : i, eh = last ? NE - 1 : i + 1;
              lo7[i] = first || last || ORDER == 1 ? D[first || !last ? el : eh]
                                                   : D[el] + E[el];
              hi7[i] = first || last || ORDER == 1 ? D[last || !first ? eh : el]
                                                   : D[eh] - E[eh];
            }
          }
#pragma unroll
          for (int i = 0; i < NE; i++) {
            const float f = vc[i];
            const float ve = __ldg(s.ev + i), we = fabsf(ve) * g.ke;
            const float fex = ve * cs6, fey = ve * sn6;
            float Hs = flow[at + i], ds = diss[at + i], lo, hi;
            float2 xylo, xyhi;
            node_slopes_pair<ORDER>(make_float2(col[i - 2 * sx], col[i - 2 * sy]),
                                    make_float2(col[i - sx], col[i - sy]), two(f),
                                    make_float2(col[i + sx], col[i + sy]),
                                    make_float2(col[i + 2 * sx], col[i + 2 * sy]), xy, xylo,
                                    xyhi);
            const float2 gxy = mul2(two(.5f), plus2(xylo, xyhi));
            const float2 jxy = minus(xyhi, xylo);
            Hs += fex * gxy.x;
            ds += .5f * fabsf(fex) * jxy.x;
            Hs += fey * gxy.y;
            ds += .5f * fabsf(fey) * jxy.y;
            node_slopes<ORDER>(col[i + om2], col[i + om1], f, col[i + op1], col[i + op2],
                               a.axis[2], lo, hi);
            const float g6 = .5f * (lo + hi);
            ds += .5f * we * (hi - lo);
            const float g7 = .5f * (lo7[i] + hi7[i]);
            ds += .5f * g.ae * (hi7[i] - lo7[i]);
            const float ealo = i == 0 ? 0 : -g.ae, eahi = i == NE - 1 ? 0 : g.ae;
            const float e_lo = ealo * g7, e_hi = eahi * g7;
            Hs += turn[at + i] + we * fabsf(g6) + accel[at + i] + (e_lo < e_hi ? e_hi : e_lo);
            flow[at + i] = Hs + ds;
          }
        }
        __syncthreads();  // the group's sums are complete
        if (c1 == a.ncols) {  // and the padded block is free
          const int next = o + gridDim.x;
          if (next < a.outer) stage_block(next);
          cp_async_commit();
        }
        // ---- C (a thread's own cells of pass A, so the next group or pose may
        // write its sums without a barrier)
        const float *base_o = s.base ? s.base + j0 + e0 : nullptr;
        for (int eb = tid; eb < count; eb += kBatch * kT) {
          float fv[kBatch], bv[kBatch], tv[kBatch];
#pragma unroll
          for (int h = 0; h < kBatch; h++) {
            const int c = min(eb + h * kT, count - 1);
            fv[h] = __ldg(src_o + e0 + c);
            bv[h] = base_o ? __ldg(base_o + c) : fv[h];
            tv[h] = flow[c];
          }
#pragma unroll
          for (int h = 0; h < kBatch; h++) {
            const int c = eb + h * kT;
            if (c >= count) break;
            const int64_t j = j0 + e0 + c;
            float value = fv[h] + s.dt * tv[h];
            if (base_o) value = .5f * (bv[h] + value);
            if (!isfinite(tv[h]) || !isfinite(value)) {
              const CellFlags f = general_cell(g, s, o, inner, e0 + c);
              change_max = fmaxf(change_max, f.change);
              bad |= f.bad;
              tiny |= f.tiny;
              continue;
            }
            if (g.order == 1 || base_o) {
              const float previous = bv[h];  // the partner, or the stage input
              const float tube = previous < value ? previous : value;
              value = tube < avoid ? avoid : tube;
              if (previous > 0 && value <= 0 && isnan(s.arrival[j]))
                s.arrival[j] = (float)s.tau + s.dt * previous / (previous - value);
              change_max = fmaxf(change_max, fabsf(value - previous));
            }
            bad |= !isfinite(value);
            tiny |= w8::tiny_value(value);
            s.dst[j] = value;
          }
        }
      }
    }
    cp_async_wait_all();
  }

  if (__syncthreads_or(bad) && tid == 0) atomicOr(&s.stats->nonfinite, 1u);
  if (__syncthreads_or(tiny) && tid == 0) atomicOr(s.dst_tiny, 1u);
  for (int off = 16; off > 0; off >>= 1)
    change_max = fmaxf(change_max, __shfl_xor_sync(0xffffffffu, change_max, off));
  if (lane == 0) warp_max[warp] = change_max;
  __syncthreads();
  if (tid == 0) {
    float m = 0.f;
    for (int w = 0; w < nwarps; w++) m = fmaxf(m, warp_max[w]);
    if (m > 0.f)
      atomicMax(&s.stats->residual, (unsigned long long)__double_as_longlong((double)m));
  }
}

__global__ void scan_tiny_kernel(const float *__restrict__ field, int64_t n, unsigned *tiny) {
  bool any = false;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x)
    any |= w8::tiny_value(field[j]);
  if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(tiny, 1u);
}

size_t pad_bytes(const World8Grid &g) {
  return sizeof(float) * (size_t)g.nh * g.shape[7] * (g.n + 4) * (g.n + 4);
}

// vE columns per group: all of them, else the largest multiple of the CTA's
// threads (every thread of pass B then has a column) with which two CTAs -- or,
// for large blocks, one -- fit an SM; 0: none fits.
int group_columns(const World8Grid &g) {
  const int ncols = g.shape[4] * g.shape[5] * g.shape[6];
  const size_t column = sizeof(float) * 4 * (size_t)g.shape[7];
  for (int ctas = 2; ctas >= 1; ctas--) {
    const size_t room = kPerSm / ctas - 2048;
    if (pad_bytes(g) >= room) continue;
    const int fit = (int)((room - pad_bytes(g)) / column);
    if (fit >= ncols) return ncols;
    if (fit >= kT) return fit / kT * kT;
  }
  return 0;
}

template <int ORDER, int NE, int SKIND>
cudaError_t launch_kind(const ColExactArgs &a, size_t smem, cudaStream_t stream) {
  auto kernel = world8_column_exact_kernel<ORDER, NE, SKIND>;
  static thread_local LaunchShape shape;
  const cudaError_t e = launch_shape(reinterpret_cast<const void *>(kernel), kT, smem, shape);
  if (e != cudaSuccess) return e;
  const int ctas = shape.sms * shape.resident;
  kernel<<<a.outer < ctas ? a.outer : ctas, kT, smem, stream>>>(a);
  return cudaGetLastError();
}

template <int ORDER, int NE>
cudaError_t launch_ne(const ColExactArgs &a, size_t smem, cudaStream_t stream) {
  return a.g.linear_speed ? launch_kind<ORDER, NE, kInward>(a, smem, stream)
                          : launch_kind<ORDER, NE, kExtrapolated>(a, smem, stream);
}

template <int ORDER>
cudaError_t launch(const ColExactArgs &a, size_t smem, cudaStream_t stream) {
  switch (a.g.shape[7]) {
    case 3: return launch_ne<ORDER, 3>(a, smem, stream);
    case 4: return launch_ne<ORDER, 4>(a, smem, stream);
    case 5: return launch_ne<ORDER, 5>(a, smem, stream);
    case 6: return launch_ne<ORDER, 6>(a, smem, stream);
    case 7: return launch_ne<ORDER, 7>(a, smem, stream);
    default: return launch_ne<ORDER, 8>(a, smem, stream);
  }
}

AxisQ axis_of(const World8Grid &g, int k) {
  const float h = g.spacing[k];
  return AxisQ{h, g.inv_spacing[k], h * h, g.inv_spacing_sq[k], .5f * h};
}

}  // namespace

bool world8_column_exact_applies(const World8Grid &g) {
  // block offsets are 32-bit
  return g.shape[7] >= 3 && g.shape[7] <= 8 && g.cells < ((int64_t)1 << 31) &&
         group_columns(g) > 0;
}

cudaError_t world8_stage_column(const World8Grid &g, const World8Stage &s,
                                cudaStream_t stream) {
  ColExactArgs a;
  a.g = g;
  a.s = s;
  a.axis[0] = axis_of(g, 0);
  a.axis[1] = axis_of(g, 3);
  a.axis[2] = axis_of(g, 2);
  a.axis[3] = axis_of(g, 7);
  a.inner = g.shape[4] * g.shape[5] * g.shape[6] * g.shape[7];
  a.outer = (int)(g.cells / a.inner);
  a.ncols = a.inner / g.shape[7];
  a.group = group_columns(g);
  a.dnh = make_divisor(g.nh);
  a.dn = make_divisor(g.n);
  const size_t smem = pad_bytes(g) + sizeof(float) * 4 * (size_t)a.group * g.shape[7];
  return g.order == 1 ? launch<1>(a, smem, stream) : launch<2>(a, smem, stream);
}

cudaError_t world8_scan_tiny(const World8Grid &g, const float *field, unsigned *tiny,
                             cudaStream_t stream) {
  scan_tiny_kernel<<<148 * 8, 256, 0, stream>>>(field, g.cells, tiny);
  return cudaGetLastError();
}

}  // namespace pe
