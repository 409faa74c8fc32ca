// Relative 5D ENO/LF stage, exact variant, tiled: the results of
// relative5d_exact.cu bit for bit (double local arithmetic in the order of
// native_relative.cpp:38-67, :124-172, float32 storage), on the streaming
// scheme of the float32 stage (relative5d_ring.cuh): a work item is `rows` y
// rows of one (vP, vE) pair over a chunk of headings, a consumer thread owns
// 4 consecutive x cells of a row and walks the headings, a producer warp
// streams the planes by bulk copies.  Compiled with -fmad=false.
//
// The thread-per-cell kernel forms 25 quotients, 10 selections and 21
// conversions per cell, with a range check on every quotient; here the
// heading axis' are carried from step to step, the x axis' shared inside the
// chunk, and the range checks are replaced by one test of the result
// (relative5d_exact_walk.cuh): about 165 double operations per cell (64 per
// clock and SM), whose dependent chains bound it with 10 to 16 warps per SM (FP64
// pipe 38 to 42 % busy at 33x24x11x11): 1.82 ms per stage at 65x48x21x21 (4.0 ms
// for the thread-per-cell kernel), of which the double operations are 0.85.
#include "launch_shape.cuh"
#include "relative5d_exact_walk.cuh"
#include "relative5d_ring.cuh"

namespace pe {
namespace {

using namespace ring;

// The spacings' constants are made on the host: as kernel parameters they are
// operands in the constant bank, where 20 doubles made in the kernel took
// registers of the 128 that two CTAs per SM leave a thread (RK2 step of
// 33x24x11x11 0.208 -> 0.202 ms, 57x36x17x17 1.75 -> 1.67, 64x48x21x21 3.33 ->
// 3.24).  65x48x21x21 takes 3.63 ms: 3.78 before, and 3.59 in a variant compiled
// for its row pitch and 13 rows, which no other grid could use.
struct WalkArgs {
  RingArgs ring;
  exact::AxisSteps st;
};

// heading (cos, sin) pairs and x positions, in double
__host__ __device__ inline int table_bytes(const Rel5Grid &g) { return 16 * g.nh + 8 * g.xp; }

template <int ORDER, int BLEND, int XR, bool OVERLAP>
__global__ void __launch_bounds__(TARGET_THREADS, 2)
    rel5_walk_exact_kernel(const __grid_constant__ WalkArgs args) {
  const RingArgs &a = args.ring;
  extern __shared__ __align__(128) float smem[];
  const Rel5Grid &g = a.g;
  const int R = a.rows, XP = g.xp, XC = a.xc;
  const SmemLayout L = smem_layout(R, XP, table_bytes(g));
  float *own = smem + L.own_off;  // [8][R+4][XP]
  float *nbr = smem + L.nb_off;   // [2][9][R][XP]
  char *raw = reinterpret_cast<char *>(smem);
  uint64_t *full = reinterpret_cast<uint64_t *>(raw + L.bar_off);
  uint64_t *empty = full + STEP_SLOTS;
  double2 *trig = reinterpret_cast<double2 *>(raw + L.trig_off);  // [nh] cos, sin
  double *xtab = reinterpret_cast<double *>(trig + g.nh);         // [xp]

  const int64_t PP = (int64_t)g.nx * XP;  // plane pitch
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool producer = warp == a.consumer_warps;
  unsigned int *timeout = &a.s.stats->timeout;

  if (tid == 0) {
    for (int i = 0; i < STEP_SLOTS; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 32 * a.consumer_warps);
    }
    fence_barrier_init();
  }
  for (int k = tid; k < g.nh; k += blockDim.x)
    trig[k] = make_double2(__ldg(a.s.cs + k), __ldg(a.s.sn + k));
  for (int k = tid; k < XP; k += blockDim.x) xtab[k] = -g.extent + k * g.dx;
  if (OVERLAP) {
    grid_launch_next();
    grid_wait_previous();  // the fields the stage before this one wrote
    // the step's residual starts at its second stage: clear it in the first
    if (ORDER == 2 && !BLEND && blockIdx.x == 0 && tid == 0) a.s.stats->residual = 0ull;
  }
  __syncthreads();

  bool bad = false;
  exact::ChangeMax change;

  if (producer) {
    if (lane == 0) produce<BLEND>(a, L, own, nbr, full, empty, XP);
  } else {
    const int r = tid / XC, c = tid % XC;
    const int x0 = 4 * c;
    const bool first = x0 == 0;
    constexpr int KP = (XR + 2) & 3, IEND = (XR + 3) & 3;
    const bool kend = x0 == g.nx - 2 - KP, iend = x0 == g.nx - 1 - IEND;
    const int valid = iend ? IEND + 1 : 4;
    const exact::AxisSteps &st = args.st;
    const int ctr = (r + 2) * XP + x0;  // this chunk in an own slot
    const int nbo = r * XP + x0;        // this chunk in a neighbour slot
    bool alive = true;
    unsigned og = 0, gs = 0;

    for (int idx = blockIdx.x; idx < a.items && alive; idx += gridDim.x) {
      const Item it = decode_item(a, idx);
      const bool active = r < it.r_eff;
      // warps holding a row within two of a y end take the general y rules
      const int rw0 = (32 * warp) / XC;
      const int rw1 = min((32 * warp + 31) / XC, it.r_eff - 1);
      exact::ItemCoef q;
      q.set(g, it.iv, it.ie, a.s.dt);
      exact::RowCoef row;
      row.iy = it.y0 + r;
      row.y = -g.extent + row.iy * g.dx;
      row.general = it.y0 + rw0 < 2 || it.y0 + rw1 + 2 >= g.nx;
      const unsigned base = og;  // issue index of own plane d = -2
      og += it.steps + 4;
      int64_t j = (((int64_t)(it.iv - g.slab_lo) * g.nve + it.ie) * g.nh + it.p0) * PP +
                  (int64_t)row.iy * XP + x0;
      auto own_at = [&](unsigned p) -> const float * {
        return own + (p & (OWN_SLOTS - 1)) * L.own_floats + ctr;
      };
      auto own4 = [&](unsigned p) { return *reinterpret_cast<const float4 *>(own_at(p)); };

      // Step 0's set holds planes -2..2: start the heading differences.
      if (alive) alive = wait_phase(&full[gs & 1u], (gs >> 1) & 1u, timeout);
      exact::HeadingCarry<ORDER> carry;
      if (active)  // lanes past the item's rows read nothing
        carry.start(own4(base), own4(base + 1), own4(base + 2), own4(base + 3), st.psi);

#pragma unroll 1
      for (int k = 0; k < it.steps; k++) {
        const unsigned slot = gs & 1u;
        if (k > 0 && alive) alive = wait_phase(&full[slot], (gs >> 1) & 1u, timeout);
        if (active && alive) {
          const float *o0 = own_at(base + k + 2);  // centre plane k
          const float *nb = nbr + slot * NB_PLANES * L.nb_floats + nbo;
          const float4 C = *reinterpret_cast<const float4 *>(o0);
          const double2 cssn = trig[it.p0 + k];
          double H[4];
          exact::walk_hamiltonian<ORDER, XR>(
              *reinterpret_cast<const float2 *>(o0 - 2), C,
              *reinterpret_cast<const float2 *>(o0 + 4), own4(base + k + 3),
              own4(base + k + 4), o0, XP, nb, L.nb_floats, first, kend, iend, 0, 0,
              xtab + x0, cssn.x, cssn.y, q, row, st, carry, H);
          const float4 P =
              BLEND ? *reinterpret_cast<const float4 *>(nb + NEIGHBOURS * L.nb_floats) : C;
          bad |= exact::walk_update<ORDER, BLEND>(g, a.s, x0, it.p0 + k, j, valid, q, row,
                                                  xtab + x0, C, P, H, change);
        }
        mbar_arrive(&empty[slot]);  // release this step's set
        gs++;
        j += PP;
      }
    }
  }

  // Block reductions: non-finite flag, largest change and increase.
  if (__syncthreads_or(bad) && tid == 0) atomicOr(&a.s.stats->nonfinite, 1u);
  if (BLEND || ORDER == 1) {
    double m_abs = change.abs_max, m_up = change.up_max;
    for (int off = 16; off > 0; off >>= 1) {
      m_abs = fmax(m_abs, __shfl_xor_sync(0xffffffffu, m_abs, off));
      m_up = fmax(m_up, __shfl_xor_sync(0xffffffffu, m_up, off));
    }
    if (lane == 0) {
      exact::atomic_max_nonneg(&a.s.stats->residual, m_abs);
      exact::atomic_max_nonneg(&a.s.stats->increase, m_up);
    }
  }
}

template <int ORDER, int BLEND, int XR, bool OVERLAP>
cudaError_t launch_xr(const RingArgs &args, size_t smem, int threads, cudaStream_t stream) {
  auto kernel = rel5_walk_exact_kernel<ORDER, BLEND, XR, OVERLAP>;
  static thread_local LaunchShape shape;
  const cudaError_t e =
      launch_shape(reinterpret_cast<const void *>(kernel), threads, smem, shape);
  if (e != cudaSuccess) return e;
  const int ctas = std::min(args.items, shape.sms * shape.resident);
  const Rel5Grid &g = args.g;
  const WalkArgs walk{args, exact::AxisSteps{exact::axis_step(g.dx, g.rdx, g.rdx2),
                                             exact::axis_step(g.dphi, g.rdphi, g.rdphi2),
                                             exact::axis_step(g.dvp, g.rdvp, g.rdvp2),
                                             exact::axis_step(g.dve, g.rdve, g.rdve2)}};
  return launch_overlapped(OVERLAP, kernel, dim3((unsigned)ctas), threads, smem, stream, walk);
}

template <int ORDER, int BLEND, bool OVERLAP>
cudaError_t launch_nx(const RingArgs &args, size_t smem, int threads, cudaStream_t stream) {
  switch (args.g.nx & 3) {
    case 0: return launch_xr<ORDER, BLEND, 0, OVERLAP>(args, smem, threads, stream);
    case 1: return launch_xr<ORDER, BLEND, 1, OVERLAP>(args, smem, threads, stream);
    case 2: return launch_xr<ORDER, BLEND, 2, OVERLAP>(args, smem, threads, stream);
    default: return launch_xr<ORDER, BLEND, 3, OVERLAP>(args, smem, threads, stream);
  }
}

template <int ORDER, int BLEND>
cudaError_t launch(const RingArgs &args, size_t smem, int threads, cudaStream_t stream) {
  return args.overlap ? launch_nx<ORDER, BLEND, true>(args, smem, threads, stream)
                      : launch_nx<ORDER, BLEND, false>(args, smem, threads, stream);
}

}  // namespace

// The tiled kernel takes the padded layout on 16-byte bounds, in a tile whose
// rings and tables fit, where it is the faster one: its stage takes about 3.4
// times the float32 stage's, the thread-per-cell stage 4 us and 45 us per
// million cells, row padding not counted.  Near equal estimates the tiled one is
// up to 17 % low, so it has to be 8 % below (B200, us per RK2 step in tiles and
// per cell: 21x16x7x7 42.7, 38.1; 21x16x9x9 60.2, 59.0; 25x18x7x7 65.1, 53.2;
// 25x18x9x9 64, 88; 33x24x11x11 202, 293; 65x48x21x21 3630, 8000.  It costs
// 23x16x7x7 44.7, 46.7).
bool rel5_walk_exact_applies(const Rel5Grid &g, const Rel5Tile &t, const Rel5Stage &s) {
  if (g.xp % 4 != 0 || g.sy != g.xp ||
      ((reinterpret_cast<uintptr_t>(s.src) | reinterpret_cast<uintptr_t>(s.dst)) & 15) != 0)
    return false;
  if (!rel5_tile_valid(g, t) ||
      smem_layout(t.rows, g.xp, table_bytes(g)).bytes > 227 * 1024)
    return false;
  const double cells =
      (double)g.nx * g.nx * g.nh * g.nve * (g.own_n > 0 ? g.own_n : g.nvp);
  return 3.4 * rel5_tile_cost(g, t) < 0.92 * (4.0 + 45e-6 * cells);
}

cudaError_t rel5_stage_f64_tiled(const Rel5Grid &g, const Rel5Tile &t, const Rel5Stage &s,
                                 int blend, cudaStream_t stream) {
  const RingArgs args = ring_args(g, t, s);
  const int threads = 32 * (args.consumer_warps + 1);
  const size_t smem = (size_t)smem_layout(t.rows, g.xp, table_bytes(g)).bytes;
  const cudaError_t e = ring::clear_residual(args, blend, stream);
  if (e != cudaSuccess) return e;
  if (g.order == 1) return launch<1, 0>(args, smem, threads, stream);
  if (blend) return launch<2, 1>(args, smem, threads, stream);
  return launch<2, 0>(args, smem, threads, stream);
}

}  // namespace pe
