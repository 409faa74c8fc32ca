// Batched relative 5D solves with the exact cell update, tiled: every solve
// of a batch reproduces the reference executable bit for bit
// (native_relative.cpp:38-67, :124-172), on the item and staging scheme of the
// float32 batched kernel (relative5d_batch_stage.cuh) with the arithmetic of
// the single-grid tiled exact kernel (relative5d_exact_walk.cuh).  Compiled
// with -fmad=false.
//
// A work item is `rows` y rows of one (vP, vE) plane stack over `chunk`
// headings; a thread owns 4 x cells of a row and walks the headings.  The
// chunks keep a batch of few solves spread over the SMs: a stage ends at a
// grid barrier, so its time is that of the CTA with the most items.
//
// Bound by the CTA's barrier per heading (its warps wait there 6 times as long
// as they take to issue) and the latency of the double operations, at 16 warps
// per SM (128 registers; the item's constants lie in shared memory); the FP64
// pipe is 30 % busy.  4 solves of 17-49
// positions, 6.7e8 cell-stages: 56 ms on the cell-per-thread kernel, 22.7 ms
// here; 32 solves, 7.7e9: 233 ms.  Handling two of the four cells at a time
// keeps fewer values live but measured 22 % slower.
#include "launch_shape.cuh"
#include "relative5d_batch_stage.cuh"
#include "relative5d_exact_walk.cuh"

namespace pe {
namespace {

// The solve and item a CTA is on.
struct SharedSolve {
  Rel5Grid g;
  exact::AxisSteps st;
  exact::ItemCoef q;
};

// One stage of one item: headings p0 .. p0 + steps - 1.
template <int BLEND>
__device__ __forceinline__ void item_stage(SharedSolve &ss, const Rel5Stage &s,
                                           const ItemGeom &it, int p0, int steps, float *smem,
                                           StageRing &ring, exact::ChangeMax &change,
                                           bool &bad) {
  const Rel5Grid &g = ss.g;
  const int xp = g.xp, xc = it.xc, nh = g.nh;
  const int64_t PP = (int64_t)g.nx * xp;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int r = tid / xc, c = tid - r * xc;
  const bool active = tid < it.R * xc && r < it.r_eff;
  const int x0 = 4 * c, bufsz = buffer_floats(it.R, xp);
  const bool first = x0 == 0;
  const int kcell = g.nx - 2 - x0, icell = g.nx - 1 - x0;
  const int valid = icell < 3 ? icell + 1 : 4;
  double xs[4];
#pragma unroll
  for (int i = 0; i < 4; i++) xs[i] = -g.extent + (x0 + i) * g.dx;
  // warps holding a row within two of a y end take the general y rules
  const int rw0 = (32 * warp) / xc, rw1 = min((32 * warp + 31) / xc, it.r_eff - 1);
  exact::RowCoef row;
  row.iy = it.y0 + r;
  row.y = -g.extent + row.iy * g.dx;
  row.general = it.y0 + rw0 < 2 || it.y0 + rw1 + 2 >= g.nx;
  // (read after the first heading's barrier; the last item's readers are done)
  if (tid == 0) ss.q.set(g, it.iv, it.ie, s.dt);
  const exact::ItemCoef &q = ss.q;
  const int64_t cell0 = ((int64_t)it.iv * g.nve + it.ie) * nh * PP + (int64_t)row.iy * xp + x0;
  auto load_plane = [&](int p) {
    p = p < 0 ? p + nh : (p >= nh ? p - nh : p);
    return active ? *reinterpret_cast<const float4 *>(s.src + cell0 + (int64_t)p * PP)
                  : make_float4(0.f, 0.f, 0.f, 0.f);
  };

  if (tid < 32) stage_heading(g, s.src, it, p0, smem, &stage_bar[0]);
  ring.filled(0);
  // VN, VNEW: headings k + 1, k + 2 of this chunk
  float4 VN = load_plane(p0 + 1), VNEW = load_plane(p0 + 2);
  exact::HeadingCarry<2> carry;
  carry.start(load_plane(p0 - 2), load_plane(p0 - 1), load_plane(p0), VN, ss.st.psi);
#pragma unroll 1
  for (int k = 0; k < steps; k++) {
    const int b = k & 1;
    wait_staged(ring, b);
    __syncthreads();  // heading k staged; heading k-1's buffer no longer read
    if (k + 1 < steps) {
      if (tid < 32)
        stage_heading(g, s.src, it, p0 + k + 1, smem + (b ^ 1) * bufsz, &stage_bar[b ^ 1]);
      ring.filled(b ^ 1);
    }
    const float4 next = k + 1 < steps ? load_plane(p0 + k + 3) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
      const float *own = smem + b * bufsz;
      const float *o0 = own + (r + 2) * xp + x0;
      const float *nb = own + (it.R + 4) * xp + r * xp + x0;
      const float4 C = *reinterpret_cast<const float4 *>(o0);
      const int64_t cell = cell0 + (int64_t)(p0 + k) * PP;
      const float4 P = BLEND ? *reinterpret_cast<const float4 *>(s.dst + cell) : C;
      double H[4];
      exact::walk_hamiltonian<2, -1>(*reinterpret_cast<const float2 *>(o0 - 2), C,
                                     *reinterpret_cast<const float2 *>(o0 + 4), VN, VNEW, o0, xp,
                                     nb, it.R * xp, first, false, false, kcell,
                                     icell, xs, s.cs[p0 + k], s.sn[p0 + k], q, row, ss.st, carry, H);
      bad |= exact::walk_update<2, BLEND>(g, s, x0, p0 + k, cell, valid, q, row, xs, C, P, H, change);
    }
    VN = VNEW;
    VNEW = next;
  }
  __syncthreads();  // the buffers are restaged by the next item
}

template <int BLEND>
__device__ __forceinline__ void exact_stage(const Rel5BatchArgs &A, int step, int64_t n_items,
                                            double *scratch, SharedSolve *ss, float *smem,
                                            StageRing &ring) {
  int64_t lo = 0, hi = 0;
  const Rel5BatchSolve *S = nullptr;
  Rel5Stage s{};
  int rows = 1, slabs = 1, chunk = 1;
  exact::ChangeMax change;
  bool bad = false;
  auto flush = [&]() {
    if (!S) return;
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&S->stats->nonfinite, 1u);
    if (BLEND) {
      const double m_abs = batch_impl::block_max(change.abs_max, scratch);
      const double m_up = batch_impl::block_max(change.up_max, scratch);
      if (threadIdx.x == 0) {
        batch_impl::atomic_max_nonneg(&S->stats->residual, m_abs);
        batch_impl::atomic_max_nonneg(&S->stats->increase, m_up);
      }
    }
    change = exact::ChangeMax();
    bad = false;
  };
  for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    if (item < lo || item >= hi) {  // the same for every thread of the CTA
      flush();
      S = &A.solves[batch_impl::find_solve(A, item)];
      lo = S->item_base;
      hi = lo + S->items;
      __syncthreads();  // the previous solve's grid copy is no longer read
      if (threadIdx.x == 0) {
        ss->g = S->g;
        ss->st = exact::AxisSteps{exact::axis_step(S->g.dx, S->g.rdx, S->g.rdx2),
                                  exact::axis_step(S->g.dphi, S->g.rdphi, S->g.rdphi2),
                                  exact::axis_step(S->g.dvp, S->g.rdvp, S->g.rdvp2),
                                  exact::axis_step(S->g.dve, S->g.rdve, S->g.rdve2)};
      }
      const double2 td = S->steps[step];
      s.src = BLEND ? S->b : S->a;
      s.dst = BLEND ? S->a : S->b;
      s.arrival = S->arrival;
      s.sn = S->sn;
      s.cs = S->cs;
      s.t = td.x;
      s.dt = td.y;
      s.stats = S->stats;
      rows = S->rows;
      chunk = S->chunk;
      __syncthreads();
      slabs = (ss->g.nx + rows - 1) / rows;
    }
    const Rel5Grid &g = ss->g;
    int64_t local = item - lo;
    ItemGeom it;
    const int slab = (int)(local % slabs);
    local /= slabs;
    it.ie = (int)(local % g.nve);
    local /= g.nve;
    it.iv = (int)(local % g.nvp);
    const int p0 = (int)(local / g.nvp) * chunk;
    it.R = rows;
    it.xc = g.xp / 4;
    it.y0 = slab * rows;
    it.r_eff = min(rows, g.nx - it.y0);
    item_stage<BLEND>(*ss, s, it, p0, min(chunk, g.nh - p0), smem, ring, change, bad);
  }
  flush();
}

__global__ void __launch_bounds__(kThreads, 2)
    rel5_batch_tiled_exact_kernel(const __grid_constant__ Rel5BatchArgs A) {
  extern __shared__ __align__(16) float smem[];
  __shared__ double scratch[kThreads / 32];
  __shared__ SharedSolve ss;
  if (threadIdx.x == 0) {
    bulk::mbar_init(&stage_bar[0], 1);
    bulk::mbar_init(&stage_bar[1], 1);
    bulk::fence_barrier_init();
    stage_timeout = &A.sync[2];
  }
  __syncthreads();
  StageRing ring;
  unsigned round = 0;
  for (int step = 0; step < A.max_steps; step++) {
    const int64_t n_items = A.active_items[step];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < A.count;
         k += gridDim.x * blockDim.x)
      if (step < A.solves[k].nsteps) A.solves[k].stats->residual = 0ull;
    exact_stage<0>(A, step, n_items, scratch, &ss, smem, ring);
    if (!batch_impl::grid_barrier(A.sync, ++round)) break;
    // order the other CTAs' stores before the next stage's bulk copies
    if (threadIdx.x < 32) bulk::fence_async_global();
    exact_stage<1>(A, step, n_items, scratch, &ss, smem, ring);
    if (!batch_impl::grid_barrier(A.sync, ++round)) break;
    if (threadIdx.x < 32) bulk::fence_async_global();
  }
  // no bulk copy may still be landing when the CTA exits
  if (threadIdx.x == 0) {
    if (ring.used(0)) wait_staged(ring, 0);
    if (ring.used(1)) wait_staged(ring, 1);
  }
}

}  // namespace

int rel5_batch_grid_tiled_exact(size_t smem) {
  return cooperative_ctas(reinterpret_cast<const void *>(rel5_batch_tiled_exact_kernel), kThreads,
                          smem);
}

cudaError_t rel5_batch_run_tiled_exact(const Rel5BatchArgs &args, int grid, size_t smem,
                                       cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, rel5_batch_tiled_exact_kernel, args);
}

}  // namespace pe
