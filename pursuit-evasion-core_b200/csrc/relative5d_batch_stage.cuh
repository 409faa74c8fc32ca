// Staging of the tiled batched kernels (relative5d_batch_tiled.cu,
// relative5d_batch_tiled_exact.cu): per heading of a work item, the own rows
// with a y halo and the rows of the 8 speed-neighbour planes by bulk copies
// into one of two shared-memory buffers, and the persistent stage loop.
#pragma once
#include "bulk_copy.cuh"
#include "relative5d_batch_impl.cuh"

namespace pe {
namespace {

constexpr int kThreads = kRel5BatchThreads;
constexpr int kNb = 8;  // vE-2, vE-1, vE+1, vE+2, vP-2, vP-1, vP+1, vP+2
// tries of a bounded wait for a staged heading
constexpr unsigned kStageWaitLimit = 1u << 22;

// The two heading buffers' mbarriers, and the flag a wait that gives up
// raises (set once per launch).
__shared__ uint64_t stage_bar[2];
__shared__ unsigned *stage_timeout;

// Fill state of the two heading buffers, the same in every thread of the
// CTA: bit b = number of fills of buffer b mod 2, bit 2 + b = buffer b was
// filled at least once.
struct StageRing {
  unsigned bits = 0;
  // parity of the mbarrier phase of buffer b's latest fill
  __device__ __forceinline__ unsigned parity(int b) const { return ((bits >> b) & 1u) ^ 1u; }
  __device__ __forceinline__ void filled(int b) { bits = (bits ^ (1u << b)) | (4u << b); }
  __device__ __forceinline__ bool used(int b) const { return (bits >> (2 + b)) & 1u; }
};

__device__ __forceinline__ void wait_staged(const StageRing &ring, int b) {
  for (unsigned i = 0; i < kStageWaitLimit; i++)
    if (bulk::mbar_try_wait(&stage_bar[b], ring.parity(b))) return;
  atomicOr(stage_timeout, 1u);
}

// Shared memory of one heading: own rows [R + 4][xp] then [kNb][R][xp].
__host__ __device__ inline int buffer_floats(int rows, int xp) {
  return (rows + 4) * xp + kNb * rows * xp;
}

// A thread of an item owns chunk c0 + (thread mod xc) of one of its rows.
struct ItemGeom {
  int iv, ie, y0, r_eff, R, xc;
  int c0 = 0;
};

// Stage heading `psi` of an item into buffer `buf` (called by warp 0): the
// own plane rows y0-2 .. y0+r_eff+1 inside the box (lane 8) and rows
// y0 .. y0+r_eff-1 of each speed-neighbour plane inside the grid (lane q for
// neighbour q), each a contiguous range (rows are xp floats, xp a multiple
// of 4, so every range starts and ends on 16 bytes), completing on `bar`.
// Lane 0 first posts the byte count of all of them.
__device__ __forceinline__ void stage_heading(const Rel5Grid &g, const float *__restrict__ src,
                                              const ItemGeom &it, int psi, float *buf,
                                              uint64_t *bar) {
  const int lane = threadIdx.x & 31;
  const int xp = g.xp;
  const int64_t PP = (int64_t)g.nx * xp;
  const uint32_t nb_bytes = (uint32_t)(it.r_eff * xp * 4);
  const int lo = max(0, it.y0 - 2), hi = min(g.nx, it.y0 + it.r_eff + 2);
  const uint32_t own_bytes = (uint32_t)((hi - lo) * xp * 4);
  if (lane == 0) {
    // speed neighbours inside the grid: vE-2..vE+2 and vP-2..vP+2 minus the
    // centre, cut at the ends
    const int count = min(it.ie + 2, g.nve - 1) - max(it.ie - 2, 0) +
                      min(it.iv + 2, g.nvp - 1) - max(it.iv - 2, 0);
    bulk::mbar_expect_tx(bar, own_bytes + (uint32_t)count * nb_bytes);
  }
  __syncwarp();
  if (lane < kNb) {
    const int d = (lane & 3) < 2 ? (lane & 3) - 2 : (lane & 3) - 1;  // -2, -1, +1, +2
    const int nv = it.iv + (lane < 4 ? 0 : d), ne = it.ie + (lane < 4 ? d : 0);
    if (nv >= 0 && nv < g.nvp && ne >= 0 && ne < g.nve) {
      bulk::fence_async_shared();
      bulk::bulk_load(buf + (it.R + 4 + lane * it.R) * xp,
                      src + (((int64_t)nv * g.nve + ne) * g.nh + psi) * PP + (int64_t)it.y0 * xp,
                      nb_bytes, bar);
    }
  } else if (lane == kNb) {
    bulk::fence_async_shared();
    bulk::bulk_load(buf + (lo - it.y0 + 2) * xp,
                    src + (((int64_t)it.iv * g.nve + it.ie) * g.nh + psi) * PP + (int64_t)lo * xp,
                    own_bytes, bar);
  }
}

}  // namespace
}  // namespace pe
