// Persistent, warp-specialised streaming of a relative 5D stage: work items,
// the shared-memory rings of own and speed-neighbour planes, and the producer
// that fills them by bulk asynchronous copies.  Shared by the float32 stage
// (relative5d_fast.cu, whose head comment describes the scheme) and the exact
// one (relative5d_tiled_exact.cu).
#pragma once
#include <algorithm>

#include "bulk_copy.cuh"
#include "relative5d.cuh"

namespace pe {
namespace ring {

using namespace bulk;

constexpr int OWN_SLOTS = 8;   // own-plane ring (power of two)
constexpr int STEP_SLOTS = 2;  // neighbour sets and step barriers
constexpr int NEIGHBOURS = 8;  // vE-2, vE-1, vE+1, vE+2, vP-2, vP-1, vP+1, vP+2
// a neighbour set also holds, on RK2 stage 2, the item's rows of the
// stage's old value V (the blend partner), prefetched with the neighbours
constexpr int NB_PLANES = NEIGHBOURS + 1;
constexpr int MAX_THREADS = 512;
constexpr int TARGET_THREADS = 256;  // launch bound: two CTAs of 256 per SM
constexpr int MIN_ITEM_STEPS = 4;    // own-ring reuse needs items of >= 4 headings
// A try waits for up to the hardware's own time limit before it returns
// false; a wait gives up after WAIT_LIMIT tries.  (On the 89M-cell grid a
// suspend-time hint of 1 us per try measured 0.8 % slower, and a
// %globaltimer bound in the loop 1.3 % slower.)
constexpr unsigned WAIT_LIMIT = 1u << 21;

// Bounded wait for one mbarrier phase.  Returns false (and flags the handle)
// when the limit is reached.
__device__ __forceinline__ bool wait_phase(uint64_t *bar, uint32_t parity,
                                           unsigned int *timeout_flag) {
  return bulk::wait_phase(bar, parity, timeout_flag, WAIT_LIMIT);
}

struct RingArgs {
  Rel5Grid g;
  Rel5Stage s;
  int rows, psi_chunk, slabs, chunks, xc, consumer_warps, items;
  int vp_first, vp_count;  // the vP slabs this launch updates (a shard's own)
  float ihx, ihp, ihv, ihe;
  float dt;
  bool overlap;  // launch under the previous kernel's tail (short stages)
};

// Shared memory layout of one CTA.
struct SmemLayout {
  int own_floats, nb_floats;
  int own_off, nb_off;                 // floats
  int bar_off, red_off, trig_off;      // bytes (trig_off: the kernel's own tables)
  int bytes;
};

__host__ __device__ inline SmemLayout smem_layout(int rows, int xp, int table_bytes) {
  SmemLayout L;
  L.own_floats = (rows + 4) * xp;
  L.nb_floats = rows * xp;
  L.own_off = 0;
  L.nb_off = OWN_SLOTS * L.own_floats;
  L.bar_off = 4 * (L.nb_off + STEP_SLOTS * NB_PLANES * L.nb_floats);
  L.red_off = L.bar_off + 8 * 2 * STEP_SLOTS;
  L.trig_off = L.red_off + 4 * (MAX_THREADS / 32);
  L.bytes = L.trig_off + table_bytes;
  return L;
}

// One work item: `rows` y rows (from y0) of one (vP, vE) pair over `steps`
// headings from p0.  Items are numbered heading chunk first, so that the
// CTAs resident at any moment share the planes of a few headings in L2.
struct Item {
  int iv, ie, y0, r_eff, p0, steps;
};

__device__ __forceinline__ Item decode_item(const RingArgs &a, int idx) {
  Item it;
  const int slab = idx % a.slabs;
  idx /= a.slabs;
  it.ie = idx % a.g.nve;
  idx /= a.g.nve;
  it.iv = a.vp_first + idx % a.vp_count;
  const int chunk = idx / a.vp_count;
  it.y0 = slab * a.rows;
  it.r_eff = min(a.rows, a.g.nx - it.y0);
  it.p0 = chunk * a.psi_chunk;
  it.steps = min(a.psi_chunk, a.g.nh - it.p0);
  return it;
}

// The producer: lane 0 of a CTA's last warp issues every bulk copy of the
// CTA's items in the order the consumers need them (see relative5d_fast.cu).
template <int BLEND>
__device__ __forceinline__ void produce(const RingArgs &a, const SmemLayout &L, float *own,
                                        float *nbr, uint64_t *full, uint64_t *empty, int XP) {
  const Rel5Grid &g = a.g;
  const int64_t PP = (int64_t)g.nx * XP;  // plane pitch
  unsigned int *timeout = &a.s.stats->timeout;
  bool alive = true;
  auto plane_index = [&](int v_idx, int e_idx, int psi) -> int64_t {
    return ((int64_t)(v_idx - g.slab_lo) * g.nve + e_idx) * g.nh + psi;
  };
  unsigned og = 0, gs = 0;  // own planes / steps issued so far
  for (int idx = blockIdx.x; idx < a.items && alive; idx += gridDim.x) {
    const Item it = decode_item(a, idx);
    const int row_lo = max(0, it.y0 - 2), row_hi = min(g.nx, it.y0 + it.r_eff + 2);
    const uint32_t own_bytes = (uint32_t)((row_hi - row_lo) * XP * 4);
    const float *own_src = a.s.src + (int64_t)row_lo * XP;
    const int own_dst = (row_lo - (it.y0 - 2)) * XP;
    const uint32_t nb_bytes = (uint32_t)(it.r_eff * XP * 4);
    int nb_e[NEIGHBOURS], nb_v[NEIGHBOURS], nb_count = 0;
    {
      const int de[NEIGHBOURS] = {-2, -1, 1, 2, 0, 0, 0, 0};
      const int dv[NEIGHBOURS] = {0, 0, 0, 0, -2, -1, 1, 2};
      for (int q = 0; q < NEIGHBOURS; q++) {
        nb_e[q] = it.ie + de[q];
        nb_v[q] = it.iv + dv[q];
        const bool ok = nb_e[q] >= 0 && nb_e[q] < g.nve && nb_v[q] >= 0 && nb_v[q] < g.nvp;
        if (!ok) nb_e[q] = -1;
        nb_count += ok;
      }
    }
    for (int k = 0; k < it.steps; k++) {
      const int slot = (int)(gs & 1u);
      // the slot's previous step (gs - 2) must be released first
      if (gs >= STEP_SLOTS)
        alive = wait_phase(&empty[slot], ((gs >> 1) - 1) & 1u, timeout);
      if (!alive) break;
      fence_async_shared();
      const int d_first = k == 0 ? -2 : k + 2;
      const int n_own = k + 3 - d_first;
      mbar_expect_tx(&full[slot], (uint32_t)n_own * own_bytes +
                                      nb_bytes * (nb_count + (BLEND ? 1 : 0)));
      for (int d = d_first; d <= k + 2; d++) {
        const int psi = ((it.p0 + d) % g.nh + g.nh) % g.nh;
        bulk_load(own + (og & (OWN_SLOTS - 1)) * L.own_floats + own_dst,
                  own_src + plane_index(it.iv, it.ie, psi) * PP, own_bytes, &full[slot]);
        og++;
      }
      float *set = nbr + slot * NB_PLANES * L.nb_floats;
      for (int q = 0; q < NEIGHBOURS; q++)
        if (nb_e[q] >= 0)
          bulk_load(set + q * L.nb_floats,
                    a.s.src + plane_index(nb_v[q], nb_e[q], it.p0 + k) * PP +
                        (int64_t)it.y0 * XP,
                    nb_bytes, &full[slot]);
      // the blend partner V of this step's rows: read here before any
      // consumer writes them (they wait for this set first)
      if (BLEND)
        bulk_load(set + NEIGHBOURS * L.nb_floats,
                  a.s.dst + plane_index(it.iv, it.ie, it.p0 + k) * PP +
                      (int64_t)it.y0 * XP,
                  nb_bytes, &full[slot]);
      gs++;
    }
  }
  // After a timeout, let the copies already issued (the last two steps'
  // sets at most) land before the CTA exits.
  if (!alive)
    for (unsigned q = gs > STEP_SLOTS ? gs - STEP_SLOTS : 0; q < gs; q++)
      wait_phase(&full[q & 1u], (q >> 1) & 1u, timeout);
}

// Arguments of a launch over the grid (or a shard's own vP slabs) in tiles `t`.
inline RingArgs ring_args(const Rel5Grid &g, const Rel5Tile &t, const Rel5Stage &s) {
  RingArgs args;
  args.g = g;
  args.s = s;
  args.rows = t.rows;
  args.psi_chunk = t.psi_chunk;
  args.xc = g.xp / 4;
  args.consumer_warps = (t.rows * args.xc + 31) / 32;
  args.slabs = (g.nx + t.rows - 1) / t.rows;
  args.chunks = (g.nh + t.psi_chunk - 1) / t.psi_chunk;
  args.vp_first = g.own_n > 0 ? g.own_lo : 0;
  args.vp_count = g.own_n > 0 ? g.own_n : g.nvp;
  args.items = args.slabs * g.nve * args.vp_count * args.chunks;
  args.ihx = (float)(1.0 / g.dx);
  args.ihp = (float)(1.0 / g.dphi);
  args.ihv = (float)(1.0 / g.dvp);
  args.ihe = (float)(1.0 / g.dve);
  args.dt = (float)s.dt;
  // Short stages, where launch latency counts: the 16 RK2 steps of a 17x12x7x7
  // solve take 415 us without and 342 us with it.  Long ones lose by it, since the
  // next stage's CTAs then fill the SMs unevenly as this one's leave
  // (33x24x11x11 exact 12.95 against 13.3 ms, 65x48x21x21 float32 71.7 against
  // 73.2 ms per solve).
  args.overlap = rel5_tile_cost(g, t) < 12;
  return args;
}

// Clear the step's residual before its first stage, unless the kernel does.
inline cudaError_t clear_residual(const RingArgs &a, int blend, cudaStream_t stream) {
  if (blend || (a.overlap && a.g.order == 2)) return cudaSuccess;
  return cudaMemsetAsync(&a.s.stats->residual, 0, sizeof(unsigned long long), stream);
}

}  // namespace ring
}  // namespace pe
