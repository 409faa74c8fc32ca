// The surrogate network (hidden width 256) as whole-network kernels on the
// 5th-generation tensor cores: the forward pass of all layers and the head in
// one launch, the backward pass of the activations in one, every weight
// gradient in one.
//
// Forward.  A CTA owns TPC tiles of 128 rows and takes them through all
// layers: the tile's activations stay in shared memory (K-major, 128B
// swizzle, 64 KB a tile) from one layer's epilogue to the next layer's
// tcgen05.mma (M = 128, N = 256, K = 16), whose FP32 accumulator fills 256
// tensor-memory columns; only the weights stream in (32 KB slices of 64 K
// columns, a TMA ring from L2).  Warps 0-15 run the epilogues (warp w reads
// lanes 32 (w mod 4) .. of its tile's accumulator, 64 TPC columns), warp 16
// loads weights, warp 17 issues the MMAs.  With two tiles one tile's MMAs run
// under the other's epilogue, which is the bound: SiLU takes two special
// function operations (four clocks of an SM's unit per warp) and about 9
// instructions per element; that unit is 61 % busy, issue 52 %, the tensor pipe
// 23 %, and the largest stall is the wait for accumulator reads.  Training
// (TPC = 1) also writes each layer's pre-activation and activation (below); inference
// writes the 128 outputs of a tile and can make its own input features, so
// nothing of a row but its output touches memory.
//
// Measured: 8.5 M grid nodes (41x30x13x13) 45.7 ms with a launch per layer,
// 10.7 ms with this kernel and the division of the C expression, 6.7 ms with
// the packed SiLU; a query of 1000 states 116 -> 25 us.
//
// Backward (per 128-row tile): dz of the last layer from the head, then
// dz_{l-1} = (dz_l W_l) silu'(z_{l-1}) down the layers, with the head gradients
// summed on the way.  Weight gradients: dW_l = dz_l^T prev_l over the rows,
// both operands as they lie in memory (MN-major tiles), the rows split over the
// CTAs, partial sums added with 16-byte atomics; the bias gradients are column
// sums of the same dz tiles.
//
// A training batch of 8192 rows is 64 tiles for 148 SMs and each tile a chain
// of layers, so a training pass's time is that chain: MMA, epilogue, MMA, ..
// Two CTAs of a cluster share a tile: each takes 128 columns of every layer
// and writes its half of the next operand into both CTAs' shared memory.  The
// epilogue hands the tile to the next MMAs before it writes z, h or dz to
// memory, in whole rows (z by TMA from a staged block per warp, and one layer
// ahead by TMA in the backward pass): with a row per lane and before the
// hand-over those stores were 6,000 of a layer's 16,000 clocks.  A step at 8192
// rows, launch per layer, then one CTA per tile, then this: forward 145, 43,
// 34 us; backward with all gradients 400, 66, 40 us.
//
// Every mbarrier wait is bounded; a wait that gives up sets the error flag
// of pe_mlp_gemm_tc_timeouts and the CTA still releases its tensor memory.  The
// outputs of the rows that it concerns are NaN, and the loss with them.
#include "mlp_features.cuh"
#include "mlp_tc.cuh"

#include <algorithm>
#include <cfloat>

namespace pe {
namespace {

using namespace tc;

constexpr int H = 256;          // hidden width
constexpr int MAX_LAYERS = 8;
constexpr int EW = 16;          // epilogue warps
constexpr int THREADS = 32 * (EW + 2);
constexpr int A_CHUNK = TM * 128;   // 64 K columns of a 128-row tile, bytes
constexpr int A_TILE = 4 * A_CHUNK;
constexpr int W_SLICE = H * 128;    // 64 K columns of 256 weight rows, bytes

enum Input { FEATURES = 0, RELATIVE_NODES = 1, RELATIVE_STATES = 2, WORLD_NODES = 3 };

struct ForwardArgs {
  CUtensorMap w[MAX_LAYERS], feat, zmap[MAX_LAYERS];
  int layers, rows, groups;
  const float *bias[MAX_LAYERS], *w_out, *b_out;
  float *z[MAX_LAYERS];          // training: pre-activations [rows][256]
  __nv_bfloat16 *h[MAX_LAYERS];  // training: activations [rows][256]
  const float *target;           // training: labels (with dy, loss)
  float *y, *dy, *loss;
  float inv_rows;
  NodeGrid grid;                 // RELATIVE_NODES, WORLD_NODES
  int64_t first;                 // ... index of row 0's node
  const float *states;           // RELATIVE_STATES [rows][5]
  unsigned *error;
};

struct BackwardArgs {
  CUtensorMap wt[MAX_LAYERS];  // transposed weights [in][out]
  CUtensorMap zmap[MAX_LAYERS];
  int layers;
  const float *dy, *w_out;
  const __nv_bfloat16 *h_last;
  __nv_bfloat16 *dz[MAX_LAYERS];
  float *gw_out, *gb_out;
  unsigned *error;
};

struct WeightGradArgs {
  CUtensorMap dz[MAX_LAYERS], prev[MAX_LAYERS];
  float *gw[MAX_LAYERS], *gb[MAX_LAYERS];
  int width0;  // input columns of layer 0 (128 or 256)
  int ksteps;  // 64-row steps over all rows
  unsigned *error;
};

__device__ __forceinline__ void mma256(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

// BF16 x BF16 -> FP32, M = 128; MN: both operands MN-major.
__host__ __device__ constexpr uint32_t instr_desc(int n, bool mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (1u << 15) | (1u << 16) : 0u) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// --- a cluster of two CTAs on one tile (CL = 2): each takes 128 of the 256
// columns of every layer and writes its half of the next operand into both
// CTAs' shared memory.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_addr(const void *p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// bounded wait that also acquires what the peer CTA released
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity,
                                                  unsigned *error) {
  for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  atomicOr(error, 1u);
  return false;
}
template <int CL>
__device__ __forceinline__ bool tile_wait(uint64_t *bar, uint32_t parity, unsigned *error) {
  return CL == 2 ? mbar_wait_cluster(bar, parity, error) : mbar_wait(bar, parity, error);
}
// the same by a whole warp, one answer for all lanes (the warp-wide operations
// that follow need them together also after a wait that gave up)
template <int CL>
__device__ __forceinline__ bool tile_wait_warp(uint64_t *bar, uint32_t parity, unsigned *error) {
  return __all_sync(0xffffffffu, tile_wait<CL>(bar, parity, error)) != 0;
}
// A warp's part of the tile is written: the tensor core (async proxy) of every
// CTA of the cluster may read it.
template <int CL>
__device__ __forceinline__ void tile_arrive(uint64_t *bar, uint32_t rank) {
  if (CL == 1) {
    fence_async_shared();
    mbar_arrive(bar);
    return;
  }
  asm volatile("fence.proxy.async.shared::cluster;" ::: "memory");
  __syncwarp();
  if ((threadIdx.x & 31) < CL)
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(
                     peer_addr(bar, threadIdx.x & 31))
                 : "memory");
}
// arrivals per phase of a tile barrier that `warps` warps a CTA complete
template <int CL>
__host__ __device__ constexpr int tile_arrivals(int warps) { return CL == 1 ? 32 * warps : CL * warps; }
// the issued MMAs are done reading the tile, told to every CTA that writes it
template <int CL>
__device__ __forceinline__ void acc_commit(uint64_t *bar) {
  if (CL == 1)
    mma_commit(bar);
  else
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster"
        ".b64 [%0], %1;" ::"r"(smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t r[32], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, "
      "%10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, "
      "%27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 two(float a) { return make_float2(a, a); }

// -(1 + exp(-z)) of a pair, finite.  Its approximate reciprocal is 0 beyond
// 2^126 (z < -87.34, where SiLU is above -1.03e-36), and with it SiLU and its
// derivative, however large -z is.
__device__ __forceinline__ float2 neg_denominator(float2 z) {
  const float2 x = __fmul2_rn(z, two(-1.44269504f));
  const float2 nd = __ffma2_rn(make_float2(ex2(x.x), ex2(x.y)), two(-1.f), two(-1.f));
  return make_float2(max_nan(nd.x, -FLT_MAX), max_nan(nd.y, -FLT_MAX));
}
// 1 / -nd by the approximate reciprocal and one Newton step
__device__ __forceinline__ float2 reciprocal(float2 nd) {
  const float2 r = make_float2(rcp(-nd.x), rcp(-nd.y));
  return __ffma2_rn(r, __ffma2_rn(nd, r, two(1.f)), r);
}
// silu of a pair, in packed FP32: z / (1 + exp(-z)) with the quotient from the
// reciprocal and one FMA correction (P. Markstein, "IA-64 and Elementary
// Functions", 2000), free of the division's branches: 9 instead of 21
// instructions per element.  An infinite z takes the largest float (its bf16
// is infinite again), NaN stays NaN.
__device__ __forceinline__ float2 silu2(float2 z) {
  z = make_float2(min_nan(z.x, 0x1.fffffep127f), min_nan(z.y, 0x1.fffffep127f));
  const float2 nd = neg_denominator(z), r = reciprocal(nd);
  const float2 q = __fmul2_rn(z, r);
  return __ffma2_rn(__ffma2_rn(nd, q, z), r, q);
}
// silu'(z) = s (1 + z (1 - s)), s = 1 / (1 + exp(-z))
__device__ __forceinline__ float2 silu_grad2(float2 z) {
  const float2 nd = neg_denominator(z), r = reciprocal(nd);
  const float2 s = __ffma2_rn(__ffma2_rn(nd, r, two(1.f)), r, r);
  const float2 t = __ffma2_rn(s, two(-1.f), two(1.f));
  return __fmul2_rn(s, __ffma2_rn(z, t, two(1.f)));
}

// 32-byte global accesses: a thread's row segment fills whole sectors.
__device__ __forceinline__ void st_global32(void *p, const uint32_t v[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&p);
}
__device__ __forceinline__ float lo16(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi16(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// Byte offset of 16-byte unit `u` (0..31 over the 256 columns) of row r in a
// swizzled 128 x 256 tile of four 64-column chunks.
__device__ __forceinline__ int unit_off(int r, int u) {
  return (u >> 3) * A_CHUNK + r * 128 + (((u & 7) ^ (r & 7)) << 4);
}

// 32 columns (c0 ..) of row r, packed bf16 pairs, into the swizzled tile.
__device__ __forceinline__ void store_tile32(uint8_t *tile, int r, int c0, const uint32_t p[16]) {
#pragma unroll
  for (int k = 0; k < 4; k++)
    *reinterpret_cast<uint4 *>(tile + unit_off(r, c0 / 8 + k)) =
        make_uint4(p[4 * k], p[4 * k + 1], p[4 * k + 2], p[4 * k + 3]);
}
// the same into the peer's tile
__device__ __forceinline__ void store_peer32(uint32_t tile, int r, int c0, const uint32_t p[16]) {
#pragma unroll
  for (int k = 0; k < 4; k++)
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                     tile + unit_off(r, c0 / 8 + k)),
                 "r"(p[4 * k]), "r"(p[4 * k + 1]), "r"(p[4 * k + 2]), "r"(p[4 * k + 3])
                 : "memory");
}

// 32 columns from c0 of 32 rows from r0 of the tile to a [rows][256] array,
// four lanes a row (whole sectors; a lane a row took 62 clocks an instruction)
__device__ __forceinline__ void write_out32(__nv_bfloat16 *out, int64_t row0, const uint8_t *tile,
                                            int r0, int c0, int lane) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = r0 + 8 * i + lane / 4, u = c0 / 8 + lane % 4;
    *reinterpret_cast<uint4 *>(out + (row0 + r) * H + 8 * u) =
        *reinterpret_cast<const uint4 *>(tile + unit_off(r, u));
  }
}
// A warp's 32 x 32 block of z in shared memory: the 128B-swizzled box of zmap.
constexpr int Z_BLOCK = 32 * 32 * 4;
__device__ __forceinline__ int z_unit(int r, int u) { return r * 128 + ((u ^ (r & 7)) << 4); }
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, int x, int y,
                                             const void *src) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(x), "r"(y), "r"(smem_u32(src))
      : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

template <int TPC, int CL>
struct ForwardLayout {
  static constexpr int STAGES = TPC == 2 ? 2 : 4;
  static constexpr int W = TPC * A_TILE;
  static constexpr int Z = W + STAGES * W_SLICE / CL;  // (CL = 2) a block per warp
  static constexpr int BIAS = Z + (CL == 2 ? EW * Z_BLOCK : 0);  // [layers][256], then w_out
  static constexpr int BARS = BIAS + (MAX_LAYERS + 1) * H * 4;
  static constexpr int BYTES = BARS + 8 * (2 * STAGES + 3 * TPC) + 16;
};

template <int TPC, int INPUT, bool TRAIN, int CL>
__global__ void __launch_bounds__(THREADS, 1)
    forward_kernel(const __grid_constant__ ForwardArgs g) {
  using L = ForwardLayout<TPC, CL>;
  static_assert(CL == 1 || (TPC == 1 && TRAIN && INPUT == FEATURES), "");
  constexpr int WPT = EW / TPC;        // epilogue warps of a tile
  constexpr int N = H / CL;            // columns of this CTA
  constexpr int COLS = N * 4 / WPT;    // columns of one warp
  constexpr int SLICE = W_SLICE / CL;
  constexpr int S = L::STAGES;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sA = base, *sW = base + L::W;
  float *bias = reinterpret_cast<float *>(base + L::BIAS);
  float *wout = bias + MAX_LAYERS * H;
  uint64_t *w_full = reinterpret_cast<uint64_t *>(base + L::BARS);
  uint64_t *w_empty = w_full + S, *a_ready = w_empty + S, *acc_full = a_ready + TPC;
  uint64_t *f_full = acc_full + TPC;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(f_full + TPC);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = CL == 1 ? 0 : cluster_rank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
    }
    for (int t = 0; t < TPC; t++) {
      mbar_init(&a_ready[t], tile_arrivals<CL>(WPT));
      mbar_init(&acc_full[t], CL);
      mbar_init(&f_full[t], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == EW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TPC * N)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = threadIdx.x; i < g.layers * H; i += THREADS)
    bias[i] = g.bias[i / H][i % H];
  for (int i = threadIdx.x; i < H; i += THREADS) wout[i] = g.w_out[i];
  fence_before();
  __syncthreads();
  if (CL == 2) cluster_sync();  // the peer's barriers are initialised
  fence_after();
  const uint32_t tmem = *tmem_slot;

  // weight slices of layer l: the features fill K = 16 of one slice when made
  // here, 128 columns (two slices) when read
  auto slices = [&](int l) { return l > 0 ? 4 : INPUT == FEATURES ? 2 : 1; };

  if (warp == EW) {  // ---- loader
    if (lane == 0) {
      bool ok = true;
      unsigned n = 0;  // slices issued
      for (int grp = blockIdx.x / CL; grp < g.groups && ok; grp += gridDim.x / CL) {
        if (INPUT == FEATURES)
          for (int t = 0; t < TPC; t++) {
            mbar_expect_tx(&f_full[t], 2 * A_CHUNK);
            for (int k = 0; k < 2; k++)
              tma_load_2d(sA + t * A_TILE + k * A_CHUNK, &g.feat, k * TK,
                          (grp * TPC + t) * TM, &f_full[t]);
          }
        for (int l = 0; l < g.layers && ok; l++)
          for (int t = 0; t < TPC && ok; t++)
            for (int k = 0; k < slices(l); k++) {
              const int s = n % S;
              if (n >= S) ok = mbar_wait(&w_empty[s], ((n / S) - 1) & 1, g.error);
              if (!ok) break;
              mbar_expect_tx(&w_full[s], SLICE);
              tma_load_2d(sW + s * SLICE, &g.w[l], k * TK, (int)rank * N, &w_full[s]);
              n++;
            }
      }
      // no copy may still be landing when the CTA leaves
      for (unsigned k = n > S ? n - S : 0; k < n; k++)
        mbar_wait(&w_full[k % S], (k / S) & 1, g.error);
      if (INPUT == FEATURES)
        for (int t = 0; t < TPC; t++) mbar_wait(&f_full[t], 0, g.error);
    }
  } else if (warp == EW + 1) {  // ---- MMA issuer
    if (lane == 0) {
      constexpr uint32_t ID = instr_desc(N, false);
      bool ok = true;
      unsigned n = 0, pass = 0;
      for (int grp = blockIdx.x / CL; grp < g.groups && ok; grp += gridDim.x / CL)
        for (int l = 0; l < g.layers && ok; l++, pass++)
          for (int t = 0; t < TPC && ok; t++) {
            ok = tile_wait<CL>(&a_ready[t], pass & 1, g.error);
            if (CL == 2) asm volatile("fence.proxy.async.shared::cluster;" ::: "memory");
            if (ok && INPUT == FEATURES && l == 0) ok = mbar_wait(&f_full[t], 0, g.error);
            for (int k = 0; k < slices(l) && ok; k++, n++) {
              const int s = n % S;
              ok = mbar_wait(&w_full[s], (n / S) & 1, g.error);
              if (!ok) break;
              fence_after();
              const uint32_t a0 = smem_u32(sA + t * A_TILE + k * A_CHUNK);
              const uint32_t b0 = smem_u32(sW + s * SLICE);
              const int steps = INPUT != FEATURES && l == 0 ? 1 : TK / 16;
              for (int kk = 0; kk < steps; kk++)
                mma256(tmem + t * N, smem_desc_sw128(a0 + kk * 32),
                       smem_desc_sw128(b0 + kk * 32), ID, (k | kk) != 0);
              mma_commit(&w_empty[s]);
            }
            acc_commit<CL>(&acc_full[t]);  // (also after a wait that gave up)
          }
    }
  } else {  // ---- epilogues
    const int t = warp / WPT, part = (warp % WPT) / 4, quarter = warp & 3;
    const int r = quarter * 32 + lane;   // row in the tile
    const int col0 = (int)rank * N + part * COLS;
    uint8_t *tile = sA + t * A_TILE;
    const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + t * N + part * COLS;
    const uint32_t peer = CL == 1 ? 0 : peer_addr(tile, rank ^ 1);
    uint8_t *zblock = base + L::Z + warp * Z_BLOCK;  // (CL = 2)
    bool ok = true;  // after a wait that gave up every warp still meets every barrier
    unsigned pass = 0;
    float sq = 0.f;
    for (int grp = blockIdx.x / CL; grp < g.groups; grp += gridDim.x / CL) {
      const int64_t row = (int64_t)(grp * TPC + t) * TM + r;
      if (INPUT != FEATURES && part == 0) {
        float v[kMaxFeatures] = {};
        if (row < g.rows) {
          if (INPUT == RELATIVE_NODES) relative_node_features(v, g.grid, g.first + row);
          if (INPUT == WORLD_NODES) world_node_features(v, g.grid, g.first + row);
          if (INPUT == RELATIVE_STATES) {
            const float *s = g.states + row * 5;
            state_features(v, g.grid.f, s[0], s[1], s[2], s[3], s[4]);
          }
        }
        *reinterpret_cast<uint4 *>(tile + unit_off(r, 0)) = pack_features(v);
        *reinterpret_cast<uint4 *>(tile + unit_off(r, 1)) = pack_features(v + 8);
      }
      tile_arrive<CL>(&a_ready[t], rank);
      for (int l = 0; l < g.layers; l++, pass++) {
        // (one answer per warp for the warp-wide hand-over of a training pass;
        // inference has none and does without the vote, 6.70 against 6.87 ms for
        // 8.5 M nodes)
        if (ok)
          ok = TRAIN ? tile_wait_warp<CL>(&acc_full[t], pass & 1, g.error)
                     : mbar_wait(&acc_full[t], pass & 1, g.error);
        if (!ok) continue;
        fence_after();
        const bool last = l == g.layers - 1;
        const float *bl = bias + l * H + col0;
#pragma unroll 1
        for (int c0 = 0; c0 < COLS; c0 += 32) {
          uint32_t a[32], p[16];
          tmem_ld32(a, acc + c0);
          tmem_wait();
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            const float4 b = *reinterpret_cast<const float4 *>(bl + c0 + k);
            const float2 z0 = __fadd2_rn(
                make_float2(__uint_as_float(a[k]), __uint_as_float(a[k + 1])),
                make_float2(b.x, b.y));
            const float2 z1 = __fadd2_rn(
                make_float2(__uint_as_float(a[k + 2]), __uint_as_float(a[k + 3])),
                make_float2(b.z, b.w));
            const float2 h0 = silu2(z0), h1 = silu2(z1);
            p[k / 2] = pack2(h0.x, h0.y);
            p[k / 2 + 1] = pack2(h1.x, h1.y);
            if (TRAIN) {
              a[k] = __float_as_uint(z0.x);
              a[k + 1] = __float_as_uint(z0.y);
              a[k + 2] = __float_as_uint(z1.x);
              a[k + 3] = __float_as_uint(z1.y);
            }
          }
          if (TRAIN && CL == 1) {
            if (g.z[l])
              for (int k = 0; k < 4; k++) st_global32(g.z[l] + row * H + col0 + c0 + 8 * k, a + 8 * k);
            for (int k = 0; k < 2; k++)
              st_global32(g.h[l] + row * H + col0 + c0 + 16 * k, p + 8 * k);
          }
          store_tile32(tile, r, col0 + c0, p);
          if (CL == 2) {
            // the next layer starts on the tile first; z and h leave under it
            store_peer32(peer, r, col0, p);
            fence_before();
            tile_arrive<CL>(&a_ready[t], rank);
            if (g.z[l]) {
              if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              __syncwarp();
#pragma unroll
              for (int u = 0; u < 8; u++)
                *reinterpret_cast<uint4 *>(zblock + z_unit(lane, u)) =
                    make_uint4(a[4 * u], a[4 * u + 1], a[4 * u + 2], a[4 * u + 3]);
              fence_async_shared();
              __syncwarp();
              if (lane == 0) tma_store_2d(&g.zmap[l], col0, (int)row - lane, zblock);
            }
            write_out32(g.h[l], row - r, tile, quarter * 32, col0, lane);
          }
        }
        if (CL == 1) {
          fence_before();
          if (!last) tile_arrive<CL>(&a_ready[t], rank);
        }
      }
      // the head, a warp per row: lane l sums columns l, l + 32, ..; a cluster's
      // CTAs take half of the rows each, once both halves of the columns are in
      if (CL == 2 && ok) ok = tile_wait_warp<CL>(&a_ready[t], pass & 1, g.error);
      // columns of the tile are not there: every output of the CTA becomes NaN
      if (!ok) wout[lane] = __int_as_float(0x7fc00000);
      asm volatile("bar.sync %0, %1;" ::"r"(1 + t), "n"(32 * WPT) : "memory");
      float w[H / 32];
#pragma unroll
      for (int i = 0; i < H / 32; i++) w[i] = wout[lane + 32 * i];
      const float b_out = g.b_out[0];
#pragma unroll 4
      for (int q = 0; q < TM / CL / WPT; q++) {
        const int rr = (int)rank * (TM / CL) + (warp % WPT) * (TM / CL / WPT) + q;
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < H / 32; i++) {
          const uint16_t hv = *reinterpret_cast<const uint16_t *>(
              tile + unit_off(rr, lane / 8 + 4 * i) + (lane & 7) * 2);
          sum = fmaf(__uint_as_float((uint32_t)hv << 16), w[i], sum);
        }
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        const int64_t out_row = (int64_t)(grp * TPC + t) * TM + rr;
        if (lane == 0 && out_row < g.rows) {
          const float out = sum + b_out;
          g.y[out_row] = out;
          if (TRAIN && g.target) {
            const float e = out - g.target[out_row];
            g.dy[out_row] = 2.f * e * g.inv_rows;
            sq += e * e * g.inv_rows;
          }
        }
      }
      // every row has been read: the next group may overwrite the tile
      asm volatile("bar.sync %0, %1;" ::"r"(1 + t), "n"(32 * WPT) : "memory");
    }
    if (TRAIN && g.target && lane == 0) atomicAdd(g.loss, sq);
    if (CL == 2 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (CL == 2) cluster_sync();  // the peer is done with this shared memory
  if (warp == EW + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TPC * N)
                 : "memory");
}

// ------------------------------------------------------------- backward
constexpr int BCL = 2;  // CTAs per tile, always
struct BackwardLayout {
  static constexpr int STAGES = 4;
  static constexpr int W = A_TILE;
  static constexpr int Z = W + STAGES * W_SLICE / BCL;  // a block per warp
  static constexpr int WOUT = Z + EW * Z_BLOCK;
  static constexpr int DY = WOUT + H * 4;
  static constexpr int RED = DY + TM * 4;  // [8 ranges][128] partial column sums
  static constexpr int BARS = RED + 4 * H * 4;
  static constexpr int BYTES = BARS + 8 * (2 * STAGES + 2 + EW) + 16;
};

__global__ void __launch_bounds__(THREADS, 1)
    backward_kernel(const __grid_constant__ BackwardArgs g) {
  using L = BackwardLayout;
  constexpr int CL = BCL;
  constexpr int S = L::STAGES;
  constexpr int N = H / CL;     // columns of this CTA
  constexpr int COLS = N / 4;   // columns of one epilogue warp
  static_assert(COLS == 32, "a warp takes one 32 x 32 block");
  constexpr int SLICE = W_SLICE / CL;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *tile = base, *sW = base + L::W;
  float *wout = reinterpret_cast<float *>(base + L::WOUT);
  float *dys = reinterpret_cast<float *>(base + L::DY);
  float *red = reinterpret_cast<float *>(base + L::RED);
  uint64_t *w_full = reinterpret_cast<uint64_t *>(base + L::BARS);
  uint64_t *w_empty = w_full + S, *a_ready = w_empty + S, *acc_full = a_ready + 1;
  uint64_t *z_full = acc_full + 1;  // one per epilogue warp
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(z_full + EW);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int64_t row0 = (int64_t)(blockIdx.x / CL) * TM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
    }
    mbar_init(a_ready, tile_arrivals<CL>(EW));
    mbar_init(acc_full, CL);
    for (int w = 0; w < EW; w++) mbar_init(&z_full[w], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == EW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(N)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = threadIdx.x; i < H; i += THREADS) wout[i] = g.w_out[i];
  for (int i = threadIdx.x; i < TM; i += THREADS) dys[i] = g.dy[row0 + i];
  fence_before();
  __syncthreads();
  cluster_sync();  // the peer's barriers are initialised
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == EW) {
    if (lane == 0) {
      bool ok = true;
      unsigned n = 0;
      for (int l = g.layers - 1; l > 0 && ok; l--)
        for (int k = 0; k < 4; k++, n++) {
          const int s = n % S;
          if (n >= S) ok = mbar_wait(&w_empty[s], ((n / S) - 1) & 1, g.error);
          if (!ok) break;
          mbar_expect_tx(&w_full[s], SLICE);
          tma_load_2d(sW + s * SLICE, &g.wt[l], k * TK, (int)rank * N, &w_full[s]);
        }
      for (unsigned k = n > S ? n - S : 0; k < n; k++)
        mbar_wait(&w_full[k % S], (k / S) & 1, g.error);
    }
  } else if (warp == EW + 1) {
    if (lane == 0) {
      constexpr uint32_t ID = instr_desc(N, false);
      bool ok = true;
      unsigned n = 0, pass = 0;
      for (int l = g.layers - 1; l > 0 && ok; l--, pass++) {
        ok = tile_wait<CL>(a_ready, pass & 1, g.error);
        asm volatile("fence.proxy.async.shared::cluster;" ::: "memory");
        for (int k = 0; k < 4 && ok; k++, n++) {
          const int s = n % S;
          ok = mbar_wait(&w_full[s], (n / S) & 1, g.error);
          if (!ok) break;
          fence_after();
          const uint32_t a0 = smem_u32(tile + k * A_CHUNK);
          const uint32_t b0 = smem_u32(sW + s * SLICE);
          for (int kk = 0; kk < TK / 16; kk++)
            mma256(tmem, smem_desc_sw128(a0 + kk * 32), smem_desc_sw128(b0 + kk * 32), ID,
                   (k | kk) != 0);
          mma_commit(&w_empty[s]);
        }
        acc_commit<CL>(acc_full);
      }
    }
  } else {
    const int part = warp / 4, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int col0 = (int)rank * N + part * COLS;
    const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + part * COLS;
    const uint32_t peer = peer_addr(tile, rank ^ 1);
    const float d = dys[r];
    // Column pair and row range of the head's sums: this CTA's 64 pairs x 8
    // ranges of 16 rows.
    constexpr int ROWS = 32 / CL;
    const int pair = (int)rank * (N / 2) + threadIdx.x % (N / 2), range = threadIdx.x / (N / 2);
    bool ok = true;
    unsigned pass = 0;
    // column sums over the tile: the ranges in shared memory first, so that a
    // CTA adds one partial sum per column
    auto add_columns = [&](float *out, float v0, float v1) {
      const int c = 2 * (threadIdx.x % (N / 2));
      *reinterpret_cast<float2 *>(red + range * N + c) = make_float2(v0, v1);
      asm volatile("bar.sync 1, %0;" ::"n"(32 * EW) : "memory");
      if (threadIdx.x >= N || !ok) return;
      float part[4 * CL];
#pragma unroll
      for (int i = 0; i < 4 * CL; i++) part[i] = red[i * N + threadIdx.x];
#pragma unroll
      for (int w = 2 * CL; w > 0; w /= 2)
#pragma unroll
        for (int i = 0; i < w; i++) part[i] += part[i + w];
      atomicAdd(out + (int)rank * N + threadIdx.x, part[0]);
    };
    // z of the next layer down arrives while this one is worked on
    uint8_t *zblock = base + L::Z + warp * Z_BLOCK;
    auto load_z = [&](int l) {
      if (lane != 0) return;
      fence_async_shared();  // the block's reads come before the copy
      mbar_expect_tx(&z_full[warp], Z_BLOCK);
      tma_load_2d(zblock, &g.zmap[l], col0, (int)row0 + quarter * 32, &z_full[warp]);
    };
    bool z_asked = true;
    load_z(g.layers - 1);
    for (int l = g.layers - 1; l >= 0; l--) {
      const bool head = l == g.layers - 1;
      uint32_t zr[32];
      // (a copy is asked for only while no wait has given up, and always
      // waited for: none is in flight when the CTA leaves)
      if (z_asked) ok = tile_wait_warp<1>(&z_full[warp], (g.layers - 1 - l) & 1, g.error) && ok;
#pragma unroll
      for (int u = 0; u < 8; u++)
        *reinterpret_cast<uint4 *>(zr + 4 * u) =
            *reinterpret_cast<const uint4 *>(zblock + z_unit(lane, u));
      __syncwarp();
      z_asked = ok && l > 0;
      if (z_asked) load_z(l - 1);
      if (!head) {
        if (ok) ok = tile_wait_warp<CL>(acc_full, pass & 1, g.error);
        pass++;
        fence_after();
      }
      uint32_t a[32], p[16];
      if (!head) {
        tmem_ld32(a, acc);
        tmem_wait();
      }
#pragma unroll
      for (int k = 0; k < 32; k += 2) {
        const float u0 = head ? d * wout[col0 + k] : __uint_as_float(a[k]);
        const float u1 = head ? d * wout[col0 + k + 1] : __uint_as_float(a[k + 1]);
        const float2 sg = silu_grad2(
            make_float2(__uint_as_float(zr[k]), __uint_as_float(zr[k + 1])));
        p[k / 2] = pack2(u0 * sg.x, u1 * sg.y);
      }
      store_tile32(tile, r, col0, p);
      if (l > 0) store_peer32(peer, r, col0, p);
      fence_before();
      if (l > 0) tile_arrive<CL>(a_ready, rank);
      __syncwarp();
      write_out32(g.dz[l], row0, tile, quarter * 32, col0, lane);
      if (head) {  // head gradients: dw_out = sum_r dy_r h_r, db_out = sum_r dy_r
        float w0 = 0.f, w1 = 0.f, sd = 0.f;
        const uint32_t *hp =
            reinterpret_cast<const uint32_t *>(g.h_last + (row0 + range * ROWS) * H) + pair;
#pragma unroll 8
        for (int q = 0; q < ROWS; q++) {
          const uint32_t v = hp[q * (H / 2)];
          const float dr = dys[range * ROWS + q];
          w0 = fmaf(dr, lo16(v), w0);
          w1 = fmaf(dr, hi16(v), w1);
          sd += dr;
        }
        add_columns(g.gw_out, w0, w1);
        if (pair == 0) atomicAdd(g.gb_out, sd);
      }
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  cluster_sync();  // the peer is done with this shared memory
  if (warp == EW + 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(N)
                 : "memory");
}

// ------------------------------------------------------ weight gradients
// One CTA: 128 rows (out) x N columns (in) of one layer's gradient over its
// share of the batch rows.  Both operands lie [row][column], so a TMA box of
// 64 columns x 64 rows is an MN-major tile: 128-byte rows, consecutive K rows
// 128 bytes apart (8-row groups 1024), 64-column blocks 8 KB apart.
constexpr int G_STAGES = 4;
constexpr int G_BLOCK = 64 * 128;            // one 64 x 64 box
constexpr int G_STAGE = (2 + 4) * G_BLOCK;   // A: 128 columns, B: up to 256
constexpr int G_WARPS = 8;
constexpr int G_THREADS = 32 * (G_WARPS + 2);
constexpr int G_BYTES = 1024 + G_STAGES * G_STAGE + 8 * (2 * G_STAGES + 1) + 16;

__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(G_BLOCK >> 4) << 16;  // leading: next 64-column block
  d |= (uint64_t)(1024 >> 4) << 32;     // stride: next 8 K rows
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;               // 128-byte swizzle
  return d;
}

__global__ void __launch_bounds__(G_THREADS, 1)
    weight_grad_kernel(const __grid_constant__ WeightGradArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *base = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(base + G_STAGES * G_STAGE);
  uint64_t *empty = full + G_STAGES, *done = empty + G_STAGES;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = blockIdx.x >> 1, m0 = (blockIdx.x & 1) * TM;
  const int N = l == 0 ? g.width0 : H;
  const int k0 = (int)((int64_t)g.ksteps * blockIdx.y / gridDim.y);
  const int k1 = (int)((int64_t)g.ksteps * (blockIdx.y + 1) / gridDim.y);

  if (threadIdx.x == 0) {
    for (int s = 0; s < G_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1 + G_WARPS);  // the MMAs, and each summing warp
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(2 * H)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == G_WARPS) {
    if (lane == 0) {
      bool ok = true;
      int n = 0;
      for (int k = k0; k < k1; k++, n++) {
        const int s = n % G_STAGES;
        if (n >= G_STAGES) ok = mbar_wait(&empty[s], ((n / G_STAGES) - 1) & 1, g.error);
        if (!ok) break;
        uint8_t *st = base + s * G_STAGE;
        mbar_expect_tx(&full[s], (2 + N / 64) * G_BLOCK);
        for (int b = 0; b < 2; b++)
          tma_load_2d(st + b * G_BLOCK, &g.dz[l], m0 + 64 * b, k * 64, &full[s]);
        for (int b = 0; b < N / 64; b++)
          tma_load_2d(st + (2 + b) * G_BLOCK, &g.prev[l], 64 * b, k * 64, &full[s]);
      }
      for (int k = n > G_STAGES ? n - G_STAGES : 0; k < n; k++)
        mbar_wait(&full[k % G_STAGES], (k / G_STAGES) & 1, g.error);
    }
  } else if (warp == G_WARPS + 1) {
    if (lane == 0) {
      const uint32_t ID = instr_desc(N, true);
      // the two halves of the rows in two accumulators: their sum rounds less
      // than one chain over all rows
      const int half = (k1 - k0 + 1) / 2;
      bool ok = true;
      for (int n = 0; n < k1 - k0 && ok; n++) {
        const int s = n % G_STAGES;
        ok = mbar_wait(&full[s], (n / G_STAGES) & 1, g.error);
        if (!ok) break;
        fence_after();
        const uint32_t a0 = smem_u32(base + s * G_STAGE), b0 = a0 + 2 * G_BLOCK;
        const int second = n >= half;
        for (int kk = 0; kk < 4; kk++)  // K = 16 rows per instruction: two 8-row groups
          mma256(tmem + second * H, smem_desc_mn(a0 + kk * 2048), smem_desc_mn(b0 + kk * 2048),
                 ID, ((n - second * half) | kk) != 0);
        mma_commit(&empty[s]);
      }
      mma_commit(done);
    }
  } else {
    // Bias gradients: the column sums of the dz tiles while the MMAs read them
    // (64 column pairs x 4 groups of 16 rows a stage).  Here a column takes
    // one partial sum per row split (18 at 8192 rows), against one per 128-row
    // tile where dz is made, and off that kernel's chain of layers.
    const int pair = threadIdx.x & 63, group = threadIdx.x >> 6;
    float s0 = 0.f, s1 = 0.f;
    bool summed = true;
    for (int n = 0; n < k1 - k0; n++) {
      const int s = n % G_STAGES;
      summed = tile_wait_warp<1>(&full[s], (n / G_STAGES) & 1, g.error);
      if (!summed) break;
      const uint8_t *block = base + s * G_STAGE + (pair >> 5) * G_BLOCK + (pair & 3) * 4;
      float t0 = 0.f, t1 = 0.f;
#pragma unroll
      for (int q = 0; q < 16; q++) {
        const int r = group * 16 + q, u = (pair & 31) >> 2;
        const uint32_t v =
            *reinterpret_cast<const uint32_t *>(block + r * 128 + ((u ^ (r & 7)) << 4));
        t0 += lo16(v);
        t1 += hi16(v);
      }
      s0 += t0;
      s1 += t1;
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    const bool ok = mbar_wait(done, 0, g.error) && k1 > k0;
    fence_after();
    // every warp is done with the ring: its space is free for what follows
    float *sums = reinterpret_cast<float *>(base + 2 * G_STAGE);  // [4][128]
    asm volatile("bar.sync 1, %0;" ::"n"(32 * G_WARPS) : "memory");
    *reinterpret_cast<float2 *>(sums + group * TM + 2 * pair) = make_float2(s0, s1);
    asm volatile("bar.sync 1, %0;" ::"n"(32 * G_WARPS) : "memory");
    if (threadIdx.x < TM && ok && summed)
      atomicAdd(g.gb[l] + m0 + threadIdx.x,
                (sums[threadIdx.x] + sums[TM + threadIdx.x]) +
                    (sums[2 * TM + threadIdx.x] + sums[3 * TM + threadIdx.x]));
    // warp w: accumulator lanes 32 (w mod 4) .., columns of half w / 4; each
    // 32 x 32 block is turned around in shared memory (the ring is idle now)
    // so that 8 lanes add 128 contiguous bytes of one row
    float *stage = reinterpret_cast<float *>(base) + warp * 32 * 33;
    const int quarter = warp & 3, half = warp >> 2;
    const bool two = k1 - k0 > 1;
#pragma unroll 1
    for (int c0 = half * (N / 2); c0 < (half + 1) * (N / 2); c0 += 32) {
      uint32_t a[32], b[32];
      tmem_ld32(a, tmem + ((uint32_t)(quarter * 32) << 16) + c0);
      tmem_ld32(b, tmem + ((uint32_t)(quarter * 32) << 16) + H + c0);
      tmem_wait();
#pragma unroll
      for (int j = 0; j < 32; j++)
        stage[lane * 33 + j] = __uint_as_float(a[j]) + (two ? __uint_as_float(b[j]) : 0.f);
      __syncwarp();
      if (ok) {
        const int rs = lane >> 3, cq = (lane & 7) * 4;
#pragma unroll
        for (int rr = 0; rr < 32; rr += 4) {
          const float *src = stage + (rr + rs) * 33 + cq;
          float *dst = g.gw[l] + (size_t)(m0 + quarter * 32 + rr + rs) * N + c0 + cq;
          atomicAdd(reinterpret_cast<float4 *>(dst),
                    make_float4(src[0], src[1], src[2], src[3]));
        }
      }
      __syncwarp();
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * H)
                 : "memory");
}

// ------------------------------------------------------------------ Adam
// Every parameter in one launch: blocks of 32 x 32 weights (their bf16 copy
// and its transpose written through a shared tile), then the vectors.
struct AdamArgs {
  float *w[2 * MAX_LAYERS + 2];
  const float *g[2 * MAX_LAYERS + 2];
  float *m[2 * MAX_LAYERS + 2], *v[2 * MAX_LAYERS + 2];
  __nv_bfloat16 *w16[MAX_LAYERS], *w16t[MAX_LAYERS];
  int layers, width0, hidden;
  float lr, b1, b2, eps;
  const float *corr;
};

__device__ __forceinline__ float adam_update(const AdamArgs &a, int p, int64_t i, float c1,
                                             float c2) {
  const float gr = a.g[p][i];
  const float mi = a.b1 * a.m[p][i] + (1.f - a.b1) * gr;
  const float vi = a.b2 * a.v[p][i] + (1.f - a.b2) * gr * gr;
  a.m[p][i] = mi;
  a.v[p][i] = vi;
  const float wi = a.w[p][i] - a.lr * (mi / c1) / (sqrtf(vi / c2) + a.eps);
  a.w[p][i] = wi;
  return wi;
}

__global__ void adam_all_kernel(const __grid_constant__ AdamArgs a) {
  __shared__ __nv_bfloat16 tile[32][34];
  const float c1 = a.corr[0], c2 = a.corr[1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
  const int per_row0 = a.width0 / 32, per_row = a.hidden / 32;
  const int tiles0 = per_row * per_row0, tiles = per_row * per_row;
  int b = blockIdx.x;
  int l = -1;
  if (b < tiles0) {
    l = 0;
  } else if (b < tiles0 + (a.layers - 1) * tiles) {
    l = 1 + (b - tiles0) / tiles;
    b = (b - tiles0) % tiles;
  }
  if (l >= 0) {
    const int across = l == 0 ? per_row0 : per_row, K = 32 * across;
    const int n0 = (b / across) * 32, k0 = (b % across) * 32;
    for (int j = ty; j < 32; j += 8) {
      const int64_t i = (int64_t)(n0 + j) * K + k0 + tx;
      const __nv_bfloat16 w = __float2bfloat16_rn(adam_update(a, l, i, c1, c2));
      a.w16[l][i] = w;
      tile[j][tx] = w;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
      a.w16t[l][(int64_t)(k0 + j) * a.hidden + n0 + tx] = tile[tx][j];
  } else {  // one block per bias vector, the head's weights, the head's bias
    const int q = blockIdx.x - tiles0 - (a.layers - 1) * tiles;
    const int n = q <= a.layers ? a.hidden : 1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) adam_update(a, a.layers + q, i, c1, c2);
  }
}

// ------------------------------------------------------------------ host
int check_net(const pe_mlp_net *n) {
  if (!n || n->hidden != H || n->layers < 1 || n->layers > MAX_LAYERS || n->in_width != 128)
    return fail(PE_EINVAL, "mlp: hidden width 256, input width 128, 1 to 8 layers");
  for (int l = 0; l < n->layers; l++)
    if (!n->w16[l] || !n->b[l] || reinterpret_cast<uintptr_t>(n->w16[l]) % 16)
      return fail(PE_EINVAL, "mlp: weights and biases required, weights 16-byte aligned");
  if (!n->w_out || !n->b_out) return fail(PE_EINVAL, "mlp: head required");
  return PE_OK;
}

// z [rows][256] in 128B-swizzled boxes of 32 x 32
CUresult make_z_map(CUtensorMap *map, const float *z, int rows) {
  const cuuint64_t dims[2] = {H, (cuuint64_t)rows}, strides[1] = {H * sizeof(float)};
  const cuuint32_t box[2] = {32, 32}, elem[2] = {1, 1};
  EncodeTiled encode = encoder();
  if (!encode) return CUDA_ERROR_NOT_FOUND;
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(z), dims, strides,
                box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// cl: CTAs that share the columns of a tile
int forward_args(const pe_mlp_net *n, ForwardArgs &g, int cl) {
  g.layers = n->layers;
  for (int l = 0; l < n->layers; l++) {
    const int K = l == 0 ? n->in_width : H;
    if (make_map(&g.w[l], n->w16[l], H, K, K, H / cl) != CUDA_SUCCESS)
      return fail(PE_EINVAL, "mlp: tensor map encoding failed");
    g.bias[l] = n->b[l];
  }
  g.w_out = n->w_out;
  g.b_out = n->b_out;
  g.error = error_word();
  if (!g.error) return fail(PE_ENOMEM, "mlp: error word");
  return PE_OK;
}

template <class... P, class... A>
cudaError_t launch_tiles(void (*kernel)(P...), int grid, int cl, int bytes, cudaStream_t stream,
                         A &...args) {
  cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim = {(unsigned)cl, 1, 1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = cl > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int TPC, int INPUT, bool TRAIN, int CL = 1>
cudaError_t launch_forward(ForwardArgs &g, cudaStream_t stream) {
  g.groups = (g.rows + TPC * TM - 1) / (TPC * TM);
  // read features: one group per CTA (or cluster); made ones: a persistent CTA per SM
  const int grid = INPUT == FEATURES || g.groups < 148 ? g.groups : 148;
  return launch_tiles(forward_kernel<TPC, INPUT, TRAIN, CL>, grid * CL, CL,
                      ForwardLayout<TPC, CL>::BYTES + 1024, stream, g);
}

// CTAs per 128-row tile of a forward training pass: two while that many fit the
// SMs (8192 rows 43.6 us with one, 34.6 with two), one beyond (9600 rows 40.4
// with one, 64.1 with two, which then take a second wave; 65536: 163 and 240).
// The backward pass takes two at every size (9600 rows, with the weight
// gradients, 74 us with one, 72 with two; 19072: 144, 111; 65536: 325, 278).
inline int cluster_of(int rows) { return 2 * (rows / TM) <= 148 ? 2 : 1; }

// Inference on made features: two tiles per CTA once every SM has two, one
// (half the latency, twice the CTAs) below that.
template <int INPUT>
int infer(const pe_mlp_net *net, ForwardArgs &g, cudaStream_t stream) {
  int rc = forward_args(net, g, 1);
  if (rc) return rc;
  const cudaError_t e = g.rows > 148 * TM ? launch_forward<2, INPUT, false>(g, stream)
                                          : launch_forward<1, INPUT, false>(g, stream);
  if (e != cudaSuccess) return cuda_fail(e, "pe_mlp inference");
  count_launches(1);
  return PE_OK;
}

}  // namespace
}  // namespace pe

extern "C" {

int pe_mlp_forward(const pe_mlp_net *net, const void *feat, int rows, float *const *z,
                   void *const *h, const float *target, float *y, float *dy, float *loss,
                   void *cuda_stream) {
  using namespace pe;
  int rc = check_net(net);
  if (rc) return rc;
  if (!feat || !h || !y || rows <= 0 || rows % TM || (target && (!dy || !loss)) ||
      reinterpret_cast<uintptr_t>(feat) % 16)
    return fail(PE_EINVAL, "mlp_forward: rows a multiple of 128, features 16-byte aligned");
  ForwardArgs g{};
  const int cl = cluster_of(rows);
  rc = forward_args(net, g, cl);
  if (rc) return rc;
  if (tc::make_map(&g.feat, feat, rows, net->in_width, net->in_width, TM) != CUDA_SUCCESS)
    return fail(PE_EINVAL, "mlp_forward: tensor map encoding failed");
  g.rows = rows;
  for (int l = 0; l < net->layers; l++) {
    g.z[l] = z ? z[l] : nullptr;
    g.h[l] = static_cast<__nv_bfloat16 *>(h[l]);
    if (!g.h[l] || (reinterpret_cast<uintptr_t>(g.h[l]) | reinterpret_cast<uintptr_t>(g.z[l])) % 32)
      return fail(PE_EINVAL, "mlp_forward: activation buffers 32-byte aligned");
    if (cl == 2 && g.z[l] && make_z_map(&g.zmap[l], g.z[l], rows) != CUDA_SUCCESS)
      return fail(PE_EINVAL, "mlp_forward: tensor map encoding failed");
  }
  g.target = target;
  g.y = y;
  g.dy = dy;
  g.loss = loss;
  g.inv_rows = 1.f / rows;
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  const cudaError_t e = cl == 2 ? launch_forward<1, FEATURES, true, 2>(g, s)
                                : launch_forward<1, FEATURES, true, 1>(g, s);
  if (e != cudaSuccess) return cuda_fail(e, "pe_mlp_forward");
  count_launches(1);
  return PE_OK;
}

int pe_mlp_backward(const pe_mlp_net *net, const void *feat, int rows, const float *const *z,
                    const void *const *h, const float *dy, void *const *dz, float *const *gw,
                    float *const *gb, float *gw_out, float *gb_out, void *cuda_stream) {
  using namespace pe;
  int rc = check_net(net);
  if (rc) return rc;
  if (!feat || !z || !h || !dy || !dz || !gw || !gb || !gw_out || !gb_out || rows <= 0 ||
      rows % TM)
    return fail(PE_EINVAL, "mlp_backward: invalid arguments");
  BackwardArgs b{};
  WeightGradArgs w{};
  b.layers = net->layers;
  b.error = w.error = tc::error_word();
  if (!b.error) return fail(PE_ENOMEM, "mlp_backward: error word");
  CUresult r = CUDA_SUCCESS;
  auto map = [&](CUtensorMap *m, const void *p, int nrows, int K, int box) {
    if (r == CUDA_SUCCESS) r = tc::make_map(m, p, nrows, K, K, box);
  };
  for (int l = 0; l < net->layers; l++) {
    const int K = l == 0 ? net->in_width : H;
    if (!z[l] || !h[l] || !dz[l] || !gw[l] || !gb[l] || (l > 0 && !net->w16t[l]) ||
        (reinterpret_cast<uintptr_t>(z[l]) | reinterpret_cast<uintptr_t>(dz[l])) % 32 ||
        reinterpret_cast<uintptr_t>(gw[l]) % 16)
      return fail(PE_EINVAL, "mlp_backward: buffers of every layer required, aligned");
    if (l > 0) map(&b.wt[l], net->w16t[l], H, H, H / BCL);
    if (r == CUDA_SUCCESS) r = make_z_map(&b.zmap[l], z[l], rows);
    map(&w.dz[l], dz[l], rows, H, 64);
    map(&w.prev[l], l == 0 ? feat : h[l - 1], rows, K, 64);
    b.dz[l] = static_cast<__nv_bfloat16 *>(dz[l]);
    w.gb[l] = gb[l];
    w.gw[l] = gw[l];
  }
  if (r != CUDA_SUCCESS) return fail(PE_EINVAL, "mlp_backward: tensor map encoding failed");
  b.h_last = static_cast<const __nv_bfloat16 *>(h[net->layers - 1]);
  b.dy = dy;
  b.w_out = net->w_out;
  b.gw_out = gw_out;
  b.gb_out = gb_out;
  w.width0 = net->in_width;
  w.ksteps = rows / 64;
  cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  cudaError_t e = cudaFuncSetAttribute(weight_grad_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, G_BYTES);
  if (e == cudaSuccess)
    e = launch_tiles(backward_kernel, rows / TM * BCL, BCL, BackwardLayout::BYTES + 1024, s, b);
  if (e != cudaSuccess) return cuda_fail(e, "pe_mlp_backward");
  // about one CTA per SM, none with fewer than two 64-row steps; nor more than
  // eight (chains of 16 MMAs into each accumulator: twice that at 16384 rows
  // put the gradients 4.9e-7 from 64 bits, against 2.7e-7)
  const int tiles = 2 * net->layers;
  const int splits =
      std::max({1, std::min(148 / tiles, w.ksteps / 2), (w.ksteps + 7) / 8});
  weight_grad_kernel<<<dim3(tiles, splits), G_THREADS, G_BYTES, s>>>(w);
  PE_CUDA_TRY(cudaGetLastError());
  count_launches(2);
  return PE_OK;
}

int pe_mlp_adam_all(const pe_mlp_net *net, float *const *w, const float *const *grad,
                    float *const *m, float *const *v, void *const *w16, void *const *w16t,
                    float lr, float beta1, float beta2, float eps, const float *corr,
                    void *cuda_stream) {
  using namespace pe;
  if (!net || net->layers < 1 || net->layers > MAX_LAYERS || net->hidden < 128 ||
      net->hidden % 32 || net->in_width < 32 || net->in_width % 32 || !w || !grad || !m || !v ||
      !w16 || !w16t || !corr)
    return fail(PE_EINVAL, "mlp_adam_all: invalid arguments");
  AdamArgs a{};
  for (int p = 0; p < 2 * net->layers + 2; p++) {
    if (!w[p] || !grad[p] || !m[p] || !v[p]) return fail(PE_EINVAL, "mlp_adam_all: NULL array");
    a.w[p] = w[p];
    a.g[p] = grad[p];
    a.m[p] = m[p];
    a.v[p] = v[p];
  }
  for (int l = 0; l < net->layers; l++) {
    if (!w16[l] || !w16t[l]) return fail(PE_EINVAL, "mlp_adam_all: NULL weight copy");
    a.w16[l] = static_cast<__nv_bfloat16 *>(w16[l]);
    a.w16t[l] = static_cast<__nv_bfloat16 *>(w16t[l]);
  }
  a.layers = net->layers;
  a.width0 = net->in_width;
  a.hidden = net->hidden;
  a.lr = lr;
  a.b1 = beta1;
  a.b2 = beta2;
  a.eps = eps;
  a.corr = corr;
  const int t = net->hidden / 32;
  const int blocks = t * (net->in_width / 32) + (net->layers - 1) * t * t + net->layers + 2;
  adam_all_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(cuda_stream)>>>(a);
  PE_CUDA_TRY(cudaGetLastError());
  count_launches(1);
  return PE_OK;
}

int pe_mlp_predict_relative_nodes(const pe_mlp_net *net, int64_t first, int64_t n, int positions,
                                  int headings, int p_speeds, int e_speeds, double extent,
                                  double p_min, double p_max, double e_min, double e_max,
                                  float *out, void *cuda_stream) {
  using namespace pe;
  int rc = check_net(net);
  if (rc) return rc;
  if (first < 0 || n <= 0 || n > INT32_MAX - 1024 || !out)
    return fail(PE_EINVAL, "predict_relative_nodes: invalid arguments");
  ForwardArgs g{};
  g.grid = node_grid(positions, headings, p_speeds, e_speeds, extent, p_min, p_max, e_min, e_max);
  g.first = first;
  g.rows = (int)n;
  g.y = out;
  return infer<RELATIVE_NODES>(net, g, static_cast<cudaStream_t>(cuda_stream));
}

int pe_mlp_predict_world_nodes(const pe_mlp_net *net, int64_t first, int64_t n, int positions,
                               int headings, int p_speeds, int e_speeds, double extent,
                               double p_min, double p_max, double e_min, double e_max,
                               float *out, void *cuda_stream) {
  using namespace pe;
  int rc = check_net(net);
  if (rc) return rc;
  if (first < 0 || n <= 0 || n > INT32_MAX - 1024 || !out)
    return fail(PE_EINVAL, "predict_world_nodes: invalid arguments");
  ForwardArgs g{};
  g.grid = node_grid(positions, headings, p_speeds, e_speeds, extent, p_min, p_max, e_min, e_max);
  g.first = first;
  g.rows = (int)n;
  g.y = out;
  return infer<WORLD_NODES>(net, g, static_cast<cudaStream_t>(cuda_stream));
}

int pe_mlp_predict_relative_states(const pe_mlp_net *net, const float *states, int n,
                                   double extent, double p_min, double p_max, double e_min,
                                   double e_max, float *out, void *cuda_stream) {
  using namespace pe;
  int rc = check_net(net);
  if (rc) return rc;
  if (!states || n <= 0 || n > INT32_MAX - 1024 || !out)
    return fail(PE_EINVAL, "predict_relative_states: invalid arguments");
  ForwardArgs g{};
  g.grid.f = feature_scale((float)extent, (float)p_min, (float)p_max, (float)e_min, (float)e_max);
  g.states = states;
  g.rows = n;
  g.y = out;
  return infer<RELATIVE_STATES>(net, g, static_cast<cudaStream_t>(cuda_stream));
}

}  // extern "C"
