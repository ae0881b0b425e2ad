// bf16 GEMM for sm_100a with CTA pairs: tcgen05.mma.cta_group::2, 256 x 256 output tile per pair.
//
//   C[M,N] (+)= alpha * A[M,K] * B[N,K]^T (+ bias)        same contract as gemm_bf16.cu
//
// Two CTAs on neighbouring SMs form a cluster. Each loads its own 128 rows of A and its own 128
// rows (half) of the B tile, 32 KB per stage instead of 48 KB, so the ring is 6 stages deep and
// every byte of B is fetched once per pair. The leader CTA (cluster rank 0) issues the MMAs for
// both SMs; each CTA's tensor memory receives its own 128 rows of the 256 x 256 accumulator and
// each CTA runs its own epilogue. No TMA copy here is shared between CTAs: every load lands in
// the shared memory of the CTA that issued it and only its completion is signalled to the leader.
//
// Barrier protocol (per stage s, per accumulator a):
//   full[s]    leader only : leader's producer arrives with the pair's byte count (64 KB); the TMA
//                            loads of BOTH CTAs complete on it
//   empty[s]   both CTAs   : tcgen05.commit from the leader arrives on both
//   tfull[a]   both CTAs   : tcgen05.commit from the leader arrives on both
//   tempty[a]  leader only : the 8 epilogue warps of both CTAs arrive (16 arrivals)
//
// Fused with collectives over NVLink (tensor parallelism with sequence-sharded activations):
//   all-gather -> GEMM   the rows of A arrive shard by shard in a local buffer (copy engines pulling the
//                        peers' shards); `Gate` carries one arrival flag per shard, the TMA producer of a
//                        tile waits (bounded) for the flag of the shard that holds its rows, and the tiles
//                        are visited starting with this rank's own shard, so the math starts at once and
//                        the transfers hide behind it
//   GEMM -> reduce-scatter  the epilogue adds every output row into the fp32 accumulation buffer of the
//                        rank that owns the row (`red.add.f32` on peer pointers): no partial-sum tensor, no
//                        separate collective, the reduction traffic overlaps the remaining tiles
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace {
using namespace atb;

constexpr int BM = 128;   // rows of A per CTA (256 per pair)
constexpr int BK = 64;
constexpr int A_BYTES = BM * BK * 2;

// BN = accumulator columns of the pair's tile (256 or 128); each CTA loads BN/2 rows of B.
// The narrower tile exists for wave quantisation: 256 tiles of 256x256 fill 74 CTA pairs 3.46 times
// (4 waves, 86 % busy), the same problem in 256x128 tiles takes 7 waves of half the length (99 %).
//
// SPLIT = 2: two pairs, a cluster of four CTAs, share a tile: pair p takes half p of the reduction and finishes half of the
// columns, whose partial sums it gets from its counterpart (same rows) through distributed shared memory, 64 KB each way per
// tile; half of the epilogue is left to each. For products with too few tiles, see split_pays.
template <int BN, int SPLIT = 1>
struct Cfg {
  static constexpr int BNH = BN / 2;
  static constexpr int STAGES = SPLIT == 2 ? 5 : BN == 256 ? 6 : 8;
  static constexpr int B_BYTES = BNH * BK * 2;
  static constexpr int X_OFF = STAGES * (A_BYTES + B_BYTES);         // partial sums from the other pair, fp32
  // output boxes on their way out (see the epilogue): 4 KB per epilogue warp, [32 rows][128 bytes] with 128-byte swizzle, in
  // the place of the operands, all of which have been multiplied by then. Space of their own took half of the L1 cache, in
  // which an epilogue that adds to fp32 values keeps their lines: 4096 x 4096 x 256 68.0 us, 84.2 with it.
  static constexpr int OUT_OFF = 0;
  static constexpr int BAR_OFF = X_OFF + (SPLIT == 2 ? BM * (BN / 2) * 4 : 0);
  static constexpr int TQ = 4;                     // tile-id ring of the dynamic scheduler
  static constexpr int SMEM_TOTAL = BAR_OFF + (2 * STAGES + 4 + 2 * TQ + 3) * 8 + 16 + TQ * 4 + 1024;
  static_assert(SMEM_TOTAL <= 232448, "shared memory of the pair kernel exceeds 227 KB");
};

struct Epi {
  void* C;
  const void* bias;
  long long ldc;
  float alpha;
  int out_fp32, accumulate;
  const void* residual;  // optional bf16 [M, N] added in the epilogue (pitch ldr); bf16 output only
  long long ldr;
  // reduce-scatter epilogue (rs_rows > 0): row r goes to rank r / rs_rows, as fp32 atomic adds into
  // rs_base[rank] + (r % rs_rows) * ldc + column; C is not written
  float* rs_base[8];
  int rs_rows;
  // gated (SwiGLU) epilogue: B is the fused gate|up weight [2 N, K] (K-major); a tile pairs gate rows
  // [f0, f0 + BN/2) (CTA 0's half of B) with up rows [N + f0, ...) (CTA 1's half), so that accumulator columns c
  // and BN/2 + c belong to the same output feature, and C[:, f0 + c] = silu(gate) * up is written as bf16. With
  // gu_out != null the bf16 gate and up values are stored too ([M, 2 N], pitch ldgu) for the backward pass.
  int gated;
  void* gu_out;
  long long ldgu;
  // rotary epilogue (rope_cos != null; bf16 output, no accumulation, no residual): columns [0, rope_cols) are heads of
  // rope_dim (128 or 64) columns and leave the epilogue rotated, out[c] = x[c] cos - x[c + D/2] sin, out[c + D/2] =
  // x[c + D/2] cos + x[c] sin, with fp32 tables [rope_s, D/2] at position rope_pos[row], or row % rope_s
  const float* rope_cos;
  const float* rope_sin;
  const int* rope_pos;
  int rope_s, rope_dim, rope_cols;
  int split;  // (host) pairs per tile: 0 by split_pays, -1 one, 1 two wherever the kernel can
  int boxed;  // nothing but a rounding to bf16 on the way out, and a tensor map for it (set by launch)
  int wide;   // every 16 columns of an output row start on a 32-byte boundary and N is a multiple of 16 (set by launch)
};

// 32 packed bf16 columns of a row, of which `cols` (a multiple of 8) are inside the matrix
ATB_DEVICE void store_row_bf16(__nv_bfloat16* p, const uint32_t (&o)[16], int cols, bool wide) {
  if (wide) {
    stg_v8(p, o);
    if (cols > 16) stg_v8(p + 16, o + 8);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i * 8 < cols) *reinterpret_cast<uint4*>(p + i * 8) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
  }
}
// v[0..8) += 8 bf16 values (16-byte aligned)
ATB_DEVICE void add_row_bf16(const __nv_bfloat16* p, float* v) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = unpack_bf16x2(w[i]);
    v[2 * i] += f.x;
    v[2 * i + 1] += f.y;
  }
}

// Arrival flags of the A operand (all-gather -> GEMM): rows [g * rows, (g + 1) * rows) are in place once
// flags[g] >= epoch (wrap-safe). rot = first tile row to visit (this rank's own shard).
// on_b: the flags describe rows of B (a weight gathered from row shards) instead of rows of A; rot then counts
// tile columns.
struct Gate {
  const unsigned int* flags;
  unsigned int epoch;
  int rows, rot;
  int on_b;
};

__device__ unsigned long long g_gate_wait_ns = ATB_WAIT_LIMIT_NS;

// An error that a kernel has recorded in the status word.
ATB_DEVICE bool error_recorded(const int* status) {
  return status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
}

// True as well, at once, when an error has been recorded: what would arrive is not needed any more (see `stopped`).
ATB_DEVICE bool gate_wait(const Gate& gate, int row_lo, int row_hi, volatile int* abort_flag, int* status) {
  for (int g = row_lo / gate.rows; g <= (row_hi - 1) / gate.rows; ++g) {
    const unsigned int* f = gate.flags + g;
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
    if ((int)(v - gate.epoch) >= 0) continue;
    const unsigned long long limit = g_gate_wait_ns;
    const uint64_t t0 = globaltimer_ns();
    while (true) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(f) : "memory");
      if ((int)(v - gate.epoch) >= 0) break;
      if (*abort_flag) return false;
      if (error_recorded(status)) return true;
      if (globaltimer_ns() - t0 > limit) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, (int)ATB_ERR_PEER_TIMEOUT);
        return false;
      }
      __nanosleep(200);
    }
  }
  // the rows were written by the copy engines / generic proxy; the loads that follow go through TMA
  asm volatile("fence.proxy.async.global;" ::: "memory");
  return true;
}

// Row groups with device-resident fill counts (mixture-of-experts buffers: `rows` slots per group, only
// the first counts[g] hold data and the rest is zero).
//   m_rows > 0 : rows of A / C form groups of m_rows (a multiple of 256). A tile that starts at or beyond
//                its group's count does no loads and no MMAs; its output is written as zeros.
//   b_rows > 0 : every bm_rows rows of A / C (a multiple of 256; one expert's slots from all sources)
//                multiply with their own B: the B tile coordinate is shifted by (m0 / bm_rows) * b_rows
//                along B's row axis (N for K-major B, K for MN-major B): B is [n_b * b_rows, ...].
//   k_rows > 0 : the reduction dim forms groups of k_rows (a multiple of 64); k-blocks at or beyond their
//                group's count are skipped (both operands are zero there).
struct Groups {
  const int* counts;
  int m_rows, b_rows, k_rows, bm_rows;
};

// Consecutive row groups of any length (routed tokens sorted by expert; the lengths are known on the host): group g
// holds rows [row0[g], row0[g + 1]) of A / C and is cut into tiles of its own, m-tiles [mt0[g], mt0[g + 1]) of the
// launch. Its B is shifted by g * Groups::b_rows as above. A tile's loads may run into the rows of the next group,
// its stores stop at the group's end. n == 0: off.
constexpr int RAGGED_MAX = 64;
struct Ragged {
  int n;
  int row0[RAGGED_MAX + 1], mt0[RAGGED_MAX + 1];
};

// Weight gradients of the same groups, C_g = A_g^T B_g (both operands MN-major, the reduction runs over the group's rows):
// one tensor map per group and operand, so that a group's last k-block ends with its rows (the rest reads as zero). The
// outputs are stacked, [n * M, N]; a group without rows writes zeros (nothing when accumulating).
// One launch for up to 16 groups. Against one per group (each with its own prologue, last wave and exposed last epilogue):
// gradients of 8 experts x 14336 x 4096 over 8192 rows 2518 -> 2468 us; forward and backward of an expert MLP
// 8 x 4096 x 1024 on 131 tokens 782 -> 515 us, 8 x 3520 x 1024 on 2049 tokens 797 -> 550, 4 x 8192 x 2048 on 1000 tokens
// 707 -> 657, 4 x 9024 x 4096 on 2000 tokens 2765 -> 2712.
constexpr int KGROUP_MAX = 16;
template <bool KG>
struct KGroups {};
template <>
struct KGroups<true> {
  CUtensorMap a[KGROUP_MAX], b[KGROUP_MAX];
  int rows[KGROUP_MAX];
  int n;
};

template <bool KG>
uint64_t kg_count(const KGroups<KG>& kg) {
  if constexpr (KG) return kg.n;
  return 1;
}

ATB_DEVICE uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
ATB_DEVICE void cluster_arrive_all() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
ATB_DEVICE void cluster_wait_all() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
ATB_DEVICE void cluster_sync_all() {
  cluster_arrive_all();
  cluster_wait_all();
}
// shared::cluster address of `ptr` (a shared::cta pointer of this CTA) in CTA `rank` of the cluster
ATB_DEVICE uint32_t map_to_cta(const void* ptr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(ptr)), "r"(rank));
  return r;
}
// TMA load into this CTA's shared memory whose completion is counted on a barrier given by its
// shared::cluster address (the leader's).
ATB_DEVICE void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tm, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
// Dynamic tile scheduling: tiles are handed out by an atomic counter instead of a fixed stride, so that a CTA pair
// that shares its SMs with another kernel (a reduce-scatter or copy kernel of the communication streams takes part
// of the SM's path to L2, on which this kernel's operand loads depend) simply takes fewer tiles, instead of making
// the whole launch wait for it. Where two pairs share a tile, their cluster of four draws as one. counters[0] = next tile,
// counters[1] = clusters that have finished; both are zero between launches (the cluster that finishes last clears them).
struct Sched {
  int* counters;   // nullptr: static schedule (tile = pair + i * pairs)
  int early;       // the launch after this one may take the SMs that this one leaves
};

ATB_DEVICE void st_remote_u32(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
ATB_DEVICE void st_remote_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Wait (by a whole converged warp, one answer for all lanes) on a barrier whose phase is completed by an arrive of
// another CTA of the cluster that published data with it.
ATB_DEVICE bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
    if ((++spins & 0x3ff) == 0) {
      const uint64_t now = warp_uniform(globaltimer_ns());
      if (t0 == 0) t0 = now;
      const bool late = now - t0 > ATB_WAIT_LIMIT_NS;
      if (late) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, (int)ATB_ERR_WAIT_TIMEOUT);
      }
      if (__any_sync(0xffffffffu, late || *abort_flag != 0)) return false;
    }
  }
}
ATB_DEVICE void mbar_arrive_remote(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// Epilogue: two warps per lane quarter of tensor memory, each with one half of the tile's columns; the next 32 columns
// are loaded out of tensor memory while the current ones are converted and stored, 32 bytes per thread and store where
// the output's alignment allows it. With four warps and 16-byte stores a tile took 11,000 clocks, more than the main
// loop of a reduction over 1000 (16 k-blocks of 570 clocks), and it is exposed in full after the last tile of any launch.
// The twelve products of a 7B block on 4096 tokens: 3471 -> 3311 us (1500 TFLOP/s); of a 1.3B block on 3000 tokens:
// 883 -> 833 us; weight gradients of 8 experts x 14336 x 4096 over 8192 routed rows: 2767 -> 2429 us.
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;

template <int BN, bool A_MN, bool B_MN, bool KG, int SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, Epi ep, int M,
                      int N, int K, Groups grp, Gate gate, Sched sched, const __grid_constant__ Ragged rag,
                      const __grid_constant__ KGroups<KG> kg, int* status) {
  static_assert(!KG || (A_MN && B_MN), "groups along the reduction are rows of MN-major operands");
  static_assert(SPLIT == 1 || (BN == 256 && !KG), "two pairs share a 256-wide tile");
  using C = Cfg<BN, SPLIT>;
  constexpr int BNH = C::BNH, STAGES = C::STAGES, B_BYTES = C::B_BYTES, BAR_OFF = C::BAR_OFF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  constexpr int TQ = C::TQ;
  uint64_t* tq_full = tempty + 2;
  uint64_t* tq_empty = tq_full + TQ;
  uint64_t* xfull = tq_empty + TQ;        // partial sums of the other pair are in the exchange buffer
  uint64_t* xfree = xfull + 1;            // the other pair has read those sent to it
  uint64_t* tmem_ready = xfree + 1;       // tensor memory has been allocated
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* tq_tile = reinterpret_cast<volatile int*>(tmem_slot + 4);   // [TQ] tile ids (-1: no more tiles)

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t cta = warp_uniform(cluster_ctarank());
  const uint32_t rank = cta & 1, pair0 = cta & ~1u;     // place in the pair; the pair's first CTA in the cluster
  const int part = SPLIT == 2 ? (int)(cta >> 1) : 0;    // which half of the reduction and of the columns
  const bool leader = rank == 0;
  const int tiles_m = rag.n > 0 ? rag.mt0[rag.n] : (M + 2 * BM - 1) / (2 * BM);
  const int tile_cols = ep.gated ? BN / 2 : BN;      // output columns per tile
  const int tiles_n = (N + tile_cols - 1) / tile_cols;
  int groups = 1;
  if constexpr (KG) groups = kg.n;
  // k-blocks [first, end) of a tile for this pair
  auto tile_kbs = [&](int b_idx, int& first) -> int {
    first = 0;
    if constexpr (KG) return (kg.rows[b_idx] + BK - 1) / BK;
    const int n = (K + BK - 1) / BK, mid = (n + 1) / 2;
    if constexpr (SPLIT == 2) {
      first = part ? mid : 0;
      return part ? n : mid;
    }
    return n;
  };
  const int cluster_id = blockIdx.x / (2 * SPLIT), num_clusters = gridDim.x / (2 * SPLIT);
  constexpr int BAND = 8;

  // What every role waits for is the barriers of all CTAs of the cluster, so they come first, and the wait for them last: the
  // allocation of tensor memory and the coordinates of the first tile lie between arriving and waiting. One after the other
  // the first load went out 4060 clocks after the start of a CTA, now 3140.
  if (warp == 2) {
    if (lane == 0) {
      for (int i = 0; i < STAGES; ++i) {
        mbar_init(&full[i], 1);
        mbar_init(&empty[i], 1);
      }
      mbar_init(&tfull[0], 1);
      mbar_init(&tfull[1], 1);
      mbar_init(&tempty[0], 2 * EPI_WARPS);
      mbar_init(&tempty[1], 2 * EPI_WARPS);
      for (int i = 0; i < TQ; ++i) {
        mbar_init(&tq_full[i], 1);
        // read by every CTA's epilogue warps, every pair's MMA warp and every producer but the one that draws
        mbar_init(&tq_empty[i], SPLIT * (2 + 2 * EPI_WARPS) + SPLIT - 1);
      }
      mbar_init(xfull, EPI_WARPS);
      mbar_init(xfree, EPI_WARPS);
      mbar_init(tmem_ready, 1);
      *abort_flag = 0;
      mbar_fence_init();
    }
    __syncwarp();
  }
  cluster_arrive_all();
  if (!KG && warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc<2>(tmem_slot, 2 * BN);
    tmem_relinquish<2>();
    tc_fence_before();
    if (lane == 0 && sched.early) grid_go();
  }
  const int num_tiles = tiles_m * tiles_n * groups;

  // identical decisions in every role: which tiles and which k-blocks carry data
  auto tile_active = [&](int m0, int b_idx) -> bool {
    if constexpr (KG) return kg.rows[b_idx] > 0;
    if (grp.counts == nullptr) return true;
    if (grp.m_rows > 0) {
      const int g = m0 / grp.m_rows;
      if (m0 - g * grp.m_rows >= grp.counts[g]) return false;
    }
    if (grp.k_rows > 0) {   // nothing to reduce over at all?
      const int ng = (K + grp.k_rows - 1) / grp.k_rows;
      bool any = false;
      for (int g = 0; g < ng; ++g) any |= grp.counts[g] > 0;
      return any;
    }
    return true;
  };
  auto kb_active = [&](int kb) -> bool {
    if (grp.counts == nullptr || grp.k_rows <= 0) return true;
    const int k0 = kb * BK, g = k0 / grp.k_rows;
    return k0 - g * grp.k_rows < grp.counts[g];
  };

  // first row / column of a tile, the end of its rows and the index of its B operand
  auto tile_coords = [&](int tile, int& m0, int& n0, int& m_end, int& b_idx) {
    int kg_idx = 0;
    if constexpr (KG) {
      kg_idx = tile / (tiles_m * tiles_n);
      tile -= kg_idx * tiles_m * tiles_n;
    }
    const int band_tiles = BAND * tiles_n;
    const int band = tile / band_tiles;
    const int rem = tile - band * band_tiles;
    const int rows_in_band = min(BAND, tiles_m - band * BAND);
    int tn = rem / rows_in_band;
    int tm = band * BAND + (rem - tn * rows_in_band);
    if (gate.rot > 0) {          // start with the rows that are already here
      if (gate.on_b) {
        tn += gate.rot;
        if (tn >= tiles_n) tn -= tiles_n;
      } else {
        tm += gate.rot;
        if (tm >= tiles_m) tm -= tiles_m;
      }
    }
    n0 = tn * tile_cols;
    if (rag.n > 0) {
      int g = 0;
      while (tm >= rag.mt0[g + 1]) ++g;
      m0 = rag.row0[g] + (tm - rag.mt0[g]) * 2 * BM;
      m_end = rag.row0[g + 1];
      b_idx = g;
    } else {
      m0 = tm * 2 * BM;
      m_end = M;
      b_idx = KG ? kg_idx : grp.b_rows > 0 ? m0 / grp.bm_rows : 0;
    }
  };

  // The idx-th tile of this cluster, the same number in every role of all its CTAs. Static: a fixed stride. Dynamic: the
  // first CTA's producer thread draws it from the global counter and publishes it through a ring of tile ids in the
  // shared memory of all CTAs; every other role reads it there and frees the slot.
  const bool dyn = sched.counters != nullptr, draws = cta == 0;
  // A cluster of four begins with the tile of its own number and draws and publishes the next one AHEAD k-blocks before
  // the end of its loads: four CTAs take longer to hear of it.
  constexpr int GIVEN = SPLIT == 2 ? 1 : 0, AHEAD = 8;
  auto static_tile = [&](int idx) -> int {
    const int t = cluster_id + idx * num_clusters;
    return t < num_tiles ? t : -1;
  };
  auto publish_tile = [&](int idx, int t) -> bool {          // the producer warp that draws
    const int slot = (idx - GIVEN) % TQ;
    if (!mbar_wait_warp(&tq_empty[slot], (((idx - GIVEN) / TQ) & 1) ^ 1, abort_flag, status)) return false;
    if (lane == 0) {
      tq_tile[slot] = t;
      mbar_arrive(&tq_full[slot]);
#pragma unroll
      for (uint32_t to = 1; to < 2 * SPLIT; ++to) {
        st_remote_u32(map_to_cta(const_cast<int*>(&tq_tile[slot]), to), (uint32_t)t);
        mbar_arrive_remote(map_to_cta(&tq_full[slot], to));     // release.cluster: orders the store above
      }
    }
    return true;
  };
  auto read_tile = [&](int idx) -> int {                      // any other role, a whole warp
    if (!dyn || idx < GIVEN) return static_tile(idx);
    const int slot = (idx - GIVEN) % TQ;
    if (!mbar_wait_cluster(&tq_full[slot], ((idx - GIVEN) / TQ) & 1, abort_flag, status)) return -1;
    return warp_uniform((int)tq_tile[slot]);
  };
  auto free_tile_slot = [&](int idx) {                        // once per consumer warp, after read_tile by all its lanes
    __syncwarp();
    if (dyn && idx >= GIVEN && lane == 0) mbar_arrive_remote(map_to_cta(&tq_empty[(idx - GIVEN) % TQ], 0));
  };

  if (warp == 0) {
    {
      uint32_t it = 0;
      // lane 0 draws, all lanes know the number
      auto draw = [&]() -> int {
        int d = 0;
        if (lane == 0) d = atomicAdd(&sched.counters[0], 1);
        return warp_uniform(d) + GIVEN * num_clusters;
      };
      grid_wait();
      int drawn = (dyn && draws && GIVEN == 0) ? draw() : 0;
      // the first tile, as far as it is known without the cluster
      int tile = dyn && GIVEN == 0 ? (draws && drawn < num_tiles ? drawn : -1) : static_tile(0);
      int m0 = 0, n0 = 0, m_end = 0, b_idx = 0;
      if (tile >= 0) tile_coords(tile, m0, n0, m_end, b_idx);
      cluster_wait_all();
      for (int idx = 0;; ++idx) {
        if (idx > 0 || (dyn && !draws && GIVEN == 0)) {
          if (dyn && draws) {
            tile = drawn < num_tiles ? drawn : -1;
          } else {
            tile = read_tile(idx);
            free_tile_slot(idx);
          }
          if (tile >= 0) tile_coords(tile, m0, n0, m_end, b_idx);
        }
        if (dyn && draws) {
          if (GIVEN == 0) {
            if (tile >= 0) drawn = draw();                     // the next one, fetched under this tile's loads
            if (!publish_tile(idx, tile)) goto producer_done;
          }
          if (tile < 0 && lane == 0) {   // every cluster draws exactly one number past the end; the last to do so resets
            if (atomicAdd(&sched.counters[1], 1) == num_clusters - 1) {
              sched.counters[0] = 0;
              sched.counters[1] = 0;
              __threadfence();
            }
          }
        }
        if (tile < 0) break;
        if (!tile_active(m0, b_idx)) continue;
        int kb_first;
        const int kb_end = tile_kbs(b_idx, kb_first);
        const CUtensorMap *mapA = &tmA, *mapB = &tmB;
        if constexpr (KG) {
          mapA = &kg.a[b_idx];
          mapB = &kg.b[b_idx];
        }
        const int am0 = m0 + (int)rank * BM;   // this CTA's rows of A
        const int bshift = b_idx * grp.b_rows;   // this expert's own B
        // this CTA's rows of B (gated: CTA 0 takes gate rows, CTA 1 the up rows of the same features)
        const int bn0 = n0 + (int)rank * (ep.gated ? N : BNH) + (B_MN ? 0 : bshift);
        const int bk0 = B_MN ? bshift : 0;
        if (gate.flags != nullptr) {
          bool here = true;
          if (lane == 0)
            here = gate.on_b ? gate_wait(gate, min(bn0, N - 1), min(bn0 + BNH, N), abort_flag, status)
                             : gate_wait(gate, am0, min(am0 + BM, M), abort_flag, status);
          if (!__all_sync(0xffffffffu, here)) goto producer_done;
        }
        for (int kb = kb_first; kb < kb_end; ++kb) {
          if (GIVEN > 0 && dyn && draws && kb == max(kb_end - AHEAD, kb_first)) {
            drawn = draw();
            if (!publish_tile(idx + 1, drawn < num_tiles ? drawn : -1)) goto producer_done;
          }
          if (!kb_active(kb)) continue;
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait_warp(&empty[s], ph ^ 1, abort_flag, status)) goto producer_done;
          if (lane == 0) {
            if (leader) mbar_expect_tx(&full[s], 2 * (A_BYTES + B_BYTES));
            const uint32_t bar = map_to_cta(&full[s], pair0);
            uint8_t* a_dst = sA + s * A_BYTES;
            uint8_t* b_dst = sB + s * B_BYTES;
            if constexpr (!A_MN) {
              tma_load_2d_pair(a_dst, mapA, bar, kb * BK, am0);
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(a_dst + j * 8192, mapA, bar, am0 + j * 64, kb * BK);
            }
            if constexpr (!B_MN) {
              tma_load_2d_pair(b_dst, mapB, bar, kb * BK, bn0);
            } else {
#pragma unroll
              for (int j = 0; j < BNH / 64; ++j)
                tma_load_2d_pair(b_dst + j * 8192, mapB, bar, bn0 + j * 64, bk0 + kb * BK);
            }
          }
          ++it;
        }
      }
    }
  producer_done:;
  } else if (warp == 1) {
    cluster_wait_all();
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(*tmem_slot);
    if (lane == 0) mbar_arrive(tmem_ready);
    if (leader) {
      grid_wait();                          // counts of rows lie in device memory; a wait with a limit starts when work can
      const uint32_t el = elect_one();      // the lane that issues and commits
      const uint32_t a_desc = umma_desc_lo(smem_u32(sA), A_MN ? 8192 : 16), b_desc = umma_desc_lo(smem_u32(sB), B_MN ? 8192 : 16);
      const uint32_t empty0 = map_to_cta(empty, pair0), empty1 = map_to_cta(empty, pair0 + 1);
      const uint32_t tfull0 = map_to_cta(tfull, pair0), tfull1 = map_to_cta(tfull, pair0 + 1);
      constexpr uint32_t idesc = umma_idesc(2 * BM, BN, 1, 1, A_MN, B_MN);
      uint32_t it = 0;
      int local = 0;
      for (int idx = 0;; ++idx) {
        const int tile = read_tile(idx);
        free_tile_slot(idx);
        if (tile < 0) break;
        int kb_first, kb_end;
        {
          int m0, n0, m_end, b_idx;
          tile_coords(tile, m0, n0, m_end, b_idx);
          if (!tile_active(m0, b_idx)) continue;
          kb_end = tile_kbs(b_idx, kb_first);
        }
        const int acc = local & 1;
        const uint32_t acc_ph = (local >> 1) & 1;
        if (!mbar_wait_warp(&tempty[acc], acc_ph ^ 1, abort_flag, status)) goto mma_done;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        bool first_kb = true;
        for (int kb = kb_first; kb < kb_end; ++kb) {
          if (!kb_active(kb)) continue;
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait_warp(&full[s], ph, abort_flag, status)) goto mma_done;
          tc_fence_after();
          const uint32_t a_s = a_desc + ((s * A_BYTES) >> 4), b_s = b_desc + ((s * B_BYTES) >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)   // 16 elements of the reduction: 16 rows MN-major, 32 bytes of a row K-major
            umma_ss_issue<2>(d_tmem, a_s + k * (A_MN ? 128 : 2), b_s + k * (B_MN ? 128 : 2), idesc,
                             (first_kb && k == 0) ? 0u : 1u, el);
          first_kb = false;
          umma_commit_cg2_issue(empty0 + s * 8, el);
          umma_commit_cg2_issue(empty1 + s * 8, el);
          ++it;
        }
        umma_commit_cg2_issue(tfull0 + acc * 8, el);
        umma_commit_cg2_issue(tfull1 + acc * 8, el);
        ++local;
      }
    }
  mma_done:;
  } else {
    cluster_wait_all();
    const int q = warp & 3;                 // lane quarter
    const int half = (warp - 2) >> 2;       // column half
    grid_wait();
    // After an error of a kernel before this one nothing is stored. Only the epilogue asks, and here, where that kernel has
    // completed: every role of every CTA of the cluster goes through all tiles either way, so no answer has to be the same in
    // two of them. The load runs under the first tile's products.
    bool stopped = warp_uniform((int)error_recorded(status)) != 0;
    const bool have_tmem = mbar_wait_warp(tmem_ready, 0, abort_flag, status);
    tc_fence_after();
    const uint32_t tmem_base = warp_uniform(*tmem_slot);
    const bool wide = ep.wide != 0;
    int local = 0;
    const uint32_t tempty_leader[2] = {map_to_cta(&tempty[0], pair0), map_to_cta(&tempty[1], pair0)};
    // What becomes of 32 accumulators of a row (the operands' sum over the whole reduction) at column col0 of the output.
    // gate and up of the same 32 features
    auto finish_gated = [&](const uint32_t (&g)[32], const uint32_t (&u)[32], int row, int col0) {
      __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(ep.C) + (long long)row * ep.ldc + col0;
      __nv_bfloat16* grow = ep.gu_out == nullptr ? nullptr
          : reinterpret_cast<__nv_bfloat16*>(ep.gu_out) + (long long)row * ep.ldgu + col0;
      uint32_t gp[16], up[16], op[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        // round to bf16 first: the same values and the same formula as the separate SwiGLU kernel
        gp[j] = pack_bf16x2(__uint_as_float(g[2 * j]), __uint_as_float(g[2 * j + 1]));
        up[j] = pack_bf16x2(__uint_as_float(u[2 * j]), __uint_as_float(u[2 * j + 1]));
        const float2 a = unpack_bf16x2(gp[j]), b = unpack_bf16x2(up[j]);
        op[j] = pack_bf16x2(a.x / (1.f + __expf(-a.x)) * b.x, a.y / (1.f + __expf(-a.y)) * b.y);
      }
      store_row_bf16(crow, op, N - col0, wide);
      if (grow != nullptr) {
        store_row_bf16(grow, gp, N - col0, wide);
        store_row_bf16(grow + N, up, N - col0, wide);
      }
    };
    // the two sides of a rotation, x1 at col0 and x2 half a head further
    auto finish_rope = [&](const uint32_t (&x1)[32], const uint32_t (&x2)[32], int row, int col0) {
      const int hd2 = ep.rope_dim / 2, pos = ep.rope_pos != nullptr ? ep.rope_pos[row] : row % ep.rope_s;
      const long long at = (long long)pos * hd2 + (col0 % ep.rope_dim);
      uint32_t o1[16], o2[16];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 cs = *reinterpret_cast<const float4*>(ep.rope_cos + at + i);
        const float4 sn = *reinterpret_cast<const float4*>(ep.rope_sin + at + i);
        const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
        float a[4], b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float u = __uint_as_float(x1[i + e]) * ep.alpha, v = __uint_as_float(x2[i + e]) * ep.alpha;
          a[e] = u * cv[e] - v * sv[e];
          b[e] = v * cv[e] + u * sv[e];
        }
        o1[i / 2] = pack_bf16x2(a[0], a[1]);
        o1[i / 2 + 1] = pack_bf16x2(a[2], a[3]);
        o2[i / 2] = pack_bf16x2(b[0], b[1]);
        o2[i / 2 + 1] = pack_bf16x2(b[2], b[3]);
      }
      __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(ep.C) + (long long)row * ep.ldc + col0;
      store_row_bf16(crow, o1, N - col0, wide);
      store_row_bf16(crow + hd2, o2, N - col0 - hd2, wide);
    };
    // A body for each kind of output, chosen outside of the loop over the columns: with one for all, the registers for what is
    // added and the choices cost those that need neither 6 % (32000 x 2048 x 512 75.8 us, with one body 81.9; with a bias 101
    // and 120).
    constexpr int PLAIN = 0, FP32 = 1, ADD = 2, ANY = 3;   // bf16; fp32, alone or added to; bf16 and one thing added; the rest
    constexpr std::integral_constant<int, ANY> any{};
    const int output = ep.bias != nullptr || ep.rs_rows > 0 || (ep.residual != nullptr && (ep.accumulate || ep.out_fp32)) ? ANY
                       : ep.out_fp32 ? FP32 : ep.residual == nullptr && !ep.accumulate ? PLAIN : ADD;
    // 32 bf16 values that are added to a row's accumulators, the residual or, when accumulating, the output so far, in four loads
    // at once; with a test of the column around each, they came one after the other, 16 times the latency of the L2 per tile.
    // They are asked for one piece ahead; in the grouped weight gradients, where that slowed down the plain body (8 groups of
    // 1024 rows, 4096 x 14336, 766 -> 836 us), with the piece: added to 861 us, one after the other 972.
    const bool bias16 = (reinterpret_cast<uintptr_t>(ep.bias) & 15) == 0;
    const __nv_bfloat16* added = ep.residual != nullptr ? reinterpret_cast<const __nv_bfloat16*>(ep.residual)
                                 : ep.accumulate && !ep.out_fp32 ? reinterpret_cast<const __nv_bfloat16*>(ep.C) : nullptr;
    const long long added_ld = ep.residual != nullptr ? ep.ldr : ep.ldc;
    auto fetch = [&](uint4 (&x)[4], long long row, int col0) {
      const uint4* p = reinterpret_cast<const uint4*>(added + row * added_ld + col0);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = p[i];
    };
    auto add8 = [&](float* v, const uint4& x) {
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(w[k]);
        v[2 * k] += f.x;
        v[2 * k + 1] += f.y;
      }
    };
    // x: as fetched, if `fetched` (whole pieces)
    auto finish_plain = [&](auto kind, const uint32_t (&r)[32], int row, int col0, long long c_row0, uint4 (&x)[4], bool fetched) {
      constexpr int KIND = decltype(kind)::value;
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * ep.alpha;
      if (KIND == ANY && ep.bias != nullptr) {
        const __nv_bfloat16* bias = reinterpret_cast<const __nv_bfloat16*>(ep.bias);
        if (bias16 && col0 + 32 <= N) {
          uint4 b[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) b[i] = *reinterpret_cast<const uint4*>(bias + col0 + 8 * i);
#pragma unroll
          for (int i = 0; i < 4; ++i) add8(v + 8 * i, b[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (col0 + i < N) v[i] += __bfloat162float(bias[col0 + i]);
        }
      }
      if (KIND == ANY && ep.rs_rows > 0) {
        const int owner = row / ep.rs_rows;
        float* crow = ep.rs_base[owner] + (long long)(row - owner * ep.rs_rows) * ep.ldc + col0;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          if (col0 + i < N)
            asm volatile("red.relaxed.sys.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(crow + i), "f"(v[i]),
                         "f"(v[i + 1]), "f"(v[i + 2]), "f"(v[i + 3])
                         : "memory");
        }
      } else if (KIND == FP32 || (KIND == ANY && ep.out_fp32)) {
        float* crow = reinterpret_cast<float*>(ep.C) + (c_row0 + row) * ep.ldc + col0;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          if (col0 + i < N) {
            if (ep.accumulate) {
              const float4 old = *reinterpret_cast<const float4*>(crow + i);
              v[i] += old.x; v[i + 1] += old.y; v[i + 2] += old.z; v[i + 3] += old.w;
            }
            if (!wide) *reinterpret_cast<float4*>(crow + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
          }
        }
        if (wide) {
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            if (col0 + i < N) stg_v8(crow + i, reinterpret_cast<const uint32_t*>(v + i));
        }
      } else {
        __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(ep.C) + (c_row0 + row) * ep.ldc + col0;
        if ((KIND == ANY || KIND == ADD) && fetched) {
#pragma unroll
          for (int i = 0; i < 4; ++i) add8(v + 8 * i, x[i]);
        }
        const bool more = ep.accumulate && ep.residual != nullptr;      // both: the second one here
        if ((KIND == ANY && more) || ((KIND == ANY || KIND == ADD) && (ep.accumulate || ep.residual != nullptr) && !fetched)) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            if (col0 + i < N) {
              if (ep.accumulate) add_row_bf16(crow + i, v + i);
              if (ep.residual != nullptr && !fetched)
                add_row_bf16(reinterpret_cast<const __nv_bfloat16*>(ep.residual) + (long long)row * ep.ldr + col0 + i,
                             v + i);
            }
          }
        }
        uint32_t o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
        store_row_bf16(crow, o, N - col0, wide);
      }
    };
    int next = -1;
    if (have_tmem) {
      next = read_tile(0);
      free_tile_slot(0);
    }
    for (int idx = 0; next >= 0; ++idx) {
      const int tile = next;
      next = read_tile(idx + 1);      // known by the time this tile's accumulators are: the producer is past its loads
      free_tile_slot(idx + 1);
      int m0, n0, m_end, b_idx;
      tile_coords(tile, m0, n0, m_end, b_idx);
      const long long c_row0 = KG ? (long long)b_idx * M : 0;      // this group's rows of C
      if (!tile_active(m0, b_idx)) {
        // an empty tile: its output is all zeros (left alone when accumulating)
        const int zrow = m0 + (int)rank * BM + q * 32 + lane;
        if (!stopped && !ep.accumulate && ep.rs_rows <= 0 && zrow < M) {
          for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 8) {
            if (n0 + c >= N) break;
            if (ep.out_fp32) {
              float* z = reinterpret_cast<float*>(ep.C) + (c_row0 + zrow) * ep.ldc + n0 + c;
              *reinterpret_cast<float4*>(z) = make_float4(0.f, 0.f, 0.f, 0.f);
              *reinterpret_cast<float4*>(z + 4) = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(ep.C) + (c_row0 + zrow) * ep.ldc + n0 + c) =
                  make_uint4(0u, 0u, 0u, 0u);
            }
          }
        }
        continue;
      }
      const int acc = local & 1;
      const uint32_t acc_ph = (local >> 1) & 1;
      const int row = m0 + (int)rank * BM + q * 32 + lane;
      const bool fetching = added != nullptr && row < m_end;
      uint4 xa[4], xb[4];
      if (SPLIT == 1 && !KG && fetching && n0 + half * (BN / 2) + 32 <= N) fetch(xa, c_row0 + row, n0 + half * (BN / 2));
      if (!mbar_wait_warp(&tfull[acc], acc_ph, abort_flag, status)) break;
      tc_fence_after();
      // a producer that found an error in place of its rows went on without them: look again behind it
      if (gate.flags != nullptr) stopped = stopped || warp_uniform((int)error_recorded(status)) != 0;
      if (stopped) m_end = m0;
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN;
      const bool in = row < m_end;
      const int row0 = m0 + (int)rank * BM + q * 32;      // first of this warp's rows
      // The last tile's epilogue is exposed in full: boxes of 32 rows x 64 columns go through shared memory (swizzled, no bank
      // conflicts) and the TMA unit. 512 x 512 x 512: 11.6 -> 10.3 us, 2048 x 2048 x 4096 weight gradient 30.8 -> 28.8. Earlier
      // tiles keep to direct stores: the operands of the products that run beside them take the whole bandwidth of shared
      // memory.
      if (SPLIT == 1 && ep.boxed != 0 && next < 0 && row0 + 32 <= m_end && n0 + (half + 1) * (BN / 2) <= N) {
        uint8_t* box = smem + C::OUT_OFF + (warp - 2) * 4096;
#pragma unroll 1
        for (int e = 0; e < BN / 128; ++e) {
          uint32_t r0[32], r1[32];
          tmem_ld_32x32(t_addr + half * (BN / 2) + e * 64, r0);
          tmem_ld_32x32(t_addr + half * (BN / 2) + e * 64 + 32, r1);
          tmem_ld_wait();
          if (e > 0) {                   // the box before has been read
            if (lane == 0) tma_store_wait_read<0>();
            __syncwarp();
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t (&r)[32] = i < 4 ? r0 : r1;
            const int k = (i & 3) * 8;
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[k]), __uint_as_float(r[k + 1]));
            o.y = pack_bf16x2(__uint_as_float(r[k + 2]), __uint_as_float(r[k + 3]));
            o.z = pack_bf16x2(__uint_as_float(r[k + 4]), __uint_as_float(r[k + 5]));
            o.w = pack_bf16x2(__uint_as_float(r[k + 6]), __uint_as_float(r[k + 7]));
            *reinterpret_cast<uint4*>(box + lane * 128 + ((i ^ (lane & 7)) << 4)) = o;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmC, box, n0 + half * (BN / 2) + e * 64, (int)(c_row0 + row0));
            tma_store_commit();
          }
        }
        if (lane == 0) tma_store_wait_read<0>();      // shared memory has to outlive its readers
        tc_fence_before();
        __syncwarp();
        break;
      }
      if constexpr (SPLIT == 2) {
        // 32-column pieces: this CTA finishes four of the eight, 4 part .. 4 part + 3, of gate|up columns two of each. This warp
        // sends two of the counterpart's and finishes two of its own, the two sides of what belongs together.
        const bool cross = ep.gated || (ep.rope_cos != nullptr && ep.rope_dim == 128 && n0 + part * 128 < ep.rope_cols);
        auto piece = [&](int owner, int i) -> int { return ep.gated ? (i >> 1) * 4 + 2 * owner + (i & 1) : 4 * owner + i; };
        const int first = cross ? half : 2 * half, second = cross ? half + 2 : 2 * half + 1;      // of the four
        const uint32_t other = cta ^ 2;
        if (!mbar_wait_cluster(xfree, (local & 1) ^ 1, abort_flag, status)) break;
        const uint32_t xout = map_to_cta(smem + C::X_OFF, other) + (q * 32 + lane) * 16;
        uint32_t ra[32], rb[32];
        tmem_ld_32x32(t_addr + piece(1 - part, first) * 32, ra);
        tmem_ld_32x32(t_addr + piece(1 - part, second) * 32, rb);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 8; ++k) {      // four columns of 128 rows are 2 KB: lanes write and read 16 bytes side by side
          st_remote_v4(xout + (first * 8 + k) * BM * 16, ra[4 * k], ra[4 * k + 1], ra[4 * k + 2], ra[4 * k + 3]);
          st_remote_v4(xout + (second * 8 + k) * BM * 16, rb[4 * k], rb[4 * k + 1], rb[4 * k + 2], rb[4 * k + 3]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(map_to_cta(xfull, other));
        tmem_ld_32x32(t_addr + piece(part, first) * 32, ra);
        tmem_ld_32x32(t_addr + piece(part, second) * 32, rb);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(tempty_leader[acc]);
        const int col_a = n0 + piece(part, first) * 32, col_b = n0 + piece(part, second) * 32;
        if (fetching && col_a + 32 <= N) fetch(xa, c_row0 + row, col_a);
        if (fetching && col_b + 32 <= N) fetch(xb, c_row0 + row, col_b);
        if (!mbar_wait_cluster(xfull, local & 1, abort_flag, status)) break;
        const uint8_t* xin = smem + C::X_OFF + (q * 32 + lane) * 16;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float4 a = *reinterpret_cast<const float4*>(xin + (first * 8 + k) * BM * 16);
          const float4 b = *reinterpret_cast<const float4*>(xin + (second * 8 + k) * BM * 16);
          const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ra[4 * k + e] = __float_as_uint(__uint_as_float(ra[4 * k + e]) + av[e]);
            rb[4 * k + e] = __float_as_uint(__uint_as_float(rb[4 * k + e]) + bv[e]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(map_to_cta(xfree, other));
        ++local;
        if (!in) continue;
        if (ep.gated) {
          if (col_a < N) finish_gated(ra, rb, row, col_a);
        } else if (ep.rope_cos != nullptr && col_a < ep.rope_cols) {
          if (col_a < N) finish_rope(ra, rb, row, col_a);
        } else {
          if (col_a < N) finish_plain(any, ra, row, col_a, c_row0, xa, fetching && col_a + 32 <= N);
          if (col_b < N) finish_plain(any, rb, row, col_b, c_row0, xb, fetching && col_b + 32 <= N);
        }
        continue;
      }
      if (ep.gated) {
#pragma unroll 1
        for (int c = half * (BN / 128); c < (half + 1) * (BN / 128); ++c) {
          uint32_t g[32], u[32];
          tmem_ld_32x32(t_addr + c * 32, g);
          tmem_ld_32x32(t_addr + BN / 2 + c * 32, u);
          tmem_ld_wait();
          if (in && n0 + c * 32 < N) finish_gated(g, u, row, n0 + c * 32);
        }
      } else if (ep.rope_cos != nullptr && n0 + half * (BN / 2) < ep.rope_cols) {
        // this warp's half of the columns is one head of 128 or two of 64 (launch checks BN == 256): the pieces that
        // hold the two sides of a rotation are loaded together
        const int gap = ep.rope_dim / 64;      // pieces between them: 2 or 1
#pragma unroll 1
        for (int pr = 0; pr < 2; ++pr) {
          const int c = half * (BN / 64) + pr * (gap == 1 ? 2 : 1);     // first piece of the pair
          uint32_t x1[32], x2[32];
          tmem_ld_32x32(t_addr + c * 32, x1);
          tmem_ld_32x32(t_addr + (c + gap) * 32, x2);
          tmem_ld_wait();
          if (in && n0 + c * 32 < N) finish_rope(x1, x2, row, n0 + c * 32);
        }
      } else {
        constexpr int CH = BN / 64;              // 32-column pieces of this warp's half
        auto pieces = [&](auto kind) {
          uint32_t ra[32], rb[32];
          tmem_ld_32x32(t_addr + half * (BN / 2), ra);
#pragma unroll
          for (int cc = 0; cc < CH; ++cc) {
            const int c = half * CH + cc;
            uint32_t (&r)[32] = (cc & 1) ? rb : ra;
            uint32_t (&rn)[32] = (cc & 1) ? ra : rb;
            tmem_ld_wait();
            if (cc + 1 < CH) {
              tmem_ld_32x32(t_addr + (c + 1) * 32, rn);
              if (kind == ADD && !KG && fetching && n0 + (c + 2) * 32 <= N)
                fetch((cc & 1) ? xa : xb, c_row0 + row, n0 + (c + 1) * 32);
            }
            if (kind == ADD && KG && fetching && n0 + (c + 1) * 32 <= N) fetch(xa, c_row0 + row, n0 + c * 32);
            if (in && n0 + c * 32 < N)
              finish_plain(kind, r, row, n0 + c * 32, c_row0, (kind == ADD && !KG && (cc & 1)) ? xb : xa,
                           (kind == ADD || (cc == 0 && !KG)) && fetching && n0 + (c + 1) * 32 <= N);
          }
        };
        if (output == PLAIN) pieces(std::integral_constant<int, PLAIN>{});
        else if (output == FP32) pieces(std::integral_constant<int, FP32>{});
        else if (output == ADD) pieces(std::integral_constant<int, ADD>{});
        else pieces(any);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(tempty_leader[acc]);
      ++local;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  // neither CTA may leave (or free tensor memory) while its partner can still signal its barriers
  // or while the leader's MMAs can still write into the partner's tensor memory
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<2>(warp_uniform(*tmem_slot), 2 * BN);
  }
}

int g_sms = 0;
int sm_count() {
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 148;
  }
  return g_sms;
}

// Counters of the dynamic tile scheduler: one pair per (device, stream), because launches on different streams can
// overlap. Allocated and zeroed on first use (never during a stream capture: such launches use the static schedule).
struct SchedWs {
  int dev;
  cudaStream_t stream;
  int* counters;
};
constexpr int SCHED_MAX_STREAMS = 16;
SchedWs g_sched_ws[SCHED_MAX_STREAMS];
int g_sched_n = 0;
int g_dynamic = -1;      // -1: read ATB_GEMM_DYNAMIC on first use (default on)
std::mutex g_sched_mu;

int* sched_counters(cudaStream_t stream) {
  // A graph may be replayed on any stream, beside launches of the one that it was captured on.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_sched_mu);
  int dev = 0;
  cudaGetDevice(&dev);
  for (int i = 0; i < g_sched_n; ++i)
    if (g_sched_ws[i].dev == dev && g_sched_ws[i].stream == stream) return g_sched_ws[i].counters;
  if (g_sched_n >= SCHED_MAX_STREAMS) return nullptr;
  void* p = nullptr;
  if (cudaMalloc(&p, 256) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (cudaMemsetAsync(p, 0, 256, stream) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(p);
    return nullptr;
  }
  g_sched_ws[g_sched_n++] = SchedWs{dev, stream, reinterpret_cast<int*>(p)};
  return reinterpret_cast<int*>(p);
}

// Clusters of four CTAs of the split kernel that run at a time (fewer than a quarter of the SMs where a GPC's number of
// them is no multiple of four); 0 if none. The same for all operand layouts: asked once.
int split_clusters() {
  static std::atomic<int> known{-1};
  int n = known.load(std::memory_order_relaxed);
  if (n >= 0) return n;
  auto kern = gemm_bf16_2cta_kernel<256, false, false, false, 2>;
  constexpr int smem = Cfg<256, 2>::SMEM_TOTAL;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(4 * sm_count(), 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 4;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known.store(n, std::memory_order_relaxed);
  return n;
}

// Whether two pairs per tile finish earlier than one, in waves of k-blocks: a wave of half tiles takes a tenth longer per
// k-block when all SMs load, the exchange at its end costs as much as 14 k-blocks (4 us), and a further tile, drawn by four CTAs,
// 1.5 more. Cold L2, one / two pairs (us), tiles and k-blocks: 8 x 172 59.4 / 43.0; 16 x 86 36.9 / 28.7; 32 x 86 36.9 / 30.7;
// 96 x 86 71.7 / 67.6; 96 x 172 124.9 / 110.6; about even: 80 x 64 55.3 / 55.3, 96 x 64 57.3 / 55.3; not: 80 x 58 51.2 / 53.2,
// 48 x 86 38.9 / 49.2, 104 x 86 73.7 / 81.9, 222 x 86 104.4 / 133.1.
// Beside a kernel that takes 24 SMs for itself fewer clusters of four find room than pairs: 16 x 86 36.9 / 32.8, 24 x 86 36.9 /
// 34.8, but 32 x 86 38.9 / 57.3, 96 x 86 73.7 / 92.2 (115.6 with a fixed share of tiles); one that takes 8, 96 x 86 73.7 /
// 67.6.
bool split_pays(int tiles, int kbs, int wish) {
  if (kbs < 2 || wish < 0) return false;
  const int pairs = sm_count() / 2;
  const long long whole = (long long)((tiles + pairs - 1) / pairs) * kbs;
  auto pays = [&](int clusters) {
    if (clusters <= 0) return false;
    const long long waves = (tiles + clusters - 1) / clusters;
    return wish > 0 || waves * ((kbs + 1) / 2) * 110 + 1400 + 150 * (waves - 1) < whole * 95;
  };
  return pays(pairs / 2) && pays(split_clusters());      // the second number takes a driver call: only where it can matter
}

template <int BN, bool A_MN, bool B_MN, bool KG = false, int SPLIT = 1>
int launch(const void* A, const void* B, const Epi& ep, int M, int N, int K, long long lda, long long ldb,
           int max_ctas, const Groups& grp, int b_extent_rows, const Gate& gate, const Ragged& rag, cudaStream_t stream,
           int* status, const KGroups<KG>& kg = KGroups<KG>()) {
  const int tile_cols = ep.gated ? BN / 2 : BN;
  int tiles = (rag.n > 0 ? rag.mt0[rag.n] : (M + 2 * BM - 1) / (2 * BM)) * ((N + tile_cols - 1) / tile_cols);
  if constexpr (KG) tiles *= kg.n;
  if constexpr (SPLIT == 1 && BN == 256 && !KG) {
    if (rag.n == 0 && grp.counts == nullptr && grp.b_rows == 0 && gate.flags == nullptr && ep.rs_rows <= 0 && max_ctas <= 0 &&
        split_pays(tiles, (K + BK - 1) / BK, ep.split))
      return launch<BN, A_MN, B_MN, KG, 2>(A, B, ep, M, N, K, lda, ldb, max_ctas, grp, b_extent_rows, gate, rag, stream, status,
                                           kg);
  }
  CUtensorMap tmA = {}, tmB = {}, tmC = {};
  bool ok = true;
  if (KG) {              // a map per group, made by the caller
  } else if (!A_MN)
    ok = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, K, lda, BM, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    ok = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, M, lda, BK, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (!ok) return -2;
  // with per-group B the tensor map spans all groups' weights (b_extent_rows rows)
  if (KG) {
  } else if (!B_MN)
    ok = make_tmap_2d(&tmB, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, b_extent_rows > 0 ? b_extent_rows : N, K, ldb,
                      Cfg<BN>::BNH, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    ok = make_tmap_2d(&tmB, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, b_extent_rows > 0 ? b_extent_rows : K,
                      ep.gated ? 2 * N : N, ldb, BK,
                      64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (!ok) return -3;
  Epi epw = ep;
  const long long out_bytes = ep.out_fp32 ? 4 : 2;
  epw.wide = ep.C != nullptr && ep.rs_rows <= 0 && N % 16 == 0 && (reinterpret_cast<uintptr_t>(ep.C) & 31) == 0 &&
             (ep.ldc * out_bytes) % 32 == 0 &&
             (ep.gu_out == nullptr || ((reinterpret_cast<uintptr_t>(ep.gu_out) & 31) == 0 && (ep.ldgu * 2) % 32 == 0));
  epw.boxed = SPLIT == 1 && ep.C != nullptr && ep.rs_rows <= 0 && ep.bias == nullptr && ep.residual == nullptr && !ep.accumulate &&
              !ep.out_fp32 && ep.alpha == 1.f && !ep.gated && ep.rope_cos == nullptr &&
              make_tmap_2d(&tmC, ep.C, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)M * kg_count(kg), N, ep.ldc, 32, 64,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  auto kern = gemm_bf16_2cta_kernel<BN, A_MN, B_MN, KG, SPLIT>;
  constexpr int SMEM_TOTAL = Cfg<BN, SPLIT>::SMEM_TOTAL;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL) != cudaSuccess) return -4;
    attr_set = true;
  }
  int clusters = SPLIT == 2 ? split_clusters() : sm_count() / 2;
  if (tiles < clusters) clusters = tiles;
  if (max_ctas > 0 && clusters > max_ctas / 2) clusters = max_ctas / 2 > 0 ? max_ctas / 2 : 1;
  // Dynamic tile scheduling for plain launches with more tiles than clusters (see Sched). A launch that waits for other ranks, and
  // one with a limit on its CTAs, keep the SMs that they leave free for what runs beside them, a transfer: the launch after
  // them would sit there and wait.
  Sched sched{nullptr, gate.flags == nullptr && max_ctas <= 0};
  if (g_dynamic < 0) {
    const char* e = getenv("ATB_GEMM_DYNAMIC");
    g_dynamic = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  if (g_dynamic > 0 && tiles > clusters && grp.counts == nullptr && (grp.b_rows == 0 || rag.n > 0) &&
      gate.flags == nullptr)
    sched.counters = sched_counters(stream);
  const cudaError_t e = launch_after(kern, dim3(2 * SPLIT * clusters), THREADS, SMEM_TOTAL, stream, 2 * SPLIT, tmA, tmB, tmC, epw, M,
                                     N, K, grp, gate, sched, rag, kg, status);
  return e == cudaSuccess ? 0 : -5;
}

const Ragged kNoGroups = {};

// extra arguments of the next launch of this host thread (set and cleared by atb_gemm_bf16_2cta_fused)
struct FusedArgs {
  bool active;
  Gate gate;
  float* rs_base[8];
  int rs_rows;
};
thread_local FusedArgs g_fused_args = {false, {nullptr, 0u, 1, 0}, {nullptr}, 0};

}  // namespace

// Same arguments as atb_gemm_bf16 (gemm_bf16.cu) minus the tile choice, plus row groups (see Groups):
// `group_counts` int32 device array or null with m_group_rows (multiple of 256) and / or k_group_rows
// (multiple of 64); b_group_rows > 0: every bm_group_rows rows of A use their own B out of n_b stacked
// ones, as described there. Best for M, N >= 256.
extern "C" int atb_gemm_bf16_2cta_grouped(const void* A, const void* B, void* C, const void* bias, int M, int N, int K,
                                          long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major,
                                          int out_fp32, int accumulate, float alpha, int tile_n, int max_ctas,
                                          const void* residual, long long ldr, const int* group_counts,
                                          int m_group_rows, int k_group_rows, int b_group_rows, int bm_group_rows,
                                          int n_b, void* stream, int* status) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldc & 3) || (!out_fp32 && (ldc & 7))) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return -1;
  if (residual != nullptr && (out_fp32 || (ldr & 7) || (reinterpret_cast<uintptr_t>(residual) & 15))) return -1;
  Groups grp{nullptr, 0, 0, 0, 0};
  int b_extent = 0;
  if ((m_group_rows % 256) || (k_group_rows % 64) || (bm_group_rows % 256) || m_group_rows < 0 ||
      k_group_rows < 0 || b_group_rows < 0)
    return -1;
  if (group_counts != nullptr) {
    grp.counts = group_counts;
    grp.m_rows = m_group_rows;
    grp.k_rows = k_group_rows;
  }
  if (b_group_rows > 0) {
    if (bm_group_rows <= 0 || n_b <= 0) return -1;
    grp.b_rows = b_group_rows;
    grp.bm_rows = bm_group_rows;
    b_extent = n_b * b_group_rows;
  }
  Epi ep{C, bias, ldc, alpha, out_fp32, accumulate, residual, ldr, {nullptr}, 0, 0, nullptr, 0};
  Gate gate{nullptr, 0u, 1, 0};
  if (g_fused_args.active) {   // set by atb_gemm_bf16_2cta_fused for this one launch
    gate = g_fused_args.gate;
    for (int i = 0; i < 8; ++i) ep.rs_base[i] = g_fused_args.rs_base[i];
    ep.rs_rows = g_fused_args.rs_rows;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // The 256-wide tile is the default. The 128-wide one fills short waves better, but per product of a pair it reads one and a
  // half times the operand bytes out of shared memory for the same work. Products of a 1.3B layer (hidden 2048, 5504),
  // 256 / 128 wide, cold L2: 4096 rows 83 / 124 (q|k|v), 131 / 203 (gate|up), 37 / 54 us (o); 1500 rows 39 / 55, 64 / 89,
  // 25 / 34; 777 rows 37 / 44, 50 / 66, 22.5 / 20.7. It wins only where the 256-wide tiles are fewer than the pairs, by 4 to
  // 9 % (333 rows, o: 22.5 / 20.5; 777 rows, dgrad of gate|up: 65.5 / 59.6), and not in weight gradients. It stays
  // selectable with tile_n = 128.
  const bool narrow = tile_n == 128;
  ep.split = tile_n == 256 ? -1 : tile_n == 512 ? 1 : 0;
#define ATB_PAIR_DISPATCH(BN_)                                                                                     \
  do {                                                                                                             \
    if (!a_mn_major && !b_mn_major)                                                                                \
      return launch<BN_, false, false>(A, B, ep, M, N, K, lda, ldb, max_ctas, grp, b_extent, gate, kNoGroups, st, status);  \
    if (!a_mn_major && b_mn_major)                                                                                 \
      return launch<BN_, false, true>(A, B, ep, M, N, K, lda, ldb, max_ctas, grp, b_extent, gate, kNoGroups, st, status);  \
    if (a_mn_major && b_mn_major)                                                                                  \
      return launch<BN_, true, true>(A, B, ep, M, N, K, lda, ldb, max_ctas, grp, b_extent, gate, kNoGroups, st, status);  \
    return launch<BN_, true, false>(A, B, ep, M, N, K, lda, ldb, max_ctas, grp, b_extent, gate, kNoGroups, st, status);  \
  } while (0)
  if (narrow) ATB_PAIR_DISPATCH(128);
  ATB_PAIR_DISPATCH(256);
#undef ATB_PAIR_DISPATCH
}

extern "C" int atb_gemm_bf16_2cta(const void* A, const void* B, void* C, const void* bias, int M, int N, int K,
                                  long long lda, long long ldb, long long ldc, int a_mn_major, int b_mn_major,
                                  int out_fp32, int accumulate, float alpha, int tile_n, int max_ctas,
                                  const void* residual, long long ldr, void* stream, int* status) {
  return atb_gemm_bf16_2cta_grouped(A, B, C, bias, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major, out_fp32,
                                    accumulate, alpha, tile_n, max_ctas, residual, ldr, nullptr, 0, 0, 0, 0, 0, stream,
                                    status);
}

// C[rows of group g] = A[rows of group g] * B_g^T for `n_groups` (at most 64) consecutive row groups of `sizes` rows
// (host memory, the sum is M) and as many stacked operands: B is [n_groups * N, K] (K-major) or [n_groups * K, N]
// (MN-major, K a multiple of 64 so that no k-block reaches into the next operand). A is K-major, C is bf16.
// One launch in place of one per group: the tiles of all groups share the waves. Experts of a routed layer get unequal
// numbers of rows, and a launch of its own leaves 74 CTA pairs with a short last wave once per expert. Forward and
// backward of the expert MLP 8 x 14336 x 4096 on 8192 routed rows: 8.5 ms, against 148 ms when every group whose
// length is no multiple of 8 took the fp32 fallback and w2 was transposed by a copy first.
// gated: every operand holds gate | up features (2 N of them), C [M, N] is silu(gate) * up and gu_out, if given,
// [M, 2 N] the two as they are, as in atb_gemm_bf16_2cta_swiglu below. Against this
// launch and the SwiGLU kernel after it, cold L2: 8192 rows, 8 x 14336 x 4096 1687 -> 1541 us, 4000 rows, 4 x 9024 x 4096
// 490 -> 450, 1000 rows, 4 x 8192 x 2048 103 -> 97.
extern "C" int atb_gemm_bf16_2cta_ragged(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                         long long ldb, long long ldc, int b_mn_major, const int* sizes, int n_groups,
                                         int gated, void* gu_out, void* stream, int* status) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldc & 7)) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(gu_out)) & 15)
    return -1;
  const int b_cols = gated ? 2 * N : N;
  if (n_groups < 1 || n_groups > RAGGED_MAX || (b_mn_major && (K % BK))) return -1;
  Ragged rag = {};
  rag.n = n_groups;
  for (int g = 0; g < n_groups; ++g) {
    if (sizes[g] < 0 || sizes[g] > M - rag.row0[g]) return -1;
    rag.row0[g + 1] = rag.row0[g] + sizes[g];
    rag.mt0[g + 1] = rag.mt0[g] + (sizes[g] + 2 * BM - 1) / (2 * BM);
  }
  if (rag.row0[n_groups] != M) return -1;
  Epi ep{C, nullptr, ldc, 1.f, 0, 0, nullptr, 0, {nullptr}, 0, gated != 0, gated ? gu_out : nullptr, b_cols};
  Groups grp{nullptr, 0, b_mn_major ? K : b_cols, 0, 0};
  Gate gate{nullptr, 0u, 1, 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (b_mn_major)
    return launch<256, false, true>(A, B, ep, M, N, K, lda, ldb, 0, grp, n_groups * K, gate, rag, st, status);
  return launch<256, false, false>(A, B, ep, M, N, K, lda, ldb, 0, grp, n_groups * b_cols, gate, rag, st, status);
}

// C[g] (+)= A_g^T B_g for `n_groups` consecutive row groups of `sizes` rows (host memory, T in all): A [T, M] and B [T, N]
// hold the groups' rows, C [n_groups, M, N] is bf16 or fp32 (see KGroups).
extern "C" int atb_gemm_bf16_2cta_kgroups(const void* A, const void* B, void* C, int M, int N, int T, long long lda,
                                          long long ldb, const int* sizes, int n_groups, int out_fp32, int accumulate,
                                          void* stream, int* status) {
  if (M <= 0 || N <= 0 || n_groups <= 0) return 0;
  if ((M & 7) || (N & 7) || (lda & 7) || (ldb & 7) || T < 0) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -1;
  const Groups grp{nullptr, 0, 0, 0, 0};
  const Gate gate{nullptr, 0u, 1, 0};
  long long row = 0;
  for (int g = 0; g < n_groups; ++g) {
    if (sizes[g] < 0 || sizes[g] > T - row) return -1;
    row += sizes[g];
  }
  if (row != T) return -1;
  row = 0;
  for (int g0 = 0; g0 < n_groups; g0 += KGROUP_MAX) {
    KGroups<true> kg = {};
    kg.n = n_groups - g0 < KGROUP_MAX ? n_groups - g0 : KGROUP_MAX;
    for (int i = 0; i < kg.n; ++i) {
      kg.rows[i] = sizes[g0 + i];
      if (kg.rows[i] == 0) continue;
      if (!make_tmap_2d(&kg.a[i], reinterpret_cast<const __nv_bfloat16*>(A) + row * lda, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                        kg.rows[i], M, lda, BK, 64, CU_TENSOR_MAP_SWIZZLE_128B))
        return -2;
      if (!make_tmap_2d(&kg.b[i], reinterpret_cast<const __nv_bfloat16*>(B) + row * ldb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                        kg.rows[i], N, ldb, BK, 64, CU_TENSOR_MAP_SWIZZLE_128B))
        return -3;
      row += kg.rows[i];
    }
    char* c = reinterpret_cast<char*>(C) + (long long)g0 * M * N * (out_fp32 ? 4 : 2);
    Epi ep{c, nullptr, N, 1.f, out_fp32, accumulate, nullptr, 0, {nullptr}, 0, 0, nullptr, 0};
    const int rc = launch<256, true, true, true>(A, B, ep, M, N, T, lda, ldb, 0, grp, 0, gate, kNoGroups,
                                                 reinterpret_cast<cudaStream_t>(stream), status, kg);
    if (rc != 0) return rc;
  }
  return 0;
}

// out[M, N] = rope(x W^T): the projection onto fused q | k | v heads with the first rope_heads heads of head_dim (128 or
// 64) columns rotated in the epilogue (see Epi; the values are rotated before they are rounded). W is [N, K] K-major with
// rows for whole heads, N a multiple of 128; cos / sin [rope_s, head_dim / 2] fp32, 16-byte aligned; pos may be null.
// The separate kernel read and wrote the q and k heads again: 24 us after a 290 us product at 4096 x 12288 x 4096, and a
// launch per layer. Loss without gradients of 8 layers of a 1.3B model on one odd batch: 2536 -> 2350 us, of which
// 27 us are device time (1495 -> 1468) and the rest is the launches.
extern "C" int atb_gemm_bf16_2cta_rope(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                       long long ldb, long long ldc, const float* cos_t, const float* sin_t,
                                       const int* pos, int rope_s, int rope_heads, int head_dim, void* stream,
                                       int* status) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 127) || (lda & 7) || (ldb & 7) || (ldc & 7) || (head_dim != 128 && head_dim != 64) || rope_s < 1 ||
      rope_heads < 0 || (rope_heads * head_dim) % 128 || rope_heads * head_dim > N)
    return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15)
    return -1;
  Epi ep = {};
  ep.C = C;
  ep.ldc = ldc;
  ep.alpha = 1.f;
  ep.rope_cos = cos_t;
  ep.rope_sin = sin_t;
  ep.rope_pos = pos;
  ep.rope_s = rope_s;
  ep.rope_dim = head_dim;
  ep.rope_cols = rope_heads * head_dim;
  Groups grp{nullptr, 0, 0, 0, 0};
  Gate gate{nullptr, 0u, 1, 0};
  return launch<256, false, false>(A, B, ep, M, N, K, lda, ldb, 0, grp, 0, gate, kNoGroups,
                                   reinterpret_cast<cudaStream_t>(stream), status);
}

// act[M, F] = silu(x Wg^T) * (x Wu^T) for the fused weight W = [Wg; Wu] ([2 F, K], K-major, pitch ldb): the GEMM with
// the gated epilogue (see Epi). gu_out (optional, [M, 2 F] bf16, pitch ldgu) receives the gate and up values the
// backward pass needs. F % 8 == 0; x is [M, K] K-major with pitch lda.
extern "C" int atb_gemm_bf16_2cta_swiglu(const void* A, const void* B, void* act, void* gu_out, int M, int F, int K,
                                         long long lda, long long ldb, long long ld_act, long long ldgu, void* stream,
                                         int* status) {
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if ((F & 7) || (lda & 7) || (ldb & 7) || (ld_act & 7) || (gu_out != nullptr && (ldgu & 7))) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(act) |
       reinterpret_cast<uintptr_t>(gu_out)) & 15)
    return -1;
  Epi ep{act, nullptr, ld_act, 1.f, 0, 0, nullptr, 0, {nullptr}, 0, 1, gu_out, ldgu};
  Groups grp{nullptr, 0, 0, 0, 0};
  Gate gate{nullptr, 0u, 1, 0};
  return launch<256, false, false>(A, B, ep, M, F, K, lda, ldb, 0, grp, 2 * F, gate, kNoGroups,
                                   reinterpret_cast<cudaStream_t>(stream), status);
}

// Weight all-gather -> GEMM (a linear layer whose weight is sharded by rows over the ranks): C = A B^T with
// B [N, K] K-major arriving in shards of gate_rows rows (a multiple of 128); shard g is in place once
// gate_flags[g] >= gate_epoch. Tiles start at column gate_first_row (a multiple of 256: this rank's own shard).
extern "C" int atb_gemm_bf16_2cta_wgather(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                          long long ldb, long long ldc, const unsigned int* gate_flags,
                                          unsigned int gate_epoch, int gate_rows, int gate_first_row, void* stream,
                                          int* status) {
  if (gate_flags == nullptr || gate_rows <= 0 || (gate_rows % 128) || gate_first_row < 0 || (gate_first_row % 256))
    return -1;
  FusedArgs fa = {true, {gate_flags, gate_epoch, gate_rows, gate_first_row / 256, 1}, {nullptr}, 0};
  g_fused_args = fa;
  const int rc = atb_gemm_bf16_2cta_grouped(A, B, C, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, 0, 1.f, 0, 0, nullptr, 0,
                                            nullptr, 0, 0, 0, 0, 0, stream, status);
  g_fused_args.active = false;
  return rc;
}

// 1 / 0: hand tiles out dynamically or by a fixed stride (default: dynamic unless ATB_GEMM_DYNAMIC=0).
extern "C" void atb_gemm_set_dynamic(int on) { g_dynamic = on ? 1 : 0; }

// Upper bound of the arrival-flag waits of the all-gather -> GEMM form, in nanoseconds (default 2 s).
extern "C" int atb_set_gate_wait_ns(unsigned long long ns) {
  return cudaMemcpyToSymbol(g_gate_wait_ns, &ns, sizeof(ns)) == cudaSuccess ? 0 : -5;
}

// The GEMM fused with a collective (see the file header). On top of atb_gemm_bf16_2cta:
//   gate_flags != null : all-gather -> GEMM. A's rows arrive in shards of gate_rows rows (a multiple of 128);
//                        shard g is in place once gate_flags[g] >= gate_epoch; tiles start at row gate_first_row.
//   rs_ptrs != null    : GEMM -> reduce-scatter. rs_ptrs = `rs_world` device addresses of the ranks' fp32
//                        accumulation buffers [rs_rows, N] (pitch ldc); output row r is added into rank
//                        r / rs_rows' buffer. C may be null.
extern "C" int atb_gemm_bf16_2cta_fused(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                        long long ldb, long long ldc, int a_mn_major, int b_mn_major, float alpha,
                                        const unsigned int* gate_flags, unsigned int gate_epoch, int gate_rows,
                                        int gate_first_row, const unsigned long long* rs_ptrs, int rs_world,
                                        int rs_rows, void* stream, int* status) {
  FusedArgs fa = {true, {nullptr, 0u, 1, 0}, {nullptr}, 0};
  if (gate_flags != nullptr) {
    if (gate_rows <= 0 || (gate_rows % 128) || a_mn_major || gate_first_row < 0 || (gate_first_row % 256)) return -1;
    fa.gate = Gate{gate_flags, gate_epoch, gate_rows, gate_first_row / 256};
  }
  void* c_arg = C;
  int out_fp32 = 0;
  if (rs_ptrs != nullptr) {
    if (rs_world < 1 || rs_world > 8 || rs_rows <= 0 || (long long)rs_rows * rs_world < M) return -1;
    for (int i = 0; i < rs_world; ++i) fa.rs_base[i] = reinterpret_cast<float*>(rs_ptrs[i]);
    fa.rs_rows = rs_rows;
    c_arg = fa.rs_base[0];     // only its alignment is checked; the epilogue never writes through it
    out_fp32 = 1;
  }
  g_fused_args = fa;
  const int rc = atb_gemm_bf16_2cta_grouped(A, B, c_arg, nullptr, M, N, K, lda, ldb, ldc, a_mn_major, b_mn_major,
                                            out_fp32, 0, alpha, 0, 0, nullptr, 0, nullptr, 0, 0, 0, 0, 0, stream,
                                            status);
  g_fused_args.active = false;
  return rc;
}
