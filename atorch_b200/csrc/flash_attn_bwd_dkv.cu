// Flash attention backward, key/value-gradient kernel for sm_100a (head dim 128 or 64, bf16), tcgen05 + TMEM + TMA.
//
// One CTA per (128 keys, key/value head, batch) walks the query blocks that can see its keys, for all query heads of
// the group, and accumulates dV and dK in tensor memory:
//   S  = Q K^T,  dP = dO V^T                      smem x smem -> TMEM   (lane = query, column = key)
//   P  = exp2(S c - lse),  dS = P (dP - delta) s    registers -> bf16 tiles in swizzled shared memory
//   dV += P^T dO,  dK += dS^T Q                    smem x smem (MN-major both) -> TMEM
// A [rows][64] bf16 panel with 128-byte swizzle is at the same time a K-major tile of the matrix and an MN-major tile of
// its transpose, so P, dS, Q and dO are each stored once and read both ways. TMEM: S | dP | dV | dK.
// The query gradient comes from flash_attn_bwd_dq.cu.
//
// The element-wise warps bound the kernel, so the tensor core works around them:
//   S(i+1) is issued as soon as the warps hold S(i) in registers and runs under the exponentials of block i,
//   dV(i) starts when P(i) is stored and runs under dS(i),
//   dK(i), dP(i+1) run under the exponentials of block i+1.
// S=8192, 32 heads of 128, causal: 822 us (861 with a CTA per block; 1188 when S(i+1) was issued after P and dS were both
// stored); 2800 clocks a block, 1024 of them exponentials. For long causal inputs P^T and dS^T once went through tensor memory
// instead, whose element-wise warps need the row statistics per column.
// For grouped queries the gradients of the group are summed in the accumulator in fp32; with one CTA per query head the
// bf16 results have to be added by a separate pass over them.
//
// Warp 0 = TMA producer, warp 1 = MMA issuer / TMEM owner, warp 10 = scheduler (block_queue.cuh), warps 2..9 = element-wise
// work: thread (row r, half h) owns columns [64h, 64h+64) of row r. Masks are per-row key intervals [lo, hi) as in the forward
// kernel.
#include "block_queue.cuh"

namespace {
using namespace atb;

constexpr int BQ = 128, BKV = 128;
constexpr int PANEL = 128 * 64 * 2;
constexpr int EW_TILE = 2 * PANEL;      // P, dS: [128 queries][128 keys]
constexpr int N_EW = 256;
constexpr int THREADS = 96 + N_EW;
constexpr int SCHED_WARP = 10;

struct DkvParams {
  const float* lse;    // [B, Hq, Sq]
  const float* delta;  // [B, Hq, Sq]
  __nv_bfloat16* dk;   // token-major, head h at columns [h*HD, h*HD+HD) of a row of pitch dkv_stride
  __nv_bfloat16* dv;
  long long dkv_stride;
  const int* row_lo;
  const int* row_hi;
  int B, Sq, Sk, Hq, Hkv, causal;
  const int2* key_range;   // [B, query blocks]: first, last+1 key that a row of the block sees (null with the intervals)
  int fold;            // query heads per CTA, a divisor of Hq / Hkv: Hq / Hkv (gradients of a key/value head) down to 1
  int wide;            // rows of dk and dv start on 32-byte boundaries
  float scale, scale_log2;
  int* status;
  BlockOrder order;
};

template <int HD>
struct SmemK {
  static constexpr int TILE = (HD / 64) * PANEL;
  static constexpr int DO_STAGES = HD == 128 ? 1 : 2;       // shared memory is full at head dim 128
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = K_OFF + TILE;
  static constexpr int Q_OFF = V_OFF + TILE;                // two stages
  static constexpr int DO_OFF = Q_OFF + 2 * TILE;
  static constexpr int P_OFF = DO_OFF + DO_STAGES * TILE;
  static constexpr int DS_OFF = P_OFF + EW_TILE;
  static constexpr int BAR_OFF = DS_OFF + EW_TILE;          // 224 KB at head dim 128
  static constexpr int NBARS = 2 + 4 + 4 + 8;
  static constexpr int QUEUE_OFF = BAR_OFF + NBARS * 8 + 16;
  static constexpr int TOTAL = QUEUE_OFF + (int)sizeof(WorkQueue) + 1024;
};
static_assert(SmemK<128>::QUEUE_OFF % 16 == 0 && SmemK<64>::QUEUE_OFF % 16 == 0, "the queue is 16-byte aligned");
static_assert(SmemK<128>::TOTAL <= 232448, "shared memory of the dK/dV kernel exceeds 227 KB");

struct RowInfo {       // one query row as the element-wise thread sees it; -inf as lse: takes no part (P becomes 0)
  float lse, delta;
  int lo, hi;          // key interval
};

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, DkvParams p) {
  using L = SmemK<HD>;
  constexpr int TILE = L::TILE, DO_STAGES = L::DO_STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem + L::K_OFF;
  uint8_t* sV = smem + L::V_OFF;
  uint8_t* sQ = smem + L::Q_OFF;
  uint8_t* sdO = smem + L::DO_OFF;
  uint8_t* sP = smem + L::P_OFF;
  uint8_t* sdS = smem + L::DS_OFF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* kv_full = bars;
  uint64_t* kv_free = bars + 1;    // the last S and dP of a unit have read K and V
  uint64_t* q_full = bars + 2;     // [2]
  uint64_t* q_free = bars + 4;     // [2]  dK(i) has read Q(i)
  uint64_t* do_full = bars + 6;    // [DO_STAGES]
  uint64_t* do_free = bars + 8;    // [DO_STAGES]  dV(i) has read dO(i)
  uint64_t* s_full = bars + 10;    // S(i) is in TMEM
  uint64_t* s_read = bars + 11;    // every element-wise warp holds S(i) in registers
  uint64_t* dp_full = bars + 12;   // dP(i) is in TMEM
  uint64_t* p_full = bars + 13;    // P(i) is in shared memory
  uint64_t* ds_full = bars + 14;   // dS(i) is in shared memory, dP(i) has been read
  uint64_t* p_free = bars + 15;    // dV(i) has read P(i)
  uint64_t* ds_free = bars + 16;   // dK(i) has read dS(i)
  uint64_t* acc_free = bars + 17;  // dV and dK of a unit have been read out of TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  WorkQueue* queue = reinterpret_cast<WorkQueue*>(smem + L::QUEUE_OFF);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int shift = p.Sk - p.Sq;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(kv_free, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1); mbar_init(&q_free[i], 1);
      mbar_init(&do_full[i], 1); mbar_init(&do_free[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_read, N_EW / 32);
    mbar_init(dp_full, 1);
    mbar_init(p_full, N_EW / 32);
    mbar_init(ds_full, N_EW / 32);
    mbar_init(p_free, 1);
    mbar_init(ds_free, 1);
    mbar_init(acc_free, N_EW / 32);
    queue_init(queue, 2 + N_EW / 32);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc<1>(tmem_slot, 512);
    tmem_relinquish<1>();
    if (lane == 0) grid_go();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_wait();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  // Units of this CTA, one after another: key block w.place (the first is the heaviest) of head w.head of the results and
  // sample w.sample, query blocks [w.v0, w.v0 + w.v1). Block i of a unit: query block v0 + i % v1 of query head
  // head * fold + i / v1. Barriers of the blocks count on through all units (g), those of K, V and the accumulators count
  // the units that have any block (u).
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 384;

  if (warp == SCHED_WARP) {
    queue_run(queue, p.order, [&](Work& w, int) {
      // query blocks that see this block of keys
      const int kv0 = w.place * BKV, nqb = (p.Sq + BQ - 1) / BQ;
      if (p.key_range == nullptr) {
        const int rmin = p.causal ? max(0, kv0 - shift) : 0;
        w.v0 = rmin / BQ;
        w.v1 = rmin < p.Sq ? nqb - w.v0 : 0;
      } else {
        int first = nqb, end = 0;
        for (int i = lane; i < nqb; i += 32) {
          const int2 r = p.key_range[(long long)w.sample * nqb + i];
          if (max(r.x, kv0) < min(min(r.y, p.Sk), kv0 + BKV)) { first = min(first, i); end = i + 1; }
        }
        w.v0 = __reduce_min_sync(0xffffffffu, first);
        w.v1 = max(__reduce_max_sync(0xffffffffu, end) - w.v0, 0);
      }
    }, abort_flag, p.status);
  } else if (warp == 0) {
    const bool el = elect_one();
    if (el) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
    uint32_t g = 0;
    int u = 0;
    Work w;
    for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
      const int n = w.v1 * p.fold;
      if (n == 0) { queue_claim(queue); continue; }
      int h = w.head * p.fold, qb = 0;
      const int hk = h / (p.Hq / p.Hkv);
      const int krow = (int)((long long)w.sample * p.Sk + w.place * BKV);
      if (!mbar_wait_warp(kv_free, (u & 1) ^ 1, abort_flag, p.status)) break;
      ++u;
      if (el) {
        mbar_expect_tx(kv_full, 2 * TILE);
#pragma unroll
        for (int c2 = 0; c2 < HD / 64; ++c2) {
          tma_load_2d(sK + c2 * PANEL, &tmK, kv_full, hk * HD + c2 * 64, krow);
          tma_load_2d(sV + c2 * PANEL, &tmV, kv_full, hk * HD + c2 * 64, krow);
        }
      }
      bool ok = true;
      for (int it = 0; it < n; ++it, ++g) {
        if (it == max(n - 3, 0)) queue_claim(queue);
        const int qs = g & 1, ds = g % DO_STAGES;
        const int qrow = (int)((long long)w.sample * p.Sq + (long long)(w.v0 + qb) * BQ);
        ok = mbar_wait_warp(&q_free[qs], ((g >> 1) & 1) ^ 1, abort_flag, p.status);
        if (!ok) break;
        if (el) {
          mbar_expect_tx(&q_full[qs], TILE);
#pragma unroll
          for (int c2 = 0; c2 < HD / 64; ++c2)
            tma_load_2d(sQ + qs * TILE + c2 * PANEL, &tmQ, &q_full[qs], h * HD + c2 * 64, qrow);
        }
        ok = mbar_wait_warp(&do_free[ds], ((g / DO_STAGES) & 1) ^ 1, abort_flag, p.status);
        if (!ok) break;
        if (el) {
          mbar_expect_tx(&do_full[ds], TILE);
#pragma unroll
          for (int c2 = 0; c2 < HD / 64; ++c2)
            tma_load_2d(sdO + ds * TILE + c2 * PANEL, &tmdO, &do_full[ds], h * HD + c2 * 64, qrow);
        }
        if (++qb == w.v1) { qb = 0; ++h; }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    const uint32_t el = elect_one();   // the lane that issues and commits
    constexpr uint32_t id_kk = umma_idesc(128, 128, 1, 1, false, false);
    constexpr uint32_t id_mm = umma_idesc(128, HD, 1, 1, true, true);      // dV, dK: [keys x d]
    const uint32_t dQk = umma_desc_lo(smem_u32(sQ), 16), dQm = umma_desc_lo(smem_u32(sQ), PANEL);
    const uint32_t dOk = umma_desc_lo(smem_u32(sdO), 16), dOm = umma_desc_lo(smem_u32(sdO), PANEL);
    const uint32_t dKk = umma_desc_lo(smem_u32(sK), 16), dVk = umma_desc_lo(smem_u32(sV), 16);
    const uint32_t dPm = umma_desc_lo(smem_u32(sP), PANEL), dSm = umma_desc_lo(smem_u32(sdS), PANEL);
    auto issue_s = [&](uint32_t g) -> bool {   // S(g) = Q(g) K^T over d
      if (!mbar_wait_warp(&q_full[g & 1], (g >> 1) & 1, abort_flag, p.status)) return false;
      const uint32_t qd = dQk + (((g & 1) * TILE) >> 4);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
        const uint32_t off = ((k >> 2) * PANEL + (k & 3) * 32) >> 4;
        umma_ss_issue(tS, qd + off, dKk + off, id_kk, k != 0, el);
      }
      umma_commit_issue(s_full, el);
      return true;
    };
    auto issue_dp = [&](uint32_t g, bool last) -> bool {  // dP(g) = dO(g) V^T over d
      const int ds = g % DO_STAGES;
      if (!mbar_wait_warp(&do_full[ds], (g / DO_STAGES) & 1, abort_flag, p.status)) return false;
      const uint32_t od = dOk + ((ds * TILE) >> 4);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
        const uint32_t off = ((k >> 2) * PANEL + (k & 3) * 32) >> 4;
        umma_ss_issue(tdP, od + off, dVk + off, id_kk, k != 0, el);
      }
      umma_commit_issue(dp_full, el);
      if (last) umma_commit_issue(kv_free, el);
      return true;
    };
    uint32_t g = 0;
    int u = 0;
    Work w;
    for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
      const int n = w.v1 * p.fold;
      if (n == 0) continue;
      // the first scores of a unit follow the last products of the one before and run under its results' way out
      bool ok = mbar_wait_warp(kv_full, u & 1, abort_flag, p.status) &&
                (g == 0 || mbar_wait_warp(s_read, (g - 1) & 1, abort_flag, p.status));
      tc_fence_after();
      ok = ok && issue_s(g) && issue_dp(g, n == 1);
      for (int it = 0; ok && it < n; ++it, ++g) {
        if (it + 1 < n) {
          ok = mbar_wait_warp(s_read, g & 1, abort_flag, p.status);
          tc_fence_after();
          ok = ok && issue_s(g + 1);
        }
        if (ok && it == 0 && u > 0) ok = mbar_wait_warp(acc_free, (u - 1) & 1, abort_flag, p.status);
        ok = ok && mbar_wait_warp(p_full, g & 1, abort_flag, p.status);
        if (!ok) break;
        tc_fence_after();
        const int ds = g % DO_STAGES;
        const uint32_t om = dOm + ((ds * TILE) >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)  // dV += P^T dO over q
          umma_ss_issue(tdV, dPm + k * 128, om + k * 128, id_mm, (it | k) != 0, el);
        umma_commit_issue(&do_free[ds], el);
        umma_commit_issue(p_free, el);
        ok = mbar_wait_warp(ds_full, g & 1, abort_flag, p.status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t qm = dQm + (((g & 1) * TILE) >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)  // dK += dS^T Q over q
          umma_ss_issue(tdK, dSm + k * 128, qm + k * 128, id_mm, (it | k) != 0, el);
        umma_commit_issue(&q_free[g & 1], el);
        umma_commit_issue(ds_free, el);
        if (it + 1 < n) ok = issue_dp(g + 1, it + 2 == n);
      }
      if (!ok) break;
      ++u;
    }
  } else {
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = ((uint32_t)(quarter * 32) << 16);
    uint8_t* prow = sP + half * PANEL + r * 128;
    uint8_t* dsrow = sdS + half * PANEL + r * 128;
    // values of a row of sample b: loads only, used one block later
    auto row_info = [&](int b, int h, int i, bool any) -> RowInfo {
      RowInfo ri{-INFINITY, 0.f, 0, p.Sk};
      if (any && i < p.Sq) {
        const long long ridx = ((long long)b * p.Hq + h) * p.Sq + i;
        ri.lse = p.lse[ridx];
        ri.delta = p.delta[ridx];
        if (p.causal) ri.hi = i + 1 + shift;
        if (p.row_lo) ri.lo = p.row_lo[(long long)b * p.Sq + i];
        if (p.row_hi) ri.hi = p.row_hi[(long long)b * p.Sq + i];
      }
      return ri;
    };
    // the first row of a unit: the loads go out before the results of the one before are stored
    auto first_row = [&](const Work& w) -> RowInfo {
      return row_info(w.sample, w.head * p.fold, w.v0 * BQ + r, w.more && w.v1 > 0);
    };
    uint32_t g = 0;
    bool ok = queue_wait(queue, 0, abort_flag, p.status);
    RowInfo raw = ok ? first_row(queue_read(queue, 0)) : RowInfo{};
    for (int c = 0; ok; ++c) {
      const Work w = queue_read(queue, c);
      if (!w.more) break;
      const int b = w.sample, ho = w.head, kv0 = w.place * BKV, n = w.v1 * p.fold;
      const int c0 = kv0 + half * 64;              // first key of this thread
      int h = ho * p.fold, qb = 0;
      for (int it = 0; it < n; ++it, ++g) {
        const bool valid = raw.lse != -INFINITY;
        const float lse2 = valid ? raw.lse * 1.4426950408889634f : 0.f, delta = valid ? raw.delta : 0.f;
        const int lo = max(raw.lo, 0), hi = valid ? min(raw.hi, p.Sk) : 0;
        // this block's values are out of `raw` before the loads of the next block's are issued: with both in flight the wait
        // for the old ones also waited for the new ones, 500 to 700 clocks per block
        asm volatile("" ::"f"(lse2), "f"(delta), "r"(lo), "r"(hi) : "memory");
        if (++qb == w.v1) { qb = 0; ++h; }
        raw = row_info(b, h, (w.v0 + qb) * BQ + r, it + 1 < n);
        // ---- P(g) = exp2(S c - lse)
        // warp-uniform, so that the interval tests are a separate path that full tiles never enter
        const bool row_full = __all_sync(0xffffffffu, lo <= kv0 && hi >= kv0 + BKV);
        if (!mbar_wait_warp(s_full, g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        float pv[64];
        {
          uint32_t s0[32], s1[32];
          tmem_ld_32x32(tS + lane_addr + half * 64, s0);
          tmem_ld_32x32(tS + lane_addr + half * 64 + 32, s1);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_read);
          const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2), nl2 = f2_pack(-lse2, -lse2);
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float a0, a1, b0, b1;
            f2_unpack(f2_fma(f2_pack_bits(s0[c], s0[c + 1]), sc2, nl2), a0, a1);
            f2_unpack(f2_fma(f2_pack_bits(s1[c], s1[c + 1]), sc2, nl2), b0, b1);
            pv[c] = fast_exp2(a0); pv[c + 1] = fast_exp2(a1);
            pv[32 + c] = fast_exp2(b0); pv[33 + c] = fast_exp2(b1);
          }
          if (!row_full) {
            const uint32_t m0 = visible_keys(c0, lo, hi), m1 = visible_keys(c0 + 32, lo, hi);
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (!(m0 & (1u << c))) pv[c] = 0.f;
              if (!(m1 & (1u << c))) pv[32 + c] = 0.f;
            }
          }
        }
        // dV(g-1) has read P(g-1)
        if (g > 0 && !mbar_wait_warp(p_free, (g - 1) & 1, abort_flag, p.status)) { ok = false; break; }
#pragma unroll
        for (int c8 = 0; c8 < 8; ++c8) {
          const int c = c8 * 8, slot = (c8 ^ (r & 7)) << 4;
          *reinterpret_cast<uint4*>(prow + slot) =
              make_uint4(pack_bf16x2(pv[c], pv[c + 1]), pack_bf16x2(pv[c + 2], pv[c + 3]),
                         pack_bf16x2(pv[c + 4], pv[c + 5]), pack_bf16x2(pv[c + 6], pv[c + 7]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
        // ---- dS(g) = P (dP - delta) scale
        if (!mbar_wait_warp(dp_full, g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        uint32_t ds[32];
        {
          uint32_t d0[32], d1[32];
          tmem_ld_32x32(tdP + lane_addr + half * 64, d0);
          tmem_ld_32x32(tdP + lane_addr + half * 64 + 32, d1);
          tmem_ld_wait();
          const uint64_t nd2 = f2_pack(-delta, -delta), scl2 = f2_pack(p.scale, p.scale);
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float x0, x1, y0, y1;
            f2_unpack(f2_mul(f2_mul(f2_pack(pv[c], pv[c + 1]), scl2), f2_add(f2_pack_bits(d0[c], d0[c + 1]), nd2)), x0, x1);
            f2_unpack(f2_mul(f2_mul(f2_pack(pv[32 + c], pv[33 + c]), scl2), f2_add(f2_pack_bits(d1[c], d1[c + 1]), nd2)),
                      y0, y1);
            ds[c >> 1] = pack_bf16x2(x0, x1);
            ds[16 + (c >> 1)] = pack_bf16x2(y0, y1);
          }
        }
        // dK(g-1) has read dS(g-1)
        if (g > 0 && !mbar_wait_warp(ds_free, (g - 1) & 1, abort_flag, p.status)) { ok = false; break; }
#pragma unroll
        for (int c8 = 0; c8 < 8; ++c8)
          *reinterpret_cast<uint4*>(dsrow + ((c8 ^ (r & 7)) << 4)) =
              make_uint4(ds[4 * c8], ds[4 * c8 + 1], ds[4 * c8 + 2], ds[4 * c8 + 3]);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
      }
      if (!ok) break;
      // the next unit is known and its first values are on their way before this one's results leave
      ok = queue_wait(queue, c + 1, abort_flag, p.status);
      if (!ok) break;
      raw = first_row(queue_read(queue, c + 1));
      if (n > 0)
        ok = mbar_wait_warp(p_free, (g - 1) & 1, abort_flag, p.status) &&
             mbar_wait_warp(ds_free, (g - 1) & 1, abort_flag, p.status);
      if (!ok) break;
      // dV / dK of this key block: TMEM lane = key row. tcgen05.ld is a warp-wide (.sync.aligned)
      // instruction: every lane executes it, only the global stores are predicated per row.
      const Work again = queue_read(queue, c);
      const int j = again.place * BKV + r;
      const long long at = ((long long)again.sample * p.Sk + j) * p.dkv_stride + again.head * HD + half * (HD / 2);
      if (n > 0) tc_fence_after();
#pragma unroll
      for (int cc = 0; cc < HD / 64; ++cc) {
        uint32_t tv[32], tk[32];
        if (n > 0) {
          tmem_ld_32x32(tdV + lane_addr + half * (HD / 2) + cc * 32, tv);
          tmem_ld_32x32(tdK + lane_addr + half * (HD / 2) + cc * 32, tk);
          tmem_ld_wait();
          if (cc == HD / 64 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) { tv[i] = 0u; tk[i] = 0u; }
        }
        if (j < p.Sk) {
          store_bf16_32(p.dv + at + cc * 32, tv, p.wide);
          store_bf16_32(p.dk + at + cc * 32, tk, p.wide);
        }
      }
      queue_free(queue, c);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

template <int HD>
int launch_dkv(const void* dout, const void* q, const void* k, const void* v, DkvParams p, long long q_stride,
               long long k_stride, long long v_stride, long long do_stride, cudaStream_t stream) {
  CUtensorMap tmQ, tmdO, tmK, tmV;
  const auto bf16 = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  if (!make_tmap_2d(&tmQ, q, bf16, 2, (uint64_t)p.B * p.Sq, (uint64_t)p.Hq * HD, q_stride, BQ, 64, sw) ||
      !make_tmap_2d(&tmdO, dout, bf16, 2, (uint64_t)p.B * p.Sq, (uint64_t)p.Hq * HD, do_stride, BQ, 64, sw) ||
      !make_tmap_2d(&tmK, k, bf16, 2, (uint64_t)p.B * p.Sk, (uint64_t)p.Hkv * HD, k_stride, BKV, 64, sw) ||
      !make_tmap_2d(&tmV, v, bf16, 2, (uint64_t)p.B * p.Sk, (uint64_t)p.Hkv * HD, v_stride, BKV, 64, sw))
    return -2;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_bwd_dkv_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemK<HD>::TOTAL) !=
        cudaSuccess)
      return -4;
    attr_set = true;
  }
  dim3 grid;
  make_block_order(&p.order, &grid, (p.Sk + BKV - 1) / BKV, p.Hq / p.fold, p.B, p.causal != 0, p.Sq, HD);
  launch_after(flash_bwd_dkv_kernel<HD>, grid, THREADS, SmemK<HD>::TOTAL, stream, 1, tmQ, tmdO, tmK, tmV, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace

// dk, dv: token-major rows of pitch dkv_stride elements, one head per `fold` query heads (fold == Hq / Hkv: the
// gradients of a key/value head; below, the caller sums what is left of a group); lse, delta: [B, Hq, Sq] fp32.
extern "C" int atb_flash_bwd_dkv(const void* dout, const void* q, const void* k, const void* v, const float* lse,
                                 const float* delta, void* dk, void* dv, const int* row_lo, const int* row_hi, int B,
                                 int Sq, int Sk, int Hq, int Hkv, long long q_stride, long long k_stride,
                                 long long v_stride, long long do_stride, long long dkv_stride, int causal,
                                 float softmax_scale, int fold, int head_dim, const int* key_range, void* stream,
                                 int* status) {
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if (Hq % Hkv || fold < 1 || (Hq / Hkv) % fold || (head_dim != 128 && head_dim != 64)) return -1;
  if ((q_stride | k_stride | v_stride | do_stride | dkv_stride) & 7) return -1;
  DkvParams p;
  p.lse = lse; p.delta = delta; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv; p.dkv_stride = dkv_stride;
  p.row_lo = row_lo; p.row_hi = row_hi;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal;
  p.fold = fold;
  p.key_range = reinterpret_cast<const int2*>(key_range);
  p.wide = ((reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 31) == 0 && (dkv_stride & 15) == 0;
  p.scale = softmax_scale; p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  return head_dim == 64
             ? launch_dkv<64>(dout, q, k, v, p, q_stride, k_stride, v_stride, do_stride, (cudaStream_t)stream)
             : launch_dkv<128>(dout, q, k, v, p, q_stride, k_stride, v_stride, do_stride, (cudaStream_t)stream);
}
