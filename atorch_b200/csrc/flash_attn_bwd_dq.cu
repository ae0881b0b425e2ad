// Flash attention backward, query-gradient kernel for sm_100a (head dim 128 or 64, bf16), tcgen05 + TMEM + TMA.
//
// One CTA per (128 query rows, head, batch) walks the key blocks its rows can see and keeps dQ in tensor
// memory from the first block to the last, so the query gradient needs no atomic adds, no fp32 scratch buffer
// and no conversion pass (the key/value gradients come from flash_attn_bwd_dkv.cu):
//   S  = Q K_j^T,  dP = dO V_j^T              2 x tcgen05.mma  smem x smem -> TMEM
//   P  = exp2(S c - lse),  dS = P (dP - delta) s   registers; dS written as bf16 over the dP columns
//   dQ += dS K_j                                tcgen05.mma  TMEM x smem (MN-major K) -> TMEM
// TMEM: S | dP (two buffers) | dQ = 4 x 128 columns. While the element-wise warps work on block j the tensor
// core already forms S and dP of block j+1 (S is free as soon as the warps hold it in registers, dP has a
// second buffer); dQ of block j follows when dS(j) is in place.
//
// Warp 0 = TMA producer (Q, dO once; K in three stages because a K tile serves S and, later, dQ; V in two), warp 1 = MMA issuer
// / TMEM owner, warp 2 = scheduler (block_queue.cuh), warps 4..11 = element-wise work: thread (row r, half h) owns columns
// [64h, 64h+64) of row r. The two threads of a row sit in different warps and the bf16 dS of one overwrites fp32 dP columns of
// the other, so the two warps of a lane quarter meet at a barrier between loading and storing (an mbarrier with a bounded
// wait). Masks are per-row key intervals [lo, hi) as in the forward kernel.
#include "block_queue.cuh"

namespace {
using namespace atb;

constexpr int BQ = 128, BKV = 128;
constexpr int PANEL = 128 * 64 * 2;
constexpr int K_STAGES = 3, V_STAGES = 2;
constexpr int N_EW = 256;
constexpr int THREADS = 128 + N_EW;

struct DqParams {
  const float* lse;            // [B, Hq, Sq]
  float* delta;                // [B, Hq, Sq], written: rowsum(dO * O)
  const __nv_bfloat16* dO;     // token-major rows of pitch do_stride, 16-byte aligned like the tensor maps
  const __nv_bfloat16* O;      // [B, Sq, Hq, HD]
  long long do_stride;
  __nv_bfloat16* dq;   // token-major, head h at columns [h*HD, h*HD+HD) of a row of pitch dq_stride
  long long dq_stride;
  const int* row_lo;
  const int* row_hi;
  int2* key_range;     // [B, query blocks], written for the dK/dV kernel unless null: first, last+1 key that a row sees
  int wide;            // rows of dq start on 32-byte boundaries
  int B, Sq, Sk, Hq, Hkv, causal;
  float scale, scale_log2;
  int* status;
  BlockOrder order;
};

template <int HD>
struct SmemQ {
  static constexpr int TILE = (HD / 64) * PANEL;
  static constexpr int Q_OFF = 0;
  static constexpr int DO_OFF = Q_OFF + TILE;
  static constexpr int K_OFF = DO_OFF + TILE;
  static constexpr int V_OFF = K_OFF + K_STAGES * TILE;
  static constexpr int BAR_OFF = V_OFF + V_STAGES * TILE;  // 224 KB
  static constexpr int NBARS = 2 + 2 * K_STAGES + 2 * V_STAGES + 4 + 4 + 2;
  static constexpr int QUEUE_OFF = BAR_OFF + NBARS * 8 + 16;
  static constexpr int DOT_OFF = QUEUE_OFF + (int)sizeof(WorkQueue);   // float [2][BQ]: dO . O of the rows of a unit
  static constexpr int TOTAL = DOT_OFF + 2 * BQ * 4 + 1024;
};
static_assert(SmemQ<128>::QUEUE_OFF % 16 == 0 && SmemQ<64>::QUEUE_OFF % 16 == 0, "the queue is 16-byte aligned");
static_assert(SmemQ<128>::TOTAL <= 232448, "shared memory of the dQ kernel exceeds 227 KB");

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, DqParams p) {
  using L = SmemQ<HD>;
  constexpr int TILE = L::TILE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::Q_OFF;
  uint8_t* sdO = smem + L::DO_OFF;
  uint8_t* sK = smem + L::K_OFF;
  uint8_t* sV = smem + L::V_OFF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* qdo_full = bars;
  uint64_t* qdo_free = bars + 1;               // the last S and dP of a unit have read Q and dO
  uint64_t* k_full = bars + 2;                 // [K_STAGES]
  uint64_t* k_empty = k_full + K_STAGES;       // [K_STAGES]  dQ(j) has read K_j
  uint64_t* v_full = k_empty + K_STAGES;       // [V_STAGES]
  uint64_t* v_empty = v_full + V_STAGES;       // [V_STAGES]  dP(j) has read V_j
  uint64_t* sdp_full = v_empty + V_STAGES;     // S(j), dP(j) are in TMEM
  uint64_t* s_free = sdp_full + 1;             // every element-wise warp holds S(j), dP(j) in registers
  uint64_t* ds_full = s_free + 1;              // dS(j) is in TMEM
  uint64_t* dq_full = ds_full + 1;             // the last dQ product of a unit has completed
  uint64_t* acc_free = dq_full + 1;            // dQ of a unit has been read out of TMEM
  uint64_t* pair_bar = acc_free + 1;           // [4] the two warps of a lane quarter both hold S(j), dP(j)
  uint64_t* dot_bar = pair_bar + 4;            // every element-wise warp has written its rows' dO . O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  WorkQueue* queue = reinterpret_cast<WorkQueue*>(smem + L::QUEUE_OFF);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int shift = p.Sk - p.Sq;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    mbar_init(qdo_free, 1);
    for (int i = 0; i < K_STAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < V_STAGES; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(sdp_full, 1);
    mbar_init(s_free, N_EW / 32);
    mbar_init(ds_full, N_EW / 32);
    mbar_init(dq_full, 1);
    mbar_init(acc_free, N_EW / 32);
    for (int i = 0; i < 4; ++i) mbar_init(&pair_bar[i], 2);
    mbar_init(dot_bar, N_EW / 32);
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
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdQ = tmem_base + 384;   // dP buffer of block g at tdP + 128*(g&1)

  // Units of this CTA, one after another: query block w.place of head w.head and sample w.sample, key blocks
  // [w.v0, w.v0 + w.v1), of which all rows see the keys [w.v2, w.v3). Barriers of the key blocks count on through all units
  // (g), those of Q, dO and the accumulator count the units that have any block (u).
  if (warp < 4) {
    if (warp == 2) {
      queue_run(queue, p.order, [&](Work& w, int blocks) {
        w.place = blocks - 1 - w.place;   // heaviest (last) causal blocks first
        const int q0 = w.place * BQ;
        int umin = INT_MAX, umax = 0, ilo = 0, ihi = INT_MAX;   // union and intersection of the rows' intervals
        int rlo[BQ / 32], rhi[BQ / 32];      // all loads first, then their use
#pragma unroll
        for (int e = 0; e < BQ / 32; ++e) {
          const int i = min(q0 + lane + 32 * e, p.Sq - 1);
          rlo[e] = p.row_lo ? p.row_lo[(long long)w.sample * p.Sq + i] : 0;
          rhi[e] = p.row_hi ? p.row_hi[(long long)w.sample * p.Sq + i] : (p.causal ? i + 1 + shift : p.Sk);
        }
#pragma unroll
        for (int e = 0; e < BQ / 32; ++e) {
          if (q0 + lane + 32 * e >= p.Sq) continue;
          const int lo = max(rlo[e], 0), hi = min(rhi[e], p.Sk);
          if (hi <= lo) { ilo = INT_MAX; ihi = 0; continue; }
          umin = min(umin, lo); umax = max(umax, hi);
          ilo = max(ilo, lo); ihi = min(ihi, hi);
        }
        umin = __reduce_min_sync(0xffffffffu, umin);
        umax = __reduce_max_sync(0xffffffffu, umax);
        w.v0 = umax > umin ? umin / BKV : 0;
        w.v1 = (umax > umin ? (umax + BKV - 1) / BKV : 0) - w.v0;
        w.v2 = __reduce_max_sync(0xffffffffu, ilo);
        w.v3 = __reduce_min_sync(0xffffffffu, ihi);
        if (p.key_range != nullptr && w.head == 0 && lane == 0)
          p.key_range[(long long)w.sample * blocks + w.place] = make_int2(umin, umax);
      }, abort_flag, p.status);
    } else if (warp == 0) {
      const bool el = elect_one();
      if (el) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
      uint32_t g = 0;
      int u = 0;
      Work w;
      for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
        const int n = w.v1, h = w.head, hk = h / (p.Hq / p.Hkv);
        if (n == 0) { queue_claim(queue); continue; }
        const int qrow = (int)((long long)w.sample * p.Sq + w.place * BQ);
        if (!mbar_wait_warp(qdo_free, (u & 1) ^ 1, abort_flag, p.status)) break;
        ++u;
        if (el) mbar_expect_tx(qdo_full, 2 * TILE);
        if (el) tma_load_2d(sQ, &tmQ, qdo_full, h * HD, qrow);
        if (HD == 128 && el) tma_load_2d(sQ + PANEL, &tmQ, qdo_full, h * HD + 64, qrow);
        if (el) tma_load_2d(sdO, &tmdO, qdo_full, h * HD, qrow);
        if (HD == 128 && el) tma_load_2d(sdO + PANEL, &tmdO, qdo_full, h * HD + 64, qrow);
        bool ok = true;
        for (int j = 0; j < n; ++j, ++g) {
          if (j == max(n - 3, 0)) queue_claim(queue);
          const int ks = g % K_STAGES, vs = g % V_STAGES;
          const int krow = (int)((long long)w.sample * p.Sk + (long long)(w.v0 + j) * BKV);
          ok = mbar_wait_warp(&k_empty[ks], ((g / K_STAGES) & 1) ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (el) mbar_expect_tx(&k_full[ks], TILE);
          if (el) tma_load_2d(sK + ks * TILE, &tmK, &k_full[ks], hk * HD, krow);
          if (HD == 128 && el) tma_load_2d(sK + ks * TILE + PANEL, &tmK, &k_full[ks], hk * HD + 64, krow);
          ok = mbar_wait_warp(&v_empty[vs], ((g / V_STAGES) & 1) ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (el) mbar_expect_tx(&v_full[vs], TILE);
          if (el) tma_load_2d(sV + vs * TILE, &tmV, &v_full[vs], hk * HD, krow);
          if (HD == 128 && el) tma_load_2d(sV + vs * TILE + PANEL, &tmV, &v_full[vs], hk * HD + 64, krow);
        }
        if (!ok) break;
      }
    } else if (warp == 1) {
      const uint32_t el = elect_one();   // the lane that issues and commits
      constexpr uint32_t id_kk = umma_idesc(128, 128, 1, 1, false, false);
      constexpr uint32_t id_km = umma_idesc(128, HD, 1, 1, false, true);
      const uint32_t dQk = umma_desc_lo(smem_u32(sQ), 16), dOk = umma_desc_lo(smem_u32(sdO), 16);
      const uint32_t dKk0 = umma_desc_lo(smem_u32(sK), 16), dKm0 = umma_desc_lo(smem_u32(sK), PANEL);
      const uint32_t dVk0 = umma_desc_lo(smem_u32(sV), 16);
      // S(g) = Q K_g^T and dP(g) = dO V_g^T
      auto issue_sdp = [&](uint32_t g, bool last) -> bool {
        const int ks = g % K_STAGES, vs = g % V_STAGES;
        if (!mbar_wait_warp(&k_full[ks], (g / K_STAGES) & 1, abort_flag, p.status)) return false;
        tc_fence_after();
        const uint32_t kd = dKk0 + ((ks * TILE) >> 4);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * PANEL + (k & 3) * 32;
          umma_ss_issue(tS, dQk + (off >> 4), kd + (off >> 4), id_kk, k != 0, el);
        }
        if (!mbar_wait_warp(&v_full[vs], (g / V_STAGES) & 1, abort_flag, p.status)) return false;
        tc_fence_after();
        const uint32_t vd = dVk0 + ((vs * TILE) >> 4);
        const uint32_t dst = tdP + 128 * (g & 1);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * PANEL + (k & 3) * 32;
          umma_ss_issue(dst, dOk + (off >> 4), vd + (off >> 4), id_kk, k != 0, el);
        }
        umma_commit_issue(sdp_full, el);
        umma_commit_issue(&v_empty[vs], el);
        if (last) umma_commit_issue(qdo_free, el);
        return true;
      };
      uint32_t g = 0;
      int u = 0;
      Work w;
      for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
        const int n = w.v1;
        if (n == 0) continue;
        // the first scores of a unit follow the last product of the one before and run under its results' way out
        bool ok = mbar_wait_warp(qdo_full, u & 1, abort_flag, p.status) &&
                  (g == 0 || mbar_wait_warp(s_free, (g - 1) & 1, abort_flag, p.status));
        tc_fence_after();
        ok = ok && issue_sdp(g, n == 1);
        for (int j = 0; ok && j < n; ++j, ++g) {
          if (j + 1 < n) {
            ok = mbar_wait_warp(s_free, g & 1, abort_flag, p.status);
            tc_fence_after();
            ok = ok && issue_sdp(g + 1, j + 2 == n);
          }
          if (ok && j == 0 && u > 0) ok = mbar_wait_warp(acc_free, (u - 1) & 1, abort_flag, p.status);
          ok = ok && mbar_wait_warp(ds_full, g & 1, abort_flag, p.status);
          if (!ok) break;
          tc_fence_after();
          const uint32_t km = dKm0 + (((g % K_STAGES) * TILE) >> 4);
          const uint32_t a = tdP + 128 * (g & 1);
#pragma unroll
          for (int k = 0; k < 8; ++k)   // dQ += dS K_j: 16 keys per step = 8 TMEM columns of packed bf16
            umma_ts_issue(tdQ, a + k * 8, km + k * 128, id_km, (j | k) != 0, el);
          umma_commit_issue(&k_empty[g % K_STAGES], el);
          if (j == n - 1) umma_commit_issue(dq_full, el);
        }
        if (!ok) break;
        ++u;
      }
    }
  } else {
    const int quarter = warp & 3;
    const int half = (warp - 4) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = ((uint32_t)(quarter * 32) << 16);
    // delta = dO . O of the block's rows, 16 rows per warp and HD / 8 lanes per row: a separate pass over both tensors took
    // 26 us at S=4096, 32 heads of 128. A unit's values are loaded when it begins, under its first products: holding them from the
    // end of the unit before took registers that the loop over the tiles needs (16 heads on 8192 keys, all visible, head dim 64
    // 565 us, now 512; 128 604, now 562). They are asked into L2 there (backward of 4096 in 30 documents, 32 heads of 128 on 8,
    // 148 us without, 144 with).
    constexpr int LANES = HD / 8, AT_ONCE = 32 / LANES, STEPS = 16 / AT_ONCE;
    const int first = (warp - 4) * 16 + lane / LANES, sub = lane % LANES;
    uint32_t g = 0;
    int u = 0;
    Work w;
    bool ok = queue_next(queue, 0, w, abort_flag, p.status);
    for (int c = 0; ok && w.more;) {
      const int b = w.sample, h = w.head, n = w.v1, full_lo = w.v2, full_hi = w.v3;
      const int i = w.place * BQ + r;   // global query row
      float delta, lse;
      int lo, hi;
      {
        uint4 x[STEPS], y[STEPS];
#pragma unroll
        for (int e = 0; e < STEPS; ++e) {
          const long long tok = (long long)b * p.Sq + min(w.place * BQ + first + e * AT_ONCE, p.Sq - 1);
          x[e] = *reinterpret_cast<const uint4*>(p.dO + tok * p.do_stride + h * HD + sub * 8);
          y[e] = *reinterpret_cast<const uint4*>(p.O + (tok * p.Hq + h) * HD + sub * 8);
        }
        const int at = min(i, p.Sq - 1);
        lse = p.lse[((long long)b * p.Hq + h) * p.Sq + at];
        lo = p.row_lo ? p.row_lo[(long long)b * p.Sq + at] : 0;
        hi = p.row_hi ? p.row_hi[(long long)b * p.Sq + at] : (p.causal ? at + 1 + shift : p.Sk);
        float* dots = reinterpret_cast<float*>(smem + L::DOT_OFF) + (c & 1) * BQ;
#pragma unroll
        for (int e = 0; e < STEPS; ++e) {
          const uint32_t xs[4] = {x[e].x, x[e].y, x[e].z, x[e].w}, ys[4] = {y[e].x, y[e].y, y[e].z, y[e].w};
          float acc = 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 a = unpack_bf16x2(xs[k]), d = unpack_bf16x2(ys[k]);
            acc += a.x * d.x + a.y * d.y;
          }
#pragma unroll
          for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          if (sub == 0) dots[first + e * AT_ONCE] = acc;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(dot_bar);
        ok = mbar_wait_warp(dot_bar, c & 1, abort_flag, p.status);
        if (!ok) break;
        delta = dots[r];
        if (half == 0 && i < p.Sq) p.delta[((long long)b * p.Hq + h) * p.Sq + i] = delta;
      }
      const bool valid = i < p.Sq && lse != -INFINITY;
      if (!valid) delta = 0.f;
      const float lse2 = valid ? lse * 1.4426950408889634f : 0.f;
      lo = valid ? max(lo, 0) : 0;
      hi = valid ? min(hi, p.Sk) : 0;
      const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2), nl2 = f2_pack(-lse2, -lse2);
      const uint64_t nd2 = f2_pack(-delta, -delta), scl2 = f2_pack(p.scale, p.scale);
      for (int j = 0; j < n; ++j, ++g) {
        const int kv0 = (w.v0 + j) * BKV;
        const uint32_t dp_addr = tdP + 128 * (g & 1) + lane_addr;
        if (!mbar_wait_warp(sdp_full, g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        uint32_t s0[32], s1[32], d0[32], d1[32];
        tmem_ld_32x32(tS + lane_addr + half * 64, s0);
        tmem_ld_32x32(tS + lane_addr + half * 64 + 32, s1);
        tmem_ld_32x32(dp_addr + half * 64, d0);
        tmem_ld_32x32(dp_addr + half * 64 + 32, d1);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(s_free);
          mbar_arrive(&pair_bar[quarter]);
        }
        // both threads of every row of this lane quarter hold their S and dP before either stores dS (a bounded
        // mbarrier wait, not a named barrier, so that a warp whose partner gave up cannot wait forever)
        if (!mbar_wait_warp(&pair_bar[quarter], g & 1, abort_flag, p.status)) { ok = false; break; }
        // tiles inside the intersection of the rows' intervals run without per-element tests
        const bool tile_full = (kv0 >= full_lo) && (kv0 + BKV <= full_hi);
        const int c0 = kv0 + half * 64;
        float pa[32], pb[32];   // P for keys c0 .. c0+31 and c0+32 .. c0+63
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float a0, a1, b0, b1;
          f2_unpack(f2_fma(f2_pack_bits(s0[c], s0[c + 1]), sc2, nl2), a0, a1);
          f2_unpack(f2_fma(f2_pack_bits(s1[c], s1[c + 1]), sc2, nl2), b0, b1);
          pa[c] = fast_exp2(a0); pa[c + 1] = fast_exp2(a1);
          pb[c] = fast_exp2(b0); pb[c + 1] = fast_exp2(b1);
        }
        if (!tile_full) {   // a separate pass, so that fully visible tiles execute no interval tests at all
          const uint32_t m0 = valid ? visible_keys(c0, lo, hi) : 0u, m1 = valid ? visible_keys(c0 + 32, lo, hi) : 0u;
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (!(m0 & (1u << c))) pa[c] = 0.f;
            if (!(m1 & (1u << c))) pb[c] = 0.f;
          }
        }
        uint32_t ds[32];
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float x0, x1, y0, y1;   // dS = P (dP - delta) scale
          f2_unpack(f2_mul(f2_mul(f2_pack(pa[c], pa[c + 1]), scl2), f2_add(f2_pack_bits(d0[c], d0[c + 1]), nd2)), x0, x1);
          f2_unpack(f2_mul(f2_mul(f2_pack(pb[c], pb[c + 1]), scl2), f2_add(f2_pack_bits(d1[c], d1[c + 1]), nd2)), y0, y1);
          ds[c >> 1] = pack_bf16x2(x0, x1);
          ds[16 + (c >> 1)] = pack_bf16x2(y0, y1);
        }
        // keys [64h, 64h+64) of the row as packed bf16: columns [32h, 32h+32) of the dP buffer
        tmem_st_32x32(dp_addr + half * 32, ds);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
      }
      if (!ok) break;
      Work nw;
      ok = queue_next(queue, ++c, nw, abort_flag, p.status);
      if (!ok) break;
      if (nw.more) {      // on their way into L2 while this unit's results leave
#pragma unroll
        for (int e = 0; e < STEPS; ++e) {
          const long long tok = (long long)nw.sample * p.Sq + min(nw.place * BQ + first + e * AT_ONCE, p.Sq - 1);
          if ((sub & 3) == 0) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.dO + tok * p.do_stride + nw.head * HD + sub * 8));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.O + (tok * p.Hq + nw.head) * HD + sub * 8));
          }
        }
      }
      if (n > 0) {
        ok = mbar_wait_warp(dq_full, u & 1, abort_flag, p.status);
        if (!ok) break;
        ++u;
        tc_fence_after();
      }
      __nv_bfloat16* row = p.dq + ((long long)b * p.Sq + i) * p.dq_stride + h * HD + half * (HD / 2);
#pragma unroll
      for (int cc = 0; cc < HD / 64; ++cc) {
        uint32_t t[32];
        if (n > 0) {
          tmem_ld_32x32(tdQ + lane_addr + half * (HD / 2) + cc * 32, t);
          tmem_ld_wait();
          if (cc == HD / 64 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free);
          }
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) t[k] = 0u;
        }
        if (i < p.Sq) store_bf16_32(row + cc * 32, t, p.wide);
      }
      w = nw;
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
int launch_dq(const void* dout, const void* q, const void* k, const void* v, DqParams p, long long q_stride,
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
    if (cudaFuncSetAttribute(flash_bwd_dq_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmemQ<HD>::TOTAL) !=
        cudaSuccess)
      return -4;
    attr_set = true;
  }
  dim3 grid;
  make_block_order(&p.order, &grid, (p.Sq + BQ - 1) / BQ, p.Hq, p.B, p.causal != 0, p.Sk, HD);
  launch_after(flash_bwd_dq_kernel<HD>, grid, THREADS, SmemQ<HD>::TOTAL, stream, 1, tmQ, tmdO, tmK, tmV, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace

// dq rows of pitch dq_stride elements (head h at columns [h*head_dim, (h+1)*head_dim)); lse: [B, Hq, Sq] fp32;
// delta: [B, Hq, Sq] fp32, written (rowsum(dO * O), which the key/value-gradient kernel reads); out: [B, Sq, Hq, head_dim].
extern "C" int atb_flash_bwd_dq(const void* dout, const void* q, const void* k, const void* v, const void* out,
                                const float* lse, float* delta, void* dq, const int* row_lo, const int* row_hi, int B, int Sq,
                                int Sk, int Hq, int Hkv, long long q_stride, long long k_stride, long long v_stride,
                                long long do_stride, long long dq_stride, int causal, float softmax_scale, int head_dim,
                                int* key_range, void* stream, int* status) {
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if (Hq % Hkv || (head_dim != 128 && head_dim != 64)) return -1;
  if ((q_stride | k_stride | v_stride | do_stride | dq_stride) & 7) return -1;
  if ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out)) & 15) return -2;
  DqParams p;
  p.dO = (const __nv_bfloat16*)dout; p.O = (const __nv_bfloat16*)out; p.do_stride = do_stride;
  p.lse = lse; p.delta = delta; p.dq = (__nv_bfloat16*)dq; p.dq_stride = dq_stride;
  p.row_lo = row_lo; p.row_hi = row_hi; p.key_range = reinterpret_cast<int2*>(key_range);
  p.wide = (reinterpret_cast<uintptr_t>(dq) & 31) == 0 && (dq_stride & 15) == 0;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal;
  p.scale = softmax_scale; p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  return head_dim == 64
             ? launch_dq<64>(dout, q, k, v, p, q_stride, k_stride, v_stride, do_stride, (cudaStream_t)stream)
             : launch_dq<128>(dout, q, k, v, p, q_stride, k_stride, v_stride, do_stride, (cudaStream_t)stream);
}
