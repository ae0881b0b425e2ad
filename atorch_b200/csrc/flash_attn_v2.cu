// Flash attention forward, two query tiles per CTA (head dim 128 or 64, bf16) for sm_100a.
//
// One CTA owns 256 query rows as two 128-row tiles A and B that share every K/V tile. Warp 0 = TMA
// producer, warp 1 = MMA issuer / TMEM owner, warp 2 = scheduler (block_queue.cuh), warps 4..7 = softmax of tile A, warps 8..11 =
// softmax of tile B; a softmax thread owns one whole row (128 scores), so no row statistics are exchanged.
//
//   TMEM:  S_A | S_B | O_A | O_B   (4 x 128 fp32 columns); P_T (bf16) overwrites the first 64 columns of S_T
//   per K/V tile j:   S_T = Q_T K_j^T  ->  P_T = 2^(S_T c - m_T c)  ->  O_T += P_T V_j
//
// P never leaves tensor memory: the softmax thread stores its packed row with tcgen05.st and the P.V
// product reads it as the A operand of tcgen05.mma. O accumulates in tensor memory. What bounds the kernel is the
// chain S -> maximum -> exponentials -> P -> P.V -> next S of one tile, so it is kept short: the 128 scores of a row
// are read out of tensor memory once and stay in registers, hidden keys are turned into -inf there (32 keys per bit
// mask, so that a partly visible tile costs little more than a full one), and P is handed over in two halves of 64
// keys, so that the first half of P.V runs under the second half of the exponentials. The reference maximum
// m_T of a row is only raised when the new row maximum exceeds it by more than 2^8 (head dim 128; in the exponent
// domain); then the row of O_T is rescaled in TMEM by the owning thread, which is safe because the scores
// S_T(j) it has just waited for were issued after the product P_T(j-1) V and complete after it.
// While tile A's warps exponentiate, the tensor core works for tile B and vice versa:
// issue order  PV_A(j), S_A(j+1), PV_B(j), S_B(j+1).
//
// 8192 keys, 32 heads of 128: full 775 us (1420 TFLOP/s), causal 419 us (450 with a CTA per block); 16 x 512, 16 heads of 64,
// all keys 45 us (55 with a CTA per block). A step of both tiles takes 3100 clocks, 1900 of them softmax and 1200 tensor work
// of the same tile. Tried: K/V tiles of 64 keys with two score buffers per tile, which takes the tensor work out of that chain
// - 887 us, because a 128 x 64 x 16 score product takes 48 clocks for its shared-memory operands where it should take 32; P in
// one piece - 859 us.
//
// Masks: per-row key interval [lo, hi) exactly as in flash_attn.cu; each query tile walks only the K/V
// tiles up to the last one that any of its rows can see.
#include "block_queue.cuh"
#include <type_traits>

namespace {
using namespace atb;

constexpr int BQ = 128, BKV = 128;
constexpr int PANEL = 128 * 64 * 2;
constexpr int THREADS = 128 + 256;
// 168 registers a thread at launch (384 x 168 = 64512); the control warpgroup gives up what the softmax warps need to
// hold a row of scores: 128 x 80 + 256 x 208 = 63488
constexpr int REGS_CONTROL = 80, REGS_SOFTMAX = 208;
// How far (log2 units) a row's maximum may run ahead of its reference before the row is rescaled. A lag moves the rounding
// of P to bf16 to other mantissas: 0.00234 from the 64-bit result (2 x 2048 of normal values, head dim 128) against 0.00226
// with the exact maximum of the single-tile kernel. Head dim 64 takes the exact maximum: 0.00220, 0.00230 with the lag
// (16 x 512), for 55 us in place of 51 there and 498 in place of 395 at 8192 x 16 heads, all keys.
template <int HD>
constexpr float RESCALE_THRESHOLD = HD == 64 ? 0.f : 8.f;

struct Params {
  __nv_bfloat16* O;
  float* lse;
  const int* row_lo;
  const int* row_hi;
  int B, Sq, Sk, Hq, Hkv, causal;
  float scale_log2;
  int* status;
  const int* holes;    // [B] or null: if any is set, the launch does nothing
  int wide;            // rows of O start on 32-byte boundaries
  BlockOrder order;
};

template <int HD>
struct L2 {
  static constexpr int TILE = (HD / 64) * PANEL;
  static constexpr int Q_OFF = 0;                    // tile A, tile B
  static constexpr int K_OFF = Q_OFF + 2 * TILE;     // 2 stages
  static constexpr int V_OFF = K_OFF + 2 * TILE;     // 2 stages
  static constexpr int BAR_OFF = V_OFF + 2 * TILE;   // 192 KB
  static constexpr int NBARS = 2 + 8 + 2 + 4 + 2 + 2;
  static constexpr int QUEUE_OFF = BAR_OFF + NBARS * 8 + 16;
  static constexpr int TOTAL = QUEUE_OFF + (int)sizeof(WorkQueue) + 1024;
  static_assert(QUEUE_OFF % 16 == 0, "the queue is 16-byte aligned");
};

// -inf in place of the scores of hidden keys: key kv0 + c is visible when it lies in [lo, hi)
ATB_DEVICE void mask_scores(uint32_t (&x)[32], int kv0, int lo, int hi) {
  const uint32_t vis = visible_keys(kv0, lo, hi);
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (!(vis & (1u << c))) x[c] = 0xff800000u;
}

ATB_DEVICE float max_of(const uint32_t (&x)[32]) {
  float m0 = __uint_as_float(x[0]), m1 = __uint_as_float(x[1]);
#pragma unroll
  for (int c = 2; c < 32; c += 2) {
    m0 = fmaxf(m0, __uint_as_float(x[c]));
    m1 = fmaxf(m1, __uint_as_float(x[c + 1]));
  }
  return fmaxf(m0, m1);
}

// P = 2^(S c - m c) of 64 scores as packed bf16; the sums of the even and the odd keys are added to `sum`
ATB_DEVICE void exp_half(const uint32_t (&xa)[32], const uint32_t (&xb)[32], uint64_t sc2, uint64_t nm2, uint64_t& sum0,
                         uint64_t& sum1, uint32_t (&pk)[32]) {
#pragma unroll
  for (int c = 0; c < 32; c += 2) {
    float t0, t1, u0, u1;
    f2_unpack(f2_fma(f2_pack_bits(xa[c], xa[c + 1]), sc2, nm2), t0, t1);
    f2_unpack(f2_fma(f2_pack_bits(xb[c], xb[c + 1]), sc2, nm2), u0, u1);
    const float p0 = fast_exp2(t0), p1 = fast_exp2(t1), r0 = fast_exp2(u0), r1 = fast_exp2(u1);
    sum0 = f2_add(sum0, f2_pack(p0, p1));
    sum1 = f2_add(sum1, f2_pack(r0, r1));
    pk[c >> 1] = pack_bf16x2(p0, p1);
    pk[16 + (c >> 1)] = pack_bf16x2(r0, r1);
  }
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
flash_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, Params p) {
  using L = L2<HD>;
  constexpr int TILE = L::TILE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::Q_OFF;
  uint8_t* sK = smem + L::K_OFF;
  uint8_t* sV = smem + L::V_OFF;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* q_full = bars;
  uint64_t* q_free = bars + 1;      // the last scores of a unit have read Q
  uint64_t* k_full = bars + 2;      // [2]
  uint64_t* k_empty = bars + 4;     // [2]
  uint64_t* v_full = bars + 6;      // [2]
  uint64_t* v_empty = bars + 8;     // [2]
  uint64_t* s_full = bars + 10;     // [2] per query tile: S_T(j) is in TMEM (and P_T(j-1) V has completed)
  uint64_t* p_full = bars + 12;     // [2][2] per query tile and half of the keys: P_T(j) is in TMEM
  uint64_t* o_full = bars + 16;     // [2] per query tile: the last P.V product of a unit has completed
  uint64_t* o_free = bars + 18;     // [2] per query tile: O_T of a unit has been read out of TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBARS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  WorkQueue* queue = reinterpret_cast<WorkQueue*>(smem + L::QUEUE_OFF);

  const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p.holes != nullptr) {
    grid_wait();
    int any = 0;
    for (int i = threadIdx.x; i < p.B; i += THREADS) any |= p.holes[i];
    if (__syncthreads_or(any)) return;
  }
  const int shift = p.Sk - p.Sq;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_free, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&o_full[i], 1); mbar_init(&o_free[i], 4);
    }
    for (int i = 0; i < 4; ++i) mbar_init(&p_full[i], 4);
    queue_init(queue, 2 + 8);
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

  // Units of this CTA, one after another: 256 query rows w.place of head w.head and sample w.sample, w.v1 (w.v2) K/V tiles
  // from w.v0 on for query tile A (B). Barriers of the K/V ring count its tiles through all units (g), those of a query tile
  // the tiles that it multiplied, those of Q and O the units that have any.
  if (warp < 4) {
    reg_dealloc<REGS_CONTROL>();
    if (warp == 2) {
      queue_run(queue, p.order, [&](Work& w, int blocks) {
        w.place = blocks - 1 - w.place;   // heaviest (last) causal blocks first
        const int q0 = w.place * 2 * BQ;
        // union of the key intervals of the rows of each tile (all loads first, then their use)
        int rlo[2 * BQ / 32], rhi[2 * BQ / 32];
#pragma unroll
        for (int e = 0; e < 2 * BQ / 32; ++e) {
          const int i = min(q0 + lane + 32 * e, p.Sq - 1);
          rlo[e] = p.row_lo ? p.row_lo[(long long)w.sample * p.Sq + i] : 0;
          rhi[e] = p.row_hi ? p.row_hi[(long long)w.sample * p.Sq + i] : (p.causal ? i + 1 + shift : p.Sk);
        }
        int umin = INT_MAX, umax[2] = {0, 0};
#pragma unroll
        for (int e = 0; e < 2 * BQ / 32; ++e) {
          const int lo = max(rlo[e], 0), hi = min(rhi[e], p.Sk), t = e / (BQ / 32);
          if (q0 + lane + 32 * e < p.Sq && hi > lo) { umin = min(umin, lo); umax[t] = max(umax[t], hi); }
        }
        umin = __reduce_min_sync(0xffffffffu, umin);
        umax[0] = __reduce_max_sync(0xffffffffu, umax[0]);
        umax[1] = __reduce_max_sync(0xffffffffu, umax[1]);
        w.v0 = umin == INT_MAX ? 0 : umin / BKV;
        w.v1 = umax[0] > 0 ? (umax[0] + BKV - 1) / BKV - w.v0 : 0;
        w.v2 = umax[1] > 0 ? (umax[1] + BKV - 1) / BKV - w.v0 : 0;
      }, abort_flag, p.status);
    }
    if (warp == 0) {
      const bool el = elect_one();
      if (el) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); }
      uint32_t g = 0;
      int u = 0;
      Work w;
      for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
        const int n = max(w.v1, w.v2), h = w.head, hk = h / (p.Hq / p.Hkv);
        if (n == 0) { queue_claim(queue); continue; }
        if (!mbar_wait_warp(q_free, (u & 1) ^ 1, abort_flag, p.status)) break;
        ++u;
        if (el) mbar_expect_tx(q_full, 2 * TILE);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int qrow = (int)((long long)w.sample * p.Sq + w.place * 2 * BQ + t * BQ);
          if (el) tma_load_2d(sQ + t * TILE, &tmQ, q_full, h * HD, qrow);
          if (HD == 128 && el) tma_load_2d(sQ + t * TILE + PANEL, &tmQ, q_full, h * HD + 64, qrow);
        }
        bool ok = true;
        for (int j = 0; j < n; ++j, ++g) {
          if (j == max(n - 2, 0)) queue_claim(queue);
          const int s = g & 1;
          const uint32_t ph = (g >> 1) & 1;
          const int krow = (int)((long long)w.sample * p.Sk + (long long)(w.v0 + j) * BKV);
          ok = mbar_wait_warp(&k_empty[s], ph ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (el) mbar_expect_tx(&k_full[s], TILE);
          if (el) tma_load_2d(sK + s * TILE, &tmK, &k_full[s], hk * HD, krow);
          if (HD == 128 && el) tma_load_2d(sK + s * TILE + PANEL, &tmK, &k_full[s], hk * HD + 64, krow);
          ok = mbar_wait_warp(&v_empty[s], ph ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (el) mbar_expect_tx(&v_full[s], TILE);
          if (el) tma_load_2d(sV + s * TILE, &tmV, &v_full[s], hk * HD, krow);
          if (HD == 128 && el) tma_load_2d(sV + s * TILE + PANEL, &tmV, &v_full[s], hk * HD + 64, krow);
        }
        if (!ok) break;
      }
    }
    if (warp == 1) {
      const uint32_t el = elect_one();  // the lane that issues and commits
      constexpr uint32_t idesc_s = umma_idesc(BQ, BKV, 1, 1, false, false);
      constexpr uint32_t idesc_o = umma_idesc(BQ, HD, 1, 1, false, true);
      uint32_t k_ready = 0, v_ready = 0;   // K / V tiles whose arrival has been waited for
      // descriptors of the tiles' first MMA operands; the loops below only advance them
      // (kept in scalars and picked with selects: an array indexed at run time would live in local memory)
      const uint32_t q_desc0 = umma_desc_lo(smem_u32(sQ), 16), k_desc0 = umma_desc_lo(smem_u32(sK), 16),
                     v_desc0 = umma_desc_lo(smem_u32(sV), PANEL);
      auto wait_k = [&](uint32_t g) -> bool {
        if (k_ready > g) return true;
        k_ready = g + 1;
        return mbar_wait_warp(&k_full[g & 1], (g >> 1) & 1, abort_flag, p.status);
      };
      auto wait_v = [&](uint32_t g) -> bool {
        if (v_ready > g) return true;
        v_ready = g + 1;
        return mbar_wait_warp(&v_full[g & 1], (g >> 1) & 1, abort_flag, p.status);
      };
      // S_T(g) = Q_T K_g^T into the tile's S columns (K_g has arrived)
      auto issue_s = [&](int t, uint32_t g) {
        const uint32_t qd = q_desc0 + ((t ? TILE : 0) >> 4), kd = k_desc0 + (((g & 1) ? TILE : 0) >> 4);
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t off = (k >> 2) * PANEL + (k & 3) * 32;
          umma_ss_issue(tmem_base + t * BKV, qd + (off >> 4), kd + (off >> 4), idesc_s, k != 0, el);
        }
        umma_commit_issue(&s_full[t], el);
      };
      uint32_t g = 0, done_a = 0, done_b = 0;      // K/V tiles so far: of the ring, multiplied by query tile A, B
      int u = 0, units_a = 0, units_b = 0;
      Work w;
      for (int c = 0; queue_next(queue, c, w, abort_flag, p.status) && w.more; ++c) {
        const int n_a = w.v1, n_b = w.v2, n = max(n_a, n_b);
        if (n == 0) continue;
        bool ok = mbar_wait_warp(q_full, u & 1, abort_flag, p.status) && wait_k(g);
        if (!ok) break;
        if (n_a > 0) issue_s(0, g);
        if (n_b > 0) issue_s(1, g);
        umma_commit_issue(&k_empty[g & 1], el);
        if (n == 1) umma_commit_issue(q_free, el);
        // one half-step of the ping-pong for query tile T (compile-time, so that nothing is indexed at run time):
        // P_T(j) V_j into O_T, then the next scores S_T(j+1). The waits for V_j and K_{j+1} come before the wait for P,
        // so that nothing lies between P's arrival and the products that depend on it.
        auto half_step = [&](auto tile, int j) -> bool {
          constexpr int t = decltype(tile)::value;
          const int n_t = t ? n_b : n_a;
          const uint32_t gj = g + j, ph = ((t ? done_b : done_a) + j) & 1;
          const int s = gj & 1;
          if (j < n_t) {
            if (!wait_v(gj) || (j + 1 < n_t && !wait_k(gj + 1))) return false;
            const int units = t ? units_b : units_a;
            if (j == 0 && units > 0 && !mbar_wait_warp(&o_free[t], (units - 1) & 1, abort_flag, p.status)) return false;
            const uint32_t vd = v_desc0 + ((s ? TILE : 0) >> 4);
#pragma unroll
            for (int k = 0; k < BKV / 16; ++k) {   // A = P_T: 16 bf16 keys per step = 8 TMEM columns
              if (k % (BKV / 32) == 0) {
                if (!mbar_wait_warp(&p_full[2 * t + k / (BKV / 32)], ph, abort_flag, p.status)) return false;
                tc_fence_after();
              }
              umma_ts_issue(tmem_base + 2 * BKV + t * HD, tmem_base + t * BKV + k * 8, vd + k * 128,
                            idesc_o, (j | k) != 0, el);
            }
            if (j == n_t - 1) umma_commit_issue(&o_full[t], el);
          }
          if (j + 1 < n_t) issue_s(t, gj + 1);
          if (t == 1) umma_commit_issue(&v_empty[s], el);
          if (t == 1 && j + 1 < n) umma_commit_issue(&k_empty[(gj + 1) & 1], el);
          if (t == 1 && j + 2 == n) umma_commit_issue(q_free, el);
          return true;
        };
        for (int j = 0; ok && j < n; ++j)
          ok = half_step(std::integral_constant<int, 0>{}, j) && half_step(std::integral_constant<int, 1>{}, j);
        if (!ok) break;
        g += n;
        ++u;
        done_a += n_a;
        done_b += n_b;
        units_a += n_a > 0;
        units_b += n_b > 0;
      }
    }
  } else {
    reg_alloc<REGS_SOFTMAX>();
    const int t = (warp - 4) >> 2;            // query tile of this warp
    const int quarter = warp & 3;             // TMEM lane quarter
    const int r = quarter * 32 + lane;        // row inside the tile
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + t * BKV, o_addr = lane_addr + 2 * BKV + t * HD;
    int lo = 0, hi = 0;
    auto load_unit = [&](const Work& w) {     // the row's interval, loaded before the results of the last unit are stored
      const int i = w.place * 2 * BQ + t * BQ + r;
      lo = hi = 0;
      if (w.more && i < p.Sq) {
        lo = p.row_lo ? p.row_lo[(long long)w.sample * p.Sq + i] : 0;
        hi = p.row_hi ? p.row_hi[(long long)w.sample * p.Sq + i] : (p.causal ? i + 1 + shift : p.Sk);
      }
    };
    uint32_t g = 0;
    int u = 0;
    bool ok = queue_wait(queue, 0, abort_flag, p.status);
    if (ok) load_unit(queue_read(queue, 0));
    for (int c = 0; ok; ++c) {
      const Work unit = queue_read(queue, c);
      if (!unit.more) break;
      const int n_t = t ? unit.v2 : unit.v1;
      lo = max(lo, 0); hi = min(hi, p.Sk);             // (0, 0) in a row that there is not
      float m_ref = -INFINITY, l_run = 0.f;
      for (int j = 0; j < n_t; ++j, ++g) {
        const int kv0 = (unit.v0 + j) * BKV;
        if (!mbar_wait_warp(&s_full[t], g & 1, abort_flag, p.status)) { ok = false; break; }
        tc_fence_after();
        // the mask tests are compiled into a separate path taken only by warps with a partly visible row
        const bool full = __all_sync(0xffffffffu, lo <= kv0 && hi >= kv0 + BKV);
        uint32_t x0[32], x1[32], x2[32], x3[32];
        tmem_ld_32x32(s_addr, x0);
        tmem_ld_32x32(s_addr + 32, x1);
        tmem_ld_32x32(s_addr + 64, x2);
        tmem_ld_32x32(s_addr + 96, x3);
        tmem_ld_wait();
        if (!full) {
          mask_scores(x0, kv0, lo, hi);
          mask_scores(x1, kv0 + 32, lo, hi);
          mask_scores(x2, kv0 + 64, lo, hi);
          mask_scores(x3, kv0 + 96, lo, hi);
        }
        const float mx = fmaxf(fmaxf(max_of(x0), max_of(x1)), fmaxf(max_of(x2), max_of(x3)));
        // raise the reference maximum only when it pays: 2^(gap) of a stale one fits bf16 and fp32
        const bool raise = (mx > m_ref) && (m_ref == -INFINITY || (mx - m_ref) * p.scale_log2 > RESCALE_THRESHOLD<HD>);
        if (__any_sync(0xffffffffu, raise)) {
          float alpha = 1.f;
          if (raise) {
            alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - mx) * p.scale_log2);
            m_ref = mx;
            l_run *= alpha;
          }
          if (j > 0) {   // O_T holds the products up to tile j-1 (complete: S_T(j) was issued after them)
#pragma unroll 1
            for (int cc = 0; cc < HD / 32; ++cc) {
              uint32_t tr[32];
              tmem_ld_32x32(o_addr + cc * 32, tr);
              tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 32; ++c) tr[c] = __float_as_uint(__uint_as_float(tr[c]) * alpha);
              tmem_st_32x32(o_addr + cc * 32, tr);
            }
          }
        }
        // ---- P = 2^(S c - m c) as packed bf16 over the first 64 columns of S, in two halves
        const float neg_ms = (m_ref == -INFINITY) ? 0.f : -m_ref * p.scale_log2;
        const uint64_t sc2 = f2_pack(p.scale_log2, p.scale_log2), nm2 = f2_pack(neg_ms, neg_ms);
        uint64_t sum0 = 0ull, sum1 = 0ull;   // (0.f, 0.f)
        uint32_t pk[32];
        exp_half(x0, x1, sc2, nm2, sum0, sum1, pk);
        tmem_st_32x32(s_addr, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[2 * t]);
        exp_half(x2, x3, sc2, nm2, sum0, sum1, pk);
        tmem_st_32x32(s_addr + 32, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[2 * t + 1]);
        float a, b2, c2, d2;
        f2_unpack(sum0, a, b2);
        f2_unpack(sum1, c2, d2);
        l_run += (a + b2) + (c2 + d2);
      }
      if (!ok) break;
      ok = queue_wait(queue, c + 1, abort_flag, p.status);
      if (!ok) break;
      load_unit(queue_read(queue, c + 1));
      const Work w = queue_read(queue, c);
      const int b = w.sample, h = w.head, i = w.place * 2 * BQ + t * BQ + r;     // global query row
      const bool row_valid = i < p.Sq;
      if (n_t > 0) {
        ok = mbar_wait_warp(&o_full[t], u & 1, abort_flag, p.status);
        if (!ok) break;
        ++u;
        tc_fence_after();
      }
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      __nv_bfloat16* orow = p.O + (((long long)b * p.Sq + i) * p.Hq + h) * HD;
#pragma unroll
      for (int cc = 0; cc < HD / 32; ++cc) {
        uint32_t tr[32];
        if (n_t > 0) {
          tmem_ld_32x32(o_addr + cc * 32, tr);
          tmem_ld_wait();
          if (cc == HD / 32 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_free[t]);
          }
#pragma unroll
          for (int k = 0; k < 32; ++k) tr[k] = __float_as_uint(__uint_as_float(tr[k]) * inv);
        } else {
#pragma unroll
          for (int k = 0; k < 32; ++k) tr[k] = 0u;
        }
        if (row_valid) store_bf16_32(orow + cc * 32, tr, p.wide);
      }
      if (row_valid)
        p.lse[((long long)b * p.Hq + h) * p.Sq + i] =
            l_run > 0.f ? (m_ref * p.scale_log2 + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
      queue_free(queue, c);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc<1>(tmem_base, 512); }
}

template <int HD>
int launch_fwd2(const void* q, const void* k, const void* v, Params p, long long q_stride, long long k_stride,
                long long v_stride, cudaStream_t stream) {
  CUtensorMap tmQ, tmK, tmV;
  const auto bf16 = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const auto sw = CU_TENSOR_MAP_SWIZZLE_128B;
  if (!make_tmap_2d(&tmQ, q, bf16, 2, (uint64_t)p.B * p.Sq, (uint64_t)p.Hq * HD, q_stride, BQ, 64, sw) ||
      !make_tmap_2d(&tmK, k, bf16, 2, (uint64_t)p.B * p.Sk, (uint64_t)p.Hkv * HD, k_stride, BKV, 64, sw) ||
      !make_tmap_2d(&tmV, v, bf16, 2, (uint64_t)p.B * p.Sk, (uint64_t)p.Hkv * HD, v_stride, BKV, 64, sw))
    return -2;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_fwd2_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, L2<HD>::TOTAL) !=
        cudaSuccess)
      return -4;
    attr_set = true;
  }
  dim3 grid;
  make_block_order(&p.order, &grid, (p.Sq + 2 * BQ - 1) / (2 * BQ), p.Hq, p.B, p.causal != 0, p.Sk, HD);
  launch_after(flash_fwd2_kernel<HD>, grid, THREADS, L2<HD>::TOTAL, stream, 1, tmQ, tmK, tmV, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace

// Same contract as atb_flash_fwd (flash_attn.cu), for a positive softmax_scale and head dim 128 or 64. With
// `holes` (int32 [B], may be null) the launch writes nothing if any of them is set: the caller, who is about to learn the
// same, takes another path then.
extern "C" int atb_flash_fwd_v2(const void* q, const void* k, const void* v, void* o, float* lse, const int* row_lo,
                                const int* row_hi, int B, int Sq, int Sk, int Hq, int Hkv, long long q_stride,
                                long long k_stride, long long v_stride, int causal, float softmax_scale, void* stream,
                                int* status, int head_dim, const int* holes) {
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  if (Hq % Hkv || (head_dim != 128 && head_dim != 64) || !(softmax_scale > 0.f)) return -1;
  if ((q_stride | k_stride | v_stride) & 7) return -1;
  Params p;
  p.O = (__nv_bfloat16*)o; p.lse = lse; p.row_lo = row_lo; p.row_hi = row_hi;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.status = status;
  p.holes = holes;
  p.wide = (reinterpret_cast<uintptr_t>(o) & 31) == 0;     // rows of whole heads of 128 or 256 bytes
  return head_dim == 64 ? launch_fwd2<64>(q, k, v, p, q_stride, k_stride, v_stride, (cudaStream_t)stream)
                        : launch_fwd2<128>(q, k, v, p, q_stride, k_stride, v_stride, (cudaStream_t)stream);
}
