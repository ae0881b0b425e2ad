// Blocks of a grid worked off by the CTAs that are already running.
//
// One CTA of the attention kernels fills an SM, so nothing overlapped the start of a block (tensor memory, barriers, first
// loads, first products: 4 to 5 us) and its end (last products, results out of tensor memory: 2 us) with other work. Here a
// running CTA takes over blocks that have not started (clusterlaunchcontrol.try_cancel: the hardware scheduler withdraws the
// next block of the grid and hands its index to the caller), in the order in which they would have started, and the roles
// of the CTA go from one block into the next on their own: the producer loads the next block's tiles and the first products run
// while the element-wise warps still finish the last one. No counter in memory, nothing to reset, nothing shared between
// launches; a launch of one wave finds nothing to take over and runs as before.
//
// A scheduler warp asks, works out what the roles need to know about a block and publishes it in a ring of two entries; the
// roles (readers) take the entries in order. It asks for the next block when the producer says so (queue_claim, close to the
// end of the loads of the current one): a block claimed early cannot go to an SM that becomes free.
#pragma once
#include "common.cuh"

namespace atb {

// One unit of work: place, head and sample of block_of, four values of the kernel's own, and whether there is any.
struct alignas(16) Work {
  int place, head, sample, more;
  int v0, v1, v2, v3;
};

struct alignas(16) WorkQueue {
  uint4 answer;                // of try_cancel, written by the asynchronous proxy
  Work ring[2];
  uint64_t full[2], empty[2];  // per entry
  uint64_t claim;              // the producer wants the next block
  uint64_t answered;
};

ATB_DEVICE void queue_init(WorkQueue* q, int reader_warps) {
  for (int i = 0; i < 2; ++i) {
    mbar_init(&q->full[i], 1);
    mbar_init(&q->empty[i], reader_warps);
  }
  mbar_init(&q->claim, 1);
  mbar_init(&q->answered, 1);
}

// The c-th unit of this CTA, by every lane of a reader warp: wait for it (false: the wait ran out), read it, give its place back.
// The element-wise warps of the forward and the dK/dV kernel hold it until its results are stored, and read it again where
// they need it: eight values kept in registers through the loop over the tiles slowed that loop by 6 to 8 % (one wave of
// 8192 keys: head dim 64 139 -> 128 us, 128 128 -> 121). In the dQ kernel it makes no difference.
ATB_DEVICE bool queue_wait(WorkQueue* q, int c, volatile int* abort_flag, int* status) {
  return mbar_wait_warp(&q->full[c & 1], (c >> 1) & 1, abort_flag, status);
}
ATB_DEVICE Work queue_read(const WorkQueue* q, int c) {
  const int4 a = *reinterpret_cast<const int4*>(&q->ring[c & 1].place), b = *reinterpret_cast<const int4*>(&q->ring[c & 1].v0);
  return Work{warp_uniform(a.x), warp_uniform(a.y), warp_uniform(a.z), warp_uniform(a.w),
              warp_uniform(b.x), warp_uniform(b.y), warp_uniform(b.z), warp_uniform(b.w)};
}
ATB_DEVICE void queue_free(WorkQueue* q, int c) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(&q->empty[c & 1]);
}
// All three, for the warps that feed the tensor core.
ATB_DEVICE bool queue_next(WorkQueue* q, int c, Work& w, volatile int* abort_flag, int* status) {
  if (!queue_wait(q, c, abort_flag, status)) return false;
  w = queue_read(q, c);
  queue_free(q, c);
  return true;
}

// Once per unit, by one reader warp (the producer).
ATB_DEVICE void queue_claim(WorkQueue* q) {
  if ((threadIdx.x & 31) == 0) mbar_arrive(&q->claim);
}

ATB_DEVICE void clc_ask(WorkQueue* q) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(&q->answer)),
               "r"(smem_u32(&q->answered))
               : "memory");
}
// True: the block `idx` was withdrawn and is this CTA's to do. After a false no further question may be asked.
ATB_DEVICE bool clc_answer(const WorkQueue* q, uint3& idx) {
  uint32_t ok, x, y, z;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      ".reg .b128 r;\n"
      "ld.shared.b128 r, [%4];\n"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "mov.u32 %1, 0;\n"
      "mov.u32 %2, 0;\n"
      "mov.u32 %3, 0;\n"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, r;\n"
      "}\n"
      : "=r"(ok), "=r"(x), "=r"(y), "=r"(z)
      : "r"(smem_u32(&q->answer))
      : "memory");
  idx = make_uint3(warp_uniform(x), warp_uniform(y), warp_uniform(z));
  return warp_uniform(ok) != 0;
}

// The scheduler warp's whole life, by all its lanes, after grid_wait. describe(Work&, blocks) fills in v0..v3 of a block
// (`blocks`: blocks of a head); its lanes may load and shuffle. After an error of a kernel before this one the first unit
// is published as none: one warp looks, the roles all take the same from the queue, and the load runs beside those of the unit.
template <class F>
ATB_DEVICE void queue_run(WorkQueue* q, const BlockOrder& order, F describe, volatile int* abort_flag, int* status) {
  const bool first_lane = (threadIdx.x & 31) == 0;
  const int failed = status != nullptr ? *reinterpret_cast<volatile int*>(status) : 0;
  uint3 idx = blockIdx;
  bool have = true;
  uint32_t asked = 0;
  // one question; false: a wait ran out
  auto ask = [&]() -> bool {
    if (first_lane) {
      fence_proxy_async_smem();        // the last answer has been read
      mbar_expect_tx(&q->answered, 16);
      clc_ask(q);
    }
    __syncwarp();
    if (!mbar_wait_warp(&q->answered, asked & 1, abort_flag, status)) return false;
    ++asked;
    have = clc_answer(q, idx);
    __syncwarp();
    return true;
  };
  for (int c = 0;; ++c) {
    Work w = {};
    int blocks = 0;
    while (have && !block_of(order, idx, w.place, blocks, w.head, w.sample))   // an index without a block
      if (!ask()) return;
    if (have) describe(w, blocks);
    if (c == 0 && warp_uniform(failed) != 0) have = false;
    w.more = have;
    const int e = c & 1;
    if (!mbar_wait_warp(&q->empty[e], ((c >> 1) & 1) ^ 1, abort_flag, status)) return;
    if (first_lane) {
      q->ring[e] = w;
      mbar_arrive(&q->full[e]);
    }
    __syncwarp();
    if (!have) return;
    if (!mbar_wait_warp(&q->claim, c & 1, abort_flag, status) || !ask()) return;
  }
}

}  // namespace atb
