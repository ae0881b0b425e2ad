// Shared device-side primitives for the sm_100a kernels of atorch_b200:
// mbarrier, TMA (cp.async.bulk.tensor), tcgen05 (TMEM alloc / MMA / load / commit),
// bounded waits and small vector/reduction helpers.
//
// Every wait in this library is bounded: a wait that does not complete within
// ATB_WAIT_LIMIT_NS records an error code in a host-visible word and returns false,
// after which the calling kernel drains and exits without touching the result.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#define ATB_DEVICE __device__ __forceinline__
#define ATB_HOST_DEVICE __host__ __device__ __forceinline__

#ifndef ATB_WAIT_LIMIT_NS
#define ATB_WAIT_LIMIT_NS 2000000000ull  // 2 s: far above any legal wait in these kernels
#endif

// Error codes written to the status word (0 = ok).
enum AtbStatus : int {
  ATB_OK = 0,
  ATB_ERR_WAIT_TIMEOUT = 1,   // an mbarrier / flag wait ran out
  ATB_ERR_BAD_ARG = 2,        // launcher rejected the arguments
  ATB_ERR_TMEM_ALLOC = 3,
  ATB_ERR_PEER_TIMEOUT = 4,   // a peer flag was never set
};

namespace atb {

ATB_DEVICE uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

ATB_DEVICE uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A value that is the same in every lane, as one the compiler knows to be (it can then use uniform registers and branches).
template <typename T>
ATB_DEVICE T warp_uniform(T v) { return __shfl_sync(0xffffffffu, v, 0); }

ATB_DEVICE bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n"
      ".reg .b32 rx;\n"
      ".reg .pred px;\n"
      "elect.sync rx|px, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, px;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// ----------------------------------------------------------------------------------
// mbarrier
// ----------------------------------------------------------------------------------
ATB_DEVICE void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
ATB_DEVICE void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
ATB_DEVICE void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
ATB_DEVICE void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrive on the same-offset barrier of another CTA of the cluster (rank `cta`).
ATB_DEVICE void mbar_arrive_cluster(uint64_t* bar, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(bar)), "r"(cta));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
ATB_DEVICE bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. `abort_flag` is a shared-memory word: once any role of the CTA has
// timed out, all later waits return false at once so the CTA can drain.
// The clock is read only after a thousand polls: a read of %globaltimer costs several hundred clocks, which every wait
// that was not already satisfied used to pay between its first and its second poll.
ATB_DEVICE bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3ff) == 0) {
      if (*abort_flag) return false;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > ATB_WAIT_LIMIT_NS) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, (int)ATB_ERR_WAIT_TIMEOUT);
        return false;
      }
    }
  }
  return true;
}

// The same by a whole converged warp, with one answer for all lanes: a satisfied wait costs 27 clocks, against 103 in the
// loop above, which every lane may leave on its own, and 267 when that loop runs in an `if (lane == 0)` branch (2000
// waits on a completed barrier, clock64). The warps that feed the tensor core wait several times per tile in series with
// the products, so they use this one, and leave to one elected lane only the instructions that must be issued once.
ATB_DEVICE bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
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
  return true;
}

// ----------------------------------------------------------------------------------
// TMA: tiled bulk tensor copies, each into the issuing CTA's own shared memory
// ----------------------------------------------------------------------------------
ATB_DEVICE void tma_prefetch_desc(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tm)) : "memory");
}
ATB_DEVICE void tma_load_2d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
ATB_DEVICE void tma_load_3d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
ATB_DEVICE void tma_load_4d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z),
      "r"(w)
      : "memory");
}
ATB_DEVICE void tma_store_2d(const CUtensorMap* tm, const void* smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tm)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// Element-wise fp32 add of a shared-memory tile into global memory by the TMA unit (asynchronous; completion
// through the bulk group of the issuing thread). Coordinates must be non-negative, x a multiple of 4 floats.
ATB_DEVICE void tma_reduce_add_2d(const CUtensorMap* tm, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
ATB_DEVICE void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
ATB_DEVICE void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
ATB_DEVICE void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
ATB_DEVICE void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ----------------------------------------------------------------------------------
// tcgen05: tensor memory and 5th-generation tensor-core MMA
// ----------------------------------------------------------------------------------
template <int CTA_GROUP = 1>
ATB_DEVICE void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  if constexpr (CTA_GROUP == 1)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
                 "r"(ncols)
                 : "memory");
  else
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
                 "r"(ncols)
                 : "memory");
}
template <int CTA_GROUP = 1>
ATB_DEVICE void tmem_relinquish() {
  if constexpr (CTA_GROUP == 1)
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  else
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <int CTA_GROUP = 1>
ATB_DEVICE void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  if constexpr (CTA_GROUP == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
  else
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
ATB_DEVICE void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
ATB_DEVICE void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 lanes x 32 consecutive fp32 columns: thread t of the warp gets lane (base_lane + t).
ATB_DEVICE void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
ATB_DEVICE void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
ATB_DEVICE void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
ATB_DEVICE void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
ATB_DEVICE void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for tcgen05.mma, 128-byte swizzle.
//   K-major  operand tile: rows of 64 x 16-bit (128 B); 8-row groups 1024 B apart (SBO).
//   MN-major operand tile: k-rows of 64 x 16-bit along MN (128 B); 8 k-rows = 1024 B (SBO);
//                          successive 64-element MN chunks `lbo_bytes` apart.
// It is kept as its low word (start address in 16-byte units, which cannot carry out of its 14 bits inside the 227 KB of a
// CTA, and LBO): adding to it moves on in shared memory, and the high word (SBO, descriptor version, swizzle) is the same for
// every tile with 1024-byte row groups.
//
// The issue path of a whole warp: every lane runs the code, lanes with issue != 0 (one, from elect_one()) execute the
// instruction; the predicate sits on the instruction itself, not on a branch around it. D (+)= A B, accumulate == 0
// overwrites D; `ss`: both operands from shared memory, `ts`: A from tensor memory. A commit makes the mbarrier (cg2: one
// given by its shared::cluster address, own or partner CTA) track all tcgen05 operations that this lane has issued. Measured
// for groups of 8 products of 32 clocks, each group behind a satisfied barrier: 268 clocks a group, 336 with `if (issue)`
// around 64-bit descriptors.
constexpr uint32_t UMMA_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
ATB_DEVICE uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFF) >> 4) | ((lbo_bytes >> 4) << 16);
}
template <int CTA_GROUP = 1>
ATB_DEVICE void umma_ss_issue(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate,
                              uint32_t issue) {
#define ATB_UMMA_SS(GROUP)                                          \
  asm volatile(                                                     \
      "{\n"                                                         \
      ".reg .pred p, q;\n"                                          \
      ".reg .b64 a, b;\n"                                           \
      "mov.b64 a, {%1, %3};\n"                                      \
      "mov.b64 b, {%2, %3};\n"                                      \
      "setp.ne.b32 p, %5, 0;\n"                                     \
      "setp.ne.b32 q, %6, 0;\n"                                     \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], a, b, %4, p;\n" \
      "}\n" ::"r"(tmem_d),                                          \
      "r"(a_lo), "r"(b_lo), "r"(UMMA_DESC_HI), "r"(idesc), "r"(accumulate), "r"(issue) \
      : "memory")
  if constexpr (CTA_GROUP == 1) ATB_UMMA_SS("1");
  else ATB_UMMA_SS("2");
#undef ATB_UMMA_SS
}
// kind::f8f6f4, shared-memory operands, one CTA
ATB_DEVICE void umma_f8_issue(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate,
                              uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      ".reg .b64 a, b;\n"
      "mov.b64 a, {%1, %3};\n"
      "mov.b64 b, {%2, %3};\n"
      "setp.ne.b32 p, %5, 0;\n"
      "setp.ne.b32 q, %6, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %4, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(a_lo), "r"(b_lo), "r"(UMMA_DESC_HI), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
ATB_DEVICE void umma_ts_issue(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate,
                              uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      ".reg .b64 b;\n"
      "mov.b64 b, {%2, %3};\n"
      "setp.ne.b32 p, %5, 0;\n"
      "setp.ne.b32 q, %6, 0;\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "r"(b_lo), "r"(UMMA_DESC_HI), "r"(idesc), "r"(accumulate), "r"(issue)
      : "memory");
}
ATB_DEVICE void umma_commit_issue(uint64_t* bar, uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %1, 0;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(smem_u32(bar)), "r"(issue)
      : "memory");
}

ATB_DEVICE void umma_commit_cg2_issue(uint32_t bar_cluster_addr, uint32_t issue) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %1, 0;\n"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(bar_cluster_addr), "r"(issue)
      : "memory");
}

// Instruction descriptor for kind::f16 / kind::f8f6f4 with fp32 accumulation.
//   fmt: kind::f16: 0 = f16, 1 = bf16;  kind::f8f6f4: 0 = e4m3, 1 = e5m2
ATB_DEVICE constexpr uint32_t umma_idesc(int m, int n, int a_fmt, int b_fmt, bool a_mn_major, bool b_mn_major) {
  return (1u << 4) | ((uint32_t)a_fmt << 7) | ((uint32_t)b_fmt << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Registers per thread of this warpgroup (executed by all its warps; N a multiple of 8). The warpgroups' shares must
// add up to no more than the block was launched with, or the increase waits forever.
template <int N>
ATB_DEVICE void reg_alloc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
ATB_DEVICE void reg_dealloc() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ----------------------------------------------------------------------------------
// Launches that overlap the end of the kernel before them (programmatic dependent launch)
// ----------------------------------------------------------------------------------
// grid_go(): the next launch of the stream, if it is made by launch_after(), may take the SMs that become free from here on.
// grid_wait(): the kernels before have completed and their writes are visible. A kernel launched by launch_after() waits in
// every thread that touches device memory, before it does, on every path: barriers, tensor memory and tensor maps are set up
// before it, under the last blocks of the kernel in front. A kernel that allocates tensor memory says grid_go() in the warp
// that allocates, after it: then no CTA of a successor runs before every CTA of this grid has its tensor memory, and none can
// hold, while it waits for this kernel, what this kernel still needs. Such a kernel takes its inputs by plain pointers: const
// __restrict__ selects the read-only path, which promises that nobody writes while the kernel runs. Kernels that are not worth
// it only say grid_go(). The gap between two kernels was 1.9 us. Before / after matrix products and attention had it: loss of 8
// layers of a 1.3B model on 777 tokens (68 launches) 1479 / 1444 us, forward and backward of one layer on 3000 tokens (23) 1073
// / 1049, a training step of 8 layers (286) 18687 / 18431. Norms, SwiGLU and rotary then: the loss 1485 / 1466, a step of a
// small model (83 launches) 2901 / 2816, the large ones even.
ATB_DEVICE void grid_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
ATB_DEVICE void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ----------------------------------------------------------------------------------
// small helpers
// ----------------------------------------------------------------------------------
ATB_DEVICE float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
ATB_DEVICE float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum; `red` is a shared float[33]. Result is returned to every thread.
ATB_DEVICE float block_sum(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
ATB_DEVICE float block_max(float v, float* red) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

// Order of attention blocks. Under a causal mask the work of a block of rows grows (of a block of keys: shrinks) with its
// place in the sequence, and one CTA fills an SM: head after head, each from its heaviest block down, the last heads' heavy
// blocks started when the other SMs were about to run dry. Here the heaviest blocks of all heads of all samples come first
// and the lightest last (grid: head, place, run), in runs of as many heads as keep what their CTAs stream, two tensors of
// `rows` rows, in half of the L2, three eighths for heads of 3 MB and more, but of 4 heads at least, and all runs as long as
// each other or one head longer.
// The share of the L2 (32 heads of 128, forward and backward, a quarter, three eighths, a half; head after head): 4096 rows
// 568, 568, 566 us; 616. 5120 822, 828, 828; 880. 6144 1132, 1143, 1143; 1203. 7168 1491, 1501, 1520; 1575. 8192 1923, 1925,
// 1953; 2001. 10240 2926, 2916, 2949; 3011. Over 7 to 48 heads three eighths are within 1 % of the best from 3 MB on. Below,
// a half is as good under a plain causal mask and keeps 32 heads of 4096 in one run, which short packed documents like better
// (mean of 8 draws of 9 documents, 32 heads on 8, forward 70.7 against 71.9 us).
// Equal runs: with a short last run the order lost what it gains (7168 x 20 in 18 + 2 heads 1075, in 10 + 10 947, head after
// head 1034; 12288 x 16 2289, 2060, 2182; 10240 x 20 1952, 1845, 1937). Without a causal mask the blocks weigh the same, and
// neighbours that stream the same rows are worth more (4096 x 32 heads: 241 us forward, 254 in the other order): grid (place,
// head, sample) as it was.
struct BlockOrder {
  int heads, all;      // heads of a sample, of the batch; all == 0: the order without a causal mask
  int run, longer;     // heads of a run; the first `longer` runs have one more
};
inline void make_block_order(BlockOrder* o, dim3* grid, int blocks, int heads, int batch, bool causal, long long rows,
                             int head_dim) {
  const long long all = (long long)heads * batch, head = rows * head_dim * 4;
  const long long fit = (head < (3LL << 20) ? 64LL << 20 : 48LL << 20) / head, least = fit < 4 ? 4 : fit;
  const long long want = least < all ? least : all, runs = (all + want - 1) / want;
  if (causal && blocks <= 65535 && runs <= 65535 && all <= 0x7fffffffLL) {
    *o = BlockOrder{heads, (int)all, (int)(all / runs), (int)(all % runs)};
    *grid = dim3((unsigned)((all + runs - 1) / runs), blocks, (unsigned)runs);
  } else {
    *o = BlockOrder{heads, 0, 0, 0};
    *grid = dim3(blocks, heads, batch);
  }
}
// place: 0 = the heaviest block of its head; idx: the block's index in the grid. False: no block (a run that is one head
// shorter).
ATB_DEVICE bool block_of(const BlockOrder& o, const uint3& idx, int& place, int& blocks, int& head, int& sample) {
  if (o.all == 0) {
    place = idx.x;
    blocks = gridDim.x;
    head = idx.y;
    sample = idx.z;
    return true;
  }
  const int run = idx.z;
  if ((int)idx.x >= o.run + (run < o.longer ? 1 : 0)) return false;
  place = idx.y;
  blocks = gridDim.y;
  head = run * o.run + min(run, o.longer) + idx.x;
  sample = 0;
  if (o.all != o.heads) {
    sample = head / o.heads;
    head -= sample * o.heads;
  }
  return true;
}

// 32-byte global store (32-byte aligned): one whole sector per thread.
ATB_DEVICE void stg_v8(void* p, const uint32_t* r) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Two fp32 values in one 64-bit register and the packed arithmetic of sm_100 on them: one instruction
// does two fused multiply-adds (or adds), which halves the issue slots of element-wise fp32 work.
ATB_DEVICE uint64_t f2_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
ATB_DEVICE uint64_t f2_pack_bits(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
ATB_DEVICE void f2_unpack(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
ATB_DEVICE uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
ATB_DEVICE uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
ATB_DEVICE uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// bit c set: key k0 + c lies in [lo, hi)
ATB_DEVICE uint32_t visible_keys(int k0, int lo, int hi) {
  const int a = min(max(lo - k0, 0), 32), e = min(max(hi - k0, 0), 32);
  const uint32_t below_e = e == 32 ? 0xffffffffu : (1u << e) - 1u, below_a = a == 32 ? 0xffffffffu : (1u << a) - 1u;
  return below_e & ~below_a;
}

// Attention dropout: a counter-based keep decision per (batch*head, query row, key column), the same in the
// forward and the backward kernels and reproducible on the host (ops/flash.py: dropout_keep_mask). One hash
// serves two neighbouring columns: the low 16 bits decide the even column, the high 16 bits the odd one;
// an element is kept when its 16 bits are >= thr16 = round(p * 65536).
struct DropParams {
  uint32_t thr16;      // 0: no dropout
  uint32_t seed_lo, seed_hi;
  float keep_scale;    // 65536 / (65536 - thr16)
};
// Additive attention bias (bf16), added to the scaled scores: element (b, h, i, j) at ptr[b sb + h sh + i sq + j];
// sb / sh = 0 broadcast over batch / heads. Rows are read in 16-byte pieces: sq, sb, sh and the key count are
// multiples of 8 and ptr is 16-byte aligned. ptr == nullptr: none.
struct BiasParams {
  const __nv_bfloat16* ptr;
  long long sb, sh, sq;
};
ATB_HOST_DEVICE uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}
ATB_HOST_DEVICE uint32_t drop_row_key(const DropParams& d, uint32_t bh, uint32_t row) {
  const uint32_t base = hash32(d.seed_lo ^ (bh * 0x9E3779B1U)) ^ d.seed_hi;
  return hash32(base + row * 0x85EBCA77U);
}
// bits for columns (col, col + 1), col even
ATB_HOST_DEVICE uint32_t drop_pair_bits(uint32_t row_key, uint32_t col) {
  return hash32(row_key ^ ((col >> 1) * 0xC2B2AE3DU));
}

// 2^x on the special-function unit (ex2.approx.ftz): -inf -> 0, relative error ~2^-22
ATB_DEVICE float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

ATB_DEVICE uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
ATB_DEVICE float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(h);
}

// 32 fp32 bit patterns of a row as bf16: whole 32-byte sectors where the row allows it (`wide`), else 16-byte pieces
ATB_DEVICE void store_bf16_32(__nv_bfloat16* p, const uint32_t (&x)[32], bool wide) {
  uint32_t o[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i] = pack_bf16x2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1]));
  if (wide) {
    stg_v8(p, o);
    stg_v8(p + 16, o + 8);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<uint4*>(p + 8 * i) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
  }
}

template <typename T>
ATB_DEVICE float to_f32(T v);
template <>
ATB_DEVICE float to_f32<float>(float v) { return v; }
template <>
ATB_DEVICE float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
ATB_DEVICE float to_f32<__half>(__half v) { return __half2float(v); }
template <typename T>
ATB_DEVICE T from_f32(float v);
template <>
ATB_DEVICE float from_f32<float>(float v) { return v; }
template <>
ATB_DEVICE __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
ATB_DEVICE __half from_f32<__half>(float v) { return __float2half_rn(v); }

}  // namespace atb

// Host-side: encode a 2-D tiled tensor map through the driver entry point (no libcuda link).
#include <mutex>
#include <cstdio>
#include <utility>
namespace atb {
// Launch that may start before the kernel in front has ended (see grid_wait), in clusters of `cluster` CTAs.
template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, int cluster,
                                A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline PFN_encodeTiled get_encode_tiled() {
  static PFN_encodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encodeTiled>(p);
  });
  return fn;
}
// rows x cols row-major matrix of `elt_bytes` elements with row pitch `ld` (elements); box = box_rows x box_cols.
// Returns false if the driver rejects it (alignment: base 16 B, pitch multiple of 16 B).
inline bool make_tmap_2d(CUtensorMap* tm, const void* base, CUtensorMapDataType dt, int elt_bytes, uint64_t rows,
                         uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle sw) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * (uint64_t)elt_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // first CUDA work of this host thread (e.g. an autograd worker): bind the primary context
    // through the runtime, then encode again
    cudaFree(nullptr);
    r = enc(tm, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS)
    fprintf(stderr, "atb: cuTensorMapEncodeTiled failed (%d): base=%p rows=%llu cols=%llu ld=%llu box=%ux%u elt=%d\n",
            (int)r, base, (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)ld, box_rows,
            box_cols, elt_bytes);
  return r == CUDA_SUCCESS;
}
}  // namespace atb
