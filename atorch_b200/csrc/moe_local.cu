// Row movement of a routed layer on one GPU (bf16 rows of H elements, H a multiple of 8). `slot_of[t * k + j]` is the row
// of the expert-sorted buffer that holds choice j of token t (-1: none).
//   gather_sum    out[t] = sum_j w[t, j] src[slot_of[t, j]]     unpermute forward (w = routing probabilities) and
//                                                               permute backward (no w)
//   gather_rows   out[i] = src[order[i] / k]                    permute forward
//   ungather      dsrc[i] = w[s] dout[s / k], dw[s] = <dout[s / k], src[i]> with s = order[i]        unpermute backward
// Bound by memory, one pass each with 16-byte pieces and fp32 sums. As tensor operations (zeros, index_copy, product,
// sum; index_add with atomics backward) this was 13 passes over [T k, H]: for 4096 tokens, top 2, H = 4096 0.75 ms of an
// 8.5 ms forward and backward, 0.1 ms here.
#include "common.cuh"

namespace {
using namespace atb;

ATB_DEVICE float weight_at(const void* w, int dtype, long long i) {
  return dtype == 0 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w)[i]) : reinterpret_cast<const float*>(w)[i];
}

__global__ void invert_perm_kernel(const long long* __restrict__ order, int* __restrict__ slot_of, int n) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) {
    const long long s = order[i];
    if (s >= 0 && s < n) slot_of[s] = i;
  }
}

__global__ void __launch_bounds__(256) gather_sum_kernel(const __nv_bfloat16* __restrict__ src,
                                                         const int* __restrict__ slot_of, const void* __restrict__ w,
                                                         int w_dtype, __nv_bfloat16* __restrict__ out, int k, int H) {
  grid_go();
  const long long t = blockIdx.x;
  for (int c = threadIdx.x; c < H / 8; c += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < k; ++j) {
      const int s = slot_of[t * k + j];
      if (s < 0) continue;
      const float f = w ? weight_at(w, w_dtype, t * k + j) : 1.f;
      const uint4 u = *reinterpret_cast<const uint4*>(src + (long long)s * H + c * 8);
      const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 v = unpack_bf16x2(x[e]);
        acc[2 * e] += f * v.x;
        acc[2 * e + 1] += f * v.y;
      }
    }
    *reinterpret_cast<uint4*>(out + t * H + c * 8) =
        make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                   pack_bf16x2(acc[6], acc[7]));
  }
}

__global__ void __launch_bounds__(256) ungather_kernel(const __nv_bfloat16* __restrict__ dout,
                                                       const __nv_bfloat16* __restrict__ src,
                                                       const long long* __restrict__ order, const void* __restrict__ w,
                                                       int w_dtype, __nv_bfloat16* __restrict__ dsrc,
                                                       void* __restrict__ dw, int k, int H) {
  grid_go();
  __shared__ float red[33];
  const long long s = order[blockIdx.x];
  if (s < 0 || s >= (long long)gridDim.x) return;
  const long long t = s / k, row = (long long)blockIdx.x * H;
  float dot = 0.f;
  {
    const float f = w ? weight_at(w, w_dtype, s) : 1.f;
    for (int c = threadIdx.x; c < H / 8; c += 256) {
      const uint4 d = *reinterpret_cast<const uint4*>(dout + t * H + c * 8);
      const uint32_t x[4] = {d.x, d.y, d.z, d.w};
      uint4 u = make_uint4(0u, 0u, 0u, 0u);
      if (dw != nullptr) u = *reinterpret_cast<const uint4*>(src + row + c * 8);
      const uint32_t y[4] = {u.x, u.y, u.z, u.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 a = unpack_bf16x2(x[e]), b = unpack_bf16x2(y[e]);
        dot += a.x * b.x + a.y * b.y;
        o[e] = pack_bf16x2(f * a.x, f * a.y);
      }
      if (dsrc != nullptr) *reinterpret_cast<uint4*>(dsrc + row + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (dw != nullptr) {
    dot = block_sum(dot, red);
    if (threadIdx.x == 0) {
      if (w_dtype == 0) reinterpret_cast<__nv_bfloat16*>(dw)[s] = __float2bfloat16_rn(dot);
      else reinterpret_cast<float*>(dw)[s] = dot;
    }
  }
}

// Stable counting sort of n routed expert ids by one block: counts[e], order (the sorted positions) and slot, its inverse.
// Every warp owns a run of the ids and walks it twice, 32 ids a step: lanes with the same id find each other by
// match_any, so a step adds each id once (first walk, the warp's histogram) or hands out consecutive places (second walk).
// Between the walks the histograms become starting places, expert by expert and warp by warp within an expert. Bound by
// latency: the ids of 8 steps are loaded together. Ids outside [0, E) are counted nowhere and go to the end.
// 8192 ids of 8 experts: 10 us, in place of a histogram (with a host synchronisation of its own), a radix sort of 64-bit
// keys and two inversions, 32 launches and 100 us of device time. Forward and backward of 8 experts of 4096 x 1024 on
// 131 tokens 1200 -> 760 us, of 4 x 8192 x 2048 on 1000 tokens 1000 -> 700. The block takes 84 us for
// 32768 ids of 256 experts (34 us for 8 experts), by then no less device time than the sort's launches: the limit.
constexpr int ROUTE_MAX_E = 256, ROUTE_MAX_N = 32768, ROUTE_STEPS = 8;
__global__ void __launch_bounds__(1024) route_kernel(const long long* __restrict__ idx, int n, int E,
                                                     long long* __restrict__ counts, long long* __restrict__ order,
                                                     int* __restrict__ slot) {
  __shared__ int place[32][ROUTE_MAX_E + 1];
  __shared__ int scan[2][ROUTE_MAX_E + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int run = ((n + 31) / 32 + 31) / 32 * 32;      // ids per warp, whole steps
  const int lo = min(n, warp * run), hi = min(n, lo + run);
  for (int i = threadIdx.x; i < 32 * (ROUTE_MAX_E + 1); i += 1024) (&place[0][0])[i] = 0;
  __syncthreads();
  auto walk = [&](auto&& step) {
    for (int base = lo; base < hi; base += 32 * ROUTE_STEPS) {
      int e[ROUTE_STEPS];
#pragma unroll
      for (int s = 0; s < ROUTE_STEPS; ++s) {
        const int i = base + s * 32 + lane;
        const long long v = i < hi ? idx[i] : 0;
        e[s] = i >= hi ? -1 : v < 0 || v >= E ? E : (int)v;
      }
#pragma unroll
      for (int s = 0; s < ROUTE_STEPS; ++s) {
        const unsigned same = __match_any_sync(0xffffffffu, e[s]);
        step(base + s * 32 + lane, e[s], same);
        __syncwarp();
        if (e[s] >= 0 && lane == __ffs(same) - 1) place[warp][e[s]] += __popc(same);
        __syncwarp();
      }
    }
  };
  walk([](int, int, unsigned) {});
  __syncthreads();
  const int b = threadIdx.x;
  int total = 0;
  if (b <= E) {
    for (int w = 0; w < 32; ++w) {
      const int c = place[w][b];
      place[w][b] = total;
      total += c;
    }
    scan[0][b] = total;
    if (b < E) counts[b] = total;
  }
  __syncthreads();
  int cur = 0;
  for (int d = 1; d <= E; d <<= 1, cur ^= 1) {         // inclusive scan over the experts
    if (b <= E) scan[cur ^ 1][b] = scan[cur][b] + (b >= d ? scan[cur][b - d] : 0);
    __syncthreads();
  }
  if (b <= E) {
    const int first = scan[cur][b] - total;
    for (int w = 0; w < 32; ++w) place[w][b] += first;
  }
  __syncthreads();
  walk([&](int i, int e, unsigned same) {
    if (e >= 0) {
      const int p = place[warp][e] + __popc(same & ((1u << lane) - 1));
      order[p] = i;
      slot[i] = p;
    }
  });
}

__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ src, const long long* __restrict__ order,
                                                          uint4* __restrict__ out, int k, int pieces) {
  grid_go();
  const long long s = order[blockIdx.x] / k;
  for (int c = threadIdx.x; c < pieces; c += 256) out[(long long)blockIdx.x * pieces + c] = src[s * pieces + c];
}

bool aligned16(const void* a, const void* b, const void* c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}
}  // namespace

// slot_of[order[i]] = i; entries that `order` (int64 [n]) does not name become -1.
extern "C" int atb_invert_perm(const long long* order, int* slot_of, int n, void* stream) {
  if (n <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(slot_of, 0xff, (size_t)n * 4, st) != cudaSuccess) return -5;
  invert_perm_kernel<<<(n + 255) / 256, 256, 0, st>>>(order, slot_of, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// counts [E], order [n] int64, slot [n] int32 from idx [n]; n at most 32768, E at most 256.
extern "C" int atb_moe_sort_ids(const long long* idx, int n, int E, long long* counts, long long* order, int* slot,
                             void* stream) {
  if (n < 0 || n > ROUTE_MAX_N || E < 1 || E > ROUTE_MAX_E) return -1;
  route_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(idx, n, E, counts, order, slot);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// out[i] = src[order[i] / k] for n rows of H bf16; order names rows of src (0 <= order[i] / k < rows).
extern "C" int atb_moe_gather_rows(const void* src, const long long* order, void* out, int n, int k, int H, void* stream) {
  if (n <= 0 || H <= 0) return 0;
  if ((H & 7) || k < 1 || !aligned16(src, out, nullptr)) return -1;
  gather_rows_kernel<<<n, 256, 0, (cudaStream_t)stream>>>((const uint4*)src, order, (uint4*)out, k, H / 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// w_dtype: 0 bf16, 2 fp32; w may be null (weights of 1).
extern "C" int atb_moe_gather_sum(const void* src, const int* slot_of, const void* w, int w_dtype, void* out, int T, int k,
                                  int H, void* stream) {
  if (T <= 0 || H <= 0) return 0;
  if ((H & 7) || k < 1 || !aligned16(src, out, nullptr)) return -1;
  gather_sum_kernel<<<T, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, slot_of, w, w_dtype,
                                                        (__nv_bfloat16*)out, k, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// n sorted rows; dsrc or dw may be null, dw has the type of w (bf16 or fp32). Rows whose entry of `order` is outside [0, n)
// are left alone.
extern "C" int atb_moe_ungather(const void* dout, const void* src, const long long* order, const void* w, int w_dtype,
                                void* dsrc, void* dw, int n, int k, int H, void* stream) {
  if (n <= 0 || H <= 0) return 0;
  if ((H & 7) || k < 1 || !aligned16(dout, src, dsrc)) return -1;
  ungather_kernel<<<n, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)src, order, w,
                                                       w_dtype, (__nv_bfloat16*)dsrc, dw, k, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
