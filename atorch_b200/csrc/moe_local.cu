// Row movement of a routed layer on one GPU (bf16 rows of H elements, H a multiple of 8). `slot_of[t * k + j]` is the row
// of the expert-sorted buffer that holds choice j of token t (-1: none).
//   gather_sum    out[t] = sum_j w[t, j] src[slot_of[t, j]]     unpermute forward (w = routing probabilities) and
//                                                               permute backward (no w)
//   scatter_mul   dsrc[slot_of[t, j]] = w[t, j] dout[t],  dw[t, j] = <dout[t], src[slot_of[t, j]]>   unpermute backward
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

__global__ void __launch_bounds__(256) scatter_mul_kernel(const __nv_bfloat16* __restrict__ dout,
                                                          const __nv_bfloat16* __restrict__ src,
                                                          const int* __restrict__ slot_of, const void* __restrict__ w,
                                                          int w_dtype, __nv_bfloat16* __restrict__ dsrc,
                                                          void* __restrict__ dw, int k, int H) {
  __shared__ float red[33];
  const long long t = blockIdx.x / k;
  const int s = slot_of[blockIdx.x];
  float dot = 0.f;
  if (s >= 0) {
    const float f = w ? weight_at(w, w_dtype, blockIdx.x) : 1.f;
    for (int c = threadIdx.x; c < H / 8; c += 256) {
      const uint4 d = *reinterpret_cast<const uint4*>(dout + t * H + c * 8);
      const uint32_t x[4] = {d.x, d.y, d.z, d.w};
      uint4 u = make_uint4(0u, 0u, 0u, 0u);
      if (dw != nullptr) u = *reinterpret_cast<const uint4*>(src + (long long)s * H + c * 8);
      const uint32_t y[4] = {u.x, u.y, u.z, u.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 a = unpack_bf16x2(x[e]), b = unpack_bf16x2(y[e]);
        dot += a.x * b.x + a.y * b.y;
        o[e] = pack_bf16x2(f * a.x, f * a.y);
      }
      if (dsrc != nullptr) *reinterpret_cast<uint4*>(dsrc + (long long)s * H + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (dw != nullptr) {
    dot = block_sum(dot, red);
    if (threadIdx.x == 0) {
      if (w_dtype == 0) reinterpret_cast<__nv_bfloat16*>(dw)[blockIdx.x] = __float2bfloat16_rn(dot);
      else reinterpret_cast<float*>(dw)[blockIdx.x] = dot;
    }
  }
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

// w_dtype: 0 bf16, 2 fp32; w may be null (weights of 1).
extern "C" int atb_moe_gather_sum(const void* src, const int* slot_of, const void* w, int w_dtype, void* out, int T, int k,
                                  int H, void* stream) {
  if (T <= 0 || H <= 0) return 0;
  if ((H & 7) || k < 1 || !aligned16(src, out, nullptr)) return -1;
  gather_sum_kernel<<<T, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)src, slot_of, w, w_dtype,
                                                        (__nv_bfloat16*)out, k, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// dsrc (rows that no choice names are left alone) or dw may be null; dw has the type of w (bf16 or fp32).
extern "C" int atb_moe_scatter_mul(const void* dout, const void* src, const int* slot_of, const void* w, int w_dtype,
                                   void* dsrc, void* dw, int T, int k, int H, void* stream) {
  if (T <= 0 || H <= 0) return 0;
  if ((H & 7) || k < 1 || (long long)T * k > 0x7fffffffLL || !aligned16(dout, src, dsrc)) return -1;
  scatter_mul_kernel<<<(unsigned)T * (unsigned)k, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)dout, (const __nv_bfloat16*)src, slot_of, w, w_dtype, (__nv_bfloat16*)dsrc, dw, k, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
