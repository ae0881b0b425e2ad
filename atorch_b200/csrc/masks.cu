// Per-row key intervals [lo, hi) of the flash-attention kernels from the mask arguments of the attention operator, in
// one launch: causal, GLM break points, packed GLM pairs, key padding (left or right; `holes[b]` reports a sample whose
// valid keys are not contiguous), packed sequences. In separate tensor operations the lowering took 13 to 27 launches,
// 0.2 to 0.3 ms of host time in front of attention kernels of 0.1 ms.
#include "common.cuh"

namespace {
using namespace atb;

struct MaskArgs {
  const void *glm, *pack, *cu;       // int32 or int64, null: absent
  const unsigned char* keys;         // [B, Sk], nonzero = valid key
  int glm64, pack64, cu64;
  int pairs, n_cu;                   // packed GLM pairs per sample; entries of cu (sequences + 1)
};

ATB_DEVICE long long ld_index(const void* p, int is64, long long i) {
  return is64 ? reinterpret_cast<const long long*>(p)[i] : reinterpret_cast<const int*>(p)[i];
}

__global__ void __launch_bounds__(256) row_intervals_kernel(int* __restrict__ row_lo, int* __restrict__ row_hi,
                                                            int* __restrict__ holes, int Sq, int Sk, int causal_like,
                                                            MaskArgs m) {
  grid_go();
  __shared__ int s_cnt, s_first, s_last;
  const int b = blockIdx.y, i = blockIdx.x * 256 + threadIdx.x;
  if (m.keys != nullptr) {
    if (threadIdx.x == 0) { s_cnt = 0; s_first = INT_MAX; s_last = -1; }
    __syncthreads();
    int cnt = 0, first = INT_MAX, last = -1;
#pragma unroll 4
    for (int j = threadIdx.x; j < Sk; j += 256) {
      if (m.keys[(long long)b * Sk + j] != 0) { ++cnt; first = min(first, j); last = j; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
      last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
    }
    if ((threadIdx.x & 31) == 0) { atomicAdd(&s_cnt, cnt); atomicMin(&s_first, first); atomicMax(&s_last, last); }
    __syncthreads();
    if (threadIdx.x == 0 && blockIdx.x == 0) holes[b] = s_cnt > 0 && s_last - s_first + 1 != s_cnt;
  }
  if (i >= Sq) return;
  long long lo = 0, hi = Sk;
  if (causal_like) hi = min((long long)i + 1 + Sk - Sq, (long long)Sk);
  if (m.glm != nullptr) hi = max(hi, ld_index(m.glm, m.glm64, b));
  if (m.pack != nullptr) {
    hi = max(hi, 0LL);
    for (int k = 0; k < m.pairs; ++k) {
      const long long s = ld_index(m.pack, m.pack64, (2LL * b) * m.pairs + k);
      const long long e = ld_index(m.pack, m.pack64, (2LL * b + 1) * m.pairs + k);
      if (s >= 0 && e >= 0 && s <= i) hi = max(hi, e);
    }
  }
  if (m.cu != nullptr) {
    int a = 0, e = m.n_cu - 1;                   // sequences whose end (cu[1..]) is at or before this row
    while (a < e) {
      const int mid = (a + e) >> 1;
      if (ld_index(m.cu, m.cu64, mid + 1) <= i) a = mid + 1;
      else e = mid;
    }
    const int seg = min(a, m.n_cu - 2);
    lo = max(lo, ld_index(m.cu, m.cu64, seg));
    if (!causal_like) hi = min(hi, ld_index(m.cu, m.cu64, seg + 1));
  }
  if (m.keys != nullptr) {
    lo = max(lo, (long long)(s_cnt > 0 ? s_first : 0));
    hi = min(hi, (long long)(s_cnt > 0 ? s_last + 1 : 0));
  }
  hi = min(hi, (long long)Sk);
  row_lo[(long long)b * Sq + i] = (int)lo;
  row_hi[(long long)b * Sq + i] = (int)hi;
}
}  // namespace

// row_lo, row_hi: int32 [B, Sq]; holes: int32 [B], written when keys != null. glm [B], pack [B, 2, pairs], cu [n_cu] are
// int32 (x64 == 0) or int64; any may be null. causal_like: causal, or any GLM form.
extern "C" int atb_row_intervals(int* row_lo, int* row_hi, int* holes, int B, int Sq, int Sk, int causal_like,
                                 const void* glm, int glm64, const void* pack, int pack64, int pairs,
                                 const unsigned char* keys, const void* cu, int cu64, int n_cu, void* stream) {
  if (B <= 0 || Sq <= 0) return 0;
  if (B > 65535 || (cu != nullptr && n_cu < 2) || (keys != nullptr && holes == nullptr)) return -1;
  MaskArgs m{glm, pack, cu, keys, glm64, pack64, cu64, pairs, n_cu};
  row_intervals_kernel<<<dim3((Sq + 255) / 256, B), 256, 0, (cudaStream_t)stream>>>(row_lo, row_hi, holes, Sq, Sk,
                                                                                   causal_like, m);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
