// Gradient of an embedding table: row v (+)= the sum of the gradients of the tokens whose id is v, in the order of the
// tokens, in fp32, rounded once. Two kernels, no atomics on values and no order that depends on timing:
//   embed_sort    a stable counting sort of the ids. A CTA owns a range of rows and reads all ids twice: the first time it counts
//                 its own per row and warp and the ids below its range (which is where its part of the result begins), the
//                 second time it writes the tokens. The ids are small (64 KB for 8192) and come out of L2; in exchange no CTA
//                 waits for another and nothing has to be cleared before.
//   embed_rows    a warp per row and 512 columns; a row with many tokens (padding) is summed by the eight warps of its block.
// Bound by memory: the gradients of the tokens are read once, the rows that have any are read and written. The library wrote a
// gradient of the whole table (zeros, then rows) that was then added to the gradient buffer, three more passes over the
// table, after a sort in several launches. 4096 tokens on 32000 rows of 2048, random ids: 315 us in 30 launches, now 5 + 37 us; the
// training step of 8 layers that it belongs to 18431 -> 18202 us.
#include "common.cuh"

namespace {
using namespace atb;

constexpr int SORT_WARPS = 16, BATCH = 8;
constexpr int MAX_RANGE = 1024;          // rows of a CTA: 16 warps x 1024 counters are 64 KB of shared memory
constexpr int ROWS = 32, COLS = 512;     // rows of a block, columns of a block
constexpr int MANY = 64;                 // tokens from which on the whole block sums a row

__global__ void __launch_bounds__(SORT_WARPS * 32)
embed_sort_kernel(const long long* __restrict__ ids, int* __restrict__ start, int* __restrict__ order, int T, int V, int range) {
  extern __shared__ int cnt[];           // [SORT_WARPS][range]
  __shared__ int scan[SORT_WARPS], base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long lo = (long long)blockIdx.x * range;
  const int rows = (int)min((long long)range, V - lo);
  for (int i = threadIdx.x; i < SORT_WARPS * range; i += SORT_WARPS * 32) cnt[i] = 0;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();

  const int span = ((T + SORT_WARPS - 1) / SORT_WARPS + 31) & ~31;
  const int beg = min(warp * span, T), end = min(beg + span, T);
  int* mine = cnt + warp * range;
  auto load = [&](int at, long long (&id)[BATCH]) {       // V behind the end, counted nowhere
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const int i = at + u * 32 + lane;
      id[u] = i < end ? ids[i] : (long long)V;
    }
  };
  int below = 0;
  for (int at = beg; at < end; at += 32 * BATCH) {
    long long id[BATCH];
    load(at, id);
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const long long r = id[u] - lo;
      below += r < 0;
      if (r >= 0 && r < rows) atomicAdd(&mine[r], 1);
    }
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0) atomicAdd(&base, below);
  __syncthreads();

  // where each row begins, and in it each warp
  const int per = (range + SORT_WARPS * 32 - 1) / (SORT_WARPS * 32);
  const int r0 = min((int)threadIdx.x * per, rows), r1 = min(r0 + per, rows);
  int sum = 0;
  for (int r = r0; r < r1; ++r)
    for (int w = 0; w < SORT_WARPS; ++w) sum += cnt[w * range + r];
  int before = sum;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const int o = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += o;
  }
  if (lane == 31) scan[warp] = before;
  __syncthreads();
  int at_row = base + before - sum, total = 0;
  for (int w = 0; w < SORT_WARPS; ++w) {
    if (w < warp) at_row += scan[w];
    total += scan[w];
  }
  for (int r = r0; r < r1; ++r) {
    start[lo + r] = at_row;
    for (int w = 0; w < SORT_WARPS; ++w) {
      const int n = cnt[w * range + r];
      cnt[w * range + r] = at_row;
      at_row += n;
    }
  }
  if (threadIdx.x == 0 && lo + rows == V) start[V] = base + total;
  if (total == 0) return;
  __syncthreads();

  for (int at = beg; at < end; at += 32 * BATCH) {
    long long id[BATCH];
    load(at, id);
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const long long r = id[u] - lo;
      const bool in = r >= 0 && r < rows;
      if (!__any_sync(0xffffffffu, in)) continue;
      const unsigned same = __match_any_sync(0xffffffffu, in ? (int)r : -1);
      const int rank = __popc(same & ((1u << lane) - 1));
      if (in) order[mine[r] + rank] = at + u * 32 + lane;
      __syncwarp();
      if (in && rank == 0) mine[r] += __popc(same);
      __syncwarp();
    }
  }
}

ATB_DEVICE void add8(float (&acc)[8], const uint4& u) {
  const uint32_t x[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 v = unpack_bf16x2(x[e]);
    acc[2 * e] += v.x;
    acc[2 * e + 1] += v.y;
  }
}

// sums the gradients of tokens order[b], order[b + step], ... below e for columns c + {0, 256} + [0, 8) of `dy`
template <int U>
ATB_DEVICE void sum_tokens(float (&acc)[2][8], const __nv_bfloat16* dy, const int* order, int b, int e, int step, int H, int c,
                           const bool (&live)[2]) {
  for (int m = b; m < e; m += U * step) {
    uint4 x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = m + u * step < e ? order[m + u * step] : -1;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        x[u][h] = t >= 0 && live[h] ? *reinterpret_cast<const uint4*>(dy + (long long)t * H + c + 256 * h) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) add8(acc[h], x[u][h]);
  }
}

template <typename TO>
ATB_DEVICE void put8(TO* out, const float (&acc)[8], bool accumulate) {
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = acc[e];
  if constexpr (sizeof(TO) == 2) {
    if (accumulate) add8(v, *reinterpret_cast<const uint4*>(out));
    *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                                pack_bf16x2(v[6], v[7]));
  } else {
    float4* o = reinterpret_cast<float4*>(out);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 f = make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
      if (accumulate) {
        const float4 p = o[h];
        f = make_float4(f.x + p.x, f.y + p.y, f.z + p.z, f.w + p.w);
      }
      o[h] = f;
    }
  }
}

template <typename TO>
__global__ void __launch_bounds__(256)
embed_rows_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ start, const int* __restrict__ order,
                  TO* __restrict__ out, int V, int H, int accumulate) {
  __shared__ int s[ROWS + 1];
  __shared__ float part[8][COLS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row0 = blockIdx.x * ROWS, c = blockIdx.y * COLS + lane * 8;
  const bool live[2] = {c < H, c + 256 < H};
  if (threadIdx.x <= ROWS) s[threadIdx.x] = start[min(row0 + (int)threadIdx.x, V)];
  __syncthreads();
  for (int j = warp; j < ROWS; j += 8) {
    const int b = s[j], e = s[j + 1], row = row0 + j;
    if (row >= V || e - b > MANY || (accumulate && e == b)) continue;
    float acc[2][8] = {};
    if (e - b == 1) sum_tokens<1>(acc, dy, order, b, e, 1, H, c, live);
    else sum_tokens<4>(acc, dy, order, b, e, 1, H, c, live);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (live[h]) put8(out + (long long)row * H + c + 256 * h, acc[h], accumulate != 0);
  }
  for (int j = 0; j < ROWS; ++j) {
    const int b = s[j], e = s[j + 1];
    if (e - b <= MANY) continue;
    float acc[2][8] = {};
    sum_tokens<8>(acc, dy, order, b + warp, e, 8, H, c, live);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 8; ++i) part[warp][256 * h + lane * 8 + i] = acc[h][i];
    __syncthreads();
    if (warp < 2 && live[warp]) {
      float v[8] = {};
      for (int w = 0; w < 8; ++w)
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += part[w][256 * warp + lane * 8 + i];
      put8(out + (long long)(row0 + j) * H + c + 256 * warp, v, accumulate != 0);
    }
    __syncthreads();
  }
}

}  // namespace

// dy: bf16 [T, H]; ids: int64 [T], ids outside [0, V) are left out; out: [V, H] (H a multiple of 8, rows of 16-byte pieces),
// fp32 if out_fp32, else bf16; accumulate = 0 writes every row. scratch: int32 [V + 1 + T].
extern "C" int atb_embedding_bwd(const void* dy, const long long* ids, void* out, int* scratch, int T, int V, int H, int out_fp32,
                                 int accumulate, void* stream) {
  if (T < 0 || V <= 0 || H <= 0 || H % 8 != 0) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int range = V > 148 * MAX_RANGE ? MAX_RANGE : (V + 147) / 148;      // a CTA per SM up to 150 thousand rows
  const int smem = SORT_WARPS * range * (int)sizeof(int);
  if (smem > 40 * 1024 && cudaFuncSetAttribute(embed_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               SORT_WARPS * MAX_RANGE * (int)sizeof(int)) != cudaSuccess)
    return -4;
  int *start = scratch, *order = scratch + V + 1;
  embed_sort_kernel<<<(V + range - 1) / range, SORT_WARPS * 32, smem, st>>>(ids, start, order, T, V, range);
  const dim3 grid((V + ROWS - 1) / ROWS, (H + COLS - 1) / COLS);
  if (out_fp32)
    embed_rows_kernel<float><<<grid, 256, 0, st>>>(reinterpret_cast<const __nv_bfloat16*>(dy), start, order,
                                                   reinterpret_cast<float*>(out), V, H, accumulate);
  else
    embed_rows_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(reinterpret_cast<const __nv_bfloat16*>(dy), start, order,
                                                           reinterpret_cast<__nv_bfloat16*>(out), V, H, accumulate);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
