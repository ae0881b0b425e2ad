// Gradient of an embedding table: row v (+)= the sum of the gradients of the tokens whose id is v, in fp32, rounded once. A row
// of up to MANY tokens is summed in their order, a longer one as eight interleaved sums, from PART tokens on eight per PART
// tokens, which are then added in a fixed order. Two kernels, no atomics on values and no order that depends on timing:
//   embed_sort    a stable counting sort of the ids. A CTA owns a range of rows and reads all ids twice: the first time it counts
//                 its own per row and warp and the ids below its range (which is where its part of the result begins), the
//                 second time it writes the tokens. The ids are small (64 KB for 8192) and come out of L2; in exchange no CTA
//                 waits for another.
//   embed_rows    a warp per row and 512 columns; a row with many tokens by the eight warps of its block, a long one by several
//                 blocks. With one block for every row and 32 rows a block, 65536 tokens took, nine in ten of them on one row
//                 (padding; 32000 x 2048), 2670 us, now 163; on a table of 256 x 1024 482, now 67; spread over 32000 x
//                 2048 155, now 152.
// Bound by memory: the gradients of the tokens are read once, the rows that have any are read and written. The library wrote a
// gradient of the whole table (zeros, then rows) that was then added to the gradient buffer, three more passes over the
// table, after a sort in several launches. 4096 tokens on 32000 rows of 2048, random ids, cold: 357 us in 30 launches, now 48.
#include "common.cuh"
#include <type_traits>

namespace {
using namespace atb;

constexpr int SORT_WARPS = 16, BATCH = 8;
constexpr int MAX_RANGE = 1024;          // rows of a CTA: 16 warps x 1024 counters are 64 KB of shared memory
constexpr int COLS = 512;                // columns of a block; its rows are 32, 8 or 2
constexpr int FEW_BLOCKS = 2 * 148;      // blocks that there should be (4096 tokens on 1000 x 256: 32 rows a block 34 us, 2 17)
// Tokens above which the whole block sums a row: 16 to 128 are all even, 256 takes half as long again on 256 x 1024 with 65536 tokens.
constexpr int MANY = 64;
constexpr int PART = 512;                // tokens above which several blocks sum a row, as many of them each

__global__ void __launch_bounds__(SORT_WARPS * 32)
embed_sort_kernel(const long long* __restrict__ ids, int* __restrict__ start, int* __restrict__ order, int* __restrict__ done,
                  int n_done, int T, int V, int range) {
  extern __shared__ int cnt[];           // [SORT_WARPS][range]
  __shared__ int scan[SORT_WARPS], base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long lo = (long long)blockIdx.x * range;
  const int rows = (int)min((long long)range, V - lo);
  for (int i = threadIdx.x; i < SORT_WARPS * range; i += SORT_WARPS * 32) cnt[i] = 0;
  if (threadIdx.x == 0) base = 0;
  for (int i = blockIdx.x * SORT_WARPS * 32 + threadIdx.x; i < n_done; i += gridDim.x * SORT_WARPS * 32) done[i] = 0;
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

// The sums of the eight warps of a block, in their order, of 512 columns: put(which 256 of them, eight sums of a lane).
template <class F>
ATB_DEVICE void sum_warps(float (&part)[8][COLS], const float (&acc)[2][8], int warp, int lane, F put) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 8; ++i) part[warp][256 * h + lane * 8 + i] = acc[h][i];
  __syncthreads();
  if (warp < 2) {
    float v[8] = {};
    for (int w = 0; w < 8; ++w)
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += part[w][256 * warp + lane * 8 + i];
    put(warp, v);
  }
  __syncthreads();
}

// The pieces that parts [PART * at, PART * (at + 1)) of `order` hold of rows with more than PART tokens: at most two, the end (or
// all) of one row and the beginning of another. f(which, row, its first token, the one behind its last).
template <class F>
ATB_DEVICE void long_rows(const long long* ids, const int* start, const int* order, int V, int at, F f) {
  const int lo = max(at * PART, start[0]), hi = min((at + 1) * PART, start[V]);
  if (lo >= hi) return;
  const int r0 = (int)ids[order[lo]], r1 = (int)ids[order[hi - 1]];
  if (start[r0 + 1] - start[r0] > PART) f(0, r0, start[r0], start[r0 + 1]);
  if (r1 != r0 && start[r1 + 1] - start[r1] > PART) f(1, r1, start[r1], start[r1 + 1]);
}

// The first `parts` blocks sum PART tokens each of the long rows into sums[2 * part + which][H]; the one that finishes a row's last
// part (done: how many have been, counted where the row begins) adds them up, always in the same order. The other blocks
// take ROWS rows each.
template <typename TO, int ROWS>
__global__ void __launch_bounds__(256)
embed_rows_kernel(const __nv_bfloat16* __restrict__ dy, const long long* __restrict__ ids, const int* __restrict__ start,
                  const int* __restrict__ order, TO* __restrict__ out, float* sums, int* done, int V, int H, int accumulate,
                  int parts) {
  __shared__ int s[ROWS + 1], last;
  __shared__ float part[8][COLS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.y * COLS + lane * 8;
  const bool live[2] = {c < H, c + 256 < H};
  const int at = blockIdx.x;
  if (at < parts) {
    long_rows(ids, start, order, V, at, [&](int which, int row, int b, int e) {
      float acc[2][8] = {};
      sum_tokens<8>(acc, dy, order, max(b, at * PART) + warp, min(e, (at + 1) * PART), 8, H, c, live);
      sum_warps(part, acc, warp, lane, [&](int h, const float (&v)[8]) {
        if (c + 256 * h < H) put8(sums + (2ll * at + which) * H + c + 256 * h, v, false);
        __threadfence();
      });
      const int first = b / PART, end = (e - 1) / PART + 1, place = b > max(first * PART, start[0]) ? 1 : 0;
      if (threadIdx.x == 0) {
        last = atomicAdd(&done[(2 * first + place) * gridDim.y + blockIdx.y], 1) == end - first - 1;
        __threadfence();
      }
      __syncthreads();
      if (!last) return;
      float all[2][8] = {};
      for (int p = first + warp; p < end; p += 8) {
        const float* x = sums + (2ll * p + (p == first ? place : 0)) * H + c;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (live[h]) {
            const float4 u = __ldcg(reinterpret_cast<const float4*>(x + 256 * h));
            const float4 w = __ldcg(reinterpret_cast<const float4*>(x + 256 * h + 4));
            const float y[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) all[h][i] += y[i];
          }
      }
      sum_warps(part, all, warp, lane, [&](int h, const float (&v)[8]) {
        if (c + 256 * h < H) put8(out + (long long)row * H + c + 256 * h, v, accumulate != 0);
      });
    });
    return;
  }
  const int row0 = (at - parts) * ROWS;
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
    if (e - b <= MANY || e - b > PART) continue;
    float acc[2][8] = {};
    sum_tokens<8>(acc, dy, order, b + warp, e, 8, H, c, live);
    sum_warps(part, acc, warp, lane, [&](int h, const float (&v)[8]) {
      if (c + 256 * h < H) put8(out + (long long)(row0 + j) * H + c + 256 * h, v, accumulate != 0);
    });
  }
}

template <typename TO>
void launch_rows(const void* dy, const long long* ids, const int* start, const int* order, void* out, float* sums, int* done,
                 int parts, int V, int H, int accumulate, cudaStream_t st) {
  const int cols = (H + COLS - 1) / COLS;
  auto rows = [&](auto n) {
    constexpr int ROWS = decltype(n)::value;
    embed_rows_kernel<TO, ROWS><<<dim3(parts + (V + ROWS - 1) / ROWS, cols), 256, 0, st>>>(
        reinterpret_cast<const __nv_bfloat16*>(dy), ids, start, order, reinterpret_cast<TO*>(out), sums, done, V, H, accumulate, parts);
  };
  const long long pieces = (long long)V * cols;
  if (pieces >= 32 * FEW_BLOCKS) rows(std::integral_constant<int, 32>{});
  else if (pieces >= 8 * FEW_BLOCKS) rows(std::integral_constant<int, 8>{});
  else rows(std::integral_constant<int, 2>{});
}

}  // namespace

// Words of the scratch, 16-byte aligned: int32 [V + 1 + T], with more than 512 tokens also counters and, from the next multiple
// of 16 bytes on, fp32 sums of the parts of long rows.
extern "C" long long atb_embedding_bwd_scratch(int T, int V, int H) {
  const long long parts = T > PART ? (T + PART - 1) / PART : 0, words = (long long)V + 1 + T + 2 * parts * ((H + COLS - 1) / COLS);
  return parts > 0 ? ((words + 3) & ~3ll) + 2 * parts * H : words;
}

// dy: bf16 [T, H]; ids: int64 [T], ids outside [0, V) are left out; out: [V, H] (H a multiple of 8, rows of 16-byte pieces),
// fp32 if out_fp32, else bf16; accumulate = 0 writes every row. scratch: as many int32 words as atb_embedding_bwd_scratch says.
extern "C" int atb_embedding_bwd(const void* dy, const long long* ids, void* out, int* scratch, int T, int V, int H, int out_fp32,
                                 int accumulate, void* stream) {
  if (T < 0 || V <= 0 || H <= 0 || H % 8 != 0) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int range = V > 148 * MAX_RANGE ? MAX_RANGE : (V + 147) / 148;      // a CTA per SM up to 150 thousand rows
  const int smem = SORT_WARPS * range * (int)sizeof(int);
  if (smem > 40 * 1024 && cudaFuncSetAttribute(embed_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               SORT_WARPS * MAX_RANGE * (int)sizeof(int)) != cudaSuccess)
    return -4;
  const int parts = T > PART ? (T + PART - 1) / PART : 0, n_done = 2 * parts * ((H + COLS - 1) / COLS);
  int *start = scratch, *order = scratch + V + 1, *done = order + T;
  float* sums = reinterpret_cast<float*>(scratch + (((long long)V + 1 + T + n_done + 3) & ~3ll));
  embed_sort_kernel<<<(V + range - 1) / range, SORT_WARPS * 32, smem, st>>>(ids, start, order, done, n_done, T, V, range);
  if (out_fp32) launch_rows<float>(dy, ids, start, order, out, sums, done, parts, V, H, accumulate, st);
  else launch_rows<__nv_bfloat16>(dy, ids, start, order, out, sums, done, parts, V, H, accumulate, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
