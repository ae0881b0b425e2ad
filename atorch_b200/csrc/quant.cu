// Group-wise integer quantisation kernels for sm_100a (memory-bound, 16-byte accesses):
//   quantize / dequantize       int8 or packed int4, symmetric (scale) or asymmetric (scale, offset),
//                               one set of parameters per group of `group_size` consecutive elements
//   swizzle_quantize            quantise and emit groups in (pipeline, device, node)-major order so that
//                               a two-hop (intra-node, inter-node) all-to-all sends contiguous blocks
//   dequant_reduce              dequantise the chunks received from N peers, sum, requantise
//   optimizer-state packing     absmax-linear 8/16-bit and nonlinear (lookup-table) 4/8-bit codes with
//                               optional stochastic rounding (Philox counter per element)
// Conventions: symmetric  q = rint(x / s), s = absmax / qmax;  asymmetric q = rint((x - lo) / s) - 2^(b-1),
// s = (hi - lo) / (2^b - 1). 4-bit values are packed low nibble first.
// Counterparts in the reference: atorch/ops/csrc/quantization/{quantize,dequantize,swizzled_quantize,
// quant_reduce}.cu and atorch/ops/csrc/quantization_optimizer/quantization_optimizer.cu.
#include "common.cuh"
#include <type_traits>

namespace {
using namespace atb;

template <typename T>
ATB_DEVICE float ldf(const T* p, long long i) { return to_f32<T>(p[i]); }

// one CTA (256 threads) per group
template <typename T>
__global__ void __launch_bounds__(256) quantize_kernel(const T* __restrict__ x, int8_t* __restrict__ q,
                                                       float* __restrict__ params, int group_size, int bits,
                                                       int asym, const int* __restrict__ group_map, int out_groups) {
  __shared__ float red[33];
  const int g = blockIdx.x;
  const T* xg = x + (long long)g * group_size;
  float lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < group_size; i += 256) {
    const float v = ldf(xg, i);
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  hi = block_max(hi, red);
  lo = -block_max(-lo, red);
  const int qmax = (1 << (bits - 1)) - 1, half = 1 << (bits - 1);
  float s, off;
  if (asym) {
    s = (hi - lo) / (float)((1 << bits) - 1);
    off = lo;
  } else {
    s = fmaxf(fabsf(hi), fabsf(lo)) / (float)qmax;
    off = 0.f;
  }
  if (s == 0.f) s = 1.f;
  const float inv = 1.f / s;
  const int og = group_map ? group_map[g] : g;   // destination group (swizzled layouts)
  if (threadIdx.x == 0) {
    params[(long long)og * (asym ? 2 : 1)] = s;
    if (asym) params[(long long)og * 2 + 1] = off;
  }
  if (bits == 8) {
    int8_t* qg = q + (long long)og * group_size;
    for (int i = threadIdx.x; i < group_size; i += 256) {
      float r = rintf((ldf(xg, i) - off) * inv) - (asym ? half : 0);
      qg[i] = (int8_t)fminf(fmaxf(r, -half), qmax);
    }
  } else {
    int8_t* qg = q + (long long)og * (group_size / 2);
    for (int i = threadIdx.x; i < group_size / 2; i += 256) {
      float a = rintf((ldf(xg, 2 * i) - off) * inv) - (asym ? half : 0);
      float b = rintf((ldf(xg, 2 * i + 1) - off) * inv) - (asym ? half : 0);
      const int ia = (int)fminf(fmaxf(a, -half), qmax) & 0xF, ib = (int)fminf(fmaxf(b, -half), qmax) & 0xF;
      qg[i] = (int8_t)(ia | (ib << 4));
    }
  }
}

// The same quantisation with every group held in registers: one read of x. LANES lanes of a warp, or a block of WARPS warps
// (LANES = 32), own a group of at most WARPS * LANES * V pieces of 8 elements; the i-th of them takes pieces i,
// i + LANES * WARPS, ...
// Bound by memory: 16-byte loads, all V pieces of a thread in flight, 8- or 4-byte stores, and few enough instructions, which
// bounded it before: extrema of 16-bit values two at a time, and codes by adding 1.5 * 2^23, whose low bits then are the
// rounded integer, packed by byte permutes; rintf and the conversion to int each take a slot of the slow unit (16 a clock).
// 67 M bf16 values in groups of 2048 to int8 (201 MB, cold): 47.1 us with those, 36.9 now (5.5 TB/s); fp32 57.4 either way.
// The kernel above reads x twice, 2 bytes a thread: 87.5 us.
template <typename T>
struct Piece8 {
  uint4 r[sizeof(T) / 2];
  ATB_DEVICE void load(const T* p) {
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 2); ++i) r[i] = reinterpret_cast<const uint4*>(p)[i];
  }
  ATB_DEVICE float at(int i) const { return to_f32<T>(reinterpret_cast<const T*>(r)[i]); }
};

// Running extrema of pieces; NaN is passed over. abs_only: hi is that of the magnitudes, lo is not kept.
template <typename T>
struct Extrema {
  float hi = -INFINITY, lo = INFINITY;
  ATB_DEVICE void add(const Piece8<T>& v, bool abs_only) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      hi = fmaxf(hi, abs_only ? fabsf(v.at(j)) : v.at(j));
      if (!abs_only) lo = fminf(lo, v.at(j));
    }
  }
  ATB_DEVICE void done(float& h, float& l) const { h = hi; l = lo; }
};
template <typename T2>
struct Extrema16 {
  T2 hi, lo;
  template <typename P>
  ATB_DEVICE void add(const P& v, bool abs_only) {
    const T2* x = reinterpret_cast<const T2*>(v.r);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      hi = __hmax2(hi, abs_only ? __habs2(x[j]) : x[j]);
      if (!abs_only) lo = __hmin2(lo, x[j]);
    }
  }
};
template <>
struct Extrema<__nv_bfloat16> : Extrema16<__nv_bfloat162> {
  ATB_DEVICE Extrema() { hi = __float2bfloat162_rn(-INFINITY); lo = __float2bfloat162_rn(INFINITY); }
  ATB_DEVICE void done(float& h, float& l) const {
    h = fmaxf(__low2float(hi), __high2float(hi));
    l = fminf(__low2float(lo), __high2float(lo));
  }
};
template <>
struct Extrema<__half> : Extrema16<__half2> {
  ATB_DEVICE Extrema() { hi = __float2half2_rn(-INFINITY); lo = __float2half2_rn(INFINITY); }
  ATB_DEVICE void done(float& h, float& l) const {
    h = fmaxf(__low2float(hi), __high2float(hi));
    l = fminf(__low2float(lo), __high2float(lo));
  }
};

// Low bytes of four words in one.
ATB_DEVICE uint32_t low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
// Low nibbles of the bytes of x as 16 bits.
ATB_DEVICE uint32_t nibbles(uint32_t x) {
  x &= 0x0F0F0F0Fu;
  x = (x | (x >> 4)) & 0x00FF00FFu;
  return (x | (x >> 8)) & 0xFFFFu;
}

template <typename T, int WARPS, int LANES, int V>
__global__ void __launch_bounds__(128) quantize_regs_kernel(const T* __restrict__ x, int8_t* __restrict__ q,
                                                            float* __restrict__ params, int groups, int group_size,
                                                            int bits, int asym, const int* __restrict__ group_map) {
  __shared__ float red[2][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int PER_WARP = 32 / LANES, TEAM = LANES * WARPS;      // groups of a warp; threads of a group
  int g = WARPS == 1 ? (blockIdx.x * 4 + warp) * PER_WARP + lane / LANES : blockIdx.x;
  if (WARPS == 1 && g - lane / LANES >= groups) return;      // whole warps leave, nothing below syncs the block
  const bool mine = WARPS > 1 || g < groups;                 // the last warp may have lanes without a group
  if (!mine) g = groups - 1;
  const int t = WARPS == 1 ? lane % LANES : threadIdx.x;
  const int n = group_size / 8;
  const T* xg = x + (long long)g * group_size;
  Piece8<T> v[V];
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (t + i * TEAM < n) v[i].load(xg + (t + i * TEAM) * 8);
  Extrema<T> ext;
#pragma unroll
  for (int i = 0; i < V; ++i)
    if (t + i * TEAM < n) ext.add(v[i], !asym);
  float lo, hi;
  ext.done(hi, lo);
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) {
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
  }
  if (WARPS > 1) {
    if (lane == 0) { red[0][warp] = hi; red[1][warp] = lo; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WARPS; ++i) { hi = fmaxf(hi, red[0][i]); lo = fminf(lo, red[1][i]); }
  }
  const int qmax = (1 << (bits - 1)) - 1, half = 1 << (bits - 1);
  float s = asym ? (hi - lo) / (float)((1 << bits) - 1) : fabsf(hi) / (float)qmax;
  const float off = asym ? lo : 0.f;
  if (s == 0.f) s = 1.f;
  const float inv = 1.f / s;
  const int og = group_map ? group_map[g] : g;
  if (t == 0 && mine) {
    params[(long long)og * (asym ? 2 : 1)] = s;
    if (asym) params[(long long)og * 2 + 1] = off;
  }
  // rint(clamp(x)) is clamp(rint(x)) for whole bounds; asymmetric codes are rounded before the offset of half the range, which
  // turns over their highest bit. NaN takes the lowest code, as fmaxf has it.
  const float low = asym ? 0.f : -(float)half, high = asym ? (float)(2 * half - 1) : (float)qmax;
  const uint32_t turn = !asym ? 0u : bits == 8 ? 0x80808080u : 0x08080808u;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int k = t + i * TEAM;
    if (k >= n || !mine) continue;
    uint32_t c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // off is 0 for symmetric codes; two roundings, product and sum, are wanted
      const float x = __fmul_rn(asym ? v[i].at(j) - off : v[i].at(j), inv);
      c[j] = __float_as_uint(__fadd_rn(fminf(fmaxf(x, low), high), 12582912.f));
    }
    const uint32_t w0 = low_bytes(c[0], c[1], c[2], c[3]) ^ turn, w1 = low_bytes(c[4], c[5], c[6], c[7]) ^ turn;
    if (bits == 8)
      *reinterpret_cast<uint2*>(q + (long long)og * group_size + (long long)k * 8) = make_uint2(w0, w1);
    else
      *reinterpret_cast<uint32_t*>(q + (long long)og * (group_size / 2) + (long long)k * 4) = nibbles(w0) | (nibbles(w1) << 16);
  }
}

// Four pieces a lane as far as the group has them, and as many lanes as it takes: 8 up to 256 elements, 16 up to 512, a warp up
// to 2048 (8 pieces a lane: 32 registers of 16-bit, 64 of 32-bit values), a block of 4 warps up to 8192. With a whole warp
// for every group 67 M bf16 values in groups of 128 (512) took 121 (46) us, now
// 45 (38); fp32 in groups of 128 119 -> 57. Longer groups, groups that are no
// multiple of 8 and unaligned inputs take quantize_kernel.
template <typename T>
bool quantize_regs(const T* x, int8_t* q, float* params, int groups, int group_size, int bits, int asym,
                   const int* group_map, cudaStream_t st) {
  if (group_size % 8 || group_size > 8192 || (reinterpret_cast<uintptr_t>(x) & 15) ||
      (reinterpret_cast<uintptr_t>(q) & 7))
    return false;
#define ATB_QUANT(W_, L_, V_)                                                                                           \
  quantize_regs_kernel<T, W_, L_, V_><<<(W_) == 1 ? (groups + 4 * (32 / (L_)) - 1) / (4 * (32 / (L_))) : groups, 128, 0, st>>>( \
      x, q, params, groups, group_size, bits, asym, group_map)
  if (group_size <= 64) ATB_QUANT(1, 8, 1);
  else if (group_size <= 128) ATB_QUANT(1, 8, 2);
  else if (group_size <= 256) ATB_QUANT(1, 8, 4);
  else if (group_size <= 512) ATB_QUANT(1, 16, 4);
  else if (group_size <= 1024) ATB_QUANT(1, 32, 4);
  else if (group_size <= 2048) ATB_QUANT(1, 32, 8);
  else if (group_size <= 4096) ATB_QUANT(4, 32, 4);
  else ATB_QUANT(4, 32, 8);
#undef ATB_QUANT
  return true;
}

ATB_DEVICE float deq(int v, float s, float off, int asym, int half) { return asym ? (v + half) * s + off : v * s; }
ATB_DEVICE int sext4(int v) { return (v & 8) ? v - 16 : v; }

template <typename T>
__global__ void dequantize_kernel(const int8_t* __restrict__ q, const float* __restrict__ params, T* __restrict__ out,
                                  long long total, int group_size, int bits, int asym) {
  const int half = 1 << (bits - 1);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long g = i / group_size;
    const float s = params[g * (asym ? 2 : 1)], off = asym ? params[g * 2 + 1] : 0.f;
    int v;
    if (bits == 8) v = q[i];
    else {
      const int byte = q[i >> 1];
      v = sext4((i & 1) ? (byte >> 4) & 0xF : byte & 0xF);
    }
    out[i] = from_f32<T>(deq(v, s, off, asym, half));
  }
}

// The same for groups of a multiple of 8 elements: a thread turns pieces of 8 codes into 16-byte stores, four pieces in
// flight, one division by the group length per piece in place of one (64-bit) per element. Bound by memory: 67 M int8
// codes to bf16 146.5 -> 29.4 us (201 MB, part of the codes still in L2).
template <typename T>
__global__ void __launch_bounds__(256) dequantize8_kernel(const int8_t* __restrict__ q, const float* __restrict__ params,
                                                          T* __restrict__ out, unsigned pieces, unsigned per_group,
                                                          int bits, int asym) {
  constexpr int U = 4;
  const int half = 1 << (bits - 1);
  const unsigned first = blockIdx.x * (256u * U) + threadIdx.x;
  uint2 c[U];
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const unsigned k = first + i * 256u;
    if (k >= pieces) break;
    if (bits == 8) c[i] = reinterpret_cast<const uint2*>(q)[k];
    else c[i].x = reinterpret_cast<const uint32_t*>(q)[k];
  }
#pragma unroll
  for (int i = 0; i < U; ++i) {
    const unsigned k = first + i * 256u;
    if (k >= pieces) break;
    const unsigned g = k / per_group;
    const float s = params[(size_t)g * (asym ? 2 : 1)], off = asym ? params[(size_t)g * 2 + 1] : 0.f;
    Piece8<T> o;
    T* ov = reinterpret_cast<T*>(o.r);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int v;
      if (bits == 8) v = (int)(int8_t)((j < 4 ? c[i].x : c[i].y) >> (8 * (j & 3)));
      else v = sext4((c[i].x >> (4 * j)) & 0xF);
      ov[j] = from_f32<T>(deq(v, s, off, asym, half));
    }
#pragma unroll
    for (int j = 0; j < (int)(sizeof(T) / 2); ++j)
      reinterpret_cast<uint4*>(out + (size_t)k * 8)[j] = o.r[j];
  }
}

template <typename T>
bool dequantize8(const int8_t* q, const float* params, T* out, long long total, int group_size, int bits, int asym,
                 cudaStream_t st) {
  if (group_size % 8 || total % 8 || total / 8 > 0x7fffffffLL || (reinterpret_cast<uintptr_t>(out) & 15) ||
      (reinterpret_cast<uintptr_t>(q) & 7))
    return false;
  const unsigned pieces = (unsigned)(total / 8);
  dequantize8_kernel<T><<<(pieces + 1023) / 1024, 256, 0, st>>>(q, params, out, pieces, (unsigned)group_size / 8, bits,
                                                                asym);
  return true;
}

// out group g = requantised sum over `n_in` tensors' group g (all tensors share the group layout);
// input tensor t is at q_in + t * in_stride_bytes, params_in + t * groups * P.
__global__ void __launch_bounds__(256)
dequant_reduce_kernel(const int8_t* __restrict__ q_in, const float* __restrict__ p_in, int8_t* __restrict__ q_out,
                      float* __restrict__ p_out, int n_in, long long in_stride_bytes, int groups, int group_size,
                      int bits, int asym) {
  extern __shared__ float vals[];
  __shared__ float red[33];
  const int g = blockIdx.x, P = asym ? 2 : 1, half = 1 << (bits - 1), qmax = half - 1;
  float lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < group_size; i += 256) {
    float acc = 0.f;
    for (int t = 0; t < n_in; ++t) {
      const int8_t* qt = q_in + t * in_stride_bytes;
      const float s = p_in[((long long)t * groups + g) * P], off = asym ? p_in[((long long)t * groups + g) * P + 1] : 0.f;
      int v;
      if (bits == 8) v = qt[(long long)g * group_size + i];
      else {
        const int byte = qt[((long long)g * group_size + i) >> 1];
        v = sext4((i & 1) ? (byte >> 4) & 0xF : byte & 0xF);
      }
      acc += deq(v, s, off, asym, half);
    }
    vals[i] = acc;
    lo = fminf(lo, acc);
    hi = fmaxf(hi, acc);
  }
  hi = block_max(hi, red);
  lo = -block_max(-lo, red);
  float s = asym ? (hi - lo) / (float)((1 << bits) - 1) : fmaxf(fabsf(hi), fabsf(lo)) / (float)qmax;
  const float off = asym ? lo : 0.f;
  if (s == 0.f) s = 1.f;
  if (threadIdx.x == 0) {
    p_out[(long long)g * P] = s;
    if (asym) p_out[(long long)g * P + 1] = off;
  }
  __syncthreads();
  const float inv = 1.f / s;
  if (bits == 8) {
    for (int i = threadIdx.x; i < group_size; i += 256)
      q_out[(long long)g * group_size + i] =
          (int8_t)fminf(fmaxf(rintf((vals[i] - off) * inv) - (asym ? half : 0), -half), qmax);
  } else {
    for (int i = threadIdx.x; i < group_size / 2; i += 256) {
      const int a = (int)fminf(fmaxf(rintf((vals[2 * i] - off) * inv) - (asym ? half : 0), -half), qmax) & 0xF;
      const int b = (int)fminf(fmaxf(rintf((vals[2 * i + 1] - off) * inv) - (asym ? half : 0), -half), qmax) & 0xF;
      q_out[(long long)g * (group_size / 2) + i] = (int8_t)(a | (b << 4));
    }
  }
}

// ---- optimizer-state codes ---------------------------------------------------------------
ATB_DEVICE uint32_t philox_hash(uint64_t seed, uint64_t idx) {   // counter-based, reproducible per element
  uint64_t z = seed + idx * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (uint32_t)((z ^ (z >> 31)) >> 32);
}

// absmax-linear: code = rint(x / absmax(group) * qmax) stored as int8 / int16; absmax per group
template <typename CODE>
__global__ void __launch_bounds__(256) pack_linear_kernel(const float* __restrict__ x, CODE* __restrict__ code,
                                                          float* __restrict__ absmax, long long n, int group_size,
                                                          int qmax) {
  __shared__ float red[33];
  const long long g0 = (long long)blockIdx.x * group_size;
  float am = 0.f;
  for (int i = threadIdx.x; i < group_size && g0 + i < n; i += 256) am = fmaxf(am, fabsf(x[g0 + i]));
  am = block_max(am, red);
  if (threadIdx.x == 0) absmax[blockIdx.x] = am;
  const float inv = am > 0.f ? (float)qmax / am : 0.f;
  for (int i = threadIdx.x; i < group_size && g0 + i < n; i += 256) code[g0 + i] = (CODE)rintf(x[g0 + i] * inv);
}
template <typename CODE>
__global__ void unpack_linear_kernel(const CODE* __restrict__ code, const float* __restrict__ absmax,
                                     float* __restrict__ out, long long n, int group_size, int qmax) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = (float)code[i] * absmax[i / group_size] / (float)qmax;
}

// nonlinear: x / absmax(group) in [-1, 1] is mapped to the nearest entry of a sorted table `qmap`
// (2^bits entries); with stochastic rounding the two neighbours are chosen with probability
// proportional to proximity. 4-bit codes are packed two per byte.
__global__ void __launch_bounds__(256)
pack_nonlinear_kernel(const float* __restrict__ x, uint8_t* __restrict__ code, float* __restrict__ absmax,
                      const float* __restrict__ qmap, long long n, int group_size, int bits, int stochastic,
                      unsigned long long seed) {
  __shared__ float red[33];
  __shared__ float smap[256];
  const int nq = 1 << bits;
  for (int i = threadIdx.x; i < nq; i += 256) smap[i] = qmap[i];
  const long long g0 = (long long)blockIdx.x * group_size;
  float am = 0.f;
  for (int i = threadIdx.x; i < group_size && g0 + i < n; i += 256) am = fmaxf(am, fabsf(x[g0 + i]));
  am = block_max(am, red);
  if (threadIdx.x == 0) absmax[blockIdx.x] = am;
  const float inv = am > 0.f ? 1.f / am : 0.f;
  auto encode = [&](long long idx) -> int {
    if (idx >= n) return 0;
    const float v = x[idx] * inv;
    int lo = 0, hi = nq - 1;           // binary search: largest entry <= v
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (smap[mid] <= v) lo = mid; else hi = mid - 1;
    }
    if (lo == nq - 1) return lo;
    const float a = smap[lo], b = smap[lo + 1];
    if (stochastic) {
      const float u = (philox_hash(seed, (uint64_t)idx) >> 8) * (1.f / 16777216.f);
      return (v - a) > u * (b - a) ? lo + 1 : lo;
    }
    return (v - a) > (b - v) ? lo + 1 : lo;
  };
  if (bits == 8) {
    for (int i = threadIdx.x; i < group_size && g0 + i < n; i += 256) code[g0 + i] = (uint8_t)encode(g0 + i);
  } else {
    for (int i = threadIdx.x; i < group_size / 2 && g0 + 2 * i < n; i += 256)
      code[(g0 >> 1) + i] = (uint8_t)(encode(g0 + 2 * i) | (encode(g0 + 2 * i + 1) << 4));
  }
}
__global__ void unpack_nonlinear_kernel(const uint8_t* __restrict__ code, const float* __restrict__ absmax,
                                        const float* __restrict__ qmap, float* __restrict__ out, long long n,
                                        int group_size, int bits) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int c;
    if (bits == 8) c = code[i];
    else c = (i & 1) ? code[i >> 1] >> 4 : code[i >> 1] & 0xF;
    out[i] = qmap[c] * absmax[i / group_size];
  }
}

inline int cap_grid(long long work, int threads) {
  long long g = (work + threads - 1) / threads;
  const long long cap = 148LL * 16;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}
}  // namespace

// dtype: 0 bf16, 1 fp16, 2 fp32. `group_map` (optional int32[groups]) redirects group g to output slot group_map[g].
extern "C" int atb_quantize(const void* x, void* q, float* params, int groups, int group_size, int bits, int asym,
                            const int* group_map, int dtype, void* stream) {
  if (groups <= 0) return 0;
  if ((bits != 4 && bits != 8) || (bits == 4 && (group_size & 1))) return -1;
  auto run = [&](auto* xt) {
    using T = std::remove_cv_t<std::remove_pointer_t<decltype(xt)>>;
    cudaStream_t st = (cudaStream_t)stream;
    if (!quantize_regs<T>(xt, (int8_t*)q, params, groups, group_size, bits, asym, group_map, st))
      quantize_kernel<T><<<groups, 256, 0, st>>>(xt, (int8_t*)q, params, group_size, bits, asym, group_map, groups);
  };
  if (dtype == 0) run((const __nv_bfloat16*)x);
  else if (dtype == 1) run((const __half*)x);
  else run((const float*)x);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_dequantize(const void* q, const float* params, void* out, long long total, int group_size, int bits,
                              int asym, int dtype, void* stream) {
  if (total <= 0) return 0;
  auto run = [&](auto* o) {
    using T = std::remove_pointer_t<decltype(o)>;
    cudaStream_t st = (cudaStream_t)stream;
    if (!dequantize8<T>((const int8_t*)q, params, o, total, group_size, bits, asym, st))
      dequantize_kernel<T><<<cap_grid(total, 256), 256, 0, st>>>((const int8_t*)q, params, o, total, group_size, bits,
                                                                 asym);
  };
  if (dtype == 0) run((__nv_bfloat16*)out);
  else if (dtype == 1) run((__half*)out);
  else run((float*)out);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_dequant_reduce(const void* q_in, const float* p_in, void* q_out, float* p_out, int n_in,
                                  long long in_stride_bytes, int groups, int group_size, int bits, int asym,
                                  void* stream) {
  if (groups <= 0) return 0;
  if (group_size * 4 > 160 * 1024) return -1;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(dequant_reduce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    attr = true;
  }
  dequant_reduce_kernel<<<groups, 256, group_size * 4, (cudaStream_t)stream>>>(
      (const int8_t*)q_in, p_in, (int8_t*)q_out, p_out, n_in, in_stride_bytes, groups, group_size, bits, asym);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_pack_linear(const float* x, void* code, float* absmax, long long n, int group_size, int bits,
                               void* stream) {
  if (n <= 0) return 0;
  const int groups = (int)((n + group_size - 1) / group_size);
  if (bits == 8) pack_linear_kernel<int8_t><<<groups, 256, 0, (cudaStream_t)stream>>>(x, (int8_t*)code, absmax, n, group_size, 127);
  else if (bits == 16) pack_linear_kernel<int16_t><<<groups, 256, 0, (cudaStream_t)stream>>>(x, (int16_t*)code, absmax, n, group_size, 32767);
  else return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_unpack_linear(const void* code, const float* absmax, float* out, long long n, int group_size,
                                 int bits, void* stream) {
  if (n <= 0) return 0;
  const int g = cap_grid(n, 256);
  if (bits == 8) unpack_linear_kernel<int8_t><<<g, 256, 0, (cudaStream_t)stream>>>((const int8_t*)code, absmax, out, n, group_size, 127);
  else if (bits == 16) unpack_linear_kernel<int16_t><<<g, 256, 0, (cudaStream_t)stream>>>((const int16_t*)code, absmax, out, n, group_size, 32767);
  else return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_pack_nonlinear(const float* x, void* code, float* absmax, const float* qmap, long long n,
                                  int group_size, int bits, int stochastic, unsigned long long seed, void* stream) {
  if (n <= 0) return 0;
  if ((bits != 4 && bits != 8) || (bits == 4 && (group_size & 1))) return -1;
  const int groups = (int)((n + group_size - 1) / group_size);
  pack_nonlinear_kernel<<<groups, 256, 0, (cudaStream_t)stream>>>(x, (uint8_t*)code, absmax, qmap, n, group_size, bits, stochastic, seed);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int atb_unpack_nonlinear(const void* code, const float* absmax, const float* qmap, float* out, long long n,
                                    int group_size, int bits, void* stream) {
  if (n <= 0) return 0;
  unpack_nonlinear_kernel<<<cap_grid(n, 256), 256, 0, (cudaStream_t)stream>>>((const uint8_t*)code, absmax, qmap, out, n, group_size, bits);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
