// Per-token-group INT8 quantisation (bf16 / fp16 / fp32 -> int8 + fp32 scale per group).
//
// Arithmetic (must stay bit-identical to the reference's torch model,
// test/moe_w8a8/benchmark_moe_int8.py:60-83):
//   amax  = max |x| over the group, clamped from below by eps rounded to x's type
//   scale = amax / 127                 (IEEE fp32 division)
//   q     = trunc(clamp(x / scale, -128, 127))   (IEEE fp32 division, then round toward zero)
// Memory-bound streaming kernel: a few lanes own one group, each lane moves 32 bytes of
// input (64 of fp32 in large calls) and stores as many int8 as it has elements.
#include "common.h"
#include <type_traits>

namespace lo {
namespace {

template <typename T> struct Load8;
template <> struct Load8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16 *p, float (&v)[8]) {
    uint4 raw = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <> struct Load8<__half> {
  static __device__ __forceinline__ void load(const __half *p, float (&v)[8]) {
    uint4 raw = *reinterpret_cast<const uint4 *>(p);
    const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __half22float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
};
template <> struct Load8<float> {
  static __device__ __forceinline__ void load(const float *p, float (&v)[8]) {
    float4 a = *reinterpret_cast<const float4 *>(p);
    float4 b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
};

// Four quotients to four bytes: truncation toward zero, a NaN to -128.
__device__ __forceinline__ uint32_t pack4_rz(const float (&r)[4]) {
  int q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = __float2int_rz(fmaxf(r[i], -128.0f));
  uint32_t hi, lo;      // (saturating: 127 from above)
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q[3]), "r"(q[2]));
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(lo) : "r"(q[1]), "r"(q[0]), "r"(hi));
  return lo;
}

// A thread's N elements (16 or 8) of a group of LANES x N: maximum over the group's lanes, scale, codes.  Every lane of the warp
// calls it; the ones without a group (the last block's, absent tokens') give zeros for the maximum and get no codes: zeros over a
// scale of zero or of eps take the longest way through the library's division, which made 1 x 7168 fp32 3.2 us instead of 1.9.
// Two-byte types take the quotient from the refined reciprocal wherever the scale is finite and not near the ends of the range
// (all but groups with an infinity or, with a tiny eps, of next to nothing).  The codes are those of the IEEE quotient: every pair
// of maximum and element of bf16 and fp16 is compared with the library's division in the tests; fp32 elements keep that one.
// With the library's division and eight elements a thread the kernels were bound by their instructions: 4096 x 7168 bf16 alone
// 33 -> 22 us (the bytes take 14), into eight sorted places 60 -> 49, 8192 rows of which a shard wants two thirds 82 -> 40.
template <typename T, int LANES, int N>
__device__ __forceinline__ float quantise(const float (&v)[N], float eps_t, bool active, uint32_t (&packed)[N / 4]) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if (!active) return 0.f;
  const float scale = __fdiv_rn(fmaxf(amax, eps_t), 127.0f);
  const bool plain = sizeof(T) == 2 && scale >= 1e-30f && scale <= 1e37f;
  if (plain) {
    const float y = rcp_refined(scale);
#pragma unroll
    for (int w = 0; w < N / 4; ++w) {
      float r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = div_by(v[4 * w + i], scale, y);
      packed[w] = pack4_rz(r);
    }
  } else {
#pragma unroll
    for (int w = 0; w < N / 4; ++w) {
      float r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = __fdiv_rn(v[4 * w + i], scale);
      packed[w] = pack4_rz(r);
    }
  }
  return scale;
}

// LANES lanes x N elements = one group.  Sixteen elements a thread halve the shuffles and the address arithmetic an element costs;
// fp32, which the library's division binds in either form, has twice the warps with eight: see launch_group_quant().
template <typename T, int LANES, int N>
__global__ void __launch_bounds__(256) group_quant_kernel(const T *__restrict__ x, int8_t *__restrict__ q,
                                                          float *__restrict__ s, int64_t num_groups,
                                                          float eps_t, int q16) {
  dependency_wait();
  dependency_release();      // (a dependent kernel waits for the whole grid before it reads)
  const int64_t gthread = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t group = gthread / LANES;
  const bool active = group < num_groups;
  float v[N];
#pragma unroll
  for (int i = 0; i < N; i += 8) {
    float (&part)[8] = *reinterpret_cast<float (*)[8]>(&v[i]);
    if (active) Load8<T>::load(x + gthread * N + i, part);
    else {
#pragma unroll
      for (int j = 0; j < 8; ++j) part[j] = 0.f;
    }
  }
  uint32_t packed[N / 4];
  const float scale = quantise<T, LANES, N>(v, eps_t, active, packed);
  if (!active) return;
  int8_t *dst = q + gthread * N;
  if (N == 16 && q16) {
    *reinterpret_cast<uint4 *>(dst) = make_uint4(packed[0], packed[1], packed[N / 4 - 2], packed[N / 4 - 1]);
  } else {
#pragma unroll
    for (int w = 0; w < N / 4; w += 2) *reinterpret_cast<uint2 *>(dst + 4 * w) = make_uint2(packed[w], packed[w + 1]);
  }
  if (gthread % LANES == 0) s[group] = scale;
}

// bf16 rows [M, H], group 128: quantise once, store to each of the token's sorted positions.
// The rows are loaded and quantised while the alignment kernel is still at work.  Where many tokens are to be expected without any
// position (`positions_first`), the positions are read before that and those tokens' rows are passed over.
__global__ void __launch_bounds__(256) group_quant_scatter_kernel(const __nv_bfloat16 *__restrict__ x, int64_t M,
                                                                  int groups_per_row, int topk,
                                                                  const int32_t *__restrict__ inv_pos, float eps_t,
                                                                  int8_t *__restrict__ q_sorted,
                                                                  float *__restrict__ s_sorted, int positions_first) {
  const int64_t gthread = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t group = (uint32_t)(gthread / 8);            // (2^32 groups would be a terabyte of activations)
  const uint32_t row = group / (uint32_t)groups_per_row;
  const int gi = (int)(group - row * (uint32_t)groups_per_row);
  const int64_t token = row;
  const bool active = token < M;
  const int32_t *pos_of = inv_pos + token * topk;
  if (positions_first) dependency_wait();
  bool wanted = active;
  if (positions_first && active) {
    wanted = false;
    for (int j = 0; j < topk; ++j) wanted |= pos_of[j] >= 0;
  }
  float v[16];
  if (wanted) {
    Load8<__nv_bfloat16>::load(x + gthread * 16, *reinterpret_cast<float (*)[8]>(&v[0]));
    Load8<__nv_bfloat16>::load(x + gthread * 16 + 8, *reinterpret_cast<float (*)[8]>(&v[8]));
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.f;
  }
  if (!__any_sync(0xffffffffu, wanted)) return;          // (an exited block counts as released for the dependent launch)
  uint32_t packed[4];
  const float scale = quantise<__nv_bfloat16, 8, 16>(v, eps_t, wanted, packed);
  // everything above reads the caller's activations only; the positions come from the align kernel before this one
  if (!positions_first) dependency_wait();
  dependency_release();
  if (!wanted) return;
  const uint4 codes = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  const int64_t row_bytes = (int64_t)groups_per_row * 128;
  int8_t *dst = q_sorted + gi * 128 + (gthread & 7) * 16;
  const bool first = (gthread & 7) == 0;
#pragma unroll 4
  for (int j = 0; j < topk; ++j) {
    const int32_t pos = pos_of[j];
    if (pos < 0) continue;
    *reinterpret_cast<uint4 *>(dst + pos * row_bytes) = codes;
    if (first) s_sorted[(int64_t)pos * groups_per_row + gi] = scale;
  }
}

// ---------------------------------------------------------------------------
// Alignment and quantisation of a small call in one kernel.
//
// As kernels of their own the two are a launch each around a few hundred ids, and the second waits for one CTA of the first.  Here
// every CTA works the positions out for itself: experts of all ids in shared memory, one id a thread, rank = earlier ids of the
// same expert (counted by comparison), segments from one scan over the experts' counts.  CTA 0 writes the tables that the GEMMs
// read; the others quantise a share of one token's row each and store it at the token's positions.  Same order, tables, codes
// and scales as the two kernels.  Bound by latency (ids, count, scan, store).
// ---------------------------------------------------------------------------
constexpr int ROUTE_THREADS = 256;
static_assert(ROUTE_SMALL_IDS == ROUTE_THREADS, "one id a thread");

template <typename IdT>
__global__ void __launch_bounds__(ROUTE_THREADS) route_quant_kernel(
    const __nv_bfloat16 *__restrict__ x, int groups_per_row, int blocks_per_row, int topk, const IdT *__restrict__ ids, int numel, int E,
    const int32_t *__restrict__ expert_map, int map_mode, float eps_t, int8_t *__restrict__ q_sorted, float *__restrict__ s_sorted,
    int32_t *__restrict__ sorted_ids, int64_t sorted_capacity, int32_t *__restrict__ num_tokens_post_pad, Chunk *__restrict__ chunks,
    int32_t *__restrict__ num_chunks, int64_t chunk_capacity, int chunk_max) {
  __shared__ __align__(16) int32_t expert_of[ROUTE_SMALL_IDS];
  __shared__ int32_t pos_of[ROUTE_SMALL_IDS];
  __shared__ __align__(16) uint32_t count[1024];       // ids per expert
  __shared__ __align__(16) uint32_t offset[1024];      // before the expert: padded rows in the low half, chunks in the high half
  __shared__ uint32_t warp_tot[ROUTE_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  *reinterpret_cast<uint4 *>(&count[tid * 4]) = make_uint4(0u, 0u, 0u, 0u);
  dependency_wait();
  dependency_release();
  // a share of a token's row: eight lanes a group, sixteen elements a lane
  const int share = (int)blockIdx.x - 1, token = share / blocks_per_row;
  const int part = (share - token * blocks_per_row) * ROUTE_THREADS + tid;
  const bool active = share >= 0 && part < groups_per_row * 8;
  float v[16];
  if (active) {
    const __nv_bfloat16 *src = x + ((int64_t)token * groups_per_row * 8 + part) * 16;
    Load8<__nv_bfloat16>::load(src, *reinterpret_cast<float (*)[8]>(&v[0]));
    Load8<__nv_bfloat16>::load(src + 8, *reinterpret_cast<float (*)[8]>(&v[8]));
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.f;
  }
  const int e = load_expert<IdT>(ids, tid, numel, E, expert_map, map_mode);
  expert_of[tid] = e;
  if (blockIdx.x == 0)
    for (int64_t i = tid; i < sorted_capacity; i += ROUTE_THREADS) sorted_ids[i] = numel;
  __syncthreads();
  int rank = 0;
  if (e >= 0) {
    atomicAdd(&count[e], 1u);
    for (int i = 0; i < tid; i += 4) {
      const int4 o = *reinterpret_cast<const int4 *>(&expert_of[i]);
      rank += (o.x == e) + (i + 1 < tid && o.y == e) + (i + 2 < tid && o.z == e) + (i + 3 < tid && o.w == e);
    }
  }
  __syncthreads();
  // exclusive scan over the experts, four a thread (E <= 1024)
  {
    const uint4 c4 = *reinterpret_cast<const uint4 *>(&count[tid * 4]);
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
    uint32_t own[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      own[i] = sum;
      sum += (c[i] + FUSED_ALIGN_BLOCK - 1) / FUSED_ALIGN_BLOCK * FUSED_ALIGN_BLOCK + ((c[i] + chunk_max - 1) / chunk_max << 16);
    }
    uint32_t run = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, run, off);
      if (lane >= off) run += t;
    }
    if (lane == 31) warp_tot[warp] = run;
    __syncthreads();
    uint32_t base = run - sum;
#pragma unroll
    for (int w = 0; w < ROUTE_THREADS / 32; ++w) base += w < warp ? warp_tot[w] : 0u;
    *reinterpret_cast<uint4 *>(&offset[tid * 4]) = make_uint4(base + own[0], base + own[1], base + own[2], base + own[3]);
    if (blockIdx.x == 0 && tid == ROUTE_THREADS - 1) {
      const uint32_t total = base + sum;
      *num_tokens_post_pad = (int32_t)(total & 0xffffu);
      *num_chunks = (int64_t)(total >> 16) < chunk_capacity ? (int32_t)(total >> 16) : (int32_t)chunk_capacity;
    }
  }
  __syncthreads();
  const int pos = e >= 0 ? (int)(offset[e] & 0xffffu) + rank : -1;
  if (blockIdx.x == 0) {
    if (pos >= 0 && pos < sorted_capacity) sorted_ids[pos] = tid;
    for (int x0 = tid; x0 < E; x0 += ROUTE_THREADS) {
      // equal chunks, rounded up to segments, as the alignment kernel cuts them
      const int c = (int)count[x0], nch = (c + chunk_max - 1) / chunk_max;
      const int per = nch > 0 ? ((c + nch - 1) / nch + FUSED_ALIGN_BLOCK - 1) / FUSED_ALIGN_BLOCK * FUSED_ALIGN_BLOCK : 0;
      int ci = (int)(offset[x0] >> 16);
      for (int r = 0; r < c; r += per, ++ci)
        if (ci < chunk_capacity) {
          Chunk ch;
          ch.expert = x0;
          ch.row0 = (int)(offset[x0] & 0xffffu) + r;
          ch.rows = c - r < per ? c - r : per;
          ch.pad = (c - r - 1) / per;
          chunks[ci] = ch;
        }
    }
    return;
  }
  pos_of[tid] = pos;
  __syncthreads();
  uint32_t packed[4];
  const float scale = quantise<__nv_bfloat16, 8, 16>(v, eps_t, active, packed);
  if (!active) return;
  const uint4 codes = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  for (int j = 0; j < topk; ++j) {
    const int64_t p = pos_of[token * topk + j];
    if (p < 0) continue;
    *reinterpret_cast<uint4 *>(q_sorted + p * groups_per_row * 128 + part * 16) = codes;
    if ((part & 7) == 0) s_sorted[p * groups_per_row + (part >> 3)] = scale;
  }
}

// ---------------------------------------------------------------------------
// Per-token (whole-row) INT8 quantisation, the activation format of the per-channel W8A8 mode.
//
// Arithmetic of the reference's kernel (python/lightop/_lmslim_native/layers/gemm/int8_utils.py:21-44):
//   absmax = max(max |x|, 1e-10)       (fp32)
//   scale  = absmax / 127              (IEEE fp32 division)
//   q      = rint(x * (127 / absmax))  (one fp32 division per row, fp32 product, round half to even)
// One CTA per row: pass 1 takes the maximum, pass 2 re-reads the row (it is still in L1/L2) and
// stores 8 int8 per thread and step.  With inv_pos the int8 row and its scale are written to every
// sorted position of the token instead of to row `token` (same layout trick as the group kernel).
// ---------------------------------------------------------------------------
constexpr int TOKEN_QUANT_THREADS = 256;

__device__ __forceinline__ float block_max_256(float v, float *red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = red[lane & 7];
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, off));
  __syncthreads();   // red may be reused by the caller
  return r;
}

// Eight codes: value x inv, rounded half to even, saturated, a NaN to -128.  Adding 1.5 x 2^23 rounds to an integer and leaves its
// two's complement in the low byte (the conversion instruction runs at an eighth of the rate).
__device__ __forceinline__ uint2 quant8_rn(const float (&v)[8], float inv) {
  uint32_t b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) b[i] = __float_as_uint(__fadd_rn(fminf(fmaxf(__fmul_rn(v[i], inv), -128.0f), 127.0f), 12582912.0f));
  return make_uint2(__byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410),
                    __byte_perm(__byte_perm(b[4], b[5], 0x0040), __byte_perm(b[6], b[7], 0x0040), 0x5410));
}

template <typename T>
__global__ void __launch_bounds__(TOKEN_QUANT_THREADS) token_quant_kernel(const T *__restrict__ x, int64_t K, int topk,
                                                                          const int32_t *__restrict__ inv_pos,
                                                                          int8_t *__restrict__ q, float *__restrict__ s) {
  __shared__ float red[8];
  const int64_t row = blockIdx.x;
  dependency_wait();
  dependency_release();
  const T *xr = x + row * K;
  // rows of a length that is not a multiple of 8 are not 16-byte aligned: they take the scalar loops only
  const int64_t vecs = (K & 7) == 0 ? K / 8 : 0;
  float amax = 0.f;
  for (int64_t i = threadIdx.x; i < vecs; i += TOKEN_QUANT_THREADS) {
    float v[8];
    Load8<T>::load(xr + i * 8, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
  }
  for (int64_t i = vecs * 8 + threadIdx.x; i < K; i += TOKEN_QUANT_THREADS) amax = fmaxf(amax, fabsf((float)xr[i]));
  amax = fmaxf(block_max_256(amax, red), 1e-10f);
  const float scale = __fdiv_rn(amax, 127.0f);
  const float inv = __fdiv_rn(127.0f, amax);
  if (inv_pos == nullptr) {
    for (int64_t i = threadIdx.x; i < vecs; i += TOKEN_QUANT_THREADS) {
      float v[8];
      Load8<T>::load(xr + i * 8, v);
      *reinterpret_cast<uint2 *>(q + row * K + i * 8) = quant8_rn(v, inv);
    }
    for (int64_t i = vecs * 8 + threadIdx.x; i < K; i += TOKEN_QUANT_THREADS) {
      const float r = fminf(fmaxf(__fmul_rn((float)xr[i], inv), -128.0f), 127.0f);
      q[row * K + i] = (int8_t)__float2int_rn(r);
    }
    if (threadIdx.x == 0) s[row] = scale;
    return;
  }
  for (int64_t i = threadIdx.x; i < vecs; i += TOKEN_QUANT_THREADS) {
    float v[8];
    Load8<T>::load(xr + i * 8, v);
    const uint2 pk = quant8_rn(v, inv);
    for (int j = 0; j < topk; ++j) {
      const int32_t pos = inv_pos[row * topk + j];
      if (pos >= 0) *reinterpret_cast<uint2 *>(q + (int64_t)pos * K + i * 8) = pk;
    }
  }
  if (threadIdx.x < topk) {
    const int32_t pos = inv_pos[row * topk + threadIdx.x];
    if (pos >= 0) s[pos] = scale;
  }
}

// ---------------------------------------------------------------------------
// SiLU(gate) * up followed by per-token INT8 quantisation, one CTA per row of a bf16 [rows, 2*d]
// matrix (gate columns first).  Semantics of the reference's fused kernel
// (csrc/kernels/gated_activation/fuse_silu_mul_quant.cu:90-131), the SiLU rounded as with fp32 expf and division
// (silu_of_bf16()): act = bf16(bf16(silu(gate)) * up); scale = max|act| / 127; q = rint(act * (127 / max)),
// saturated; a row of zeros gets scale 0 and q 0.  Rows whose entry in row_ids is a padding
// sentinel (< 0 or >= numel_valid) are skipped.
// A row's loads are on their way before its id is looked up.  24 000 rows of 2048 channels take 49 us (the bytes 38); with the library's
// exponential and a refined quotient, 25 instructions an element more, 70; with the library's division and the loads behind the look-ups 139.
// 4000 x 8192 45.6 -> 29.9, 2368 x 2048 9.4 -> 7.0.  Threads a row, in us with 128 and 256:
//   1 x 2048: 1.9, 1.7    148 x 4096: 2.2, 2.2    296 x 1408: 2.1, 2.1    444 x 1408: 2.2, 2.7    2368 x 2048: 7.0, 8.6    24000 x 2048: 49, 69
//   64 x 8192: 5.1, 2.7    4000 x 8192: 49, 30    16 x 18432: 9.4, 7.0    2000 x 18432: 63, 56
// 256 up to two rows a SM, where a row's chain is all there is, and for rows of more than 4096 channels, half of which would not
// stay in the registers of 128; 128 else, where the blocks fill the SMs and fewer warps wait at a row's barrier.
// ---------------------------------------------------------------------------

// Eight activations, as bf16, of eight gates and up values; amax takes their largest magnitude.
__device__ __forceinline__ uint4 act8(const uint4 &g, const uint4 &u, float &amax) {
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
  uint32_t out[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 sl = __floats2bfloat162_rn(silu_of_bf16(__uint_as_float(gw[i] << 16)), silu_of_bf16(__uint_as_float(gw[i] & 0xffff0000u)));
    const float2 f = __bfloat1622float2(sl);
    const __nv_bfloat162 a = __floats2bfloat162_rn(f.x * __uint_as_float(uw[i] << 16), f.y * __uint_as_float(uw[i] & 0xffff0000u));
    out[i] = *reinterpret_cast<const uint32_t *>(&a);
    amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(out[i] << 16)), fabsf(__uint_as_float(out[i] & 0xffff0000u))));
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}
__device__ __forceinline__ uint2 quant8_bf16(const uint4 &a, float inv) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  return quant8_rn(v, inv);
}

constexpr int SILU_VECS = 4;      // vectors of eight channels a thread keeps: rows of up to 32 channels a thread stay in registers
template <int THREADS>
__global__ void __launch_bounds__(THREADS) silu_mul_token_quant_kernel(
    const __nv_bfloat16 *__restrict__ in, int64_t d, const int32_t *__restrict__ row_ids, int64_t numel_valid,
    const int32_t *__restrict__ num_rows_dev, int64_t group_rows, const int32_t *__restrict__ group_counts,
    int8_t *__restrict__ q, float *__restrict__ s) {
  __shared__ float red[THREADS / 32];
  const int64_t row = blockIdx.x;
  dependency_wait();
  dependency_release();
  // The grid is the capacity.  Rows that do not exist are passed over before anything of them is loaded: in the masked layout [groups,
  // group_rows, 2d] all but the first group_counts[g] rows of a group, in the sorted one all from *num_rows_dev on.  What is left there
  // is the padding of the experts' blocks, whose ids are looked up beside the loads.
  if (group_counts && row % group_rows >= group_counts[row / group_rows]) return;
  if (num_rows_dev && row >= *num_rows_dev) return;
  const uint4 *g = reinterpret_cast<const uint4 *>(in + row * 2 * d);
  const int64_t vecs = d / 8;
  const uint4 *u = g + vecs;
  const bool kept = vecs <= SILU_VECS * THREADS;      // the row's activations stay in registers
  uint4 gv[SILU_VECS], uv[SILU_VECS];
  if (kept) {
#pragma unroll
    for (int v = 0; v < SILU_VECS; ++v) {
      const int64_t i = threadIdx.x + v * THREADS;
      if (i < vecs) {
        gv[v] = g[i];
        uv[v] = u[i];
      }
    }
  }
  if (row_ids) {
    const int32_t id = row_ids[row];
    if (id < 0 || id >= numel_valid) return;
  }
  float amax = 0.f;
  if (kept) {
#pragma unroll
    for (int v = 0; v < SILU_VECS; ++v) {
      if (threadIdx.x + v * THREADS < vecs) gv[v] = act8(gv[v], uv[v], amax);
    }
  } else {
    for (int64_t i = threadIdx.x; i < vecs; i += THREADS) act8(g[i], u[i], amax);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) amax = fmaxf(amax, red[w]);
  const float inv = amax == 0.f ? 0.f : __fdiv_rn(127.0f, amax);
  if (threadIdx.x == 0) s[row] = __fdiv_rn(amax, 127.0f);
  uint2 *dst = reinterpret_cast<uint2 *>(q + row * d);
  if (kept) {
#pragma unroll
    for (int v = 0; v < SILU_VECS; ++v) {
      const int64_t i = threadIdx.x + v * THREADS;
      if (i < vecs) dst[i] = quant8_bf16(gv[v], inv);
    }
  } else {
    for (int64_t i = threadIdx.x; i < vecs; i += THREADS) {
      float again = 0.f;
      dst[i] = quant8_bf16(act8(g[i], u[i], again), inv);
    }
  }
}

template <typename T, int N>
int launch_typed(const void *x, int64_t num_groups, int group_size, float eps_t, int8_t *q, float *s,
                 cudaStream_t stream) {
  const int lanes = group_size / N;
  const int threads = 256;
  const int64_t total_threads = num_groups * lanes;
  const int64_t blocks = ceil_div(total_threads, threads);
  if (blocks > 0x7fffffffLL) return fail(LO_ERR_INVALID_ARGUMENT, "group quant: too many groups");
  const T *xp = static_cast<const T *>(x);
  const int q16 = (reinterpret_cast<uintptr_t>(q) & 15) == 0 ? 1 : 0;      // (the caller's q may begin on 8 bytes only)
  auto kernel = group_quant_kernel<T, 128 / N, N>;
  switch (group_size) {
    case 64: kernel = group_quant_kernel<T, 64 / N, N>; break;
    case 128: break;
    case 256: kernel = group_quant_kernel<T, 256 / N, N>; break;
    default: return fail(LO_ERR_UNSUPPORTED, "group quant: group_size %d not in {64,128,256}", group_size);
  }
  LO_CUDA_OK(launch_dependent(kernel, dim3((unsigned)blocks), dim3(threads), 0, stream, xp, q, s, num_groups, eps_t, q16));
  return LO_OK;
}

// ---------------------------------------------------------------------------
// Dense block-INT8 linear of one to four rows in one kernel: quantisation, dot products, promotion.
//
// With so few rows the linear is a read of the weights; the tensor cores' tile (128 outputs, one CTA) leaves most SMs without work or
// needs the K extent dealt out and a second kernel behind it, and quantisation is a launch of its own in front.  Here a CTA owns a
// few outputs over the whole K extent: it quantises the rows itself (every CTA the same ones, from L2), takes the int32 dot
// product of every 128-wide K block with dp4a, and carries the fp32 chain over the K blocks in their order: the arithmetic and
// the bits of the quantiser and of the tensor-core forms.
//
// Bound by latency: one read of weights (the first loads in flight before the rows are quantised), the quantisation, the chain.  512
// threads a CTA instead of 256 shorten the quantisation: 1 x 576 x 7168 5.2 -> 4.0 us, 1 x 4096 x 7168 14.0 -> 11.3.  Two CTAs a SM
// hold the registers to 64, at 12 to 24 bytes of spills.  By itself the form of four rows takes 79: one CTA a SM, which is the better form up to
// one CTA a SM (4 x 576 x 7168 7.3, with 64 registers 7.5) and a second wave, with the quantisation repeated, beyond: 4 x 600 x 7168 12.5, with
// 64 registers 8.8, 4 x 1187 x 3584 8.9, 6.7, 4 x 2304 x 1280 5.5, 4.2, 3 x 4745 x 896 7.0, 5.7.
// ---------------------------------------------------------------------------
constexpr int ROW_THREADS = 512, ROW_WARPS = ROW_THREADS / 32;
constexpr int ROW_CTAS = 2;      // resident CTAs a SM where there are more CTAs than SMs: what the rules below count with
constexpr int ROWS_MAX = 4;
constexpr int ROW_OUTS_MAX = 32;      // outputs of a CTA at most
constexpr int ROW_AHEAD = 4;         // 16-byte weight loads a lane has in flight
constexpr int KB_UNIT = 4;       // K blocks that a warp takes with one load: eight lanes each

// Shared memory: codes [ROWS][K], scales [ROWS][KB], dot products as fp32 [outs][ROWS][KB].
constexpr size_t rows_smem(int rows, int64_t KB, int outs) { return (size_t)rows * KB * 128 + (size_t)rows * KB * 4 + (size_t)outs * rows * KB * 4; }
constexpr size_t ROWS_SMEM_PLAIN = 48 * 1024;      // what a kernel gets without asking
static_assert(ROW_CTAS * (ROWS_SMEM_PLAIN + 1024) <= 227 * 1024, "shared memory of the resident CTAs of a SM");

template <typename T, int ROWS, int CTAS>
__global__ void __launch_bounds__(ROW_THREADS, CTAS) linear_rows_kernel(const T *__restrict__ x, const int8_t *__restrict__ B,
                                                                    const float *__restrict__ b_scale, int M, int N, int KB, int outs,
                                                                    float eps_t, __nv_bfloat16 *__restrict__ C) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t *codes = smem;                                                  // [ROWS][KB * 128]
  float *scale = reinterpret_cast<float *>(smem + ROWS * KB * 128);       // [ROWS][KB]: token scale, then times the weight block's
  float *dots = scale + ROWS * KB;                                        // [outs][ROWS][KB]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * outs;
  const int64_t K = (int64_t)KB * 128;
  const int units_per_row = (KB + KB_UNIT - 1) / KB_UNIT, units = outs * units_per_row;
  dependency_wait();
  dependency_release();      // (a dependent kernel waits for the whole grid before it reads)

  // unit u: four K blocks of one output's weights, 512 consecutive bytes
  auto load = [&](int u) {
    const int r = u / units_per_row, kb = (u - r * units_per_row) * KB_UNIT + (lane >> 3);
    if (u >= units || kb >= KB || n0 + r >= N) return make_uint4(0u, 0u, 0u, 0u);
    return __ldg(reinterpret_cast<const uint4 *>(B + (int64_t)(n0 + r) * K + kb * 128 + (lane & 7) * 16));
  };
  uint4 w[ROW_AHEAD];
#pragma unroll
  for (int i = 0; i < ROW_AHEAD; ++i) w[i] = load(warp + i * ROW_WARPS);

  // the rows, sixteen elements a thread (rows that do not exist: zero codes)
  const int parts = ROWS * KB * 8, present = M * KB * 8;
  for (int i0 = warp * 32; i0 < parts; i0 += ROW_THREADS) {
    const int i = i0 + lane;
    const bool active = i < present;
    float v[16];
    if (active) {
      Load8<T>::load(x + (int64_t)i * 16, *reinterpret_cast<float (*)[8]>(&v[0]));
      Load8<T>::load(x + (int64_t)i * 16 + 8, *reinterpret_cast<float (*)[8]>(&v[8]));
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0.f;
    }
    uint32_t packed[4] = {0u, 0u, 0u, 0u};
    const float s = quantise<T, 8, 16>(v, eps_t, active, packed);
    if (i < parts) {
      *reinterpret_cast<uint4 *>(codes + i * 16) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      // (a CTA's outputs lie in one block of 128 weight rows: their number is a power of two, at most 32)
      if ((i & 7) == 0) {
        const int g = i >> 3, kb = g % KB;
        scale[g] = active ? __fmul_rn(s, __ldg(b_scale + (int64_t)(n0 / 128) * KB + kb)) : 0.f;
      }
    }
  }
  __syncthreads();

  auto dot_unit = [&](int u, const uint4 &wv) {
    const int r = u / units_per_row, kb = (u - r * units_per_row) * KB_UNIT + (lane >> 3);
    int d[ROWS];
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      const uint4 a = kb < KB ? *reinterpret_cast<const uint4 *>(codes + (m * KB + kb) * 128 + (lane & 7) * 16) : make_uint4(0u, 0u, 0u, 0u);
      d[m] = __dp4a((int)a.x, (int)wv.x, __dp4a((int)a.y, (int)wv.y, __dp4a((int)a.z, (int)wv.z, __dp4a((int)a.w, (int)wv.w, 0))));
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)
#pragma unroll
      for (int m = 0; m < ROWS; ++m) d[m] += __shfl_xor_sync(0xffffffffu, d[m], off);
    if ((lane & 7) == 0 && kb < KB) {
#pragma unroll
      for (int m = 0; m < ROWS; ++m) dots[(r * ROWS + m) * KB + kb] = __int2float_rn(d[m]);
    }
  };
#pragma unroll
  for (int i = 0; i < ROW_AHEAD; ++i)
    if (warp + i * ROW_WARPS < units) dot_unit(warp + i * ROW_WARPS, w[i]);
  for (int u0 = warp + ROW_AHEAD * ROW_WARPS; u0 < units; u0 += ROW_AHEAD * ROW_WARPS) {
#pragma unroll
    for (int i = 0; i < ROW_AHEAD; ++i) w[i] = load(u0 + i * ROW_WARPS);
#pragma unroll
    for (int i = 0; i < ROW_AHEAD; ++i)
      if (u0 + i * ROW_WARPS < units) dot_unit(u0 + i * ROW_WARPS, w[i]);
  }
  __syncthreads();

  // acc = fma(float(dot), a_s * b_s, acc) over the K blocks in their order
  if (threadIdx.x < outs * ROWS) {
    const int r = threadIdx.x / ROWS, m = threadIdx.x - r * ROWS;
    if (m < M && n0 + r < N) {
      const float *d = dots + threadIdx.x * KB, *s = scale + m * KB;
      float acc = 0.f;
#pragma unroll 8
      for (int kb = 0; kb < KB; ++kb) acc = __fmaf_rn(d[kb], s[kb], acc);
      C[(int64_t)m * N + n0 + r] = __float2bfloat16_rn(acc);
    }
  }
}

// Outputs a CTA: a power of two, one wave of CTAs where the outputs allow it.
inline int rows_outs(int64_t N) {
  const int64_t ctas = (int64_t)ROW_CTAS * sm_count();
  int outs = 4;
  while (outs < ROW_OUTS_MAX && N > outs * ctas) outs *= 2;
  return outs;
}

template <typename T>
int launch_rows(const void *x, const int8_t *B, const float *b_scale, int64_t M, int64_t N, int64_t K, float eps_t, void *C, cudaStream_t st) {
  const int KB = (int)(K / 128);
  const int outs = rows_outs(N);
  const dim3 grid((unsigned)ceil_div(N, outs));
  const T *xt = static_cast<const T *>(x);
  __nv_bfloat16 *c = static_cast<__nv_bfloat16 *>(C);
#define LO_ROWS_CASE(R, CTAS) \
  LO_CUDA_OK(launch_dependent(linear_rows_kernel<T, R, CTAS>, grid, dim3(ROW_THREADS), rows_smem(R, KB, outs), st, xt, B, b_scale, (int)M, (int)N, KB, outs, eps_t, c))
  if (M <= 1) LO_ROWS_CASE(1, ROW_CTAS);
  else if (M <= 2) LO_ROWS_CASE(2, ROW_CTAS);
  else if constexpr (std::is_same<T, float>::value) return fail(LO_ERR_UNSUPPORTED, "linear of a few rows: more than two rows of fp32");      // linear_rows_fit() sends none
  else if ((int)grid.x <= sm_count()) LO_ROWS_CASE(ROWS_MAX, 1);
  else LO_ROWS_CASE(ROWS_MAX, ROW_CTAS);
#undef LO_ROWS_CASE
  return LO_OK;
}

}  // namespace

// eps rounded to the element type of x, the way a torch clamp(min=eps) on a tensor of
// that type sees it.
float round_eps_to_dtype(float eps, int dtype) {
  if (dtype == LO_BF16) return __bfloat162float(__float2bfloat16_rn(eps));
  if (dtype == LO_F16) return __half2float(__float2half_rn(eps));
  return eps;
}

int launch_group_quant_scatter(const void *x, int64_t M, int64_t H, int topk, const int32_t *inv_pos, float eps,
                               int8_t *q_sorted, float *s_sorted, bool positions_first, cudaStream_t stream) {
  if (M == 0) return LO_OK;
  LO_REQUIRE(H % 128 == 0, "group quant: hidden size must be a multiple of 128");
  const int64_t total_threads = M * (H / 128) * 8;
  const int64_t blocks = ceil_div(total_threads, 256);
  LO_REQUIRE(blocks <= 0x7fffffffLL, "group quant: too many groups");
  LO_CUDA_OK(launch_dependent(group_quant_scatter_kernel, dim3((unsigned)blocks), dim3(256), 0, stream,
                              static_cast<const __nv_bfloat16 *>(x), M, (int)(H / 128), topk, inv_pos,
                              round_eps_to_dtype(eps, LO_BF16), q_sorted, s_sorted, positions_first ? 1 : 0));
  return LO_OK;
}

// Up to 256 ids and one CTA a SM for the rows; every CTA repeats the counting, so more of them take longer than one that counts for all.
// Layers in a graph in us, as two kernels and as one (experts 256, narrow, unless said):
//   top-8 of 1 x 7168 44.9, 42.2   8 x 7168 71.5, 69.2   32 x 7168 170.2, 169.6 (one shard of eight 50.2, 49.4)   4 x 4096, Qwen3 widths 107.2, 103.9
//   top-2 of 32 x 256 17.7, 15.7   128 x 2048 27.8, 26.4     top-1 of 256 x 1024 (256 CTAs) 26.6, 26.6   256 x 7168 (512) 50.5, 53.0
bool route_quant_small_fits(int64_t M, int64_t H, int topk) {
  return M * topk <= ROUTE_SMALL_IDS && M * ceil_div(H / 128 * 8, ROUTE_THREADS) <= sm_count();
}
int launch_route_quant_small(const void *x, int64_t M, int64_t H, int topk, const void *topk_ids, int ids_dtype, int num_experts,
                             const int32_t *expert_map, float eps, int8_t *q_sorted, float *s_sorted, int32_t *sorted_ids, int64_t sorted_capacity,
                             int32_t *num_tokens_post_pad, Chunk *chunks, int32_t *num_chunks, int64_t chunk_capacity, int chunk_max, cudaStream_t stream) {
  LO_REQUIRE(M >= 1 && topk >= 1 && M * topk <= ROUTE_SMALL_IDS && H % 128 == 0 && num_experts >= 1 && num_experts <= 1024, "route and quantise: bad shape");
  const int groups = (int)(H / 128), per_row = (int)ceil_div(groups * 8, ROUTE_THREADS);
  const dim3 grid((unsigned)(1 + M * per_row));
  const int map_mode = expert_map ? 1 : 0;
  const float eps_t = round_eps_to_dtype(eps, LO_BF16);
  const __nv_bfloat16 *xt = static_cast<const __nv_bfloat16 *>(x);
  if (ids_dtype == LO_I32)
    LO_CUDA_OK(launch_dependent(route_quant_kernel<int32_t>, grid, dim3(ROUTE_THREADS), 0, stream, xt, groups, per_row, topk, static_cast<const int32_t *>(topk_ids),
                                (int)(M * topk), num_experts, expert_map, map_mode, eps_t, q_sorted, s_sorted, sorted_ids, sorted_capacity, num_tokens_post_pad,
                                chunks, num_chunks, chunk_capacity, chunk_max));
  else
    LO_CUDA_OK(launch_dependent(route_quant_kernel<int64_t>, grid, dim3(ROUTE_THREADS), 0, stream, xt, groups, per_row, topk, static_cast<const int64_t *>(topk_ids),
                                (int)(M * topk), num_experts, expert_map, map_mode, eps_t, q_sorted, s_sorted, sorted_ids, sorted_capacity, num_tokens_post_pad,
                                chunks, num_chunks, chunk_capacity, chunk_max));
  return LO_OK;
}

constexpr int64_t FP32_SMALL = 1 << 24;
int launch_group_quant(const void *x, int x_dtype, int64_t num_groups, int group_size, float eps, int8_t *q, float *s,
                       cudaStream_t st) {
  const float eps_t = round_eps_to_dtype(eps, x_dtype);
  switch (x_dtype) {
    case LO_BF16: return launch_typed<__nv_bfloat16, 16>(x, num_groups, group_size, eps_t, q, s, st);
    case LO_F16: return launch_typed<__half, 16>(x, num_groups, group_size, eps_t, q, s, st);
    case LO_F32:
      // Eight elements a thread up to 2^24 elements, sixteen above (the input no longer stays in L2, loads count more than warps).
      // Eight, sixteen, us: 257 x 7168 2.8, 3.8; 1024 x 2048 2.9, 4.0; 1024 x 7168 5.9, 6.3; 4096 x 2048 6.6, 6.9; 4096 x 7168 23.9,
      // 22.9 (from HBM 32.8, 30.9).
      return num_groups * group_size <= FP32_SMALL ? launch_typed<float, 8>(x, num_groups, group_size, eps_t, q, s, st)
                                                   : launch_typed<float, 16>(x, num_groups, group_size, eps_t, q, s, st);
    default: return fail(LO_ERR_UNSUPPORTED, "group quant: unsupported input dtype code %d", x_dtype);
  }
}

// Whether the one-kernel form takes the call: up to 30 million weights with one or two rows (14 million with two of fp32), 4.5 million
// with three or four, one wave of CTAs (further ones repeat the quantisation: 1 x 29184 x 1024 12.4 us against 10.4 of the other kernels, 3 x 33024
// x 128 17.5 against 5.9), and K up to the line below.  A CTA's time is that of outs * K weights, dp4a and loads in turn; the other kernels
// (quantisation, GEMM, promotion where split) give a CTA of 128 outputs to the tensor core, whose time grows with K alone and less steeply.  So
// the line falls with the outputs a CTA, and where more rows or a dearer quantisation (fp32 quotients are the library's divisions) come on top.
// Device time in us, weights from HBM, the other kernels and this one, around the lines:
//   1 row, 16 outputs: 2400 x 10240 15.0, 13.9   2400 x 12288 16.8, 17.2     32: 8192 x 3584 11.5, 11.0   6144 x 4096 12.0, 11.8 (fp16 14.5, 15.2)   4800 x 6144 14.9, 15.1
//   2 rows, 8 outputs: 1200 x 10240 12.9, 12.3   1200 x 12288 14.3, 14.8     16: 4096 x 7168 16.4, 14.1   2400 x 7168 14.0, 13.4   3072 x 8192 14.4, 17.0
//           32: 7168 x 2048 8.9, 8.1   5120 x 2560 9.3, 9.6   7168 x 4096 12.2, 15.0   (the worst inside: 2400 x 6144 11.6, 11.7, of fp16 14.9, 15.3)
//   1 row of fp32, 8: 1200 x 20480 22.6, 21.8   1200 x 24576 25.5, 25.6      16: 4096 x 7168 19.1, 16.8   3072 x 8192 17.4, 18.0
//           32: 6144 x 2048 11.4, 10.8   8192 x 3072 13.5, 14.4
//   2 rows of fp32, 8: 1536 x 6144 13.5, 13.6   1200 x 8192 15.0, 15.6       16: 2400 x 4096 13.5, 13.6   32: 6144 x 2048 12.0, 12.1
//   Far from the lines: 1 x 576 x 7168 10.7, 4.0   1 x 1536 x 1536 6.8, 3.3   2 x 576 x 7168 10.9, 5.1   2 x 2048 x 4096 11.0, 6.5
//   3 and 4 rows: 4 x 576 x 7168 11.0, 7.2   4 x 600 x 7168 11.3, 8.8   4 x 1536 x 1536 6.6, 4.2   3 x 4745 x 896 6.8, 5.7   4 x 9472 x 384 5.8, 4.4
// A pass from Python is 16 to 18 us with the other kernels and 11 to 12 with this one wherever the device takes less.
constexpr int64_t ROWS_ANY_K = 1LL << 20;
constexpr int64_t ROWS_K[4][4] = {
    // outputs a CTA: 4, 8, 16, 32
    {ROWS_ANY_K, ROWS_ANY_K, 10240, 3584},      // one row of bf16 or fp16
    {ROWS_ANY_K, 10240, 7168, 2048},            // two
    {ROWS_ANY_K, 20480, 7168, 2048},            // one row of fp32
    {8192, 5120, 3072, 1536},                   // two
};
bool linear_rows_fit(int64_t M, int64_t N, int64_t K, int x_dtype) {
  if (M < 1 || M > ROWS_MAX || N < 1 || N > (int64_t)ROW_OUTS_MAX * ROW_CTAS * sm_count() || K > ROWS_ANY_K) return false;
  const bool fp32 = x_dtype == LO_F32;
  if (fp32 && M > 2) return false;
  const int outs = rows_outs(N);
  if (M <= 2 && K > ROWS_K[(fp32 ? 2 : 0) + (M - 1)][outs == 4 ? 0 : (outs == 8 ? 1 : (outs == 16 ? 2 : 3))]) return false;
  const int64_t most = M > 2 ? 4500000 : (M == 2 && fp32 ? 14000000 : 30000000);
  const int rows = M <= 2 ? (int)M : ROWS_MAX;
  return N * K <= most && rows_smem(rows, K / 128, outs) <= ROWS_SMEM_PLAIN;
}

int launch_linear_rows(const void *x, int x_dtype, const int8_t *B, const float *b_scale, int64_t M, int64_t N, int64_t K, float eps, void *C,
                       cudaStream_t st) {
  const float eps_t = round_eps_to_dtype(eps, x_dtype);
  switch (x_dtype) {
    case LO_BF16: return launch_rows<__nv_bfloat16>(x, B, b_scale, M, N, K, eps_t, C, st);
    case LO_F16: return launch_rows<__half>(x, B, b_scale, M, N, K, eps_t, C, st);
    case LO_F32: return launch_rows<float>(x, B, b_scale, M, N, K, eps_t, C, st);
    default: return fail(LO_ERR_UNSUPPORTED, "group quant: unsupported input dtype code %d", x_dtype);
  }
}

int launch_token_quant(const void *x, int x_dtype, int64_t M, int64_t K, int topk, const int32_t *inv_pos, int8_t *q,
                       float *s, cudaStream_t stream) {
  if (M == 0) return LO_OK;
  LO_REQUIRE(K >= 1, "per-token quant: empty rows");
  LO_REQUIRE(inv_pos == nullptr || K % 8 == 0, "per-token quant: the sorted layout needs a row length that is a multiple of 8");
  LO_REQUIRE(M <= 0x7fffffffLL, "per-token quant: too many rows");
  LO_REQUIRE(inv_pos == nullptr || (topk >= 1 && topk <= TOKEN_QUANT_THREADS), "per-token quant: bad top-k");
  const unsigned blocks = (unsigned)M;
  switch (x_dtype) {
    case LO_BF16:
      LO_CUDA_OK(launch_dependent(token_quant_kernel<__nv_bfloat16>, dim3(blocks), dim3(TOKEN_QUANT_THREADS), 0, stream, static_cast<const __nv_bfloat16 *>(x), K, topk, inv_pos, q, s));
      break;
    case LO_F16:
      LO_CUDA_OK(launch_dependent(token_quant_kernel<__half>, dim3(blocks), dim3(TOKEN_QUANT_THREADS), 0, stream, static_cast<const __half *>(x), K, topk, inv_pos, q, s));
      break;
    case LO_F32:
      LO_CUDA_OK(launch_dependent(token_quant_kernel<float>, dim3(blocks), dim3(TOKEN_QUANT_THREADS), 0, stream, static_cast<const float *>(x), K, topk, inv_pos, q, s));
      break;
    default: return fail(LO_ERR_UNSUPPORTED, "per-token quant: unsupported input dtype code %d", x_dtype);
  }
  return LO_OK;
}

int launch_silu_mul_token_quant(const void *in, int64_t rows, int64_t d, const int32_t *row_ids, int64_t numel_valid,
                                const int32_t *num_rows_dev, int8_t *q, float *s, cudaStream_t stream,
                                int64_t group_rows, const int32_t *group_counts) {
  if (rows == 0) return LO_OK;
  LO_REQUIRE(d >= 8 && d % 8 == 0, "silu-mul quant: width %lld must be a multiple of 8", (long long)d);
  LO_REQUIRE(rows <= 0x7fffffffLL, "silu-mul quant: too many rows");
  const bool wide = d > 128 * 8 * SILU_VECS || rows <= 2 * (int64_t)sm_count();
  auto kernel = wide ? silu_mul_token_quant_kernel<256> : silu_mul_token_quant_kernel<128>;
  LO_CUDA_OK(launch_dependent(kernel, dim3((unsigned)rows), dim3(wide ? 256 : 128), 0, stream,
                              static_cast<const __nv_bfloat16 *>(in), d, row_ids, numel_valid, num_rows_dev,
                              group_rows > 0 ? group_rows : (int64_t)1, group_counts, q, s));
  return LO_OK;
}

}  // namespace lo

extern "C" int lo_per_token_quant_int8(const void *x, int x_dtype, int64_t M, int64_t K, int8_t *q, float *s,
                                       void *stream) {
  using namespace lo;
  LO_REQUIRE(M >= 0, "per-token quant: negative row count");
  if (M == 0) return LO_OK;
  LO_REQUIRE(x && q && s, "per-token quant: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
             "per-token quant: x must be 16-byte and q 8-byte aligned");
  return launch_token_quant(x, x_dtype, M, K, 0, nullptr, q, s, static_cast<cudaStream_t>(stream));
}

extern "C" int lo_silu_mul_quant_int8(const void *input, int64_t rows, int64_t d, int8_t *q, float *s, void *stream) {
  using namespace lo;
  LO_REQUIRE(rows >= 0, "silu-mul quant: negative row count");
  if (rows == 0) return LO_OK;
  LO_REQUIRE(input && q && s, "silu-mul quant: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(input) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
             "silu-mul quant: input must be 16-byte and q 8-byte aligned");
  return launch_silu_mul_token_quant(input, rows, d, nullptr, 0, nullptr, q, s, static_cast<cudaStream_t>(stream));
}

extern "C" int lo_silu_mul_quant_int8_masked(const void *input, int64_t groups, int64_t group_rows, int64_t d,
                                             const int32_t *tokens_per_group, int8_t *q, float *s, void *stream) {
  using namespace lo;
  LO_REQUIRE(groups >= 0 && group_rows >= 0, "silu-mul quant: negative shape");
  if (groups * group_rows == 0) return LO_OK;
  LO_REQUIRE(input && q && s, "silu-mul quant: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(input) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
             "silu-mul quant: input must be 16-byte and q 8-byte aligned");
  return launch_silu_mul_token_quant(input, groups * group_rows, d, nullptr, 0, nullptr, q, s,
                                     static_cast<cudaStream_t>(stream), group_rows, tokens_per_group);
}

extern "C" int lo_group_quant_int8(const void *x, int x_dtype, int64_t num_groups, int group_size,
                                   float eps, int8_t *q, float *s, void *stream) {
  using namespace lo;
  LO_REQUIRE(num_groups >= 0, "group quant: negative group count");
  if (num_groups == 0) return LO_OK;
  LO_REQUIRE(x && q && s, "group quant: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
             "group quant: x must be 16-byte and q 8-byte aligned");
  return launch_group_quant(x, x_dtype, num_groups, group_size, eps, q, s, static_cast<cudaStream_t>(stream));
}
