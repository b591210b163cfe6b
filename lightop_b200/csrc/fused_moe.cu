// Host-side composition of the fused block-INT8 MoE layer and of the stand-alone
// grouped GEMM entry point.  Everything here only carves the caller's workspace
// and enqueues kernels on the caller's stream.
#include "common.h"
#include <mutex>

namespace lo {
float round_eps_to_dtype(float eps, int dtype);   // quant.cu
namespace {

constexpr int64_t ALIGN_BYTES = 256;

struct Carver {
  uint8_t *base;
  size_t off = 0;
  explicit Carver(void *b) : base(static_cast<uint8_t *>(b)) {}
  template <typename T> T *take(int64_t count) {
    T *p = base ? reinterpret_cast<T *>(base + off) : nullptr;
    off += (size_t)round_up(count * (int64_t)sizeof(T), ALIGN_BYTES);
    return p;
  }
};

struct FusedLayout {
  int8_t *xq;           // [sorted_cap, H] quantised activations in sorted-position order
  float *xs;            // [sorted_cap, H/128]
  int32_t *header;      // [0] num_tokens_post_pad, [1] num_chunks
  int32_t *sorted_ids;
  int32_t *inv_pos;     // [M*topk] position of every (token, slot), -1 if dropped; written and read by calls that align in a kernel of its own
  Chunk *chunks;
  int8_t *act_q;
  float *act_s;
  int64_t sorted_cap;
  int64_t chunk_cap;
  size_t bytes;
};

FusedLayout carve_fused(void *ws, int64_t M, int num_experts_for_align, int topk, int64_t H, int64_t I) {
  FusedLayout L;
  Carver c(ws);
  const int64_t numel = M * topk;
  L.sorted_cap = numel + (int64_t)num_experts_for_align * (FUSED_ALIGN_BLOCK - 1);
  L.chunk_cap = numel / 32 + num_experts_for_align + 1;   // enough for the smallest chunk size (32 rows)
  L.header = c.take<int32_t>(64);
  L.xq = c.take<int8_t>(L.sorted_cap * H);
  L.xs = c.take<float>(L.sorted_cap * (H / 128));
  L.sorted_ids = c.take<int32_t>(L.sorted_cap);
  L.inv_pos = c.take<int32_t>(numel);
  L.chunks = c.take<Chunk>(L.chunk_cap);
  L.act_q = c.take<int8_t>(L.sorted_cap * I);
  L.act_s = c.take<float>(L.sorted_cap * (I / 128));
  L.bytes = c.off;
  return L;
}

// Chunk sizes of the block-scaled layer, by the rows an expert gets on average (rows / experts).  The GEMM is instantiated per
// chunk cap and the caps differ in what fits beside the operands: 8 weight slots and 8 partial buffers with 64 rows, 7 and 4
// with 128, 7 and 3 with 160 on pairs of CTAs (5 and 3 on single ones).  Layer times in us, caps of 64 (single CTAs) / 128 / 160 rows (pairs):
//   rows per expert          32                    48                    56                    64                    100                   120                   128
//   DeepSeek-V3, even       1836 / 1931 / 1974     1988 / 2080 / 2140     2244 / 2134 / 2235     2682 / 2245 / 2314     3613 / 2665 / 2717     3950 / 3127 / 2927     4226 / 3543 / 3034
//   Zipf (1.2) routing      1228 / 1178 / 1200     1614 / 1506 / 1492     1877 / 1723 / 1694     2018 / 1842 / 1836     2812 / 2560 / 2513     3274 / 2886 / 2817     3446 / 3035 / 2946
//   Qwen3, even              417 /  448 /  459      450 /  480 /  510      493 /  498 /  524      579 /  531 /  553      786 /  630 /  653      852 /  731 /  699      942 /  842 /  730
//   Zipf                     359 /  369 /  374      454 /  445 /  451      487 /  470 /  496      542 /  520 /  523      729 /  684 /  699      853 /  801 /  797      894 /  842 /  813
//   <= 48 rows per expert : 64-row chunks.  A weight-streaming call wants the deep rings: 4 to 7 % with even routing.  With Zipf routing 128-row
//                           chunks are up to 7 % ahead from 32 rows per expert on; the routing is not known on the host.  At 56 the two
//                           are within 5 % either way with even routing, by shape, and 128 is ahead with Zipf.
//   49 .. 119             : 128-row chunks
//   176 .. 232            : 128-row chunks: nearly every expert has two chunks with either cap, and the narrower ones have the deeper rings.
//                           128 / 160 rows, even routing: Qwen3 168 rows 1028 / 1003, 176 1052 / 1066, 184 1067 / 1106, 216 1190 / 1233, 232 1234 /
//                           1265, 240 1253 / 1255; 7168 tokens of a shard with 32 experts (224) 719 / 743, 5376 (168) 610 / 612, 8192 (256) 828 / 789;
//                           Zipf 176 1012 / 1023, 224 1238 / 1197.  On single CTAs (odd tile counts, small layers) the same: 32 experts of 1024 x 384
//                           176 rows 55.4 / 59.6, 200 56.2 / 57.8, 232 59.5 / 61.2, Zipf 200 59.2 / 63.6; 64 of 4224 x 1408 184 500 / 532, 200 533 / 568, 232
//                           575 / 583, Zipf 216 606 / 596; 16 of 7296 x 1920 200 320 / 329, 232 342 / 344, Zipf 200 331 / 315, 232 348 / 366
//   otherwise >= 120      : 160-row chunks: with 128 rows per expert half of the experts have a few rows more than 128, and a
//                           second chunk means a second pass over the expert's weights (256 rows: 1374 / 1313, Zipf 1368 / 1322).
constexpr int CHUNK_ROWS = 128;
constexpr int CHUNK_ROWS_WIDE = 160;
constexpr int CHUNK_ROWS_SMALL = 64;
inline int chunk_rows_for(int64_t rows, int experts) {
  const int64_t avg = rows / experts;
  if (avg >= 176 && avg <= 232) return CHUNK_ROWS;
  return avg >= 120 ? CHUNK_ROWS_WIDE : (avg <= 48 ? CHUNK_ROWS_SMALL : CHUNK_ROWS);
}

// Rows that a chunk of a call's table may hold: the smallest size the GEMM is instantiated for that holds min(rows, chunk_max).  The
// alignment cuts the table at this size and the GEMM's instantiation is chosen by it, so that no chunk is wider than the instantiation that reads
// it.  `rows` is the number of tokens, the most an expert gets where the experts of a token are distinct; nothing makes them so (a batch
// of padding tokens may carry one id in every slot), and an expert with more rows then has more chunks.
inline int table_chunk_rows(int64_t rows, int chunk_max) {
  for (int cap : {32, CHUNK_ROWS_SMALL, CHUNK_ROWS, CHUNK_ROWS_WIDE})
    if (rows <= cap || chunk_max <= cap) return cap;
  return 256;
}

// Chunks that a table of that size can have: one an expert with rows, and one more for every full chunk.
inline int64_t most_chunks(int64_t rows, int experts, int chunk_rows) { return (rows < experts ? rows : experts) + rows / chunk_rows; }

// Whether the quantiser of the block-scaled layer reads a token's positions before its row, so that rows of tokens without a local
// expert are not read.  It then starts behind the alignment instead of beside it, which costs about 1 us: worth it where a fifth of
// the tokens or more can be expected to have no local expert (ids spread evenly over the experts) and their rows are 8 MB or more.
// Layer in us, rows first and positions first, narrow experts (I = 256), 1 of 8 shards with top-8 (34 % absent) unless said:
//   64 x 7168 52.7, 53.6    1600 x 7168 (7.9 MB) 104.2, 103.2    8192 x 7168 (40 MB) 283.5, 277.8    8192 x 7168, 1 of 4 (10 % absent) 443.8, 445.1
//   64 x 1024 21.9, 22.9    8192 x 1024 (5.8 MB) 70.1, 71.3      8192 x 4096 (23 MB) 176.6, 174.2    64 x 7168, 1 of 2 131.9, 133.0
inline bool positions_first(int64_t M, int64_t H, int topk, int E_local, int experts) {
  double absent = 1.0;
  for (int j = 0; j < topk; ++j) absent *= 1.0 - (double)E_local / experts;
  return absent >= 0.2 && absent * (double)M * (double)H * 2.0 >= 8e6;
}

// Optional per-stage timing of the fused call (cudaEvents recorded between its five kernels).
struct StageProfile {
  bool enabled = false;
  bool created = false;
  bool recorded = false;
  bool joined = false;      // alignment and quantisation were one kernel: there is no event 1
  cudaEvent_t ev[6];
};
thread_local StageProfile g_prof;

inline void prof_mark(int i, cudaStream_t st) {
  if (g_prof.enabled && g_prof.created) cudaEventRecord(g_prof.ev[i], st);
}

}  // namespace
}  // namespace lo

extern "C" int lo_profile_enable(int on) {
  using namespace lo;
  if (on && !g_prof.created) {
    for (int i = 0; i < 6; ++i) LO_CUDA_OK(cudaEventCreate(&g_prof.ev[i]));
    g_prof.created = true;
  }
  g_prof.enabled = on != 0;
  g_prof.recorded = false;
  return LO_OK;
}

extern "C" int lo_profile_read(float *ms5) {
  using namespace lo;
  LO_REQUIRE(ms5 != nullptr, "profile read: null output");
  LO_REQUIRE(g_prof.created && g_prof.recorded, "profile read: no fused call was recorded on this thread");
  LO_CUDA_OK(cudaEventSynchronize(g_prof.ev[5]));
  for (int i = 0; i < 5; ++i) {
    if (g_prof.joined && i == 0) ms5[i] = 0.f;
    else LO_CUDA_OK(cudaEventElapsedTime(&ms5[i], g_prof.ev[g_prof.joined && i == 1 ? 0 : i], g_prof.ev[i + 1]));
  }
  return LO_OK;
}

extern "C" size_t lo_fused_moe_workspace_bytes(int64_t M, int E_local, int global_num_experts, int topk, int64_t H,
                                               int64_t I) {
  const int e = global_num_experts > E_local ? global_num_experts : E_local;
  return lo::carve_fused(nullptr, M, e, topk, H, I).bytes;
}

extern "C" int lo_fused_moe_workspace_layout(int64_t M, int E_local, int global_num_experts, int topk, int64_t H,
                                            int64_t I, int64_t *out8) {
  using namespace lo;
  LO_REQUIRE(out8 != nullptr, "workspace layout: null output");
  const int e = global_num_experts > E_local ? global_num_experts : E_local;
  uint8_t *base = reinterpret_cast<uint8_t *>(uintptr_t(4096));   // any non-null base: only differences are used
  FusedLayout L = carve_fused(base, M, e, topk, H, I);
  out8[0] = reinterpret_cast<uint8_t *>(L.header) - base;
  out8[1] = reinterpret_cast<uint8_t *>(L.xq) - base;
  out8[2] = reinterpret_cast<uint8_t *>(L.xs) - base;
  out8[3] = reinterpret_cast<uint8_t *>(L.sorted_ids) - base;
  out8[4] = reinterpret_cast<uint8_t *>(L.chunks) - base;
  out8[5] = reinterpret_cast<uint8_t *>(L.act_q) - base;
  out8[6] = reinterpret_cast<uint8_t *>(L.act_s) - base;
  out8[7] = L.sorted_cap;
  return LO_OK;
}

extern "C" int lo_fused_moe_block_int8(const void *x, const int8_t *w1, const int8_t *w2, const float *w1_scale,
                                       const float *w2_scale, const float *topk_weights, const void *topk_ids,
                                       int ids_dtype, const int32_t *expert_map, int global_num_experts, int64_t M,
                                       int E_local, int topk, int64_t H, int64_t I, void *cache3,
                                       const void *shared_output, void *out, int apply_router_weight_on_input,
                                       float routed_scaling_factor, void *workspace, size_t workspace_bytes,
                                       int32_t *status, void *stream) {
  using namespace lo;
  LO_REQUIRE(M >= 0 && E_local >= 1 && topk >= 1, "fused moe: bad shape");
  if (M == 0) return LO_OK;
  LO_REQUIRE(x && w1 && w2 && w1_scale && w2_scale && topk_weights && topk_ids && cache3 && out && workspace,
             "fused moe: null pointer");
  LO_REQUIRE(H % 128 == 0 && I % 128 == 0, "fused moe: hidden (%lld) and intermediate (%lld) sizes must be multiples of 128",
             (long long)H, (long long)I);
  LO_REQUIRE(ids_dtype == LO_I32 || ids_dtype == LO_I64, "fused moe: topk_ids must be int32 or int64");
  LO_REQUIRE(!apply_router_weight_on_input || topk == 1, "fused moe: apply_router_weight_on_input requires topk == 1");
  LO_REQUIRE(M * topk < (1LL << 30), "fused moe: too many (token, slot) pairs; split the call into chunks");
  if (global_num_experts <= 0) global_num_experts = E_local;
  LO_REQUIRE(expert_map != nullptr || global_num_experts == E_local, "fused moe: global_num_experts != E needs an expert_map");
  const int align_E = expert_map ? global_num_experts : E_local;
  LO_REQUIRE(align_E <= 1024, "fused moe: more than 1024 experts");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "fused moe: workspace must be 256-byte aligned");
  LO_REQUIRE(aligned16(x, cache3, shared_output, out), "fused moe: activations, cache, shared output and result must be 16-byte aligned");
  FusedLayout L = carve_fused(workspace, M, align_E, topk, H, I);
  LO_REQUIRE(workspace_bytes >= L.bytes, "fused moe: workspace of %zu bytes, %zu needed", workspace_bytes, L.bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t numel = M * topk;
  int rc;

  const int chunk_max = table_chunk_rows(M, chunk_rows_for(numel, align_E));
  prof_mark(0, st);
  g_prof.joined = route_quant_small_fits(M, H, topk);
  if (g_prof.joined) {
    // 1 and 2 in one kernel: a launch and the wait of one kernel for the other less
    rc = launch_route_quant_small(x, M, H, topk, topk_ids, ids_dtype, align_E, expert_map, 1e-10f, L.xq, L.xs, L.sorted_ids, L.sorted_cap,
                                  L.header, L.chunks, L.header + 1, L.chunk_cap, chunk_max, st);
    if (rc != LO_OK) return rc;
  } else {
    // 1. expert-major stable order, chunk table, position of every (token, slot)
    rc = launch_align(topk_ids, ids_dtype, numel, align_E, FUSED_ALIGN_BLOCK, expert_map, expert_map ? 1 : 0,
                      L.sorted_ids, L.sorted_cap, nullptr, 0, L.header, L.chunks, L.header + 1, L.chunk_cap, L.inv_pos,
                      chunk_max, st);
    if (rc != LO_OK) return rc;

    // 2. activations -> int8 + per-128 scales, written once per routed slot into sorted order so
    //    that every chunk of the grouped GEMM is a run of consecutive rows (one TMA box)
    prof_mark(1, st);
    rc = launch_group_quant_scatter(x, M, H, topk, L.inv_pos, 1e-10f, L.xq, L.xs,
                                    expert_map != nullptr && positions_first(M, H, topk, E_local, align_E), st);
    if (rc != LO_OK) return rc;
  }

  // 3. gate_up GEMM, SiLU*mul and re-quantisation in the epilogue -> act_q/act_s in sorted order
  prof_mark(2, st);
  GemmArgs g1{};
  g1.A = L.xq; g1.a_scale = L.xs; g1.rows_a = L.sorted_cap;
  g1.max_chunk_rows = chunk_max; g1.expected_rows = ceil_div(numel, align_E); g1.max_chunks = most_chunks(numel, align_E, chunk_max);
  g1.B = w1; g1.b_scale = w1_scale; g1.E = E_local;
  g1.n_rows_per_expert = 2 * I; g1.K = H; g1.n_tiles = (int)(I / 128);
  g1.sorted_ids = L.sorted_ids; g1.numel_valid = numel;
  g1.chunks = L.chunks; g1.num_chunks = L.header + 1;
  g1.act_q = L.act_q; g1.act_s = L.act_s; g1.C = nullptr;
  g1.topk_weights = topk_weights;
  g1.weight_mode = apply_router_weight_on_input ? LO_WEIGHT_FP32 : LO_WEIGHT_NONE;
  g1.act_eps = round_eps_to_dtype(1e-10f, LO_BF16);
  g1.status = status;
  rc = launch_grouped_gemm(GEMM_GATE_UP, g1, st);
  if (rc != LO_OK) return rc;

  // 4. down GEMM, routed weight in the epilogue -> cache3[token, slot, :]
  prof_mark(3, st);
  GemmArgs g2{};
  g2.A = L.act_q; g2.a_scale = L.act_s; g2.rows_a = L.sorted_cap;
  g2.max_chunk_rows = g1.max_chunk_rows; g2.expected_rows = g1.expected_rows; g2.max_chunks = g1.max_chunks; g2.B = w2; g2.b_scale = w2_scale; g2.E = E_local;
  g2.n_rows_per_expert = H; g2.K = I; g2.n_tiles = (int)(H / 128);
  g2.sorted_ids = L.sorted_ids; g2.numel_valid = numel;
  g2.chunks = L.chunks; g2.num_chunks = L.header + 1;
  g2.C = static_cast<__nv_bfloat16 *>(cache3);
  g2.topk_weights = topk_weights;
  g2.weight_mode = apply_router_weight_on_input ? LO_WEIGHT_NONE : LO_WEIGHT_BF16_PRODUCT;
  g2.act_eps = 0.f;
  g2.status = status;
  rc = launch_grouped_gemm(GEMM_SINGLE, g2, st);
  if (rc != LO_OK) return rc;

  // 5. top-k reduction (slots of non-local experts are skipped, their rows were never written)
  prof_mark(4, st);
  rc = launch_moe_sum_masked(static_cast<const __nv_bfloat16 *>(cache3), static_cast<__nv_bfloat16 *>(out),
                             static_cast<const __nv_bfloat16 *>(shared_output), M, topk, H, routed_scaling_factor,
                             topk_ids, ids_dtype, expert_map, align_E, E_local, st);
  prof_mark(5, st);
  if (g_prof.enabled && g_prof.created) g_prof.recorded = true;
  return rc;
}

namespace lo {
namespace {
struct GemmWs {
  int32_t *num_chunks;
  Chunk *chunks;
  int8_t *a_sorted;
  float *as_sorted;
  size_t bytes;
};
GemmWs carve_gemm(void *ws, int64_t sorted_capacity, int block_size, int64_t K) {
  GemmWs W;
  Carver c(ws);
  const int64_t blocks = ceil_div(sorted_capacity, block_size);
  const int per_block = block_size <= 128 ? 1 : block_size / 128;
  W.num_chunks = c.take<int32_t>(64);
  W.chunks = c.take<Chunk>(blocks * per_block + 1);
  W.a_sorted = c.take<int8_t>(sorted_capacity * K);
  W.as_sorted = c.take<float>(sorted_capacity * (K / 128));
  W.bytes = c.off;
  return W;
}
}  // namespace
}  // namespace lo

extern "C" size_t lo_grouped_gemm_workspace_bytes(int64_t sorted_capacity, int block_size, int64_t K) {
  if (block_size <= 0 || sorted_capacity <= 0 || K <= 0) return 0;
  return lo::carve_gemm(nullptr, sorted_capacity, block_size, K).bytes;
}

namespace lo {
namespace {
// Both scale formats of the stand-alone grouped GEMM: chunk table from the caller's block table, rows and
// scales permuted into sorted order, then the kernel of the format.
int grouped_gemm_on_blocks(GemmMode mode, const int8_t *A, const float *a_scale, int64_t rows_a, const int8_t *B,
                           const float *b_scale, int E, int64_t N, int64_t K, void *C, const float *topk_weights,
                           int weight_mode, const int32_t *sorted_ids, int64_t sorted_capacity,
                           const int32_t *expert_ids, const int32_t *num_tokens_post_pad, int64_t numel_valid,
                           int top_k, int block_size, void *workspace, size_t workspace_bytes, void *stream) {
  LO_REQUIRE(A && a_scale && B && b_scale && C && sorted_ids && expert_ids && num_tokens_post_pad && workspace,
             "grouped gemm: null pointer");
  LO_REQUIRE(block_size >= 1 && (block_size <= 128 || block_size % 128 == 0),
             "grouped gemm: block_size %d must be <= 128 or a multiple of 128", block_size);
  LO_REQUIRE(top_k >= 1 && E >= 1 && rows_a >= 0 && sorted_capacity >= 1, "grouped gemm: bad shape");
  LO_REQUIRE(K % 128 == 0 && N % 128 == 0, "grouped gemm: N and K must be multiples of 128");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "grouped gemm: workspace must be 256-byte aligned");
  LO_REQUIRE(aligned16(A), "grouped gemm: operands and scales must be 16-byte aligned");
  GemmWs W = carve_gemm(workspace, sorted_capacity, block_size, K);   // sized for block scales; per-token scales need less
  LO_REQUIRE(workspace_bytes >= W.bytes, "grouped gemm: workspace of %zu bytes, %zu needed", workspace_bytes, W.bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = launch_permute_rows(A, a_scale, rows_a, K, sorted_ids, sorted_capacity, num_tokens_post_pad, numel_valid, top_k,
                           W.a_sorted, W.as_sorted, st, mode == GEMM_CHANNEL ? 1 : 0, 0, expert_ids, block_size, W.chunks, W.num_chunks);
  if (rc != LO_OK) return rc;
  GemmArgs g{};
  g.A = W.a_sorted; g.a_scale = W.as_sorted; g.rows_a = sorted_capacity;
  g.max_chunk_rows = block_size < 128 ? block_size : 128; g.expected_rows = ceil_div(numel_valid, E); g.B = B; g.b_scale = b_scale; g.E = E;
  g.n_rows_per_expert = N; g.K = K; g.n_tiles = (int)(N / 128);
  g.sorted_ids = sorted_ids; g.numel_valid = numel_valid;
  g.chunks = W.chunks; g.num_chunks = W.num_chunks;
  g.C = static_cast<__nv_bfloat16 *>(C);
  g.topk_weights = topk_weights; g.weight_mode = weight_mode; g.act_eps = 0.f; g.status = nullptr;
  return launch_grouped_gemm(mode, g, st);
}
}  // namespace
}  // namespace lo

extern "C" int lo_moe_grouped_gemm_i8_block(const int8_t *A, const float *a_scale, int64_t rows_a, const int8_t *B,
                                            const float *b_scale, int E, int64_t N, int64_t K, void *C,
                                            const float *topk_weights, int weight_mode, const int32_t *sorted_ids,
                                            int64_t sorted_capacity, const int32_t *expert_ids,
                                            const int32_t *num_tokens_post_pad, int64_t numel_valid, int top_k,
                                            int block_size, void *workspace, size_t workspace_bytes, void *stream) {
  return lo::grouped_gemm_on_blocks(lo::GEMM_SINGLE, A, a_scale, rows_a, B, b_scale, E, N, K, C, topk_weights, weight_mode,
                                    sorted_ids, sorted_capacity, expert_ids, num_tokens_post_pad, numel_valid, top_k,
                                    block_size, workspace, workspace_bytes, stream);
}

// Per-channel form of the grouped GEMM: a_scale [rows_a] (one per token), b_scale [E, N].
extern "C" int lo_moe_grouped_gemm_i8_channel(const int8_t *A, const float *a_scale, int64_t rows_a, const int8_t *B,
                                              const float *b_scale, int E, int64_t N, int64_t K, void *C,
                                              const float *topk_weights, int weight_mode, const int32_t *sorted_ids,
                                              int64_t sorted_capacity, const int32_t *expert_ids,
                                              const int32_t *num_tokens_post_pad, int64_t numel_valid, int top_k,
                                              int block_size, void *workspace, size_t workspace_bytes, void *stream) {
  return lo::grouped_gemm_on_blocks(lo::GEMM_CHANNEL, A, a_scale, rows_a, B, b_scale, E, N, K, C, topk_weights, weight_mode,
                                    sorted_ids, sorted_capacity, expert_ids, num_tokens_post_pad, numel_valid, top_k,
                                    block_size, workspace, workspace_bytes, stream);
}

// ---------------------------------------------------------------------------
// Fused layer without any caller-supplied or allocated scratch.
//
// Some hosts of this library have no way to obtain device memory at the moment they need the
// layer: a serving thread that must not trigger the implicit device-wide synchronisation of
// cudaMalloc, a plugin that is handed raw pointers by a runtime which owns the only allocator,
// a foreign-language binding (cgo / JNI / Rust FFI) that was given no allocator handle.  For
// them the scratch of the fused layer lives in a fixed array that is part of the library image:
// every GPU that loads the library reserves LO_NOALLOC_SCRATCH_BYTES for it until the process ends.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[LO_NOALLOC_SCRATCH_BYTES];

namespace lo {
namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void *g_noalloc_ptr[kMaxDevices] = {};   // device address of g_noalloc_scratch, per device ordinal

// The name g_noalloc_scratch is a host-side handle here, not an address a kernel may use: the
// device address is looked up once per device, with that device current.
int noalloc_scratch(void **out) {
  int dev = -1;
  LO_CUDA_OK(cudaGetDevice(&dev));
  LO_REQUIRE(dev >= 0 && dev < kMaxDevices, "no-alloc fused moe: device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void *ptr = nullptr;
    LO_CUDA_OK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    LO_REQUIRE(ptr != nullptr, "no-alloc fused moe: the scratch symbol has no device address");
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return LO_OK;
}
}  // namespace
}  // namespace lo

extern "C" int lo_fused_moe_block_int8_noalloc(const void *x, const int8_t *w1, const int8_t *w2,
                                               const float *w1_scale, const float *w2_scale,
                                               const float *topk_weights, const void *topk_ids, int ids_dtype,
                                               const int32_t *expert_map, int global_num_experts, int64_t M,
                                               int E_local, int topk, int64_t H, int64_t I, void *cache3,
                                               const void *shared_output, void *out,
                                               int apply_router_weight_on_input, float routed_scaling_factor,
                                               int32_t *status, void *stream) {
  using namespace lo;
  LO_REQUIRE(M >= 0 && E_local >= 1 && topk >= 1 && H >= 128 && I >= 128, "no-alloc fused moe: bad shape");
  const size_t need = lo_fused_moe_workspace_bytes(M, E_local, global_num_experts, topk, H, I);
  if (need > (size_t)LO_NOALLOC_SCRATCH_BYTES)
    return fail(LO_ERR_INVALID_ARGUMENT,
                "no-alloc fused moe: this shape needs %zu bytes of scratch, the built-in array holds %zu; "
                "use fewer tokens per call or lo_fused_moe_block_int8 with a caller-owned workspace",
                need, (size_t)LO_NOALLOC_SCRATCH_BYTES);
  void *scratch = nullptr;
  const int rc = noalloc_scratch(&scratch);
  if (rc != LO_OK) return rc;
  // Nothing in the scratch has to start at zero: every region a kernel reads for a result was written
  // earlier in the same call (sentinel fill, header, chunk table, sorted rows), so the previous call's
  // contents that remain in it are never interpreted.
  return lo_fused_moe_block_int8(x, w1, w2, w1_scale, w2_scale, topk_weights, topk_ids, ids_dtype, expert_map,
                                 global_num_experts, M, E_local, topk, H, I, cache3, shared_output, out,
                                 apply_router_weight_on_input, routed_scaling_factor, scratch, need, status, stream);
}

// ---------------------------------------------------------------------------
// Per-channel W8A8 mode of the same layer: one scale per token (activations) and one per output
// channel (weights).  The GEMMs accumulate int32 over the whole K extent on the tensor core and
// apply both scales once in the epilogue; SiLU*mul and the per-token re-quantisation need the
// maximum of a whole row, so they run as a kernel of their own between the two GEMMs, as in the
// reference (python/lightop/_lmslim_native/layers/fused_moe/int8.py:771-905).
// ---------------------------------------------------------------------------
namespace lo {
namespace {
// Chunk sizes of the per-channel layer, by the rows an expert gets on average.  A chunk is one pass over the expert's weights and
// one MMA N extent; the GEMM is instantiated per chunk cap, and on pairs of CTAs the wider caps keep the weight rings as deep as the narrow
// ones (weight slots and accumulators: 9 and 8 with 64 rows; pairs 9 and 4 with 128, 9 and 3 with 160, 9 and 2 with 256; single CTAs 9 and 4, 8 and 3,
// 5 and 2).  Layer times in us, caps of 64 (single CTAs) / 128 / 160 / 256 rows (pairs):
//   rows per expert          16                            48                            56                            93                            128
//   DeepSeek-V3, even        1747 / 1752 / 1758 / 1851     1941 / 1929 / 1952 / 2080     2085 / 1984 / 2011 / 2127     3142 / 2246 / 2248 / 2372     3825 / 3006 / 2574 / 2614
//   Zipf (1.2) routing        822 /  726 /  722 /  736     1571 / 1270 / 1229 / 1215     1789 / 1441 / 1384 / 1353     2576 / 2016 / 1864 / 1808     3294 / 2509 / 2319 / 2211
//   Qwen3, even               408 /  407 /  408 /  410      462 /  454 /  459 /  469      501 /  467 /  470 /  486      756 /  551 /  548 /  565      907 /  714 /  635 /  629
//   Zipf                      258 /  251 /  247 /  248      444 /  402 /  383 /  387      484 /  418 /  414 /  410      694 /  580 /  548 /  540      886 /  721 /  680 /  666
//   <= 136 rows per expert: 160-row chunks: as fast as narrower ones where the rows are spread evenly (within 1 %), up to 28 % faster where
//                           a few experts are hot; the routing is not known on the host.  At 2 rows per expert (66 tokens) the same.
//   above                 : 256-row chunks
// On single CTAs a weight-streaming call wants the narrow chunks (up to 56 rows per expert 64-row ones are up to 4 % ahead with even routing).
inline int channel_chunk_rows_for(int64_t rows, int experts, bool pairs) {
  const int64_t avg = rows / experts;
  return avg <= 56 && !pairs ? CHUNK_ROWS_SMALL : (avg <= 136 ? CHUNK_ROWS_WIDE : 256);
}
struct ChannelLayout {
  int32_t *header;      // [0] num_tokens_post_pad, [1] num_chunks
  int8_t *xq;           // [sorted_cap, H]
  float *xs;            // [sorted_cap]
  int32_t *sorted_ids;
  int32_t *inv_pos;
  Chunk *chunks;
  __nv_bfloat16 *cache1;   // [sorted_cap, 2I] gate_up output by sorted position
  int8_t *act_q;        // [sorted_cap, I]
  float *act_s;         // [sorted_cap]
  int64_t sorted_cap;
  int64_t chunk_cap;
  size_t bytes;
};
ChannelLayout carve_channel(void *ws, int64_t M, int num_experts_for_align, int topk, int64_t H, int64_t I) {
  ChannelLayout L;
  Carver c(ws);
  const int64_t numel = M * topk;
  L.sorted_cap = numel + (int64_t)num_experts_for_align * (FUSED_ALIGN_BLOCK - 1);
  L.chunk_cap = numel / 32 + num_experts_for_align + 1;
  L.header = c.take<int32_t>(64);
  L.xq = c.take<int8_t>(L.sorted_cap * H);
  L.xs = c.take<float>(L.sorted_cap);
  L.sorted_ids = c.take<int32_t>(L.sorted_cap);
  L.inv_pos = c.take<int32_t>(numel);
  L.chunks = c.take<Chunk>(L.chunk_cap);
  L.cache1 = c.take<__nv_bfloat16>(L.sorted_cap * 2 * I);
  L.act_q = c.take<int8_t>(L.sorted_cap * I);
  L.act_s = c.take<float>(L.sorted_cap);
  L.bytes = c.off;
  return L;
}
}  // namespace
}  // namespace lo

extern "C" size_t lo_fused_moe_channel_workspace_bytes(int64_t M, int E_local, int global_num_experts, int topk,
                                                       int64_t H, int64_t I) {
  const int e = global_num_experts > E_local ? global_num_experts : E_local;
  return lo::carve_channel(nullptr, M, e, topk, H, I).bytes;
}

extern "C" int lo_fused_moe_channel_int8(const void *x, int x_dtype, const int8_t *w1, const int8_t *w2,
                                         const float *w1_scale, const float *w2_scale, const float *topk_weights,
                                         const void *topk_ids, int ids_dtype, const int32_t *expert_map,
                                         int global_num_experts, int64_t M, int E_local, int topk, int64_t H, int64_t I,
                                         void *cache3, const void *shared_output, void *out,
                                         int apply_router_weight_on_input, float routed_scaling_factor, void *workspace,
                                         size_t workspace_bytes, int32_t *status, void *stream) {
  using namespace lo;
  LO_REQUIRE(M >= 0 && E_local >= 1 && topk >= 1, "channel moe: bad shape");
  if (M == 0) return LO_OK;
  LO_REQUIRE(x && w1 && w2 && w1_scale && w2_scale && topk_weights && topk_ids && cache3 && out && workspace,
             "channel moe: null pointer");
  LO_REQUIRE(x_dtype == LO_BF16, "channel moe: activations must be bfloat16");
  LO_REQUIRE(H % 128 == 0 && I % 128 == 0, "channel moe: hidden (%lld) and intermediate (%lld) sizes must be multiples of 128",
             (long long)H, (long long)I);
  LO_REQUIRE(ids_dtype == LO_I32 || ids_dtype == LO_I64, "channel moe: topk_ids must be int32 or int64");
  LO_REQUIRE(!apply_router_weight_on_input || topk == 1, "channel moe: apply_router_weight_on_input requires topk == 1");
  LO_REQUIRE(M * topk < (1LL << 30), "channel moe: too many (token, slot) pairs; split the call into chunks");
  if (global_num_experts <= 0) global_num_experts = E_local;
  LO_REQUIRE(expert_map != nullptr || global_num_experts == E_local, "channel moe: global_num_experts != E needs an expert_map");
  const int align_E = expert_map ? global_num_experts : E_local;
  LO_REQUIRE(align_E <= 1024, "channel moe: more than 1024 experts");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "channel moe: workspace must be 256-byte aligned");
  LO_REQUIRE(aligned16(x, cache3, shared_output, out), "channel moe: activations, cache, shared output and result must be 16-byte aligned");
  ChannelLayout L = carve_channel(workspace, M, align_E, topk, H, I);
  LO_REQUIRE(workspace_bytes >= L.bytes, "channel moe: workspace of %zu bytes, %zu needed", workspace_bytes, L.bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t numel = M * topk;
  const int64_t per_expert = ceil_div(numel, align_E);
  const bool pairs = grouped_gemm_on_pairs(GEMM_CHANNEL, E_local, per_expert, (int)(2 * I / 128), H) &&
                     grouped_gemm_on_pairs(GEMM_CHANNEL, E_local, per_expert, (int)(H / 128), I);
  const int chunk_max = table_chunk_rows(M, channel_chunk_rows_for(numel, align_E, pairs));
  // 1. expert-major stable order, chunk table, position of every (token, slot)
  prof_mark(0, st);
  g_prof.joined = false;
  int rc = launch_align(topk_ids, ids_dtype, numel, align_E, FUSED_ALIGN_BLOCK, expert_map, expert_map ? 1 : 0,
                        L.sorted_ids, L.sorted_cap, nullptr, 0, L.header, L.chunks, L.header + 1, L.chunk_cap,
                        L.inv_pos, chunk_max, st);
  if (rc != LO_OK) return rc;
  // 2. per-token quantisation, written once per routed slot into sorted order
  prof_mark(1, st);
  rc = launch_token_quant(x, x_dtype, M, H, topk, L.inv_pos, L.xq, L.xs, st);
  if (rc != LO_OK) return rc;
  // 3. gate_up GEMM -> bf16 [position, 2I]
  prof_mark(2, st);
  GemmArgs g1{};
  g1.A = L.xq; g1.a_scale = L.xs; g1.rows_a = L.sorted_cap;
  g1.max_chunk_rows = chunk_max; g1.expected_rows = ceil_div(numel, align_E); g1.max_chunks = most_chunks(numel, align_E, chunk_max);
  g1.B = w1; g1.b_scale = w1_scale; g1.E = E_local;
  g1.n_rows_per_expert = 2 * I; g1.K = H; g1.n_tiles = (int)(2 * I / 128);
  g1.sorted_ids = L.sorted_ids; g1.numel_valid = numel; g1.out_by_position = 1;
  g1.chunks = L.chunks; g1.num_chunks = L.header + 1;
  g1.C = L.cache1;
  g1.topk_weights = topk_weights;
  g1.weight_mode = apply_router_weight_on_input ? LO_WEIGHT_FP32 : LO_WEIGHT_NONE;
  g1.status = status;
  rc = launch_grouped_gemm(GEMM_CHANNEL, g1, st);
  if (rc != LO_OK) return rc;
  // SiLU*mul + per-token re-quantisation of the rows that exist (padding positions are skipped)
  rc = launch_silu_mul_token_quant(L.cache1, L.sorted_cap, I, L.sorted_ids, numel, L.header, L.act_q, L.act_s, st);
  if (rc != LO_OK) return rc;
  // 4. down GEMM, routed weight in the epilogue -> cache3[token, slot, :]
  prof_mark(3, st);
  GemmArgs g2{};
  g2.A = L.act_q; g2.a_scale = L.act_s; g2.rows_a = L.sorted_cap; g2.max_chunk_rows = g1.max_chunk_rows; g2.expected_rows = g1.expected_rows; g2.max_chunks = g1.max_chunks;
  g2.B = w2; g2.b_scale = w2_scale; g2.E = E_local;
  g2.n_rows_per_expert = H; g2.K = I; g2.n_tiles = (int)(H / 128);
  g2.sorted_ids = L.sorted_ids; g2.numel_valid = numel;
  g2.chunks = L.chunks; g2.num_chunks = L.header + 1;
  g2.C = static_cast<__nv_bfloat16 *>(cache3);
  g2.topk_weights = topk_weights;
  g2.weight_mode = apply_router_weight_on_input ? LO_WEIGHT_NONE : LO_WEIGHT_FP32;
  g2.status = status;
  rc = launch_grouped_gemm(GEMM_CHANNEL, g2, st);
  if (rc != LO_OK) return rc;
  // 5. top-k reduction
  prof_mark(4, st);
  rc = launch_moe_sum_masked(static_cast<const __nv_bfloat16 *>(cache3), static_cast<__nv_bfloat16 *>(out),
                             static_cast<const __nv_bfloat16 *>(shared_output), M, topk, H, routed_scaling_factor,
                             topk_ids, ids_dtype, expert_map, align_E, E_local, st);
  prof_mark(5, st);
  if (g_prof.enabled && g_prof.created) g_prof.recorded = true;
  return rc;
}

// ---------------------------------------------------------------------------
// Expert side of expert parallelism: rows arrive already quantised (int8 + group scales), each with
// the local expert that has to process it and, optionally, its routed weight.
// ---------------------------------------------------------------------------
namespace lo {
namespace {
// xs == nullptr: the rows are records of `x_stride` bytes, int8 row first, its group scales right behind it
int expert_rows_impl(const int8_t *xq, const float *xs, int64_t x_stride, const int32_t *row_expert,
                     const float *row_weight, const int8_t *w1, const int8_t *w2, const float *w1_scale,
                     const float *w2_scale, int64_t T, int E_local, int64_t H, int64_t I, void *out, void *workspace,
                     size_t workspace_bytes, int32_t *status, void *stream, const int64_t *row_dst = nullptr) {
  LO_REQUIRE(T >= 0 && E_local >= 1 && E_local <= 1024, "expert rows: bad shape");
  if (T == 0) return LO_OK;
  LO_REQUIRE(xq && row_expert && w1 && w2 && w1_scale && w2_scale && (out || row_dst) && workspace, "expert rows: null pointer");
  LO_REQUIRE(H % 128 == 0 && I % 128 == 0, "expert rows: hidden and intermediate sizes must be multiples of 128");
  LO_REQUIRE(T < (1LL << 30), "expert rows: too many rows");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "expert rows: workspace must be 256-byte aligned");
  LO_REQUIRE(aligned16(xq), "expert rows: rows must be 16-byte aligned");
  FusedLayout L = carve_fused(workspace, T, E_local, 1, H, I);
  LO_REQUIRE(workspace_bytes >= L.bytes, "expert rows: workspace of %zu bytes, %zu needed", workspace_bytes, L.bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // chunk sizes: the rule of lo_fused_moe_block_int8
  const int chunk_max = table_chunk_rows(T, chunk_rows_for(T, E_local));
  // 1. expert-major stable order of the rows (ids outside [0, E_local) are dropped)
  int rc = launch_align(row_expert, LO_I32, T, E_local, FUSED_ALIGN_BLOCK, nullptr, 0, L.sorted_ids, L.sorted_cap,
                        nullptr, 0, L.header, L.chunks, L.header + 1, L.chunk_cap, nullptr, chunk_max, st);
  if (rc != LO_OK) return rc;
  // 2. rows and scales into sorted order
  rc = launch_permute_rows(xq, xs, T, H, L.sorted_ids, L.sorted_cap, L.header, T, 1, L.xq, L.xs, st, 0, x_stride);
  if (rc != LO_OK) return rc;
  GemmArgs g1{};
  g1.A = L.xq; g1.a_scale = L.xs; g1.rows_a = L.sorted_cap; g1.max_chunk_rows = chunk_max; g1.expected_rows = ceil_div(T, E_local); g1.max_chunks = most_chunks(T, E_local, chunk_max);
  g1.B = w1; g1.b_scale = w1_scale; g1.E = E_local;
  g1.n_rows_per_expert = 2 * I; g1.K = H; g1.n_tiles = (int)(I / 128);
  g1.sorted_ids = L.sorted_ids; g1.numel_valid = T;
  g1.chunks = L.chunks; g1.num_chunks = L.header + 1;
  g1.act_q = L.act_q; g1.act_s = L.act_s;
  g1.weight_mode = LO_WEIGHT_NONE;
  g1.act_eps = round_eps_to_dtype(1e-10f, LO_BF16);
  g1.status = status;
  rc = launch_grouped_gemm(GEMM_GATE_UP, g1, st);
  if (rc != LO_OK) return rc;
  GemmArgs g2{};
  g2.A = L.act_q; g2.a_scale = L.act_s; g2.rows_a = L.sorted_cap; g2.max_chunk_rows = g1.max_chunk_rows; g2.expected_rows = g1.expected_rows; g2.max_chunks = g1.max_chunks;
  g2.B = w2; g2.b_scale = w2_scale; g2.E = E_local;
  g2.n_rows_per_expert = H; g2.K = I; g2.n_tiles = (int)(H / 128);
  g2.sorted_ids = L.sorted_ids; g2.numel_valid = T;
  g2.chunks = L.chunks; g2.num_chunks = L.header + 1;
  g2.C = static_cast<__nv_bfloat16 *>(out);      // top_k = 1: the sorted id is the row itself
  g2.row_dst = row_dst;                          // or: every row has an address of its own
  g2.topk_weights = row_weight;
  g2.weight_mode = row_weight ? LO_WEIGHT_BF16_PRODUCT : LO_WEIGHT_NONE;
  g2.status = status;
  return launch_grouped_gemm(GEMM_SINGLE, g2, st);
}
}  // namespace
}  // namespace lo

extern "C" int lo_expert_rows_block_int8(const int8_t *xq, const float *xs, const int32_t *row_expert,
                                         const float *row_weight, const int8_t *w1, const int8_t *w2,
                                         const float *w1_scale, const float *w2_scale, int64_t T, int E_local,
                                         int64_t H, int64_t I, void *out, void *workspace, size_t workspace_bytes,
                                         int32_t *status, void *stream) {
  LO_REQUIRE(xs != nullptr || T == 0, "expert rows: null pointer");
  return lo::expert_rows_impl(xq, xs, 0, row_expert, row_weight, w1, w2, w1_scale, w2_scale, T, E_local, H, I, out,
                              workspace, workspace_bytes, status, stream);
}

extern "C" size_t lo_expert_rows_packed_workspace_bytes(int64_t T, int E_local, int64_t H, int64_t I) {
  using namespace lo;
  return carve_fused(nullptr, T, E_local, 1, H, I).bytes + 2 * (size_t)round_up(T * 4, ALIGN_BYTES) +
         (size_t)round_up(T * 8, ALIGN_BYTES);
}

namespace lo {
namespace {
int expert_rows_packed_impl(const uint8_t *packed, int64_t T, const int8_t *w1, const int8_t *w2, const float *w1_scale,
                            const float *w2_scale, int E_local, int64_t H, int64_t I, void *out, const int32_t *seg_first,
                            const int64_t *seg_ret, int world, void *workspace, size_t workspace_bytes, int32_t *status,
                            void *stream) {
  LO_REQUIRE(T >= 0 && E_local >= 1 && H % 128 == 0 && I % 128 == 0, "expert rows (packed): bad shape");
  if (T == 0) return LO_OK;
  LO_REQUIRE(packed && workspace, "expert rows (packed): null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(packed) & 15) == 0, "expert rows (packed): records must be 16-byte aligned");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "expert rows (packed): workspace must be 256-byte aligned");
  const size_t fused_bytes = carve_fused(nullptr, T, E_local, 1, H, I).bytes;
  const size_t meta_bytes = (size_t)round_up(T * 4, ALIGN_BYTES);
  const size_t table_bytes = (size_t)round_up(T * 8, ALIGN_BYTES);
  LO_REQUIRE(workspace_bytes >= fused_bytes + 2 * meta_bytes + table_bytes,
             "expert rows (packed): workspace of %zu bytes, %zu needed", workspace_bytes, fused_bytes + 2 * meta_bytes + table_bytes);
  uint8_t *ws = static_cast<uint8_t *>(workspace);
  int32_t *row_expert = reinterpret_cast<int32_t *>(ws + fused_bytes);
  float *row_weight = reinterpret_cast<float *>(ws + fused_bytes + meta_bytes);
  int64_t *row_dst = seg_ret ? reinterpret_cast<int64_t *>(ws + fused_bytes + 2 * meta_bytes) : nullptr;
  const int64_t stride = lo_ep_dispatch_row_bytes(H);
  int rc = launch_ep_unpack_meta(packed, T, stride, H + 4 * (H / 128), row_expert, row_weight, static_cast<cudaStream_t>(stream),
                                 seg_first, seg_ret, world, 2 * H, row_dst);
  if (rc != LO_OK) return rc;
  return expert_rows_impl(reinterpret_cast<const int8_t *>(packed), nullptr, stride, row_expert, row_weight, w1, w2, w1_scale,
                          w2_scale, T, E_local, H, I, out, workspace, fused_bytes, status, stream, row_dst);
}
}  // namespace
}  // namespace lo

extern "C" int lo_expert_rows_block_int8_packed(const uint8_t *packed, int64_t T, const int8_t *w1, const int8_t *w2,
                                                const float *w1_scale, const float *w2_scale, int E_local, int64_t H,
                                                int64_t I, void *out, void *workspace, size_t workspace_bytes,
                                                int32_t *status, void *stream) {
  using namespace lo;
  LO_REQUIRE(out != nullptr || T == 0, "expert rows (packed): null pointer");
  return expert_rows_packed_impl(packed, T, w1, w2, w1_scale, w2_scale, E_local, H, I, out, nullptr, nullptr, 0, workspace,
                                 workspace_bytes, status, stream);
}

extern "C" int lo_expert_rows_block_int8_packed_put(const uint8_t *packed, int64_t T, const int8_t *w1, const int8_t *w2,
                                                    const float *w1_scale, const float *w2_scale, int E_local, int64_t H,
                                                    int64_t I, const int32_t *seg_first, const int64_t *seg_ret, int world,
                                                    void *workspace, size_t workspace_bytes, int32_t *status, void *stream) {
  using namespace lo;
  LO_REQUIRE(world >= 1 && world <= 1024 && (T == 0 || (seg_first && seg_ret)), "expert rows (put): bad return route");
  return expert_rows_packed_impl(packed, T, w1, w2, w1_scale, w2_scale, E_local, H, I, nullptr, seg_first, seg_ret, world,
                                 workspace, workspace_bytes, status, stream);
}

// ---------------------------------------------------------------------------
// Dense block-INT8 linear: the grouped GEMM with a single "expert" that owns every row.
// ---------------------------------------------------------------------------
namespace lo {
namespace {
// How a dense call is cut.  Chunks of at most 128 rows; equally many each where all items run at the same time (129 rows: 80 and
// 49), else full ones with the short one last, where it shortens the last wave (300 x 7168 x 2048: 18.7 against 20.6 us).
//
// Where the tiles would leave half of the SMs or more without work, the K extent of a tile can be dealt to n_split items of
// split_steps K blocks.  The items write the int32 sum of every K block and a second kernel carries the fp32 chain over them in
// the order of K, so a row has the same bits whatever the form and whatever the other rows of the call are.  (fp32 sums of
// the parts are a quarter of the traffic and less, but associate differently: one bf16 output in 5000 changed with the batch.)
// split_gain_us() is the rule, in microseconds: a K block taken off a CTA's chain saves 0.17 us and 0.0015 us a row; the second
// kernel costs 2.5 us and 0.08 us a K block of its chain, the sums 0.55 us a million (written and read through L2, up to 9
// million of them).  Undivided and split, kernel time in us:
//     1 x 576 x 7168: 13.6, 9.2     32 x 576 x 7168: 14.1, 11.0    128 x 576 x 7168: 22.7, 13.9    200 x 576 x 7168: 23.2, 16.5
//     1 x 4096 x 7168: 14.6, 13.5    8 x 4096 x 7168: 14.6, 14.4   16 x 4096 x 7168: 14.8, 16.1     64 x 4096 x 7168: 16.9, 27.3
//    16 x 2048 x 7168: 14.2, 12.3   64 x 2048 x 7168: 16.1, 16.0   96 x 2048 x 7168: 20.6, 22.8    128 x 2048 x 7168: 23.1, 26.2
//     1 x 576 x 4096: 9.0, 6.9      300 x 576 x 4096: 15.9, 14.4   16 x 2048 x 4096: 9.5, 8.5       32 x 2048 x 4096: 9.6, 10.1
// The rule errs by up to 0.8 us at 64 to 128 x 2048 x 4096 (15.4, 16.2) and by 2 us at 500 x 520 x 4096 (15.6, 17.6).
// Below 32 K blocks it changes little or loses: 576 x 2048 from 5.9, 5.5 (1 row) to 9.7, 9.3 (128), 1024 x 3072 from 7.6, 7.1 to
// 12.6, 11.9 with losses up to 1 us between, 1536 x 1536 5.3, 7.1.
constexpr int64_t LINEAR_CHUNK = 128;
constexpr int SPLIT_MIN_STEPS = 2, SPLIT_MIN_K = 32, SPLIT_MAX_K = 512;      // K blocks: of a part, of a split call
constexpr int64_t SPLIT_MAX_SUMS = 9000000;
inline double split_gain_us(int64_t KB, int64_t steps, int64_t chunk_rows, int64_t sums) {
  return (double)(KB - steps) * (0.17 + 0.0015 * (double)chunk_rows) - (2.5 + 0.08 * (double)KB + 0.55e-6 * (double)sums);
}
struct LinearPlan {
  int chunk_rows, n_chunks, n_tiles, split_steps, n_split;
  size_t partial_bytes;
};
LinearPlan plan_linear(int64_t M, int64_t N, int64_t K) {
  LinearPlan L;
  const int64_t n0 = ceil_div(M, LINEAR_CHUNK);
  L.n_tiles = (int)ceil_div(N, 128);
  L.chunk_rows = (int)(n0 == 1 ? M : (n0 * L.n_tiles <= sm_count() ? round_up(ceil_div(M, n0), 16) : LINEAR_CHUNK));
  L.n_chunks = (int)ceil_div(M, L.chunk_rows);
  const int64_t KB = K / 128, items = (int64_t)L.n_chunks * L.n_tiles;
  const int64_t want = sm_count() / items;       // parts that fill the SMs once
  L.split_steps = 0; L.n_split = 1; L.partial_bytes = 0;
  if (want >= 2 && KB >= SPLIT_MIN_K && KB <= SPLIT_MAX_K) {
    int64_t steps = ceil_div(KB, want);
    if (steps < SPLIT_MIN_STEPS) steps = SPLIT_MIN_STEPS;
    const int64_t sums = KB * M * N;
    if (ceil_div(KB, steps) >= 2 && sums <= SPLIT_MAX_SUMS && split_gain_us(KB, steps, L.chunk_rows, sums) > 0) {
      L.split_steps = (int)steps;
      L.n_split = (int)ceil_div(KB, steps);
      L.partial_bytes = (size_t)round_up(sums * 4, ALIGN_BYTES);
    }
  }
  return L;
}

// C from the int32 sums of the K blocks: acc = fma(float(dot), a_s * b_s, acc) over the K blocks in their order, the chain that the
// promotion warps of the undivided form carry, so both forms give the same bits.  One block per row and 128 columns; bound by the
// latency of its loads (sixteen in flight a thread): 3 us of the 9.2 at 1 x 576 x 7168.
__global__ void __launch_bounds__(128) linear_promote_kernel(const int32_t *__restrict__ partial, const float *__restrict__ a_scale,
                                                             const float *__restrict__ b_scale, int64_t M, int64_t N, int KB,
                                                             __nv_bfloat16 *__restrict__ C) {
  __shared__ float sc[SPLIT_MAX_K];
  const int64_t row = blockIdx.y, n = (int64_t)blockIdx.x * 128 + threadIdx.x;
  dependency_wait();
  for (int kb = threadIdx.x; kb < KB; kb += 128) sc[kb] = __fmul_rn(a_scale[row * KB + kb], b_scale[(int64_t)blockIdx.x * KB + kb]);
  __syncthreads();
  if (n >= N) return;
  const int64_t slab = M * N;
  const int32_t *src = partial + row * N + n;
  float acc = 0.f;
#pragma unroll 16
  for (int kb = 0; kb < KB; ++kb) acc = __fmaf_rn(__int2float_rn(__ldg(src + kb * slab)), sc[kb], acc);
  C[row * N + n] = __float2bfloat16_rn(acc);
}

int check_linear(int64_t M, int64_t N, int64_t K) {
  LO_REQUIRE(M >= 0 && N >= 1 && K >= 128 && K % 128 == 0, "block int8 linear: bad shape (K must be a multiple of 128)");
  LO_REQUIRE(M < (1LL << 30), "block int8 linear: too many rows");
  return LO_OK;
}

int run_linear(const int8_t *A, const float *a_scale, const int8_t *B, const float *b_scale, int64_t M, int64_t N, int64_t K,
               void *C, const LinearPlan &L, int32_t *partial, int32_t *status, cudaStream_t st) {
  GemmArgs g{};
  g.A = A; g.a_scale = a_scale; g.rows_a = M; g.max_chunk_rows = L.chunk_rows; g.expected_rows = L.chunk_rows;
  g.B = B; g.b_scale = b_scale; g.E = 1;
  g.n_rows_per_expert = N; g.n_store = N; g.K = K; g.n_tiles = L.n_tiles;
  g.numel_valid = M; g.fixed_chunks = L.n_chunks;
  g.C = static_cast<__nv_bfloat16 *>(C);
  g.weight_mode = LO_WEIGHT_NONE; g.status = status;
  if (L.n_split > 1 && partial != nullptr) { g.split_steps = L.split_steps; g.partial = partial; }
  const int rc = launch_grouped_gemm(GEMM_SINGLE, g, st);
  if (rc != LO_OK || g.partial == nullptr) return rc;
  LO_CUDA_OK(launch_dependent(linear_promote_kernel, dim3((unsigned)L.n_tiles, (unsigned)M), dim3(128), 0, st, (const int32_t *)partial, a_scale,
                              b_scale, M, N, (int)(K / 128), static_cast<__nv_bfloat16 *>(C)));
  return LO_OK;
}
}  // namespace
}  // namespace lo

// (the undivided form writes nothing but C)
extern "C" size_t lo_block_int8_linear_workspace_bytes(int64_t) { return 0; }

extern "C" size_t lo_block_int8_linear_split_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K < 128) return 0;
  return lo::plan_linear(M, N, K).partial_bytes;
}

extern "C" int lo_block_int8_linear(const int8_t *A, const float *a_scale, const int8_t *B, const float *b_scale,
                                    int64_t M, int64_t N, int64_t K, void *C, void *workspace, size_t workspace_bytes,
                                    int32_t *status, void *stream) {
  using namespace lo;
  const int rc = check_linear(M, N, K);
  if (rc != LO_OK || M == 0) return rc;
  LO_REQUIRE(A && a_scale && B && b_scale && C, "block int8 linear: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "block int8 linear: workspace must be 256-byte aligned");
  const LinearPlan L = plan_linear(M, N, K);
  // the K extent is split where the workspace has room for the parts
  int32_t *partial = L.n_split > 1 && workspace != nullptr && workspace_bytes >= L.partial_bytes ? static_cast<int32_t *>(workspace) : nullptr;
  return run_linear(A, a_scale, B, b_scale, M, N, K, C, L, partial, status, static_cast<cudaStream_t>(stream));
}

namespace lo {
namespace {
struct DynLinearLayout {
  int8_t *xq;
  float *xs;
  int32_t *partial;
  size_t bytes;
};
DynLinearLayout carve_dyn_linear(void *ws, int64_t M, int64_t K, const LinearPlan &L) {
  DynLinearLayout D;
  Carver c(ws);
  D.xq = c.take<int8_t>(M * K);
  D.xs = c.take<float>(M * (K / 128));
  D.partial = c.take<int32_t>((int64_t)(L.partial_bytes / 4));
  D.bytes = c.off;
  return D;
}
inline bool overlap(const void *a, size_t a_bytes, const void *b, size_t b_bytes) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
  return x < y + b_bytes && y < x + a_bytes;
}
}  // namespace
}  // namespace lo

// (enough for every call of these sizes, whichever kernels take it)
extern "C" size_t lo_block_int8_linear_dynamic_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K < 128) return 0;
  return lo::carve_dyn_linear(nullptr, M, K, lo::plan_linear(M, N, K)).bytes;
}

// (the one-kernel form keeps no scratch, and the type of x has a say in whether it takes the call)
extern "C" size_t lo_block_int8_linear_dynamic_scratch_bytes(int64_t M, int64_t N, int64_t K, int x_dtype) {
  return lo::linear_rows_fit(M, N, K, x_dtype) ? 0 : lo_block_int8_linear_dynamic_workspace_bytes(M, N, K);
}

extern "C" int lo_block_int8_linear_dynamic(const void *x, int x_dtype, const int8_t *B, const float *b_scale, int64_t M,
                                            int64_t N, int64_t K, void *C, void *workspace, size_t workspace_bytes,
                                            int32_t *status, void *stream) {
  using namespace lo;
  int rc = check_linear(M, N, K);
  if (rc != LO_OK || M == 0) return rc;
  // (every CTA of the one-kernel form reads x while others write C: a call in place takes the kernels that quantise first)
  const bool rows = linear_rows_fit(M, N, K, x_dtype) && !overlap(x, (size_t)(M * K) * (x_dtype == LO_F32 ? 4 : 2), C, (size_t)(M * N) * 2);
  LO_REQUIRE(x && B && b_scale && C && (workspace || rows), "block int8 linear: null pointer");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0, "group quant: x must be 16-byte and q 8-byte aligned");
  LO_REQUIRE((reinterpret_cast<uintptr_t>(workspace) & (ALIGN_BYTES - 1)) == 0, "block int8 linear: workspace must be 256-byte aligned");
  if (rows) {
    // (the operands that the grouped GEMM refuses are refused here too)
    LO_REQUIRE(aligned16(B, b_scale), "grouped gemm: operands and scales must be 16-byte aligned");
    LO_REQUIRE((reinterpret_cast<uintptr_t>(C) & 1) == 0, "grouped gemm: the output must be aligned to its bf16 elements");
    return launch_linear_rows(x, x_dtype, B, b_scale, M, N, K, 1e-10f, C, static_cast<cudaStream_t>(stream));
  }
  const LinearPlan L = plan_linear(M, N, K);
  DynLinearLayout D = carve_dyn_linear(workspace, M, K, L);
  LO_REQUIRE(workspace_bytes >= D.bytes, "block int8 linear: workspace of %zu bytes, %zu needed", workspace_bytes, D.bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = launch_group_quant(x, x_dtype, M * (K / 128), 128, 1e-10f, D.xq, D.xs, st);
  if (rc != LO_OK) return rc;
  return run_linear(D.xq, D.xs, B, b_scale, M, N, K, C, L, D.partial, status, st);
}
