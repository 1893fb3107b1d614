// Paged grouped-query attention of the true 32-bit path, any query length, all float32 arithmetic on the CUDA cores.
//
// What it computes is what attention_generic.cu says (one row: a token's query of one head; causal, with a window or runs of
// positions, kept first keys, soft cap, distance bias, sinks).  That kernel gives a warp a row and reads every key and value
// for it alone, 32 keys one after another; here a CTA takes R rows of one sequence that share a kv head (tokens times the
// heads of its group) and brings each 32 keys and values to shared memory once for all of them (cp.async, two buffers, the
// next tile on its way while this one is worked on).  A thread forms the scores of R / 16 rows by two keys, then the outputs of
// the same rows by D / 16 columns; the sixteen threads of a row are neighbours in a warp, so maxima and sums take four shuffles.
//
// A row's result does not depend on what else is in the batch, nor on R: keys are walked in tiles of 32 at multiples of
// 32, a key that the row does not see adds nothing, and every 64 keys (a chunk) are an attention of their own whose
// (maximum, sum, outputs) are merged into the row's in ascending order.  So the chunks of a few decoding requests can run on
// CTAs of their own (R = 16, grid over chunks, `merge_kernel`) and give the bits of a prompt's CTA that walks them all (R = 64).
// Where such tiles would stay nearly empty (few keys, heads that share their keys with nobody) a warp takes a row (`warps_kernel`),
// with every operation in the same order.
//
// Measured (one B200; a warp a row before): 3 requests of 200 tokens, 12 heads of 128 over 2: 83.6 us a layer before, 13.0
// and 3.6 for the merge now; 333 tokens, 14 heads of 64 over 2: 123 us before, 37 now.
#include "common.cuh"

#ifndef SHRIKE_HEAD_DIM
#error "compile with -DSHRIKE_HEAD_DIM=<head size>"
#endif

namespace attn32 {

constexpr int D = SHRIKE_HEAD_DIM;
constexpr int THREADS = 256;
constexpr int KEYS = 32;          // keys of a tile
constexpr int CHUNK = 64;         // keys of a chunk
constexpr int ROW = D + 4;        // a row in shared memory: neighbouring rows' 16-byte pieces fall into different banks
constexpr int COLS = (D + 63) / 64;   // groups of four output columns of a thread: 4 (t % 16) + 64 i
constexpr int P_ROW = KEYS + 4;
constexpr float UNSEEN = -1.f;    // in the place of a weight, which is never negative

struct Params {
  const float* q;
  const float* k_cache;
  const float* v_cache;
  const int* block_table;
  const int* q_start;
  const int* ctx_len;
  const int* seq_of_token;
  const float* slopes;
  const float* sinks;
  float* out;
  float* partial;        // [seqs][heads][chunks][D + 2]: outputs, maximum, sum; null: rows are finished here
  int max_blocks, num_heads, num_kv_heads, page_size, num_pages, window, keep_first, num_tokens, num_seqs, chunks;
  int heads_per_cta, head_groups, skip_single;
  int early_metadata;    // 1: no kernel still running writes the tables, starts and lengths: they are read before the wait
  int aligned;           // q and out lie on 16 bytes
  float scale, softcap;
};

template <int R> constexpr size_t shared_floats() { return static_cast<size_t>(R) * ROW + 4 * KEYS * ROW + static_cast<size_t>(R) * P_ROW; }

__device__ __forceinline__ void copy16(float* smem, const float* from, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(smem))), "l"(from),
               "r"(valid ? 16 : 0));
}

// One row's running softmax.  Explicit roundings: every use of the row gives the same bits.
struct Running {
  float top, sum;
};
// (top, sum, outputs) of `next` joins those of `all`; returns the two factors of the outputs.
__device__ __forceinline__ float2 join(Running& all, const Running& next) {
  const float top = fmaxf(all.top, next.top);
  if (top == -INFINITY) return make_float2(0.f, 0.f);
  const float a = expf(all.top - top), b = expf(next.top - top);
  all.sum = __fadd_rn(__fmul_rn(all.sum, a), __fmul_rn(next.sum, b));
  all.top = top;
  return make_float2(a, b);
}
__device__ __forceinline__ float joined(float all, float a, float next, float b) { return __fadd_rn(__fmul_rn(all, a), __fmul_rn(next, b)); }

// The sink: one more term of the denominator, taken where the row is finished.  Returns the factor of the outputs.
__device__ __forceinline__ float finish(Running& row, const float* sinks, int head) {
  float shrink = 1.f;
  if (sinks != nullptr) {
    const float top = fmaxf(row.top, sinks[head]);
    shrink = expf(row.top - top);
    row.sum = __fadd_rn(__fmul_rn(row.sum, shrink), expf(sinks[head] - top));
  }
  return row.sum > 0.f ? __fdiv_rn(shrink, row.sum) : 0.f;
}

// acc += weights x values of one tile for RI rows; !FULL: some weights are marked as not seen.
template <int RI, bool FULL>
__device__ __forceinline__ void add_values(float (&acc)[RI][COLS * 4], const float* p_rows, const float* v_tile, int tx) {
#pragma unroll 2
  for (int key = 0; key < KEYS; key += 4) {
    float4 w[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) w[i] = *reinterpret_cast<const float4*>(p_rows + 16 * i * P_ROW + key);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        if (D % 64 != 0 && tx * 4 + 64 * c >= D) continue;
        const float4 v = *reinterpret_cast<const float4*>(v_tile + (key + e) * ROW + tx * 4 + 64 * c);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const float weight = e == 0 ? w[i].x : (e == 1 ? w[i].y : (e == 2 ? w[i].z : w[i].w));
          if (FULL || weight != UNSEEN) {
            acc[i][c * 4 + 0] = fmaf(weight, v.x, acc[i][c * 4 + 0]);
            acc[i][c * 4 + 1] = fmaf(weight, v.y, acc[i][c * 4 + 1]);
            acc[i][c * 4 + 2] = fmaf(weight, v.z, acc[i][c * 4 + 2]);
            acc[i][c * 4 + 3] = fmaf(weight, v.w, acc[i][c * 4 + 3]);
          }
        }
      }
    }
  }
}

// Rows: the tokens [token, token + count) of sequence `seq`, heads [head, head + heads) of one kv head; chunks [c_begin, c_end).
template <int R>
__device__ void attend(const Params& p, float* smem, int seq, int token, int count, int head, int heads, int kv_head, int c_begin, int c_end,
                       bool whole, int slot = 0) {
  constexpr int RI = R / 16;
  float* q_s = smem;                       // [R][ROW]
  float* k_s = q_s + R * ROW;              // [2][KEYS][ROW]
  float* v_s = k_s + 2 * KEYS * ROW;       // [2][KEYS][ROW]
  float* p_s = v_s + 2 * KEYS * ROW;       // [R][P_ROW]
  __shared__ long long row_s[4][KEYS];     // where a key's row lies in the pages, or -1: the lookups run two tiles ahead
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int start = p.q_start[seq], q_len = p.q_start[seq + 1] - start;
  const int position = p.ctx_len[seq] - q_len + (token - start);   // of the first of these tokens
  const int rows = count * heads;
  const int* table = p.block_table + static_cast<size_t>(seq) * p.max_blocks;
  const size_t key_stride = static_cast<size_t>(p.num_kv_heads) * D;
  const int last_key = position + count - 1;
  const int first_key = first_visible_key(position, p.window);     // the earliest that any of these rows sees (kept ones apart)
  const int kept = p.window > 0 ? min(p.keep_first, first_key) : 0;

  // tiles that some row sees, in ascending order
  auto next_tile = [&](int tile) {
    const int wanted = first_key / KEYS;
    if (tile * KEYS < kept) return tile;
    return tile < wanted ? wanted : tile;
  };
  const int tile_end = min(c_end * (CHUNK / KEYS), last_key / KEYS + 1);
  auto lookup = [&](int tile) -> long long {
    const int key = tile * KEYS + t, block = key / p.page_size;
    const int page = key <= last_key && block < p.max_blocks ? table[block] : -1;
    return page >= 0 && page < p.num_pages ? static_cast<long long>(page) * p.page_size + (key - block * p.page_size) : -1;
  };
  auto load = [&](int walked, int buffer) {
    float* k_to = k_s + buffer * KEYS * ROW;
    float* v_to = v_s + buffer * KEYS * ROW;
    for (int i = t; i < KEYS * (D / 4); i += THREADS) {
      const int r = i / (D / 4), c = i % (D / 4);
      const long long row = row_s[walked & 3][r];
      const size_t at = row >= 0 ? static_cast<size_t>(row) * key_stride + static_cast<size_t>(kv_head) * D + c * 4 : 0;
      copy16(k_to + r * ROW + c * 4, p.k_cache + at, row >= 0);
      copy16(v_to + r * ROW + c * 4, p.v_cache + at, row >= 0);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };

  int row_at[RI], row_head[RI], row_first[RI];   // position, head, first visible key; a row beyond `rows` sees nothing
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = ty + 16 * i;
    row_at[i] = r < rows ? position + r / heads : -1;
    row_head[i] = head + (r < rows ? r % heads : 0);
    row_first[i] = first_visible_key(row_at[i], p.window);
  }
  Running all[RI], run[RI];
  float total[RI][COLS * 4], acc[RI][COLS * 4];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    all[i] = Running{-INFINITY, 0.f};
    run[i] = Running{-INFINITY, 0.f};
#pragma unroll
    for (int c = 0; c < COLS * 4; ++c) total[i][c] = acc[i][c] = 0.f;
  }
  int tile = next_tile(c_begin * (CHUNK / KEYS)), buffer = 0, walked = 0;
  if (t < KEYS && tile < tile_end) {
    const int second = next_tile(tile + 1);
    row_s[0][t] = lookup(tile);
    if (second < tile_end) row_s[1][t] = lookup(second);
  }
  if (p.early_metadata) wait_for_previous();   // so far the step's metadata alone was read
  for (int i = t; i < R * (D / 4); i += THREADS) {
    const int r = i / (D / 4), c = i % (D / 4);
    const bool valid = r < rows;
    const float* from = p.q + (static_cast<size_t>(token + (valid ? r / heads : 0)) * p.num_heads + head + (valid ? r % heads : 0)) * D + c * 4;
    if (p.aligned) {
      copy16(q_s + r * ROW + c * 4, from, valid);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) q_s[r * ROW + c * 4 + e] = valid ? from[e] : 0.f;
    }
  }
  __syncthreads();
  if (tile < tile_end) load(0, 0);
  while (tile < tile_end) {
    const int following = next_tile(tile + 1), third = next_tile(following + 1);
    long long ahead = -1;
    if (t < KEYS && third < tile_end) ahead = lookup(third);
    if (following < tile_end) {
      load(walked + 1, buffer ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::);
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::);
    }
    __syncthreads();
    const float* k_tile = k_s + buffer * KEYS * ROW;
    const float* v_tile = v_s + buffer * KEYS * ROW;
    const bool held[2] = {row_s[walked & 3][tx] >= 0, row_s[walked & 3][tx + 16] >= 0};   // whether the key's page is there at all
    float s[RI][2];
#pragma unroll
    for (int i = 0; i < RI; ++i) s[i][0] = s[i][1] = 0.f;
#pragma unroll 4
    for (int c = 0; c < D / 4; ++c) {
      const float4 k0 = *reinterpret_cast<const float4*>(k_tile + tx * ROW + c * 4);
      const float4 k1 = *reinterpret_cast<const float4*>(k_tile + (tx + 16) * ROW + c * 4);
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(q_s + (ty + 16 * i) * ROW + c * 4);
        s[i][0] = fmaf(a.w, k0.w, fmaf(a.z, k0.z, fmaf(a.y, k0.y, fmaf(a.x, k0.x, s[i][0]))));
        s[i][1] = fmaf(a.w, k1.w, fmaf(a.z, k1.z, fmaf(a.y, k1.y, fmaf(a.x, k1.x, s[i][1]))));
      }
    }
    bool full = true;   // every row of this thread's sixteen sees the whole tile
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      bool seen[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int key = tile * KEYS + tx + 16 * j;
        seen[j] = held[j] && key <= row_at[i] && (key >= row_first[i] || (p.window > 0 && key < p.keep_first));
        float score = __fmul_rn(s[i][j], p.scale);
        if (p.softcap > 0.f) score = __fmul_rn(p.softcap, tanhf(__fdiv_rn(score, p.softcap)));
        if (p.slopes != nullptr) score = __fmaf_rn(-p.slopes[row_head[i]], static_cast<float>(row_at[i] - key), score);
        s[i][j] = seen[j] ? score : -INFINITY;
      }
      float top = fmaxf(s[i][0], s[i][1]);
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, offset));
      const float now = fmaxf(run[i].top, top);
      seen[0] = seen[0] && now != -INFINITY;   // nothing but -inf so far: the keys weigh nothing
      seen[1] = seen[1] && now != -INFINITY;
      full = full && ((seen[0] && seen[1]) || ty + 16 * i >= rows);
      const float p0 = seen[0] ? expf(__fadd_rn(s[i][0], -now)) : 0.f, p1 = seen[1] ? expf(__fadd_rn(s[i][1], -now)) : 0.f;
      float sum = __fadd_rn(p0, p1);
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, offset));
      if (now != -INFINITY) {
        const float shrink = expf(__fadd_rn(run[i].top, -now));
        run[i].sum = __fadd_rn(__fmul_rn(run[i].sum, shrink), sum);
        run[i].top = now;
#pragma unroll
        for (int c = 0; c < COLS * 4; ++c) acc[i][c] = __fmul_rn(acc[i][c], shrink);
      }
      // a key that the row does not see is marked, so that whatever lies in its value (a later token's) stays out
      p_s[(ty + 16 * i) * P_ROW + tx] = seen[0] ? p0 : UNSEEN;
      p_s[(ty + 16 * i) * P_ROW + tx + 16] = seen[1] ? p1 : UNSEEN;
    }
    full = __all_sync(0xffffffffu, full);   // a row's probabilities are written and read by one half warp
    __syncwarp();
    if (full) add_values<RI, true>(acc, p_s + ty * P_ROW, v_tile, tx);
    else add_values<RI, false>(acc, p_s + ty * P_ROW, v_tile, tx);
    if (t < KEYS) row_s[(walked + 2) & 3][t] = ahead;
    __syncthreads();   // the tile's buffer may be filled again
    ++walked;
    if (following >= tile_end || following / (CHUNK / KEYS) != tile / (CHUNK / KEYS)) {   // a chunk ends: it joins the row
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        if (run[i].top != -INFINITY) {
          const float2 f = join(all[i], run[i]);
#pragma unroll
          for (int c = 0; c < COLS * 4; ++c) total[i][c] = joined(total[i][c], f.x, acc[i][c], f.y);
        }
        run[i] = Running{-INFINITY, 0.f};
#pragma unroll
        for (int c = 0; c < COLS * 4; ++c) acc[i][c] = 0.f;
      }
    }
    tile = following;
    buffer ^= 1;
  }
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = ty + 16 * i;
    if (r >= rows) continue;
    if (whole) {
      const float inverse = finish(all[i], p.sinks, row_head[i]);
      float* to = p.out + (static_cast<size_t>(token + r / heads) * p.num_heads + row_head[i]) * D;
#pragma unroll
      for (int c = 0; c < COLS; ++c) {
        if (D % 64 != 0 && tx * 4 + 64 * c >= D) continue;
        float* at = to + tx * 4 + 64 * c;
        const float4 v = make_float4(total[i][c * 4] * inverse, total[i][c * 4 + 1] * inverse, total[i][c * 4 + 2] * inverse, total[i][c * 4 + 3] * inverse);
        if (p.aligned) {
          *reinterpret_cast<float4*>(at) = v;
        } else {
          at[0] = v.x, at[1] = v.y, at[2] = v.z, at[3] = v.w;
        }
      }
    } else {
      float* to = p.partial + ((static_cast<size_t>(seq) * p.num_heads + row_head[i]) * p.chunks + slot) * (D + 2);
#pragma unroll
      for (int c = 0; c < COLS; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (D % 64 == 0 || tx * 4 + 64 * c < D) to[tx * 4 + 64 * c + e] = total[i][c * 4 + e];
      if (tx == 0) {
        to[D] = all[i].top;
        to[D + 1] = all[i].sum;
      }
    }
  }
}

// The chunks that a single token's row sees: `kept` of the kept first keys, then those from `from` on that hold its window.
struct Visible {
  int kept, from, count;
};
__device__ __forceinline__ Visible visible_chunks(const Params& p, int position) {
  const int first = first_visible_key(position, p.window), kept = p.window > 0 ? (min(p.keep_first, first) + CHUNK - 1) / CHUNK : 0;
  const int from = max(first / CHUNK, kept);
  return Visible{kept, from, position < 0 ? 0 : min(p.chunks, kept + max(0, position / CHUNK - from + 1))};
}

// Single tokens: grid (chunks that a row can see, kv heads times head groups, sequences).
__global__ void __launch_bounds__(THREADS) single_kernel(const Params p) {
  extern __shared__ __align__(16) float smem[];
  let_dependents_start();
  if (!p.early_metadata) wait_for_previous();
  const int seq = blockIdx.z, kv_head = blockIdx.y / p.head_groups, group = blockIdx.y % p.head_groups;
  const int token = p.q_start[seq];
  // a longer entry: the portions kernel's; or the table is wider than the sequence is long
  const int index = blockIdx.x;
  const Visible seen = visible_chunks(p, p.ctx_len[seq] - 1);
  const int chunk = p.chunks == 1 ? 0 : (index < seen.kept ? index : seen.from + index - seen.kept);
  if (p.q_start[seq + 1] - token != 1 || (p.chunks > 1 && index >= seen.count)) {
    if (p.early_metadata) wait_for_previous();   // every CTA waits before it leaves
    return;
  }
  const int share = p.num_heads / p.num_kv_heads, head = kv_head * share + group * p.heads_per_cta;
  const int heads = min(p.heads_per_cta, share - group * p.heads_per_cta);
  attend<16>(p, smem, seq, token, 1, head, heads, kv_head, chunk, p.chunks > 1 ? chunk + 1 : 0x7ffffff, p.chunks == 1, index);
}

// A warp a (sequence, head): the chunks of a single token's row, in ascending order.
__global__ void __launch_bounds__(128) merge_kernel(const Params p) {
  let_dependents_start();
  wait_for_previous();
  const int lane = threadIdx.x & 31, work = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (work >= p.num_seqs * p.num_heads) return;
  const int seq = work / p.num_heads, head = work % p.num_heads;
  const int token = p.q_start[seq];
  if (p.q_start[seq + 1] - token != 1) return;
  const int chunks = visible_chunks(p, p.ctx_len[seq] - 1).count;
  const float* from = p.partial + static_cast<size_t>(work) * p.chunks * (D + 2);
  constexpr int OWN = (D + 31) / 32;
  float total[OWN];
#pragma unroll
  for (int i = 0; i < OWN; ++i) total[i] = 0.f;
  Running all{-INFINITY, 0.f};
#pragma unroll 4
  for (int c = 0; c < chunks; ++c) {
    const float* mine = from + static_cast<size_t>(c) * (D + 2);
    float value[OWN];
#pragma unroll
    for (int i = 0; i < OWN; ++i) value[i] = lane + 32 * i < D ? mine[lane + 32 * i] : 0.f;
    const Running run{mine[D], mine[D + 1]};
    if (run.top == -INFINITY) continue;
    const float2 f = join(all, run);
#pragma unroll
    for (int i = 0; i < OWN; ++i) total[i] = joined(total[i], f.x, value[i], f.y);
  }
  const float inverse = finish(all, p.sinks, head);
  float* to = p.out + (static_cast<size_t>(token) * p.num_heads + head) * D;
#pragma unroll
  for (int i = 0; i < OWN; ++i)
    if (lane + 32 * i < D) to[lane + 32 * i] = total[i] * inverse;
}

// Portions: grid (tiles of tokens of the flat batch, kv heads times head groups); a tile's sequences one after another.
template <int R>
__global__ void __launch_bounds__(THREADS) portions_kernel(const Params p) {
  extern __shared__ __align__(16) float smem[];
  let_dependents_start();
  if (!p.early_metadata) wait_for_previous();
  const int kv_head = blockIdx.y / p.head_groups, group = blockIdx.y % p.head_groups;
  const int share = p.num_heads / p.num_kv_heads, head = kv_head * share + group * p.heads_per_cta;
  const int heads = min(p.heads_per_cta, share - group * p.heads_per_cta);
  const int a_tile = R / p.heads_per_cta;
  // the last tiles walk the most keys: they start first
  const int first = (gridDim.x - 1 - blockIdx.x) * a_tile, end = min(p.num_tokens, first + a_tile);
  for (int token = first; token < end;) {
    const int seq = p.seq_of_token[token];
    const int stop = min(end, p.q_start[seq + 1]);
    if (!p.skip_single || p.q_start[seq + 1] - p.q_start[seq] > 1) {
      __syncthreads();   // the sequence before is done with shared memory
      attend<R>(p, smem, seq, token, stop - token, head, heads, kv_head, 0, 0x7ffffff, true);
    }
    token = stop > token ? stop : token + 1;
  }
  if (p.early_metadata) wait_for_previous();
}

// A warp a row: short contexts, and rows that share their keys with nobody, for which a CTA's tiles stay nearly empty.  A lane
// forms a key's score, then the warp walks the tile's keys, a lane D / 32 columns.  Every operation and its order are those of
// `attend`, so are the bits.  `which`: 0 every token, 1 those of entries of one token, 2 the others.  WIDE: keys lie on 16 bytes.
constexpr int WARPS = 4;
template <bool WIDE>
__global__ void __launch_bounds__(WARPS * 32) warps_kernel(const Params p, int which) {
  __shared__ __align__(16) float q_s[WARPS][D];
  let_dependents_start();
  if (!p.early_metadata) wait_for_previous();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long work = static_cast<long long>(blockIdx.x) * WARPS + warp;
  const int token = static_cast<int>(work / p.num_heads), head = static_cast<int>(work % p.num_heads);
  const int seq = token < p.num_tokens ? p.seq_of_token[token] : 0;
  const int start = p.q_start[seq], q_len = p.q_start[seq + 1] - start;
  if (token >= p.num_tokens || (which == 1 && q_len != 1) || (which == 2 && q_len == 1)) {
    if (p.early_metadata) wait_for_previous();
    return;
  }
  constexpr int OWN = (D + 31) / 32, AHEAD = OWN <= 4 ? 8 : 4;   // columns of a lane; keys whose values are on their way together
  const int position = p.ctx_len[seq] - q_len + (token - start), first = first_visible_key(position, p.window);
  const int kept = p.window > 0 ? min(p.keep_first, first) : 0;
  const int* table = p.block_table + static_cast<size_t>(seq) * p.max_blocks;
  const size_t key_stride = static_cast<size_t>(p.num_kv_heads) * D, column = static_cast<size_t>(head / (p.num_heads / p.num_kv_heads)) * D;
  const float slope = p.slopes != nullptr ? p.slopes[head] : 0.f;
  if (p.early_metadata) wait_for_previous();
  const float* q = p.q + (static_cast<size_t>(token) * p.num_heads + head) * D;
  for (int d = lane; d < D; d += 32) q_s[warp][d] = q[d];
  __syncwarp();
  Running all{-INFINITY, 0.f}, run{-INFINITY, 0.f};
  float total[OWN], acc[OWN];
#pragma unroll
  for (int i = 0; i < OWN; ++i) total[i] = acc[i] = 0.f;
  const int tile_end = position / KEYS + 1;
  auto next_tile = [&](int tile) { return tile * KEYS < kept || tile >= first / KEYS ? tile : first / KEYS; };
  for (int tile = next_tile(0); position >= 0 && tile < tile_end;) {
    const int key = tile * KEYS + lane, block = key / p.page_size;
    const int page = key <= position && block < p.max_blocks ? table[block] : -1;
    const long long row = page >= 0 && page < p.num_pages ? static_cast<long long>(page) * p.page_size + (key - block * p.page_size) : -1;
    bool seen = row >= 0 && (key >= first || (p.window > 0 && key < p.keep_first));
    float score = 0.f;
    if (seen) {
      const float* k = p.k_cache + static_cast<size_t>(row) * key_stride + column;
#pragma unroll 32
      for (int c = 0; c < D; c += 4) {
        float4 b;
        if (WIDE) b = *reinterpret_cast<const float4*>(k + c);
        else b = make_float4(k[c], k[c + 1], k[c + 2], k[c + 3]);
        const float4 a = *reinterpret_cast<const float4*>(&q_s[warp][c]);
        score = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, score))));
      }
      score = __fmul_rn(score, p.scale);
      if (p.softcap > 0.f) score = __fmul_rn(p.softcap, tanhf(__fdiv_rn(score, p.softcap)));
      if (p.slopes != nullptr) score = __fmaf_rn(-slope, static_cast<float>(position - key), score);
    }
    const float now = fmaxf(run.top, warp_max(seen ? score : -INFINITY));
    seen = seen && now != -INFINITY;   // nothing but -inf so far: the keys weigh nothing
    const float weight = seen ? expf(__fadd_rn(score, -now)) : 0.f;
    float sum = weight;
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, offset));
    if (now != -INFINITY) {
      const float shrink = expf(__fadd_rn(run.top, -now));
      run.sum = __fadd_rn(__fmul_rn(run.sum, shrink), sum);
      run.top = now;
#pragma unroll
      for (int i = 0; i < OWN; ++i) acc[i] = __fmul_rn(acc[i], shrink);
    }
    for (unsigned left = __ballot_sync(0xffffffffu, seen); left != 0;) {   // the keys that the row sees, in ascending order
      float v[AHEAD][OWN], w[AHEAD];
      int count = 0;
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int j = left != 0 ? __ffs(left) - 1 : 0;
        w[a] = __shfl_sync(0xffffffffu, weight, j);
        const long long row_j = __shfl_sync(0xffffffffu, row, j);
        if (left != 0) {
          const float* from = p.v_cache + static_cast<size_t>(row_j) * key_stride + column;
#pragma unroll
          for (int i = 0; i < OWN; ++i) v[a][i] = lane + 32 * i < D ? from[lane + 32 * i] : 0.f;
          count = a + 1;
          left &= left - 1;
        }
      }
#pragma unroll
      for (int a = 0; a < AHEAD; ++a)
        if (a < count) {
#pragma unroll
          for (int i = 0; i < OWN; ++i) acc[i] = fmaf(w[a], v[a][i], acc[i]);
        }
    }
    const int following = next_tile(tile + 1);
    if (following >= tile_end || following / (CHUNK / KEYS) != tile / (CHUNK / KEYS)) {   // a chunk ends: it joins the row
      if (run.top != -INFINITY) {
        const float2 f = join(all, run);
#pragma unroll
        for (int i = 0; i < OWN; ++i) total[i] = joined(total[i], f.x, acc[i], f.y);
      }
      run = Running{-INFINITY, 0.f};
#pragma unroll
      for (int i = 0; i < OWN; ++i) acc[i] = 0.f;
    }
    tile = following;
  }
  const float inverse = finish(all, p.sinks, head);
  float* to = p.out + (static_cast<size_t>(token) * p.num_heads + head) * D;
#pragma unroll
  for (int i = 0; i < OWN; ++i)
    if (lane + 32 * i < D) to[lane + 32 * i] = total[i] * inverse;
}

}  // namespace attn32

SHRIKE_API int shrike_attention_head_dim() { return attn32::D; }

// Chunks of single tokens' keys: what tables of `keys` keys hold, no more than a window (or run of positions, `window` < 0) and the
// kept first keys can reach.
SHRIKE_API int shrike_attention_fp32_chunks(int keys, int window, int keep_first) {
  constexpr long long C = attn32::CHUNK;
  const long long all = (static_cast<long long>(keys) + C - 1) / C, span = window < 0 ? -static_cast<long long>(window) : window;
  if (window == 0) return static_cast<int>(all);
  const long long seen = (span + C - 1) / C + 1 + (window > 0 ? (keep_first + C - 1) / C : 0);
  return static_cast<int>(seen < all ? seen : all);
}

// How single tokens (portions) should run: 1 the CTA forms, 2 a warp a row.  `keys`: the most that a row can see.
//
// A CTA's sixteen rows are the heads of one kv head; with one or two of them it multiplies mostly zeros, which costs nothing
// while SMs are idle, and many such pairs are quicker with a warp a row.  Measured, us with tiles and with warps: 8 heads of 64 over 8: 16
// requests (128 pairs) 64 keys 14.9 and 9.2, 128 keys 14.9 and 16.5, 200 keys 21.7 and 25.4; 32 requests 200 keys 34.2 and 25.6, 1,000
// keys 111 and 201; 64 requests 400 keys 85 and 84, 1,000 keys 195 and 202; 128 requests 1,000 keys 382 and 243; 32 heads of 128 over
// 32: 8 requests 200 keys 49.5 and 34.1, 400 keys 85 and 109; 16 requests 1,000 keys 363 and 278; 16 heads of 64 over 8: 64 requests 200
// keys 49.8 and 44.9, 1,000 keys 195 and 245; 128 requests 1,000 keys 378 and 308.  From three heads a kv head on only the first few
// keys are quicker that way (12 heads of 128 over 2, 64 requests: 3 keys 9.5 and 5.1, 20 keys 10.0 and 9.3, 64 keys 16.4 and 21.8).
SHRIKE_API int shrike_attention_fp32_single_form(int num_seqs, int num_heads, int num_kv_heads, int keys) {
  if (keys <= 8) return 2;
  const int share = num_kv_heads > 0 ? num_heads / num_kv_heads : 0;
  if (share < 1 || share > 2) return 1;
  const long long pairs = static_cast<long long>(num_seqs) * num_kv_heads;
  return pairs >= 512 * share || (pairs >= 256 && keys <= 256) || (pairs >= 128 && keys <= 128) ? 2 : 1;
}
// A CTA takes its tokens' sequences one after another: with entries of few rows, several of them to a tile of sixteen (us with tiles and
// with warps: 8 heads of 64 over 8: 8 entries of 2 tokens 26.8 and 3.5, 32 of 4 tokens over 60 keys 23.1 and 14.7, of 8 tokens over
// 200 keys 44.2 and 60.9; 16 heads over 8: 100 entries of 3 tokens 55.8 and 26.1 [6 rows], 32 of 4 over 60 keys 15.4 and 21.9 [8 rows]).
SHRIKE_API int shrike_attention_fp32_portion_form(int num_tokens, int num_seqs, int num_heads, int num_kv_heads) {
  if (num_kv_heads <= 0) return 1;
  return num_seqs > 1 && static_cast<long long>(num_tokens) * (num_heads / num_kv_heads) <= 6LL * num_seqs ? 2 : 1;
}

// `has_single` 1: single tokens run on CTAs per chunk (scratch: float32 [seqs][heads][chunks][head size + 2]); `has_portions` 1: the
// entries of more than one token (all entries when there is no `has_single`) run on tiles of tokens; 2: a warp a row.  All give
// the same bits.  Keys or values that do not lie on 16 bytes, and more sequences or kv heads than a grid has places for, go to
// the warps.  `early_metadata` 1: the caller knows that whatever wrote the block table, q_start, ctx_len and seq_of_token has
// finished (a copy, or an earlier step).
SHRIKE_API int shrike_paged_attention_fp32(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                                           int max_blocks, const int* q_start, const int* ctx_len, const int* seq_of_token,
                                           int num_tokens, int num_seqs, int num_heads, int num_kv_heads, int page_size, int num_pages,
                                           float scale, int window, float softcap, const float* slopes, const float* sinks,
                                           int keep_first, int has_single, int has_portions, int chunks, float* scratch,
                                           int early_metadata, void* out, cudaStream_t stream) {
  using namespace attn32;
  if (num_tokens <= 0) return SHRIKE_OK;
  if (keep_first < 0 || num_heads <= 0 || num_kv_heads <= 0 || num_heads % num_kv_heads || page_size <= 0 || max_blocks <= 0 || num_seqs <= 0 ||
      chunks < 1 || (has_single == 1 && chunks > 1 && scratch == nullptr))
    return SHRIKE_BAD_ARGUMENT;
  Params p = {};
  p.q = static_cast<const float*>(q);
  p.k_cache = static_cast<const float*>(k_cache);
  p.v_cache = static_cast<const float*>(v_cache);
  p.block_table = block_table;
  p.q_start = q_start;
  p.ctx_len = ctx_len;
  p.seq_of_token = seq_of_token;
  p.slopes = slopes;
  p.sinks = sinks;
  p.out = static_cast<float*>(out);
  p.partial = scratch;
  p.max_blocks = max_blocks;
  p.num_heads = num_heads;
  p.num_kv_heads = num_kv_heads;
  p.page_size = page_size;
  p.num_pages = num_pages;
  p.window = window;
  p.keep_first = keep_first;
  p.num_tokens = num_tokens;
  p.num_seqs = num_seqs;
  p.chunks = chunks;
  p.skip_single = has_single;
  p.early_metadata = early_metadata;
  p.aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  p.scale = scale;
  p.softcap = softcap;
  const bool wide_keys = (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0, wide = wide_keys && (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0;
  const int share = num_heads / num_kv_heads;
  static PerDevice raised[4];
  int rc = shrike_raise_smem(raised[0], single_kernel, shared_floats<16>() * 4);
  if (rc == 0) rc = shrike_raise_smem(raised[1], portions_kernel<16>, shared_floats<16>() * 4);
  if (rc == 0) rc = shrike_raise_smem(raised[2], portions_kernel<32>, shared_floats<32>() * 4);
  if (rc == 0) rc = shrike_raise_smem(raised[3], portions_kernel<64>, shared_floats<64>() * 4);
  if (rc != 0) return rc;
  const bool places = static_cast<long long>(num_kv_heads) * ((share + 15) / 16) <= 65535;
  if (has_single && (!wide || !places || num_seqs > 65535)) has_single = 2;
  if (has_portions && (!wide || !places)) has_portions = 2;
  if (has_single == 2 || has_portions == 2) {
    const long long blocks = (static_cast<long long>(num_tokens) * num_heads + WARPS - 1) / WARPS;
    if (blocks > 0x7fffffffLL) return SHRIKE_BAD_ARGUMENT;
    const int which = has_portions != 2 ? 1 : (has_single == 1 ? 2 : 0);
    const cudaError_t err = launch_dependent(wide_keys ? warps_kernel<true> : warps_kernel<false>, dim3(static_cast<unsigned>(blocks)),
                                             dim3(WARPS * 32), 0, stream, p, which);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  if (has_portions == 1) {
    // 64 rows a CTA read a key from shared memory for 64 rows, 16 only for 16; but fewer of them live on an SM (two for heads of
    // 64, one for wider ones; of 16 rows three, two and one), and where they are few the device waits for the last tokens' CTAs,
    // which walk every key.  Measured, us with 16, 32 and 64 rows: 14 heads of 64 over 2: 100 tokens 12.8, 15.6, 22.6; 333 tokens
    // 43.5, 43.1, 54.1; 1,500 tokens 371, 285, 300; 28 heads of 128 over 4: 100 tokens 24.4, 23.3, 31.6; 400 tokens 131, 95.7,
    // 91.3; 1,500 tokens 1,402, 881, 771.  What is chosen is within 7% of the best at 17 to 1,500 tokens of five head layouts.
    const long long rows = static_cast<long long>(num_tokens) * share, sms = shrike_device().sm_count;
    const int a_cta = (rows + 63) / 64 * num_kv_heads >= 2 * sms ? 64 : ((rows + 31) / 32 * num_kv_heads * 5 >= 4 * sms ? 32 : 16);
    p.heads_per_cta = share < a_cta ? share : a_cta;
    p.head_groups = (share + p.heads_per_cta - 1) / p.heads_per_cta;
    const int a_tile = a_cta / p.heads_per_cta;
    const dim3 grid((num_tokens + a_tile - 1) / a_tile, num_kv_heads * p.head_groups);
    const cudaError_t err = a_cta == 64   ? launch_dependent(portions_kernel<64>, grid, dim3(THREADS), shared_floats<64>() * 4, stream, p)
                            : a_cta == 32 ? launch_dependent(portions_kernel<32>, grid, dim3(THREADS), shared_floats<32>() * 4, stream, p)
                                          : launch_dependent(portions_kernel<16>, grid, dim3(THREADS), shared_floats<16>() * 4, stream, p);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  if (has_single == 1) {
    p.heads_per_cta = share < 16 ? share : 16;
    p.head_groups = (share + p.heads_per_cta - 1) / p.heads_per_cta;
    cudaError_t err = launch_dependent(single_kernel, dim3(chunks, num_kv_heads * p.head_groups, num_seqs), dim3(THREADS),
                                       shared_floats<16>() * 4, stream, p);
    if (err == cudaSuccess && chunks > 1)
      err = launch_dependent(merge_kernel, dim3((num_seqs * num_heads + 3) / 4), dim3(128), 0, stream, p);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  return shrike_launch_status();
}
