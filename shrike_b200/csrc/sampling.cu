// Sampling: one block per row of float32 logits.
//
// temperature == 0: the largest logit, lowest index on ties
//   (shrike/engine/sampler.py:15-17).
// otherwise: p = softmax(logits / temperature) in float32 (sampler.py:21-22);
//   with top_p < 1 a token is kept while the probability mass strictly above it is
//   below top_p (sampler.py:24-28: the most probable token is always kept); one
//   token is then drawn from the kept ones in proportion to p.  The draw is the
//   Gumbel-max form of a categorical sample, token = argmax(logit / T + g_i), with
//   g_i = -log(-log(u_i)) and u_i a hash of (seed, i): the same seed gives the same
//   token whatever else is in the batch (the reference's torch.multinomial on the
//   global generator, sampler.py:29, does not have that property).
#include <cooperative_groups.h>

#include "common.cuh"

constexpr int SAMPLE_THREADS = 1024;

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xFF51AFD7ED558CCDull;
  x ^= x >> 33;
  x *= 0xC4CEB9FE1A85EC53ull;
  x ^= x >> 33;
  return x;
}
__device__ __forceinline__ float gumbel(unsigned long long seed, int index) {
  const unsigned long long word = mix64(seed + static_cast<unsigned long long>(index) * 0x9E3779B97F4A7C15ull);
  const float u = (static_cast<float>(word >> 40) + 0.5f) * (1.0f / 16777216.0f);
  return -logf(-logf(u));
}

struct Best {
  float value;
  int index;
};
__device__ __forceinline__ Best better(Best a, Best b) {
  if (b.value > a.value || (b.value == a.value && b.index < a.index)) return b;
  return a;
}
__device__ Best block_best(Best mine, Best* scratch /* 33 entries */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    Best other;
    other.value = __shfl_xor_sync(0xffffffffu, mine.value, offset);
    other.index = __shfl_xor_sync(0xffffffffu, mine.index, offset);
    mine = better(mine, other);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = mine;
  __syncthreads();
  if (warp == 0) {
    const int warps = (blockDim.x + 31) >> 5;
    Best w = lane < warps ? scratch[lane] : Best{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      Best other;
      other.value = __shfl_xor_sync(0xffffffffu, w.value, offset);
      other.index = __shfl_xor_sync(0xffffffffu, w.index, offset);
      w = better(w, other);
    }
    if (lane == 0) scratch[32] = w;
  }
  __syncthreads();
  return scratch[32];
}

// A row whose logits are all NaN has no winner (no comparison with NaN holds): it yields token
// 0, a valid id, and leaves ERR_NO_FINITE_LOGIT in the status word when the caller gave one.
constexpr int ERR_NO_FINITE_LOGIT = 31;
__device__ __forceinline__ int valid_token(int index, int vocab, int* status) {
  if (index >= 0 && index < vocab) return index;
  if (status != nullptr && *status == 0) *status = ERR_NO_FINITE_LOGIT;
  return 0;
}

// Stage 1: the vocabulary of every row is cut into `chunks` slices; each block finds the
// best (score, index) of its slice, the score being the logit (greedy) or
// logit / T + Gumbel noise (sampled without top_p).  Rows with top_p < 1 are left to
// stage 2, which needs the whole row's probabilities.
constexpr int SLICE_THREADS = 256;
__global__ void __launch_bounds__(SLICE_THREADS)
sample_slices_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
                     const float* __restrict__ top_p, const long long* __restrict__ seeds,
                     float* __restrict__ partial_value, int* __restrict__ partial_index, int vocab, int chunks) {
  __shared__ Best best_scratch[33];
  let_dependents_start();
  wait_for_previous();
  const int row = blockIdx.y, chunk = blockIdx.x;
  const float temp = temperature[row];
  if (temp != 0.f && top_p[row] < 1.0f) return;
  const int per = (vocab + chunks - 1) / chunks;
  const int begin = chunk * per, end = min(vocab, begin + per);
  const float* x = logits + static_cast<size_t>(row) * vocab;
  Best mine{-INFINITY, 0x7fffffff};
  if (temp == 0.f) {
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) mine = better(mine, Best{x[i], i});
  } else {
    const float inv_temp = 1.0f / temp;
    const unsigned long long seed = static_cast<unsigned long long>(seeds[row]);
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x)
      mine = better(mine, Best{x[i] * inv_temp + gumbel(seed, i), i});
  }
  const Best top = block_best(mine, best_scratch);
  if (threadIdx.x == 0) {
    partial_value[static_cast<size_t>(row) * chunks + chunk] = top.value;
    partial_index[static_cast<size_t>(row) * chunks + chunk] = top.index;
  }
}

// Stage 2 for vocabularies whose rows do not fit a cluster's shared memory (above some 400,000 tokens), and for small ones, whose
// rows are quickly read: one block per row, the row read at every step of the bisection.
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
              const float* __restrict__ top_p, const long long* __restrict__ seeds, int* __restrict__ out,
              const float* __restrict__ partial_value, const int* __restrict__ partial_index, int vocab,
              int chunks, int* __restrict__ status) {
  __shared__ float scratch[33];
  __shared__ Best best_scratch[33];
  let_dependents_start();
  wait_for_previous();
  const int row = blockIdx.x;
  const float* x = logits + static_cast<size_t>(row) * vocab;
  const float temp = temperature[row];
  const float nucleus = top_p[row];

  if (temp == 0.f || nucleus >= 1.0f) {
    Best mine{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < chunks; i += blockDim.x)
      mine = better(mine, Best{partial_value[static_cast<size_t>(row) * chunks + i],
                               partial_index[static_cast<size_t>(row) * chunks + i]});
    const Best top = block_best(mine, best_scratch);
    if (threadIdx.x == 0) out[row] = valid_token(top.index, vocab, status);
    return;
  }

  const float inv_temp = 1.0f / temp;
  float local_max = -INFINITY;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) local_max = fmaxf(local_max, x[i]);
  const float row_max = block_max(local_max, scratch);
  float local_sum = 0.f;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) local_sum += expf((x[i] - row_max) * inv_temp);
  const float total = block_sum(local_sum, scratch);
  const float inv_total = 1.0f / total;
  // Bisection on the bit pattern of a positive float: mass_above(lo) >= top_p and
  // mass_above(hi) < top_p hold throughout; at the end no probability lies
  // strictly between lo and hi, and the kept set is {p > lo}.
  unsigned lo = 0u, hi = __float_as_uint(1.0f);  // mass_above(0) = 1 >= top_p; mass_above(1) = 0
  while (hi - lo > 1u) {
    const unsigned mid = lo + (hi - lo) / 2u;
    const float cut = __uint_as_float(mid);
    float above = 0.f;
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
      const float p = expf((x[i] - row_max) * inv_temp) * inv_total;
      if (p > cut) above += p;
    }
    above = block_sum(above, scratch);
    if (above < nucleus) hi = mid;
    else lo = mid;
  }
  const float threshold = lo == 0u ? -1.f : __uint_as_float(lo);
  Best mine{-INFINITY, 0x7fffffff};
  const unsigned long long seed = static_cast<unsigned long long>(seeds[row]);
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const float p = expf((x[i] - row_max) * inv_temp) * inv_total;
    if (p > threshold) mine = better(mine, Best{x[i] * inv_temp + gumbel(seed, i), i});
  }
  const Best top = block_best(mine, best_scratch);
  if (threadIdx.x == 0) out[row] = valid_token(top.index, vocab, status);
}

// Stage 2: a cluster of eight CTAs per row.  Rows handled by stage 1 only pick the best slice result (the first CTA
// does); rows with top_p < 1 run the whole nucleus procedure here.
//
// The procedure is a bisection of some thirty steps, each a sum over the row, so the row's probabilities stay in the
// cluster's shared memory, and two steps cost a scan of a thread's own entries and one cluster barrier.  An entry at or below
// the bisection's lower end can never count again and is dropped from its thread's list, in place, now and then.  The sums are those of one block of 1,024 threads that walk the row with a
// stride of 1,024, to the bit: thread t of CTA r is that block's thread 128 r + t, dropped entries add nothing, and the 32
// warps' sums meet in one warp in the same order.
// HELP threads share what a place's entries cost one by one (copies, exponentials, the draw's noise), one or two.  Where two
// CTAs fill an SM's shared memory, or rows are few, the time is that of their few warps, and two threads pay; where an SM holds
// many CTAs the second thread only takes another CTA's place.  Measured (one B200, top_p 0.95), us with one and two threads a
// place: 64 rows of 152,064 logits 177 and 148, one row 72 and 58; 64 rows of 5,000 39 and 46, 128 rows of 12,000 58 and 89; and
// 1,391 for the first with a block a row that reads the row from memory thirty times.  Four threads: 191 where two took 180.
constexpr int ROW_CTAS = 8, ROW_THREADS = SAMPLE_THREADS / ROW_CTAS;

struct RowShare {
  float warps[2][4][32];   // up to four values per warp of the cluster, two buffers: one barrier a sum
  Best best[ROW_CTAS];
};

// Every HELP-th of the row's entries x[0], x[SAMPLE_THREADS], ... that belong to a place, from the `which`-th on, into
// shared memory.  All copies are under way together: read through registers, eight at a time and eight warps an SM, a row
// came at a sixth of the memory's rate.
template <int HELP>
__device__ __forceinline__ void fetch_entries(float* place, const float* x, int which, int count) {
  const unsigned to = static_cast<unsigned>(__cvta_generic_to_shared(place));
#pragma unroll 4
  for (int j = which; j < count; j += HELP)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + j * static_cast<unsigned>(ROW_THREADS * sizeof(float))),
                 "l"(x + static_cast<size_t>(j) * SAMPLE_THREADS) : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ void row_publish(float4 mine, RowShare& share, int buffer, cooperative_groups::cluster_group& cluster) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane < ROW_CTAS && warp < ROW_THREADS / 32) {
    RowShare* to = cluster.map_shared_rank(&share, lane);
    const int at = cluster.block_rank() * (ROW_THREADS / 32) + warp;
    to->warps[buffer][0][at] = mine.x;
    to->warps[buffer][1][at] = mine.y;
    to->warps[buffer][2][at] = mine.z;
    to->warps[buffer][3][at] = mine.w;
  }
  cluster.sync();
}

template <int HELP>
__global__ void __launch_bounds__(ROW_THREADS * HELP)
sample_cluster_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
                      const float* __restrict__ top_p, const long long* __restrict__ seeds, int* __restrict__ out,
                      const float* __restrict__ partial_value, const int* __restrict__ partial_index, int vocab,
                      int chunks, int* __restrict__ status) {
  extern __shared__ float held[];   // [entries of a thread][ROW_THREADS]
  __shared__ RowShare share;
  __shared__ Best best_scratch[33];
  let_dependents_start();
  wait_for_previous();
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int row = blockIdx.x / ROW_CTAS, rank = blockIdx.x % ROW_CTAS, lane = threadIdx.x & 31;
  const float temp = temperature[row];
  const float nucleus = top_p[row];
  if (temp == 0.f || nucleus >= 1.0f) {
    if (rank != 0) return;
    Best mine{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < chunks; i += ROW_THREADS * HELP)
      mine = better(mine, Best{partial_value[static_cast<size_t>(row) * chunks + i],
                               partial_index[static_cast<size_t>(row) * chunks + i]});
    const Best top = block_best(mine, best_scratch);
    if (threadIdx.x == 0) out[row] = valid_token(top.index, vocab, status);
    return;
  }
  cluster.sync();   // every CTA of the cluster runs: its shared memory may be written from the others
  const float* x = logits + static_cast<size_t>(row) * vocab;
  // A place's entries are shared out among HELP threads wherever each stands for itself; what is added up in order, and the
  // list of the bisection, is the first's alone (the others go along with a list of none).
  const int place = threadIdx.x % ROW_THREADS, which = threadIdx.x / ROW_THREADS;
  float* own = held + place;
  const int first = rank * ROW_THREADS + place;
  const int all = first < vocab ? (vocab - first + SAMPLE_THREADS - 1) / SAMPLE_THREADS : 0;
  int count = which == 0 ? all : 0;
  const float inv_temp = 1.0f / temp;
  float local_max = -INFINITY;
  fetch_entries<HELP>(own, x + first, which, all);
  __syncthreads();
#pragma unroll 8
  for (int j = 0; j < count; ++j) local_max = fmaxf(local_max, own[j * ROW_THREADS]);
  row_publish(make_float4(warp_max(local_max), 0.f, 0.f, 0.f), share, 0, cluster);
  const float row_max = warp_max(share.warps[0][0][lane]);
#pragma unroll 4
  for (int j = which; j < all; j += HELP) own[j * ROW_THREADS] = expf((own[j * ROW_THREADS] - row_max) * inv_temp);
  __syncthreads();
  float local_sum = 0.f;
#pragma unroll 8
  for (int j = 0; j < count; ++j) local_sum += own[j * ROW_THREADS];
  row_publish(make_float4(warp_sum(local_sum), 0.f, 0.f, 0.f), share, 1, cluster);
  const float total = warp_sum(share.warps[1][0][lane]);
  const float inv_total = 1.0f / total;
#pragma unroll 4
  for (int j = which; j < all; j += HELP) own[j * ROW_THREADS] *= inv_total;
  __syncthreads();
  // Bisection on the bit pattern of a positive float: mass_above(lo) >= top_p and
  // mass_above(hi) < top_p hold throughout; at the end no probability lies
  // strictly between lo and hi, and the kept set is {p > lo}.
  unsigned lo = 0u, hi = __float_as_uint(1.0f);  // mass_above(0) = 1 >= top_p; mass_above(1) = 0
  // Two levels of it a pass: the middle and the middles of both halves, a sum each.
  int buffer = 0, passes = 0;
  while (hi - lo > 1u) {
    const unsigned mid = lo + (hi - lo) / 2u, low = lo + (mid - lo) / 2u, high = mid + (hi - mid) / 2u;
    const float cut = __uint_as_float(mid), cut_low = __uint_as_float(low), cut_high = __uint_as_float(high);
    const float floor = __uint_as_float(lo), ceiling = __uint_as_float(hi);
    float above = 0.f, above_low = 0.f, above_high = 0.f;
    bool between = false;
#pragma unroll 8
    for (int j = 0; j < count; ++j) {
      const float p = own[j * ROW_THREADS];
      if (p > cut_low) above_low += p;
      if (p > cut) above += p;
      if (p > cut_high) above_high += p;
      between = between || (p > floor && p < ceiling);
    }
    above = warp_sum(above), above_low = warp_sum(above_low), above_high = warp_sum(above_high);
    row_publish(make_float4(above, above_low, above_high, __any_sync(0xffffffffu, between) ? 1.f : 0.f), share, buffer, cluster);
    const bool upper = !(warp_sum(share.warps[buffer][0][lane]) < nucleus);
    // No probability lies strictly between the ends: every later middle has this one's mass above it, and the search would
    // end just below `hi` or at `lo` (a `lo` of zero is no threshold: it keeps the tokens of probability zero too).
    if (warp_max(share.warps[buffer][3][lane]) == 0.f) {
      if (upper) lo = hi - 1u;
      break;
    }
    const bool again = !(warp_sum(share.warps[buffer][upper ? 2 : 1][lane]) < nucleus);
    buffer ^= 1;
    if (upper) lo = mid;
    else hi = mid;
    if (hi - lo > 1u) {
      if (again) lo = upper ? high : low;
      else hi = upper ? high : low;
    }
    if ((++passes & 3) == 3) {   // drop what cannot count any more; eight entries are read before the first is written
      const float drop = __uint_as_float(lo);
      int kept = 0;
      for (int j = 0; j < count; j += 8) {
        float p[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e] = j + e < count ? own[(j + e) * ROW_THREADS] : 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (p[e] > drop) own[kept++ * ROW_THREADS] = p[e];
      }
      count = kept;
    }
  }
  const float threshold = lo == 0u ? -1.f : __uint_as_float(lo);
  Best mine{-INFINITY, 0x7fffffff};
  const unsigned long long seed = static_cast<unsigned long long>(seeds[row]);
  __syncthreads();   // the logits once more, over what the bisection left of their probabilities
  fetch_entries<HELP>(own, x + first, which, all);
#pragma unroll 4
  for (int j = which; j < all; j += HELP) {
    const int i = first + j * SAMPLE_THREADS;
    const float v = own[j * ROW_THREADS], p = expf((v - row_max) * inv_temp) * inv_total;
    if (p > threshold) mine = better(mine, Best{v * inv_temp + gumbel(seed, i), i});
  }
  const Best top = block_best(mine, best_scratch);
  if (threadIdx.x == 0) cluster.map_shared_rank(&share, 0)->best[rank] = top;
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    Best winner = share.best[0];
    for (int r = 1; r < ROW_CTAS; ++r) winner = better(winner, share.best[r]);
    out[row] = valid_token(winner.index, vocab, status);
  }
}

// How many slices stage 1 cuts a row into; scratch must hold rows * slices floats and ints.
SHRIKE_API int shrike_sample_slices(int vocab) {
  const int slices = (vocab + 2047) / 2048;
  return slices < 1 ? 1 : (slices > 128 ? 128 : slices);
}

namespace {
// Both stages.
int launch_sample(const float* logits, const float* temperature, const float* top_p, const long long* seeds, int* out,
                  float* scratch_value, int* scratch_index, int rows, int vocab, int chunks, int* status, cudaStream_t stream) {
  cudaError_t err = launch_dependent(sample_slices_kernel, dim3(chunks, rows), SLICE_THREADS, 0, stream, logits, temperature, top_p,
                                     seeds, scratch_value, scratch_index, vocab, chunks);
  if (err != cudaSuccess) return static_cast<int>(err);
  const size_t smem = static_cast<size_t>((vocab + SAMPLE_THREADS - 1) / SAMPLE_THREADS) * ROW_THREADS * sizeof(float);
  constexpr size_t MOST = 200 * 1024;
  // The cluster form costs 0.3 us a cluster to start, whatever a row holds; a block a row costs a scan of the row at every step of
  // the bisection.  Measured, us with clusters and with blocks: 1,000 tokens 20 and 19 (1 row), 37 and 23 (64), 96 and 29 (256);
  // 2,000 tokens 22 and 23 (8), 30 and 23 (32); 5,000 tokens 39 and 52 (64), 53 and 57 (128), 103 and 59 (256); 12,000 tokens 107
  // and 112 (256), 206 and 217 (512); 152,000 tokens 148 and 1,117 (64).  Both give the same tokens.
  const bool clusters = vocab >= 12000 || (vocab >= 4096 && rows <= 128) || (vocab >= 1536 && rows <= 8);
  if (clusters && smem <= MOST) {
    auto launch = [&](auto kernel, int help, PerDevice& raised) {
      const int rc = shrike_raise_smem(raised, kernel, MOST);
      if (rc != 0) return static_cast<cudaError_t>(rc);
      return launch_dependent_clusters(kernel, dim3(rows * ROW_CTAS), dim3(ROW_THREADS * help), smem, stream, ROW_CTAS, logits, temperature,
                                       top_p, seeds, out, static_cast<const float*>(scratch_value),
                                       static_cast<const int*>(scratch_index), vocab, chunks, status);
    };
    // Two threads a place (above) for few rows, or for rows that leave an SM few CTAs.  Measured, us with one and two: 4,096 tokens
    // 24 and 25 (16 rows), 51 and 79 (128); 8,000 25 and 24 (12), 39 and 46 (64); 20,000 30 and 28 (12), 38 and 41 (24), 61 and 85
    // (128); 32,000 49 and 40 (24), 70 and 64 (64), 72 and 93 (128); 64,000 68 and 68 (64), 160 and 171 (192); 100,000 90 and 91
    // (64), 321 and 311 (256).
    const bool pairs = vocab >= 90000 || (vocab >= 30000 && rows <= 64) || (vocab >= 6000 && rows <= 12);
    static PerDevice raised_alone, raised_pairs;
    err = pairs ? launch(sample_cluster_kernel<2>, 2, raised_pairs) : launch(sample_cluster_kernel<1>, 1, raised_alone);
  } else {
    err = launch_dependent(sample_kernel, rows, SAMPLE_THREADS, 0, stream, logits, temperature, top_p, seeds, out,
                           static_cast<const float*>(scratch_value), static_cast<const int*>(scratch_index), vocab, chunks, status);
  }
  return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
}
}  // namespace

SHRIKE_API int shrike_sample(const float* logits, const float* temperature, const float* top_p,
                             const long long* seeds, int* out, float* scratch_value, int* scratch_index,
                             int rows, int vocab, int* status, cudaStream_t stream) {
  if (rows <= 0) return SHRIKE_OK;
  if (vocab <= 0 || rows > 65535 || scratch_value == nullptr || scratch_index == nullptr) return SHRIKE_BAD_ARGUMENT;
  const int chunks = shrike_sample_slices(vocab);
  return launch_sample(logits, temperature, top_p, seeds, out, scratch_value, scratch_index, rows, vocab, chunks, status, stream);
}

// ------------------------------------------------------------------------------------
// The same two kernels with their scratch in a fixed device array, for callers that
// must not allocate (sampling_no_alloc.h says who they are and what the limits are).
#include <mutex>

#include "sampling_no_alloc.h"

static __device__ __align__(256) unsigned char sample_no_alloc_scratch[SHRIKE_SAMPLE_NO_ALLOC_BYTES];

namespace {
constexpr int NO_ALLOC_MAX_DEVICES = 64;
std::mutex no_alloc_mutex;
void* no_alloc_address[NO_ALLOC_MAX_DEVICES] = {};

// In host code `sample_no_alloc_scratch` is only a handle for the symbol, not an address a
// kernel can use; the device address is asked for once per device, with that device current.
int no_alloc_scratch(void** address) {
  int device = -1;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return static_cast<int>(err);
  if (device < 0 || device >= NO_ALLOC_MAX_DEVICES) return SHRIKE_SAMPLE_NO_ALLOC_BAD_DEVICE;
  std::lock_guard<std::mutex> guard(no_alloc_mutex);
  if (no_alloc_address[device] == nullptr) {
    void* found = nullptr;
    err = cudaGetSymbolAddress(&found, sample_no_alloc_scratch);
    if (err != cudaSuccess) return static_cast<int>(err);
    no_alloc_address[device] = found;
  }
  *address = no_alloc_address[device];
  return SHRIKE_OK;
}
}  // namespace

SHRIKE_API int shrike_sample_no_alloc(const float* logits, const float* temperature, const float* top_p,
                                      const long long* seeds, int* out, int rows, int vocab,
                                      cudaStream_t stream) {
  if (rows <= 0) return SHRIKE_OK;
  if (vocab <= 0) return SHRIKE_BAD_ARGUMENT;
  if (rows > SHRIKE_SAMPLE_NO_ALLOC_MAX_ROWS) return SHRIKE_SAMPLE_NO_ALLOC_TOO_MANY_ROWS;
  const int chunks = shrike_sample_slices(vocab);  // never more than SHRIKE_SAMPLE_NO_ALLOC_MAX_SLICES
  void* base = nullptr;
  const int status = no_alloc_scratch(&base);
  if (status != SHRIKE_OK) return status;
  float* values = static_cast<float*>(base);
  int* indices = reinterpret_cast<int*>(static_cast<unsigned char*>(base) + SHRIKE_SAMPLE_NO_ALLOC_BYTES / 2);
  return launch_sample(logits, temperature, top_p, seeds, out, values, indices, rows, vocab, chunks, nullptr, stream);
}

SHRIKE_API const char* shrike_sample_no_alloc_message(int code) {
  if (code == SHRIKE_OK) return "ok";
  if (code == SHRIKE_SAMPLE_NO_ALLOC_TOO_MANY_ROWS)
    return "shrike_sample_no_alloc: more than 256 rows in one call; the fixed scratch array holds 256 "
           "(split the batch, or use shrike_sample with scratch of your own)";
  if (code == SHRIKE_BAD_ARGUMENT) return "shrike_sample_no_alloc: bad argument (vocab must be positive)";
  if (code == SHRIKE_SAMPLE_NO_ALLOC_BAD_DEVICE)
    return "shrike_sample_no_alloc: the current device's index is 64 or more; the library keeps the scratch "
           "address of devices 0 to 63 only";
  return cudaGetErrorString(static_cast<cudaError_t>(code));
}
