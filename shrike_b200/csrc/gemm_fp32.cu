// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), all float32 with float32 FMA on the CUDA
// cores: no TF32, no reduced-precision staging.  This is the matrix product of the
// true 32-bit path.
//
// Order of the sums.  K is cut into `segments` runs of `segment_length` (the last one shorter); every run is one
// chain of FMAs in ascending k from zero, and the runs are added in ascending order, then the bias.  Both numbers
// follow from N and K alone (shrike_gemm_fp32_segments), so a row's result does not depend on the batch it was in,
// whichever of the kernels below forms it.
//
//   few rows (M <= 16)   `rows_kernel`: bound by reading W once.  A warp owns ROWS rows of W and one run of K, a
//                        lane one row (and some of the tokens): its chain.  W and A arrive by TMA in boxes of 32
//                        elements in the 128-byte swizzle, in which neighbouring rows' 16-byte pieces fall into
//                        different banks.  A matrix with few rows has few chains, so it is cut into runs: the warps
//                        of a CTA share its rows and the runs meet in shared memory, or, where the consumer adds
//                        slices, they are CTAs of their own and leave as a stack.
//   more rows            `tile_kernel`: bound by the FMA pipe.  A CTA owns BM x 128 outputs, a thread TM x 8 of
//                        them; both operands stay K-major as TMA brings them, and a thread reads a
//                        column's worth of pieces, two rows' FMAs in one instruction.  Three stages, two CTAs an SM.
//                        Where the tiles alone would not fill the device the runs go to CTAs of their own and leave
//                        as a stack that the consumer, or `sum_runs_kernel`, adds in order.
//   small products       `plain_kernel`: 64 x 64 tiles, 16 of k at a time (also K not a multiple of four, and operands not aligned to
//                        16 bytes)
//
// Measured (one B200, the plain kernel's time first): 1.5B widths, 3 tokens: the products of a decode step 30.3 and 1.55 ms,
// the 17,920 x 1,536 matrix 20.1 us (5.5 TB/s) and the 1,536 x 8,960 one 15.3 (3.6 TB/s); 0.5B widths, 333 tokens: the
// products of a prompt 16.9 and 8.6 ms; 512 tokens against the 37,888 x 3,584 matrix 47.9 TFLOP/s of FMA.
#include "blackwell.cuh"

namespace fp32 {
using namespace bw;

enum : int { ERR_ROWS = 41, ERR_TILE_PRODUCER = 42, ERR_TILE = 43, ERR_DRAIN = 44 };

constexpr int BM = 64, BN = 64, BK = 16;   // the plain kernel's tile
constexpr int PLAIN_THREADS = 256;

// VEC: rows and operands lie on 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(PLAIN_THREADS)
plain_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
             float* __restrict__ C, int M, int N, int K, int segment_length) {
  __shared__ __align__(16) float a_tile[BK][BM + 4];
  __shared__ __align__(16) float w_tile[BK][BN + 4];
  let_dependents_start();
  wait_for_previous();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int load_row = tid >> 2, load_k = (tid & 3) * 4;
  const int ty = tid >> 4, tx = tid & 15;
  const int am = m0 + load_row, wn = n0 + load_row;
  float acc[4][4], total[4][4];
  for (int begin = 0; begin < K; begin += segment_length) {   // a run: a multiple of BK
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const int end = min(K, begin + segment_length);
    for (int k0 = begin; k0 < end; k0 += BK) {
      float a_reg[4] = {0.f, 0.f, 0.f, 0.f}, w_reg[4] = {0.f, 0.f, 0.f, 0.f};
      const int k = k0 + load_k;
      if (am < M) {
        const float* src = A + static_cast<size_t>(am) * K + k;
        if (VEC) {
          if (k < K) load4<float>(src, a_reg);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) if (k + i < K) a_reg[i] = src[i];
        }
      }
      if (wn < N) {
        const float* src = W + static_cast<size_t>(wn) * K + k;
        if (VEC) {
          if (k < K) load4<float>(src, w_reg);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) if (k + i < K) w_reg[i] = __ldg(src + i);
        }
      }
      __syncthreads();  // the previous tile has been consumed
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a_tile[load_k + i][load_row] = a_reg[i];
        w_tile[load_k + i][load_row] = w_reg[i];
      }
      __syncthreads();
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        const float4 a = *reinterpret_cast<const float4*>(&a_tile[kk][ty * 4]);
        const float4 w = *reinterpret_cast<const float4*>(&w_tile[kk][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) total[i][j] = begin == 0 ? acc[i][j] : total[i][j] + acc[i][j];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[static_cast<size_t>(m) * N + n] = bias ? total[i][j] + bias[n] : total[i][j];
    }
  }
}

// The runs of a stack added up in order, then the bias: what the kernels above leave when they add the runs themselves.
template <int VEC>
__global__ void __launch_bounds__(256) sum_runs_kernel(const float* __restrict__ runs, int count, const float* __restrict__ bias, float* __restrict__ C,
                                                       long long total, int N) {
  let_dependents_start();
  wait_for_previous();
  const long long at = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * VEC;
  if (at >= total) return;
  float v[VEC];
  if constexpr (VEC == 4) sum_partials4(runs + at, total, count, v);
  else v[0] = sum_partials(runs + at, total, count);
  if (bias != nullptr) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) v[e] += bias[(at + e) % N];
  }
  if constexpr (VEC == 4) store4<float>(C + at, v);
  else C[at] = v[0];
}

// Tiles want 1024-byte alignment: the swizzle pattern repeats every 1024 bytes.
__device__ __forceinline__ unsigned char* aligned_tiles(unsigned char* raw) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
}
__device__ __forceinline__ float4 tile_read(const unsigned char* row, int piece, int swizzle) {
  return *reinterpret_cast<const float4*>(row + ((piece ^ swizzle) << 4));
}

constexpr int ROWS_MAX_STAGES = 8;
template <int S> struct RowsWarps { static constexpr int value = S > 1 ? S : 2; };   // warps of a CTA: a run of K each, or two row groups

// Few tokens.  A warp takes ROWS * RPL rows of W, a lane RPL of them; MT: tokens, rounded up to a power of two; S: runs of
// K (at most), one a warp; S = 1: one run, the blockIdx.y-th, whose sums leave as that slice of the stack.  What a lane reads of A is the same for every row, and shared memory hands a warp 128 bytes a
// clock however many lanes share them: two or four rows a lane keep those reads below the rate at which W arrives.
template <int ROWS, int RPL, int MT, int S>
__global__ void __launch_bounds__(32 * RowsWarps<S>::value)
rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const float* __restrict__ bias,
            float* __restrict__ C, int M, int N, int K, int segment_length, int stages, int* status) {
  constexpr int WARPS = RowsWarps<S>::value, PER_WARP = ROWS * RPL;
  constexpr int GROUPS = 32 / ROWS;                       // lanes that share a row, each with its own tokens
  constexpr int OWN = MT > GROUPS ? MT / GROUPS : 1;      // tokens of a lane: group + GROUPS * i
  constexpr int W_BYTES = PER_WARP * 128, A_SLOT = MT > 8 ? MT * 128 : 1024, STAGE = W_BYTES + A_SLOT;
  extern __shared__ unsigned char raw[];
  __shared__ unsigned long long full[WARPS][ROWS_MAX_STAGES];
  __shared__ volatile int abort_flag;
  unsigned char* tiles = aligned_tiles(raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int w = 0; w < WARPS; ++w)
      for (int s = 0; s < stages; ++s) mbar_init(&full[w][s], 1);
    abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();
  let_dependents_start();
  const int segment = S > 1 ? warp : blockIdx.y, n0 = (S > 1 ? blockIdx.x : blockIdx.x * WARPS + warp) * PER_WARP;
  const int k_begin = segment * segment_length, k_end = min(K, k_begin + segment_length);
  const int steps = n0 < N && k_end > k_begin ? (k_end - k_begin + 31) / 32 : 0;
  unsigned char* mine = tiles + static_cast<size_t>(warp) * stages * STAGE;
  // neighbouring lanes hand their copies to the engine together: one thread that issues them one after another keeps a short
  // run waiting for its last ones (2,048 x 1,536 and 1,536 x 1,536, 3 tokens: 6.7 us a product, 4.9 together)
  int issued = min(steps, stages);
  if (lane < issued) {   // W is written by nobody: it is on its way before the kernel before this one ends
    mbar_expect_tx(&full[warp][lane], W_BYTES + MT * 128);
    tma_load_2d(mine + lane * STAGE, &map_w, &full[warp][lane], k_begin + lane * 32, n0);
  }
  wait_for_previous();
  if (lane < issued) tma_load_2d(mine + lane * STAGE + W_BYTES, &map_a, &full[warp][lane], k_begin + lane * 32, 0);
  __syncwarp();
  const int row = lane % ROWS, group = lane / ROWS;
  float acc[RPL][OWN];
#pragma unroll
  for (int r = 0; r < RPL; ++r)
#pragma unroll
    for (int i = 0; i < OWN; ++i) acc[r][i] = 0.f;
  int stage = 0;
  unsigned phase = 0;
  for (int step = 0; step < steps; ++step) {
    if (!__all_sync(0xffffffffu, mbar_wait(&full[warp][stage], phase, &abort_flag, status, ERR_ROWS))) break;
    const unsigned char* w_row = mine + stage * STAGE + row * 128;
    const unsigned char* a_tile = mine + stage * STAGE + W_BYTES;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      float4 w[RPL];
#pragma unroll
      for (int r = 0; r < RPL; ++r) w[r] = tile_read(w_row + r * (ROWS * 128), c, row & 7);
#pragma unroll
      for (int i = 0; i < OWN; ++i) {
        const int m = MT >= GROUPS ? group + GROUPS * i : group % MT;
        const float4 a = tile_read(a_tile + m * 128, c, m & 7);
#pragma unroll
        for (int r = 0; r < RPL; ++r) {
          acc[r][i] = fmaf(a.x, w[r].x, acc[r][i]);
          acc[r][i] = fmaf(a.y, w[r].y, acc[r][i]);
          acc[r][i] = fmaf(a.z, w[r].z, acc[r][i]);
          acc[r][i] = fmaf(a.w, w[r].w, acc[r][i]);
        }
      }
    }
    __syncwarp();   // every lane has read the stage
    if (step + stages < steps) {
      if (lane == 0) mbar_expect_tx(&full[warp][stage], W_BYTES + MT * 128);
      __syncwarp();
      if (lane < 2)
        tma_load_2d(mine + stage * STAGE + (lane == 0 ? 0 : W_BYTES), lane == 0 ? &map_w : &map_a, &full[warp][stage],
                    k_begin + (step + stages) * 32, lane == 0 ? n0 : 0);
      issued = step + stages + 1;
    }
    if (++stage == stages) { stage = 0; phase ^= 1; }
  }
  if (lane == 0 && abort_flag) {   // copies may still be in flight: wait for the stages armed last before leaving
    for (int i = max(0, issued - stages); i < issued; ++i) {
      bool landed = false;
      for (unsigned tries = 0; tries < WAIT_LIMIT && !landed; ++tries) landed = mbar_try_wait(&full[warp][i % stages], (i / stages) & 1);
      if (!landed && status != nullptr) *status = ERR_DRAIN;
    }
  }
  if (S == 1) {
    C += static_cast<size_t>(segment) * M * N;
#pragma unroll
    for (int r = 0; r < RPL; ++r) {
      const int n = n0 + row + ROWS * r;
#pragma unroll
      for (int i = 0; i < OWN; ++i) {
        const int m = group + GROUPS * i;
        if (m < MT && m < M && n < N) C[static_cast<size_t>(m) * N + n] = bias ? acc[r][i] + bias[n] : acc[r][i];
      }
    }
    return;
  }
  float* part = reinterpret_cast<float*>(tiles);   // [S][MT][PER_WARP], once every warp has read its last stage
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RPL; ++r)
#pragma unroll
    for (int i = 0; i < OWN; ++i) {
      const int m = group + GROUPS * i;
      if (m < MT) part[(warp * MT + m) * PER_WARP + row + ROWS * r] = acc[r][i];
    }
  __syncthreads();
  const int runs = (K + segment_length - 1) / segment_length;
  for (int at = threadIdx.x; at < MT * PER_WARP; at += 32 * WARPS) {
    const int r = at % PER_WARP, m = at / PER_WARP, n = n0 + r;
    if (m >= M || n >= N) continue;
    float sum = part[m * PER_WARP + r];
    for (int s = 1; s < runs; ++s) sum += part[(s * MT + m) * PER_WARP + r];
    C[static_cast<size_t>(m) * N + n] = bias ? sum + bias[n] : sum;
  }
}

constexpr int TILE_N = 128, TILE_THREADS = 128, TILE_STAGES = 3;

// 8 TM rows of A by 128 of W.  blockIdx.z: the run of K when the runs leave as a stack (gridDim.z > 1), else all
// runs one after another, each added to what the earlier ones left in C.
template <int TM>
__global__ void __launch_bounds__(TILE_THREADS, 2)
tile_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ bias,
            float* __restrict__ C, int M, int N, int K, int segment_length, int* status) {
  constexpr int TILE_M = 8 * TM, A_BYTES = TILE_M * 128, STAGE = A_BYTES + TILE_N * 128;
  extern __shared__ unsigned char raw[];
  __shared__ unsigned long long full[TILE_STAGES], empty[TILE_STAGES];
  __shared__ volatile int abort_flag;
  unsigned char* tiles = aligned_tiles(raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * TILE_M, n0 = blockIdx.x * TILE_N;
  const int k_begin = gridDim.z > 1 ? blockIdx.z * segment_length : 0;
  const int k_end = gridDim.z > 1 ? min(K, k_begin + segment_length) : K;
  const int steps = (k_end - k_begin + 31) / 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < TILE_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], TILE_THREADS / 32);
    }
    abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();
  let_dependents_start();
  wait_for_previous();
  auto load = [&](int step) {
    unsigned char* to = tiles + (step % TILE_STAGES) * STAGE;
    unsigned long long* bar = &full[step % TILE_STAGES];
    mbar_expect_tx(bar, STAGE);
    tma_load_2d(to, &map_a, bar, k_begin + step * 32, m0);
    tma_load_2d(to + A_BYTES, &map_w, bar, k_begin + step * 32, n0);
  };
  int issued = min(steps, TILE_STAGES);
  if (threadIdx.x == 0)
    for (int i = 0; i < issued; ++i) load(i);
  // a thread's rows: m = m_first + 8 i, n = n_first + 16 j; the rows that lanes read side by side differ modulo eight
  const int m_first = (warp & 1) * 4 + (lane >> 3), n_first = (warp >> 1) * 8 + (lane & 7);
  float* out = C + static_cast<size_t>(blockIdx.z) * M * N;
  unsigned long long acc[TM / 2][8];   // rows i and i + 1 of the thread, side by side
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  const int steps_a_run = gridDim.z > 1 ? steps : segment_length / 32;
  int left = steps_a_run, stage = 0;
  unsigned phase = 0;
  bool first_run = true;
  for (int step = 0; step < steps; ++step) {
    bool ok = mbar_wait(&full[stage], phase, &abort_flag, status, ERR_TILE);
    if (ok && threadIdx.x == 0 && step > 0 && step - 1 + TILE_STAGES < steps) {   // the stage that every warp has left
      ok = mbar_wait(&empty[(step - 1) % TILE_STAGES], ((step - 1) / TILE_STAGES) & 1, &abort_flag, status, ERR_TILE_PRODUCER);
      if (ok) {
        load(step - 1 + TILE_STAGES);
        issued = step + TILE_STAGES;
      }
    }
    if (!__all_sync(0xffffffffu, ok)) break;
    const unsigned char* a_rows = tiles + stage * STAGE + m_first * 128;
    const unsigned char* w_rows = tiles + stage * STAGE + A_BYTES + n_first * 128;
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {
      // Two rows' FMAs in one instruction (the same roundings): single FMAs here lose a third of their issue slots to
      // register bank conflicts, and pairs leave issue slots for the reads.  Scalar reads put the pairs together.
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        unsigned long long w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float v = reinterpret_cast<const volatile float*>(w_rows + j * 2048 + ((c ^ (n_first & 7)) << 4))[e];
          asm("mov.b64 %0, {%1, %1};" : "=l"(w[j]) : "f"(v));
        }
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) {
          const unsigned char* a_row = a_rows + 2 * i * 1024 + ((c ^ (m_first & 7)) << 4);
          const float a0 = reinterpret_cast<const volatile float*>(a_row)[e], a1 = reinterpret_cast<const volatile float*>(a_row + 1024)[e];
          unsigned long long a;
          asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
#pragma unroll
          for (int j = 0; j < 8; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(a), "l"(w[j]));
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
    if (++stage == TILE_STAGES) { stage = 0; phase ^= 1; }
    const bool last = step + 1 == steps;
    if (--left == 0 || last) {   // a run ends: its chains are added to the earlier runs' sum
      left = steps_a_run;
      // a few of a thread's rows at a time: their earlier sums are all on their way before the first is needed
      constexpr int BATCH = TM % 4 == 0 ? 4 : 2;
#pragma unroll
      for (int i0 = 0; i0 < TM; i0 += BATCH) {
        float before[BATCH][8];
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = m0 + m_first + 8 * (i0 + i), n = n0 + n_first + 16 * j;
            before[i][j] = !first_run && m < M && n < N ? out[static_cast<size_t>(m) * N + n] : 0.f;
          }
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = m0 + m_first + 8 * (i0 + i), n = n0 + n_first + 16 * j;
            const unsigned long long both = acc[(i0 + i) / 2][j];
            const float mine = __uint_as_float(static_cast<unsigned>((i & 1) ? both >> 32 : both));
            if (m < M && n < N) {
              float sum = first_run ? mine : before[i][j] + mine;
              if (last && bias != nullptr) sum += bias[n];
              out[static_cast<size_t>(m) * N + n] = sum;
            }
          }
#pragma unroll
        for (int i = 0; i < BATCH / 2; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i0 / 2 + i][j] = 0ull;
      }
      first_run = false;
    }
  }
  if (threadIdx.x == 0 && abort_flag) {   // copies may still be in flight: wait for the stages armed last before leaving
    for (int i = max(0, issued - TILE_STAGES); i < issued; ++i) {
      bool landed = false;
      for (unsigned tries = 0; tries < WAIT_LIMIT && !landed; ++tries) landed = mbar_try_wait(&full[i % TILE_STAGES], (i / TILE_STAGES) & 1);
      if (!landed && status != nullptr) *status = ERR_DRAIN;
    }
  }
}

template <int ROWS, int RPL, int MT, int S>
int launch_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int segment_length, int stack, int* status,
                cudaStream_t stream) {
  constexpr int WARPS = RowsWarps<S>::value, STAGE = ROWS * RPL * 128 + (MT > 8 ? MT * 128 : 1024);
  constexpr int PER_CTA = ROWS * RPL * (S > 1 ? 1 : WARPS), MOST = 200 * 1024;
  const int tiles = (N + PER_CTA - 1) / PER_CTA, ctas = tiles * stack, sms = shrike_device().sm_count;
  // stages: the SM's shared memory shared among the CTAs that will live on it (at most four), two stages at least
  const int resident = ctas >= 4 * sms ? 4 : (ctas + sms - 1) / sms;
  int stages = MOST / (resident < 1 ? 1 : resident) / (WARPS * STAGE);
  const int steps = (segment_length < K ? segment_length : K) / 32 + 1;
  stages = stages < 2 ? 2 : (stages > ROWS_MAX_STAGES ? ROWS_MAX_STAGES : stages);
  if (stages > steps) stages = steps;
  const size_t smem = static_cast<size_t>(WARPS) * stages * STAGE + 1024;
  static_assert(WARPS * 2 * STAGE <= MOST, "two stages must fit");
  static_assert(S == 1 || S * MT * ROWS * RPL * 4 <= WARPS * STAGE, "the runs' partial sums lie in the first stages");
  static PerDevice raised;
  int rc = shrike_raise_smem(raised, rows_kernel<ROWS, RPL, MT, S>, MOST + 1024);
  if (rc != 0) return rc;
  CUtensorMap map_w, map_a;
  rc = tensor_map_f32(W, N, K, ROWS * RPL, &map_w);
  if (rc != SHRIKE_OK) return rc;
  rc = tensor_map_f32(A, M, K, MT, &map_a);
  if (rc != SHRIKE_OK) return rc;
  const cudaError_t err = launch_dependent(rows_kernel<ROWS, RPL, MT, S>, dim3(tiles, stack), dim3(32 * WARPS), smem, stream,
                                           map_w, map_a, bias, C, M, N, K, segment_length, stages, status);
  return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
}

// Rows a warp takes: as many as leave every SM two warps.  Fewer rows a warp read A from shared memory more often for
// the same W; fewer warps leave the chains' latency uncovered.
template <int MT, int S>
int rows_of_width(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int length, int stack, int* status,
                  cudaStream_t stream) {
  const long long wanted = 2LL * shrike_device().sm_count, chains = static_cast<long long>(N) * S * stack;
  if constexpr (S <= 4) {
    if constexpr (MT >= 8)
      if (chains >= 128 * wanted) return launch_rows<32, 4, MT, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
    if (chains >= 64 * wanted) return launch_rows<32, 2, MT, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  }
  if (chains >= 32 * wanted) return launch_rows<32, 1, MT, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  if constexpr (S <= 4)
    if (chains >= 16 * wanted) return launch_rows<16, 1, MT, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  return launch_rows<8, 1, MT, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
}

template <int S>
int rows_of_tokens(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int length, int stack, int* status,
                   cudaStream_t stream) {
  if (M <= 1) return rows_of_width<1, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  if (M <= 2) return rows_of_width<2, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  if (M <= 4) return rows_of_width<4, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  if (M <= 8) return rows_of_width<8, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
  return rows_of_width<16, S>(A, W, bias, C, M, N, K, length, stack, status, stream);
}

template <int TM>
int launch_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int length, int stack, int* status,
                 cudaStream_t stream) {
  constexpr int TILE_M = 8 * TM, STAGE = (TILE_M + TILE_N) * 128;
  constexpr size_t smem = static_cast<size_t>(TILE_STAGES) * STAGE + 1024;
  static PerDevice raised;
  int rc = shrike_raise_smem(raised, tile_kernel<TM>, smem);
  if (rc != 0) return rc;
  CUtensorMap map_w, map_a;
  rc = tensor_map_f32(W, N, K, TILE_N, &map_w);
  if (rc != SHRIKE_OK) return rc;
  rc = tensor_map_f32(A, M, K, TILE_M, &map_a);
  if (rc != SHRIKE_OK) return rc;
  const dim3 grid((N + TILE_N - 1) / TILE_N, (M + TILE_M - 1) / TILE_M, stack);
  if (grid.y > 65535) return SHRIKE_BAD_ARGUMENT;
  const cudaError_t err = launch_dependent(tile_kernel<TM>, grid, dim3(TILE_THREADS), smem, stream, map_a, map_w, bias, C, M, N, K,
                                           length, status);
  return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
}

// Elements of a run of K: a multiple of 32.  A matrix is cut into as many runs as give every SM of a B200 two warps of 64 rows when
// a few tokens are multiplied (the number of SMs is written out: it fixes the order of the sums, which is the matrix's alone; 1.5B
// widths, 3 tokens, the 1,536 x 8,960 matrix: 22.5 us with eight runs of 1,120, 15.3 with the sixteen of 576 that this gives); never
// shorter than a hundred elements or so, for every run of a prompt's product is one more addition to its result.
int segment_length(int n, int k) {
  const int most = k < 512 ? 1 : (k < 1024 ? 4 : (k < 8192 ? 8 : 16));
  int runs = 1;
  while (runs < most && static_cast<long long>(n) * runs < 64LL * 2 * 148) runs *= 2;
  return ((k + runs - 1) / runs + 31) / 32 * 32;
}

// Eighths of a tile's rows (TM) for a product of M rows and `stack` slices: what an SM's CTAs cost, rounds of as many as
// live on it (two by their registers; three of 32 rows by their shared memory), the last round at least the cost of two where it is
// the only one (a CTA alone hides nothing of its latencies) and of 1.25 behind others (its CTAs start as places fall free).
// Smaller tiles read more from shared memory an FMA.  The rows beyond M and the empty places of the last round are what the
// choice avoids.  Measured over 17 to 2,048 rows of ten matrices of 0.5B, 1.5B and 7B widths (183 products, every height
// each): 0.7% above the best height's time on average, 12% at worst (333 rows, 2,048 x 1,536 in one slice: 164 us with 32, 147
// with 48 rows a tile).  333 rows: the 896 x 4,864 matrix 84 us with the chosen 80 rows a tile, 112 to 136 with 32, 64, 112 or 128;
// 1,152 x 896: 28 with 32, 45 with 96.  96 rows are slower than both neighbours (1,024 rows, 9,728 x 896: 497 us, 435 with 80).
int tile_rows(int M, int N, int stack) {
  constexpr int sizes[] = {16, 14, 12, 10, 8, 4}, resident[] = {2, 2, 2, 2, 2, 3};
  constexpr float rate[] = {1.f, 1.f, 0.9f, 1.f, 0.95f, 0.75f};
  const long long sms = shrike_device().sm_count, columns = static_cast<long long>((N + TILE_N - 1) / TILE_N) * stack;
  int best = 16;
  float least = 0.f;
  for (int i = 0; i < 6; ++i) {
    const long long rows = (M + 8LL * sizes[i] - 1) / (8 * sizes[i]);
    if (i > 0 && rows > 65535) continue;   // more than a grid's y
    const long long ctas = columns * rows, places = sms * resident[i];
    const long long rounds = ctas / places, rest = ctas % places, an_sm = (rest + sms - 1) / sms;
    const float alone = rounds > 0 ? 1.25f : 2.f, last = rest == 0 ? 0.f : (an_sm > alone ? an_sm : alone);
    const float cost = (rounds * resident[i] + last) * sizes[i] / rate[i];
    if (i == 0 || cost < least) {
      least = cost;
      best = sizes[i];
    }
  }
  return best;
}

}  // namespace fp32

// Runs that K is cut into for a product with a [n, k] matrix, whatever the number of rows.
SHRIKE_API int shrike_gemm_fp32_segments(int n, int k) {
  if (n <= 0 || k <= 0) return 1;
  const int length = fp32::segment_length(n, k);
  return (k + length - 1) / length;
}

// Slices of the stack in which a product of m rows should leave when its consumer adds slices (1: a plain result).
// The runs get CTAs of their own where the 128 x 128 tiles alone would leave places empty (two CTAs an SM); with few rows
// always: a CTA that holds all runs of its rows leaves SMs without one when the matrix has few rows.
SHRIKE_API int shrike_gemm_fp32_stack(int m, int n, int k) {
  if (k % 4) return 1;
  if (m <= 16) return shrike_gemm_fp32_segments(n, k);
  const long long tiles = static_cast<long long>((n + fp32::TILE_N - 1) / fp32::TILE_N) * ((m + 127) / 128);
  return tiles < 2LL * shrike_device().sm_count ? shrike_gemm_fp32_segments(n, k) : 1;
}

// `stack` > 1 (as shrike_gemm_fp32_stack says, no bias): C is [stack][M][N], one slice a run of K, to be added in order.
// `tile` 0: the tile height that the rule above gives; n: 8 n rows.  `scratch` (float32 [runs][M][N], or null; for a plain result of more
// than 16 rows where shrike_gemm_fp32_stack says more than 1): the runs go there on CTAs of their own and are then added up.  Measured,
// us with the runs one after another in a CTA and with them side by side and a sum: 17 rows, 1,152 x 896: 57.6 and 16.4; 500 rows 80.3
// and 31.2; 300 rows, 9,728 x 896: 180 and 164; 300 rows, 1,536 x 8,960: 756 and 237; at worst 300 rows, 9,472 x 516: 80.6 and 83.6.
SHRIKE_API int shrike_gemm_fp32(const float* A, const float* W, const float* bias, float* C, int M, int N,
                                int K, int stack, int tile, float* scratch, int* status, cudaStream_t stream) {
  using namespace fp32;
  if (M <= 0 || N <= 0) return SHRIKE_OK;
  if (K <= 0 || stack < 1) return SHRIKE_BAD_ARGUMENT;
  const int length = segment_length(N, K), runs = (K + length - 1) / length;
  const bool aligned = (K % 4 == 0) && (reinterpret_cast<uintptr_t>(A) % 16 == 0) && (reinterpret_cast<uintptr_t>(W) % 16 == 0);
  if (stack > 1 && (stack != runs || bias != nullptr || !aligned)) return SHRIKE_BAD_ARGUMENT;
  if (!aligned) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return SHRIKE_BAD_ARGUMENT;
    const cudaError_t err = launch_dependent(plain_kernel<false>, grid, dim3(PLAIN_THREADS), 0, stream, A, W, bias, C, M, N, K, length);
    return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
  }
  if (M <= 16) {
    if (runs == 1 || stack > 1) return rows_of_tokens<1>(A, W, bias, C, M, N, K, length, stack, status, stream);
    if (runs <= 2) return rows_of_tokens<2>(A, W, bias, C, M, N, K, length, stack, status, stream);
    if (runs <= 4) return rows_of_tokens<4>(A, W, bias, C, M, N, K, length, stack, status, stream);
    if (runs > 8) return rows_of_tokens<16>(A, W, bias, C, M, N, K, length, stack, status, stream);
    return rows_of_tokens<8>(A, W, bias, C, M, N, K, length, stack, status, stream);
  }
  if (tile == 0 && runs == 1) {
    // A chain of FMAs that nothing hides runs quicker in the small tiles, as long as they are one round of CTAs (us with large and
    // with small tiles: 129 rows, 192 x 192: 13.3 and 11.2; 500 rows, 640 x 384 [80 small tiles]: 27.2 and 23.7; 1,000 rows [160]: 40.7 and
    // 40.5; 2,000 rows [320]: 45.9 and 57.5; 129 rows, 4,000 x 300 [189]: 35.7 and 35.0).
    const long long small = static_cast<long long>((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    if (small <= shrike_device().sm_count) {
      const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
      const cudaError_t err = launch_dependent(plain_kernel<true>, grid, dim3(PLAIN_THREADS), 0, stream, A, W, bias, C, M, N, K, length);
      return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
    }
  }
  if (scratch != nullptr && stack == 1 && runs > 1) {
    const int rc = shrike_gemm_fp32(A, W, nullptr, scratch, M, N, K, runs, tile, nullptr, status, stream);
    if (rc != SHRIKE_OK) return rc;
    const long long total = static_cast<long long>(M) * N;
    const bool vec = N % 4 == 0 && ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(scratch)) & 15) == 0;
    const long long blocks = ((vec ? total / 4 : total) + 255) / 256;
    if (blocks > 0x7fffffffLL) return SHRIKE_BAD_ARGUMENT;
    const cudaError_t err = launch_dependent(vec ? sum_runs_kernel<4> : sum_runs_kernel<1>, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream,
                                             static_cast<const float*>(scratch), runs, bias, C, total, N);
    return err == cudaSuccess ? shrike_launch_status() : static_cast<int>(err);
  }
  switch (tile > 0 ? tile : tile_rows(M, N, stack)) {
#define SHRIKE_TILE(TM) case TM: return launch_tiles<TM>(A, W, bias, C, M, N, K, length, stack, status, stream)
    SHRIKE_TILE(4);
    SHRIKE_TILE(8);
    SHRIKE_TILE(10);
    SHRIKE_TILE(12);
    SHRIKE_TILE(14);
    SHRIKE_TILE(16);
    default: return SHRIKE_BAD_ARGUMENT;
#undef SHRIKE_TILE
  }
}
