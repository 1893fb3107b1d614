// Every layer of a decode step for few sequences in one cooperative kernel (bfloat16, pre-norm layers of this package's
// attention and gated feed-forward: shrike/models/qwen.py:147-150).
//
// What bounds it.  Issued kernel by kernel, a layer of a small model is a chain of eight dependent launches at 3 to 5 us each,
// while its weights take 4.6 us (0.5B widths) to 14 us (1.5B) to stream: every kernel pays its start, the first trips
// to memory and the drain of its last CTA.  Here one CTA lives on every SM for the whole step.  A warp of its own streams the
// CTA's share of all weights, layer after layer, through a ring in shared memory and runs ahead of the arithmetic by the depth
// of that ring (it needs nothing but the layer table), so that HBM keeps busy while the other warps wait for one another.
//
// Measured (500 keys, us a step as separate launches and as one kernel, in turn): 0.5B widths 1 sequence 654 and 440, 4 sequences
// 670 and 533; 1.5B 1,058 and 773, 1,099 and 1,055; 3B 1,673 and 1,332; 7B 2,694 and 2,538.  A layer takes 14.8 us at 0.5B widths
// and 23.5 at 1.5B (12 against 24 layers, 14 against 28); one of 256 columns, which has next to no weights, 13.2: that is what the
// five exchanges, the norms and the attention take by themselves.
//
// A layer:  norm + q/k/v product | rotation, store, attention | output product + residual | norm + gate/up product +
// activation | down product + residual.  A product gives every CTA the same number of weight rows (the gated one units of 8 gate rows
// and the 8 up rows of the same features) over the whole of K: no sum crosses a CTA, so the residual is added and the activation
// applied where the product ends.  The eight warps of a CTA share the K steps of a ring stage (mma.sync m16n8k16: 16 weight rows by
// 8 sequences; the step is bound by bytes and by latency, and a warp-wide product takes any number of rows, where a tcgen05 tile
// wants 64 or 128 of them that few CTAs would then share) and add up in shared memory in a fixed order.  Each CTA norms the rows
// it reads by itself.
//
// How CTAs hand values on.  Every value that crosses CTAs travels as one 64-bit word with the number of the exchange beside it:
// a reader polls the very words it needs until they carry the number it expects.  That takes one trip to L2 to write
// and one to read, where stores, a fence, a counter, a poll and the loads took 1.5 us (fence and counter 0.7, poll 0.4, loads 0.4).
// The numbers grow with every layer and launch, so nothing is ever cleared.  A reader wants the very number it expects, so a
// word may be written again only when all its readers have it.  One buffer an exchange suffices, because every reader publishes
// something after it has read, and whoever writes the words again has read that, directly or through others:
//   residual, part 0  read by the CTAs with q/k/v rows; the output rows that replace it need all heads, those need all q/k/v rows.
//                     A CTA without such rows must not read it: nothing that waits for that CTA lies between the two.
//   q/k/v             read by the CTAs with a pair; the next layer's rows need all down rows, those all gated units, of which
//                     every CTA has one, and it comes to that behind its attention.
//   runs' sums        read by the CTAs with a pair, replaced by them behind the next q/k/v rows: as above.
//   heads             read by all CTAs in part 1; replaced behind the next q/k/v rows, which need every CTA's gated units.
//   residual, part 2  read by all CTAs; the down rows that replace it need all gated units.
//   activation        read by the CTAs with down rows; the next units need all output rows, those all heads, those the q/k/v rows,
//                     and each of those needs all down rows.
//
// Rounding points are those of the separate kernels: normed rows, rotated q and k, v, probabilities, attention output,
// gate, up and their product in bfloat16, all sums in float32.
//
// Attention: a CTA takes a (sequence, kv head) pair, or, where pairs are few, a run of its keys; the keys of earlier positions
// are brought to shared memory before q is there.  The runs of a pair exchange their sums, and each adds up a share of the
// pair's columns.
//
// Every layer walks once through the same code, so loops stay rolled, loads unconditional (a load under a condition is a branch of
// 30 clocks and more), and nothing spills: 220 KB of shared memory leave no L1 to hold local memory, 300 clocks an access.
//
// Every wait is bounded; one that runs out leaves its code in the status word, and the CTA runs through the rest of its
// schedule without waiting (no thread leaves the common path, so that no barrier is left short of an arrival).
#include "blackwell.cuh"

namespace step {
using namespace bw;
typedef unsigned long long Word;               // a value below, the exchange's number above

constexpr int WARPS = 8;                       // warps that compute
constexpr int COMPUTE = WARPS * 32;
// The ninth streams weights, the tenth fetches to L2; two more, idle, make them a warpgroup, whose registers go to the computing
// ones: what these held beyond 168 registers lay in local memory (0.5B widths, in an early
// state of this kernel: 657 us a step with such spills, 546 without).
constexpr int THREADS = COMPUTE + 128;
constexpr int COMPUTE_REGISTERS = 232, STREAM_REGISTERS = 40;
static_assert(COMPUTE * COMPUTE_REGISTERS + 128 * STREAM_REGISTERS <= THREADS * 168, "no more than the launch brings");
constexpr int SLOT = 16 * 1024;                // bytes of a ring stage
constexpr int MAX_SLOTS = 8;
constexpr int X_BYTES = 42 * 1024;             // a product's input rows, or attention's queries, later tiles and sums
constexpr int TILE_SPACE = 36 * 1024;          // attention's first tile, brought a layer ahead
constexpr int RED_BYTES = 25 * 1024;           // what the warps add up
constexpr int LEAD = 4;                        // ring stages on their way to L2 ahead of the ring's last
constexpr int MAX_TOKENS = 8;
constexpr int MAX_SPLITS = 16;                 // runs of a pair's keys
constexpr int MAX_ROWS = 32;                   // weight rows of a CTA in a product
constexpr int MAX_LAYERS = 96;
#ifndef SHRIKE_STEP_POLL_LIMIT
#define SHRIKE_STEP_POLL_LIMIT 4000000u
#endif
constexpr unsigned POLL_LIMIT = SHRIKE_STEP_POLL_LIMIT;   // looks at a word before it is given up: seconds

constexpr int NOT_TOGETHER = -2;   // the launcher's answer where the device will not run all CTAs at once: nothing has run
enum : int { ERR_PRODUCER = 51, ERR_STAGE = 52, ERR_WORD = 53, ERR_DRAIN = 54 };

// A product: `n` rows of weights, K = 64 * chunks, `rows` of them a CTA (gated: a unit's 16), `depth` chunks to a ring stage.
struct Product {
  int n, chunks, rows, depth;
};

struct Fields {
  const float* norm_mixer;
  const float* norm_ffn;
  const float* b_qkv;    // or null
  __nv_bfloat16* keys;
  __nv_bfloat16* values;
  float eps_mixer, eps_ffn;
};
struct alignas(128) Layer {
  CUtensorMap maps[4];   // q/k/v, o, gate/up, down
  Fields fields;
};

struct Args {
  const Layer* layers;
  const int* positions;
  const int* slots;
  const int* block_table;
  const int* ctx_len;
  const float* inv_freq;   // or null: no rotation
  float* resid;            // [tokens][width]
  Word* x_resid;           // [tokens][width] float32
  Word* x_qkv;             // [tokens][(heads + 2 kv_heads) D] float32
  Word* x_attn;            // [tokens][heads D / 2] pairs of bfloat16
  Word* x_act;             // [tokens][inter / 2] pairs of bfloat16
  Word* x_part;            // [tokens][kv_heads][MAX_SPLITS][group D] float32, then [tokens][kv_heads][MAX_SPLITS][group][2]
  int* sync;               // [0] the number the next launch's exchanges begin with, [1] CTAs that have left
  int* status;
  long long num_slots;
  int num_layers, tokens, width, heads, kv_heads, inter, max_blocks, page_size, num_pages, max_splits, ring;
  int x_span;              // down product: chunks of the activation's columns that half of x holds
  float scale, inv_width;
  Product products[4];
};

struct Shared {
  unsigned long long full[MAX_SLOTS];
  unsigned long long empty[MAX_SLOTS];
  alignas(16) float partial[WARPS];
  float2 angle[64];
  float top[WARPS][16], den[WARPS][16];   // attention: maximum and denominator of a warp's rows
  int rows[256];               // attention: the pool's rows of the first two tiles' keys, -1 where there is none
  volatile int abort;
  volatile int issued;         // ring stages that are on their way or further
};

// As `mbar_wait`, in little code.
__device__ __forceinline__ bool wait_stage(unsigned long long* bar, unsigned parity, Shared* sh, int* status, int who) {
  unsigned tries = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (sh->abort) return false;
    if (++tries >= WAIT_LIMIT) {
      sh->abort = 1;
      if (status != nullptr && *status == 0) *status = who;
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(COMPUTE) : "memory"); }

__device__ __forceinline__ Word word_of(float v, unsigned number) {
  return static_cast<Word>(number) << 32 | __float_as_uint(v);
}
__device__ __forceinline__ float value_of(Word w) { return __uint_as_float(static_cast<unsigned>(w)); }
__device__ __forceinline__ unsigned number_of(Word w) { return static_cast<unsigned>(w >> 32); }
__device__ __forceinline__ void put(Word* p, Word w) { asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory"); }
__device__ __forceinline__ Word get(const Word* p) {
  Word w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}
// Two neighbouring words (each is whole by itself).
__device__ __forceinline__ ulonglong2 get2(const Word* p) {
  ulonglong2 w;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
  return w;
}
// 16 bytes to shared memory through L2; `bytes` 0 writes zeros and reads nothing.
__device__ __forceinline__ void copy16(unsigned dst, const void* src, int bytes = 16) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix2(unsigned (&r)[2], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ void load_box3(unsigned smem, const CUtensorMap* map, unsigned long long* bar, int row, int chunk) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem),
               "l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(bar)), "r"(0), "r"(row), "r"(chunk) : "memory");
}
__device__ __forceinline__ void load_box5(unsigned smem, const CUtensorMap* map, unsigned long long* bar, int half, int run, int chunk) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(smem),
               "l"(reinterpret_cast<unsigned long long>(map)), "r"(smem_u32(bar)), "r"(0), "r"(half), "r"(0), "r"(run), "r"(chunk) : "memory");
}
// The same to L2 alone.
__device__ __forceinline__ void fetch_box3(const CUtensorMap* map, int row, int chunk) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(0),
               "r"(row), "r"(chunk) : "memory");
}
__device__ __forceinline__ void fetch_box5(const CUtensorMap* map, int half, int run, int chunk) {
  asm volatile("cp.async.bulk.prefetch.tensor.5d.L2.global [%0, {%1, %2, %3, %4, %5}];" ::"l"(reinterpret_cast<unsigned long long>(map)),
               "r"(0), "r"(half), "r"(0), "r"(run), "r"(chunk) : "memory");
}
// Before a map in global memory is used: what the host's copy wrote there, and not an earlier table's map at this address that a
// descriptor cache may still hold.  The streaming warpgroup does it for all layers at once and meets (24 layers: no time that
// shows; map by map in the two threads that use them 0.7 us each, 65 us a step).
__device__ __forceinline__ void acquire_map(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}

// Whether CTA `cta` has rows of a product other than the gated one.
__host__ __device__ inline bool has_rows(const Product& g, int cta) { return cta * g.rows < g.n; }
// Whether it reads the residual words in part 0 (see above: those it writes q/k/v rows with, and no others).
__host__ __device__ inline bool reads_residual(const Product* products, int cta) { return has_rows(products[0], cta); }
// The gated product's units of 8 features that CTA `cta` of `ctas` takes: [first, end).
__host__ __device__ __forceinline__ void units_of(int inter, int cta, int ctas, int& first, int& end) {
  const long long units = inter / 8;
  first = static_cast<int>(units * cta / ctas);
  end = static_cast<int>(units * (cta + 1) / ctas);
}

// Streams this CTA's weights, in the order in which the other warps take them.  `fetch`: the warp beside the one that fills the
// ring, which brings the LEAD stages behind the ring's last to L2: while the CTAs wait for one another the ring is full after two
// microseconds, and what HBM brings meanwhile waits there (1.5B widths 784 us a step without, 763 with 4, 867 with 16; 3B 1,418,
// 1,347 and 1,576: fetched further ahead, a stage delays the ones that are needed first).
template <bool FETCH>
__device__ __forceinline__ void stream_weights(const Args& a, Shared* sh, unsigned ring) {
  int slot = 0, stage = 0;
  unsigned parity = 0;
  bool ok = true;
  int first_unit, end_unit;
  units_of(a.inter, blockIdx.x, gridDim.x, first_unit, end_unit);
#pragma unroll 1
  for (int l = 0; l < a.num_layers && ok; ++l) {
#pragma unroll 1
    for (int p = 0; p < 4 && ok; ++p) {
      const Product g = a.products[p];
      const CUtensorMap* map = &a.layers[l].maps[p];
      if (FETCH) prefetch_map(map);
      const int row = blockIdx.x * g.rows;
      const int first = p == 2 ? first_unit : 0, end = p == 2 ? end_unit : (has_rows(g, blockIdx.x) ? 1 : 0);
      const unsigned bytes = static_cast<unsigned>(g.rows * g.depth * 128);
#pragma unroll 1
      for (int u = first; u < end && ok; ++u) {
#pragma unroll 1
        for (int c = 0; c < g.chunks; c += g.depth) {
          if (FETCH) {
            unsigned tries = 0;
            int taken = sh->issued;
#pragma unroll 1
            while (stage >= taken + a.ring + LEAD && ok) {
              __nanosleep(100);
              ok = !sh->abort && ++tries < POLL_LIMIT;
              taken = sh->issued;
            }
            if (!ok) break;
            if (stage >= taken) {   // else the ring has overtaken it
              if (p == 2) fetch_box5(map, (u & 1) * 8, u >> 1, c);
              else fetch_box3(map, row, c);
            }
            ++stage;
            continue;
          }
          ok = wait_stage(&sh->empty[slot], parity ^ 1, sh, a.status, ERR_PRODUCER) && !sh->abort;
          if (!ok) break;
          mbar_expect_tx(&sh->full[slot], bytes);
          if (p == 2) load_box5(ring + slot * SLOT, map, &sh->full[slot], (u & 1) * 8, u >> 1, c);
          else load_box3(ring + slot * SLOT, map, &sh->full[slot], row, c);
          sh->issued = ++stage;
          if (++slot == a.ring) {
            slot = 0;
            parity ^= 1;
          }
        }
      }
    }
  }
  if (!FETCH) {   // where a wait ran out, here or later in the other warps, nobody waits for the copies still in flight: not to leave before
    const int left = stage < a.ring ? stage : a.ring;
#pragma unroll 1
    for (int i = 0; i < left; ++i) {
      if (--slot < 0) {
        slot = a.ring - 1;
        parity ^= 1;
      }
      bool landed = false;
#pragma unroll 1
      for (unsigned tries = 0; tries < WAIT_LIMIT && !landed; ++tries) landed = mbar_try_wait(&sh->full[slot], parity);
      if (!landed && a.status != nullptr) *a.status = ERR_DRAIN;
    }
  }
}

// D: head size.
template <int D>
struct Compute {
  static constexpr int KEY_GROUPS = D == 128 ? 4 : 8;    // warps along the keys of a tile; the others share the head's columns
  static constexpr int TILE = 16 * KEY_GROUPS;           // keys of a tile
  static constexpr int PARTS = WARPS / KEY_GROUPS;
  static constexpr int PITCH = D * 2 + 16;               // bytes of a tile's row: rows fall on different banks
  static constexpr int TILE_BYTES = TILE * PITCH;
  static constexpr int Q_AT = 2 * TILE_BYTES;            // in x: keys and values of every second tile, then the queries
  static constexpr int GROUPS = D / 8, ITEMS = TILE * GROUPS / COMPUTE;   // 16-byte pieces of a row; pieces of a tile for a thread
  static_assert(Q_AT + 16 * PITCH <= X_BYTES && 2 * TILE_BYTES <= TILE_SPACE, "attention's tiles fit");
  static constexpr int SUM_PITCH = D + 8;                // floats: rows fall on different banks
  static_assert(KEY_GROUPS * 16 * SUM_PITCH * 4 <= Q_AT, "the warps' sums fit where the tiles were");
  static_assert(2 * TILE <= 256, "the rows of two tiles fit");

  const Args& a;
  Shared* sh;
  const Fields* const fields;     // every layer's, in shared memory
  float* const gains;             // the weights of the next norm, in shared memory
  const unsigned xs;              // the shared address of x
  unsigned char* const x_mem;     // the same as pointers
  unsigned char* const tile_mem;
  float* const red;
  int tid, warp, lane;
  unsigned slot_at, full_at, parity = 0;   // the ring stage at hand, its barrier
  const unsigned ring_end;
  bool landed = false;            // the stage at hand is known to be there
  unsigned number;                // of the exchange at hand
  float own = 0.f;                // the residual of row `lane` of this CTA's rows, sequence `warp`
  // attention: this CTA's pair and run of keys
  int pair_token = -1, pair_head = 0, key_first = 0, key_end = 0, context = 0, run = 0, splits = 1, own_slot = -1;

  __device__ Compute(const Args& args, Shared* shared, const Fields* f, float* gain, unsigned char* ring_mem, unsigned char* x, unsigned char* tile, float* r, unsigned first)
      : a(args), sh(shared), fields(f), gains(gain), xs(smem_u32(x)), x_mem(x), tile_mem(tile), red(r), tid(threadIdx.x),
        warp(threadIdx.x >> 5), lane(threadIdx.x & 31), slot_at(smem_u32(ring_mem)), full_at(smem_u32(shared->full)), ring_end(smem_u32(ring_mem) + args.ring * SLOT),
        number(first) {}

  // True when a wait has to end: at its limit, or another thread's.
  __device__ __forceinline__ bool stop(unsigned& tries, unsigned limit, int who) {
    if (sh->abort) return true;
    if (++tries < limit) return false;
    sh->abort = 1;
    if (a.status != nullptr && *a.status == 0) *a.status = who;
    return true;
  }
  __device__ __forceinline__ bool give_up(unsigned& tries) { return stop(tries, POLL_LIMIT, ERR_WORD); }
  static constexpr unsigned EMPTY = MAX_SLOTS * 8;   // from a stage's full barrier to its empty one
  __device__ __forceinline__ static bool ready(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
  }

  __device__ __forceinline__ static bool glance(unsigned bar, unsigned parity) {   // never waits
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
  }

  // ---- inputs of a product.  Loads are unconditional, at an index that stays inside the row: a load under a condition costs a
  // branch, and those of a batch would no longer be on their way together.
  // RMS norm of the residual rows into x ([tokens][width] bfloat16, rows `pitch` bytes apart), 1 << `spread` warps a row, each lane
  // PER pairs of elements.
  template <int PER>
  __device__ __forceinline__ void norm_rows(float eps, int pitch, int spread) {
    const int rows_a_pass = WARPS >> spread, share = warp & ((1 << spread) - 1);
    const int pairs = a.width / 2, g0 = share * 32 + lane, step = 32 << spread;
#pragma unroll 1
    for (int first = 0; first < a.tokens; first += rows_a_pass) {
      // every CTA reads the same rows: each begins with another, or all of them would ask one part of L2 at a time
      const int t = min(first + static_cast<int>(((warp >> spread) + blockIdx.x) & (rows_a_pass - 1)), a.tokens - 1);
      const Word* row = a.x_resid + static_cast<size_t>(t) * a.width;
      float2 v[PER];
      unsigned tries = 0;
      bool there;
      do {
        there = true;
        ulonglong2 w[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) w[i] = get2(row + min(g0 + i * step, pairs - 1) * 2);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          there = there && number_of(w[i].x) == number && number_of(w[i].y) == number;
          v[i] = make_float2(value_of(w[i].x), value_of(w[i].y));
        }
      } while (!there && !give_up(tries));
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const float square = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
        sum += g0 + i * step < pairs ? square : 0.f;
      }
      sum = warp_sum(sum);
      if (spread > 0) {
        if (lane == 0) sh->partial[warp] = sum;
        compute_sync();
        const float4 lo = *reinterpret_cast<const float4*>(sh->partial), hi = *reinterpret_cast<const float4*>(sh->partial + 4);
        const float two[4] = {lo.x + lo.y, lo.z + lo.w, hi.x + hi.y, hi.z + hi.w};
        const float low = two[0] + two[1], high = two[2] + two[3];
        sum = spread == 3 ? low + high : (spread == 2 ? (warp < 4 ? low : high) : (warp < 4 ? (warp < 2 ? two[0] : two[1]) : (warp < 6 ? two[2] : two[3])));
        if (first + rows_a_pass < a.tokens) compute_sync();
      }
      const float inv = __frsqrt_rn(sum * a.inv_width + eps);
      unsigned* out = reinterpret_cast<unsigned*>(x_mem + t * pitch);
      const float2* gain = reinterpret_cast<const float2*>(gains);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int g = min(g0 + i * step, pairs - 1);
        const float2 w = gain[g];
        out[g] = pack(__fmul_rn(__fmul_rn(v[i].x, inv), w.x), __fmul_rn(__fmul_rn(v[i].y, inv), w.y));
      }
    }
  }
  __device__ __forceinline__ void norm(float eps, bool reads) {
    if (!reads) {
      copy_wait<0>();   // the gains and the tile: their places are written again
      compute_sync();
      return;
    }
    const int pitch = a.width * 2 + 16, pairs = a.width / 2;
    int spread = a.tokens == 1 ? 3 : (a.tokens == 2 ? 2 : (a.tokens <= 4 ? 1 : 0));   // few rows: several warps each
    while (spread < 3 && pairs > (16 * 32 << spread)) ++spread;
    copy_wait<0>();   // the gains
    compute_sync();
    if (pairs <= (2 * 32 << spread)) norm_rows<2>(eps, pitch, spread);
    else if (pairs <= (4 * 32 << spread)) norm_rows<4>(eps, pitch, spread);
    else if (pairs <= (8 * 32 << spread)) norm_rows<8>(eps, pitch, spread);
    else norm_rows<16>(eps, pitch, spread);
    compute_sync();
  }
  // The weights of the next norm on their way to shared memory.
  __device__ __forceinline__ void bring_gain(const float* from) {
#pragma unroll 1
    for (int i = tid * 4; i < a.width; i += COMPUTE * 4) copy16(smem_u32(gains + i), from + i);
    copy_commit();
  }

  // Four columns an item of a row of pairs of bfloat16 into x, COUNT items of this lane, COMPUTE apart.
  template <int COUNT>
  __device__ __forceinline__ void items_in(const Word* row, uint2* out, int first, int items) {
    unsigned tries = 0;
    bool there;
    ulonglong2 w[COUNT];
    do {
      there = true;
#pragma unroll
      for (int i = 0; i < COUNT; ++i) w[i] = get2(row + min(first + i * COMPUTE, items - 1) * 2);
#pragma unroll
      for (int i = 0; i < COUNT; ++i) there = there && number_of(w[i].x) == number && number_of(w[i].y) == number;
    } while (!there && !give_up(tries));
#pragma unroll
    for (int i = 0; i < COUNT; ++i) out[min(first + i * COMPUTE, items - 1)] = make_uint2(static_cast<unsigned>(w[i].x), static_cast<unsigned>(w[i].y));
  }
  // Columns [first, first + count) of rows of pairs of bfloat16 ([tokens][columns]) into x, rows `pitch` bytes apart.
  __device__ __forceinline__ void rows_in(const Word* from, int columns, unsigned char* to, int pitch, int first, int count) {
    const int items = count / 4;
    int t = blockIdx.x % a.tokens;   // another first row in every CTA
#pragma unroll 1
    for (int n = 0; n < a.tokens; ++n) {
      const Word* row = from + (static_cast<size_t>(t) * columns + first) / 2;
      uint2* out = reinterpret_cast<uint2*>(to + t * pitch);
      int at = warp * 32;
#pragma unroll 1
      while (at < items) {
        if (at + 6 * COMPUTE < items) {
          items_in<8>(row, out, at + lane, items);
          at += 8 * COMPUTE;
        } else if (at + 4 * COMPUTE < items) {
          items_in<6>(row, out, at + lane, items);
          at += 6 * COMPUTE;
        } else if (at + 2 * COMPUTE < items) {
          items_in<4>(row, out, at + lane, items);
          at += 4 * COMPUTE;
        } else if (at + COMPUTE < items) {
          items_in<2>(row, out, at + lane, items);
          at += 2 * COMPUTE;
        } else {
          items_in<1>(row, out, at + lane, items);
          at += COMPUTE;
        }
      }
      t = t + 1 < a.tokens ? t + 1 : 0;
    }
  }

  // ---- products
  // Where a warp's operands lie: of every stage the K steps of 16 columns `warp`, `warp` + 8, ..., two chunks apart.  The rows of a
  // chunk are a multiple of four, so the weights' addresses grow evenly too.
  template <int MT>
  struct Operands {
    unsigned w[MT], w_step, x;
  };
  template <int MT>
  __device__ __forceinline__ Operands<MT> operands(int rows, unsigned x_at, int pitch) const {
    Operands<MT> o;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int line = (warp >> 2) * rows + min(m * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, rows - 1);
      o.w[m] = line * 128 + ((((warp & 3) * 2 + (lane >> 4)) ^ (line & 7)) << 4);
    }
    o.w_step = rows * 256;
    o.x = x_at + min(lane & 7, a.tokens - 1) * pitch + ((lane >> 3) & 1) * 16 + warp * 32;
    return o;
  }
  template <int MT, int COUNT>
  __device__ __forceinline__ void steps_of(float (&acc)[2 * MT][4], unsigned (&w_at)[MT], unsigned w_step, unsigned& x_at) {
    unsigned b[COUNT][2], w[COUNT][MT][4];
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
      ldmatrix2(b[i], x_at + i * 256);
#pragma unroll
      for (int m = 0; m < MT; ++m) ldmatrix4(w[i][m], w_at[m] + i * w_step);
    }
    x_at += COUNT * 256;
#pragma unroll
    for (int m = 0; m < MT; ++m) w_at[m] += COUNT * w_step;
#pragma unroll
    for (int i = 0; i < COUNT; ++i)
#pragma unroll
      for (int m = 0; m < MT; ++m) mma(acc[m + (i & 1) * MT], w[i][m], b[i][0], b[i][1]);
  }
  // One ring stage: `count` of this warp's steps, against the columns of x from `x_at` on.
  template <int MT>
  __device__ __forceinline__ void take_stage(float (&acc)[2 * MT][4], const Operands<MT>& o, int count, unsigned x_at) {
    const unsigned full = full_at, held = parity;
    unsigned w_at[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) w_at[m] = slot_at + o.w[m];
    slot_at += SLOT;
    full_at += 8;
    if (slot_at == ring_end) {
      slot_at -= a.ring * SLOT;
      full_at -= a.ring * 8;
      parity ^= 1;
    }
    unsigned tries = 0;
    while (!landed) {
      landed = ready(full, held);
      if (!landed && stop(tries, WAIT_LIMIT, ERR_STAGE)) break;
    }
    landed = glance(full_at, parity);   // at the next stage, while this one is worked on: the answer takes 150 clocks
#pragma unroll 1
    for (int i = count >> 2; i > 0; --i) steps_of<MT, 4>(acc, w_at, o.w_step, x_at);
    if (count & 2) steps_of<MT, 2>(acc, w_at, o.w_step, x_at);
    if (count & 1) steps_of<MT, 1>(acc, w_at, o.w_step, x_at);
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full + EMPTY) : "memory");
  }

  // The warps' sums to shared memory: [warp][8 sequences][16 MT + 4 rows] (the four keep a warp's stores on different banks).
  template <int MT> static constexpr int SUMS = MT * 16 + 4;
  template <int MT>
  __device__ __forceinline__ void put_sums(const float (&acc)[2 * MT][4], float* buffer) {
    float* mine = buffer + (warp * 8 + (lane & 3) * 2) * SUMS<MT> + (lane >> 2);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      mine[m * 16] = acc[m][0] + acc[m + MT][0];
      mine[m * 16 + SUMS<MT>] = acc[m][1] + acc[m + MT][1];
      mine[m * 16 + 8] = acc[m][2] + acc[m + MT][2];
      mine[m * 16 + 8 + SUMS<MT>] = acc[m][3] + acc[m + MT][3];
    }
  }
  template <int MT>
  __device__ __forceinline__ float sum_of(const float* buffer, int row, int t) const {
    const float* at = buffer + t * SUMS<MT> + row;
    float part[WARPS];
#pragma unroll
    for (int w = 0; w < WARPS; ++w) part[w] = at[w * 8 * SUMS<MT>];
    float sum = part[0];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) sum += part[w];
    return sum;
  }

  // q/k/v (p 0), o (p 1) and down (p 3): the CTA's rows over all of K.  Row `lane` and sequence `warp` of the result are this
  // thread's: with the bias they go to the attention, added to the residual to the next norm.
  template <int MT>
  __device__ __forceinline__ void rows_product(int p, float bias, bool last) {
    const Product g = a.products[p];
    const int row0 = blockIdx.x * g.rows;
    if (!has_rows(g, blockIdx.x)) return;
    float acc[2 * MT][4] = {};   // two chains: a product waits for the one before it on the same sums
    // the input's rows: whole, or (the activation's, where they do not fit) columns a half of x at a time
    const bool whole = p != 3 || a.tokens * (g.chunks * 128 + 16) <= X_BYTES;
    const int span = whole ? g.chunks : a.x_span, pitch = span * 128 + 16;
    const Operands<MT> o = operands<MT>(g.rows, xs, pitch);
    int at = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < g.chunks; c0 += span, at ^= X_BYTES / 2) {
      const int end = min(c0 + span, g.chunks);
      if (p == 3) {
        rows_in(a.x_act, a.inter, x_mem + at, pitch, c0 * 64, (end - c0) * 64);
        compute_sync();
      }
#pragma unroll 1
      for (int c = c0; c < end; c += g.depth) take_stage<MT>(acc, o, min(g.depth, end - c) / 2, o.x + at + (c - c0) * 128);
    }
    put_sums<MT>(acc, red);
    compute_sync();
    if (lane < min(g.rows, g.n - row0) && warp < a.tokens) {
      const float sum = sum_of<MT>(red, lane, warp);
      const size_t at = static_cast<size_t>(warp) * g.n + row0 + lane;
      if (p == 0) {
        put(a.x_qkv + at, word_of(__fadd_rn(sum, bias), number));
      } else {
        own = __fadd_rn(own, sum);
        if (last) a.resid[at] = own;
        else put(a.x_resid + at, word_of(own, number + 1));
      }
    }
  }

  // gate/up with the activation: units of 8 gate rows and the 8 up rows of the same features.  The warps meet once for as many
  // units as their sums have room for.
  static constexpr int UNIT_FLOATS = WARPS * 8 * 20, UNITS_HELD = 5;
  static_assert(UNIT_FLOATS * UNITS_HELD * 4 <= RED_BYTES && WARPS * 8 * 36 * 4 <= RED_BYTES, "the warps' sums fit");
  __device__ __forceinline__ void gated_product() {
    const Product g = a.products[2];
    const Operands<1> o = operands<1>(16, xs, a.width * 2 + 16);
    int first, end;
    units_of(a.inter, blockIdx.x, gridDim.x, first, end);
#pragma unroll 1
    for (int u0 = first; u0 < end; u0 += UNITS_HELD) {
      const int units = min(UNITS_HELD, end - u0);
#pragma unroll 1
      for (int u = 0; u < units; ++u) {
        float acc[2][4] = {};
#pragma unroll 1
        for (int c = 0; c < g.chunks; c += g.depth) take_stage<1>(acc, o, min(g.depth, g.chunks - c) / 2, o.x + c * 128);
        put_sums<1>(acc, red + u * UNIT_FLOATS);
      }
      compute_sync();
      if (warp < a.tokens) {
#pragma unroll 1
        for (int u = lane >> 3; u < (units + 3 & ~3); u += 4) {
          const int f = lane & 7;
          const float* at = red + min(u, units - 1) * UNIT_FLOATS;
          const float gate = __bfloat162float(__float2bfloat16_rn(sum_of<1>(at, f, warp)));
          const float up = __bfloat162float(__float2bfloat16_rn(sum_of<1>(at, 8 + f, warp)));
          const float mine = silu_times<__nv_bfloat16>(gate, up), next = __shfl_down_sync(0xffffffffu, mine, 1);
          if (u < units && !(f & 1))
            put(a.x_act + (static_cast<size_t>(warp) * a.inter + (u0 + u) * 8 + f) / 2, static_cast<Word>(number) << 32 | pack(mine, next));
        }
      }
      if (u0 + UNITS_HELD < end) compute_sync();
    }
  }

  // ---- attention
  // Which pair and run of keys is this CTA's, the same in every layer.
  __device__ __forceinline__ void choose_pair() {
    int unit = blockIdx.x;
#pragma unroll 1
    for (int t = 0; t < a.tokens; ++t) {
      const int length = max(a.ctx_len[t], 1), tiles = (length + TILE - 1) / TILE;
      const int most = min(a.max_splits, tiles), per = (tiles + most - 1) / most, runs = (tiles + per - 1) / per;
      const int units = runs * a.kv_heads;
      if (unit >= 0 && unit < units) {
        pair_token = t;
        pair_head = unit / runs;
        run = unit - pair_head * runs;
        splits = runs;
        context = length;
        key_first = run * per * TILE;
        key_end = min(length, key_first + per * TILE);
      }
      unit -= units;
    }
    if (pair_token >= 0) {
      const long long at = a.slots[pair_token];
      own_slot = at >= 0 && at < a.num_slots ? static_cast<int>(at) : -1;   // never store outside the pool
      if (tid < 2 * TILE) sh->rows[tid] = pool_row(key_first + tid);
      if (a.inv_freq != nullptr && tid < D / 2) {
        float s, c;
        sincosf(__fmul_rn(static_cast<float>(a.positions[pair_token]), a.inv_freq[tid]), &s, &c);
        sh->angle[tid] = make_float2(s, c);
      }
    }
    compute_sync();
  }

  // The pool's row of key `key`, or -1: only keys of earlier positions (the step's own comes from `rotate`).
  __device__ __forceinline__ int pool_row(int key) const {
    if (key >= min(key_end, context - 1)) return -1;
    const int block = key / a.page_size;
    if (block >= a.max_blocks) return -1;   // never read beyond the sequence's own row of the table
    const int page = __ldg(a.block_table + static_cast<size_t>(pair_token) * a.max_blocks + block);
    return page >= 0 && page < a.num_pages ? page * a.page_size + key % a.page_size : -1;
  }
  // Where tile `j` of the run lies: keys, then values.
  __device__ __forceinline__ unsigned char* tile_at(int j) const { return j & 1 ? x_mem : tile_mem; }
  // Brings tile `j` there; zeros where there is no key.
  __device__ __forceinline__ void load_tile(const Fields& layer, int j) {
    const int r0 = tid / GROUPS;
    const unsigned at = smem_u32(tile_at(j)) + r0 * PITCH + (tid % GROUPS) * 16;
    const size_t column = static_cast<size_t>(pair_head) * D + (tid % GROUPS) * 8, pitch = static_cast<size_t>(a.kv_heads) * D;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int r = r0 + i * (COMPUTE / GROUPS), key = key_first + j * TILE + r;
      const int row = j < 2 ? sh->rows[j * TILE + r] : pool_row(key);
      if (key == context - 1) continue;
      const size_t from = row >= 0 ? row * pitch + column : 0;
      copy16(at + i * (COMPUTE / GROUPS) * PITCH, layer.keys + from, row >= 0 ? 16 : 0);
      copy16(at + TILE_BYTES + i * (COMPUTE / GROUPS) * PITCH, layer.values + from, row >= 0 ? 16 : 0);
    }
    copy_commit();
  }
  // Where the step's own key (`value` 0) or value (1) waits: in its tile, or, where that tile's buffer is still another's, in `red`.
  __device__ __forceinline__ __nv_bfloat16* own_row(int value) const {
    const int at = context - 1 - key_first, j = at / TILE;
    if (j >= 2) return reinterpret_cast<__nv_bfloat16*>(red) + value * D;
    return reinterpret_cast<__nv_bfloat16*>(tile_at(j) + value * TILE_BYTES + (at - j * TILE) * PITCH);
  }

  // Rotates the pair's queries into shared memory and, in the run that ends with it, the step's own key, which goes to its page
  // and its tile, as does its value.
  __device__ __forceinline__ void rotate(const Fields& layer) {
    constexpr int HALF = D / 2;
    const int group = a.heads / a.kv_heads;
    const Word* row = a.x_qkv + static_cast<size_t>(pair_token) * (a.heads + 2 * a.kv_heads) * D;
    const int items = (key_end == context ? group + 2 : group) * HALF;   // pairs of the queries, the key and the value
    constexpr int COUNT = 2;   // pairs of a lane whose words are on their way together
#pragma unroll 1
    for (int i0 = warp * 32; i0 < items; i0 += COUNT * COMPUTE) {
      Word lo[COUNT], hi[COUNT];
      unsigned tries = 0;
      bool there;
      do {
        there = true;
#pragma unroll
        for (int n = 0; n < COUNT; ++n) {
          const int i = min(i0 + lane + n * COMPUTE, items - 1), head = i / HALF, j = i - head * HALF;
          const Word* from = row + (head < group ? pair_head * group + head : a.heads + (head - group) * a.kv_heads + pair_head) * D + j;
          lo[n] = get(from);
          hi[n] = get(from + HALF);
        }
#pragma unroll
        for (int n = 0; n < COUNT; ++n) there = there && number_of(lo[n]) == number && number_of(hi[n]) == number;
      } while (!there && !give_up(tries));
#pragma unroll
      for (int n = 0; n < COUNT; ++n) {
        const int i = min(i0 + lane + n * COMPUTE, items - 1), head = i / HALF, j = i - head * HALF;
        const float l = value_of(lo[n]), h = value_of(hi[n]);
        const float2 turn = a.inv_freq != nullptr && head <= group ? sh->angle[j] : make_float2(0.f, 1.f);
        // with the angle 0 the value is l * 1 - h * 0, itself
        const __nv_bfloat16 bl = __float2bfloat16_rn(__fsub_rn(__fmul_rn(l, turn.y), __fmul_rn(h, turn.x)));
        const __nv_bfloat16 bh = __float2bfloat16_rn(__fadd_rn(__fmul_rn(h, turn.y), __fmul_rn(l, turn.x)));
        __nv_bfloat16* to = head < group ? reinterpret_cast<__nv_bfloat16*>(x_mem + Q_AT + head * PITCH) : own_row(head - group);
        to[j] = bl;
        to[j + HALF] = bh;
        if (head >= group && own_slot >= 0) {
          __nv_bfloat16* page = (head == group ? layer.keys : layer.values) + (static_cast<size_t>(own_slot) * a.kv_heads + pair_head) * D;
          page[j] = bl;
          page[j + HALF] = bh;
        }
      }
    }
  }

  __device__ __forceinline__ void attend(const Fields& layer) {
    constexpr int COLUMNS = D / PARTS, TILES_N = COLUMNS / 8;
    const int tiles = (key_end - key_first + TILE - 1) / TILE;
    rotate(layer);
    const int key_group = warp % KEY_GROUPS, part = warp / KEY_GROUPS;
    const float scale = a.scale * 1.44269504088896340736f;
    float top[2] = {-INFINITY, -INFINITY}, den[2] = {0.f, 0.f};
    float out[TILES_N][4] = {};
#pragma unroll 1
    for (int j = 0; j < tiles; ++j) {
      if (j + 1 < tiles) copy_wait<1>();
      else copy_wait<0>();
      compute_sync();   // the tile's copies, and (first) the queries
      const unsigned keys = smem_u32(tile_at(j)) + key_group * 16 * PITCH, values = keys + TILE_BYTES;
      if (j >= 2 && key_end == context && j == tiles - 1) {   // the step's own row waited for this buffer
        if (tid < D) {
          const int r = context - 1 - key_first - j * TILE;
          const __nv_bfloat16* from = reinterpret_cast<const __nv_bfloat16*>(red);
          unsigned char* to = tile_at(j) + r * PITCH;
          reinterpret_cast<__nv_bfloat16*>(to)[tid] = from[tid];
          reinterpret_cast<__nv_bfloat16*>(to + TILE_BYTES)[tid] = from[D + tid];
        }
        compute_sync();
      }
      float s[2][4] = {};
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
        unsigned q[4], b[4];   // keys 0..7 and 8..15 of the warp's, 16 columns each
        ldmatrix4(q, xs + Q_AT + ((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + k * 32 + (lane >> 4) * 16);
        ldmatrix4(b, keys + ((lane & 7) + (lane >> 4) * 8) * PITCH + k * 32 + ((lane >> 3) & 1) * 16);
        mma(s[0], q, b[0], b[1]);
        mma(s[1], q, b[2], b[3]);
      }
      const int key0 = key_first + j * TILE + key_group * 16 + (lane & 3) * 2;
      float high[2] = {top[0], top[1]};
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[n][e] = key0 + n * 8 + (e & 1) < key_end ? s[n][e] * scale : -INFINITY;
          high[e >> 1] = fmaxf(high[e >> 1], s[n][e]);
        }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        high[r] = fmaxf(high[r], __shfl_xor_sync(0xffffffffu, high[r], 1));
        high[r] = fmaxf(high[r], __shfl_xor_sync(0xffffffffu, high[r], 2));
        const float base = high[r] == -INFINITY ? 0.f : high[r];
        const float shrink = exp2f(top[r] - base);
        top[r] = high[r];
        high[r] = base;
        den[r] *= shrink;
#pragma unroll
        for (int n = 0; n < TILES_N; ++n) {
          out[n][r * 2] *= shrink;
          out[n][r * 2 + 1] *= shrink;
        }
      }
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[n][e] = exp2f(s[n][e] - high[e >> 1]);
          den[e >> 1] += s[n][e];
        }
      const unsigned p[4] = {pack(s[0][0], s[0][1]), pack(s[0][2], s[0][3]), pack(s[1][0], s[1][1]), pack(s[1][2], s[1][3])};
#pragma unroll
      for (int n = 0; n < TILES_N; n += 2) {
        unsigned b[4];
        ldmatrix4_trans(b, values + ((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + (part * COLUMNS + n * 8 + (lane >> 4) * 8) * 2);
        mma(out[n], p, b[0], b[1]);
        mma(out[n + 1], p, b[2], b[3]);
      }
      if (j + 2 < tiles) {
        compute_sync();   // every warp is done with this buffer
        load_tile(layer, j + 2);
      }
    }
    // the warps along the keys meet in shared memory, where tiles were, at the highest of their maxima
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (part == 0 && (lane & 3) == 0) sh->top[key_group][(lane >> 2) + r * 8] = top[r];
    compute_sync();
    float* sums = reinterpret_cast<float*>(x_mem);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = (lane >> 2) + r * 8;
      float high = sh->top[0][row];
#pragma unroll
      for (int w = 1; w < KEY_GROUPS; ++w) high = fmaxf(high, sh->top[w][row]);
      const float shrink = exp2f(top[r] - high);   // the run's first group has a key, so `high` is a number
      den[r] += __shfl_xor_sync(0xffffffffu, den[r], 1);
      den[r] += __shfl_xor_sync(0xffffffffu, den[r], 2);
      if (part == 0 && (lane & 3) == 0) sh->den[key_group][row] = den[r] * shrink;
#pragma unroll
      for (int n = 0; n < TILES_N; ++n)
        *reinterpret_cast<float2*>(sums + (key_group * 16 + row) * SUM_PITCH + part * COLUMNS + n * 8 + (lane & 3) * 2) =
            make_float2(out[n][r * 2] * shrink, out[n][r * 2 + 1] * shrink);
    }
    compute_sync();
    const int group = a.heads / a.kv_heads;
    const int pair = pair_token * a.kv_heads + pair_head;
    Word* const result = a.x_attn + (static_cast<size_t>(pair_token) * a.heads + pair_head * group) * (D / 2);
    Word* const sums_of_run = a.x_part + (static_cast<size_t>(pair) * MAX_SPLITS) * group * D;
    Word* const ends_of_run = a.x_part + (static_cast<size_t>(a.tokens) * a.kv_heads * MAX_SPLITS) * group * D + static_cast<size_t>(pair) * MAX_SPLITS * group * 2;
#pragma unroll 1
    for (int i = tid; i < group * D / 2; i += COMPUTE) {
      const int h = i / (D / 2), col = (i - h * (D / 2)) * 2;
      float s0 = 0.f, s1 = 0.f, all = 0.f;
#pragma unroll
      for (int w = 0; w < KEY_GROUPS; ++w) {
        const float2 v = *reinterpret_cast<const float2*>(sums + (w * 16 + h) * SUM_PITCH + col);
        s0 += v.x;
        s1 += v.y;
        all += sh->den[w][h];
      }
      if (splits == 1) {
        const float inv = __frcp_rn(all);
        put(result + i, static_cast<Word>(number) << 32 | pack(s0 * inv, s1 * inv));
      } else {
        Word* to = sums_of_run + (static_cast<size_t>(run) * group + h) * D + col;
        put(to, word_of(s0, number));
        put(to + 1, word_of(s1, number));
        if (col == 0) {
          float high = sh->top[0][h];
#pragma unroll 1
          for (int w = 1; w < KEY_GROUPS; ++w) high = fmaxf(high, sh->top[w][h]);
          put(ends_of_run + (run * group + h) * 2, word_of(high, number));
          put(ends_of_run + (run * group + h) * 2 + 1, word_of(all, number));
        }
      }
    }
    if (splits > 1) add_runs(sums_of_run, ends_of_run, result, group);
  }

  // This run's share of the pair's columns, added up over the runs.
  __device__ __forceinline__ void add_runs(const Word* sums, const Word* ends, Word* result, int group) {
    constexpr int AT_ONCE = 8;   // runs whose words are on their way together
    const int items = group * D / 2, share = (items + splits - 1) / splits;
#pragma unroll 1
    for (int i = run * share + tid; i < min(items, (run + 1) * share); i += COMPUTE) {
      const int h = i / (D / 2), col = (i - h * (D / 2)) * 2;
      float top = -INFINITY, den = 0.f, n0 = 0.f, n1 = 0.f;
#pragma unroll 1
      for (int r0 = 0; r0 < splits; r0 += AT_ONCE) {
        ulonglong2 m[AT_ONCE], v[AT_ONCE];
        unsigned tries = 0;
        bool ready;
        do {
          ready = true;
#pragma unroll
          for (int r = 0; r < AT_ONCE; ++r) {
            const size_t at = static_cast<size_t>(min(r0 + r, splits - 1)) * group + h;
            m[r] = get2(ends + at * 2);
            v[r] = get2(sums + at * D + col);
          }
#pragma unroll
          for (int r = 0; r < AT_ONCE; ++r)
            ready = ready && number_of(m[r].x) == number && number_of(m[r].y) == number && number_of(v[r].x) == number && number_of(v[r].y) == number;
        } while (!ready && !give_up(tries));
        float high = top;
#pragma unroll
        for (int r = 0; r < AT_ONCE; ++r) high = fmaxf(high, value_of(m[r].x));
        const float shrink = exp2f(top - high);
        den *= shrink;
        n0 *= shrink;
        n1 *= shrink;
        top = high;
#pragma unroll
        for (int r = 0; r < AT_ONCE; ++r) {
          const float f = r0 + r < splits ? exp2f(value_of(m[r].x) - high) : 0.f;
          den = fmaf(value_of(m[r].y), f, den);
          n0 = fmaf(value_of(v[r].x), f, n0);
          n1 = fmaf(value_of(v[r].y), f, n1);
        }
      }
      const float inv = __frcp_rn(den);
      put(result + i, static_cast<Word>(number) << 32 | pack(n0 * inv, n1 * inv));
    }
  }

  __device__ __forceinline__ float bias_of(int l) const {
    const Product& g = a.products[0];
    const int row = blockIdx.x * g.rows + lane;
    return fields[l].b_qkv != nullptr && lane < g.rows && row < g.n ? __ldg(fields[l].b_qkv + row) : 0.f;
  }

  __device__ __forceinline__ void run_layers() {
    choose_pair();
    bring_gain(fields[0].norm_mixer);
    if (pair_token >= 0) load_tile(fields[0], 0);
    float bias = bias_of(0);
    {   // the residual as it stands, from the CTAs that add to it
      const int row = blockIdx.x * a.products[1].rows + lane;
      if (lane < a.products[1].rows && row < a.width && warp < a.tokens) {
        own = a.resid[static_cast<size_t>(warp) * a.width + row];
        put(a.x_resid + static_cast<size_t>(warp) * a.width + row, word_of(own, number));
      }
    }
#pragma unroll 1
    for (int l = 0; l < a.num_layers; ++l) {
      const Fields& layer = fields[l];
      const bool last = l + 1 == a.num_layers;
#pragma unroll 1
      for (int at = 0; at < 4; ++at) {
        // keeps what follows from a thread's place within its part, and the parts in one copy: the compiler would write the loop
        // out and hold all parts' addresses over the layers
        int p = at;
        asm volatile("" : "+r"(p), "+r"(tid), "+r"(warp), "+r"(lane));
        if (p == 0 || p == 2) norm(p == 0 ? layer.eps_mixer : layer.eps_ffn, p == 2 || reads_residual(a.products, blockIdx.x));
        else if (p == 1 || !last) bring_gain(p == 1 ? layer.norm_ffn : fields[l + 1].norm_mixer);
        if (p == 1) {
          rows_in(a.x_attn, a.heads * D, x_mem, a.heads * D * 2 + 16, 0, a.heads * D);
          compute_sync();
        }
        if (p == 2) gated_product();
        else if (a.products[p].rows <= 16) rows_product<1>(p, bias, p == 3 && last);
        else rows_product<2>(p, bias, p == 3 && last);
        compute_sync();   // x is free
        if (p == 0) {
          if (pair_token >= 0) {
            if (TILE < key_end - key_first) load_tile(layer, 1);
            attend(layer);
            compute_sync();
            if (!last) load_tile(fields[l + 1], 0);   // a layer ahead: taking in a tile's copies holds an SM's threads up for a microsecond
          }
        }
        if (p == 2 && !last) bias = bias_of(l + 1);
        if (p & 1) ++number;
      }
    }
  }
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1) decode_step_kernel(const __grid_constant__ Args a) {
  extern __shared__ unsigned char raw[];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  unsigned char* x = ring + static_cast<size_t>(a.ring) * SLOT;
  unsigned char* tile = x + X_BYTES;
  float* red = reinterpret_cast<float*>(tile + TILE_SPACE);
  float* gains = red + RED_BYTES / 4;
  Fields* fields = reinterpret_cast<Fields*>(gains + a.width);
  Shared* sh = reinterpret_cast<Shared*>(fields + a.num_layers);
  const unsigned first = static_cast<unsigned>(*static_cast<volatile int*>(a.sync));
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.ring; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], WARPS);
    }
    sh->abort = 0;
    sh->issued = 0;
    mbar_init_fence();
  }
  for (int l = threadIdx.x; l < a.num_layers; l += THREADS) fields[l] = a.layers[l].fields;
  __syncthreads();
  if (threadIdx.x >= COMPUTE) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(STREAM_REGISTERS));
    for (int i = threadIdx.x - COMPUTE; i < 4 * a.num_layers; i += THREADS - COMPUTE) acquire_map(&a.layers[i >> 2].maps[i & 3]);
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS - COMPUTE) : "memory");
    if (threadIdx.x == COMPUTE) stream_weights<false>(a, sh, smem_u32(ring));
    if (threadIdx.x == COMPUTE + 32) stream_weights<true>(a, sh, smem_u32(ring));
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(COMPUTE_REGISTERS));
    Compute<D> compute(a, sh, fields, gains, ring, x, tile, red, first);
    compute.run_layers();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    // the last CTA to leave sets the next launch's first number: by then every CTA has read this one's
    if (atomicAdd(a.sync + 1, 1) == static_cast<int>(gridDim.x) - 1) {
      a.sync[1] = 0;
      a.sync[0] = static_cast<int>(first + 2 * a.num_layers + 2);
      __threadfence();
    }
  }
}

// How a product is cut over `ctas` CTAs; depth: chunks of K to a ring stage (even, as a warp's steps lie two chunks apart).
static bool cut(int n, int k, int ctas, bool gated, Product* out) {
  if (n < 1 || k < 128 || k % 128) return false;
  out->n = n;
  out->chunks = k / 64;
  out->rows = gated ? 16 : ((n + ctas - 1) / ctas + 3) / 4 * 4;
  if (out->rows > MAX_ROWS) return false;
  int most = SLOT / (out->rows * 128) / 2 * 2;
  if (most > out->chunks) most = out->chunks;
  const int stages = (out->chunks + most - 1) / most;
  out->depth = ((out->chunks + stages - 1) / stages + 1) / 2 * 2;
  return true;
}

struct Cuts {
  Product products[4];
  int ring, x_span;
  size_t smem;
};

// The sizes this kernel serves, on the current device.
static bool cuts_of(int tokens, int layers, int width, int heads, int kv_heads, int dim, int inter, Cuts* out) {
  const ShrikeDevice& device = shrike_device();
  const int ctas = device.sm_count, q_width = heads * dim;
  if (tokens < 1 || tokens > MAX_TOKENS || layers < 1 || layers > MAX_LAYERS || (dim != 64 && dim != 128)) return false;
  if (kv_heads < 1 || heads % kv_heads || heads / kv_heads > 16 || tokens * kv_heads > ctas) return false;
  if (inter % 16 || inter / 8 < ctas) return false;   // every CTA has a gated unit
  Product* p = out->products;
  if (!cut((heads + 2 * kv_heads) * dim, width, ctas, false, &p[0]) || !cut(width, q_width, ctas, false, &p[1]) ||
      !cut(2 * inter, width, ctas, true, &p[2]) || !cut(width, inter, ctas, false, &p[3]))
    return false;
  // What a CTA reads of the others' words in a layer: beyond it the launches one by one are quicker.  Measured at 600 to 1,024
  // keys, us a step as launches and as one kernel: up to four sequences it wins to some 350 KB (width 2,048, 3 sequences, 255 KB:
  // 1,740 and 1,600; 4, 340 KB: 1,766 and 1,761, at 100 keys 1,711 and 1,733; 3,584, 2, 294 KB: 2,712 and 2,620; 3, 441 KB, 500 keys: 2,751 and 2,817); more take
  // the norm two rounds of rows, and win to some 200 KB (896, 5, 190 KB: 704 and 699, at 500 keys 673 and 693; 7, 266 KB, 500 keys: 840 and 884).
  const long long read = 4LL * tokens * (4LL * width + q_width + inter);
  if (read > (tokens <= 4 ? 352 : 200) * 1024LL) return false;
  const int wide = width > q_width ? width : q_width;
  if (tokens * (wide * 2 + 16) > X_BYTES || width > 16 * 64 * WARPS) return false;
  out->x_span = (X_BYTES / 2 / tokens - 16) / (p[3].depth * 128) * p[3].depth;
  if (tokens * (inter * 2 + 16) > X_BYTES && out->x_span < 1) return false;
  const size_t fixed = 1024 + X_BYTES + TILE_SPACE + RED_BYTES + static_cast<size_t>(width) * 4 + layers * sizeof(Fields) + sizeof(Shared);
  if (fixed + 3 * SLOT > static_cast<size_t>(device.max_smem)) return false;
  out->ring = static_cast<int>((device.max_smem - fixed) / SLOT);
  if (out->ring > MAX_SLOTS) out->ring = MAX_SLOTS;
  out->smem = fixed + static_cast<size_t>(out->ring) * SLOT;
  return true;
}

// The longest context with which a step that is served is at least as quick as the launches one by one: this kernel's attention
// has one CTA an SM and two tiles of keys in it, the launches' two CTAs and three tiles.
// In us a layer, fitted to both ways in turn at 100 to 32,000 keys, 1 to 8 sequences and 1 to 14 kv heads:
//   here      2 for each tile of a run (64 keys of heads of 128, 128 of 64)
//   launches  1.35 for each tile of 64 keys that one of two CTAs an SM walks, or, where pairs are few and their splits meet in
//             global memory, 2.3 and up to 10 (7) for that
//   the rest  what this kernel saves in products and norms: 11 or 12 less what is read of others' words
// Measured, keys at which both are equal (and what this says), sequences in turn.  2 kv heads of 128: 1,536 wide, 1 to 4: 13,700
// (12,300), 13,400 (11,900), 11,800 (11,400), 11,000 (11,500); 2,048 wide, 1 to 4: 13,000 (11,900), 12,800 (11,000), 11,900 (9,600),
// 9,500 (10,200).  3,584 wide, 4 kv heads, 1 and 2: 11,000 (11,600), 12,000 (10,400).  1,536 wide, 12 kv heads, 1 to 4: 14,500 (16,400),
// 3,000 (2,700), 1,500 (1,300), 200 (620).  896 wide, 2 kv heads of 64, 1, 2 and 5: 25,300 (23,400), 31,000 (30,000), 12,500 (14,200);
// 14 kv heads, 1 to 4: 16,700 (18,100), 6,900 (7,700), 3,500 (3,300), 1,600 (1,500).  512 wide, 8 kv heads of 64, 5 and 8: 3,300
// (3,200), 1,700 (1,700).  Beyond it the loss grows: 1,536 wide and 32,000 keys 1,601 us a step as launches and 2,412 here; 14
// layers with 12 kv heads, 4 sequences of 16,384 keys 1,349 and 2,839.
static int most_keys(int tokens, int width, int heads, int kv_heads, int dim, int inter) {
  const int ctas = shrike_device().sm_count, pairs = tokens * kv_heads;
  int runs = ctas / pairs;
  runs = runs > MAX_SPLITS ? MAX_SPLITS : runs;
  const bool narrow = dim == 64, few = pairs <= (narrow ? 10 : 16);
  const double kilobytes = 4.0 * tokens * (4.0 * width + heads * dim + inter) / 1024;
  const double here = 2.0 / (runs * (narrow ? 128 : 64));   // a key
  const double launches = (few && tokens <= 4 ? 2.3 : 1.35) * pairs / (64.0 * 2 * ctas);
  double ahead = tokens <= 4 ? 11.7 - 0.04 * kilobytes : 11 - 0.045 * kilobytes;
  if (ahead < 0) ahead = 0;
  if (!narrow) ahead += few ? 2 : 3;   // a run's first tile, which the shortest context has too
  if (few) ahead += narrow ? 8 - 0.5 * pairs : (pairs < 6 ? 11 - 0.5 * pairs : 8);
  constexpr int FAR = 65536;   // where the two grow alike (896 wide, 4 sequences): no further than twice what was measured
  const double keys = here > launches ? ahead / (here - launches) : FAR;
  return static_cast<int>(keys < FAR ? keys : FAR);
}

// A product's weights as ring stages: rows of 64 columns, `depth` of them side by side.
static int encode_map(CUtensorMap* map, const void* w, const Product& p, bool gated) {
  EncodeTiled encode = encode_tiled();
  if (encode == nullptr || (reinterpret_cast<uintptr_t>(w) & 15)) return SHRIKE_BAD_ARGUMENT;
  const cuuint64_t row = static_cast<cuuint64_t>(p.chunks) * 128;   // bytes
  CUresult rc;
  if (gated) {   // [64 columns][16 features of a run][gate, up][runs][chunks]
    const cuuint64_t dims[5] = {64, 16, 2, static_cast<cuuint64_t>(p.n / 32), static_cast<cuuint64_t>(p.chunks)};
    const cuuint64_t strides[4] = {row, 16 * row, 32 * row, 128};
    const cuuint32_t box[5] = {64, 8, 2, 1, static_cast<cuuint32_t>(p.depth)};
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(w), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(p.n), static_cast<cuuint64_t>(p.chunks)};
    const cuuint64_t strides[2] = {row, 128};
    const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(p.rows), static_cast<cuuint32_t>(p.depth)};
    const cuuint32_t ones[3] = {1, 1, 1};
    rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(w), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  return rc == CUDA_SUCCESS ? SHRIKE_OK : 1000 + static_cast<int>(rc);
}

}  // namespace step

extern "C" {
// What a layer is, host side: one record per layer run.
struct ShrikeStepLayer {
  const void *w_qkv, *w_o, *w_gate_up, *w_down;
  const float *norm_mixer, *norm_ffn, *b_qkv;
  void *keys, *values;
  float eps_mixer, eps_ffn;
};

struct ShrikeStepArgs {
  const void* layers;   // the device table that shrike_decode_step_table filled
  const int *positions, *slots, *block_table, *ctx_len;
  const float* inv_freq;
  float* resid;
  void* words;          // shrike_decode_step_words() 64-bit words, zero before the first launch
  int *sync, *status;   // sync: two ints, 1 and 0 before the first launch
  long long num_slots;
  int num_layers, tokens, width, heads, kv_heads, head_dim, inter, max_blocks, page_size, num_pages;
  float scale;
};
}

// 1 when a step of `tokens` single tokens over `layers` layers of these sizes is served.
SHRIKE_API int shrike_decode_step_serves(int tokens, int layers, int width, int heads, int kv_heads, int head_dim, int inter) {
  step::Cuts cuts;
  return step::cuts_of(tokens, layers, width, heads, kv_heads, head_dim, inter, &cuts) ? 1 : 0;
}
// What each of `ctas` CTAs does in a layer, on the host: bit p of roles[cta] says that it has rows (units) of product p, bit 4
// that it reads the residual words in part 0.
SHRIKE_API int shrike_decode_step_roles(int ctas, int width, int heads, int kv_heads, int head_dim, int inter, int* roles) {
  using namespace step;
  Product p[4];
  if (!cut((heads + 2 * kv_heads) * head_dim, width, ctas, false, &p[0]) || !cut(width, heads * head_dim, ctas, false, &p[1]) ||
      !cut(2 * inter, width, ctas, true, &p[2]) || !cut(width, inter, ctas, false, &p[3]))
    return SHRIKE_BAD_ARGUMENT;
  for (int cta = 0; cta < ctas; ++cta) {
    int first, end;
    units_of(inter, cta, ctas, first, end);
    roles[cta] = (has_rows(p[0], cta) ? 1 : 0) | (has_rows(p[1], cta) ? 2 : 0) | (first < end ? 4 : 0) | (has_rows(p[3], cta) ? 8 : 0) |
                 (reads_residual(p, cta) ? 16 : 0);
  }
  return SHRIKE_OK;
}
// The longest context for which it is also the quicker way; 0 where it is not served.
SHRIKE_API int shrike_decode_step_keys(int tokens, int layers, int width, int heads, int kv_heads, int head_dim, int inter) {
  step::Cuts cuts;
  if (!step::cuts_of(tokens, layers, width, heads, kv_heads, head_dim, inter, &cuts)) return 0;
  return step::most_keys(tokens, width, heads, kv_heads, head_dim, inter);
}
SHRIKE_API int shrike_decode_step_layer_bytes() { return static_cast<int>(sizeof(step::Layer)); }
// 64-bit words that the exchanges of a step of up to `tokens` tokens take.
SHRIKE_API long long shrike_decode_step_words(int tokens, int width, int heads, int kv_heads, int head_dim, int inter) {
  const long long a_token = width + heads * head_dim / 2 + inter / 2 + static_cast<long long>(heads + 2 * kv_heads) * head_dim +
                            static_cast<long long>(heads) * step::MAX_SPLITS * (head_dim + 2);
  return a_token * tokens;
}

// Fills `table` (host memory, shrike_decode_step_layer_bytes() a layer) for `count` layers of equal sizes.
SHRIKE_API int shrike_decode_step_table(const ShrikeStepLayer* layers, int count, int width, int heads, int kv_heads, int head_dim,
                                        int inter, void* table) {
  step::Cuts cuts;
  if (!step::cuts_of(1, count, width, heads, kv_heads, head_dim, inter, &cuts)) return SHRIKE_BAD_ARGUMENT;
  step::Layer* out = static_cast<step::Layer*>(table);
  for (int l = 0; l < count; ++l) {
    const ShrikeStepLayer& in = layers[l];
    const void* w[4] = {in.w_qkv, in.w_o, in.w_gate_up, in.w_down};
    for (int p = 0; p < 4; ++p) {
      const int rc = step::encode_map(&out[l].maps[p], w[p], cuts.products[p], p == 2);
      if (rc != SHRIKE_OK) return rc;
    }
    out[l].fields = {in.norm_mixer, in.norm_ffn, in.b_qkv, static_cast<__nv_bfloat16*>(in.keys), static_cast<__nv_bfloat16*>(in.values),
                     in.eps_mixer, in.eps_ffn};
  }
  return SHRIKE_OK;
}

SHRIKE_API int shrike_decode_step(const ShrikeStepArgs* in, cudaStream_t stream) {
  using namespace step;
  Cuts cuts;
  if (in->page_size < 1 || in->num_pages < 1 || in->max_blocks < 1) return SHRIKE_BAD_ARGUMENT;
  if (!cuts_of(in->tokens, in->num_layers, in->width, in->heads, in->kv_heads, in->head_dim, in->inter, &cuts)) return SHRIKE_BAD_ARGUMENT;
  const ShrikeDevice& device = shrike_device();
  const size_t n = in->tokens;
  Args a;
  a.layers = static_cast<const Layer*>(in->layers);
  a.positions = in->positions;
  a.slots = in->slots;
  a.block_table = in->block_table;
  a.ctx_len = in->ctx_len;
  a.inv_freq = in->inv_freq;
  a.resid = in->resid;
  // the words of every exchange begin at an even one: they are read two at a time
  a.x_resid = static_cast<Word*>(in->words);
  a.x_qkv = a.x_resid + n * in->width;
  a.x_attn = a.x_qkv + n * (in->heads + 2 * in->kv_heads) * in->head_dim;
  a.x_act = a.x_attn + n * in->heads * in->head_dim / 2;
  a.x_part = a.x_act + n * in->inter / 2;
  a.sync = in->sync;
  a.status = in->status;
  a.num_slots = in->num_slots;
  a.num_layers = in->num_layers;
  a.tokens = in->tokens;
  a.width = in->width;
  a.heads = in->heads;
  a.kv_heads = in->kv_heads;
  a.inter = in->inter;
  a.max_blocks = in->max_blocks;
  a.page_size = in->page_size;
  a.num_pages = in->num_pages;
  a.scale = in->scale;
  a.inv_width = 1.0f / static_cast<float>(in->width);
  a.ring = cuts.ring;
  a.x_span = cuts.x_span;
  for (int p = 0; p < 4; ++p) a.products[p] = cuts.products[p];
  const int splits = device.sm_count / (in->tokens * in->kv_heads);   // runs of a pair's keys: as many as there are CTAs for
  a.max_splits = splits > MAX_SPLITS ? MAX_SPLITS : splits;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(device.sm_count);
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = cuts.smem;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  // all CTAs live at once, or none starts: they wait for one another (a process may be held to a part of the SMs)
  attribute.id = cudaLaunchAttributeCooperative;
  attribute.val.cooperative = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
#define SHRIKE_STEP_CASE(D)                                                                     \
  {                                                                                             \
    static PerDevice raised;                                                                    \
    const int rc = shrike_raise_smem(raised, decode_step_kernel<D>, device.max_smem);           \
    if (rc != 0) return rc;                                                                     \
    const cudaError_t err = cudaLaunchKernelEx(&config, decode_step_kernel<D>, a);              \
    if (err == cudaErrorCooperativeLaunchTooLarge || err == cudaErrorNotSupported) {            \
      cudaGetLastError();                                                                       \
      return NOT_TOGETHER;                                                                      \
    }                                                                                           \
    if (err != cudaSuccess) return static_cast<int>(err);                                       \
    return shrike_launch_status();                                                              \
  }
  if (in->head_dim == 64) SHRIKE_STEP_CASE(64)
  SHRIKE_STEP_CASE(128)
#undef SHRIKE_STEP_CASE
}
