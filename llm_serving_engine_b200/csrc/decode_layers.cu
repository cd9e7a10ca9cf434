// All layers of a decode step and the LM head in one launch (bfloat16, up to four rows, pre-norm layers of grouped-query
// attention with rotary positions and a SiLU-gated feed-forward).
//
// What bounds such a step is the chain: launch by launch a layer of the 1.5B sizes is nine kernels of 1 to 6 us, a third of
// the time lies between one kernel's end and the next one's first load, and the weights of a product stream only while that
// product runs or the one before ends.  Here one block an SM stays for the whole step:
//   * Two warps bring all that the block will use, in the order of use, into a ring of stages in shared memory (bulk copies of
//     up to 3 KB a row: an SM starts one about every 42 ns, so rows of 1.5 KB gave 5.4 TB/s, of 3 KB 6.7), whatever the phase:
//     while the blocks wait for one another, up to 150 KB an SM of the next products' weights, or of the next attention's keys
//     and values, are on their way.  (cp.async by the computing warps instead: 1.5 times slower, every other load then queues
//     behind the stream in the SM's memory pipe.)
//   * A phase is a product's units of 16 weight rows, dealt out to the blocks in turn (a running deal over the phases, so that
//     a block that got a unit more in one gets one less in the next); the eight computing warps share a unit's k range, their
//     sums are added in shared memory in the warps' order.  Weights ride the M side of mma.sync (m16n8k16), the step's rows the
//     N side: the product is bound by the weights' bytes, and units of 16 rows fill 148 blocks where the 128 rows of a tcgen05
//     tile would not.  Sixteen computing warps were slower: what a phase costs beside its bytes, every warp issues.
//   * There are no barriers between blocks.  What they exchange travels in 8-byte packets, a value and the epoch (layer) that it
//     belongs to, and who needs a packet polls it: one store and one load (about 1.2 us), where a grid barrier and the load behind
//     it took 3.4.  A packet's place is written again only by blocks whose own input depends, over the phases between, on every
//     reader having read.
//   * Norms are not phases: who adds to the residual multiplies by the next norm's weight and leaves the sums of squares of its
//     16 columns; who reads it adds these up and scales.  These values are float32 in places of their own for every norm, cleared
//     to a pattern that no value has: four values a read, where packets would hold two.  Rotation, bias and the cache write belong
//     to the attention, the SiLU gate to the gate/up product (a unit is eight gate rows and the eight up rows beside them).  The
//     down product's k range may be cut into parts, and a request's keys into shares: the blocks add up one another's parts, in
//     their order.
// Sums do not depend on timing: every order is fixed.
//
// Measured against nine launches a layer, one B200: 28 layers of the 1.5B sizes and the head, one request of 100 keys, 870 to 880
// us a step against 1,174 (a layer 26 us, of which 14 are the weights' time at the memory's rate: QKV 2.5 us, attention 4, O 3,
// gate/up 8, down 6, each 1.2 to 2 of it waiting for the others); more sizes beside the rule in models/decode_layers.py.
//
// Every wait is bounded: a block whose wait gives up sets the kernel's error word and the launch's abort word, the others see
// it while they wait, and all leave.  Whichever way a block leaves, the warps that bring its data wait until all that they have
// started has landed.  The launch is cooperative: all blocks are on the GPU at once or none is.
#include <type_traits>

#include "key_ring.cuh"
#include "mma_common.cuh"
#include "smem_allowance.cuh"
#include "tcgen05.cuh"

LSE_TL_DEFINE(lse_timeline_decode_layers)
LSE_CHECK_DEFINE(lse_check_decode_layers)

namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;    // warps that compute; two more bring the data
constexpr int HEAD = 128;                // head size
constexpr int MAX_LAYERS = 80;
constexpr int MAX_ROWS = 4;              // of the eight columns of the instruction: with more, the exchange between the blocks costs too much
constexpr int UNIT_SUMS = WARPS * 16 * MAX_ROWS;   // the warps' sums of a unit
constexpr int MAX_HEADS = 8;             // query heads of a key/value head
constexpr int STAGE_CHUNKS = 48;         // 32-k chunks of eight weight rows that a stage holds at most: copies of up to 3 KB a row
constexpr int ROW_BYTES = STAGE_CHUNKS * 64 + 64;   // rows of a stage lie 64 bytes apart modulo 128: two rows' 16-byte reads do not collide
constexpr int STAGE = 25 * 1024;         // 8 rows, or:
constexpr int STAGE_KEYS = 3;            // tiles of 16 keys and their values (8 KB each)
constexpr int MAX_STAGES = 6;
constexpr int KEY_TILES = 1024;          // 16-key tiles of a block whose place in the cache is looked up ahead
constexpr int SPLIT_TILES = 8;           // a share of a request's keys is at least this many tiles (128 keys) ...
constexpr int MAX_SPLITS = 24;           // ... and a request's keys are cut into at most so many shares
constexpr int Q_STRIDE = HEAD * 2 + 64;  // bytes of a query row in shared memory
constexpr unsigned SPIN_LIMIT = 1u << 22;
static_assert(STAGE % 1024 == 0 && STAGE >= STAGE_KEYS * 8192 && STAGE >= 8 * ROW_BYTES, "key tiles are swizzled in 1024-byte groups");

constexpr int MAX_DOWN_GROUPS = 2048;

__device__ int lse_decode_layers_error;
__device__ unsigned lse_decode_layers_spin_limit = SPIN_LIMIT;
__device__ int lse_decode_layers_withhold;    // test hook: the first sum of squares never comes

// Tuning builds: when the blocks passed the marks of the last layer (nanoseconds of the global timer).
#ifdef LSE_TRACE
constexpr int STAMPS = 32, STAMP_BLOCKS = 256;
__device__ unsigned long long lse_decode_layers_stamp[STAMP_BLOCKS][STAMPS];
#define STAMP(k) if (tid == 0 && block < STAMP_BLOCKS && layer == a.layers - 1) lse_decode_layers_stamp[block][k] = lse_now();
#else
#define STAMP(k)
#endif

struct Layer {
  const __nv_bfloat16 *qkv, *o, *gate_up, *down;
  const float *qkv_bias, *norm1, *norm2;
  __nv_bfloat16 *keys, *values;
  float eps1, eps2;
};

struct Common {
  const __nv_bfloat16* head;
  const float *final_norm, *inv_freq;
  const int *positions, *segment_of_token, *slot_mapping, *block_tables;
  // Packets of 8 bytes: a value (float32, or two bfloat16), and in the upper 16 bits the epoch that it belongs to.
  uint2 *input, *middle;       // the residual that a layer begins with, and behind its attention [rows][hidden]
  uint2 *qkv, *attended, *act; // [rows][n], [rows][n_q * 64], [rows][inter / 2]
  uint2 *part_o, *part_ml;     // an attention share's sums [blocks][heads][128], maximum and sum [blocks][heads][2]
  uint2* down_part;            // [splits][rows][hidden]
  // What the norms read, float32 without epochs: the residual times the norm's weight [rows][hidden], and its sums of squares of
  // 16 columns at a time [rows][hidden / 16].  Every norm of the step has a place of its own (2 l and 2 l + 1 in layer l, 2 layers
  // at the end), which holds UNSET until its values come: four values a read, where packets would hold two.
  uint32_t* normed;
  unsigned* abort;             // set: a wait gave up somewhere
  float* logits;
  int layers, rows, hidden, inter, n_q, n_kv, vocab, page_size, bt_stride, num_pages, num_slots, num_segments, pairing;
  int down_splits, batch_units, x_bytes, stages, norm_stride;   // values from a norm's place to the next one's
  float final_eps, scale_log2e;
};

struct Args {
  CUtensorMap maps[MAX_LAYERS][2];   // keys, values
  Layer layer[MAX_LAYERS];
  Common common;
};

enum Phase { QKV = 0, KV = 1, O = 2, GATE_UP = 3, DOWN = 4, HEADS = 5 };

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Two packets, each read at once.
__device__ __forceinline__ uint4 load_packets(const uint2* p) {
  unsigned long long lo, hi;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];\n" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ uint2 load_packet(const uint2* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
__device__ __forceinline__ void store_packet(uint2* p, uint32_t value, uint32_t epoch) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"((unsigned long long)epoch << 48 | value) : "memory");
}
// A float32 in a place that held UNSET: a NaN of these bits is stored as another.
constexpr uint32_t UNSET = 0xffffffffu;
__device__ __forceinline__ uint32_t set_bits(float v) {
  const uint32_t u = __float_as_uint(v);
  return u == UNSET ? 0x7fffffffu : u;
}
__device__ __forceinline__ void store_value(uint32_t* p, float v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(set_bits(v)) : "memory");
}
__device__ __forceinline__ uint4 load_values(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, unsigned long long policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2::evict_last [%0];\n" ::"l"(p)); }
__device__ __forceinline__ void mma4(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  const uint32_t a[4] = {a0, a1, a2, a3};
  mma_bf16(d, a, b0, b1);
}
// The same for at most eight rows on the M side (query heads): their two sums a thread.
__device__ __forceinline__ void mma_heads(float& d0, float& d1, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm volatile("{\n\t.reg .f32 x, y;\n\t"
               "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,x,y}, {%2,%3,%4,%3}, {%5,%6}, {%0,%1,%7,%7};\n\t}\n"
               : "+f"(d0), "+f"(d1) : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}
// All computing warps of the block (those that bring the data do not take part).
__device__ __forceinline__ void block_sync() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }
// The same; true in all of them when it was `ok` for all.
__device__ __forceinline__ bool block_sync_ok(bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
               : "=r"(all) : "r"((uint32_t)ok) : "memory");
  return all != 0;
}

// What a block does of a step's attention: one share of the keys of one (row, key/value head).
struct Item {
  int row, kv_head, split, splits, first_block;   // row -1: none
  int tile, tiles, limit;                         // 16-key tiles of the cache; keys at `limit` and beyond are not used from it
  int segment, slot, position;
};

// Units of a phase that are this block's: first, first + step, ... (count of them), and how a unit's k range is staged
struct Share {
  int first, step, count;
  int chunks, pieces, per_piece;   // 32-k chunks, pieces of it (two stages each: rows 0-7, rows 8-15), chunks of a piece
};

struct Shared {
  unsigned long long full[MAX_STAGES], empty[MAX_STAGES];
  Common common;             // read from here: loads of kernel parameters are moved ahead of the loop over layers, and spilled
  Item item;
  Share share[6];
  int down_first_chunk;      // of this block's part of the down product's k range
  int down_split;
  int abort;
  unsigned spin_limit;
  int started[MAX_STAGES];   // parity of the phase in which a slot was filled last, -1: never
  float inverse[MAX_ROWS];   // 1 / rms of the rows
  float cs[HEAD / 2], sn[HEAD / 2];
  float ml[WARPS + 1][MAX_HEADS][2];
  int row_segment[MAX_ROWS], row_position[MAX_ROWS];
  __nv_bfloat16 new_k[HEAD], new_v[HEAD];
  int pages[KEY_TILES];      // rows of the cache, in groups of 8, at which the item's tiles begin
};

__device__ __forceinline__ bool wait_for(uint32_t bar, uint32_t parity, Shared& s) {
  volatile int* abort = &s.abort;
  for (unsigned i = 0; i < s.spin_limit; ++i) {
    if (tc::mbar_test_suspend(bar, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  atomicExch(&lse_decode_layers_error, 1);
  return false;
}

// What a block does: its barriers, its units of every phase, its share of the attention.  One thread, once a launch.
__device__ __noinline__ void deal(const Common& a, Shared& s, int block, int blocks) {
  const int n_qkv = (a.n_q + 2 * a.n_kv) * HEAD;
  for (int i = 0; i < a.stages; ++i) {
    tc::mbar_init(smem_u32(&s.full[i]), 1);
    tc::mbar_init(smem_u32(&s.empty[i]), WARPS);
    s.started[i] = -1;
  }
  tc::mbar_init_fence();
  int at = 0;
  const int k_all = a.inter / 32, per = ((k_all + a.down_splits - 1) / a.down_splits + 1) / 2 * 2;   // a part: whole 64 k
  const int part = block % a.down_splits, rank = block / a.down_splits;
  for (int p = 0; p < 6; ++p) {
    const int units = p == QKV ? n_qkv / 16 : p == O ? a.hidden / 16 : p == GATE_UP ? a.inter / 8 : p == HEADS ? a.vocab / 16 : 0;
    Share sh;
    sh.step = blocks;
    sh.first = (block - at % blocks + blocks) % blocks;
    sh.count = sh.first < units ? (units - sh.first + blocks - 1) / blocks : 0;
    sh.chunks = (p == O ? a.n_q * HEAD : a.hidden) / 32;
    at += units;
    if (p == DOWN) {   // block b takes part b % splits of the k range; the groups of 16 rows are dealt out within a part
      const int groups = a.hidden / 16;
      sh.step = (blocks - part + a.down_splits - 1) / a.down_splits;
      sh.first = rank;
      sh.count = rank < groups ? (groups - rank + sh.step - 1) / sh.step : 0;
      sh.chunks = min(per, k_all - part * per);
    }
    sh.pieces = (sh.chunks + STAGE_CHUNKS - 1) / STAGE_CHUNKS;
    sh.per_piece = (sh.chunks + sh.pieces - 1) / sh.pieces;
    s.share[p] = sh;
  }
  s.down_split = part;
  s.down_first_chunk = part * per;
  s.abort = 0;
  // attention: a share is `target` tiles of 16 keys, as few as fit into one share a block
  int most = 0, total = 0;
  for (int r = 0; r < a.rows; ++r) {
    if (s.row_segment[r] < 0) continue;
    const int t = (s.row_position[r] + 15) / 16;   // the row's own key does not come from the cache
    most = max(most, t);
    total += t;
  }
  int target = max(SPLIT_TILES, max((total * a.n_kv + blocks - 1) / blocks, (most + MAX_SPLITS - 1) / MAX_SPLITS));
  for (;;) {
    int next = 0;
    s.item.row = -1;
    s.item.tiles = 0;
    for (int r = 0; r < a.rows; ++r) {
      if (s.row_segment[r] < 0) continue;
      const int t = (s.row_position[r] + 15) / 16;
      const int splits = max(1, (t + target - 1) / target), per_split = (t + splits - 1) / splits;
      if (block >= next && block < next + splits * a.n_kv) {
        const int head = (block - next) / splits, split = (block - next) % splits;
        s.item.row = r;
        s.item.kv_head = head;
        s.item.split = split;
        s.item.splits = splits;
        s.item.first_block = block - split;
        s.item.tile = min(t, split * per_split);
        s.item.tiles = max(0, min(per_split, t - split * per_split));
        s.item.position = s.item.limit = s.row_position[r];
        s.item.segment = s.row_segment[r];
              }
      next += splits * a.n_kv;
    }
    if (next <= blocks) break;
    target += max(1, target / 8);
  }
  if (s.item.row >= 0) s.item.slot = LSE_CHECKED(a.slot_mapping[s.item.row], -1, a.num_slots, -1, LSE_CHECK_CACHE_SLOT);
}

// The two warps that bring weights, keys and values: every stage that this block will use, in the order of use, by turns.
// (Copies are started at about one every 42 ns an SM: of 3 KB each that is 1.6 times what an SM's share of the memory gives.)
__device__ __forceinline__ void bring(const Args& args, const Layer* layers, Shared& s, uint32_t ring, int lane, int which) {
  const Common& a = s.common;
  const int stages = a.stages;
  Slot slot;
  bool ok = true, mine = which == 0;    // the next stage is this warp's
  unsigned long long once;              // weights are read once a step: they leave the L2 to what the blocks exchange
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(once));
  auto product = [&](int phase, const __nv_bfloat16* w, int stride, int column, int rows_a_unit, int second) {
    const Share sh = s.share[phase];
    const size_t half = (size_t)second * stride, unit = (size_t)sh.step * rows_a_unit * stride;
    const uint32_t whole = sh.per_piece * 64u, last = (sh.chunks - (sh.pieces - 1) * sh.per_piece) * 64u;
    // lane r < 8 brings row r of a stage: rows 0-7 of the unit, then rows 8-15 (or as many rows of the second half)
    const __nv_bfloat16* src = w + ((size_t)sh.first * rows_a_unit + (lane & 7)) * stride + column;
    for (int i = 0; i < sh.count && ok; ++i, src += unit) {
      const __nv_bfloat16* from = src;
      for (int p = 0; p < sh.pieces; ++p, from += sh.per_piece * 32) {
        const uint32_t bytes = p + 1 < sh.pieces ? whole : last;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (mine && ok) {
            const uint32_t bar = smem_u32(&s.full[slot.at]);
            ok = __all_sync(0xffffffffu, wait_for(smem_u32(&s.empty[slot.at]), slot.parity ^ 1u, s));   // one answer for the warp
            if (ok && lane == 0) {
              tc::mbar_expect_tx(bar, 8u * bytes);
              s.started[slot.at] = (int)slot.parity;
            }
            __syncwarp();
            if (ok && lane < 8) bulk_copy(ring + slot.at * STAGE + lane * ROW_BYTES, from + (h ? half : 0), bytes, bar, once);
          }
          mine = !mine;
          slot.step(stages);
        }
      }
    }
  };
  auto small_weights = [&](int layer) {   // (the second warp) into the L2, so that who needs them does not wait behind the stream
    const Layer& L = layers[layer];
    const int norm_lines = a.hidden / 32, bias_lines = (a.n_q + 2 * a.n_kv) * HEAD / 32;
    if (which == 0) return;
    for (int i = blockIdx.x + lane * gridDim.x; i < 2 * norm_lines + bias_lines; i += 32 * gridDim.x) {
      if (i < norm_lines) prefetch_l2(L.norm1 + i * 32);
      else if (i < 2 * norm_lines) prefetch_l2(L.norm2 + (i - norm_lines) * 32);
      else if (L.qkv_bias) prefetch_l2(L.qkv_bias + (i - 2 * norm_lines) * 32);
    }
  };
  small_weights(0);
  for (int layer = 0; layer < a.layers && ok; ++layer) {
    const Layer& L = layers[layer];
    if (layer + 1 < a.layers) {
      small_weights(layer + 1);
      if (lane < 2) asm volatile("prefetch.tensormap [%0];\n" ::"l"(&args.maps[layer + 1][lane]) : "memory");
    }
    product(QKV, L.qkv, a.hidden, 0, 16, 8);
    for (int t0 = 0; t0 < s.item.tiles && ok; t0 += STAGE_KEYS) {
      const int tiles = min(STAGE_KEYS, s.item.tiles - t0);
      if (mine) {
        const uint32_t bar = smem_u32(&s.full[slot.at]), dst = ring + slot.at * STAGE;
        ok = __all_sync(0xffffffffu, wait_for(smem_u32(&s.empty[slot.at]), slot.parity ^ 1u, s));
        if (ok && lane == 0) {
          tc::mbar_expect_tx(bar, tiles * 8192u);
          s.started[slot.at] = (int)slot.parity;
        }
        __syncwarp();
        if (ok && lane < 2 * tiles) {
          const int t = t0 + (lane >> 1);
          int at;
          if (t < KEY_TILES) {
            at = s.pages[t];
          } else {
            const int key = (s.item.tile + t) * 16;
            const int page = LSE_CHECKED(a.block_tables[(size_t)s.item.segment * a.bt_stride + key / a.page_size], 0, a.num_pages, 0,
                                         LSE_CHECK_TABLE_ENTRY);
            at = ((page * a.n_kv + s.item.kv_head) * a.page_size + key % a.page_size) / 8;
          }
          tc::tma_load_4d(dst + (lane >> 1) * 8192 + (lane & 1) * 4096, &args.maps[layer][lane & 1], bar, 0, 0, 0, at);
        }
      }
      mine = !mine;
      slot.step(stages);
    }
    product(O, L.o, a.n_q * HEAD, 0, 16, 8);
    product(GATE_UP, L.gate_up, a.hidden, 0, 8, a.inter);
    product(DOWN, L.down, a.inter, s.down_first_chunk * 32, 16, 8);
  }
  product(HEADS, a.head, a.hidden, 0, 16, 8);
  // Neither warp starts anything any more: all that is in flight lands before the block leaves, also where the computing warps
  // have left already.
  asm volatile("bar.sync 2, 64;\n" ::: "memory");
  if (which == 0 && lane < stages) {
    const int parity = s.started[lane];
    for (unsigned i = 0; parity >= 0 && i < SPIN_LIMIT; ++i)
      if (tc::mbar_test_suspend(smem_u32(&s.full[lane]), (uint32_t)parity)) break;
  }
}

__global__ void __launch_bounds__(THREADS + 64, 1) decode_layers_kernel(const __grid_constant__ Args args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ Shared s;
  __shared__ __align__(128) unsigned char q_s[MAX_HEADS * Q_STRIDE];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int block = blockIdx.x, blocks = gridDim.x;
  const Common& a = s.common;
  if (tid < (int)(sizeof(Common) / 4)) reinterpret_cast<int*>(&s.common)[tid] = reinterpret_cast<const int*>(&args.common)[tid];
  __syncthreads();
  unsigned char* smem = smem_raw + (1024u - (smem_u32(smem_raw) & 1023u)) % 1024u;
  const uint32_t ring = smem_u32(smem);
  const uint32_t x_s = ring + a.stages * STAGE;                                        // rows of x, then the units' sums
  unsigned char* work = smem + a.stages * STAGE;
  // The layers' addresses are read from shared memory: a kernel parameter that was not touched for a layer's time comes through
  // the constant cache from memory, behind the stream of weights.
  Layer* layers = reinterpret_cast<Layer*>(smem + a.stages * STAGE + a.x_bytes + 2 * a.batch_units * UNIT_SUMS * (int)sizeof(float));
  for (int i = tid; i < a.layers * (int)(sizeof(Layer) / 8); i += THREADS + 64)
    reinterpret_cast<uint2*>(layers)[i] = reinterpret_cast<const uint2*>(args.layer)[i];
  float* red = reinterpret_cast<float*>(work + a.x_bytes);                             // two batches of [unit][warp][16][rows]
  const int q_per = a.n_q / a.n_kv, n_qkv = (a.n_q + 2 * a.n_kv) * HEAD;

  LSE_TL_BEGIN(8)
  // ---- what this block does: its units of every phase, its share of the attention
  if (tid < a.rows) {
    s.row_segment[tid] = LSE_CHECKED(a.segment_of_token[tid], -1, a.num_segments, -1, LSE_CHECK_SEGMENT);
    s.row_position[tid] = a.positions[tid];
  }
  if (tid == THREADS) s.spin_limit = lse_decode_layers_spin_limit;
  __syncthreads();
  if (tid == 0) deal(a, s, block, blocks);
  __syncthreads();
  const bool attends = s.item.row >= 0;
  if (attends) {
    for (int i = tid; i < min(s.item.tiles, KEY_TILES); i += THREADS + 64) {
      const int key = (s.item.tile + i) * 16;
      const int page = LSE_CHECKED(a.block_tables[(size_t)s.item.segment * a.bt_stride + key / a.page_size], 0, a.num_pages, 0,
                                   LSE_CHECK_TABLE_ENTRY);
      s.pages[i] = ((page * a.n_kv + s.item.kv_head) * a.page_size + key % a.page_size) / 8;
    }
    if (tid < HEAD / 2) {
      float sn, cs;
      sincosf(__fmul_rn((float)s.item.position, a.inv_freq[tid]), &sn, &cs);
      s.cs[tid] = cs;
      s.sn[tid] = sn;
    }
    for (int i = tid; i < MAX_HEADS * Q_STRIDE / 4; i += THREADS + 64) reinterpret_cast<uint32_t*>(q_s)[i] = 0u;
  }
  __syncthreads();
  if (warp >= WARPS) {
    bring(args, layers, s, ring, lane, warp - WARPS);
    return;
  }

  // ---- the pieces of a phase
  bool ok = true;     // false: a wait gave up; the thread goes on as far as the next block_sync_ok, where all leave
  // Called while a packet has not come: false when there is no point in waiting on.
  auto patience = [&](unsigned& turns) -> bool {
    if (!ok) return false;
    if (++turns & 255u) return true;
    unsigned stop;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(stop) : "l"(a.abort) : "memory");
    if (turns >= s.spin_limit) atomicExch(&lse_decode_layers_error, 1);
    if (turns >= s.spin_limit || stop || *(volatile int*)&s.abort) {
      *(volatile int*)&s.abort = 1;
      atomicExch(a.abort, 1u);
      ok = false;
    }
    return ok;
  };
  // Waits for the 16 bytes load(k), k in `todo` (a bit each), until came(v[k]): every round asks for all that have not come together,
  // so that what came late costs one round trip, not one each.
  auto fetch_until = [&](auto& v, uint32_t todo, auto came, auto load) {
    constexpr int COUNT = sizeof(v) / sizeof(uint4);
    for (unsigned turns = 0; todo;) {
#pragma unroll
      for (int k = 0; k < COUNT; ++k)
        if (todo >> k & 1u) v[k] = load(k);
#pragma unroll
      for (int k = 0; k < COUNT; ++k)
        if ((todo >> k & 1u) && came(v[k])) todo &= ~(1u << k);
      if (todo && !patience(turns)) break;
    }
  };
  auto fetch = [&](auto& v, uint32_t todo, uint32_t epoch, auto at) {   // pairs of packets
    fetch_until(v, todo, [&](const uint4& got) { return got.y >> 16 == epoch && got.w >> 16 == epoch; }, [&](int k) { return load_packets(at(k)); });
  };
  auto fetch_single = [&](auto& v, uint32_t todo, auto epoch, auto at) {
    constexpr int COUNT = sizeof(v) / sizeof(uint2);
    for (unsigned turns = 0; todo;) {
#pragma unroll
      for (int k = 0; k < COUNT; ++k)
        if (todo >> k & 1u) v[k] = load_packet(at(k));
#pragma unroll
      for (int k = 0; k < COUNT; ++k)
        if ((todo >> k & 1u) && v[k].y >> 16 == epoch) todo &= ~(1u << k);
      if (todo && !patience(turns)) break;
    }
  };
  // Rows of x (bfloat16) into shared memory, COUNT times 16 bytes a thread in flight: pairs of packets of two bfloat16 each, or
  // (normed) four values of a norm's place, whose sums of squares say what they are multiplied by.
  auto load_x = [&](auto count, auto normed, int tid, const void* src, int row_quads, int quads, uint32_t epoch, const uint32_t* squares,
                    int x_row_bytes, uint32_t rows_mask, float eps) {
    constexpr int COUNT = decltype(count)::value;
    constexpr bool NORMED = decltype(normed)::value;
    constexpr int SQUARES = NORMED ? 1 : 0;
    const int lane = tid & 31, warp = tid >> 5, groups = a.hidden / 16;
    auto came = [&](const uint4& v) {
      if (NORMED) return v.x != UNSET && v.y != UNSET && v.z != UNSET && v.w != UNSET;
      return v.y >> 16 == epoch && v.w >> 16 == epoch;
    };
    auto sum_of = [](const uint4& v) { return (__uint_as_float(v.x) + __uint_as_float(v.y)) + (__uint_as_float(v.z) + __uint_as_float(v.w)); };
    const int all = quads * a.rows;
    int row = 0, column = tid;
    auto settle = [&]() {
      while (column >= quads) {
        column -= quads;
        if (++row == a.rows) row = 0;
      }
    };
    settle();
    for (int e = tid, round = 0; round == 0 || e < all; ++round) {
      uint4 v[COUNT + SQUARES] = {};    // set on every path: a register that is not stays occupied through all phases
      uint32_t quad_of[COUNT];          // row and column of the 16 bytes
      uint32_t todo = 0u;
#pragma unroll
      for (int k = 0; k < COUNT; ++k) {
        quad_of[k] = (uint32_t)row << 24 | (uint32_t)column;
        if (e < all && (rows_mask >> row & 1u)) todo |= 1u << k;     // padding rows: nobody writes them
        e += THREADS;
        column += THREADS;
        settle();
      }
      const uint32_t mine = todo;
      if (NORMED && round == 0 && warp < a.rows && 4 * lane < groups) todo |= 1u << COUNT;   // a warp adds up a row's: lanes, then the butterfly
      auto load = [&](int k) -> uint4 {
        if (NORMED && k >= COUNT) return load_values(squares + warp * groups + 4 * lane);
        const size_t at = (size_t)(quad_of[k] >> 24) * row_quads + (quad_of[k] & 0xffffffu);
        return NORMED ? load_values(reinterpret_cast<const uint32_t*>(src) + 4 * at) : load_packets(reinterpret_cast<const uint2*>(src) + 2 * at);
      };
      if (COUNT > 4) {                                        // many: one of them is waited for, then the others asked for
        fetch_until(v, todo & 1u, came, load);
        todo &= ~1u;
      }
      fetch_until(v, todo, came, load);
      if (NORMED && round == 0) {
#pragma unroll 1
        for (int r = warp; r < a.rows; r += WARPS) {
          float sq = r == warp ? sum_of(v[COUNT + SQUARES - 1]) : 0.f;
#pragma unroll 1
          for (int i = 4 * lane + (r == warp ? 128 : 0); i < groups; i += 128) {
            uint4 more[1] = {};
            fetch_until(more, 1u, came, [&](int) { return load_values(squares + r * groups + i); });
            sq += sum_of(more[0]);
          }
          sq = warp_sum(sq);
          if (lane == 0) s.inverse[r] = 1.0f / sqrtf(sq / (float)a.hidden + eps);
        }
        block_sync();
      }
#pragma unroll
      for (int k = 0; k < COUNT; ++k) {
        if (mine >> k & 1u) {
          uint2 out = make_uint2(v[k].x, v[k].z);
          if (NORMED) {
            const float inverse = s.inverse[quad_of[k] >> 24];
            out.x = pack_bf16(__uint_as_float(v[k].x) * inverse, __uint_as_float(v[k].y) * inverse);
            out.y = pack_bf16(__uint_as_float(v[k].z) * inverse, __uint_as_float(v[k].w) * inverse);
          }
          *reinterpret_cast<uint2*>(work + (quad_of[k] >> 24) * x_row_bytes + (quad_of[k] & 0xffffffu) * 8) = out;
        }
      }
    }
  };
  int rows_log = 0;     // rows, rounded up to a power of two
  while ((1 << rows_log) < a.rows) ++rows_log;
  uint32_t valid_rows = 0u;
  for (int r = 0; r < a.rows; ++r) valid_rows |= (s.row_segment[r] >= 0 ? 1u : 0u) << r;
  auto unit_sum = [&](const float* sums, int row16, int row) {   // in the order of the warps
    const float* p = sums + row16 * MAX_ROWS + row;
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) total += p[w * 16 * MAX_ROWS];
    return total;
  };

  Slot slot;          // of the next stage
  for (int layer = 0, phase = QKV;;) {
    const Layer& L = layers[layer < a.layers ? layer : 0];
    const uint32_t epoch = layer + 1;   // of this layer's packets (the residual that it leaves to the next one: epoch + 1)
    // read anew: what is worked out from the thread's number would otherwise be carried, spilled, through all phases
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;\n" : "=r"(tid));
    const int lane = tid & 31, warp = tid >> 5;
    STAMP(phase * 4)
    if (phase == KV) {
      // -------------------------------------------------------------------- attention
      if (attends) {
        const Item& it = s.item;
        const bool own = it.split == it.splits - 1;   // this share holds the row's own key
        const uint2* row = a.qkv + (size_t)it.row * n_qkv;
        {   // pairs that turn together: of the queries, of the key, and (not turned) of the value
          const int q_pairs = q_per * (HEAD / 2), all = q_pairs + (own ? HEAD : 0);
          constexpr int MOST = (MAX_HEADS * HEAD / 2 + HEAD + THREADS - 1) / THREADS;
          uint2 v[2 * MOST] = {};
          auto first_of = [&](int e, int& apart) -> const uint2* {
            const int i = e & 63;
            const bool value = e >= q_pairs + HEAD / 2, turned_apart = a.pairing != 0 && !value;
            const int head = value ? a.n_q + a.n_kv + it.kv_head : e >= q_pairs ? a.n_q + it.kv_head : it.kv_head * q_per + (e >> 6);
            apart = turned_apart ? HEAD / 2 : 1;
            return row + head * HEAD + (turned_apart ? i : 2 * i);
          };
          uint32_t mine = 0u;
#pragma unroll
          for (int k = 0; k < MOST; ++k)
            if (tid + k * THREADS < all) mine |= 3u << (2 * k);
          fetch_single(v, mine, epoch, [&](int k) {
            int apart;
            const uint2* p = first_of(tid + (k >> 1) * THREADS, apart);
            return p + (k & 1) * apart;
          });
          const size_t at = it.slot < 0 ? 0
              : (((size_t)(it.slot / a.page_size) * a.n_kv + it.kv_head) * a.page_size + it.slot % a.page_size) * HEAD;
#pragma unroll
          for (int k = 0; k < MOST; ++k) {
            const int e = tid + k * THREADS;
            if (e < all) {
              int apart;
              first_of(e, apart);
              const int i = e & 63, ea = apart == 1 ? 2 * i : i, eb = ea + apart;
              float xa = __uint_as_float(v[2 * k].x), xb = __uint_as_float(v[2 * k + 1].x);
              if (e < q_pairs + HEAD / 2) {
                const float ya = __fsub_rn(__fmul_rn(xa, s.cs[i]), __fmul_rn(xb, s.sn[i]));
                xb = __fadd_rn(__fmul_rn(xb, s.cs[i]), __fmul_rn(xa, s.sn[i]));
                xa = ya;
              }
              const __nv_bfloat16 ra = __float2bfloat16_rn(xa), rb = __float2bfloat16_rn(xb);
              __nv_bfloat16* dst = e < q_pairs ? reinterpret_cast<__nv_bfloat16*>(q_s + (e >> 6) * Q_STRIDE)
                                               : e < q_pairs + HEAD / 2 ? s.new_k : s.new_v;
              dst[ea] = ra;
              dst[eb] = rb;
              if (e >= q_pairs && it.slot >= 0) {
                __nv_bfloat16* cache = (e < q_pairs + HEAD / 2 ? L.keys : L.values) + at;
                cache[ea] = ra;
                cache[eb] = rb;
              }
            }
          }
        }
        if (!block_sync_ok(ok)) break;
        STAMP(5)
        // A warp's tiles of 16 keys: S = Q K^T (heads x keys), probabilities relative to the running maximum, O += P V.
        // A stage holds three tiles; the warps take the tiles in turn.
        const int r = lane >> 2, q = lane & 3;
        float o[HEAD / 8][2] = {};
        float m_run = -INFINITY, l_run = 0.f;
        uint4 qf[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) qf[j] = lds128(smem_u32(q_s) + r * Q_STRIDE + j * 64 + q * 16);
        auto wait_stage = [&](const Slot& at) { ok = ok && wait_for(smem_u32(&s.full[at.at]), at.parity, s); };
        auto stage_read = [&](const Slot& at) {
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(smem_u32(&s.empty[at.at]));
        };
        auto tile = [&](const Slot& at, int i, int t) {
          const uint32_t kt = ring + at.at * STAGE + i * 8192, vt = kt + 4096;
          const int left = it.limit - (it.tile + t) * 16;   // keys of the tile that are the request's
          if (left < 16) {   // whatever else lies there (NaN included) counts as zero
            const int row16 = lane >> 1;
            if (row16 >= left) {
              const uint32_t dst = vt + (row16 >> 3) * 2048 + (row16 & 7) * 128 + (lane & 1) * 1024;
              const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
              for (int c = 0; c < 8; ++c) sts128(dst + c * 16, zero);
            }
            __syncwarp();
          }
          float c[2][2] = {};
#pragma unroll
          for (int k8 = 0; k8 < 2; ++k8)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 b = lds128(kt + k8 * 2048 + (j >> 1) * 1024 + r * 128 + ((((j & 1) * 4 + q) ^ r) << 4));
              mma_heads(c[k8][0], c[k8][1], qf[j].x, qf[j].y, b.x, b.y);
              mma_heads(c[k8][0], c[k8][1], qf[j].z, qf[j].w, b.z, b.w);
            }
          float m_tile = -INFINITY;
#pragma unroll
          for (int k8 = 0; k8 < 2; ++k8)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              c[k8][e] = k8 * 8 + 2 * q + e < left ? c[k8][e] * a.scale_log2e : -INFINITY;
              m_tile = fmaxf(m_tile, c[k8][e]);
            }
          m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 1));
          m_tile = fmaxf(m_tile, __shfl_xor_sync(0xffffffffu, m_tile, 2));
          const float m_new = fmaxf(m_run, m_tile);
          const float base = m_new == -INFINITY ? 0.f : m_new;
          const float keep = fast_exp2(m_run - base);
          m_run = m_new;
          l_run *= keep;
#pragma unroll
          for (int k8 = 0; k8 < 2; ++k8)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              c[k8][e] = fast_exp2(c[k8][e] - base);
              l_run += c[k8][e];
            }
#pragma unroll
          for (int d = 0; d < HEAD / 8; ++d) { o[d][0] *= keep; o[d][1] *= keep; }
          const uint32_t p0 = pack_bf16(c[0][0], c[0][1]), p1 = pack_bf16(c[1][0], c[1][1]);
          const uint32_t v_row = vt + ((lane >> 3) & 1) * 2048 + (lane & 7) * 128;
#pragma unroll
          for (int d = 0; d < HEAD / 16; ++d) {
            uint32_t b[4];
            ldmatrix_x4_trans(b, v_row + (d >> 2) * 1024 + ((((d & 3) * 2 + (lane >> 4)) ^ (lane & 7)) << 4));
            mma_heads(o[2 * d][0], o[2 * d][1], p0, p1, b[0], b[1]);
            mma_heads(o[2 * d + 1][0], o[2 * d + 1][1], p0, p1, b[2], b[3]);
          }
          if (left < 16) tc::fence_async_smem();
        };
        walk_key_stages(warp, WARPS, it.tiles, STAGE_KEYS, a.stages, slot, wait_stage, tile, stage_read);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
        l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
        STAMP(6)
        float* sums = reinterpret_cast<float*>(work);   // [8][heads][128]; the row's own key is a ninth part
        float* dst = sums + (warp * MAX_HEADS + r) * HEAD + 2 * q;
#pragma unroll
        for (int d = 0; d < HEAD / 8; ++d) *reinterpret_cast<float2*>(dst + d * 8) = make_float2(o[d][0], o[d][1]);
        if (q == 0) { s.ml[warp][r][0] = m_run; s.ml[warp][r][1] = l_run; }
        if (warp == WARPS - 1) {
          float dot = 0.f;
          if (own) {
            const __nv_bfloat162* qh = reinterpret_cast<const __nv_bfloat162*>(q_s + r * Q_STRIDE);
            const __nv_bfloat162* kh = reinterpret_cast<const __nv_bfloat162*>(s.new_k);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float2 x = __bfloat1622float2(qh[i * 4 + q]), y = __bfloat1622float2(kh[i * 4 + q]);
              dot = fmaf(x.x, y.x, fmaf(x.y, y.y, dot));
            }
            dot += __shfl_xor_sync(0xffffffffu, dot, 1);
            dot += __shfl_xor_sync(0xffffffffu, dot, 2);
          }
          if (q == 0) { s.ml[WARPS][r][0] = own ? dot * a.scale_log2e : -INFINITY; s.ml[WARPS][r][1] = own ? 1.f : 0.f; }
        }
        block_sync();
        const int pairs = q_per * (HEAD / 2);
        uint2* out = a.attended + ((size_t)it.row * a.n_q + (size_t)it.kv_head * q_per) * (HEAD / 2);   // [q_per][64] pairs
#pragma unroll 1
        for (int e = tid; e < pairs; e += THREADS) {
          const int h = e >> 6, d = (e & 63) * 2;
          float m = -INFINITY;
#pragma unroll
          for (int w = 0; w <= WARPS; ++w) m = fmaxf(m, s.ml[w][h][0]);
          // A maximum is that of the numbers among the scores; where there are none, NaN among them still comes through the sums.
          const float base = m > -INFINITY ? m : 0.f;
          float l = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll
          for (int w = 0; w < WARPS; ++w) {
            const float f = fast_exp2(s.ml[w][h][0] - base);
            const float2 sum = *reinterpret_cast<const float2*>(sums + (w * MAX_HEADS + h) * HEAD + d);
            l += s.ml[w][h][1] * f;
            v0 += sum.x * f;
            v1 += sum.y * f;
          }
          if (own) {
            const float f = fast_exp2(s.ml[WARPS][h][0] - base);
            const float2 value = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(s.new_v + d));
            l += f;
            v0 += value.x * f;
            v1 += value.y * f;
          }
          if (it.splits == 1) {
            store_packet(out + e, pack_bf16(v0 / l, v1 / l), epoch);
          } else {
            uint2* po = a.part_o + ((size_t)block * MAX_HEADS + h) * HEAD + d;
            store_packet(po, __float_as_uint(v0), epoch);
            store_packet(po + 1, __float_as_uint(v1), epoch);
            if (d == 0) {
              uint2* ml = a.part_ml + (size_t)(block * MAX_HEADS + h) * 2;
              store_packet(ml, __float_as_uint(m), epoch);
              store_packet(ml + 1, __float_as_uint(l), epoch);
            }
          }
        }
        if (it.splits > 1) {   // every share's block adds up some of the results, over the shares in their order
          const int per = (pairs + it.splits - 1) / it.splits, e = it.split * per + tid;
          if (tid < per && e < pairs) {
            const int h = e >> 6, d = (e & 63) * 2;
            const uint2* po = a.part_o + ((size_t)it.first_block * MAX_HEADS + h) * HEAD + d;
            const uint2* pm = a.part_ml + (size_t)(it.first_block * MAX_HEADS + h) * 2;
            constexpr int AT_ONCE = 10;
            float m = -INFINITY, l = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll 1
            for (int p0 = 0; p0 < it.splits; p0 += AT_ONCE) {
              uint4 o2[AT_ONCE] = {}, ml[AT_ONCE] = {};
              const uint32_t some = (1u << min(AT_ONCE, it.splits - p0)) - 1u;
              fetch(o2, some, epoch, [&](int k) { return po + (size_t)(p0 + k) * MAX_HEADS * HEAD; });
              fetch(ml, some, epoch, [&](int k) { return pm + (size_t)(p0 + k) * MAX_HEADS * 2; });
#pragma unroll
              for (int k = 0; k < AT_ONCE; ++k)
                if (p0 + k < it.splits) {
                  const float its = __uint_as_float(ml[k].x);
                  const float m_new = fmaxf(m, its), base = m_new > -INFINITY ? m_new : 0.f;
                  const float keep = fast_exp2(m - base), f = fast_exp2(its - base);
                  l = l * keep + __uint_as_float(ml[k].z) * f;
                  v0 = v0 * keep + __uint_as_float(o2[k].x) * f;
                  v1 = v1 * keep + __uint_as_float(o2[k].z) * f;
                  m = m_new;
                }
            }
            store_packet(out + e, pack_bf16(v0 / l, v1 / l), epoch);
          }
        }
        if (!block_sync_ok(ok)) break;   // the sums are read before the next phase's x lies there
      }
    } else {
      // -------------------------------------------------------------------- a product
      const Share sh = s.share[phase];
      if (sh.count) {
        const bool normed = phase == QKV || phase == GATE_UP || phase == HEADS;
        const int x_row_bytes = sh.chunks * 64 + 64;   // rows 64 bytes apart modulo 128 (an even number of chunks)
        // A thread finishes the result (i, row) of unit j0 of every batch (a batch has at most as many units as there are turns).
        const int columns_log = phase == GATE_UP ? 3 : 4, i = tid & ((1 << columns_log) - 1), turn = tid >> columns_log;
        const int row = turn & ((1 << rows_log) - 1), j0 = turn >> rows_log;
        auto place = [&](int unit) { return ((sh.first + unit * sh.step) << columns_log) + i; };
        const uint2* old = phase == DOWN ? a.middle : a.input;   // the residual that O and down add to
        uint2* fresh = phase == DOWN ? a.input : a.middle;
        const uint32_t old_epoch = epoch, fresh_epoch = phase == DOWN ? epoch + 1 : epoch;
        const bool add_bias = phase == QKV && L.qkv_bias != nullptr, add_residual = phase == O || (phase == DOWN && a.down_splits == 1);
        const float* next_norm = phase == O ? L.norm2 : layer + 1 < a.layers ? layers[layer + 1].norm1 : a.final_norm;
        // What a sum is added to, asked for ahead of it.  A group of 16 rows of the down product whose k range is split: the block
        // of part (group % splits) adds the parts up.
        uint2 before = {};
        float norm = 0.f;
        auto look_up = [&](int unit) {
          if (row < a.rows && unit < sh.count) {
            if (add_bias) before.x = __float_as_uint(__ldg(L.qkv_bias + place(unit)));
            if (add_residual) {
              before = load_packet(old + (size_t)row * a.hidden + place(unit));
              norm = __ldg(next_norm + place(unit));
            }
          }
        };
        look_up(j0);
        const int quads = sh.chunks * 8, mine = (quads * a.rows + THREADS - 1) / THREADS;
        auto take = [&](auto count) {
          if (normed) {
            const uint32_t* src = a.normed + (size_t)(2 * layer + (phase == GATE_UP ? 1 : 0)) * a.norm_stride;
            const float eps = phase == QKV ? L.eps1 : phase == GATE_UP ? L.eps2 : a.final_eps;
            load_x(count, std::true_type(), tid, src, a.hidden / 4, quads, epoch, src + a.rows * a.hidden, x_row_bytes, 0xffffu, eps);
          } else {
            const uint2* src = phase == O ? a.attended : a.act + s.down_first_chunk * 16;
            load_x(count, std::false_type(), tid, src, (phase == O ? a.n_q * HEAD : a.inter) / 4, quads, epoch, nullptr, x_row_bytes,
                   phase == O ? valid_rows : 0xffffu, 0.f);
          }
        };
        if (mine > 4) take(std::integral_constant<int, 12>());
        else take(std::integral_constant<int, 4>());
        if (!block_sync_ok(ok)) break;
        STAMP(phase * 4 + 1)
        // A new value of the residual, and what the norm that reads it needs of it (the 16 threads of a unit's row together).
        auto publish = [&](int row, int at, float v, float weight) {
          const size_t there = (size_t)row * a.hidden + at;
          const unsigned mask = 0xffffu << (lane & 16);
          uint32_t* normed_there = a.normed + (size_t)(2 * layer + (phase == DOWN ? 2 : 1)) * a.norm_stride;
          store_packet(fresh + there, __float_as_uint(v), fresh_epoch);
          store_value(normed_there + there, v * weight);
          float sq = v * v;
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(mask, sq, o);
          if (i == 0) store_value(normed_there + a.rows * a.hidden + there / 16, sq);
        };
        const uint32_t x0 = x_s + min(lane >> 2, a.rows - 1) * x_row_bytes + (lane & 3) * 16;
        const uint32_t w0 = ring + (lane >> 2) * ROW_BYTES + (lane & 3) * 16;
        float* sums = red;
#pragma unroll 1
        for (int first = 0; first < sh.count; first += a.batch_units) {   // batch_units at a time
          const int here = min(a.batch_units, sh.count - first);
#pragma unroll 1
          for (int j = 0; j < here; ++j) {
            // The k order inside a chunk is what 16-byte reads give a thread: thread q of a quad holds k 8q .. 8q + 7, on both sides.
            float acc[2][4] = {};
#pragma unroll 1
            for (int p = 0; p < sh.pieces; ++p) {
              const Slot low = slot;
              slot.step(a.stages);
              const Slot high = slot;
              slot.step(a.stages);
              ok = ok && wait_for(smem_u32(&s.full[low.at]), low.parity, s) &&
                   wait_for(smem_u32(&s.full[high.at]), high.parity, s);
              const int c0 = p * sh.per_piece, chunks = min(sh.per_piece, sh.chunks - c0);
              const uint32_t w_low = w0 + low.at * STAGE, w_high = w0 + high.at * STAGE;
#pragma unroll 3
              for (int c = warp; c < chunks; c += WARPS) {
                const uint4 lo = lds128(w_low + c * 64), hi = lds128(w_high + c * 64), b = lds128(x0 + (c0 + c) * 64);
                mma4(acc[0], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
                mma4(acc[1], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
              }
              __syncwarp();
              if (lane == 0) {
                tc::mbar_arrive(smem_u32(&s.empty[low.at]));
                tc::mbar_arrive(smem_u32(&s.empty[high.at]));
              }
            }
            if ((lane & 3) < MAX_ROWS / 2) {     // the others hold columns beyond the rows
              float* dst = sums + j * UNIT_SUMS + (warp * 16 + (lane >> 2)) * MAX_ROWS + 2 * (lane & 3);
              *reinterpret_cast<float2*>(dst) = make_float2(acc[0][0] + acc[1][0], acc[0][1] + acc[1][1]);
              *reinterpret_cast<float2*>(dst + 8 * MAX_ROWS) = make_float2(acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]);
            }
          }
          block_sync();
          if (row < a.rows && j0 < here) {
            const int at = place(first + j0);
            const size_t there = (size_t)row * a.hidden + at;
            const float* mine = sums + j0 * UNIT_SUMS;
            float v = unit_sum(mine, i, row);
            if (phase == QKV) {
              store_packet(a.qkv + (size_t)row * n_qkv + at, __float_as_uint(v + __uint_as_float(before.x)), epoch);
            } else if (phase == GATE_UP) {
              v = __fdividef(v, 1.0f + __expf(-v)) * unit_sum(mine, i + 8, row);
              const float next = __shfl_down_sync(0xffu << (lane & 24), v, 1);
              if ((i & 1) == 0) store_packet(a.act + ((size_t)row * a.inter + at) / 2, pack_bf16(v, next), epoch);
            } else if (phase == HEADS) {
              a.logits[(size_t)row * a.vocab + at] = v;
            } else if (add_residual) {
              if (before.y >> 16 != old_epoch) {
                uint2 late[1];
                fetch_single(late, 1u, old_epoch, [&](int) { return old + there; });
                before = late[0];
              }
              publish(row, at, v + __uint_as_float(before.x), norm);
            } else {
              store_packet(a.down_part + (size_t)s.down_split * a.rows * a.hidden + there, __float_as_uint(v), epoch);
            }
          }
          if (first + a.batch_units < sh.count) look_up(first + a.batch_units + j0);
          sums = sums == red ? red + a.batch_units * UNIT_SUMS : red;    // the other half: these are still read
        }
        STAMP(phase * 4 + 2)
        if (phase == DOWN && a.down_splits > 1 && row < a.rows) {   // over the parts in their order
#pragma unroll 1
          for (int j = j0; j < sh.count; j += (THREADS >> 4) >> rows_log) {
            if ((sh.first + j * sh.step) % a.down_splits != s.down_split) continue;
            const size_t there = (size_t)row * a.hidden + place(j), part = (size_t)a.rows * a.hidden;
            const float weight = __ldg(next_norm + place(j));
            uint2 v[9] = {};     // the parts, and the residual (whose epoch is the same)
            fetch_single(v, ((1u << a.down_splits) - 1u) | 1u << 8, epoch, [&](int p) { return p < 8 ? a.down_part + p * part + there : old + there; });
            float total = 0.f;
#pragma unroll
            for (int p = 0; p < 8; ++p)
              if (p < a.down_splits) total += __uint_as_float(v[p].x);
            publish(row, place(j), __uint_as_float(v[8].x) + total, weight);
          }
        }
      }
    }
    if (phase == HEADS) break;
    STAMP(phase * 4 + 3)
    if (phase == DOWN) phase = ++layer < a.layers ? QKV : HEADS;
    else ++phase;
  }
  LSE_TL_MARK(3)
}

// The rows' embeddings as the first layer's residual (packets of epoch 1) and what its norm reads; no epoch in every other packet,
// UNSET in the other norms' places.
__global__ void __launch_bounds__(256)
decode_layers_start_kernel(const __nv_bfloat16* __restrict__ table, const int* __restrict__ ids, const float* __restrict__ norm,
                           uint2* __restrict__ input, uint32_t* __restrict__ normed, uint4* __restrict__ rest, long long rest_count,
                           uint4* __restrict__ unset, long long unset_count, int rows, int hidden, int vocab, float scale) {
  pdl_launch_dependents();
  pdl_wait();
  const int stride = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
  for (long long i = first; i < rest_count; i += stride) rest[i] = make_uint4(0u, 0u, 0u, 0u);
  for (long long i = first; i < unset_count; i += stride) unset[i] = make_uint4(UNSET, UNSET, UNSET, UNSET);
  for (int p = first; p < rows * hidden / 2; p += stride) {    // pairs of columns: eight threads hold a group of 16 (hidden % 64 == 0)
    const int row = p / (hidden / 2), column = 2 * (p % (hidden / 2));
    const int id = LSE_CHECKED(ids[row], 0, vocab, -1, LSE_CHECK_TOKEN_ID);
    float2 v = make_float2(0.f, 0.f);
    if (id >= 0 && id < vocab) {
      v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(table + (size_t)id * hidden + column));
      v.x *= scale;
      v.y *= scale;
    }
    input[2 * p] = make_uint2(__float_as_uint(v.x), 1u << 16);
    input[2 * p + 1] = make_uint2(__float_as_uint(v.y), 1u << 16);
    reinterpret_cast<uint2*>(normed)[p] = make_uint2(set_bits(v.x * norm[column]), set_bits(v.y * norm[column + 1]));
    float sq = v.x * v.x + v.y * v.y;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffu << (threadIdx.x & 24), sq, o);
    if ((p & 7) == 0) normed[rows * hidden + p / 8] = p == 0 && lse_decode_layers_withhold ? UNSET : set_bits(sq);
  }
}

constexpr int LSE_DECODE_LAYERS_REFUSED = -3;   // the blocks cannot all be on the GPU at once
constexpr size_t SMEM_LIMIT = 232448;   // 227 KB a block, static shared memory included

struct Plan {
  int stages, down_splits, batch_units, x_bytes;
  size_t smem;
};

// How a step of these sizes is laid out; false: it does not fit, or the sizes are not the kernel's.
bool make_plan(int blocks, int layers, int rows, int hidden, int inter, int n_q, int n_kv, int vocab, Plan* plan) {
  if (rows < 1 || rows > MAX_ROWS || hidden % 64 || inter % 64 || vocab % 16 || hidden <= 0 || inter <= 0 || vocab <= 0) return false;
  if (n_kv < 1 || n_q % n_kv || n_q / n_kv > MAX_HEADS || rows * n_kv > blocks || rows * n_kv > 256) return false;
  const int groups = hidden / 16, k_all = inter / 64;
  if (groups > MAX_DOWN_GROUPS) return false;
  const size_t statics = sizeof(Shared) + MAX_HEADS * Q_STRIDE + 256;
  const int hidden_bytes = rows * (hidden * 2 + 64), attended_bytes = rows * (n_q * HEAD * 2 + 64);
  const int rest = hidden_bytes > attended_bytes ? hidden_bytes : attended_bytes;
  for (int stages = MAX_STAGES; stages >= 4; --stages) {   // as many as fit: what is fetched ahead while the blocks wait for one another
    for (int batch = 4; batch >= 2; batch -= 2) {
      const size_t sums = (size_t)2 * batch * UNIT_SUMS * sizeof(float);
      // The parts of the down product's k range: the fewest tiles for the block that has most, within what the rows' share of
      // the activations may take in shared memory.
      long long best = -1;
      for (int splits = 1; splits <= 8 && splits <= k_all && splits <= blocks; ++splits) {
        const int per = (k_all + splits - 1) / splits, least = blocks / splits;
        if ((k_all + per - 1) / per != splits) continue;                 // a part without tiles
        const int rounds = (groups + least - 1) / least;
        if (rounds > 64) continue;
        const int slice = rows * (per * 128 + 64);
        int x = slice > rest ? slice : rest;
        const int merge = WARPS * MAX_HEADS * HEAD * (int)sizeof(float);   // the attention's sums lie over x and the units' sums
        if (x + (long long)sums < merge) x = merge - (int)sums;
        x = (x + 127) / 128 * 128;
        const size_t smem = (size_t)stages * STAGE + x + sums + layers * sizeof(Layer) + 1024;
        if (smem + statics > SMEM_LIMIT) continue;
        // the time of the block that has most: its weights (2 KB a tile of 64 k), its share of the activations (packets: 256 bytes a
        // row and tile, fetched at about the same rate), and a part more is a sum more to add
        const long long cost = (long long)rounds * per * 2048 + (long long)rows * per * 256 + splits * 2048;
        if (best < 0 || cost < best) {
          best = cost;
          plan->stages = stages; plan->down_splits = splits; plan->batch_units = batch; plan->x_bytes = x; plan->smem = smem;
        }
      }
      if (best >= 0) return true;
    }
  }
  return false;
}

cudaError_t allow(size_t smem) {
  static SmemAllowance allowance;
  return allow_smem(decode_layers_kernel, smem, allowance);
}

int launch(const Args& args, int blocks, size_t smem, cudaStream_t stream) {
  cudaError_t err = allow(smem);
  if (err != cudaSuccess) return (int)err;
  cudaLaunchConfig_t config = {};
  config.gridDim = blocks;
  config.blockDim = THREADS + 64;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeCooperative;
  attribute[0].val.cooperative = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  err = cudaLaunchKernelEx(&config, decode_layers_kernel, args);
  if (err == cudaSuccess) err = cudaGetLastError();
  if (err == cudaErrorCooperativeLaunchTooLarge || err == cudaErrorNotSupported) {   // a process that may use a part of the SMs only
    cudaGetLastError();              // the step goes launch by launch, and is not to meet this error there
    return LSE_DECODE_LAYERS_REFUSED;
  }
  return (int)err;
}

}  // namespace

// Whether a decode step of these sizes can be run by lse_decode_layers on a GPU of `blocks` SMs.
extern "C" int lse_decode_layers_supported(int blocks, int layers, int rows, int hidden, int inter, int n_q, int n_kv, int vocab) {
  Plan plan;
  return layers >= 1 && layers <= MAX_LAYERS && make_plan(blocks, layers, rows, hidden, inter, n_q, n_kv, vocab, &plan) ? 1 : 0;
}

// Whether the current device takes the launch of a step of these sizes: all blocks at once.  Asked once, when a model is built.
extern "C" int lse_decode_layers_fits(int blocks, int layers, int rows, int hidden, int inter, int n_q, int n_kv, int vocab) {
  Plan plan;
  int device = 0, cooperative = 0, sms = 0, a_sm = 0;
  if (layers < 1 || layers > MAX_LAYERS || !make_plan(blocks, layers, rows, hidden, inter, n_q, n_kv, vocab, &plan)) return 0;
  const bool answered = cudaGetDevice(&device) == cudaSuccess &&
                        cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, device) == cudaSuccess &&
                        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && allow(plan.smem) == cudaSuccess &&
                        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a_sm, decode_layers_kernel, THREADS + 64, plan.smem) == cudaSuccess;
  if (!answered) cudaGetLastError();
  return answered && cooperative && (long long)a_sm * sms >= blocks ? 1 : 0;
}

// Bytes of scratch memory of a launch: the packets that blocks exchange, the abort word, and the norms' places.
// offsets (11 values): where each begins, every one 256-byte aligned, and the whole.
extern "C" int lse_decode_layers_scratch(int blocks, int layers, int rows, int hidden, int inter, int n_q, int n_kv, int vocab, long long* offsets) {
  Plan plan;
  if (!make_plan(blocks, layers, rows, hidden, inter, n_q, n_kv, vocab, &plan)) return LSE_ERR_TOO_LARGE;
  const long long residual = (long long)rows * hidden;
  const long long packets[9] = {residual, residual, (long long)rows * (n_q + 2 * n_kv) * HEAD, (long long)rows * n_q * HEAD / 2,
                                (long long)rows * inter / 2, (long long)blocks * MAX_HEADS * HEAD, (long long)blocks * MAX_HEADS * 2,
                                plan.down_splits * residual, 1};
  long long at = 0;
  for (int i = 0; i < 9; ++i) {
    offsets[i] = at;
    at += (packets[i] * 8 + 255) / 256 * 256;
  }
  offsets[9] = at;
  offsets[10] = at + ((2LL * layers + 1) * (residual + residual / 16) * 4 + 255) / 256 * 256;
  return 0;
}

extern "C" int lse_decode_layers_status(void) {
  int value = 0;
  if (cudaMemcpyFromSymbol(&value, lse_decode_layers_error, sizeof(int)) != cudaSuccess) return -1;
  return value;
}
extern "C" int lse_decode_layers_status_async(int* host_dst, cudaStream_t stream) {
  return (int)cudaMemcpyFromSymbolAsync(host_dst, lse_decode_layers_error, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
}
extern "C" int lse_decode_layers_status_reset(void) {
  const int zero = 0;
  return (int)cudaMemcpyToSymbol(lse_decode_layers_error, &zero, sizeof(int));
}
// Test hooks.  spin_limit: attempts of a bounded wait before it gives up (0: the default); withhold != 0: a value that every block
// with a unit of the first product waits for never comes.
extern "C" int lse_decode_layers_test_hooks(unsigned int spin_limit, int withhold) {
  const unsigned int limit = spin_limit ? spin_limit : SPIN_LIMIT;
  cudaError_t err = cudaMemcpyToSymbol(lse_decode_layers_spin_limit, &limit, sizeof(limit));
  if (err != cudaSuccess) return (int)err;
  return (int)cudaMemcpyToSymbol(lse_decode_layers_withhold, &withhold, sizeof(withhold));
}

// One decode step (LSE_DECODE_LAYERS_REFUSED: not taken, nothing of the step has happened).  layer_pointers [layers][9]: qkv, o, gate_up, down, qkv_bias (may be 0), norm1, norm2, keys, values;
// layer_eps [layers][2].  All bfloat16 matrices row-major and 16-byte aligned (gate_up: gate rows, then up rows), norms and
// biases float32.  Every row of the step is a request's next token (segment -1: padding).  logits float32 [rows][vocab].
extern "C" int lse_decode_layers(const long long* layer_pointers, const float* layer_eps, int layers, const void* embedding,
                                 int embedding_rows, float embedding_scale, const void* head, const float* final_norm, float final_eps,
                                 const float* inv_freq, int pairing, const int* token_ids, const int* positions,
                                 const int* segment_of_token, const int* slot_mapping, const int* block_tables, int bt_stride,
                                 int num_segments, int rows, int hidden, int inter, int n_q, int n_kv, int vocab, int page_size,
                                 int num_pages, float scale, void* scratch, float* logits, int blocks, cudaStream_t stream) {
  if (rows <= 0) return 0;
  Plan plan;
  if (layers < 1 || layers > MAX_LAYERS || !make_plan(blocks, layers, rows, hidden, inter, n_q, n_kv, vocab, &plan)) return LSE_ERR_TOO_LARGE;
  if (page_size % 16 || (long long)num_pages * n_kv * page_size > 0x7fffffffLL || ((uintptr_t)head & 15) || ((uintptr_t)scratch & 255))
    return LSE_ERR_BAD_ARGUMENT;
  Args args;
  for (int i = 0; i < layers; ++i) {
    const long long* p = layer_pointers + (size_t)i * 9;
    for (int j = 0; j < 9; ++j)
      if (p[j] & 15) return LSE_ERR_BAD_ARGUMENT;
    Layer& L = args.layer[i];
    L.qkv = (const __nv_bfloat16*)p[0]; L.o = (const __nv_bfloat16*)p[1];
    L.gate_up = (const __nv_bfloat16*)p[2]; L.down = (const __nv_bfloat16*)p[3];
    L.qkv_bias = (const float*)p[4]; L.norm1 = (const float*)p[5]; L.norm2 = (const float*)p[6];
    L.keys = (__nv_bfloat16*)p[7]; L.values = (__nv_bfloat16*)p[8];
    L.eps1 = layer_eps[2 * i]; L.eps2 = layer_eps[2 * i + 1];
    const long long cache_rows = (long long)num_pages * n_kv * page_size;
    if (!tc::make_map_row_groups(&args.maps[i][0], L.keys, cache_rows, HEAD, 16) ||
        !tc::make_map_row_groups(&args.maps[i][1], L.values, cache_rows, HEAD, 16))
      return LSE_ERR_BAD_ARGUMENT;
  }
  long long at[11];
  lse_decode_layers_scratch(blocks, layers, rows, hidden, inter, n_q, n_kv, vocab, at);
  unsigned char* base = (unsigned char*)scratch;
  Common& c = args.common;
  c.head = (const __nv_bfloat16*)head; c.final_norm = final_norm; c.inv_freq = inv_freq;
  c.positions = positions; c.segment_of_token = segment_of_token; c.slot_mapping = slot_mapping;
  c.block_tables = block_tables;
  uint2** parts[8] = {&c.input, &c.middle, &c.qkv, &c.attended, &c.act, &c.part_o, &c.part_ml, &c.down_part};
  for (int i = 0; i < 8; ++i) *parts[i] = (uint2*)(base + at[i]);
  c.abort = (unsigned*)(base + at[8]);
  c.normed = (uint32_t*)(base + at[9]);
  c.norm_stride = rows * hidden + rows * hidden / 16;
  c.logits = logits;
  c.layers = layers; c.rows = rows; c.hidden = hidden; c.inter = inter; c.n_q = n_q; c.n_kv = n_kv;
  c.vocab = vocab; c.page_size = page_size; c.bt_stride = bt_stride; c.num_pages = num_pages;
  c.num_slots = num_pages * page_size; c.num_segments = num_segments; c.pairing = pairing;
  c.down_splits = plan.down_splits; c.batch_units = plan.batch_units; c.x_bytes = plan.x_bytes;
  c.stages = plan.stages;
  c.final_eps = final_eps; c.scale_log2e = scale * LOG2E;
  cudaError_t err = lse_launch(decode_layers_start_kernel, 2 * blocks, 256, 0, stream, (const __nv_bfloat16*)embedding, token_ids,
                               args.layer[0].norm1, c.input, c.normed, (uint4*)c.middle, (at[9] - at[1]) / 16,
                               (uint4*)(c.normed + c.norm_stride), 2LL * layers * c.norm_stride / 4, rows, hidden, embedding_rows, embedding_scale);
  if (err != cudaSuccess) return (int)err;
  return launch(args, blocks, plan.smem, stream);
}

#ifdef LSE_TRACE
// The stamps of the last launch, [STAMP_BLOCKS][STAMPS].
extern "C" int lse_decode_layers_stamps(unsigned long long* host_out) {
  return (int)cudaMemcpyFromSymbol(host_out, lse_decode_layers_stamp, sizeof(lse_decode_layers_stamp));
}
#endif
