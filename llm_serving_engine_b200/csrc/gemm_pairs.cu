// bfloat16 matrix products of many rows on pairs of SMs (tcgen05, cta_group::2), with the feed-forward's gate inside or over
// groups of rows with weights of their own (a mixture of experts).
//
//   gated:  out[t, n] = scale[t] * gate_mul(sum_k x[t, k] w[g0 + n, k], sum_k x[t, k] w[u0 + n, k])
//   plain:  out[t, n] = sum_k x[t, k] w[r0 + n, c0 + k]
//
// A pair of blocks owns 256 rows of w (the M side of the instruction: 128 lanes of tensor memory in each block) and up to 256
// rows of x (the N side; a group's last tile in steps of 32).  Each block brings its own half of both operands with TMA
// (128-byte swizzle, six stages of 64 k), one thread of the even block issues the instructions for both, the sums lie in two
// buffers of tensor memory, and eight warps finish one tile while the next one's products run.  Gated, a block's 128 rows of w
// are 64 rows of the gate and the 64 rows of the up projection beside them: the warps that read the up half hand it to those
// that read the gate half through shared memory, the products' sums never leave the SM, and no kernel has to read them
// (2,048 rows x 17,920 columns: 73 MB written and read again, 18 us of 95), and
// gate and up are not rounded to bfloat16 on the way.
//
// What bounds it: an SM takes its operands from the L2 at 64 bytes a clock when the tensor cores run at full rate, which is about
// what it can take: 2,048 x 18,944 x 8,192 413 us, 1,539 TFLOP/s (the library's, whose pairs own 512 x 256 and read a quarter
// less, 383; such a tile leaves no second buffer of sums, and short k ranges are what this kernel is for).  Gated, 2,048 x 1,536 x
// 8,960: 87.5 us against 94.2 of the library's product and the activation kernel behind it.  A mixture of eight experts of 2,688
// and a shared one of 2,816 columns over 2,048 rows of 2,048: 118 + 64 us against 190 for the library's products and 27 for the
// activations.
//
// The grid is persistent: pair p takes tiles p, p + pairs, ...; a group's row tiles follow one another under the same rows of w.
// Every wait is bounded; a wait that gives up sets lse_gemm_pairs_error, and what the launch wrote is not to be used.  Both blocks of
// the pair then stay until what is in flight has landed, whichever of their threads gave up.
#include <atomic>

#include "gate_act.cuh"
#include "smem_allowance.cuh"
#include "tcgen05.cuh"

namespace {
using namespace tc;
constexpr int BLOCK_K = 64, UMMA_K = 16, STAGES = 6, HALF_TILE = 128;       // rows of a block's half of either operand
constexpr uint32_t OPERAND = HALF_TILE * BLOCK_K * 2, STAGE = 2 * OPERAND;
constexpr int MAX_GROUPS = 256, CHUNK = 16;                                  // columns of the sums that a warp takes at a time
constexpr int FINISHERS = 8;                                                 // warps that finish tiles
constexpr uint32_t ACC_COLS = 256;

__device__ int lse_gemm_pairs_error;
std::atomic<int> withhold{0};  // test hook

struct Source {                // rows of x, and where their results go
  CUtensorMap rows[4];         // boxes of 32, 64, 96 and 128 rows
  void* out;
  long long ld_out;
  const float* scale;          // by row, or null
  int out_f32;
  float limit;
};

struct Args {
  CUtensorMap weights;         // boxes of 64 rows (gated) or 128
  Source source[2];
  // group g < routed: rows offsets[g - 1] .. offsets[g] of source 0 and the g-th of equally large pieces of w; the last group,
  // if `whole` rows are given: all rows of source `whole_source` and the piece behind those
  const int* offsets;
  int routed, whole, whole_source;
  int columns, whole_columns;             // results a row
  long long w_rows, w_columns;            // from one group's piece to the next one's: rows or columns of w
  int k, whole_k;
};

struct Group {
  int lo, hi, w_row, w_column, columns, k_blocks, source, tile0, row_tiles, rows_a_tile, w_tiles;
};

struct Shared {
  unsigned long long full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  Group group[MAX_GROUPS + 1];
  int groups, tiles, abort;
  uint32_t tmem;
  float hand[4][2][CHUNK][32];            // [pair of warps][buffer][column][lane]
};

__device__ __forceinline__ uint32_t block_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// TMA load whose bytes count on the even block's barrier (the same offset in its shared memory).
__device__ __forceinline__ void tma_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
               ::"r"(dst), "l"(map), "r"(bar & 0xFEFFFFFFu), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// One arrival on the barrier of this offset in both blocks when all products issued so far have finished.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
               ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void arrive_even(uint32_t bar) {   // on the even block's barrier
  asm volatile("{\n\t.reg .b32 there;\n\tmapa.shared::cluster.u32 there, %0, 0;\n\t"
               "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [there];\n\t}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}

__device__ __forceinline__ void set_abort_there(uint32_t flag, int rank) {   // the other block's
  asm volatile("{\n\t.reg .b32 there;\n\tmapa.shared::cluster.u32 there, %0, %1;\n\tst.shared::cluster.u32 [there], %2;\n\t}\n"
               ::"r"(flag), "r"(rank), "r"(1) : "memory");
}

// Whether it went well for all threads of the warps that finish tiles (they meet at barriers: all go on or none).
__device__ __forceinline__ bool together(bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 5, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
               : "=r"(all) : "r"((uint32_t)ok) : "memory");
  return all != 0;
}

// Rows of a tile of `count` rows of x, in steps of 32, what the paired instruction takes: full tiles and a rest, or even tiles,
// whichever costs less.  A tile of few rows is bound by its rows of w (about what 140 rows take): 522 rows go as three tiles of 192,
// 1,349 as five of 256 and one of 96.
__host__ __device__ __forceinline__ int rows_of_tiles(int count) {
  const int tiles = (count + 255) / 256, even = ((count + tiles - 1) / tiles + 31) / 32 * 32, rest = count - (tiles - 1) * 256;
  return tiles * (even > 140 ? even : 140) < (tiles - 1) * 256 + (rest > 140 ? rest : 140) ? even : 256;
}
__host__ __device__ __forceinline__ int rows_of_tile(int left, int rows_a_tile) {     // of a tile with `left` rows from its first one on
  const int rows = (left + 31) / 32 * 32;
  return rows < rows_a_tile ? rows : rows_a_tile;
}
__host__ __device__ __forceinline__ int box_of(int rows) { return (rows / 2 + 31) / 32; }   // half a tile's rows, in boxes of 32

// The groups' rows, tiles and pieces of w, in their order; one warp, once a block, 32 groups at a time.  (On one thread the prologue
// of 256 groups took 40 us.)
template <bool GATED>
__device__ __noinline__ void lay_out(const Args& a, Shared& s, int lane) {
  constexpr int W_TILE = GATED ? HALF_TILE : 2 * HALF_TILE;    // results a tile
  int tiles = 0, count = 0, before = 0;
  auto put = [&](int at, int tile0, int lo, int hi, int index, int columns, int k, int source) {
    Group g;
    g.lo = lo; g.hi = hi; g.source = source; g.columns = columns;
    g.w_row = (int)(index * a.w_rows); g.w_column = (int)(index * a.w_columns);
    g.k_blocks = (k + BLOCK_K - 1) / BLOCK_K;
    g.row_tiles = (hi - lo + 255) / 256;
    g.rows_a_tile = rows_of_tiles(hi - lo);
    g.tile0 = tile0;
    g.w_tiles = (columns + W_TILE - 1) / W_TILE;
    s.group[at] = g;
    return g.row_tiles * g.w_tiles;
  };
  if (a.whole) {   // the largest first
    if (lane == 0) tiles = put(0, 0, 0, a.whole, a.routed, a.whole_columns, a.whole_k, a.whole_source);
    tiles = __shfl_sync(0xffffffffu, tiles, 0);
    count = 1;
  }
  const int w_tiles = (a.columns + W_TILE - 1) / W_TILE;
  for (int first = 0; first < a.routed; first += 32) {
    const int g = first + lane, hi = g < a.routed ? a.offsets[g] : 0;
    int lo = __shfl_up_sync(0xffffffffu, hi, 1);
    if (lane == 0) lo = before;
    before = __shfl_sync(0xffffffffu, hi, 31);
    const bool some = g < a.routed && hi > lo;
    const int mine = some ? (hi - lo + 255) / 256 * w_tiles : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += up;
    }
    const unsigned present = __ballot_sync(0xffffffffu, some);
    if (some) put(count + __popc(present & ((1u << lane) - 1u)), tiles + upto - mine, lo, hi, g, a.columns, a.k, 0);
    tiles += __shfl_sync(0xffffffffu, upto, 31);
    count += __popc(present);
  }
  if (lane == 0) {
    s.groups = count;
    s.tiles = tiles;
  }
}

struct Tile {
  int group, w_tile, row0, rows;      // first row of x; rows, rounded up to what the paired instruction takes (32)
};
__device__ __forceinline__ Tile find_tile(const Shared& s, int tile, int from) {
  int g = from;
  while (g + 1 < s.groups && s.group[g + 1].tile0 <= tile) ++g;
  const Group& G = s.group[g];
  // row tiles follow one another under the same rows of w; the group's last, which may be smaller, come behind all others, so that
  // every pair gets its share of both
  const int rest = tile - G.tile0, others = G.row_tiles - 1, w_tile = rest < others * G.w_tiles ? rest / others : rest - others * G.w_tiles;
  const int row_tile = rest < others * G.w_tiles ? rest % others : others, row0 = G.lo + row_tile * G.rows_a_tile;
  return {g, w_tile, row0, rows_of_tile(G.hi - row0, G.rows_a_tile)};
}

template <bool GATED, int ACT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(128 + 32 * FINISHERS, 1) gemm_pairs_kernel(const __grid_constant__ Args a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ Shared s;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)block_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(smem_u32(&s.full[i]), 1);
      mbar_init(smem_u32(&s.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&s.acc_full[i]), 1);
      mbar_init(smem_u32(&s.acc_empty[i]), 2 * FINISHERS);     // of both blocks
    }
    s.abort = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    if (a.routed) pdl_wait();                      // the groups' ranges are an earlier kernel's
    __syncwarp();
    lay_out<GATED>(a, s, lane);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&s.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  cluster_sync();
  fence_after_sync();
  const uint32_t tmem = s.tmem;
  volatile int* abort = &s.abort;
  const int tiles = s.tiles;

  if (warp == 0) {
    if (lane == 0) {               // brings this block's halves of both operands
      int stage = 0, g = 0;
      uint32_t parity = 0;
      bool ok = true;
      for (int tile = pair; tile < tiles && ok; tile += pairs) {
        const Tile t = find_tile(s, tile, g);
        g = t.group;
        const Group& G = s.group[g];
        const int half = t.rows >> 1, box = box_of(t.rows);
        const CUtensorMap* rows = &a.source[G.source].rows[box - 1];
        const uint32_t bytes = OPERAND + (uint32_t)box * 32u * BLOCK_K * 2u;
        const int y = t.row0 + rank * half;
        auto bring_w = [&](int kb, int at) {
          const uint32_t full = smem_u32(&s.full[at]), dst = ring + at * STAGE;
          if (rank == 0) mbar_expect_tx(full, 2u * bytes);
          const int x = G.w_column + kb * BLOCK_K;
          if (GATED) {
            const int w = G.w_row + t.w_tile * HALF_TILE + rank * 64;
            tma_load_pair(dst, &a.weights, full, x, w);
            tma_load_pair(dst + OPERAND / 2, &a.weights, full, x, w + G.columns);
          } else {
            tma_load_pair(dst, &a.weights, full, x, G.w_row + (2 * t.w_tile + rank) * HALF_TILE);
          }
        };
        auto bring_x = [&](int kb, int at) { tma_load_pair(ring + at * STAGE + OPERAND, rows, smem_u32(&s.full[at]), kb * BLOCK_K, y); };
        int kb = 0;
        if (tile == pair) {        // w does not come from the kernels before: its first tiles travel while they end
          const int early = min(STAGES, G.k_blocks);
          for (int i = 0; i < early; ++i) bring_w(i, i);
          pdl_wait();
          for (; kb < early; ++kb) bring_x(kb, kb);
          stage = early % STAGES;
          parity = early == STAGES;
        }
        for (; kb < G.k_blocks; ++kb) {
          ok = mbar_wait(smem_u32(&s.empty[stage]), parity ^ 1u, abort, &lse_gemm_pairs_error);
          if (!ok) break;
          bring_w(kb, stage);
          bring_x(kb, stage);
          if (++stage == STAGES) { stage = 0; parity ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {  // issues the products of both blocks
      int stage = 0, g = 0, buffer = 0;
      uint32_t parity = 0, buffer_parity = 0;
      bool ok = true;
      for (int tile = pair; tile < tiles && ok; tile += pairs) {
        const Tile t = find_tile(s, tile, g);
        g = t.group;
        const uint32_t idesc = instr_desc_bf16(256, t.rows, false, false);
        const int k_blocks = s.group[g].k_blocks;
        ok = mbar_wait(smem_u32(&s.acc_empty[buffer]), buffer_parity ^ 1u, abort, &lse_gemm_pairs_error);
        fence_after_sync();
        for (int kb = 0; kb < k_blocks && ok; ++kb) {
          ok = mbar_poll(smem_u32(&s.full[stage]), parity, abort, &lse_gemm_pairs_error);
          if (!ok) break;
          fence_after_sync();
          const uint32_t src = ring + stage * STAGE;
#pragma unroll
          for (int kk = 0; kk < BLOCK_K / UMMA_K; ++kk)
            umma_pair(tmem + buffer * ACC_COLS, smem_desc_k_major(src + kk * UMMA_K * 2),
                      smem_desc_k_major(src + OPERAND + kk * UMMA_K * 2), idesc, (kb | kk) != 0 ? 1u : 0u);
          commit_pair(smem_u32(&s.empty[stage]));
          if (++stage == STAGES) { stage = 0; parity ^= 1u; }
        }
        if (ok) commit_pair(smem_u32(&s.acc_full[buffer]));
        buffer ^= 1;
        if (buffer == 0) buffer_parity ^= 1u;
      }
      if (!ok) set_abort_there(smem_u32(&s.abort), 1);   // the odd block's waits need not run out themselves
    }
    __syncwarp();
  } else if (warp >= 4) {          // finish the tiles: a warp reads 32 lanes and half of the columns
    const int quarter = warp & 3, half = (warp - 4) >> 2, hand = (quarter & 1) + 2 * half;
    int g = 0, buffer = 0;
    uint32_t buffer_parity = 0;
    bool ok = true;
    pdl_wait();
    for (int tile = pair; tile < tiles && ok; tile += pairs) {
      const Tile t = find_tile(s, tile, g);
      g = t.group;
      const Group& G = s.group[g];
      const Source& S = a.source[G.source];
      const long long ld = S.ld_out;
      const int columns = t.rows >> 1, begin = half * columns, rows = min(columns, G.hi - t.row0 - begin);
      ok = together(mbar_wait(smem_u32(&s.acc_full[buffer]), buffer_parity, abort, &lse_gemm_pairs_error));
      fence_after_sync();
      const uint32_t from = tmem + buffer * ACC_COLS + begin + ((uint32_t)(quarter * 32) << 16);
      const int n = GATED ? t.w_tile * HALF_TILE + rank * 64 + (quarter & 1) * 32 + lane : (2 * t.w_tile + rank) * HALF_TILE + quarter * 32 + lane;
      const bool mine = n < G.columns && ok;
      const long long first = (long long)(t.row0 + begin) * ld + n;
      uint32_t r[2][CHUNK];
      tmem_ld16(from, r[0]);
      if (GATED) {
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(S.out) + first;
        const float* scale = S.scale == nullptr ? nullptr : S.scale + t.row0 + begin;
        const float limit = S.limit;
        // The warp of the gate's lanes finishes the first columns of a chunk, the warp of the up projection's the others: each
        // hands the other what that needs.
        const bool up = quarter >= 2;
        constexpr int PART = CHUNK / 2;
        auto chunk = [&](const uint32_t (&v)[CHUNK], int c0, int turn) {
          float(&there)[CHUNK][32] = s.hand[hand][turn];
#pragma unroll
          for (int c = 0; c < PART; ++c) {
            if (up) there[c][lane] = __uint_as_float(v[c]);
            else there[PART + c][lane] = __uint_as_float(v[PART + c]);
          }
          // One meeting a chunk: what is written two chunks on was read before the next one's meeting.
          asm volatile("bar.sync %0, 64;\n" ::"r"(1 + hand) : "memory");
          float y[PART];
#pragma unroll
          for (int c = 0; c < PART; ++c) {
            const float other = there[up ? PART + c : c][lane], own = __uint_as_float(up ? v[PART + c] : v[c]);
            y[c] = gate_mul<ACT, true>(up ? other : own, up ? own : other, limit);
          }
          const int at = c0 + (up ? PART : 0), here = rows - at;
          if (mine) {
            __nv_bfloat16* dst = out + at * ld;
#pragma unroll
            for (int c = 0; c < PART; ++c, dst += ld)
              if (c < here) {
                float v = y[c];
                if (scale != nullptr) {
                  const float factor = __ldg(scale + at + c);
                  v = factor == 0.f ? 0.f : factor * v;
                }
                *dst = __float2bfloat16_rn(v);
              }
          }
        };
        for (int c0 = 0; c0 < columns; c0 += 2 * CHUNK) {
          tmem_ld_wait();
          if (c0 + CHUNK < columns) tmem_ld16(from + c0 + CHUNK, r[1]);
          chunk(r[0], c0, 0);
          if (c0 + CHUNK < columns) {
            tmem_ld_wait();
            if (c0 + 2 * CHUNK < columns) tmem_ld16(from + c0 + 2 * CHUNK, r[0]);
            chunk(r[1], c0 + CHUNK, 1);
          }
        }
      } else {
        const bool f32 = S.out_f32 != 0;
        void* out = S.out;
        auto chunk = [&](const uint32_t (&v)[CHUNK], int c0) {
          if (!mine) return;
          const int here = rows - c0;
          if (f32) {
            float* dst = reinterpret_cast<float*>(out) + first + c0 * ld;
#pragma unroll
            for (int c = 0; c < CHUNK; ++c, dst += ld)
              if (c < here) *dst = __uint_as_float(v[c]);
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out) + first + c0 * ld;
#pragma unroll
            for (int c = 0; c < CHUNK; ++c, dst += ld)
              if (c < here) *dst = __float2bfloat16_rn(__uint_as_float(v[c]));
          }
        };
        for (int c0 = 0; c0 < columns; c0 += 2 * CHUNK) {
          tmem_ld_wait();
          if (c0 + CHUNK < columns) tmem_ld16(from + c0 + CHUNK, r[1]);
          chunk(r[0], c0);
          if (c0 + CHUNK < columns) {
            tmem_ld_wait();
            if (c0 + 2 * CHUNK < columns) tmem_ld16(from + c0 + 2 * CHUNK, r[0]);
            chunk(r[1], c0 + CHUNK);
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_even(smem_u32(&s.acc_empty[buffer]));
      buffer ^= 1;
      if (buffer == 0) buffer_parity ^= 1u;
    }
  }
  fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && s.abort) set_abort_there(smem_u32(&s.abort), rank ^ 1);
  cluster_sync();                  // the other block may still count on this one's barriers, and the products on its operands
  if (s.abort) {                   // loads and products in flight end (200 us: they take some) before either block leaves
    if (threadIdx.x == 0) for (int i = 0; i < 2000; ++i) __nanosleep(100);
    __syncthreads();
    cluster_sync();
  }
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

// Tensor map of bfloat16 rows `pitch` elements apart; box = [box_rows, 64 columns], 128-byte swizzle.
bool make_rows_map(CUtensorMap* map, const void* ptr, long long rows, long long cols, long long pitch, int box_rows) {
  EncodeTiledFn fn = encode_tiled();
  if (fn == nullptr || rows <= 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BLOCK_K, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr size_t SMEM = (size_t)STAGES * STAGE + 1024;

template <bool GATED, int ACT>
cudaError_t allow() {
  static SmemAllowance allowance;
  return allow_smem(gemm_pairs_kernel<GATED, ACT>, SMEM, allowance);
}

template <bool GATED, int ACT>
int launch(const Args& args, int blocks, cudaStream_t stream) {
  cudaError_t err = allow<GATED, ACT>();
  if (err != cudaSuccess) return (int)err;
  err = lse_launch(gemm_pairs_kernel<GATED, ACT>, blocks, 128 + 32 * FINISHERS, SMEM, stream, args);
  if (err != cudaSuccess) return (int)err;
  return (int)cudaGetLastError();
}
}  // namespace

// The kernels loaded on the current device and allowed their shared memory, ahead of the first launch.
extern "C" int lse_gemm_pairs_prepare(void) {
  const cudaError_t errors[] = {allow<false, 0>(), allow<true, 0>(), allow<true, 1>(), allow<true, 2>(), allow<true, 3>()};
  for (cudaError_t err : errors)
    if (err != cudaSuccess) return (int)err;
  return 0;
}

extern "C" int lse_gemm_pairs_status(void) {
  int value = 0;
  if (cudaMemcpyFromSymbol(&value, lse_gemm_pairs_error, sizeof(int)) != cudaSuccess) return -1;
  return value;
}
extern "C" int lse_gemm_pairs_status_async(int* host_dst, cudaStream_t stream) {
  return (int)cudaMemcpyFromSymbolAsync(host_dst, lse_gemm_pairs_error, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
}
extern "C" int lse_gemm_pairs_status_reset(void) {
  const int zero = 0;
  return (int)cudaMemcpyToSymbol(lse_gemm_pairs_error, &zero, sizeof(int));
}
// Test hook.  withheld != 0: launches bring half of every box of x's rows, so that the wait for the rest gives up (after some
// tenths of a second: the waits' limits are constants.  As an argument of the launch they made 2,048 x 1,536 x 8,960 take 96.3 us, not 93.2).
extern "C" int lse_gemm_pairs_test_hook(int withheld) {
  withhold = withheld;
  return 0;
}

// Results of groups of rows, each with its own weights, and (whole_rows > 0) of all rows of another tensor with the weights behind
// those.  x [x_rows, k] and whole_x [whole_rows, whole_k] bfloat16, rows ld elements apart; offsets int32 [routed] ends of
// the groups' rows in x (routed 0: none).  w bfloat16 [w_total_rows, w_total_columns], rows ld_w apart.
// act 0 .. 3: gated (see gate_act.cuh): a group's piece is 2 * columns rows of w, gate then up; act -1: plain: a group's piece is
// all rows and k columns of w, from column g * k on.  out bfloat16 (out_f32, whole_out_f32: float32; plain only).
// blocks: SMs of the GPU.  k, ld and the pieces' columns multiples of 8, 16-byte aligned; pieces of columns multiples of 64 wide.
extern "C" int lse_gemm_pairs(const void* x, long long x_rows, long long ld_x, const int* offsets, int routed, int columns, int k, void* out,
                              long long ld_out, int out_f32, float limit, const void* whole_x, int whole_rows, long long ld_whole,
                              int whole_columns, int whole_k, void* whole_out, long long ld_whole_out, int whole_out_f32,
                              const float* whole_scale, float whole_limit, const void* w, long long w_total_rows,
                              long long w_total_columns, long long ld_w, int act, int blocks, cudaStream_t stream) {
  if (routed < 0 || routed > MAX_GROUPS || act < -1 || act > 3 || blocks < 2) return LSE_ERR_BAD_ARGUMENT;
  if ((routed && (x_rows <= 0 || x_rows > 0x7fffffff)) || whole_rows < 0) return LSE_ERR_BAD_ARGUMENT;
  if (!routed && !whole_rows) return 0;
  // whole 16-byte pieces (the tensor maps ask for aligned rows themselves)
  if (ld_w % 8 || (routed && (k % 8 || ld_x % 8)) || (whole_rows && (whole_k % 8 || ld_whole % 8))) return LSE_ERR_BAD_ARGUMENT;
  const bool gated = act >= 0;
  Args args = {};
  if (!make_rows_map(&args.weights, w, w_total_rows, w_total_columns, ld_w, gated ? 64 : 128)) return LSE_ERR_BAD_ARGUMENT;
  // the boxes that the tiles of all rows take: every tile but the last has rows_a_tile rows
  const int a_tile = whole_rows ? rows_of_tiles(whole_rows) : 32;
  const int first_box = box_of(rows_of_tile(whole_rows, a_tile)), last_box = whole_rows ? box_of(rows_of_tile((whole_rows - 1) % a_tile + 1, a_tile)) : 0;
  const int box_rows = withhold ? 16 : 32;
  for (int box = 1; box <= 4; ++box) {
    if (routed && !make_rows_map(&args.source[0].rows[box - 1], x, x_rows, k, ld_x, box_rows * box)) return LSE_ERR_BAD_ARGUMENT;
    if (whole_rows && (box == first_box || box == last_box) && !make_rows_map(&args.source[1].rows[box - 1], whole_x, whole_rows, whole_k, ld_whole, box_rows * box)) return LSE_ERR_BAD_ARGUMENT;
  }
  if (!gated && routed && k % BLOCK_K) return LSE_ERR_BAD_ARGUMENT;      // a group's last k would meet the next one's weights
  args.source[0].out = out; args.source[0].ld_out = ld_out; args.source[0].out_f32 = out_f32; args.source[0].limit = limit;
  args.source[1].out = whole_out; args.source[1].ld_out = ld_whole_out; args.source[1].out_f32 = whole_out_f32;
  args.source[1].limit = whole_limit; args.source[1].scale = whole_scale;
  args.offsets = offsets; args.routed = routed; args.whole = whole_rows; args.whole_source = 1;
  args.columns = columns; args.whole_columns = whole_columns; args.k = k; args.whole_k = whole_k;
  args.w_rows = gated ? 2LL * columns : 0; args.w_columns = gated ? 0 : k;
  const long long w_tile = gated ? HALF_TILE : 2 * HALF_TILE;
  long long tiles = routed ? (x_rows / 256 + routed) * ((columns + w_tile - 1) / w_tile) : 0;
  if (whole_rows) tiles += (whole_rows + 255) / 256 * ((whole_columns + w_tile - 1) / w_tile);
  const int grid = (int)(2 * tiles < blocks ? 2 * tiles : blocks / 2 * 2);
  switch (act) {
    case -1: return launch<false, 0>(args, grid, stream);
    case 0: return launch<true, 0>(args, grid, stream);
    case 1: return launch<true, 1>(args, grid, stream);
    case 2: return launch<true, 2>(args, grid, stream);
    default: return launch<true, 3>(args, grid, stream);
  }
}
