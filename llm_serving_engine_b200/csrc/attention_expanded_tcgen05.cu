// Latent attention over portions of prompts with keys and values made from the cached latent once for all rows
// (bfloat16, heads of 128 unrotated and 64 rotated values, values of 128).
//
// attention_latent_mma.cu attends to the cached rows themselves: a score costs 512 + 64 multiply-adds and a weight 512, for
// every row and head.  With many rows it is cheaper to make each head's key (128) and value (128) of every cached row first,
// one product over the rows, and to pay 192 and 128 a pair.  Two kernels, the product between them:
//
//   gather      copies the rows that the step's requests may read from their pages into one tensor, request by request, each
//               request's rows rounded up to whole key tiles with zeros (a tile never meets another request's rows); a latent
//               that is not finite becomes zeros with NaN in place of its rotated values
//   attention   the kernel of attention_tcgen05.cu on these: a block takes 128 rows of one request and one head; key tiles of
//               64 go alternately to two groups of four softmax warps.  A score product takes 128 columns of the head's key
//               and the 64 rotated ones that all heads share (read from the gathered rows), so that a key tile is 24 KB;
//               three key and value stages are shared by the groups, and a group has two score accumulators, so that its
//               next scores are made while it works on the last.
//
// 2,048 rows, 16 heads: 39.5 us (544 TFLOP/s of the 320 multiply-adds a pair), bounded by the softmax threads' exponentials
// and issue slots like the kernel it follows; over the latent rows themselves 611 us.
//
// Every wait is bounded (see tcgen05.cuh); lse_attention_expanded_status() reports one that gave up, and contexts on the
// device that ask for more rows than the host made room for (the rows beyond would be zeros, and count as keys).
#include "smem_allowance.cuh"
#include "tcgen05.cuh"

LSE_CHECK_DEFINE(lse_check_attention_expanded)

namespace {
using namespace tc;

constexpr int BM = 128, BN = 64;          // rows of a block, keys of a tile
constexpr int GROUPS = 2, GROUP_THREADS = 128, STAGES = 3;
constexpr int MMA_WARP = 8, LOADER_WARP = 9, PV_WARP = 10, V_LOADER_WARP = 11, THREADS = 384;
constexpr int D = 128, ROT = 64;          // values of a head: unrotated (and of its value), rotated
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.0f, REDO_STEP = 64.0f;      // in powers of two
constexpr uint32_t Q_BOX = BM * 128, KV_BOX = BN * 128;      // a box of 64 bfloat16 columns
constexpr uint32_t Q_BYTES = 3 * Q_BOX, K_BYTES = 3 * KV_BOX, V_BYTES = 2 * KV_BOX, P_BYTES = BM * 128;
constexpr size_t SMEM = 1024 + Q_BYTES + STAGES * (K_BYTES + V_BYTES) + GROUPS * P_BYTES + GROUPS * 256 * 4 + 256;

constexpr int TOO_MANY_ROWS = 2;      // in the error word: the requests hold more rows than were to be gathered (1: a wait gave up)
__device__ int lse_attn_expanded_error;

// barriers: stages of keys and values (full, empty), scores of a group (two accumulators: full, read), probabilities, outputs
enum Bar { B_Q = 0, B_KF = 1, B_KE = 4, B_VF = 7, B_VE = 10, B_SF = 13, B_SE = 17, B_PF = 21, B_OD = 23, B_COUNT = 25 };

__device__ __forceinline__ float exp2_fast(float x) {   // 2^x, 2^-inf = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void pair_barrier(int quarter) {   // the warps of the two groups that own the same 32 rows
  asm volatile("bar.sync %0, %1;\n" ::"r"(1 + quarter), "r"(64) : "memory");
}
// A request's first gathered position and its gathered rows (whole tiles).
__device__ __forceinline__ int first_kept(int first_position, int window) { return window > 0 ? max(0, first_position + 1 - window) : 0; }
__device__ __forceinline__ int padded_rows(int context, int first_position, int window) {
  return context <= 0 ? 0 : (context - first_kept(first_position, window) + BN - 1) / BN * BN;
}
// First gathered row of request `seg` (a warp's work; the same in every lane).
__device__ __forceinline__ int rows_before(const int* __restrict__ first, const int* __restrict__ context, int window, int seg) {
  int sum = 0;
  for (int s = threadIdx.x & 31; s < seg; s += 32) sum += padded_rows(context[s], first[s], window);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

// Not zero if one of two bfloat16 numbers is infinite or NaN (an exponent of ones: it carries into the sign when it is raised by one).
__device__ __forceinline__ uint32_t not_finite(uint32_t two) { return ((two & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }

// rows[r] for r < capacity: a warp a row; rows of no request, and those that round a request up, are zeros.
__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ cache, const int* __restrict__ block_tables, int bt_stride,
                     const int* __restrict__ first, const int* __restrict__ context, int num_segments, int width,
                     int page_size, int num_pages, int window, __nv_bfloat16* __restrict__ rows, int capacity) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= capacity) return;
  int seg = -1, local = 0, before = 0;
  for (int base = 0; base < num_segments && seg < 0; base += 32) {      // 32 requests at a time
    const int s = base + lane;
    const int mine = s < num_segments ? padded_rows(context[s], first[s], window) : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned vote = __ballot_sync(0xffffffffu, mine > 0 && r >= before + upto - mine && r < before + upto);
    if (vote) {
      const int src = __ffs(vote) - 1;
      seg = base + src;
      local = r - before - __shfl_sync(0xffffffffu, upto - mine, src);
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  pdl_wait();      // the step's own rows come from the kernel before
  if (blockIdx.x == 0 && threadIdx.x < 32) {      // capacity was fixed on the host (a captured step's when it was captured)
    const int wanted = rows_before(first, context, window, num_segments);
    if (threadIdx.x == 0 && wanted > capacity) atomicExch(&lse_attn_expanded_error, TOO_MANY_ROWS);
  }
  const __nv_bfloat16* src = nullptr;
  if (seg >= 0) {
    const int pos = first_kept(first[seg], window) + local;
    if (pos < context[seg]) {
      const int page = LSE_CHECKED(block_tables[(size_t)seg * bt_stride + pos / page_size], 0, num_pages, 0, LSE_CHECK_TABLE_ENTRY);
      src = cache + ((size_t)page * page_size + pos % page_size) * width;
    }
  }
  uint32_t broken = 0;
  for (int base = lane * 8; base < width; base += 4 * 256) {      // all pieces of a row of up to 1,024 values on their way together
    uint4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = src && base + 256 * i < width ? *reinterpret_cast<const uint4*>(src + base + 256 * i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = base + 256 * i;
      if (c >= width) continue;
      *reinterpret_cast<uint4*>(rows + (size_t)r * width + c) = v[i];
      broken |= c < width - ROT ? not_finite(v[i].x) | not_finite(v[i].y) | not_finite(v[i].z) | not_finite(v[i].w) : 0u;
    }
  }
  // A latent that is not finite makes NaN of every row that attends to it, and must not reach those that do not: the values made
  // of it would, as hidden keys of a tile have no weight but are multiplied by it.  So it has finite keys and values, and NaN
  // where the scores are made, which hidden keys do not have.
  if (__any_sync(0xffffffffu, broken != 0)) {
    for (int c = lane * 8; c < width; c += 256) {
      const uint32_t x = c < width - ROT ? 0u : 0x7fc07fc0u;
      *reinterpret_cast<uint4*>(rows + (size_t)r * width + c) = make_uint4(x, x, x, x);
    }
  }
}

// map_q: [rows][heads][128]; map_qr: [rows][heads][rank + 64], the rotated values behind column `rank`; map_kv: [gathered
// rows][2 own_heads][128], keys and then values of the heads first_head .. first_head + own_heads - 1, those that this launch
// works on; map_kr: the gathered rows, [rows][rank + 64].
__global__ void __launch_bounds__(THREADS, 1)
attn_expanded_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                        const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_kr,
                        __nv_bfloat16* __restrict__ out, const int* __restrict__ segment_start, const int* __restrict__ first,
                        const int* __restrict__ context, int num_segments, int heads, int first_head, int own_heads, int rank,
                        float scale_log2e, int window,
                        const float* __restrict__ sink, const float* __restrict__ out_gate) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* gbase = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_s = base, k_s = q_s + Q_BYTES, v_s = k_s + STAGES * K_BYTES, p_s = v_s + STAGES * V_BYTES;
  float* const hand_over = reinterpret_cast<float*>(gbase + (p_s - base) + GROUPS * P_BYTES);      // [GROUPS][256]
  const uint32_t bars = p_s + GROUPS * P_BYTES + GROUPS * 256 * 4;
  unsigned char* tail = gbase + (bars - base);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 8 * B_COUNT);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8 * B_COUNT + 4);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // blocks are numbered tile by tile, all heads of a tile side by side, late tiles (the longest walks) first
  const int own_head = blockIdx.x % own_heads, head = first_head + own_head;
  pdl_launch_dependents();
  int seg, r0, cnt;
  __shared__ int tile_slot[3];
  lse_find_tile(segment_start, num_segments, BM, 0, (int)(blockIdx.x / own_heads), tile_slot, seg, r0, cnt);
  if (seg < 0) return;
  const int nrows = min(BM, cnt - r0);
  const int row_base = segment_start[seg] + r0;
  const int kept = first_kept(first[seg], window);
  const int pos0 = first[seg] + r0, last_pos = pos0 + nrows - 1;
  const int j_lo = window > 0 ? max(0, pos0 + 1 - window - kept) / BN : 0;      // key tiles are counted from the request's first gathered row
  const int n_local = (last_pos - kept) / BN + 1 - j_lo;
  const int key_row = rows_before(first, context, window, seg) + j_lo * BN;

  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_SE && i < B_OD ? GROUP_THREADS : 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == MMA_WARP) tmem_alloc(tmem_slot, 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // tensor memory: scores of group g, accumulator b at (2 g + b) * BN; outputs of group g behind them
  constexpr uint32_t O_COL = 2 * GROUPS * BN;
  int* const err = &lse_attn_expanded_error;
  pdl_wait();      // queries, keys and values come from the kernels before; no bounded wait starts earlier

  if (warp == LOADER_WARP) {
    if (lane == 0) {
      mbar_expect_tx(bar(B_Q), Q_BYTES);
      tma_load_3d(q_s, &map_q, bar(B_Q), 0, head, row_base);
      tma_load_3d(q_s + Q_BOX, &map_q, bar(B_Q), 64, head, row_base);
      tma_load_3d(q_s + 2 * Q_BOX, &map_qr, bar(B_Q), rank, head, row_base);
      for (int j = 0; j < n_local; ++j) {
        const int s = j % STAGES;
        if (!mbar_wait(bar(B_KE + s), ((uint32_t)(j / STAGES) & 1u) ^ 1u, abort_flag, err)) break;
        const uint32_t dst = k_s + s * K_BYTES;
        mbar_expect_tx(bar(B_KF + s), K_BYTES);
        tma_load_3d(dst, &map_kv, bar(B_KF + s), 0, own_head, key_row + j * BN);
        tma_load_3d(dst + KV_BOX, &map_kv, bar(B_KF + s), 64, own_head, key_row + j * BN);
        tma_load_2d(dst + 2 * KV_BOX, &map_kr, bar(B_KF + s), rank, key_row + j * BN);
      }
    }
    __syncwarp();
  } else if (warp == V_LOADER_WARP) {      // a thread of its own: keys are wanted long before the values of the same tile are
    if (lane == 0) {
      for (int j = 0; j < n_local; ++j) {
        const int s = j % STAGES;
        if (!mbar_wait(bar(B_VE + s), ((uint32_t)(j / STAGES) & 1u) ^ 1u, abort_flag, err)) break;
        const uint32_t dst = v_s + s * V_BYTES;
        mbar_expect_tx(bar(B_VF + s), V_BYTES);
        tma_load_3d(dst, &map_kv, bar(B_VF + s), 0, own_heads + own_head, key_row + j * BN);
        tma_load_3d(dst + KV_BOX, &map_kv, bar(B_VF + s), 64, own_heads + own_head, key_row + j * BN);
      }
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    if (lane == 0) {      // S_j = Q K_j^T as soon as the group has read the scores that lay in the accumulator before
      const uint32_t idesc = instr_desc_bf16(BM, BN, false, false);
      bool ok = mbar_poll(bar(B_Q), 0, abort_flag, err);
      for (int j = 0; j < n_local && ok; ++j) {
        const int s = j % STAGES, a = (j & 1) * 2 + ((j >> 1) & 1);
        ok = mbar_poll(bar(B_KF + s), (uint32_t)(j / STAGES) & 1u, abort_flag, err);
        if (ok && j >= 4) ok = mbar_poll(bar(B_SE + a), ((uint32_t)(j >> 2) & 1u) ^ 1u, abort_flag, err);
        if (!ok) break;
        fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 12; ++ks)
          umma_bf16(tmem_base + a * BN, smem_desc_k_major(q_s + (ks / 4) * Q_BOX + (ks % 4) * 32),
                    smem_desc_k_major(k_s + s * K_BYTES + (ks / 4) * KV_BOX + (ks % 4) * 32), idesc, ks != 0 ? 1u : 0u);
        umma_commit(bar(B_KE + s));
        umma_commit(bar(B_SF + a));
      }
    }
    __syncwarp();
  } else if (warp == PV_WARP) {
    if (lane == 0) {      // O_g += P_j V_j as soon as the probabilities of tile j are written
      const uint32_t idesc = instr_desc_bf16(BM, D, false, true);
      bool ok = true;
      for (int j = 0; j < n_local && ok; ++j) {
        const int g = j & 1, s = j % STAGES;
        ok = mbar_poll(bar(B_VF + s), (uint32_t)(j / STAGES) & 1u, abort_flag, err) &&
             mbar_poll(bar(B_PF + g), (uint32_t)(j >> 1) & 1u, abort_flag, err);
        if (!ok) break;
        fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < BN / 16; ++ks)
          umma_bf16(tmem_base + O_COL + g * D, smem_desc_k_major(p_s + g * P_BYTES + ks * 32),
                    smem_desc_mn_major(v_s + s * V_BYTES + ks * 2048, KV_BOX, 1024u), idesc, (j >= GROUPS || ks != 0) ? 1u : 0u);
        umma_commit(bar(B_VE + s));
        umma_commit(bar(B_OD + g));
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- softmax: a thread owns one row of its group's tiles
    const int g = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t o_addr = lane_addr + O_COL + g * D;
    const int my_pos = pos0 + min(row, nrows - 1);
    unsigned char* prow = gbase + (p_s - base) + g * P_BYTES + row * 128;
    float m_used = -INFINITY, m_seen = -INFINITY, l = 0.f;   // the maximum that O and l are relative to; the largest score seen
    bool pending = false;                                    // m_seen has outgrown m_used: O and l are to be rescaled
    // `ok` is the same in all lanes of a warp (a vote after every wait); a warp whose wait gave up still meets the other
    // group's warp at the pair barrier, which has no time limit of its own
    bool ok = true;
    auto wait_all = [&](int which, uint32_t parity) {
      const bool done = mbar_test(bar(which), parity) || mbar_wait(bar(which), parity, abort_flag, err);
      return __all_sync(0xffffffffu, done ? 1 : 0) != 0;
    };
    for (int j = g; j < n_local && ok; j += GROUPS) {
      const int a = g * 2 + ((j >> 1) & 1);
      const uint32_t s_addr = lane_addr + a * BN;
      ok = wait_all(B_SF + a, (uint32_t)(j >> 2) & 1u);
      if (!ok) break;
      fence_after_sync();
      const int kv0 = kept + (j_lo + j) * BN;      // position of the tile's first key
      const bool edge = kv0 + BN - 1 > my_pos || (window > 0 && kv0 <= my_pos - window);      // some keys are hidden from this row
      uint32_t s[2][32];
      tmem_ld32(s_addr, s[0]);
      tmem_ld32(s_addr + 32, s[1]);
      tmem_ld_wait();
      fence_before_sync();
      mbar_arrive(bar(B_SE + a));      // the scores are in registers: the accumulator is free
      float mx = -INFINITY;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (edge) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int key = kv0 + 32 * h + i;
            if (key > my_pos || (window > 0 && key <= my_pos - window)) s[h][i] = 0xff800000u;
          }
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) mx = fmaxf(mx, fmaxf(__uint_as_float(s[h][i]), __uint_as_float(s[h][i + 1])));
      }
      const float m_tile = mx * scale_log2e;
      bool rescale = false;
      float alpha = 1.f;
      if (j < GROUPS) {
        m_used = m_seen = m_tile;
      } else {
        // a maximum that grew by more than 2^8 in the tile before is taken over now, one that grows by more than 2^64 in
        // this tile at once
        m_seen = fmaxf(m_seen, m_tile);
        if (pending || __any_sync(0xffffffffu, m_tile > m_used + REDO_STEP)) {
          rescale = true;
          alpha = m_used == -INFINITY ? 0.f : exp2_fast(m_used - m_seen);
          m_used = m_seen;
          l *= alpha;
        }
      }
      pending = __any_sync(0xffffffffu, m_seen > m_used + RESCALE_STEP) != 0;
      const float neg = m_used == -INFINITY ? 0.f : -m_used;   // every score is -inf then as well: p = 0
      float sum = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float p0 = exp2_fast(fmaf(__uint_as_float(s[i / 16][2 * i % 32]), scale_log2e, neg));
        const float p1 = exp2_fast(fmaf(__uint_as_float(s[i / 16][2 * i % 32 + 1]), scale_log2e, neg));
        const float p2 = exp2_fast(fmaf(__uint_as_float(s[i / 16][2 * i % 32 + 2]), scale_log2e, neg));
        const float p3 = exp2_fast(fmaf(__uint_as_float(s[i / 16][2 * i % 32 + 3]), scale_log2e, neg));
        sum += (p0 + p1) + (p2 + p3);
        pk[i] = pack_bf16(p0, p1);
        pk[i + 1] = pack_bf16(p2, p3);
      }
      l += sum;
      if (j >= GROUPS) {   // P V of this group's tile before has read the probabilities and added to O
        ok = wait_all(B_OD + g, ((uint32_t)(j >> 1) & 1u) ^ 1u);
        if (!ok) break;
        fence_after_sync();
      }
      if (rescale) {
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          tmem_ld32(o_addr + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st32(o_addr + c, o);
        }
        tmem_st_wait();
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        *reinterpret_cast<uint4*>(prow + ((k ^ (row & 7)) << 4)) = make_uint4(pk[4 * k], pk[4 * k + 1], pk[4 * k + 2], pk[4 * k + 3]);
      fence_async_smem();
      fence_before_sync();
      mbar_arrive(bar(B_PF + g));
    }
    // ---------------------------------------------------------------- merge of the two groups
    float* mine = hand_over + g * 256;
    const float* other = hand_over + (g ^ 1) * 256;
    mine[row] = m_used;
    mine[128 + row] = l;
    pair_barrier(quarter);
    const float m_other = other[row], l_other = other[128 + row];
    const float m_all = fmaxf(m_used, m_other);                      // finite: the row sees its own key
    const float w_mine = m_used == -INFINITY ? 0.f : exp2_fast(m_used - m_all);
    const float w_other = m_other == -INFINITY ? 0.f : exp2_fast(m_other - m_all);
    // group 0's term first in both groups' threads: the two threads of a row hold the same bits
    const float l_all = g == 0 ? fmaf(l_other, w_other, l * w_mine) : fmaf(l, w_mine, l_other * w_other);
    float inv = 1.0f / l_all;
    if (sink) {   // exp(sink) joins the sum; the outputs are rescaled when the sink is the new maximum
      const float sink2 = sink[head] * LOG2E;
      const float m_fin = fmaxf(m_all, sink2);
      const float w_rows = exp2_fast(m_all - m_fin);
      inv = w_rows / fmaf(l_all, w_rows, exp2_fast(sink2 - m_fin));
    }
    if (out_gate && row < nrows) inv *= out_gate[(size_t)(row_base + row) * heads + head];
    const float w0 = (g == 0 ? w_mine : w_other) * inv, w1 = (g == 0 ? w_other : w_mine) * inv;
    const int n0 = (n_local + 1) / 2, n1 = n_local / 2;      // both groups' last products must have landed
    if (ok) ok = wait_all(B_OD + 0, (uint32_t)(n0 - 1) & 1u);
    if (ok && n1 > 0) ok = wait_all(B_OD + 1, (uint32_t)(n1 - 1) & 1u);
    __nv_bfloat16* dst = out + ((size_t)(row_base + row) * heads + head) * D + g * (D / 2);
    if (ok) {
      fence_after_sync();
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        uint32_t x[32], y[32];
        tmem_ld32(lane_addr + O_COL + g * (D / 2) + c, x);
        if (n1 > 0) tmem_ld32(lane_addr + O_COL + D + g * (D / 2) + c, y);
        tmem_ld_wait();
        if (row < nrows) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              v[e] = __uint_as_float(x[8 * i + e]) * w0;
              if (n1 > 0) v[e] = fmaf(__uint_as_float(y[8 * i + e]), w1, v[e]);
            }
            *reinterpret_cast<uint4*>(dst + c + 8 * i) =
                make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
          }
        }
      }
    }
  }
  if (*abort_flag && tid == 0) {
    // a wait gave up: give copies that may still be in flight time to land before the block leaves
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, 512);
}
}  // namespace

// Whether the kernels take these sizes (else the attention runs over the cached rows).
extern "C" int lse_attention_expanded_supported(int dim, int rot, int vdim, int rank) {
  return dim == D && rot == ROT && vdim == D && rank > 0 && rank % 8 == 0 ? 1 : 0;
}
// Keys of a tile: a request's gathered rows are a multiple of it.
extern "C" int lse_attention_expanded_tile(void) { return BN; }

// 0: no bounded wait has given up (1) and no request's rows were left out (2) since the word was last cleared (synchronises
// the device).
extern "C" int lse_attention_expanded_status(void) {
  int value = 0;
  if (cudaMemcpyFromSymbol(&value, lse_attn_expanded_error, sizeof(int)) != cudaSuccess) return -1;
  return value;
}
extern "C" int lse_attention_expanded_status_async(int* host_dst, cudaStream_t stream) {
  return (int)cudaMemcpyFromSymbolAsync(host_dst, lse_attn_expanded_error, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
}
extern "C" int lse_attention_expanded_status_reset(void) {
  const int zero = 0;
  return (int)cudaMemcpyToSymbol(lse_attn_expanded_error, &zero, sizeof(int));
}

// rows [capacity, width] bfloat16 receives the cached rows (cache [pages, page_size, width]) of every request, from its
// first position - window + 1 on (window <= 0: from 0), up to context[s] (exclusive), rounded up to whole tiles; zeros beyond.
// capacity holds the sum of them (lse_attention_expanded_status: 2 if it does not).  All 16-byte aligned.
extern "C" int lse_latent_gather(const void* cache, const int* block_tables, int bt_stride, const int* segment_first_pos,
                                 const int* segment_context, int num_segments, int width, int page_size, int num_pages,
                                 int window, void* rows, int capacity, cudaStream_t stream) {
  if (capacity <= 0 || num_segments <= 0) return 0;
  if (width <= 0 || width % 8 || page_size <= 0 || (((uintptr_t)cache | (uintptr_t)rows) & 15)) return LSE_ERR_BAD_ARGUMENT;
  lse_launch(latent_gather_kernel, (unsigned)((capacity + 7) / 8), 256, 0, stream, (const __nv_bfloat16*)cache, block_tables,
             bt_stride, segment_first_pos, segment_context, num_segments, width, page_size, num_pages, window,
             (__nv_bfloat16*)rows, capacity);
  LSE_LAUNCH_CHECK();
}

// q_plain [tokens, heads, 128], q_wide [tokens, heads, rank + 64] (the rotated values behind column rank), rows [capacity,
// rank + 64] as gathered, kv [capacity, 2 own_heads, 128] (the keys of heads first_head .. first_head + own_heads - 1, then
// their values; the other heads' outputs are left alone), out [tokens, heads, 128], all bfloat16, contiguous, 16-byte aligned.  sink float32 [heads] or null; out_gate float32 [tokens, heads] or null.
extern "C" int lse_attention_expanded(const void* q_plain, const void* q_wide, const void* rows, const void* kv, void* out,
                                      const int* segment_start, const int* segment_first_pos, const int* segment_context,
                                      int num_segments, int tokens, int heads, int first_head, int own_heads, int rank,
                                      int capacity, float scale, int window,
                                      const float* sink, const float* out_gate, cudaStream_t stream) {
  if (tokens <= 0 || num_segments <= 0) return 0;
  if (heads <= 0 || first_head < 0 || own_heads <= 0 || first_head + own_heads > heads || capacity <= 0 || !(scale > 0.f) || !lse_attention_expanded_supported(D, ROT, D, rank) ||
      (((uintptr_t)q_plain | (uintptr_t)q_wide | (uintptr_t)rows | (uintptr_t)kv | (uintptr_t)out) & 15))
    return LSE_ERR_BAD_ARGUMENT;
  static SmemAllowance allowed;
  cudaError_t err = allow_smem(attn_expanded_tc_kernel, SMEM, allowed);
  if (err != cudaSuccess) return (int)err;
  CUtensorMap map_q, map_qr, map_kv, map_kr;
  if (!make_map_3d(&map_q, q_plain, tokens, heads, D, BM) || !make_map_3d(&map_qr, q_wide, tokens, heads, rank + ROT, BM) ||
      !make_map_3d(&map_kv, kv, capacity, 2 * own_heads, D, BN) || !make_map_2d(&map_kr, rows, capacity, rank + ROT, BN))
    return LSE_ERR_BAD_ARGUMENT;
  const long long blocks = ((long long)(tokens + BM - 1) / BM + num_segments) * own_heads;      // every request may end with a partial tile
  if (blocks > 0x7fffffffLL) return LSE_ERR_TOO_LARGE;
  err = lse_launch(attn_expanded_tc_kernel, (unsigned)blocks, THREADS, SMEM, stream, map_q, map_qr, map_kv, map_kr,
                               (__nv_bfloat16*)out, segment_start, segment_first_pos, segment_context, num_segments, heads, first_head,
                               own_heads, rank, scale * LOG2E, window, sink, out_gate);
  if (err != cudaSuccess) return (int)err;
  return (int)cudaGetLastError();
}
