// Paged attention, general form: any head size that is a multiple of 16 (up to
// 256), any number of heads and groups, any page size, float32 or bfloat16
// storage, optional window.
//
// For row t of the step: the request's pages are block_tables[segment_of_token[t]],
// its position is positions[t], and it attends to keys j with
//     max(0, pos + 1 - window) <= j <= pos        (window <= 0: all keys j <= pos).
// A row's keys are taken chunk by chunk (CHUNK keys, counted from key 0) with the reference's softmax
// (src/llmserve/model.py:143-176; src/llmserve/triton_kernels/paged_attention.py:62-138).  Over a chunk's visible keys:
//     s_j = (q . k_j) * scale  (one fmaf per dimension, in order);   m = max_j s_j;   p_j = exp(s_j - m)
//     l = sum_j p_j  (keys j, j + 32 first, then the 32 sums by halving distances);   acc = sum_j p_j v_j  (in order)
// and the chunks are merged in order,
//     m' = max(M, m);  a = exp(M - m');  b = exp(m - m');  A = A a + acc b;  L = L a + l b;      out = A / L.
// Chunks depend on the row's own position only and every kernel below keeps to these operations in this order, so a row's
// result is the same bit for bit whatever else is in the batch, however the prompt was cut and whichever kernel ran.
//
// Three kernels:
//   rows    a block takes one row and up to GC query heads that share a key/value head (decoding): some of its chunks, whose
//           partial results it leaves in global memory, or (many rows) all chunks of its row;
//   tiles   a block takes ROWS (token, query head) pairs of one key/value head, the tokens neighbouring rows of one
//           request (prompts): all chunks, or some, as above;
//   merge   adds up the chunks that several blocks left.
//
// Cache layout: [page][kv head][offset in page][D].
#include "common.cuh"
#include "smem_allowance.cuh"

LSE_CHECK_DEFINE(lse_check_attention_generic)

namespace {
constexpr int CHUNK = 64;     // keys per chunk
constexpr int GC = 8;         // query heads per block of the rows kernel (chunk of a group)
constexpr int THREADS = 128;  // 4 warps
constexpr int MAX_D = 256;
constexpr int ROWS = 64;      // (token, head) pairs per block of the tiles kernel
constexpr int TILES_MAX_D = 128;
// About so many blocks share the chunks of a launch, sixteen an SM.  float32, 64 requests, 12 / 2 heads of 128, a block a
// chunk against 1,184, 2,368 and 9,472 blocks: 2,000 keys 106 against 90, 88 and 93 us; 100 keys in tables of 16,384 50
// against 15, 17 and 24 us; 8 heads of 64: 155 against 143, 126 and 130 us, 140 against 16, 17 and 23 us.
constexpr long long SPLIT_BLOCKS = 2368;

// Merge a chunk's (m, l) into the running (M, L); wa and wb are the factors for the outputs.
__device__ __forceinline__ void merge_chunk(float& M, float& L, float m, float l, float& wa, float& wb) {
  if (m == -INFINITY) {    // no key of the chunk has any weight: the row stays as it is
    wa = 1.f;
    wb = 0.f;
    return;
  }
  const float m_new = fmaxf(M, m);
  wa = expf(M - m_new);    // exp(-inf) = 0 before the first chunk
  wb = expf(m - m_new);
  L = fmaf(l, wb, __fmul_rn(L, wa));
  M = m_new;
}
// The maximum, the weights and their sum of one row's chunk: this lane holds the scaled scores of keys lane and lane + 32
// (-inf: hidden) and gets their weights.  m is -inf when every key is hidden.
__device__ __forceinline__ void chunk_softmax(float (&s)[2], float& m, float& l) {
  m = warp_max(fmaxf(s[0], s[1]));
#pragma unroll
  for (int i = 0; i < 2; ++i) s[i] = s[i] == -INFINITY ? 0.f : expf(s[i] - m);
  l = warp_sum(s[0] + s[1]);
}

// Copies rows of D values into shared memory as float32, `pitch` floats apart: row r comes from src + offsets[r]
// (negative: zeros).  The offsets lie in shared memory: worked out by the copying threads, a table entry's round trip and
// the divisions by the page size stood before every sixteen bytes (35 us a chunk of a tile against 12).
// VEC: sixteen bytes at a time.
template <typename T, bool VEC>
__device__ __forceinline__ void fill_rows(float* dst, int pitch, const T* __restrict__ src, int rows, int D,
                                          const long long* offsets) {
  constexpr int N = VEC ? 16 / (int)sizeof(T) : 1;
  const int pieces = D / N;
  const int bits = pieces > 16 ? 5 : (pieces > 8 ? 4 : 3);      // lanes that share a row
  const int lane = threadIdx.x & ((1 << bits) - 1);
#pragma unroll 4
  for (int r = threadIdx.x >> bits; r < rows; r += THREADS >> bits) {
    const long long off = offsets[r];
    for (int c = lane * N; c < D; c += N << bits) {
      float* to = dst + r * pitch + c;
      if (VEC && sizeof(T) == 4) {
        // straight to shared memory, without a register in between (zeros when nothing is read)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(to)),
                     "l"(off >= 0 ? src + off + c : src), "r"(off >= 0 ? 16 : 0) : "memory");
      } else if (VEC) {
        uint4 raw = make_uint4(0u, 0u, 0u, 0u);
        if (off >= 0) raw = *reinterpret_cast<const uint4*>(src + off + c);
        const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < N; i += 4)
          *reinterpret_cast<float4*>(to + i) = make_float4(to_f32<T>(v[i % N]), to_f32<T>(v[(i + 1) % N]), to_f32<T>(v[(i + 2) % N]), to_f32<T>(v[(i + 3) % N]));
      } else {
        to[0] = off >= 0 ? to_f32<T>(src[off + c]) : 0.f;
      }
    }
  }
}
__device__ __forceinline__ void fill_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void fill_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

struct Step {      // what the kernels take from the step
  const int* block_tables;
  int bt_stride;
  const int* segment_of_token;
  const int* positions;
  const int* segment_start;       // [segments + 1] first row of each request, or null
  int num_pages, num_segments;
  int n_q, n_kv, head_dim, page_size;
  float scale;
  int window;
  int skip;                       // rows kernel and merge: see which_row
  int max_chunks, parts;          // SPLIT: chunks that a row's partial results have room for; blocks that share them
};
enum { ALL_ROWS = 0, SINGLE_ROWS = 1, ROWS_OF_PORTIONS = 2 };

// Row number `index` of a launch: ALL_ROWS: row `index`; SINGLE_ROWS: the only row of request `index` (-1: it brings
// several); ROWS_OF_PORTIONS: row `index`, unless it is its request's only one.  seg receives its request, -1 for none.
__device__ __forceinline__ int which_row(const Step& p, int index, int& seg) {
  if (p.skip == SINGLE_ROWS) {
    seg = index;
    const int first = p.segment_start[index];
    if (p.segment_start[index + 1] - first != 1) { seg = -1; return -1; }
    return first;
  }
  seg = LSE_CHECKED(p.segment_of_token[index], -1, p.num_segments, -1, LSE_CHECK_SEGMENT);
  if (seg >= 0 && p.skip == ROWS_OF_PORTIONS && p.segment_start[seg + 1] - p.segment_start[seg] == 1) seg = -1;
  return index;
}

// What a block without work does that has not waited for the kernels before yet.  A launch over some of the rows may have none
// at all (every request brings one row): it must not end ahead of the kernel before it, for the kernel after it waits for
// this launch only.
__device__ __forceinline__ void leave_unneeded(const Step& p) {
  if (p.skip != ALL_ROWS) pdl_wait();
}

// SPLIT: the block of number `part` takes every parts-th of the chunks lo .. hi of its rows: lo becomes its first one.
// (The chunks of a row are known on the device only: with a block for every chunk that the block tables have room for, 64
// rows of 100 keys in tables of 16,384 made 16,384 blocks at two key/value heads, nearly all of them without work.)
__device__ __forceinline__ void my_chunks(const Step& p, int part, int& lo, int& hi) {
  hi = min(hi, p.max_chunks - 1);
  lo += (part - lo % p.parts + p.parts) % p.parts;
}

// ---------------------------------------------------------------- rows
// Element offset of key j of the request in the cache.
__device__ __forceinline__ long long key_offset(const Step& p, const int* bt, int kv_head, int j) {
  const int page = LSE_CHECKED(bt[j / p.page_size], 0, p.num_pages, 0, LSE_CHECK_TABLE_ENTRY);
  return (((long long)page * p.n_kv + kv_head) * p.page_size + (j % p.page_size)) * p.head_dim;
}

// grid (rows * head chunks * parts, kv heads).  SPLIT: the block takes some chunks and writes acc [D], m, l of each and its
// heads to `partials` [row][head][chunk][D + 2].  Else it merges all chunks of its row and writes `out`.
// The chunk's keys and values (2 x 33 KB at 128 values of float32) are asked for at once; scores: a lane owns two keys and
// two heads, sums: two columns and four heads, which keeps the register writes from shared memory, 128 bytes a clock,
// near the time that the chunk's bytes take.
template <typename T, bool SPLIT, bool VEC>
__global__ void __launch_bounds__(THREADS)
paged_attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                               T* __restrict__ out, const Step p, float* __restrict__ partials, int rows) {
  extern __shared__ __align__(16) float smem[];
  pdl_launch_dependents();
  pdl_wait();
  const int index = blockIdx.x % rows, rest = blockIdx.x / rows;
  const int kv_head = blockIdx.y;
  const int group = p.n_q / p.n_kv;
  const int gchunks = (group + GC - 1) / GC;
  const int g0 = (rest % gchunks) * GC;
  const int gcount = min(GC, group - g0);
  int seg;
  const int t = which_row(p, index, seg);
  if (seg < 0) return;
  const int pos = p.positions[t];
  const int kv_begin = p.window > 0 ? max(0, pos + 1 - p.window) : 0;
  int chunk_lo = kv_begin / CHUNK, chunk_hi = pos / CHUNK;
  if (SPLIT) {
    my_chunks(p, rest / gchunks, chunk_lo, chunk_hi);
    if (chunk_lo > chunk_hi) return;
  }
  const int* bt = p.block_tables + (size_t)seg * p.bt_stride;
  const int D = p.head_dim, pitch = D + 4;
  float* q_s = smem;                          // [GC][D]
  float* k_s = q_s + GC * D;                  // [CHUNK][pitch]
  float* v_s = k_s + CHUNK * pitch;           // [CHUNK][pitch]
  float* p_s = v_s + CHUNK * pitch;           // [CHUNK][GC] weights, by key
  float* stat_s = p_s + CHUNK * GC;           // [2][GC] maximum and sum of the chunk
  __shared__ long long offset_s[CHUNK];       // where the chunk's keys lie in the cache
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first_head = kv_head * group + g0;
  for (int e = tid; e < GC * D; e += THREADS)
    q_s[e] = e < gcount * D ? to_f32<T>(q[((size_t)t * p.n_q + first_head) * D + e]) : 0.f;

  // the columns 2 x, 2 x + 1 (x = tid % 64, and 64 more on) of the heads h0 .. h0 + 3
  const int h0 = (tid / 64) * 4;
  float total[4][4], M[4], L[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    M[g] = -INFINITY;
    L[g] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) total[g][i] = 0.f;
  }
  for (int chunk = chunk_lo; chunk <= chunk_hi; chunk += SPLIT ? p.parts : 1) {
    const int first_key = chunk * CHUNK;
    if (tid < CHUNK) {      // (read by the fills of the chunk before, which all threads have left)
      const int j = first_key + tid;
      offset_s[tid] = j <= pos && j >= kv_begin ? key_offset(p, bt, kv_head, j) : -1;
    }
    __syncthreads();        // the chunk before has been used
    fill_rows<T, VEC>(k_s, pitch, k_cache, CHUNK, D, offset_s);
    fill_commit();
    fill_rows<T, VEC>(v_s, pitch, v_cache, CHUNK, D, offset_s);
    fill_commit();
    fill_wait<1>();
    __syncthreads();
    {   // scores of keys lane, lane + 32 and heads 2 warp, 2 warp + 1
      float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
      const float* kr = k_s + lane * pitch;
      const float* qr = q_s + 2 * warp * D;
      if (2 * warp < gcount) {
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
          const float4 k0 = *reinterpret_cast<const float4*>(kr + d), k1 = *reinterpret_cast<const float4*>(kr + 32 * pitch + d);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const float4 a = *reinterpret_cast<const float4*>(qr + g * D + d);
            s[g][0] = fmaf(a.w, k0.w, fmaf(a.z, k0.z, fmaf(a.y, k0.y, fmaf(a.x, k0.x, s[g][0]))));
            s[g][1] = fmaf(a.w, k1.w, fmaf(a.z, k1.z, fmaf(a.y, k1.y, fmaf(a.x, k1.x, s[g][1]))));
          }
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          float m, l;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int j = first_key + lane + 32 * i;
            s[g][i] = j <= pos && j >= kv_begin ? __fmul_rn(s[g][i], p.scale) : -INFINITY;
          }
          chunk_softmax(s[g], m, l);
          p_s[lane * GC + 2 * warp + g] = s[g][0];
          p_s[(lane + 32) * GC + 2 * warp + g] = s[g][1];
          if (lane == 0) { stat_s[2 * warp + g] = m; stat_s[GC + 2 * warp + g] = l; }
        }
      }
    }
    fill_wait<0>();
    __syncthreads();
    float acc[4][4];
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[g][i] = 0.f;
    // hidden keys have no weight, and zeros for values
    if (h0 < gcount) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int col = 2 * (tid % 64) + 128 * i;
        if (col < D) {
#pragma unroll 4
          for (int j = 0; j < CHUNK; ++j) {
            const float2 v = *reinterpret_cast<const float2*>(v_s + j * pitch + col);
            const float4 w = *reinterpret_cast<const float4*>(p_s + j * GC + h0);
            acc[0][2 * i] = fmaf(w.x, v.x, acc[0][2 * i]); acc[0][2 * i + 1] = fmaf(w.x, v.y, acc[0][2 * i + 1]);
            acc[1][2 * i] = fmaf(w.y, v.x, acc[1][2 * i]); acc[1][2 * i + 1] = fmaf(w.y, v.y, acc[1][2 * i + 1]);
            acc[2][2 * i] = fmaf(w.z, v.x, acc[2][2 * i]); acc[2][2 * i + 1] = fmaf(w.z, v.y, acc[2][2 * i + 1]);
            acc[3][2 * i] = fmaf(w.w, v.x, acc[3][2 * i]); acc[3][2 * i + 1] = fmaf(w.w, v.y, acc[3][2 * i + 1]);
          }
        }
      }
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      if (h0 + g >= gcount) continue;
      const float m = stat_s[h0 + g], l = stat_s[GC + h0 + g];
      if (SPLIT) {
        float* dst = partials + (((size_t)index * p.n_q + first_head + h0 + g) * p.max_chunks + chunk) * (D + 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = 2 * (tid % 64) + 128 * (i / 2) + i % 2;
          if (col < D) dst[col] = acc[g][i];
        }
        if (tid % 64 == 0) { dst[D] = m; dst[D + 1] = l; }
      } else {
        float wa, wb;
        merge_chunk(M[g], L[g], m, l, wa, wb);
#pragma unroll
        for (int i = 0; i < 4; ++i) total[g][i] = fmaf(acc[g][i], wb, __fmul_rn(total[g][i], wa));
      }
    }
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if (SPLIT || h0 + g >= gcount) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int col = 2 * (tid % 64) + 128 * (i / 2) + i % 2;
      if (col < D) out[((size_t)t * p.n_q + first_head + h0 + g) * D + col] = from_f32<T>(total[g][i] / L[g]);
    }
  }
}

// ---------------------------------------------------------------- tiles
// A block's rows are pairs (token, head): pair r is token r / heads and head r % heads of the tile, heads = min(group, ROWS)
// query heads that share the key/value head, so that its keys are read once for all of them and a short portion still
// fills a tile.  grid (tiles of tokens * head chunks * (SPLIT ? parts : 1), kv heads).
// Scores: a thread owns 8 rows x 4 keys, sums: 8 rows x TN columns; a chunk's two products are bounded by the register
// writes from shared memory about as much as by the multiply-adds.  Keys and weights share a buffer, which leaves room
// for two blocks an SM (102 KB each at 128 values): one loads while the other multiplies.
template <typename T, int DT, bool SPLIT, bool VEC>
__global__ void __launch_bounds__(THREADS, SPLIT && DT <= 64 ? 4 : 2)
paged_attention_tiles_kernel(const T* __restrict__ q, const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                             T* __restrict__ out, const Step p, const int* __restrict__ segment_first,
                             float* __restrict__ partials, int tiles) {
  constexpr int TN = DT / 16;                 // columns of a thread: 4 (up to 64 values) or 8, in groups of four
  constexpr int PITCH = DT + 4, P_PITCH = CHUNK + 4;
  extern __shared__ __align__(16) float smem[];
  __shared__ int tile_slot[3];
  pdl_launch_dependents();
  const int group = p.n_q / p.n_kv, heads = min(group, ROWS);
  const int gchunks = (group + heads - 1) / heads, tokens_per_tile = ROWS / heads;
  const int rank = blockIdx.x % tiles, rest = blockIdx.x / tiles;
  const int kv_head = blockIdx.y;
  int seg, r0, cnt;
  lse_find_tile(p.segment_start, p.num_segments, tokens_per_tile, p.skip == ROWS_OF_PORTIONS, rank, tile_slot, seg, r0, cnt);
  if (seg < 0) { leave_unneeded(p); return; }
  const int tokens = min(tokens_per_tile, cnt - r0);
  const int row_base = p.segment_start[seg] + r0;
  const int pos0 = segment_first[seg] + r0, last_pos = pos0 + tokens - 1;
  const int first_key_read = p.window > 0 ? max(0, pos0 + 1 - p.window) : 0;
  int chunk_lo = first_key_read / CHUNK, chunk_hi = last_pos / CHUNK;
  if (SPLIT) {
    my_chunks(p, rest / gchunks, chunk_lo, chunk_hi);
    if (chunk_lo > chunk_hi) return;
  }
  const int first_head = kv_head * group + (rest % gchunks) * heads;
  const int head_count = min(heads, group - (rest % gchunks) * heads);
  const int* bt = p.block_tables + (size_t)seg * p.bt_stride;
  const int D = p.head_dim;
  float* q_s = smem;                          // [ROWS][PITCH]
  float* k_s = q_s + ROWS * PITCH;            // [CHUNK][PITCH], then the weights [ROWS][P_PITCH]
  float* v_s = k_s + CHUNK * PITCH;           // [CHUNK][PITCH]
  float* stat_s = v_s + CHUNK * PITCH;        // [4][ROWS]: M, L, wa, wb
  float* p_s = k_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto row_of = [&](int r, int& token, int& head) {      // false: no such pair
    token = r / heads;
    head = r % heads;
    return token < tokens && head < head_count;
  };
  __shared__ long long offset_s[CHUNK];       // where the chunk's keys lie in the cache (first: the queries)
  __shared__ int pos_s[ROWS];                 // position of each pair's token
  static_assert(CHUNK == ROWS, "one table of offsets for both");
  if (tid < ROWS) {
    int token, head;
    offset_s[tid] = row_of(tid, token, head) ? ((long long)(row_base + token) * p.n_q + first_head + head) * D : -1;
    pos_s[tid] = pos0 + token;                // pairs beyond the tile's: nothing of theirs is used
    stat_s[tid] = -INFINITY;
    stat_s[ROWS + tid] = 0.f;
  }
  __syncthreads();
  pdl_wait();
  fill_rows<T, VEC>(q_s, PITCH, q, ROWS, D, offset_s);
  __syncthreads();

  const int lm = lane % 4, ln = lane / 4;
  const int sm = (warp % 2) * 32 + lm;                  // rows of this thread: sm + 4 i (both products)
  const int sk = (warp / 2) * 32 + ln;                  // its keys: sk + 8 j
  const int oc = (warp / 2) * (DT / 2) + ln * 4;        // its columns: oc + 32 (j / 4) + j % 4
  float total[8][TN];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) total[i][j] = 0.f;

  for (int chunk = chunk_lo; chunk <= chunk_hi; chunk += SPLIT ? p.parts : 1) {
    const int first_key = chunk * CHUNK;
    float m_chunk = -INFINITY, l_chunk = 0.f;
    if (tid < CHUNK) {
      const int j = first_key + tid;
      offset_s[tid] = j <= last_pos && j >= first_key_read ? key_offset(p, bt, kv_head, j) : -1;
    }
    __syncthreads();
    fill_rows<T, VEC>(k_s, PITCH, k_cache, CHUNK, D, offset_s);
    fill_commit();
    fill_rows<T, VEC>(v_s, PITCH, v_cache, CHUNK, D, offset_s);
    fill_commit();
    fill_wait<1>();
    __syncthreads();
    float s[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
    for (int d = 0; d < D; d += 4) {
      float4 k[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(k_s + (sk + 8 * j) * PITCH + d);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(q_s + (sm + 4 * i) * PITCH + d);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[i][j] = fmaf(a.w, k[j].w, fmaf(a.z, k[j].z, fmaf(a.y, k[j].y, fmaf(a.x, k[j].x, s[i][j]))));
      }
    }
    __syncthreads();      // the keys have been used: the scores take their place
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int pos = pos_s[sm + 4 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = first_key + sk + 8 * j;
        const bool seen = key <= pos && (p.window <= 0 || key > pos - p.window);
        p_s[(sm + 4 * i) * P_PITCH + sk + 8 * j] = seen ? __fmul_rn(s[i][j], p.scale) : -INFINITY;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int rr = 0; rr < ROWS / 4; ++rr) {      // four rows' shuffles and exponentials on their way together
      const int r = warp * (ROWS / 4) + rr;
      float w[2] = {p_s[r * P_PITCH + lane], p_s[r * P_PITCH + lane + 32]}, m, l;
      chunk_softmax(w, m, l);
      p_s[r * P_PITCH + lane] = w[0];
      p_s[r * P_PITCH + lane + 32] = w[1];
      if (lane == rr) { m_chunk = m; l_chunk = l; }
    }
    if (lane < ROWS / 4) {      // a lane merges a row
      const int r = warp * (ROWS / 4) + lane;
      if (SPLIT) {
        stat_s[r] = m_chunk;
        stat_s[ROWS + r] = l_chunk;
      } else {
        float M = stat_s[r], L = stat_s[ROWS + r], wa, wb;
        merge_chunk(M, L, m_chunk, l_chunk, wa, wb);
        stat_s[r] = M;
        stat_s[ROWS + r] = L;
        stat_s[2 * ROWS + r] = wa;
        stat_s[3 * ROWS + r] = wb;
      }
    }
    fill_wait<0>();
    __syncthreads();
    float acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    // Keys that one row of the tile sees and another does not have no weight in the latter, and may hold anything (a later
    // row of the step may carry an infinity that must not reach an earlier one): such chunks ask key by key.
    const bool mixed = first_key + CHUNK - 1 > pos0 || (p.window > 0 && first_key <= last_pos - p.window);
    if (!mixed) {
#pragma unroll 1
      for (int j0 = 0; j0 < CHUNK; j0 += 4) {
        float v[4][TN];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
#pragma unroll
          for (int c = 0; c < TN; c += 4) {
            const float4 t = *reinterpret_cast<const float4*>(v_s + (j0 + jj) * PITCH + oc + 8 * c);
            v[jj][c] = t.x; v[jj][c + 1] = t.y; v[jj][c + 2] = t.z; v[jj][c + 3] = t.w;
          }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(p_s + (sm + 4 * i) * P_PITCH + j0);
#pragma unroll
          for (int c = 0; c < TN; ++c)
            acc[i][c] = fmaf(w.w, v[3][c], fmaf(w.z, v[2][c], fmaf(w.y, v[1][c], fmaf(w.x, v[0][c], acc[i][c]))));
        }
      }
    } else {
      int pos[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) pos[i] = pos_s[sm + 4 * i];
      const int behind = p.window > 0 ? p.window : 0x7fffffff;      // how far behind its row a key may lie, itself included
      const int keys = min(CHUNK, last_pos + 1 - first_key);
#pragma unroll 2
      for (int j = 0; j < keys; ++j) {
        float v[TN];
#pragma unroll
        for (int c = 0; c < TN; c += 4) {
          const float4 t = *reinterpret_cast<const float4*>(v_s + j * PITCH + oc + 8 * c);
          v[c] = t.x; v[c + 1] = t.y; v[c + 2] = t.z; v[c + 3] = t.w;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int ago = pos[i] - first_key - j;
          const float w = p_s[(sm + 4 * i) * P_PITCH + j];
          const bool seen = ago >= 0 && ago < behind;
#pragma unroll
          for (int c = 0; c < TN; ++c) acc[i][c] = seen ? fmaf(w, v[c], acc[i][c]) : acc[i][c];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = sm + 4 * i;
      if (SPLIT) {
        int token, head;
        if (!row_of(r, token, head)) continue;
        const int pos = pos_s[r];          // the merge asks for the chunks with a visible key only
        if (first_key > pos || (p.window > 0 && first_key + CHUNK - 1 <= pos - p.window)) continue;
        float* dst = partials + (((size_t)(row_base + token) * p.n_q + first_head + head) * p.max_chunks + chunk) * (D + 2);
#pragma unroll
        for (int c = 0; c < TN; ++c) {
          const int col = oc + 32 * (c / 4) + c % 4;
          if (col < D) dst[col] = acc[i][c];
        }
        if (oc == 0) { dst[D] = stat_s[r]; dst[D + 1] = stat_s[ROWS + r]; }
      } else {
        const float wa = stat_s[2 * ROWS + r], wb = stat_s[3 * ROWS + r];
#pragma unroll
        for (int c = 0; c < TN; ++c) total[i][c] = fmaf(acc[i][c], wb, __fmul_rn(total[i][c], wa));
      }
    }
    __syncthreads();      // weights, values and factors have been used
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int token, head;
    if (SPLIT || !row_of(sm + 4 * i, token, head)) continue;
    const float sum = stat_s[ROWS + sm + 4 * i];
    T* dst = out + ((size_t)(row_base + token) * p.n_q + first_head + head) * D;
#pragma unroll
    for (int c = 0; c < TN; ++c) {
      const int col = oc + 32 * (c / 4) + c % 4;
      if (col < D) dst[col] = from_f32<T>(total[i][c] / sum);
    }
  }
}

// ---------------------------------------------------------------- merge
// The chunks of a row and head, merged in order: grid (rows, n_q), a thread per column.  The maximum before a chunk is
// the largest of the chunks' before it, so that the first warp works out the factors of 32 chunks side by side; what is
// left to do in order is a multiplication and a fused multiply-add a chunk.
constexpr int MERGE_BATCH = 32;
template <typename T>
__global__ void __launch_bounds__(MAX_D)
paged_attention_generic_merge_kernel(const float* __restrict__ partials, T* __restrict__ out, const Step p) {
  __shared__ float wa_s[MERGE_BATCH], wb_s[MERGE_BATCH], sum_s[MERGE_BATCH];
  pdl_launch_dependents();
  const int index = blockIdx.x, head = blockIdx.y, d = threadIdx.x;
  int seg;
  const int t = which_row(p, index, seg), D = p.head_dim;
  if (seg < 0) { leave_unneeded(p); return; }
  const int pos = p.positions[t];
  const int kv_begin = p.window > 0 ? max(0, pos + 1 - p.window) : 0;
  const float* src = partials + ((size_t)index * p.n_q + head) * p.max_chunks * (D + 2);
  const int hi = min(pos / CHUNK, p.max_chunks - 1);
  float total = 0.f, M = -INFINITY, L = 0.f;      // M: the first warp's
  pdl_wait();
  for (int c0 = kv_begin / CHUNK; c0 <= hi; c0 += MERGE_BATCH) {
    float a[MERGE_BATCH];
#pragma unroll
    for (int i = 0; i < MERGE_BATCH; ++i) a[i] = c0 + i <= hi && d < D ? src[(size_t)(c0 + i) * (D + 2) + d] : 0.f;
    __syncthreads();      // the batch before has been used
    if (threadIdx.x < 32) {
      const int c = c0 + threadIdx.x;
      const float m = c <= hi ? src[(size_t)c * (D + 2) + D] : -INFINITY;
      float before = m;      // becomes the maximum over this chunk and those before it, then is handed one lane on
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float other = __shfl_up_sync(0xffffffffu, before, o);
        if (threadIdx.x >= o) before = fmaxf(before, other);
      }
      const float upto = fmaxf(before, M);
      before = __shfl_up_sync(0xffffffffu, upto, 1);
      float m_run = threadIdx.x == 0 ? M : before, l_run = 0.f, wa, wb;
      merge_chunk(m_run, l_run, m, 0.f, wa, wb);
      wa_s[threadIdx.x] = wa;
      wb_s[threadIdx.x] = wb;
      sum_s[threadIdx.x] = c <= hi ? src[(size_t)c * (D + 2) + D + 1] : 0.f;
      M = __shfl_sync(0xffffffffu, upto, 31);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MERGE_BATCH; ++i) {
      if (c0 + i <= hi) {
        const float wa = wa_s[i], wb = wb_s[i];
        L = fmaf(sum_s[i], wb, __fmul_rn(L, wa));
        total = fmaf(a[i], wb, __fmul_rn(total, wa));
      }
    }
  }
  if (d < D) out[((size_t)t * p.n_q + head) * D + d] = from_f32<T>(total / L);
}

size_t rows_smem(int D) { return sizeof(float) * ((size_t)GC * D + 2 * (size_t)CHUNK * (D + 4) + CHUNK * GC + 2 * GC); }
size_t tiles_smem(int DT) { return sizeof(float) * ((size_t)(ROWS + 2 * CHUNK) * (DT + 4) + 4 * ROWS); }

template <typename T, bool SPLIT, bool VEC>
cudaError_t launch_rows(const void* q, const void* k, const void* v, void* out, const Step& p, int rows, float* partials,
                        cudaStream_t stream) {
  auto kernel = paged_attention_generic_kernel<T, SPLIT, VEC>;
  static SmemAllowance allowed;
  cudaError_t err = allow_smem(kernel, rows_smem(MAX_D), allowed);
  if (err != cudaSuccess) return err;
  const int gchunks = (p.n_q / p.n_kv + GC - 1) / GC;
  const dim3 grid((unsigned)((long long)rows * gchunks * (SPLIT ? p.parts : 1)), p.n_kv);
  return lse_launch(kernel, grid, THREADS, rows_smem(p.head_dim), stream, (const T*)q, (const T*)k, (const T*)v, (T*)out, p,
                    partials, rows);
}

template <typename T, int DT, bool SPLIT, bool VEC>
cudaError_t launch_tiles(const void* q, const void* k, const void* v, void* out, const Step& p, const int* segment_first,
                         int tiles, float* partials, cudaStream_t stream) {
  auto kernel = paged_attention_tiles_kernel<T, DT, SPLIT, VEC>;
  static SmemAllowance allowed;
  cudaError_t err = allow_smem(kernel, tiles_smem(DT), allowed);
  if (err != cudaSuccess) return err;
  const int group = p.n_q / p.n_kv, heads = group < ROWS ? group : ROWS, gchunks = (group + heads - 1) / heads;
  const dim3 grid((unsigned)((long long)tiles * gchunks * (SPLIT ? p.parts : 1)), p.n_kv);
  return lse_launch(kernel, grid, THREADS, tiles_smem(DT), stream, (const T*)q, (const T*)k, (const T*)v, (T*)out, p,
                    segment_first, partials, tiles);
}

template <typename T>
cudaError_t launch_merge(void* out, const Step& p, int rows, const float* partials, cudaStream_t stream) {
  return lse_launch(paged_attention_generic_merge_kernel<T>, dim3(rows, p.n_q), ((p.head_dim + 31) / 32) * 32, 0, stream,
                    partials, (T*)out, p);
}

template <typename T, bool VEC>
cudaError_t run(const void* q, const void* k, const void* v, void* out, const Step& p, const int* segment_first, int rows,
                int tiles, float* partials, cudaStream_t stream) {
  cudaError_t err;
  if (tiles > 0) {
    const bool small = p.head_dim <= 64;
    if (partials)
      err = small ? launch_tiles<T, 64, true, VEC>(q, k, v, out, p, segment_first, tiles, partials, stream)
                  : launch_tiles<T, 128, true, VEC>(q, k, v, out, p, segment_first, tiles, partials, stream);
    else
      err = small ? launch_tiles<T, 64, false, VEC>(q, k, v, out, p, segment_first, tiles, nullptr, stream)
                  : launch_tiles<T, 128, false, VEC>(q, k, v, out, p, segment_first, tiles, nullptr, stream);
  } else {
    err = partials ? launch_rows<T, true, VEC>(q, k, v, out, p, rows, partials, stream)
                   : launch_rows<T, false, VEC>(q, k, v, out, p, rows, nullptr, stream);
  }
  if (err == cudaSuccess && partials) err = launch_merge<T>(out, p, rows, partials, stream);
  return err;
}
}  // namespace

// Keys of a chunk (the caller sizes `partials` by it).
extern "C" int lse_attention_generic_chunk(void) { return CHUNK; }
// Whether the tiles kernel takes this head size, and the tokens of one of its tiles.
extern "C" int lse_attention_generic_tile_tokens(int head_dim, int n_q, int n_kv) {
  if (head_dim <= 0 || head_dim > TILES_MAX_D || head_dim % 16 || n_kv <= 0 || n_q % n_kv || n_q <= 0) return 0;
  const int group = n_q / n_kv;
  return ROWS / (group < ROWS ? group : ROWS);
}

// segment_start null: the rows kernel over all `tokens` rows.  Else (with segment_first, [segments]) portions != 0: the tiles
// kernel over the rows of the requests that bring several (skip_single) or all requests; portions == 0: the rows kernel
// over the requests that bring one.
// partials != null: a row's chunks are shared by several blocks and a second kernel merges them; partials holds rows * n_q *
// max_chunks * (head_dim + 2) floats (rows: tokens, or segments for single rows), and max_chunks chunks cover the longest
// context of the step (max_context; 0: what the block tables can describe).  The result is the same bit for bit either way.
extern "C" int lse_paged_attention_generic_portions(const void* q, const void* k_cache, const void* v_cache, void* out, int dtype,
                                                    const int* block_tables, int bt_stride, const int* segment_of_token,
                                                    const int* positions, int tokens, int n_q, int n_kv, int head_dim,
                                                    int page_size, float scale, int window, int num_pages, int num_segments,
                                                    float* partials, int max_chunks, int max_context,
                                                    const int* segment_start, const int* segment_first, int portions,
                                                    int skip_single, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (head_dim <= 0 || head_dim > MAX_D || head_dim % 16 || n_kv <= 0 || n_q % n_kv || page_size <= 0)
    return LSE_ERR_BAD_ARGUMENT;
  if (segment_start && (num_segments <= 0 || (portions && (!segment_first || !lse_attention_generic_tile_tokens(head_dim, n_q, n_kv)))))
    return LSE_ERR_BAD_ARGUMENT;
  long long keys = (long long)bt_stride * page_size;
  if (max_context > 0 && max_context < keys) keys = max_context;
  if (partials && (max_chunks <= 0 || (long long)max_chunks * CHUNK < keys)) return LSE_ERR_BAD_ARGUMENT;
  Step p = {block_tables, bt_stride, segment_of_token, positions, segment_start, num_pages, num_segments,
            n_q, n_kv, head_dim, page_size, scale, window, ALL_ROWS, max_chunks, 1};
  int rows = tokens, tiles = 0;
  if (segment_start && portions) {
    const int per_tile = lse_attention_generic_tile_tokens(head_dim, n_q, n_kv);
    tiles = (tokens + per_tile - 1) / per_tile + num_segments;      // every request may end with a partial tile
    p.skip = skip_single ? ROWS_OF_PORTIONS : ALL_ROWS;
  } else if (segment_start) {
    rows = num_segments;
    p.skip = SINGLE_ROWS;
  }
  const int group = n_q / n_kv, heads = tiles > 0 ? (group < ROWS ? group : ROWS) : GC;
  const long long whole = (long long)(tiles > 0 ? tiles : rows) * ((group + heads - 1) / heads);
  if (partials) {
    const long long wanted = SPLIT_BLOCKS / (whole * n_kv) + 1;
    p.parts = (int)(wanted < max_chunks ? wanted : max_chunks);
  }
  const long long blocks = whole * p.parts;
  if (blocks > 0x7fffffffLL) return LSE_ERR_TOO_LARGE;
  const bool vec = (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) == 0;
  cudaError_t err;
#define LSE_GENERIC_ARGS q, k_cache, v_cache, out, p, segment_first, rows, tiles, partials, stream
  if (dtype == LSE_DTYPE_F32) err = vec ? run<float, true>(LSE_GENERIC_ARGS) : run<float, false>(LSE_GENERIC_ARGS);
  else if (dtype == LSE_DTYPE_BF16) err = vec ? run<__nv_bfloat16, true>(LSE_GENERIC_ARGS) : run<__nv_bfloat16, false>(LSE_GENERIC_ARGS);
  else return LSE_ERR_BAD_ARGUMENT;
#undef LSE_GENERIC_ARGS
  if (err != cudaSuccess) return (int)err;
  LSE_LAUNCH_CHECK();
}
