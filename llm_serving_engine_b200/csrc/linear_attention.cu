// Linear attention with a decay per head, carried from token to token in a float32 state per request:
//     S_t = decay_h * S_(t-1) + k_t v_t^T      (S is [dim][vdim] per head)
//     o_t = S_t^T q_t
// with q, k, v = act(projection) (act: SiLU, or none), and the gated norm that follows it:
//     y = o / sqrt(mean(o^2) + eps) * weight * sigmoid(g)      over the concatenated heads.
//
// The scan kernel walks the rows of one request in order, from the state that earlier steps left in the
// request's slot, and leaves the new state there.  A block owns (request, head, a tile of state columns); a
// thread owns 32 rows of one column of S in registers, so a token costs it 32 updates and a 32-term dot
// product, and the threads that share a column (dim > 32) add their parts by shuffles.  Columns of S are
// independent of one another, which is what lets them be spread over blocks.  Tokens are staged in shared
// memory a few at a time.  Everything is float32: the projections arrive in float32, in bfloat16 or as a
// stack of float32 partial sums, and are activated in float32.
#include "common.cuh"
#include "smem_allowance.cuh"

LSE_CHECK_DEFINE(lse_check_linear_attention)

#include "linear_attention_scan.cuh"

namespace {
// out[t] = o[t] / sqrt(mean(o[t]^2) + eps) * weight * sigmoid(g[t]); g: columns g_off .. g_off + n of proj.
template <typename TD, typename TO>
__global__ void __launch_bounds__(256)
gated_rmsnorm_kernel(const float* __restrict__ o, const TD* __restrict__ proj, int n_partials, long long partial_stride,
                     long long ld, int g_off, const float* __restrict__ weight, TO* __restrict__ out, int n, float eps,
                     const int* __restrict__ segment_of_token) {
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  if (segment_of_token && segment_of_token[t] < 0) return;
  const float* row = o + (size_t)t * n;
  float sq = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sq = fmaf(row[i], row[i], sq);
  const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)n + eps);
  const TD* g = proj + (size_t)t * ld + g_off;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float gate = 1.f / (1.f + expf(-la_load(g + i, n_partials, partial_stride)));
    out[(size_t)t * n + i] = from_f32<TO>(((row[i] * inv) * weight[i]) * gate);
  }
}
// The same for rows of up to 4,096 values in one pass: a thread keeps up to four groups of four values and of gates in
// registers (2,048 rows of 2,048: one value at a time and the row read twice took 23 us; 34 MB take 5).
constexpr int GN_GROUPS = 4;
template <typename TD, typename TO>
__global__ void __launch_bounds__(256)
gated_rmsnorm_vec_kernel(const float* __restrict__ o, const TD* __restrict__ proj, long long ld, int g_off,
                         const float* __restrict__ weight, TO* __restrict__ out, int n, float eps,
                         const int* __restrict__ segment_of_token) {
  __shared__ float scratch[32];
  pdl_launch_dependents();
  const int t = blockIdx.x;
  if (segment_of_token && segment_of_token[t] < 0) return;
  pdl_wait();
  const float* row = o + (size_t)t * n;
  const TD* g = proj + (size_t)t * ld + g_off;
  float x[GN_GROUPS][4], z[GN_GROUPS][4];
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < GN_GROUPS; ++i) {
    const int c = 4 * (threadIdx.x + i * 256);
    if (c < n) {
      const float4 v = *reinterpret_cast<const float4*>(row + c);
      x[i][0] = v.x; x[i][1] = v.y; x[i][2] = v.z; x[i][3] = v.w;
      if (sizeof(TD) == 4) {
        const float4 w = *reinterpret_cast<const float4*>(g + c);
        z[i][0] = w.x; z[i][1] = w.y; z[i][2] = w.z; z[i][3] = w.w;
      } else {
        const uint2 w = *reinterpret_cast<const uint2*>(g + c);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&w.x), b = *reinterpret_cast<const __nv_bfloat162*>(&w.y);
        z[i][0] = __low2float(a); z[i][1] = __high2float(a); z[i][2] = __low2float(b); z[i][3] = __high2float(b);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < GN_GROUPS; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * (threadIdx.x + i * 256) < n) sq = fmaf(x[i][e], x[i][e], sq);
  const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)n + eps);
#pragma unroll
  for (int i = 0; i < GN_GROUPS; ++i) {
    const int c = 4 * (threadIdx.x + i * 256);
    if (c < n) {
      const float4 w = *reinterpret_cast<const float4*>(weight + c);
      const float wv[4] = {w.x, w.y, w.z, w.w};
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = ((x[i][e] * inv) * wv[e]) * (1.f / (1.f + expf(-z[i][e])));
      if (sizeof(TO) == 4) {
        *reinterpret_cast<float4*>(out + (size_t)t * n + c) = make_float4(y[0], y[1], y[2], y[3]);
      } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(y[0], y[1]), b = __floats2bfloat162_rn(y[2], y[3]);
        *reinterpret_cast<uint2*>(out + (size_t)t * n + c) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
      }
    }
  }
}
// What a state-space scan with one decay per head takes from its step sizes: dt = softplus(z + bias_h) (no clamp),
// keep = exp(-exp(a_log_h) dt), take = dt; z is column dt_off + h of proj.  A thread per (token, head).
template <typename TD>
__global__ void __launch_bounds__(256)
ssd_gates_kernel(const TD* __restrict__ proj, int n_partials, long long partial_stride, long long ld, int dt_off,
                 const float* __restrict__ dt_bias, const float* __restrict__ a_log, float* __restrict__ keep,
                 float* __restrict__ take, int tokens, int heads) {
  pdl_launch_dependents();
  pdl_wait();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= tokens * heads) return;
  const int t = e / heads, h = e % heads;
  const float z = la_load(proj + (size_t)t * ld + dt_off + h, n_partials, partial_stride) + dt_bias[h];
  const float dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
  keep[e] = expf(-expf(a_log[h]) * dt);
  take[e] = dt;
}

// A decay per channel: keep = sigmoid(z + bias)^(1 / tau) = exp(log sigmoid(z + bias) / tau); z is column off + i of proj.
template <typename TD>
__global__ void __launch_bounds__(256)
sigmoid_power_kernel(const TD* __restrict__ proj, int n_partials, long long partial_stride, long long ld, int off,
                     const float* __restrict__ bias, float inv_tau, float* __restrict__ keep, int tokens, int n) {
  pdl_launch_dependents();
  pdl_wait();
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)tokens * n) return;
  const int t = (int)(e / n), i = (int)(e % n);
  float z = la_load(proj + (size_t)t * ld + off + i, n_partials, partial_stride);
  if (bias) z += bias[i];
  const float log_sigmoid = fminf(z, 0.f) - log1pf(expf(-fabsf(z)));
  keep[e] = expf(log_sigmoid * inv_tau);
}

// The norm behind a scan, in `groups` equal parts of a row, each by its own root mean square:
//   a_i = o_i + skip[i / head_width] * x_i          (skip null: a = o;  x: columns x_off .. of `xsrc`)
//   gate_first:  b = a * act(g);  out = b / rms(b) * weight[i % weight_len] * scale
//   else:                         out = a / rms(a) * weight[i % weight_len] * act(g) * scale
// with act the SiLU (gate_act 1) or the sigmoid (0); g: columns g_off .. of proj.  A block owns one part of one row
// (grid: rows x parts); a thread keeps up to GGN_KEPT of the part's values (and gates) between the sum and the write.
constexpr int GGN_KEPT = 8;
template <typename TD, typename TO, bool SINGLE>
__global__ void __launch_bounds__(256)
gated_group_rmsnorm_kernel(const float* __restrict__ o, const TD* __restrict__ proj, int n_partials,
                           long long partial_stride, long long ld, int g_off, const TO* __restrict__ xsrc,
                           long long x_ld, int x_off, const float* __restrict__ skip, int head_width,
                           const float* __restrict__ weight, int weight_len, TO* __restrict__ out, long long out_ld,
                           int n, int groups, float eps, float scale, int gate_first, int gate_act,
                           const int* __restrict__ segment_of_token) {
  __shared__ float scratch[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, part = blockIdx.y;
  if (segment_of_token && segment_of_token[t] < 0) return;
  const int width = n / groups, lo = part * width;
  const float* row = o + (size_t)t * n;
  const TD* g = proj + (size_t)t * ld + g_off;
  auto act = [&](float z) {
    const float sg = 1.f / (1.f + expf(-z));
    return gate_act == 1 ? z * sg : sg;
  };
  auto gate = [&](int i) { return act(SINGLE ? to_f32<TD>(g[i]) : la_load(g + i, n_partials, partial_stride)); };
  auto plain = [&](int i) {
    float a = row[i];
    if (skip) a = fmaf(skip[i / head_width], to_f32<TO>(xsrc[(size_t)t * x_ld + x_off + i]), a);
    return a;
  };
  float kept[GGN_KEPT], gates[GGN_KEPT], side[GGN_KEPT];
  float sq = 0.f;
  const TO* xrow = skip ? xsrc + (size_t)t * x_ld + x_off : nullptr;
#pragma unroll
  for (int k = 0; k < GGN_KEPT; ++k) {     // every load of the thread first, so that they travel together
    const int i = lo + threadIdx.x + k * blockDim.x;
    kept[k] = gates[k] = side[k] = 0.f;
    if (i < lo + width) {
      gates[k] = SINGLE ? to_f32<TD>(g[i]) : la_load(g + i, n_partials, partial_stride);
      kept[k] = row[i];
      if (skip) side[k] = to_f32<TO>(xrow[i]);
    }
  }
#pragma unroll
  for (int k = 0; k < GGN_KEPT; ++k) {
    const int i = lo + threadIdx.x + k * blockDim.x;
    if (i < lo + width) {
      gates[k] = act(gates[k]);
      if (skip) kept[k] = fmaf(skip[i / head_width], side[k], kept[k]);
      if (gate_first) kept[k] *= gates[k];
      sq = fmaf(kept[k], kept[k], sq);
    }
  }
  for (int i = lo + threadIdx.x + GGN_KEPT * blockDim.x; i < lo + width; i += blockDim.x) {
    const float v = gate_first ? plain(i) * gate(i) : plain(i);
    sq = fmaf(v, v, sq);
  }
  const float inv = 1.0f / sqrtf(block_sum(sq, scratch) / (float)width + eps);
#pragma unroll
  for (int k = 0; k < GGN_KEPT; ++k) {
    const int i = lo + threadIdx.x + k * blockDim.x;
    if (i < lo + width) {
      float y = (kept[k] * inv) * weight[i % weight_len];
      if (!gate_first) y *= gates[k];
      out[(size_t)t * out_ld + i] = from_f32<TO>(y * scale);
    }
  }
  for (int i = lo + threadIdx.x + GGN_KEPT * blockDim.x; i < lo + width; i += blockDim.x) {
    const float gi = gate(i);
    float y = ((gate_first ? plain(i) * gi : plain(i)) * inv) * weight[i % weight_len];
    if (!gate_first) y *= gi;
    out[(size_t)t * out_ld + i] = from_f32<TO>(y * scale);
  }
}
// The same for narrow parts (up to 32 * GGN_WARP_KEPT columns): a warp owns a part of a row, eight parts a block, no
// barrier; the part's values and gates stay in registers.
constexpr int GGN_WARP_KEPT = 16;
template <typename TD, typename TO, bool SINGLE>
__global__ void __launch_bounds__(256)
gated_group_rmsnorm_warp_kernel(const float* __restrict__ o, const TD* __restrict__ proj, int n_partials,
                                long long partial_stride, long long ld, int g_off, const TO* __restrict__ xsrc,
                                long long x_ld, int x_off, const float* __restrict__ skip, int head_width,
                                const float* __restrict__ weight, int weight_len, TO* __restrict__ out, long long out_ld,
                                int tokens, int n, int groups, float eps, float scale, int gate_first, int gate_act,
                                const int* __restrict__ segment_of_token) {
  pdl_launch_dependents();
  pdl_wait();
  const long long item = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (item >= (long long)tokens * groups) return;
  const int t = (int)(item / groups), part = (int)(item % groups);
  if (segment_of_token && segment_of_token[t] < 0) return;
  const int width = n / groups, lo = part * width;
  const float* row = o + (size_t)t * n + lo;
  const TD* g = proj + (size_t)t * ld + g_off + lo;
  const TO* x = skip ? xsrc + (size_t)t * x_ld + x_off + lo : nullptr;
  float kept[GGN_WARP_KEPT], gates[GGN_WARP_KEPT];
  float sq = 0.f;
#pragma unroll
  for (int k = 0; k < GGN_WARP_KEPT; ++k) {     // every load of the lane first, so that they travel together
    const int c = lane + 32 * k;
    kept[k] = gates[k] = 0.f;
    if (c < width) {
      gates[k] = SINGLE ? to_f32<TD>(g[c]) : la_load(g + c, n_partials, partial_stride);
      kept[k] = row[c];
    }
  }
#pragma unroll
  for (int k = 0; k < GGN_WARP_KEPT; ++k) {
    const int c = lane + 32 * k;
    if (c < width) {
      const float z = gates[k];
      const float sg = 1.f / (1.f + expf(-z));
      gates[k] = gate_act == 1 ? z * sg : sg;
      if (skip) kept[k] = fmaf(skip[(lo + c) / head_width], to_f32<TO>(x[c]), kept[k]);
      if (gate_first) kept[k] *= gates[k];
      sq = fmaf(kept[k], kept[k], sq);
    }
  }
  const float inv = 1.0f / sqrtf(warp_sum(sq) / (float)width + eps);
  const int w0 = lo % weight_len;      // the part's first weight; parts are whole multiples or whole fractions of the weight
#pragma unroll
  for (int k = 0; k < GGN_WARP_KEPT; ++k) {
    const int c = lane + 32 * k;
    if (c < width) {
      float y = (kept[k] * inv) * weight[(w0 + c) % weight_len];
      if (!gate_first) y *= gates[k];
      out[(size_t)t * out_ld + lo + c] = from_f32<TO>(y * scale);
    }
  }
}

// ---------------------------------------------------------------- chunks of a prompt as products
// The scan above costs an update and a read of the whole state for every token, and a thread reads a token's q and k from
// shared memory for one column of it: bounded by those reads (462 us for 2,048 rows of 16 heads of 128 x 128, and 228 for
// the pass that builds the chunks' states).  Over a chunk of C = 64 rows the same sums are products, with the decay's powers
// worked in (p_n = decay^n, n >= 0 only, so that nothing overflows):
//     own state of the chunk    U = sum_j p_(C-1-j) k_j v_j^T                                     (K^T V)
//     outputs                   o_i = sum_(j <= i) p_(i-j) (q_i . k_j) v_j + p_(i+1) S^T q_i      (Q K^T, P V, Q S)
// which is a third of the multiply-adds and lets a thread own 16 x 8 or 8 x 8 results: 116 us for the outputs and 56 for the
// states (the multiply-adds alone take 32 and 15).  Everything is float32, products are
// paired multiply-adds (two rounded operations an instruction).  For 64 < dim <= 128 (padded to 128 in shared memory); below, the
// scan does as well.  A chunk's products cost the same however few of its rows there are, so requests of up to LC_SHORT rows
// go to the scan, row by row from and into their slots: 256 rows beside 64 single ones 914 to 248 us, 64 requests of four rows 872
// to 192, eight of 17 115 to 58, 64 of 32 (where the two meet) 551 against 763 for 64 of 33 in chunks; 16 heads of 128 x 128.
constexpr int LC_SHORT = 32;
constexpr int LC_ROWS = 64, LC_DIM = 128, LC_THREADS = 128, LC_PITCH = LC_DIM + 4, LC_P_PITCH = LC_ROWS + 4;
constexpr size_t LC_OWN_SMEM = sizeof(float) * 2 * LC_ROWS * LC_PITCH;
constexpr size_t LC_OUT_SMEM = sizeof(float) * 3 * LC_ROWS * LC_PITCH;     // q | k, then P | v; at the end the state takes k's and v's place
static_assert(2 * LC_ROWS == LC_DIM && LC_P_PITCH <= LC_PITCH, "the state fits where k and v lay");

__device__ __forceinline__ void lc_fma_pair(uint64_t& c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t lc_pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 lc_halves(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

template <typename TD> struct LcInput {
  const TD* proj;
  int n_partials;
  long long partial_stride, ld;
  int act, wide;      // wide: one set of sums, four values at a time
};
// The rows row0 .. row0 + n - 1 of the columns col .. col + width - 1 of the projection, as this thread takes them: four
// columns of every fourth row.  All of them are asked for before the first is worked on (a few at a time, the round trips
// of a chunk's q, k and v took longer than its products).
constexpr int LC_MINE = LC_ROWS / (LC_THREADS / 32);
template <typename TD> struct LcRaw;
template <> struct LcRaw<float> { using Group = float4; Group v[LC_MINE]; };
template <> struct LcRaw<__nv_bfloat16> { using Group = uint2; Group v[LC_MINE]; };
__device__ __forceinline__ void lc_unpack(const float4& t, float (&v)[4]) { v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
__device__ __forceinline__ void lc_unpack(const uint2& t, float (&v)[4]) {
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&t.x), b = *reinterpret_cast<const __nv_bfloat162*>(&t.y);
  v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
}
template <typename TD>
__device__ __forceinline__ void lc_ask(LcRaw<TD>& raw, const LcInput<TD>& in, int col, int width, int row0, int n) {
  const int c = (threadIdx.x % 32) * 4;
  if (!in.wide) return;
#pragma unroll
  for (int i = 0; i < LC_MINE; ++i) {
    const int r = threadIdx.x / 32 + i * (LC_THREADS / 32);
    raw.v[i] = typename LcRaw<TD>::Group{};
    if (r < n && c < width)      // wide: whole groups of four
      raw.v[i] = *reinterpret_cast<const typename LcRaw<TD>::Group*>(in.proj + (size_t)(row0 + r) * in.ld + col + c);
  }
}
// Into dst (zeros beyond), then, every thread its own values, activated and times factor(row).  The second pass is a loop
// of its own that is not unrolled: with the activations of all values one behind the other the kernels did not fit the
// instruction cache (four cycles in five of a warp's went to waiting for instructions).
template <typename TD, typename Factor>
__device__ __forceinline__ void lc_put(float* dst, const LcRaw<TD>& raw, const LcInput<TD>& in, int col, int width, int row0, int n,
                                       Factor factor) {
  const int c = (threadIdx.x % 32) * 4, first = threadIdx.x / 32;
  if (in.wide) {
#pragma unroll
    for (int i = 0; i < LC_MINE; ++i) {
      float v[4];
      lc_unpack(raw.v[i], v);
      *reinterpret_cast<float4*>(dst + (first + i * (LC_THREADS / 32)) * LC_PITCH + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
#pragma unroll 1
    for (int e = 0; e < LC_MINE * 4; ++e) {
      const int r = first + e / 4 * (LC_THREADS / 32), x = c + e % 4;
      dst[r * LC_PITCH + x] = r < n && x < width
          ? la_load(in.proj + (size_t)(row0 + r) * in.ld + col + x, in.n_partials, in.partial_stride) : 0.f;
    }
  }
#pragma unroll 1
  for (int r = first; r < n; r += LC_THREADS / 32) {
    float4* at = reinterpret_cast<float4*>(dst + r * LC_PITCH + c);
    const float f = factor(r);
    float4 v = *at;
    v.x = la_act(v.x, in.act) * f; v.y = la_act(v.y, in.act) * f;
    v.z = la_act(v.z, in.act) * f; v.w = la_act(v.w, in.act) * f;
    *at = v;
  }
}
// Which rows chunk `index` has (row0, n), the chunks being numbered request by request; n = 0: there is no such chunk.
// Every thread of the block calls it; pow receives decay^0 .. decay^LC_ROWS.  Requests of up to LC_SHORT rows have none.
__device__ __forceinline__ void lc_chunk(const int* __restrict__ segment_start, int num_segments, int index, float decay,
                                         float* pow, int* slot, int& row0, int& n) {
  if (threadIdx.x == 0) {
    int before = 0;
    slot[0] = slot[1] = 0;
    for (int s = 0; s < num_segments; ++s) {
      const int a = segment_start[s], b = segment_start[s + 1];
      const int chunks = la_chunks(b - a, LC_ROWS, LC_SHORT);
      if (index < before + chunks) {
        slot[0] = a + (index - before) * LC_ROWS;
        slot[1] = min(b - slot[0], LC_ROWS);
        break;
      }
      before += chunks;
    }
  }
  if (threadIdx.x <= LC_ROWS) {
    float v = 1.f;
    for (int i = 0; i < (int)threadIdx.x; ++i) v *= decay;
    pow[threadIdx.x] = v;
  }
  __syncthreads();
  row0 = slot[0];
  n = slot[1];
}

// A chunk's own state: grid (chunks, heads, tiles of 128 columns).  A thread owns 16 x 8 of its 128 x 128 values; k and v lie
// in shared memory as the product wants them, rows side by side, and neighbouring rows of the state come as pairs.
template <typename TD>
__global__ void __launch_bounds__(LC_THREADS, 2)
linear_attention_own_states_kernel(const LcInput<TD> in, int k_off, int v_off, const float* __restrict__ decay,
                                   const int* __restrict__ segment_start, float* __restrict__ chunk_state, int heads, int dim,
                                   int vdim, int num_segments) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float pow_s[LC_ROWS + 1];
  __shared__ int slot[2];
  float* const k_s = smem;
  float* const v_s = smem + LC_ROWS * LC_PITCH;
  pdl_launch_dependents();
  const int h = blockIdx.y, col0 = blockIdx.z * LC_DIM;
  int row0, n;
  lc_chunk(segment_start, num_segments, blockIdx.x, decay[h], pow_s, slot, row0, n);
  pdl_wait();      // before any block leaves: a launch without chunks must not end ahead of the kernels before it
  if (n == 0) return;
  const int k_col = k_off + h * dim, v_col = v_off + h * vdim + col0;
  {
    LcRaw<TD> k_raw, v_raw;
    lc_ask(k_raw, in, k_col, dim, row0, n);
    lc_ask(v_raw, in, v_col, vdim - col0, row0, n);
    lc_put(k_s, k_raw, in, k_col, dim, row0, n, [&](int r) { return pow_s[n - 1 - r]; });
    lc_put(v_s, v_raw, in, v_col, vdim - col0, row0, n, [](int) { return 1.f; });
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d0 = (warp % 2) * 64 + (lane % 4) * 4;      // rows d0 + 16 i + (0 .. 3)
  const int e0 = (warp / 2) * 64 + (lane / 4) * 4;      // columns e0 + 32 j + (0 .. 3)
  uint64_t acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll 4
  for (int t = 0; t < LC_ROWS; ++t) {
    ulonglong2 a[4];
    float4 b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(k_s + t * LC_PITCH + d0 + 16 * i);
#pragma unroll
    for (int j = 0; j < 2; ++j) b[j] = *reinterpret_cast<const float4*>(v_s + t * LC_PITCH + e0 + 32 * j);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = j % 4 == 0 ? b[j / 4].x : j % 4 == 1 ? b[j / 4].y : j % 4 == 2 ? b[j / 4].z : b[j / 4].w;
      const uint64_t both = lc_pair(v, v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        lc_fma_pair(acc[2 * i][j], a[i].x, both);
        lc_fma_pair(acc[2 * i + 1][j], a[i].y, both);
      }
    }
  }
  float* const st = chunk_state + ((size_t)blockIdx.x * heads + h) * dim * vdim + col0;
  const bool wide = vdim % 4 == 0 && (((uintptr_t)chunk_state) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int d = d0 + 16 * (i / 4) + i % 4;
    if (d >= dim) continue;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      const int e = e0 + 8 * j;
      float v[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 both = lc_halves(acc[i / 2][j + x]);
        v[x] = i % 2 ? both.y : both.x;
      }
      float* out = st + (size_t)d * vdim + e;
      if (wide && col0 + e + 4 <= vdim) {
        *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (col0 + e + x < vdim) out[x] = v[x];
      }
    }
  }
}

// acc += A B: A rows [64][a_pitch] k fastest, B [k][LC_PITCH] columns fastest; rows m0 + 4 i, columns e0 + 32 (j / 2) + 2 (j % 2) ..
// CAUSAL: row r takes k <= r only (not as zeros times B: a later row may hold an infinity).
template <bool CAUSAL>
__device__ __forceinline__ void lc_product(uint64_t (&acc)[8][4], const float* a_src, int a_pitch, const float* b_src, int length,
                                           int m0) {
#pragma unroll 1
  for (int k = 0; k < length; k += 4) {
    float4 a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(a_src + 4 * i * a_pitch + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(b_src + (k + kk) * LC_PITCH);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(b_src + (k + kk) * LC_PITCH + 32);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (CAUSAL && k + kk > m0 + 4 * i) continue;
        const float v = kk == 0 ? a[i].x : kk == 1 ? a[i].y : kk == 2 ? a[i].z : a[i].w;
        const uint64_t both = lc_pair(v, v);
        lc_fma_pair(acc[i][0], both, b0.x);
        lc_fma_pair(acc[i][1], both, b0.y);
        lc_fma_pair(acc[i][2], both, b1.x);
        lc_fma_pair(acc[i][3], both, b1.y);
      }
    }
  }
}

// The outputs of a chunk from the state at its start: grid (chunks, heads, tiles of 128 columns).  A thread owns 8 x 8 of its
// 64 x 128 outputs, and 8 x 4 of the chunk's q . k.  101 KB of shared memory, so that of two blocks on an SM one computes
// while the other waits for its rows or its state.
template <typename TD>
__global__ void __launch_bounds__(LC_THREADS, 2)
linear_attention_outputs_kernel(const LcInput<TD> in, int q_off, int k_off, int v_off, const float* __restrict__ decay,
                                const int* __restrict__ segment_start, const float* __restrict__ chunk_state,
                                float* __restrict__ out, int heads, int dim, int vdim, int num_segments) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float pow_s[LC_ROWS + 1];
  __shared__ int slot[2];
  float* const q_s = smem;                              // [64][LC_PITCH]
  float* const k_s = q_s + LC_ROWS * LC_PITCH;          // [64][LC_PITCH], then P [64][LC_P_PITCH]; then the state [128][LC_PITCH]
  float* const v_s = k_s + LC_ROWS * LC_PITCH;          // [64][LC_PITCH]
  pdl_launch_dependents();
  const int h = blockIdx.y, col0 = blockIdx.z * LC_DIM;
  int row0, n;
  lc_chunk(segment_start, num_segments, blockIdx.x, decay[h], pow_s, slot, row0, n);
  pdl_wait();      // before any block leaves: a launch without chunks must not end ahead of the kernels before it
  if (n == 0) return;
  const int q_col = q_off + h * dim, k_col = k_off + h * dim, v_col = v_off + h * vdim + col0;
  {
    const auto one = [](int) { return 1.f; };
    LcRaw<TD> q_raw, k_raw, v_raw;
    lc_ask(q_raw, in, q_col, dim, row0, n);
    lc_ask(k_raw, in, k_col, dim, row0, n);
    lc_ask(v_raw, in, v_col, vdim - col0, row0, n);
    lc_put(q_s, q_raw, in, q_col, dim, row0, n, one);
    lc_put(k_s, k_raw, in, k_col, dim, row0, n, one);
    lc_put(v_s, v_raw, in, v_col, vdim - col0, row0, n, one);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m0 = (warp % 2) * 32 + lane % 4;            // rows m0 + 4 i
  const int t0 = (warp / 2) * 32 + lane / 4;            // rows of k: t0 + 8 j
  const int e0 = (warp / 2) * 64 + (lane / 4) * 4;      // columns
  const int length = (dim + 3) / 4 * 4;
  float s[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
  for (int d = 0; d < length; d += 4) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(k_s + (t0 + 8 * j) * LC_PITCH + d);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(q_s + (m0 + 4 * i) * LC_PITCH + d);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, s[i][j]))));
    }
  }
  __syncthreads();      // k has been used
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = m0 + 4 * i, t = t0 + 8 * j;
      k_s[r * LC_P_PITCH + t] = t <= r ? s[i][j] * pow_s[r - t] : 0.f;
    }
  for (int e = threadIdx.x; e < LC_ROWS * LC_DIM; e += LC_THREADS) q_s[e / LC_DIM * LC_PITCH + e % LC_DIM] *= pow_s[e / LC_DIM + 1];
  __syncthreads();
  uint64_t acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  lc_product<true>(acc, k_s + m0 * LC_P_PITCH, LC_P_PITCH, v_s + e0, LC_ROWS, m0);
  __syncthreads();      // P and v have been used: the state takes their place
  const float* const st = chunk_state + ((size_t)blockIdx.x * heads + h) * dim * vdim + col0;
  const bool wide = vdim % 4 == 0 && (((uintptr_t)chunk_state) & 15) == 0;
  for (int e = threadIdx.x; e < length * (LC_DIM / 4); e += LC_THREADS) {
    const int d = e / (LC_DIM / 4), c = e % (LC_DIM / 4) * 4;
    float* to = k_s + d * LC_PITCH + c;
    if (wide) {
      const bool inside = d < dim && col0 + c < vdim;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(to)),
                   "l"(inside ? st + (size_t)d * vdim + c : chunk_state), "r"(inside ? 16 : 0) : "memory");
    } else {
#pragma unroll
      for (int x = 0; x < 4; ++x) to[x] = d < dim && col0 + c + x < vdim ? st[(size_t)d * vdim + c + x] : 0.f;
    }
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  lc_product<false>(acc, q_s + m0 * LC_PITCH, LC_PITCH, k_s + e0, length, 0);
  const bool wide_out = vdim % 4 == 0 && (((uintptr_t)out) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = m0 + 4 * i;
    if (r >= n) continue;
    float* row = out + ((size_t)(row0 + r) * heads + h) * vdim + col0;
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const int e = e0 + 16 * j;
      const float2 a = lc_halves(acc[i][j]), b = lc_halves(acc[i][j + 1]);
      const float v[4] = {a.x, a.y, b.x, b.y};
      if (wide_out && col0 + e + 4 <= vdim) {
        *reinterpret_cast<float4*>(row + e) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (col0 + e + x < vdim) row[e + x] = v[x];
      }
    }
  }
}

template <typename TD>
int linear_attention_chunks(const void* proj, int n_partials, long long partial_stride, long long ld, int q_off, int k_off,
                            int v_off, const float* decay, float* state, const int* segment_start, const int* segment_slot,
                            float* out, int max_segments, int heads, int dim, int vdim, int act, int num_slots,
                            float* chunk_state, int max_chunks, cudaStream_t stream) {
  static SmemAllowance own_allowed, out_allowed;
  cudaError_t err = allow_smem(linear_attention_own_states_kernel<TD>, LC_OWN_SMEM, own_allowed);
  if (err == cudaSuccess) err = allow_smem(linear_attention_outputs_kernel<TD>, LC_OUT_SMEM, out_allowed);
  if (err != cudaSuccess) return (int)err;
  const bool wide = n_partials == 1 && (((uintptr_t)proj) & (4 * sizeof(TD) - 1)) == 0 && ld % 4 == 0 && q_off % 4 == 0 &&
                    k_off % 4 == 0 && v_off % 4 == 0 && dim % 4 == 0 && vdim % 4 == 0;
  const LcInput<TD> in = {(const TD*)proj, n_partials, partial_stride, ld, act, wide ? 1 : 0};
  const dim3 grid(max_chunks, heads, (vdim + LC_DIM - 1) / LC_DIM);
  const size_t per_state = (size_t)heads * dim * vdim;
  lse_launch(linear_attention_own_states_kernel<TD>, grid, LC_THREADS, LC_OWN_SMEM, stream, in, k_off, v_off, decay, segment_start,
             chunk_state, heads, dim, vdim, max_segments);
  lse_launch(linear_attention_carry_kernel<16>, dim3((unsigned)((per_state + 255) / 256), max_segments), 256, 0, stream, decay, state,
             segment_start, segment_slot, chunk_state, heads, dim, vdim, num_slots, LC_ROWS, LC_SHORT);
  lse_launch(linear_attention_outputs_kernel<TD>, grid, LC_THREADS, LC_OUT_SMEM, stream, in, q_off, k_off, v_off, decay,
             segment_start, (const float*)chunk_state, out, heads, dim, vdim, max_segments);
  LSE_LAUNCH_CHECK();
}
}  // namespace

extern "C" int lse_linear_attention_scan(const void* proj, int proj_dtype, int n_partials, long long partial_stride,
                                         long long ld, int q_off, int k_off, int v_off, const float* decay,
                                         float* state, const int* segment_start, const int* segment_slot, float* out,
                                         int max_segments, int heads, int dim, int vdim, int act, int num_slots,
                                         int chunk_rows, float* chunk_state, int max_chunks, cudaStream_t stream) {
  if (chunk_rows == LC_ROWS && dim > LC_DIM / 2 && dim <= LC_DIM && max_segments > 0 && heads > 0 && heads <= 65535 && vdim > 0 &&
      chunk_state != nullptr && max_chunks > 0 && n_partials >= 1 && (proj_dtype == LSE_DTYPE_F32 || proj_dtype == LSE_DTYPE_BF16)) {
#define LSE_LC_ARGS proj, n_partials, partial_stride, ld, q_off, k_off, v_off, decay, state, segment_start, segment_slot, out, \
  max_segments, heads, dim, vdim, act, num_slots, chunk_state, max_chunks, stream
    const int err = proj_dtype == LSE_DTYPE_F32 ? linear_attention_chunks<float>(LSE_LC_ARGS)
                                                : linear_attention_chunks<__nv_bfloat16>(LSE_LC_ARGS);
#undef LSE_LC_ARGS
    if (err != 0 || (max_segments == 1 && max_chunks > 1)) return err;      // one request of 64 rows or more: none is short
    return linear_attention_scan_launch<MODE_PLAIN>(proj, proj_dtype, n_partials, partial_stride, ld, q_off, k_off, v_off,
                                                    decay, state, segment_start, segment_slot, out, max_segments, heads,
                                                    dim, vdim, act, num_slots, 0, nullptr, 0, nullptr, nullptr, 1.0f, 0, 1,
                                                    nullptr, stream, LC_SHORT);
  }
  return linear_attention_scan_launch<MODE_PLAIN>(proj, proj_dtype, n_partials, partial_stride, ld, q_off, k_off, v_off,
                                                  decay, state, segment_start, segment_slot, out, max_segments, heads,
                                                  dim, vdim, act, num_slots, chunk_rows, chunk_state, max_chunks, nullptr,
                                                  nullptr, 1.0f, 0, 1, nullptr, stream);
}

extern "C" int lse_gated_rmsnorm(const float* o, const void* proj, int proj_dtype, int n_partials,
                                 long long partial_stride, long long ld, int g_off, const float* weight, void* out,
                                 int out_dtype, int tokens, int n, float eps, const int* segment_of_token,
                                 cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (n <= 0) return LSE_ERR_BAD_ARGUMENT;
  // one set of sums, groups of four values aligned wherever they are read or written; from 512 values on (2,048 rows of 512: 6.4
  // us either way, of 100: 6.4 against 4.2 with a value a thread)
  const size_t proj_group = proj_dtype == LSE_DTYPE_F32 ? 16 : 8, out_group = out_dtype == LSE_DTYPE_F32 ? 16 : 8;
  const bool vec = n_partials == 1 && n % 4 == 0 && n >= 512 && n <= 4 * 256 * GN_GROUPS && ld % 4 == 0 && g_off % 4 == 0 &&
                   (((uintptr_t)o | (uintptr_t)weight) & 15) == 0 && ((uintptr_t)proj & (proj_group - 1)) == 0 &&
                   ((uintptr_t)out & (out_group - 1)) == 0;
#define LSE_GN_CASE(TD, TO)                                                                                   \
  if (vec)                                                                                                    \
    lse_launch(gated_rmsnorm_vec_kernel<TD, TO>, tokens, 256, 0, stream, o, (const TD*)proj, ld, g_off, weight, \
               (TO*)out, n, eps, segment_of_token);                                                            \
  else                                                                                                        \
    lse_launch(gated_rmsnorm_kernel<TD, TO>, tokens, 256, 0, stream, o, (const TD*)proj, n_partials,          \
               partial_stride, ld, g_off, weight, (TO*)out, n, eps, segment_of_token);
  const bool d32 = proj_dtype == LSE_DTYPE_F32, o32 = out_dtype == LSE_DTYPE_F32;
  if (d32 && o32) { LSE_GN_CASE(float, float) }
  else if (d32 && !o32) { LSE_GN_CASE(float, __nv_bfloat16) }
  else if (!d32 && o32) { LSE_GN_CASE(__nv_bfloat16, float) }
  else { LSE_GN_CASE(__nv_bfloat16, __nv_bfloat16) }
#undef LSE_GN_CASE
  LSE_LAUNCH_CHECK();
}

// keep, take float32 [tokens, heads]; proj float32 / bfloat16 rows or a float32 stack of partial sums.
extern "C" int lse_ssd_gates(const void* proj, int proj_dtype, int n_partials, long long partial_stride, long long ld,
                             int dt_off, const float* dt_bias, const float* a_log, float* keep, float* take, int tokens,
                             int heads, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (heads <= 0 || n_partials < 1) return LSE_ERR_BAD_ARGUMENT;
  const unsigned blocks = (unsigned)(((long long)tokens * heads + 255) / 256);
  if (proj_dtype == LSE_DTYPE_F32)
    lse_launch(ssd_gates_kernel<float>, blocks, 256, 0, stream, (const float*)proj, n_partials, partial_stride, ld, dt_off,
               dt_bias, a_log, keep, take, tokens, heads);
  else if (proj_dtype == LSE_DTYPE_BF16)
    lse_launch(ssd_gates_kernel<__nv_bfloat16>, blocks, 256, 0, stream, (const __nv_bfloat16*)proj, n_partials,
               partial_stride, ld, dt_off, dt_bias, a_log, keep, take, tokens, heads);
  else
    return LSE_ERR_BAD_ARGUMENT;
  LSE_LAUNCH_CHECK();
}

// keep float32 [tokens, n] = sigmoid(proj[:, off .. off + n] + bias)^(1 / tau); bias float32 [n] or null.
extern "C" int lse_sigmoid_power(const void* proj, int proj_dtype, int n_partials, long long partial_stride, long long ld,
                                 int off, const float* bias, float tau, float* keep, int tokens, int n,
                                 cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (n <= 0 || n_partials < 1 || !(tau > 0.f)) return LSE_ERR_BAD_ARGUMENT;
  const long long blocks = ((long long)tokens * n + 255) / 256;
  if (blocks > 0x7fffffffLL) return LSE_ERR_TOO_LARGE;
  if (proj_dtype == LSE_DTYPE_F32)
    lse_launch(sigmoid_power_kernel<float>, (unsigned)blocks, 256, 0, stream, (const float*)proj, n_partials,
               partial_stride, ld, off, bias, 1.0f / tau, keep, tokens, n);
  else if (proj_dtype == LSE_DTYPE_BF16)
    lse_launch(sigmoid_power_kernel<__nv_bfloat16>, (unsigned)blocks, 256, 0, stream, (const __nv_bfloat16*)proj,
               n_partials, partial_stride, ld, off, bias, 1.0f / tau, keep, tokens, n);
  else
    return LSE_ERR_BAD_ARGUMENT;
  LSE_LAUNCH_CHECK();
}

// o float32 [tokens, n]; the gate in proj (float32 / bfloat16 / partial sums); xsrc (the output's dtype, rows x_ld apart) and
// skip float32 [n / head_width], or both null; weight float32 [weight_len], read at i % weight_len; out rows out_ld apart.
extern "C" int lse_gated_group_rmsnorm(const float* o, const void* proj, int proj_dtype, int n_partials,
                                       long long partial_stride, long long ld, int g_off, const void* xsrc, long long x_ld,
                                       int x_off, const float* skip, int head_width, const float* weight, int weight_len,
                                       void* out, int out_dtype, long long out_ld, int tokens, int n, int groups, float eps,
                                       float scale, int gate_first, int gate_act, const int* segment_of_token,
                                       cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (n <= 0 || groups <= 0 || n % groups || weight_len <= 0 || n_partials < 1 || (skip && (!xsrc || head_width <= 0)))
    return LSE_ERR_BAD_ARGUMENT;
  if (groups > 65535) return LSE_ERR_TOO_LARGE;
  const int width = n / groups;
  const int threads = width >= 1024 ? 256 : (width >= 256 ? 128 : (width > 32 ? 64 : 32));
  const dim3 grid(tokens, groups);
  const bool narrow = width <= 32 * GGN_WARP_KEPT;
  const long long warp_blocks = ((long long)tokens * groups + 7) / 8;
  if (narrow && warp_blocks > 0x7fffffffLL) return LSE_ERR_TOO_LARGE;
#define LSE_GGN_FORM(TD, TO, SINGLE)                                                                                 \
  if ((n_partials == 1) == SINGLE) {                                                                                 \
    if (narrow)                                                                                                      \
      lse_launch(gated_group_rmsnorm_warp_kernel<TD, TO, SINGLE>, (unsigned)warp_blocks, 256, 0, stream, o,           \
                 (const TD*)proj, n_partials, partial_stride, ld, g_off, (const TO*)xsrc, x_ld, x_off, skip,          \
                 head_width, weight, weight_len, (TO*)out, out_ld, tokens, n, groups, eps, scale, gate_first,         \
                 gate_act, segment_of_token);                                                                        \
    else                                                                                                             \
      lse_launch(gated_group_rmsnorm_kernel<TD, TO, SINGLE>, grid, threads, 0, stream, o, (const TD*)proj,            \
                 n_partials, partial_stride, ld, g_off, (const TO*)xsrc, x_ld, x_off, skip, head_width, weight,       \
                 weight_len, (TO*)out, out_ld, n, groups, eps, scale, gate_first, gate_act, segment_of_token);        \
  }
#define LSE_GGN_CASE(TD, TO)                                                                                         \
  {                                                                                                                  \
  LSE_GGN_FORM(TD, TO, true) else LSE_GGN_FORM(TD, TO, false)                                                        \
  }
  const bool d32 = proj_dtype == LSE_DTYPE_F32, o32 = out_dtype == LSE_DTYPE_F32;
  if (d32 && o32) LSE_GGN_CASE(float, float)
  else if (d32 && !o32) LSE_GGN_CASE(float, __nv_bfloat16)
  else if (!d32 && o32) LSE_GGN_CASE(__nv_bfloat16, float)
  else LSE_GGN_CASE(__nv_bfloat16, __nv_bfloat16)
#undef LSE_GGN_CASE
#undef LSE_GGN_FORM
  LSE_LAUNCH_CHECK();
}
