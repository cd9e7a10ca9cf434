// True float32 matrix product for the 32-bit path: C[M,N] = A[M,K] * B[N,K]^T (+ bias[N]).
//
// B is a weight matrix kept [out, in] as the checkpoint stores it
// (nn.Linear, reference src/llmserve/model.py:51-66).  Plain FMA on CUDA
// cores: no TF32, no reduced-precision staging.  The k range is cut into at most
// eight ranges of equal length (a multiple of 64, see f32_range); an output
// element is the sum of its ranges' sums in ascending order, starting from zero,
// and a range's sum is one fmaf per k in ascending order, starting from zero.  So
// a row's result does not depend on M, on the tile it falls in, on what else is
// in the batch, or on who adds the ranges up: the kernel itself, or (too few tiles
// to fill the GPU: a block per range) the kernel that consumes the stack of
// partial sums.
//
// Both kernels bring their tiles through a ring of shared-memory stages with cp.async.
#include "smem_allowance.cuh"
#include "tcgen05.cuh"

// Length of a k range: an eighth of K rounded up to a multiple of 64.
__host__ __device__ __forceinline__ int f32_range(int K) { return (((K + 7) / 8 + 63) / 64) * 64; }

namespace {
__device__ __forceinline__ uint32_t smem_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// `bytes` of the 16 (or 4) are fetched, the rest of the destination is zeroed; with 0 the source is not read
__device__ __forceinline__ void copy16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// ---------------------------------------------------------------- many rows
// A block owns a BM x BN tile, a warp a WM x WN part of it, a thread TM rows by TN columns, in groups of four.
// What bounds it is the width of a register write from shared memory, 128 bytes a clock and SM whether or not lanes read
// the same address: a k-value costs a thread TM + TN of them for TM TN of the 128 fused multiply-adds a clock, so a
// thread's part is made as large as its registers allow, 16 x 8.  The totals over the ranges, touched at most eight
// times, then have no room in registers: they lie in tensor memory (IN_TMEM), a column for each of the thread's 128.
// Tiles lie transposed in shared memory (cp.async of four bytes, which needs no alignment either), so that neighbouring
// rows of A come as register pairs for the paired multiply-add, two rounded operations an instruction: it leaves issue
// slots for the reads, which single ones do not.
// gridDim.z == 1: the block adds the ranges up itself.  Else block z takes range z and writes its sum to
// C + z * part_stride (no bias).
__device__ __forceinline__ void fma_pair(uint64_t& c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void halves(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}

constexpr int BK = 16, STAGES = 4;
template <int BM, int BN, int WM, int WN, int TM, int TN, bool IN_TMEM>
__global__ void __launch_bounds__((BM / WM) * (BN / WN) * 32, IN_TMEM ? 2 : 1)
gemm_f32_tiles_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ bias,
                      float* __restrict__ C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                      long long part_stride) {
  constexpr int THREADS = (BM / WM) * (BN / WN) * 32, A_PITCH = BM + 4, B_PITCH = BN + 4;
  constexpr int LM = WM / TM, LN = WN / TN;
  static_assert(LM * LN == 32 && TM % 4 == 0 && TN % 4 == 0, "a warp's lanes cover its part of the tile");
  static_assert(!IN_TMEM || (THREADS == 128 && TM * TN == 128), "a lane and 128 columns of tensor memory a thread");
  extern __shared__ __align__(16) float tiles[];
  __shared__ uint32_t tmem_slot;
  float* const As = tiles;                              // [STAGES][BK][A_PITCH]
  float* const Bs = tiles + STAGES * BK * A_PITCH;      // [STAGES][BK][B_PITCH]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int am = (warp % (BM / WM)) * WM + (lane % LM) * 4;        // this thread's first four rows; the others 4 LM apart
  const int bn = (warp / (BM / WM)) * WN + (lane / LM) * 4;        // its first four columns; the others 4 LN apart
  const int range = f32_range(K);
  const bool split = gridDim.z > 1;
  const int k_lo = split ? blockIdx.z * range : 0;
  const int k_hi = split ? min(K, k_lo + range) : K;
  const int n_tiles = (k_hi - k_lo + BK - 1) / BK;
  pdl_launch_dependents();
  if (IN_TMEM && warp == 0) tc::tmem_alloc(&tmem_slot, 128);

  // sixteen lanes fetch sixteen k-values of a row, a thread every THREADS / 16th row
  const int fk = tid % BK, fr = tid / BK;
  auto fetch = [&](const float* src, long long ld, int rows, int pitch, int row0, int limit, float* dst, int t) {
    const int k = k_lo + t * BK + fk;
    const float* from = src + (size_t)(row0 + fr) * ld + k;
    const uint32_t to = smem_address(dst + (t % STAGES) * BK * pitch + fk * pitch + fr);
#pragma unroll
    for (int r = 0; r < rows; r += THREADS / BK) {
      const bool in = row0 + fr + r < limit && k < K;
      copy4(to + 4 * r, in ? from + (size_t)r * ld : src, in ? 4 : 0);
    }
  };
  auto fetch_a = [&](int t) { fetch(A, lda, BM, A_PITCH, m0, M, As, t); };
  auto fetch_b = [&](int t) { fetch(B, ldb, BN, B_PITCH, n0, N, Bs, t); };

  // the weights do not depend on the kernels before this one; the rows do
#pragma unroll 1
  for (int t = 0; t < STAGES - 1; ++t)
    if (t < n_tiles) fetch_b(t);
  uint32_t tmem = 0;
  if (IN_TMEM) {
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tmem = tmem_slot + ((uint32_t)(warp * 32) << 16);
  }
  pdl_wait();
#pragma unroll 1
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < n_tiles) fetch_a(t);
    copies_commit();
  }
  uint64_t acc[TM / 2][TN];                               // pairs of neighbouring rows
  float total[IN_TMEM ? 1 : TM][IN_TMEM ? 1 : TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      if (i % 2 == 0) acc[i / 2][j] = 0;
      if (!IN_TMEM) total[i][j] = 0.f;
    }
  bool first = true;      // no range has ended yet

  for (int t = 0; t < n_tiles; ++t) {
    copies_wait<STAGES - 2>();
    __syncthreads();      // tile t is there, and everyone is done with the stage that is filled next
    if (t + STAGES - 1 < n_tiles) {
      fetch_a(t + STAGES - 1);
      fetch_b(t + STAGES - 1);
    }
    copies_commit();
    const float* a_src = As + (t % STAGES) * BK * A_PITCH + am;
    const float* b_src = Bs + (t % STAGES) * BK * B_PITCH + bn;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      ulonglong2 a[TM / 4];
      float4 b[TN / 4];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(a_src + kk * A_PITCH + i * 4 * LM);
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) b[j] = *reinterpret_cast<const float4*>(b_src + kk * B_PITCH + j * 4 * LN);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float v = j % 4 == 0 ? b[j / 4].x : j % 4 == 1 ? b[j / 4].y : j % 4 == 2 ? b[j / 4].z : b[j / 4].w;
        const uint64_t both = pair_of(v, v);
#pragma unroll
        for (int i = 0; i < TM / 4; ++i) {
          fma_pair(acc[2 * i][j], a[i].x, both);
          fma_pair(acc[2 * i + 1][j], a[i].y, both);
        }
      }
    }
    const bool last = t + 1 == n_tiles;
    if (last || ((t + 1) * BK) % range == 0) {   // the end of a range: its sum joins the total (from zero on)
      if (IN_TMEM) {
#pragma unroll
        for (int c = 0; c < 128; c += 32) {
          uint32_t sum[32];
          if (!first) {
            tc::tmem_ld32(tmem + c, sum);
            tc::tmem_ld_wait();
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            uint64_t& mine = acc[(c + e) / 2 / TN][(c + e) / 2 % TN];
            float lo, hi;
            halves(mine, lo, hi);
            lo = (first ? 0.f : __uint_as_float(sum[e])) + lo;
            hi = (first ? 0.f : __uint_as_float(sum[e + 1])) + hi;
            sum[e] = __float_as_uint(lo);
            sum[e + 1] = __float_as_uint(hi);
            mine = last ? pair_of(lo, hi) : 0;      // at the end the totals stay in acc
          }
          if (!last) tc::tmem_st32(tmem + c, sum);
        }
        if (!last) tc::tmem_st_wait();
        first = false;
      } else {
#pragma unroll
        for (int i = 0; i < TM; i += 2)
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            float lo, hi;
            halves(acc[i / 2][j], lo, hi);
            total[i][j] += lo;
            total[i + 1][j] += hi;
            acc[i / 2][j] = last ? pair_of(total[i][j], total[i + 1][j]) : 0;
          }
      }
    }
  }
  float* const dst = C + (split ? (size_t)blockIdx.z * part_stride : 0);
  const bool wide = (((uintptr_t)dst) & 15) == 0 && ldc % 4 == 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + am + (i / 4) * 4 * LM + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j += 4) {
      const int n = n0 + bn + (j / 4) * 4 * LN;
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float lo, hi;
        halves(acc[i / 2][j + e], lo, hi);
        v[e] = i % 2 ? hi : lo;
        if (bias && !split && n + e < N) v[e] += bias[n + e];
      }
      float* out = dst + (size_t)m * ldc + n;
      if (wide && n + 4 <= N) {
        *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) out[e] = v[e];
      }
    }
  }
  if (IN_TMEM) {
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem_slot, 128);
  }
}

// ---------------------------------------------------------------- few rows (at most 16)
// Decoding: the job is to stream B once.  A block owns 32 * TN * GROUPS columns; a warp TM of the ROWS rows, a lane TN
// columns of them (32 apart).  With one column and all eight rows a lane, the register writes of A took 36 of the 40
// clocks that 512 bytes of B took, so rows are dealt out to warps, which share the columns in shared memory.  Tiles lie as
// in global memory, k fastest; a row's pitch is 4 words beyond a multiple of 32, so that lanes reading 16 bytes of
// neighbouring rows meet no bank conflict.
// gridDim.y == 1: the block adds the ranges up itself.  Else block row y takes range y and writes its sum to
// C + y * part_stride (no bias).  Needs K % 4 == 0 and 16-byte aligned rows of A and B.
constexpr int FEW_ROWS = 16;

template <int ROWS, int TM, int TN, int GROUPS, int FEW_BK, int FEW_STAGES>
__global__ void __launch_bounds__(32 * GROUPS * (ROWS / TM))
gemm_f32_few_rows_kernel(const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ bias,
                         float* __restrict__ C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                         long long part_stride, int stages) {
  constexpr int THREADS = 32 * GROUPS * (ROWS / TM), COLS = 32 * TN * GROUPS;
  constexpr int FEW_PITCH = FEW_BK + 4, PER_ROW = FEW_BK / 4;
  extern __shared__ __align__(16) float tiles[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* const As = tiles;                                   // [stages][ROWS][FEW_BK]
  float* const Bs = tiles + stages * ROWS * FEW_BK;          // [stages][COLS][FEW_PITCH]
  const int n0 = blockIdx.x * COLS, col0 = (warp % GROUPS) * 32 * TN + lane, row0 = (warp / GROUPS) * TM;
  const int range = f32_range(K);
  const bool split = gridDim.y > 1;
  const int k_lo = split ? blockIdx.y * range : 0;
  const int k_hi = split ? min(K, k_lo + range) : K;
  const int n_tiles = (k_hi - k_lo + FEW_BK - 1) / FEW_BK;   // every one of them has a stage when they are at most FEW_STAGES
  pdl_launch_dependents();
  const int fc = (threadIdx.x % PER_ROW) * 4, fr = threadIdx.x / PER_ROW;
  auto fetch_b = [&](int t) {
    const int k = k_lo + t * FEW_BK + fc;
    const float* from = B + (size_t)(n0 + fr) * ldb + k;
    const uint32_t to = smem_address(Bs + ((t % FEW_STAGES) * COLS + fr) * FEW_PITCH + fc);
#pragma unroll 8
    for (int r = 0; r < COLS; r += THREADS / PER_ROW) {
      const bool in = n0 + fr + r < N && k < K;
      copy16(to + 4 * r * FEW_PITCH, in ? from + (size_t)r * ldb : B, in ? 16 : 0);
    }
  };
  auto fetch_a = [&](int t) {
    const int k = k_lo + t * FEW_BK + fc;
#pragma unroll
    for (int r = fr; r < ROWS; r += THREADS / PER_ROW) {
      const bool in = r < M && k < K;
      copy16(smem_address(As + ((t % FEW_STAGES) * ROWS + r) * FEW_BK + fc), in ? A + (size_t)r * lda + k : A, in ? 16 : 0);
    }
  };
  // the weights do not depend on the kernels before this one; the rows do
#pragma unroll 1
  for (int t = 0; t < FEW_STAGES - 1; ++t)
    if (t < n_tiles) fetch_b(t);
  pdl_wait();
#pragma unroll 1
  for (int t = 0; t < FEW_STAGES - 1; ++t) {
    if (t < n_tiles) fetch_a(t);
    copies_commit();
  }
  float acc[TM][TN], total[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.f;
  for (int t = 0; t < n_tiles; ++t) {
    copies_wait<FEW_STAGES - 2>();
    if (THREADS > 32) __syncthreads();       // tile t is there, and everyone is done with the stage that is filled next
    else __syncwarp();
    if (t + FEW_STAGES - 1 < n_tiles) {
      fetch_b(t + FEW_STAGES - 1);
      fetch_a(t + FEW_STAGES - 1);
    }
    copies_commit();
    const float* b_src = Bs + ((t % FEW_STAGES) * COLS + col0) * FEW_PITCH;
    const float* a_src = As + ((t % FEW_STAGES) * ROWS + row0) * FEW_BK;
    float4 a[2][TM], b[2][TN];               // the next four k-values are read while four are worked on
    auto read = [&](int kk, float4 (&av)[TM], float4 (&bv)[TN]) {
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = *reinterpret_cast<const float4*>(b_src + j * 32 * FEW_PITCH + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a_src + i * FEW_BK + kk);
    };
    read(0, a[0], b[0]);
#pragma unroll
    for (int kk = 0; kk < FEW_BK; kk += 4) {
      const int now = (kk / 4) & 1;
      if (kk + 4 < FEW_BK) read(kk + 4, a[now ^ 1], b[now ^ 1]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[now][i].x, b[now][j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[now][i].y, b[now][j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[now][i].z, b[now][j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[now][i].w, b[now][j].w, acc[i][j]);
    }
    if (((t + 1) * FEW_BK) % range == 0 || t + 1 == n_tiles) {   // the end of a range
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) { total[i][j] += acc[i][j]; acc[i][j] = 0.f; }
    }
  }
  float* const dst = C + (split ? (size_t)blockIdx.y * part_stride : 0);
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + col0 + j * 32;
      if (row0 + i < M && n < N)
        dst[(size_t)(row0 + i) * ldc + n] = (bias && !split) ? total[i][j] + bias[n] : total[i][j];
    }
  }
}

struct Product {
  const float *A, *B, *bias;
  float* C;
  int M, N, K;
  long long lda, ldb, ldc, part_stride;
  int ranges;      // 1: the kernel adds the ranges up
};

template <int BM, int BN, int WM, int WN, int TM, int TN, bool IN_TMEM>
cudaError_t launch_tiles(const Product& p, cudaStream_t stream) {
  auto kernel = gemm_f32_tiles_kernel<BM, BN, WM, WN, TM, TN, IN_TMEM>;
  const size_t smem = sizeof(float) * STAGES * BK * (BM + BN + 8);
  static SmemAllowance allowed;
  cudaError_t err = allow_smem(kernel, smem, allowed);
  if (err != cudaSuccess) return err;
  // tiles of columns lie in the grid's second dimension, which ends at 65,535 (numbered in the first they cost a hundredth of
  // the product: the compiler schedules the loop worse)
  for (long long n = 0; n < p.N && err == cudaSuccess; n += 65535LL * BN) {
    const int cols = (int)(p.N - n < 65535LL * BN ? p.N - n : 65535LL * BN);
    const dim3 grid((p.M + BM - 1) / BM, (cols + BN - 1) / BN, p.ranges);
    err = lse_launch(kernel, grid, (BM / WM) * (BN / WN) * 32, smem, stream, p.A, p.B + n * p.ldb,
                     p.bias ? p.bias + n : nullptr, p.C + n, p.M, cols, p.K, p.lda, p.ldb, p.ldc, p.part_stride);
  }
  return err;
}

template <int ROWS, int TM, int TN, int GROUPS, int FEW_BK, int FEW_STAGES>
cudaError_t launch_few(const Product& p, cudaStream_t stream) {
  constexpr int COLS = 32 * TN * GROUPS;
  auto kernel = gemm_f32_few_rows_kernel<ROWS, TM, TN, GROUPS, FEW_BK, FEW_STAGES>;
  const int length = p.ranges > 1 ? f32_range(p.K) : p.K;
  const int tiles = (length + FEW_BK - 1) / FEW_BK, stages = tiles < FEW_STAGES ? tiles : FEW_STAGES;
  const size_t smem = sizeof(float) * stages * (COLS * (FEW_BK + 4) + ROWS * FEW_BK);
  static SmemAllowance allowed;
  cudaError_t err = allow_smem(kernel, smem, allowed);
  if (err != cudaSuccess) return err;
  const dim3 grid((p.N + COLS - 1) / COLS, p.ranges);
  return lse_launch(kernel, grid, 32 * GROUPS * (ROWS / TM), smem, stream, p.A, p.B, p.bias, p.C, p.M, p.N, p.K, p.lda,
                    p.ldb, p.ldc, p.part_stride, stages);
}

int gpu_sms() {
  static int count = 0;
  if (count == 0) {
    int device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device);
    if (count <= 0) count = 148;
  }
  return count;
}

bool aligned(const float* A, const float* B, int K, long long lda, long long ldb) {
  return K % 4 == 0 && lda % 4 == 0 && ldb % 4 == 0 && (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
}

// Time of a product with tiles of BM x BN, in microseconds: a wave of `at_once` blocks an SM takes `per_k` a k-value
// whether it is full or not (measured on 1,536 k-values: 288, 161 and 154 us), and what does not fill a last wave costs
// about a quarter of one.  Of 2,048 x 17,920 x 1,536 the three take 2,309, 2,581 and 3,055 us (49 TFLOP/s; 6,442 with
// 64 x 64 tiles, 4 x 4 a thread, which this kernel replaced); of 64 x 17,920 169, 93 and 111 us as a stack (455).
struct Tiling { int bm, bn, at_once; double per_k; };
constexpr Tiling TILINGS[3] = {{128, 128, 2, 0.1875}, {64, 128, 2, 0.105}, {32, 64, 6, 0.1}};
double tiling_time(const Tiling& t, int M, int N, int K, int ranges) {
  const double blocks = (double)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn) * ranges;
  const double waves = blocks / ((double)gpu_sms() * t.at_once);
  return (waves <= 1.0 ? 1.0 : waves + 0.25) * t.per_k * (ranges > 1 ? f32_range(K) : K);
}
int best_tiling(int M, int N, int K, int ranges, double* time) {
  int best = 0;
  for (int i = 0; i < 3; ++i) {
    const double t = tiling_time(TILINGS[i], M, N, K, ranges);
    if (i == 0 || t < *time) { *time = t; best = i; }
  }
  return best;
}

// Few rows.  Wide products (blocks enough for eight an SM) stream best with two columns a lane (8 rows) or four (16) and
// short tiles, many small blocks; narrow ones, whose blocks all run at once, with long tiles and what is left to a lane.
// 8 x 17,920 x 1,536 as a stack: 24.5 against 27 us (87.5 with the kernel this one replaced; the weights' 110 MB alone
// take 17), 8 x 1,536 x 8,960: 27 against 22.7 us (82), 16 rows: 35 against 57 and 50 against 34 us (88 and 82).
cudaError_t few_rows(const Product& p, cudaStream_t stream) {
  const bool wide = (long long)((p.N + 63) / 64) * p.ranges >= 8LL * gpu_sms();
  if (p.M == 1) return launch_few<1, 1, 1, 1, 64, 4>(p, stream);
  if (p.M == 2) return launch_few<2, 2, 1, 1, 64, 4>(p, stream);
  if (p.M <= 4) return launch_few<4, 2, 1, 1, 64, 4>(p, stream);
  if (p.M <= 8) return wide ? launch_few<8, 4, 2, 1, 32, 4>(p, stream) : launch_few<8, 4, 1, 1, 64, 4>(p, stream);
  // four columns a lane leave blocks of 128 columns: where those are few, one column a lane is better (2,048 x 1,536 whole 21.6
  // against 43.6 us with 16 blocks of 128 columns, 1,536 x 8,960 whole 120 against 251 with 12; as stacks 8.0 against 6.5 with
  // 128, 33 either way with 84)
  if ((long long)((p.N + 127) / 128) * p.ranges < 64) return launch_few<16, 4, 1, 1, 64, 4>(p, stream);
  return wide ? launch_few<16, 4, 4, 1, 32, 3>(p, stream) : launch_few<16, 4, 4, 1, 64, 3>(p, stream);
}
}  // namespace

// How many ranges the k range of a product is cut into (the height of a stack of partial sums).
extern "C" int lse_gemm_f32_ranges(int K) { return K <= 0 ? 0 : (K + f32_range(K) - 1) / f32_range(K); }

// stack != 0: C is a stack [lse_gemm_f32_ranges(K)][M rows of ldc] (part_stride elements apart) of the ranges' sums,
// for a consumer that adds them up in index order starting from zero; no bias.  stack 1: few rows only (M <= 16,
// K % 4 == 0, aligned: lse_gemm_f32_stack_ok); 2: any number of them (see lse_gemm_f32_stack_wanted).
extern "C" int lse_gemm_f32_stack_ok(const float* A, const float* B, int M, int K, long long lda, long long ldb) {
  return (M > 0 && M <= FEW_ROWS && K > 0 && aligned(A, B, K, lda, ldb)) ? 1 : 0;
}

// Whether a product of more than 16 rows should be taken as a stack: its tiles alone would leave much of the GPU idle,
// and a block per range wins more than it costs the consumer to read the stack (at 6.5 TB/s; 1 us is left for the rest).
extern "C" int lse_gemm_f32_stack_wanted(const float* A, const float* B, int M, int N, int K, long long lda, long long ldb) {
  if (M <= FEW_ROWS || N <= 0 || K <= 0 || !aligned(A, B, K, lda, ldb)) return 0;
  const int ranges = lse_gemm_f32_ranges(K);
  if (ranges < 2) return 0;
  double whole, cut;
  best_tiling(M, N, K, 1, &whole);
  best_tiling(M, N, K, ranges, &cut);
  return whole - cut > 4.0 * ranges * M * N / 6.5e6 + 1.0 ? 1 : 0;
}

extern "C" int lse_gemm_f32_nt(const float* A, const float* B, const float* bias, float* C, int M,
                               int N, int K, long long lda, long long ldb, long long ldc, int stack,
                               long long part_stride, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return LSE_ERR_BAD_ARGUMENT;
  const bool vec = aligned(A, B, K, lda, ldb);
  if (stack && (!vec || bias != nullptr || (stack == 1 && M > FEW_ROWS))) return LSE_ERR_BAD_ARGUMENT;
  const Product p = {A, B, bias, C, M, N, K, lda, ldb, ldc, part_stride, stack ? lse_gemm_f32_ranges(K) : 1};
  cudaError_t err;
  if (M <= FEW_ROWS && vec) {
    err = few_rows(p, stream);
  } else {
    double time;
    const int tiling = best_tiling(M, N, K, p.ranges, &time);
    err = tiling == 0 ? launch_tiles<128, 128, 64, 64, 16, 8, true>(p, stream)
        : tiling == 1 ? launch_tiles<64, 128, 32, 64, 8, 8, false>(p, stream)
                      : launch_tiles<32, 64, 16, 64, 4, 8, false>(p, stream);
  }
  if (err != cudaSuccess) return (int)err;
  LSE_LAUNCH_CHECK();
}
