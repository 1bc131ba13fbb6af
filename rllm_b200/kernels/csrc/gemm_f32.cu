// C[M, N] = A[M, K] . W[N, K]^T in true float32: FFMA on CUDA cores, no tensor
// cores and no reduced-precision matrix mode.  This is every projection of the
// 32-bit path (the reference calls a library matmul there,
// crates/rllm-model/src/layers.rs:162-175).
//
// Each output element is one thread's sequential sum over k = 0 .. K-1, so a
// row's result does not depend on M: the same token gives the same bits alone,
// in a portion of a prompt or in a mixed batch, whichever tile it falls into.
//
// Rows of A and W go into shared memory as they lie (k contiguous) through a ring of
// cp.async stages, and a thread reads four k of its TM + TN rows at a time: rows are
// BK + 4 floats apart, so eight neighbouring lanes' 16-byte reads of eight rows hit all
// banks once.  Since no sum may be cut along k, the outputs a thread makes are what
// spreads a small product over the GPU; it then has a CTA of four warps an SM, too few to
// hide a stage's loads and shared-memory reads (K dependent multiply-adds are 4 of its
// 33 us at K = 2,048); a large one is bound by FFMA issue.
#include "common.cuh"

// VEC: 16-byte copies (rows start on 16 bytes), else 4-byte copies
template <int BM, int BN, int TM, int TN, int BK, int STAGES>
struct GemmF32 {
  static constexpr int NG = BN / TN, MG = BM / TM, THREADS = NG * MG, LD = BK + 4;
  static constexpr int STAGE = (BM + BN) * LD;                 // floats
  static constexpr int SMEM = STAGES * STAGE * 4;
};

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                float* __restrict__ C, int ldc, int M, int N, int K) {
  typedef GemmF32<BM, BN, TM, TN, BK, STAGES> S;
  extern __shared__ __align__(16) float gf_smem[];
  const int tid = threadIdx.x, tn = tid % S::NG, tm = tid / S::NG;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int steps = (K + BK - 1) / BK;

  auto load = [&](int step) {
    float* st = gf_smem + (step % STAGES) * S::STAGE;
    const int k0 = step * BK;
    constexpr int WIDE = VEC ? 4 : 1, PER_ROW = BK / WIDE, TOTAL = (BM + BN) * PER_ROW;
#pragma unroll
    for (int c = tid; c < TOTAL; c += S::THREADS) {
      const int r = c / PER_ROW, k = (c % PER_ROW) * WIDE;
      const bool in_a = r < BM;
      const int g = in_a ? m0 + r : n0 + r - BM;
      const bool ok = (in_a ? g < M : g < N) && k0 + k < K;
      const float* src = in_a ? A + (size_t)g * lda + k0 + k : W + (size_t)g * ldw + k0 + k;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(st + r * S::LD + k);
      const int n = ok ? min(WIDE, K - k0 - k) * 4 : 0;         // what lies behind K or the matrix is zero
      if (VEC)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(ok ? src : A), "r"(n) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(ok ? src : A), "r"(n) : "memory");
    }
  };

  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) load(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                       // stage s has landed for everyone, and everyone has left step s - 1
    if (s + STAGES - 1 < steps) load(s + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = gf_smem + (s % STAGES) * S::STAGE + tm * S::LD;
    const float* ws = gf_smem + (s % STAGES) * S::STAGE + (BM + tn) * S::LD;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *(const float4*)(as + i * S::MG * S::LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *(const float4*)(ws + j * S::NG * S::LD + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + tm + i * S::MG;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tn + j * S::NG;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
static int gf_launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                     cudaStream_t stream) {
  typedef GemmF32<BM, BN, TM, TN, BK, STAGES> S;
  static SmemLimit limit;
  if (const int e = limit.allow(gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES, VEC>, S::SMEM)) return e;
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return RLLM_E_UNSUPPORTED;
  gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES, VEC><<<grid, S::THREADS, S::SMEM, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);
  RLLM_LAUNCH_CHECK();
  return 0;
}

// Tiles of 64 x 64 staged through registers, k by k: no padding of a short k to the ring's 32 or 64, and rows that start
// off 16 bytes cost it nothing more.
#define GF_BM 64
#define GF_BN 64
#define GF_BK 16
__global__ void __launch_bounds__(256)
gemm_f32_staged_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                       float* __restrict__ C, int ldc, int M, int N, int K) {
  __shared__ float As[GF_BK][GF_BM + 4];
  __shared__ float Ws[GF_BK][GF_BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * GF_BM, n0 = blockIdx.x * GF_BN;
  const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  // each thread loads 4 elements of A and 4 of W per k-tile: row = tid / 4, k = (tid % 4) * 4 ..
  const int lr = tid / 4, lk = (tid % 4) * 4;
  for (int k0 = 0; k0 < K; k0 += GF_BK) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + lk + u;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + u][lr] = (am < M && k < K) ? A[(size_t)am * lda + k] : 0.f;
      Ws[lk + u][lr] = (wn < N && k < K) ? W[(size_t)wn * ldw + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GF_BK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][tm + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[k][tn + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + tm + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tn + j;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

// The tile: 64 x 64 where that leaves two CTAs an SM, else 32 x 32, 16 x 32 or, for up to 8 rows or few columns, 8 x 32.
// Microseconds (one tile of 64 x 64 for everything, scalar loads, no ring -> this form; M x N x K):
// 1 x 16384 x 2048 223 -> 43, 8 x 2048 x 8192 723 -> 62, 16 x 4096 x 2048 178 -> 25, 96 x 4096 x 1024 87 -> 35,
// 96 x 1024 x 2048 155 -> 33, 128 x 16384 x 3072 592 -> 360 (36 TFLOP/s), 2048 x 4096 x 2048 1341 -> 805.
// Where the lines lie: 96 x 4096 x 1024 in tiles of 64 / 32 / 16 rows 41 / 35 / 53 us; 96 x 1024 x 2048 (96 tiles of 32)
// 76 / 33 / 35; 24 x 2048 x 8192 (64 tiles of 32, 128 of 16) 291 / 118 / 84; 8 x 16384 x 2048 in 16 / 8 rows 62 / 45.
// Results of many 64 x 64 tiles go to the staged kernel where the ring pads k (K below 64) or copies 4 bytes at a time (rows
// off 16 bytes).  Staged / ring, M x N x K: 200 x 4096 x 16 4.8 / 8.2, 2048 x 32000 x 16 103 / 137 but x 32 198 / 138,
// 64 x 16000 x 24 6.2 / 9.1, 33 x 16000 x 48 6.9 / 8.7; rows off 16 bytes 200 x 4096 x 101 14 / 18, 2048 x 32000 x 101 490 / 651,
// 64 x 16000 x 257 30 / 38 but x 1025 105 / 105, 512 x 4096 x 1025 171 / 178, and 96 x 4096 x 257 (128 tiles) 24 / 18,
// 17 x 32000 x 257 44 / 37.  Both add in the same order: the same bits.
static bool gf_staged(bool vec, int M, int N, int K) {
  const long long tiles = (long long)((M + 63) / 64) * ((N + 63) / 64);
  if (vec) return (K <= 16 && tiles >= 64) || (K < 64 && M > 16 && tiles >= 128 && tiles < 600);
  if (M <= 32) return K < 64 && M > 16 && tiles >= 128;
  return (tiles >= 64 && K < 32) || (tiles >= 128 && (K < 128 || (K < 512 && tiles >= 192) || (M >= 256 && tiles >= 192)));
}

template <bool VEC>
static int gf_choose(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                     cudaStream_t stream) {
  auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
  if (M > 32 && tiles(64, 64) >= 296) return gf_launch<64, 64, 8, 4, 32, 3, VEC>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M > 16 && tiles(32, 32) >= 96) return gf_launch<32, 32, 4, 2, 64, 3, VEC>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M > 8 && tiles(16, 32) >= 96) return gf_launch<16, 32, 2, 2, 64, 4, VEC>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  return gf_launch<8, 32, 2, 1, 64, 5, VEC>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}

RLLM_EXPORT int rllm_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                              int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return RLLM_E_BADARG;
  const bool vec = lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  if (gf_staged(vec, M, N, K)) {
    const dim3 grid((N + GF_BN - 1) / GF_BN, (M + GF_BM - 1) / GF_BM);
    if (grid.y > 65535) return RLLM_E_UNSUPPORTED;
    gemm_f32_staged_kernel<<<grid, 256, 0, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);
    RLLM_LAUNCH_CHECK();
    return 0;
  }
  return vec ? gf_choose<true>(A, lda, W, ldw, C, ldc, M, N, K, stream)
             : gf_choose<false>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}
