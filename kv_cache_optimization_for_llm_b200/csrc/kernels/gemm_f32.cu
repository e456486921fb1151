// True 32-bit matrix product for the float32 path:  C[M,N] = A[M,K] . W[N,K]^T
// (the linear layers' y = x . W^T with W stored [out, in]; upstream does this with
// cublasGemmEx on bfloat16, base/src/engine.cu:643-671).
//
// Plain FMA on CUDA cores, no tensor cores: a tf32 product would drop mantissa bits
// and this path exists to show what bfloat16 hides.  Every output element is one
// chain of fmaf over k = 0..K-1 in ascending order, so a row's result does not
// depend on how many other rows the call holds or on which tile it falls into.
//
// What bounds it: the FMA pipe (74 TFLOP/s at 1.965 GHz).  The chain's order forbids splitting K, so the only freedom is
// the tile.  A thread owns TM x TN outputs, two neighbouring columns in one 64-bit register pair: `fma.rn.f32x2` rounds
// each half as fmaf does and takes half the issue slots, which leaves room for the shared-memory loads that feed it and for pairing
// a row's value with itself (exchanging the halves of pairs of rows instead was no faster).  Pieces of 16 k are brought into a ring
// of kStages buffers, transposed on the way (4-byte cp.async, which also takes any alignment and fills what lies outside with
// zeros): with one or two warps per scheduler nothing else hides the latency of a load.  Measured (M x N x K, this kernel / one of
// 64 x 64 tiles with 4 x 4 outputs a thread and loads one by one): 338 x 16384 x 2048 581 / 1280 us, 338 x 2048 x 8192
// 512 / 660, 2048 x 2048 x 2048 400 / 780 us (43 TFLOP/s; the busiest SMs' FMA pipes are active 69 % of the time, the rest
// is the loads' latency and tiles that do not divide by the SMs).
#include "common.cuh"

constexpr int BK = 16, kStages = 4;

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 pack(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void copy4(float* to, const float* from, bool inside) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
               "r"(inside ? 4 : 0) : "memory");
}

// A warp's 32 lanes stand 4 (rows) x 8 (columns); a lane's rows come in groups of four, 16 apart, its columns in groups of
// four, 32 apart.
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(BM / (4 * TM) * (BN / (8 * TN)) * 32)
sgemm_nt_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                float* __restrict__ C, int ldc, int M, int N, int K) {
  constexpr int WM = BM / (4 * TM), WN = BN / (8 * TN), THREADS = WM * WN * 32;
  // rows of the transposed pieces are padded by four: the lanes of a copy hold 16 consecutive k of two rows
  constexpr int LD = BM + BN + 8, STAGE = BK * LD, PER = ((BM + BN) * BK + THREADS - 1) / THREADS;
  static_assert(THREADS % BK == 0, "a thread copies one k of its rows");
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int row = (warp % WM) * 4 * TM + (lane >> 3) * 4, col = BM + 4 + (warp / WM) * 8 * TN + (lane & 7) * 4;
  const int ck = tid % BK, cr = tid / BK;              // this thread's k, and the first of its rows (A's, then W's)
  auto bring = [&](int step) {
    const int k = step * BK + ck;
    float* to = sm + step % kStages * STAGE + ck * LD;
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const int r = cr + x * (THREADS / BK);
      if (r < BM) {
        const bool in = m0 + r < M && k < K;
        copy4(to + r, in ? A + (size_t)(m0 + r) * lda + k : A, in);
      } else if (r < BM + BN) {
        const bool in = n0 + r - BM < N && k < K;
        copy4(to + r + 4, in ? W + (size_t)(n0 + r - BM) * ldw + k : W, in);
      }
    }
  };
  f32x2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
  const int steps = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < steps) bring(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();                                   // the piece is there, and nobody reads the buffer that is filled next
    if (step + kStages - 1 < steps) bring(step + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* piece = sm + step % kStages * STAGE;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
      f32x2 w[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4)
        *reinterpret_cast<float4*>(a + i) = *reinterpret_cast<const float4*>(piece + kk * LD + row + (i >> 2) * 16);
#pragma unroll
      for (int j = 0; j < TN; j += 4) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(piece + kk * LD + col + (j >> 2) * 32);
        w[j / 2] = v.x;
        w[j / 2 + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const f32x2 aa = pack(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(aa, w[j], acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + row + (i >> 2) * 16 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; j += 2) {
      const int n = n0 + col - BM - 4 + (j >> 2) * 32 + (j & 3);
      const float2 v = unpack(acc[i][j / 2]);
      if (n < N) C[(size_t)m * ldc + n] = v.x;
      if (n + 1 < N) C[(size_t)m * ldc + n + 1] = v.y;
    }
  }
}

// The tiles, and what one of them costs per 2048 k (microseconds, measured): alone on its SM (`alone`; a chain cannot be
// faster than its own latencies), and as one of many that an SM works through, two to eight of them side by side (`beside`).
struct SgemmTile { int bm, bn; float alone, beside; };
static const SgemmTile kSgemmTiles[] = {{128, 128, 207, 192}, {64, 128, 130, 105}, {64, 64, 111, 72}, {32, 64, 66, 45}, {32, 32, 56, 26.5f}, {16, 32, 59, 17}};
constexpr int kSgemmTileCount = sizeof(kSgemmTiles) / sizeof(kSgemmTiles[0]);

// Padding k beyond K with zeros adds exact zeros to the chain, so the result equals
// the unpadded chain.  Any M, N, K >= 1; leading dimensions in elements.
// tile < 0: the one with which the busiest SM (ceil(tiles / SMs) of them) is done soonest; the results are the same with each.
KVB_EXPORT int kvb_sgemm_nt_tile(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                                 int M, int N, int K, int tile, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || tile >= kSgemmTileCount) return KVB_ERR_BAD_SIZE;
  if (tile < 0) {
    double best = 0.0;
    for (int i = 0; i < kSgemmTileCount; ++i) {
      const SgemmTile& t = kSgemmTiles[i];
      const long long tiles = (long long)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn);
      const double all = (double)((tiles + kvb_sm_count() - 1) / kvb_sm_count()) * t.beside, cost = all > t.alone ? all : t.alone;
      if ((M + t.bm - 1) / t.bm <= 65535 && (tile < 0 || cost < best)) { tile = i; best = cost; }
    }
    if (tile < 0) return KVB_ERR_BAD_SIZE;
  }
  const SgemmTile& t = kSgemmTiles[tile];
  const dim3 grid((N + t.bn - 1) / t.bn, (M + t.bm - 1) / t.bm);
  if (grid.y > 65535) return KVB_ERR_BAD_SIZE;
#define KVB_SGEMM(BM, BN, TM, TN)                                                                                        \
  {                                                                                                                    \
    constexpr int threads = BM / (4 * TM) * (BN / (8 * TN)) * 32, smem = kStages * BK * (BM + BN + 8) * 4;             \
    if (smem > 48 * 1024) {                                                                                            \
      cudaError_t e = cudaFuncSetAttribute(sgemm_nt_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); \
      if (e != cudaSuccess) return (int)e;                                                                             \
    }                                                                                                                  \
    sgemm_nt_kernel<BM, BN, TM, TN><<<grid, threads, smem, stream>>>(A, lda, W, ldw, C, ldc, M, N, K);                 \
    break;                                                                                                             \
  }
  switch (tile) {
    case 0: KVB_SGEMM(128, 128, 8, 16)
    case 1: KVB_SGEMM(64, 128, 8, 8)
    case 2: KVB_SGEMM(64, 64, 8, 4)
    case 3: KVB_SGEMM(32, 64, 4, 4)
    case 4: KVB_SGEMM(32, 32, 4, 4)
    case 5: KVB_SGEMM(16, 32, 4, 4)
  }
#undef KVB_SGEMM
  return kvb_launch_result();
}

KVB_EXPORT int kvb_sgemm_nt(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                            int M, int N, int K, cudaStream_t stream) {
  return kvb_sgemm_nt_tile(A, lda, W, ldw, C, ldc, M, N, K, -1, stream);
}

#include "gemm_f32_split.cuh"
