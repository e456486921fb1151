// float32 products on the tensor cores without losing precision:  C[M,N] = A[M,K] . W[N,K]^T.
//
// Every float32 operand is the sum of three bfloat16 numbers (8 + 8 + 8 bits of mantissa; each part is the rounding of what the
// parts before it left over, and what the three leave is below 2^-26 of the value).  Of the nine partial products the six
// that matter are made on tcgen05 (bfloat16 products are exact in float32): hi hi, hi mid, mid hi, hi lo, lo hi, mid mid; the
// others are below 2^-26 of the product.  A tensor core's accumulator truncates, so no sum stays in it for
// longer than 64 k: float32 additions that round to nearest add these pieces up.  Root mean square error over that of the result,
// normal operands: 3.2e-7 to 3.4e-7 for 1024 to 8192 k, a chain of K fmaf 5.7e-7 (1024), 8.1e-7 (2048), 1.6e-6 (8192).
// A result that is not finite is made again by the chain of fmaf from the float32 operands, so infinities and NaNs come out as
// that kernel's; a magnitude above the largest bfloat16 arrives there too.  Operands below 2^-110 lose the bits that bfloat16 cannot hold
// there, 2^-126 each at most; a result below 2^-64, where that could show, is made again in the same way.  (What
// remains: magnitudes above 2^38 / K beside those, and results that are all of operands below float32's own normal range, which may come out as 0.)
//
// Measured (M x N x K, this kernel with the split of A / the chain of fmaf, us): 1 x 2048 x 2048 21 / 59, 338 x 3072 x 2048 54 / 135,
// 338 x 16384 x 2048 142 / 585, 338 x 2048 x 8192 75 / 513, 2048 x 2048 x 2048 153 / 402, 1 x 128256 x 2048 291 / 455.
// What bounds it: with few rows a thread's issue of 24 products a piece (58 cycles each) and the splitting of W; with many the operands'
// way from L2 (100 KB a piece for 176 rows, about 40 bytes a cycle and SM; the tensor pipe would take 2112 cycles a piece, a piece
// takes 2400).
//
// A block makes 128 features x up to 176 rows of A (the tensor core's M is W's rows: those are many, whatever the step):
//   warp 0        loads: W as float32 and the parts of A (a small kernel makes them once per call: every block of 128 features
//                 reads the same ones) in pieces of 64 k, both by TMA with the 128-byte swizzle;
//   warps 1, 2    issue the products of every other piece, A operand (W's parts) out of tensor memory, B operand out of shared memory;
//   warps 4..7    split W: a thread reads 64 k of its row and puts the three parts into tensor memory;
//   warps 8..15   add the finished pieces of 64 k to their registers.
// W goes through tensor memory because six products read it: out of shared memory, operands and copies would ask for
// more than the 128 bytes a cycle that it delivers.  K is cut over the blocks of a cluster where N alone would leave SMs
// idle; by N and K only, and the parts are added in a fixed order, so a row's result depends neither on the other rows nor on
// their number.
#pragma once

#include "tc5.cuh"

namespace f32s {

constexpr int kRows = 128, kCols = 176;      // features and rows of A of a block
constexpr int kBlockK = 64;                  // k of a piece
constexpr int kMaxWStages = 6, kHalfBytes = kRows * 128, kWBytes = 2 * kHalfBytes;
constexpr int kRing = 230400;         // bytes of shared memory for both rings
constexpr int kMaxStages = 4;
constexpr int kThreads = 16 * 32;
constexpr unsigned kTmemCols = 512, kSlotCols = 3 * kBlockK / 4, kMaxSlots = 4;   // a slot: the parts of W's 32 k
constexpr int kChunks = (kCols / 16 + 1) / 2;   // of 16 columns, of a half of the adding warps

struct Params {
  const float* a; const float* w; float* c;
  int lda, ldw, ldc, M, N, K;
  int nt;                  // rows of A per block, a multiple of 16
  int m_tiles, splits, k_blocks;
  int stages, w_stages, slots;    // of A's parts, of W, of W's parts in tensor memory
  int* status;
};

struct Bars {
  unsigned long long w_full[kMaxWStages], w_empty[kMaxWStages], b_full[kMaxStages], a_full[kMaxSlots], a_empty[kMaxSlots], acc_empty[2];
  // piece i's products are over (its parts of A are free, its sum is there): ring of four, so that nobody who waits
  // for a piece can be passed by the piece that uses the barrier next
  unsigned long long done[4];
  unsigned tmem;
  int abort_flag;
};

// A place in a ring and the parity of the phase that fills it.
struct Turn {
  int at = 0;
  unsigned parity = 0;
  __device__ __forceinline__ void next(int places) {
    if (++at == places) { at = 0; parity ^= 1u; }
  }
};

__device__ __forceinline__ unsigned pack2(float x, float y) {
  __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<unsigned*>(&h);
}
// (x, y) -> its three bfloat16 pairs
__device__ __forceinline__ void split2(float x, float y, unsigned& h, unsigned& m, unsigned& l) {
  h = pack2(x, y);
  x -= __uint_as_float(h << 16);
  y -= __uint_as_float(h & 0xffff0000u);
  m = pack2(x, y);
  x -= __uint_as_float(m << 16);
  y -= __uint_as_float(m & 0xffff0000u);
  l = pack2(x, y);
}

// A [M, K] -> parts [3][M][Kp] in bfloat16, Kp = K rounded up to 8 (zeros behind K).  A thread makes four of a row.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ a, int lda, int M, int K, int Kp,
                                                         __nv_bfloat16* __restrict__ parts, int wide) {
  pdl_trigger();
  pdl_wait();
  const int quads = Kp >> 2;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)M * quads) return;
  const int row = (int)(i / quads), k = (int)(i - (long long)row * quads) << 2;
  const float* src = a + (size_t)row * lda + k;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (k < K) {                               // K is a multiple of four
    if (wide) v = *reinterpret_cast<const float4*>(src);
    else v = make_float4(src[0], src[1], src[2], src[3]);
  }
  uint2 h, m, l;
  split2(v.x, v.y, h.x, m.x, l.x);
  split2(v.z, v.w, h.y, m.y, l.y);
  const size_t plane = (size_t)M * Kp, at = (size_t)row * Kp + k;
  *reinterpret_cast<uint2*>(parts + at) = h;
  *reinterpret_cast<uint2*>(parts + plane + at) = m;
  *reinterpret_cast<uint2*>(parts + 2 * plane + at) = l;
}

// The element as the chain of fmaf makes it: for results that are not finite, and for those so small that the parts' lost bits could show.
__device__ __noinline__ float chain(const Params& p, int m, int n, float v) {
  if (v == 0.f) return v;
  const float *x = p.a + (size_t)m * p.lda, *w = p.w + (size_t)n * p.ldw;
  float s = 0.f;
  for (int k = 0; k < p.K; ++k) s = fmaf(x[k], w[k], s);
  return s;
}
__device__ __forceinline__ void put(const Params& p, int m, int n, float v) {
  if (m >= p.M || n >= p.N) return;
  constexpr unsigned small = 0x1f800000u, infinite = 0x7f800000u;      // 2^-64
  if ((__float_as_uint(v) & 0x7fffffffu) - small >= infinite - small) v = chain(p, m, n, v);
  p.c[(size_t)m * p.ldc + n] = v;
}

__global__ void __launch_bounds__(kThreads, 1)
split_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const Params p) {
  using namespace tc5;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int plane_bytes = p.nt * 128, stage_bytes = 3 * plane_bytes;
  unsigned char* w_s = base;
  unsigned char* b_s = base + p.w_stages * kWBytes;
  Bars* bars = reinterpret_cast<Bars*>(b_s + (size_t)p.stages * stage_bytes);
  volatile int* abort_flag = &bars->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < p.w_stages; ++i) { mbar_init(&bars->w_full[i], 1); mbar_init(&bars->w_empty[i], 4); }
    for (int i = 0; i < p.stages; ++i) mbar_init(&bars->b_full[i], 1);
    for (int i = 0; i < p.slots; ++i) { mbar_init(&bars->a_full[i], 4); mbar_init(&bars->a_empty[i], 1); }
    for (int i = 0; i < 2; ++i) mbar_init(&bars->acc_empty[i], 8);
    for (int i = 0; i < 4; ++i) mbar_init(&bars->done[i], 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&bars->tmem, kTmemCols);
  fence_before();
  __syncthreads();
  fence_after();
  const unsigned tmem = bars->tmem;
  pdl_trigger();
  pdl_wait();

  const int split = (int)blockIdx.x % p.splits, tile = (int)blockIdx.x / p.splits;
  const int m0 = tile % p.m_tiles * p.nt, n0 = tile / p.m_tiles * kRows;
  const int kb0 = (int)((long long)p.k_blocks * split / p.splits), kb1 = (int)((long long)p.k_blocks * (split + 1) / p.splits);
  const int blocks = kb1 - kb0;
  bool failed = false;
  float acc[kChunks][16];                 // warps 8..15: columns 32 c + 16 half ..
  const int half = warp >= 12;

  // These loops are chains of one thread (or of one warp): as few barriers as the flow needs, and places in the rings and
  // the parities of their barriers are counted, not divided out.
  auto wait_done = [&](int i) { return wait_or_abort(&bars->done[i & 3], (unsigned)(i >> 2) & 1u, abort_flag); };
  if (warp == 0) {
    if (lane == 0) {
      Turn bt, wt;
      int k = kb0 * kBlockK;
      for (int i = 0; i < blocks; ++i, k += kBlockK, bt.next(p.stages), wt.next(p.w_stages)) {
        if (i >= p.w_stages && !wait_or_abort(&bars->w_empty[wt.at], wt.parity ^ 1u, abort_flag)) { failed = true; break; }
        mbar_expect_tx(&bars->w_full[wt.at], kWBytes);
        tma_load_2d(w_s + wt.at * kWBytes, &map_w, k, n0, &bars->w_full[wt.at]);
        tma_load_2d(w_s + wt.at * kWBytes + kHalfBytes, &map_w, k + kBlockK / 2, n0, &bars->w_full[wt.at]);
        if (i >= p.stages && !wait_done(i - p.stages)) { failed = true; break; }
        mbar_expect_tx(&bars->b_full[bt.at], (unsigned)stage_bytes);
        for (int part = 0; part < 3; ++part)
          tma_load_2d(b_s + (size_t)bt.at * stage_bytes + part * plane_bytes, &map_a, k, part * p.M + m0, &bars->b_full[bt.at]);
      }
    }
  } else if (warp < 3) {
    if (lane == 0) {
      // two threads take turns, each with an accumulator of its own: a wait costs 200 cycles even where nothing is waited for, an
      // issue 58, and a piece's 24 products at 128 rows 1536
      const unsigned idesc = idesc_bf16(kRows, (unsigned)p.nt);
      const unsigned long long b0 = smem_desc_sw128(smem_u32(b_s));
      const unsigned plane16 = (unsigned)plane_bytes >> 4, stage16 = (unsigned)stage_bytes >> 4;
      const int which = warp - 1;
      const unsigned d = tmem + which * p.nt;
      Turn bt, at;
      if (which) { bt.next(p.stages); at.next(p.slots); at.next(p.slots); }
      unsigned parity = 0;
      for (int i = which; i < blocks && !failed; i += 2, parity ^= 1u) {
        if (!wait_or_abort(&bars->b_full[bt.at], bt.parity, abort_flag) ||
            (i >= 2 && !wait_or_abort(&bars->acc_empty[which], parity ^ 1u, abort_flag))) { failed = true; break; }
        const unsigned long long bd = b0 + bt.at * stage16;
#pragma unroll
        for (int j = 0; j < 2; ++j, at.next(p.slots)) {
          if (!wait_or_abort(&bars->a_full[at.at], at.parity, abort_flag)) { failed = true; break; }
          fence_after();
          const unsigned w = tmem + 2 * p.nt + at.at * kSlotCols;
          // the small products first, while the sum is small
          constexpr int pw[6] = {1, 2, 0, 1, 0, 0}, pa[6] = {1, 0, 2, 0, 1, 0};
#pragma unroll
          for (int x = 0; x < 6; ++x)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
              umma_ts(d, w + pw[x] * 16 + kk * 8, bd + pa[x] * plane16 + 4 * j + 2 * kk, idesc, (j | x | kk) ? 1u : 0u);
          umma_commit(&bars->a_empty[at.at]);
        }
        if (failed) break;
        umma_commit(&bars->done[i & 3]);
        bt.next(p.stages);
        bt.next(p.stages);
        at.next(p.slots);
        at.next(p.slots);
      }
    }
  } else if (warp >= 4 && warp < 8) {
    const int r = (warp & 3) * 32 + lane;
    const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16) + 2 * p.nt;
    Turn wt, at;
    for (int i = 0; i < blocks && !failed; ++i, wt.next(p.w_stages)) {
      if (!wait_or_abort(&bars->w_full[wt.at], wt.parity, abort_flag)) { failed = true; break; }
#pragma unroll 1
      for (int j = 0; j < 2; ++j, at.next(p.slots)) {
        const unsigned char* row = w_s + wt.at * kWBytes + j * kHalfBytes + r * 128;
        unsigned h[16], m[16], l[16];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(row + ((c ^ (r & 7)) << 4));
          split2(v.x, v.y, h[2 * c], m[2 * c], l[2 * c]);
          split2(v.z, v.w, h[2 * c + 1], m[2 * c + 1], l[2 * c + 1]);
        }
        if (2 * i + j >= p.slots && !wait_or_abort(&bars->a_empty[at.at], at.parity ^ 1u, abort_flag)) { failed = true; break; }
        fence_after();
        const unsigned to = lanes + at.at * kSlotCols;
        tmem_st16(to, h);
        tmem_st16(to + 16, m);
        tmem_st16(to + 32, l);
        wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars->a_full[at.at]);
          if (j) mbar_arrive(&bars->w_empty[wt.at]);
        }
      }
    }
  } else if (warp >= 8) {
    const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16);
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[c][j] = 0.f;
    Turn ct;
    for (int i = 0; i < blocks; ++i, ct.next(2)) {
      if (!wait_done(i)) { failed = true; break; }
      fence_after();
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int col = 32 * c + 16 * half;
        if (col < p.nt) {
          unsigned v[16];
          tmem_ld16(lanes + ct.at * p.nt + col, v);
          wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c][j] += __uint_as_float(v[j]);
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[ct.at]);
    }
  }
  if (failed) *abort_flag = 1;
  __syncwarp();
  const int n_row = (warp & 3) * 32 + lane;
  if (p.splits == 1) {
    if (warp >= 8) {
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = 32 * c + 16 * half + j;
          if (col < p.nt) put(p, m0 + col, n0 + n_row, acc[c][j]);
        }
    }
  } else {
    // this block's sums [nt][128] go where A's parts were (every copy and product has finished), then the cluster's blocks
    // add up a share of the rows each, the lowest k first
    __syncthreads();
    float* mine = reinterpret_cast<float*>(b_s);
    if (warp >= 8) {
#pragma unroll
      for (int c = 0; c < kChunks; ++c)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = 32 * c + 16 * half + j;
          if (col < p.nt) mine[col * kRows + n_row] = acc[c][j];
        }
    }
    cluster_sync_all();
    const unsigned rank = cluster_rank();
    const unsigned mine_u = smem_u32(mine);
    for (int i = tid; i < p.nt / p.splits * kRows; i += kThreads) {       // nt and splits: 16 and a divisor of it
      const int col = (int)rank * (p.nt / p.splits) + i / kRows, n = i % kRows;
      float s = 0.f;
      for (int q = 0; q < p.splits; ++q) {
        unsigned remote;
        float v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine_u + (unsigned)(col * kRows + n) * 4u), "r"(q));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
        s += v;
      }
      put(p, m0 + col, n0 + n, s);
    }
    cluster_sync_all();      // nobody leaves while another block may read its sums
  }
  fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) atomicCAS(p.status, 0, KVB_STATUS_WAIT_TIMEOUT);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies and products that may still run finish
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace f32s

// Blocks of a cluster that share K: as many as keep the SMs busy with one tile of rows and leave each at least 512 k.
static int kvb_split_blocks(int N, int K) {
  const int tiles = (N + f32s::kRows - 1) / f32s::kRows, k_blocks = (K + f32s::kBlockK - 1) / f32s::kBlockK;
  int s = 1;
  while (s < 4 && tiles * s * 2 <= 148 && k_blocks / (s * 2) >= 8) s *= 2;
  return s;
}

// C = A . W^T.  W and its rows on 16-byte boundaries, K a multiple of 4; A any alignment; parts: room for 3 M (K rounded up to 8) bfloat16
// elements on a 16-byte boundary.
KVB_EXPORT int kvb_sgemm_nt_split(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                                  void* parts, int* status, cudaStream_t stream) {
  using namespace f32s;
  if (M <= 0 || N <= 0) return 0;
  if (K < 4 || (K & 3)) return KVB_ERR_BAD_SIZE;
  if ((ldw & 3) || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(parts) & 15)) return KVB_ERR_ALIGN;
  const int Kp = (K + 7) / 8 * 8;
  const long long quads = (long long)M * (Kp / 4);
  if (3ll * M > 0x7fffffffll || quads / 256 + 1 > 0x7fffffffll) return KVB_ERR_BAD_SIZE;
  Params p;
  p.a = A; p.w = W; p.c = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
  p.m_tiles = (M + kCols - 1) / kCols;
  p.nt = ((M + p.m_tiles - 1) / p.m_tiles + 15) / 16 * 16;
  p.splits = kvb_split_blocks(N, K);
  p.k_blocks = (K + kBlockK - 1) / kBlockK;
  p.slots = ((int)kTmemCols - 2 * p.nt) / (int)kSlotCols;
  if (p.slots > kMaxSlots) p.slots = kMaxSlots;
  p.stages = 110592 / (3 * 128 * p.nt);
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  if (p.stages < 2) p.stages = 2;
  p.w_stages = (kRing - p.stages * 3 * 128 * p.nt) / kWBytes;
  if (p.w_stages > kMaxWStages) p.w_stages = kMaxWStages;
  p.status = status;
  const long long grid = (long long)p.m_tiles * ((N + kRows - 1) / kRows) * p.splits;
  if (grid > 0x7fffffffll) return KVB_ERR_BAD_SIZE;
  CUtensorMap map_w, map_a;
  int e = tc5::make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, W, N, K, (long long)ldw * 4, kRows);
  if (e) return e;
  e = tc5::make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, parts, 3ll * M, Kp, (long long)Kp * 2, p.nt);
  if (e) return e;
  const int wide = !(lda & 3) && !(reinterpret_cast<uintptr_t>(A) & 15);
  cudaError_t ce = kvb_launch(split_rows_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, stream, A, lda, M, K, Kp,
                              reinterpret_cast<__nv_bfloat16*>(parts), wide);
  if (ce != cudaSuccess) return (int)ce;
  constexpr int kSmem = 1024 + kRing + (int)sizeof(Bars);
  static_assert(kSmem <= 232448, "shared memory of a block");
  ce = cudaFuncSetAttribute(split_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (ce != cudaSuccess) return (int)ce;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.splits;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = kvb_pdl_enabled() ? 2 : 1;
  ce = cudaLaunchKernelEx(&cfg, split_gemm_kernel, map_w, map_a, p);
  if (ce != cudaSuccess) return (int)ce;
  return kvb_launch_result();
}
