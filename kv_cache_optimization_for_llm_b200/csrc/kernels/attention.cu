// Attention over the paged cache, general form: any mix of query runs (a prompt
// portion, a single decoded token) against the keys of their own requests.
//
// One block per (query token, query head); its four warps take the keys in chunks
// of 32 consecutive positions, chunk c going to warp c % 4.  The chunking follows
// absolute key positions, so the sums a query sees are the same however its
// request was cut into steps, whatever else is in the batch and wherever its
// pages lie.  Scores, softmax and the weighted sum of values are float32.
//
// Upstream computes the same thing in two kernels, one over a packed prompt
// (base/src/kernels.cu:361-466) and one over the cache for a single token
// (paged_attention/src/kernels.cu:150-219): score = (q.k)/sqrt(d), keys j <= pos,
// kv head = q head / (nq/nkv), online softmax.  `window` > 0 keeps only keys
// j > pos - window (upstream has none).
#include "common.cuh"

#include <math_constants.h>

constexpr int kMaxHeadDim = 256;
constexpr int kWarps = 4;

template <typename T>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_generic_kernel(const T* __restrict__ q_base, int q_row_stride,
                               const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                               const int* __restrict__ block_table, int max_pages, int page_size,
                               int num_pages, const int* __restrict__ positions,
                               const int* __restrict__ token_req, T* __restrict__ out, int nq, int nkv,
                               int d, float scale, int window, int* status) {
  __shared__ float q_s[kMaxHeadDim];
  __shared__ float acc_s[kWarps][kMaxHeadDim];
  __shared__ float m_s[kWarps], l_s[kWarps];

  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const int h = blockIdx.y;
  const int hk = h / (nq / nkv);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = positions[t];
  const int* table = block_table + (size_t)token_req[t] * max_pages;
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;

  const T* q = q_base + (size_t)t * q_row_stride + (size_t)h * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) q_s[i] = to_f32(q[i]);
  __syncthreads();

  float m = -CUDART_INF_F, l = 0.f;
  float acc[kMaxHeadDim / 32];
#pragma unroll
  for (int r = 0; r < kMaxHeadDim / 32; ++r) acc[r] = 0.f;

  for (int c = lo / 32 + ((warp - lo / 32) % kWarps + kWarps) % kWarps; c * 32 <= pos; c += kWarps) {
    const int j = c * 32 + lane;
    const bool valid = j >= lo && j <= pos;
    long long off = -1;
    float s = -CUDART_INF_F;
    if (valid) {
      const int lp = j / page_size;
      const int page = lp < max_pages ? table[lp] : -1;
      if (page < 0 || page >= num_pages) {
        atomicCAS(status, 0, KVB_STATUS_UNMAPPED_PAGE);
      } else {
        off = (((long long)page * nkv + hk) * page_size + (j % page_size)) * d;
        const T* k = k_pages + off;
        float dot = 0.f;
        for (int i = 0; i < d; ++i) dot = fmaf(q_s[i], to_f32(k[i]), dot);
        s = dot * scale;
      }
    }
    const float cm = warp_max(s);
    if (cm == -CUDART_INF_F) continue;  // nothing readable in this chunk (only after an error)
    const float m_new = fmaxf(m, cm);
    const float corr = (m == -CUDART_INF_F) ? 0.f : expf(m - m_new);
    const float p = (off >= 0) ? expf(s - m_new) : 0.f;
    l = fmaf(l, corr, warp_sum(p));
#pragma unroll
    for (int r = 0; r < kMaxHeadDim / 32; ++r) acc[r] *= corr;
    const int n_in_chunk = min(32, pos - c * 32 + 1);
    for (int jj = 0; jj < n_in_chunk; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const long long oj = __shfl_sync(0xffffffffu, off, jj);
      if (oj < 0) continue;
      const T* v = v_pages + oj;
#pragma unroll
      for (int r = 0; r < kMaxHeadDim / 32; ++r) {
        const int i = r * 32 + lane;
        if (i < d) acc[r] = fmaf(pj, to_f32(v[i]), acc[r]);
      }
    }
    m = m_new;
  }

  if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
#pragma unroll
  for (int r = 0; r < kMaxHeadDim / 32; ++r) {
    const int i = r * 32 + lane;
    if (i < d) acc_s[warp][i] = acc[r];
  }
  __syncthreads();
  if (warp == 0) {
    float M = m_s[0];
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, m_s[w]);
    float L = 0.f, f[kWarps];
    for (int w = 0; w < kWarps; ++w) {
      f[w] = (m_s[w] == -CUDART_INF_F) ? 0.f : expf(m_s[w] - M);
      L = fmaf(l_s[w], f[w], L);
    }
    T* o = out + ((size_t)t * nq + h) * d;
    for (int i = lane; i < d; i += 32) {
      float a = 0.f;
      for (int w = 0; w < kWarps; ++w) a = fmaf(acc_s[w][i], f[w], a);
      o[i] = from_f32<T>(L > 0.f ? a / L : 0.f);
    }
  }
}

// q points at the first query head of token 0; consecutive tokens are q_row_stride
// elements apart (the fused q|k|v row).  out is [T, nq*d], dense.
// Refuses: d > 256, odd d, nq not a multiple of nkv.
KVB_EXPORT int kvb_paged_attention_generic(const void* q, int q_row_stride, const void* k_pages,
                                           const void* v_pages, const int* block_table, int max_pages,
                                           int page_size, int num_pages, const int* positions,
                                           const int* token_req, void* out, int T_, int nq, int nkv,
                                           int d, float scale, int window, int dtype, int* status,
                                           cudaStream_t stream) {
  if (T_ <= 0) return 0;
  if (d > kMaxHeadDim || d < 2 || (d & 1) || nkv < 1 || nq % nkv) return KVB_ERR_BAD_SIZE;
  dim3 grid(T_, nq);
  KVB_DISPATCH_DTYPE(dtype, T, (kvb_launch(paged_attention_generic_kernel<T>, grid, dim3(kWarps * 32), 0, stream,
                                            (const T*)q, q_row_stride, (const T*)k_pages, (const T*)v_pages,
                                            block_table, max_pages, page_size, num_pages, positions, token_req,
                                            (T*)out, nq, nkv, d, scale, window, status)));
  return kvb_launch_result();
}

// ===========================================================================
// The general attention over tiles of query rows (float32 steps with runs of tokens): the same sums as the kernel above, to
// the bit, so that a token's result does not depend on which of the two its step was given to.
//
// A block takes a tile of consecutive tokens of one request with all query heads of one key/value head, up to 16 RT rows (token,
// head), and brings every chunk of 32 keys and values into shared memory once for the whole tile.  Its four groups of 128 threads
// are the four warps of the kernel above: group g takes the chunks c with c % 4 == g, with a maximum, a sum and a weighted
// sum of values of its own, merged at the end in the same order.  Within a group a thread stands at row 16 r + ty (r < RT) and
// keys tx, tx + 8, tx + 16, tx + 24 of the chunk: every score is one chain of fmaf over the head's channels; the 32
// exponentials are added as warp_sum adds them (partners 16, 8, 4, 2, 1 apart); a value channel is one chain over the keys
// in order.  A key that a row does not see adds nothing to any of the three.
//
// Keys and values of a group's next chunk are on their way (cp.async) while it works on this one, where shared memory has room for two
// (head sizes up to 64).  Two neighbouring rows' scores, and two channels' sums, go through one `fma.rn.f32x2`, which rounds each half as
// fmaf does.  The chunk's first keys that all rows of a warp see, most of them, are added up without a look at positions.  The blocks
// that start first are the ones with the latest positions of their run, which have the most keys.
//
// What bounds it: one block of sixteen warps an SM (its registers), whose loads from shared memory are 224 of 16 bytes a thread and chunk of
// 64 rows (four cycles a warp and load, 7 us of a turn's 9).  The kernel above reads a key's channels one by one, a lane per key (32 rows a warp and load), and every (token, head) reads
// them again: 575 us for 333 + 5 tokens of 32 heads of 64 over 8 key/value heads.
// Here, us: those 338 tokens 114 -> 50, the 333 alone 112 -> 36, 1024 tokens 497 -> 181, 16 tokens behind 3000 545 -> 239, twenty single tokens
// behind 3000 beside a run of two 525 -> 231; 24 heads of 128, 333 tokens 152 -> 54 (before: loads one after the other behind a look at
// the block table each, branches around every key's sums, groups of 64 threads with eight rows each; with eight warps 56, 50, 246, 304, 215).
constexpr int kTileRows = 16;                          // TY: rows of threads in a group, eight threads a row
constexpr int kTileThreads = kWarps * 8 * kTileRows, kGroupThreads = 8 * kTileRows;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void copy_16(float* to, const float* from, bool inside) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
               "r"(inside ? 16 : 0) : "memory");
}

// floats of a group's chunk of keys, in whose place its exponentials are kept
__host__ __device__ constexpr int tile_key_floats(int dmax, int rt) {
  return 32 * (dmax + 4) > kTileRows * rt * 36 ? 32 * (dmax + 4) : kTileRows * rt * 36;
}
// chunks of keys and values that a group has room for
__host__ __device__ constexpr int tile_stages(int dmax) { return dmax <= 64 ? 2 : 1; }
// floats between the rows of a pair of queries: the pair's channels side by side, eight more for the banks
__host__ __device__ constexpr int tile_pair_floats(int dmax) { return 2 * dmax + 8; }

// Scores of RP pairs of rows (of a thread: rows 16 r + ty) with four keys.
template <int RP, int LD, int LDQ>
__device__ __forceinline__ void tile_scores(f32x2 (&s)[RP][4], const float* q_s, const float* k_s, int d, int tx, int ty) {
#pragma unroll
  for (int r = 0; r < RP; ++r)
#pragma unroll
    for (int u = 0; u < 4; ++u) s[r][u] = 0ull;
#pragma unroll 2
  for (int i = 0; i < d; i += 4) {
    float4 kv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) kv[u] = *reinterpret_cast<const float4*>(k_s + (tx + 8 * u) * LD + i);
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(q_s + (kTileRows * r + ty) * LDQ + 2 * i);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(q_s + (kTileRows * r + ty) * LDQ + 2 * i + 4);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s[r][u] = fma2(a.x, pack2(kv[u].x, kv[u].x), s[r][u]);
        s[r][u] = fma2(a.y, pack2(kv[u].y, kv[u].y), s[r][u]);
        s[r][u] = fma2(b.x, pack2(kv[u].z, kv[u].z), s[r][u]);
        s[r][u] = fma2(b.y, pack2(kv[u].w, kv[u].w), s[r][u]);
      }
    }
  }
}

// Keys 0 .. n - 1 of the chunk (n a multiple of four), seen by all of the first R rows of the thread.
template <int R, int RT, int DT, int LD, int LDP>
__device__ __forceinline__ void tile_values(f32x2 (&acc)[RT][2 * DT], const float* p_s, const float* v_s, int n, int tx, int ty) {
#pragma unroll 1
  for (int jj = 0; jj < n; jj += 4) {
    float4 pv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) pv[r] = *reinterpret_cast<const float4*>(p_s + (kTileRows * r + ty) * LDP + jj);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      ulonglong2 vv[DT];
#pragma unroll
      for (int x = 0; x < DT; ++x) vv[x] = *reinterpret_cast<const ulonglong2*>(v_s + (jj + u) * LD + 32 * x + 4 * tx);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float pj = u == 0 ? pv[r].x : u == 1 ? pv[r].y : u == 2 ? pv[r].z : pv[r].w;
        const f32x2 p2 = pack2(pj, pj);
#pragma unroll
        for (int x = 0; x < DT; ++x) {
          acc[r][2 * x] = fma2(p2, vv[x].x, acc[r][2 * x]);
          acc[r][2 * x + 1] = fma2(p2, vv[x].y, acc[r][2 * x + 1]);
        }
      }
    }
  }
}

template <int DMAX, int RT>
__global__ void __launch_bounds__(kTileThreads)
paged_attention_tiles_kernel(const float* __restrict__ q_base, int q_row_stride, const float* __restrict__ k_pages,
                             const float* __restrict__ v_pages, const int* __restrict__ block_table, int max_pages,
                             int page_size, int num_pages, const int* __restrict__ positions, const int4* __restrict__ tiles,
                             float* __restrict__ out, int nq, int nkv, int d, float scale, int window, int* status) {
  constexpr int ROWS = kTileRows * RT, LD = DMAX + 4, LDP = 36, DT = DMAX / 32;      // DT: groups of four channels a thread owns
  constexpr int RP = RT / 2, LDQ = tile_pair_floats(DMAX), STAGES = tile_stages(DMAX);
  constexpr int KREG = tile_key_floats(DMAX, RT), PER_CHUNK = KREG + 32 * LD, PER_GROUP = STAGES * PER_CHUNK;
  extern __shared__ __align__(16) float tsm[];
  float* q_s = tsm;                                    // [RP * 16 pairs of rows][LDQ]: rows 32 r + ty and 32 r + 16 + ty
  const int tid = threadIdx.x, g = tid / kGroupThreads, gt = tid % kGroupThreads, tx = gt & 7, ty = gt >> 3;
  float* mine_s = q_s + RP * kTileRows * LDQ + g * PER_GROUP;  // [STAGES]{[32][LD] keys, [32][LD] values}
  __shared__ float m_s[kWarps][ROWS], l_s[kWarps][ROWS];
  pdl_trigger();
  pdl_wait();
  // the tiles come in the order of their tokens: the last ones first, for all key/value heads
  const int lin = blockIdx.y * gridDim.x + blockIdx.x;
  const int4 tile = tiles[gridDim.x - 1 - lin / nkv];
  const int hk = lin % nkv, group = nq / nkv, rows = tile.z * group, nr = (rows + kTileRows - 1) / kTileRows;     // r < nr: rows that exist
  const int* table = block_table + (size_t)tile.x * max_pages;
  int pos_lo = 0x7fffffff, pos_hi = -1;                // of the tile's tokens
  for (int t = 0; t < tile.z; ++t) {
    const int p = positions[tile.y + t];
    pos_lo = min(pos_lo, p);
    pos_hi = max(pos_hi, p);
  }
  // This group's part of a chunk, on its way to a stage; bit k of the answer: key k lies in a page (the same word in every thread
  // of the warp).  A lane looks one key's page up for the others.
  const int d4 = d >> 2;
  auto request = [&](int c, int stage) -> unsigned {
    const int j = c * 32 + (tid & 31);
    const int lp = j / page_size;
    const int page = j <= pos_hi && lp < max_pages ? table[lp] : -1;
    const bool there = page >= 0 && page < num_pages;
    if (!there && j <= pos_hi && (window <= 0 || j > pos_lo - window)) atomicCAS(status, 0, KVB_STATUS_UNMAPPED_PAGE);
    const long long off = there ? (((long long)page * nkv + hk) * page_size + (j - lp * page_size)) * d : -1;
    float* to = mine_s + stage * PER_CHUNK;
    for (int x = gt; x < 32 * d4; x += kGroupThreads) {      // (whole warps take part: 32 d4 is a multiple of 32)
      const int kk = x / d4, i = (x - kk * d4) * 4;
      const long long of = __shfl_sync(0xffffffffu, off, kk);
      copy_16(to + kk * LD + i, k_pages + (of >= 0 ? of + i : 0), of >= 0);
      copy_16(to + KREG + kk * LD + i, v_pages + (of >= 0 ? of + i : 0), of >= 0);
    }
    return __ballot_sync(0xffffffffu, there);
  };
  const int first = (window > 0 ? max(0, pos_lo - window + 1) : 0) / 32;
  int c = first + ((g - first) % kWarps + kWarps) % kWarps, stage = 0;
  unsigned mapped = c * 32 <= pos_hi ? request(c, 0) : 0u;
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int x = tid; x < ROWS * d4; x += kTileThreads) {
    const int row = x / d4, i = (x - row * d4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows)
      v = *reinterpret_cast<const float4*>(q_base + (size_t)(tile.y + row / group) * q_row_stride + (size_t)(hk * group + row % group) * d + i);
    float* to = q_s + (row / (2 * kTileRows) * kTileRows + row % kTileRows) * LDQ + 2 * i + row / kTileRows % 2;
    to[0] = v.x; to[2] = v.y; to[4] = v.z; to[6] = v.w;
  }
  int pos[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) pos[r] = kTileRows * r + ty < rows ? positions[tile.y + (kTileRows * r + ty) / group] : -1;
  __syncthreads();

  float m[RT], l[RT];
  f32x2 acc[RT][2 * DT];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    m[r] = -CUDART_INF_F;
    l[r] = 0.f;
#pragma unroll
    for (int x = 0; x < 2 * DT; ++x) acc[r][x] = 0ull;
  }
  const bool busy = (ty & ~3) < rows;                    // this warp has rows that exist; a single token's heads leave most without
  for (; c * 32 <= pos_hi; c += kWarps) {
    unsigned next = 0u;
    if (STAGES == 2) {
      if ((c + kWarps) * 32 <= pos_hi) next = request(c + kWarps, stage ^ 1);
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kGroupThreads) : "memory");
    float* k_s = mine_s + stage * PER_CHUNK;             // [32][LD]
    const float* v_s = k_s + KREG;                       // [32][LD]
    float* p_s = k_s;                                    // [ROWS][LDP], once the scores are made
    f32x2 s2[RP][4];
    if (!busy) {
#pragma unroll
      for (int r = 0; r < RP; ++r) s2[r][0] = s2[r][1] = s2[r][2] = s2[r][3] = 0ull;
    } else if (nr <= 2 && RP > 1) {
      f32x2 few[1][4];
      tile_scores<1, LD, LDQ>(few, q_s, k_s, d, tx, ty);
#pragma unroll
      for (int u = 0; u < 4; ++u) s2[0][u] = few[0][u];
#pragma unroll
      for (int r = 1; r < RP; ++r) s2[r][0] = s2[r][1] = s2[r][2] = s2[r][3] = 0ull;
    } else {
      tile_scores<RP, LD, LDQ>(s2, q_s, k_s, d, tx, ty);
    }
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kGroupThreads) : "memory");
    if (busy) {
      int every = mapped == 0xffffffffu ? 32 : 0;        // keys 0 .. every - 1: seen by all of this thread's rows
      unsigned skipped = 0;                              // bit r: row 16 r + ty takes nothing of the chunk
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        if (r >= nr) break;
        float s[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 two = unpack2(s2[r >> 1][u]);
          s[u] = r & 1 ? two.y : two.x;
        }
        unsigned seen = 0;                               // bit u: key tx + 8 u
        float cm;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int kk = tx + 8 * u, j = c * 32 + kk;
          const bool on = j <= pos[r] && (window <= 0 || j > pos[r] - window) && (mapped >> kk & 1);
          s[u] = on ? s[u] * scale : -CUDART_INF_F;
          seen |= (on ? 1u : 0u) << u;
          cm = u == 0 ? s[0] : fmaxf(cm, s[u]);          // (a NaN only if all 32 scores are, as warp_max has it)
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
        const float m_new = fmaxf(m[r], cm);
        const float corr = m[r] == -CUDART_INF_F ? 0.f : expf(m[r] - m_new);
        const bool skip = cm == -CUDART_INF_F;           // nothing seen, or no score above the lowest: the row stays as it is
        if (kTileRows * r + ty < rows) every = skip || (window > 0 && c * 32 <= pos[r] - window) ? 0 : min(every, pos[r] - c * 32 + 1);
        skipped |= (skip ? 1u : 0u) << r;
        float p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          p[u] = seen >> u & 1 && !skip ? expf(s[u] - m_new) : 0.f;
          p_s[(kTileRows * r + ty) * LDP + tx + 8 * u] = p[u];
        }
        float sum = (p[0] + p[2]) + (p[1] + p[3]);       // keys 16 apart, then 8 apart
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (!skip) {
          l[r] = fmaf(l[r], corr, sum);
#pragma unroll
          for (int x = 0; x < 2 * DT; ++x) {
            const float2 two = unpack2(acc[r][x]);
            acc[r][x] = pack2(two.x * corr, two.y * corr);
          }
          m[r] = m_new;
        }
      }
      // (rows that do not exist hold a probability of zero, or what lay there, and are never stored)
      every = __reduce_min_sync(0xffffffffu, every) & ~3;
      __syncwarp();
      if (nr <= 1) tile_values<1, RT, DT, LD, LDP>(acc, p_s, v_s, every, tx, ty);
      else tile_values<RT, RT, DT, LD, LDP>(acc, p_s, v_s, every, tx, ty);
      const int last = min(32, pos_hi - c * 32 + 1);
      for (int jj = every; jj < last; ++jj) {
        ulonglong2 vv[DT];
#pragma unroll
        for (int x = 0; x < DT; ++x) vv[x] = *reinterpret_cast<const ulonglong2*>(v_s + jj * LD + 32 * x + 4 * tx);
        const int j = c * 32 + jj;
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          if (r >= nr) break;
          // a value that the row does not see is left out, whatever it holds
          if (!(skipped >> r & 1) && j <= pos[r] && (window <= 0 || j > pos[r] - window) && (mapped >> jj & 1)) {
            const float pj = p_s[(kTileRows * r + ty) * LDP + jj];
            const f32x2 p2 = pack2(pj, pj);
#pragma unroll
            for (int x = 0; x < DT; ++x) {
              acc[r][2 * x] = fma2(p2, vv[x].x, acc[r][2 * x]);
              acc[r][2 * x + 1] = fma2(p2, vv[x].y, acc[r][2 * x + 1]);
            }
          }
        }
      }
    }
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kGroupThreads) : "memory");
    if (STAGES == 2) {
      stage ^= 1;
      mapped = next;
    } else {
      if ((c + kWarps) * 32 <= pos_hi) mapped = request(c + kWarps, 0);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  }

  // merge: every group leaves its weighted sums where its chunks of keys and values lay
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  float* acc_s = mine_s;                               // [ROWS][LD]
  static_assert(ROWS * LD <= PER_GROUP, "the weighted sums take the room of both chunks");
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int row = kTileRows * r + ty;
#pragma unroll
    for (int x = 0; x < DT; ++x) {
      const float2 a = unpack2(acc[r][2 * x]), b = unpack2(acc[r][2 * x + 1]);
      *reinterpret_cast<float4*>(acc_s + row * LD + 32 * x + 4 * tx) = make_float4(a.x, a.y, b.x, b.y);
    }
    if (tx == 0) { m_s[g][row] = m[r]; l_s[g][row] = l[r]; }
  }
  __syncthreads();
  const float* acc0 = q_s + RP * kTileRows * LDQ;
  for (int x = tid; x < rows * d; x += kTileThreads) {
    const int row = x / d, i = x - row * d;
    float M = m_s[0][row];
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, m_s[w][row]);
    float L = 0.f, a = 0.f;
    for (int w = 0; w < kWarps; ++w) {
      const float f = m_s[w][row] == -CUDART_INF_F ? 0.f : expf(m_s[w][row] - M);
      L = fmaf(l_s[w][row], f, L);
      a = fmaf(acc0[(size_t)w * PER_GROUP + row * LD + i], f, a);
    }
    out[((size_t)(tile.y + row / group) * nq + hk * group + row % group) * d + i] = L > 0.f ? a / L : 0.f;
  }
}

// Tokens in one tile of the kernel above (0: it does not take these sizes): 64 rows at head sizes up to 64, 32 up to 128.
KVB_EXPORT int kvb_paged_attention_tile_tokens(int d, int group) {
  if (d < 4 || d > 128 || d % 4 || group < 1) return 0;
  return (d <= 64 ? 64 : 32) / group;
}

// tiles [n_tiles, 4]: request row, first token row, tokens (at most kvb_paged_attention_tile_tokens), 0.  float32 only; q, the
// pages and their rows start on 16-byte boundaries.
KVB_EXPORT int kvb_paged_attention_tiles(const float* q, int q_row_stride, const float* k_pages, const float* v_pages,
                                         const int* block_table, int max_pages, int page_size, int num_pages,
                                         const int* positions, const int* tiles, int n_tiles, float* out, int nq, int nkv,
                                         int d, float scale, int window, int* status, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (nkv < 1 || nkv > 65535 || nq % nkv || kvb_paged_attention_tile_tokens(d, nq / nkv) < 1) return KVB_ERR_BAD_SIZE;
  if (q_row_stride % 4 || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) |
                            reinterpret_cast<uintptr_t>(v_pages) | reinterpret_cast<uintptr_t>(tiles)) & 15)) return KVB_ERR_ALIGN;
#define KVB_TILES(DMAX, RT)                                                                                            \
  {                                                                                                                    \
    constexpr int smem = (kTileRows * RT / 2 * tile_pair_floats(DMAX) +                                                            \
                          kWarps * tile_stages(DMAX) * (tile_key_floats(DMAX, RT) + 32 * (DMAX + 4))) * (int)sizeof(float); \
    cudaError_t e = cudaFuncSetAttribute(paged_attention_tiles_kernel<DMAX, RT>,                                       \
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);                           \
    if (e != cudaSuccess) return (int)e;                                                                               \
    kvb_launch(paged_attention_tiles_kernel<DMAX, RT>, dim3(n_tiles, nkv), dim3(kTileThreads), smem, stream, q,        \
               q_row_stride, k_pages, v_pages, block_table, max_pages, page_size, num_pages, positions,                \
               reinterpret_cast<const int4*>(tiles), out, nq, nkv, d, scale, window, status);                          \
  }
  if (d <= 64) KVB_TILES(64, 4) else KVB_TILES(128, 2)
#undef KVB_TILES
  return kvb_launch_result();
}

// ===========================================================================
// Decode attention: every request brings one query token.  Split over the keys.
//
// Block (kv head, request, key block b) takes the keys [b*KB, (b+1)*KB) of its
// request and all `group` query heads that share the kv head, so each key and
// value is read from memory once for the group (upstream reads them once per query
// head: paged_attention/src/kernels.cu:150-219).  A thread owns one key for the
// scores (its K row against the group's queries, which sit pre-scaled in shared
// memory), the block agrees on max and sum per head, then each warp folds its 32
// values into the output dims its lanes own.  The block writes an unnormalised
// partial (o, m, l) to scratch; `decode_attention_combine_kernel` merges the key
// blocks of a (request, head) in ascending order.  Key blocks are cut at absolute
// positions with a size fixed by the engine, so a token's sums do not depend on
// the batch it runs in.
// ===========================================================================

template <typename T> struct Vec8;
template <> struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* f) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float* f) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
};

constexpr int kDecThreads = 128;  // 4 warps, 128 keys per pass

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gmem_src) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Grid (kv head, request, slot): slot z takes the key blocks z, z + gridDim.z, ... of its
// request, so no block of an absent key range is ever launched and the grid does not
// depend on the contexts' lengths.  The partial result of key block b lands in
// part_*[..., b], whoever computed it.
template <typename T, int D, int GMAX>
__global__ void __launch_bounds__(kDecThreads, 5)
decode_attention_split_kernel(const T* __restrict__ q_base, int q_row_stride, const T* __restrict__ k_pages,
                              const T* __restrict__ v_pages, const int* __restrict__ block_table,
                              int max_pages, int page_size, int num_pages, const int* __restrict__ q_start,
                              const int* __restrict__ ctx_len, float* __restrict__ part_o,
                              float* __restrict__ part_ml, int nq, int nkv, int G, float scale, int window,
                              int KB, int NB, int* status) {
  constexpr int DPL = D / 32;                    // output dims per lane
  constexpr int CPK = D * (int)sizeof(T) / 16;   // 16-byte chunks per value row
  __shared__ __align__(16) float q_s[GMAX][D];
  __shared__ float red_s[4][GMAX];
  extern __shared__ __align__(16) unsigned char dec_smem[];
  T (*v_s)[32][D] = reinterpret_cast<T (*)[32][D]>(dec_smem);  // each warp stages the values of its 32 keys

  pdl_trigger();
  pdl_wait();
  const int hk = blockIdx.x, r = blockIdx.y;
  const int pos = ctx_len[r] - 1;
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((int)blockIdx.z * KB > pos) return;
  const int* table = block_table + (size_t)r * max_pages;

  const T* q = q_base + (size_t)q_start[r] * q_row_stride + (size_t)hk * G * D;
  for (int i = tid; i < G * D; i += kDecThreads) q_s[i / D][i % D] = to_f32(q[i]) * scale;
  __syncthreads();

  for (int b = blockIdx.z; b * KB <= pos && b < NB; b += gridDim.z) {
    const int k0 = b * KB;
    if (k0 + KB <= lo) continue;  // the window has passed this block; combine skips it too
    float m_run[GMAX], l_run[GMAX], acc[GMAX][DPL];
#pragma unroll
    for (int g = 0; g < GMAX; ++g) {
      m_run[g] = -CUDART_INF_F; l_run[g] = 0.f;
#pragma unroll
      for (int e = 0; e < DPL; ++e) acc[g][e] = 0.f;
    }
    const int k_end = min(k0 + KB, pos + 1);
    for (int base = k0; base < k_end; base += kDecThreads) {
      const int j = base + tid;
      const bool valid = j < k_end && j >= lo;
      long long off = -1;
      if (valid) {
        const int lp = j / page_size;
        const int page = lp < max_pages ? table[lp] : -1;
        if (page < 0 || page >= num_pages) atomicCAS(status, 0, KVB_STATUS_UNMAPPED_PAGE);
        else off = (((long long)page * nkv + hk) * page_size + (j % page_size)) * D;
      }
      // the values of this warp's keys start their way to shared memory now and
      // arrive while the scores are computed
#pragma unroll
      for (int i = 0; i < CPK; ++i) {
        const int c = i * 32 + lane;
        const int key = c / CPK, part = c % CPK;
        const long long oj = __shfl_sync(0xffffffffu, off, key);
        if (oj >= 0)
          cp_async_16(reinterpret_cast<char*>(&v_s[warp][key][0]) + part * 16,
                      reinterpret_cast<const char*>(v_pages + oj) + part * 16);
      }
      float s[GMAX];
#pragma unroll
      for (int g = 0; g < GMAX; ++g) s[g] = -CUDART_INF_F;
      if (off >= 0) {
        const T* k = k_pages + off;
#pragma unroll
        for (int g = 0; g < GMAX; ++g) s[g] = 0.f;
#pragma unroll
        for (int c = 0; c < D / 8; ++c) {
          float kf[8];
          Vec8<T>::load(k + c * 8, kf);
#pragma unroll
          for (int g = 0; g < GMAX; ++g) {
            if (g < G) {
              const float4 qa = *reinterpret_cast<const float4*>(&q_s[g][c * 8]);
              const float4 qb = *reinterpret_cast<const float4*>(&q_s[g][c * 8 + 4]);
              float t = s[g];
              t = fmaf(qa.x, kf[0], t); t = fmaf(qa.y, kf[1], t); t = fmaf(qa.z, kf[2], t); t = fmaf(qa.w, kf[3], t);
              t = fmaf(qb.x, kf[4], t); t = fmaf(qb.y, kf[5], t); t = fmaf(qb.z, kf[6], t); t = fmaf(qb.w, kf[7], t);
              s[g] = t;
            }
          }
        }
      }
      // block-wide max per head
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float wm = warp_max(g < G ? s[g] : -CUDART_INF_F);
        if (lane == 0) red_s[warp][g] = wm;
      }
      __syncthreads();
      float p[GMAX], corr[GMAX];
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float bm = fmaxf(fmaxf(red_s[0][g], red_s[1][g]), fmaxf(red_s[2][g], red_s[3][g]));
        const float m_new = fmaxf(m_run[g], bm);
        corr[g] = (m_run[g] == -CUDART_INF_F) ? 0.f : __expf(m_run[g] - m_new);
        p[g] = (off >= 0 && g < G) ? __expf(s[g] - m_new) : 0.f;
        m_run[g] = m_new;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float ws = warp_sum(p[g]);
        if (lane == 0) red_s[warp][g] = ws;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        l_run[g] = l_run[g] * corr[g] + ((red_s[0][g] + red_s[1][g]) + (red_s[2][g] + red_s[3][g]));
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[g][e] *= corr[g];
      }
      // fold the staged values of this warp's 32 keys into the dims its lanes own
      cp_async_wait_all();
      __syncwarp();
      const int n_here = min(32, k_end - (base + warp * 32));
      for (int jj = 0; jj < n_here; ++jj) {
        const long long oj = __shfl_sync(0xffffffffu, off, jj);
        float pj[GMAX];
#pragma unroll
        for (int g = 0; g < GMAX; ++g) pj[g] = __shfl_sync(0xffffffffu, p[g], jj);
        if (oj < 0) continue;
        float vf[DPL];
        const T* v = &v_s[warp][jj][lane * DPL];
        if constexpr (sizeof(T) == 2 && DPL == 2) {
          const unsigned w = *reinterpret_cast<const unsigned*>(v);
          vf[0] = __uint_as_float(w << 16); vf[1] = __uint_as_float(w & 0xffff0000u);
        } else if constexpr (sizeof(T) == 2 && DPL == 4) {
          const uint2 w = *reinterpret_cast<const uint2*>(v);
          vf[0] = __uint_as_float(w.x << 16); vf[1] = __uint_as_float(w.x & 0xffff0000u);
          vf[2] = __uint_as_float(w.y << 16); vf[3] = __uint_as_float(w.y & 0xffff0000u);
        } else {
#pragma unroll
          for (int e = 0; e < DPL; ++e) vf[e] = to_f32(v[e]);
        }
#pragma unroll
        for (int g = 0; g < GMAX; ++g)
          if (g < G)
#pragma unroll
            for (int e = 0; e < DPL; ++e) acc[g][e] = fmaf(pj[g], vf[e], acc[g][e]);
      }
      __syncthreads();  // red_s and v_s are rewritten by the next pass
    }
    // sum the four warps' partial outputs in a fixed order, through shared memory
    float* red = reinterpret_cast<float*>(dec_smem);  // the value stage is free again and large enough
    static_assert(sizeof(T) * 32 >= sizeof(float) * GMAX, "the value stage must hold the warps' partial outputs");
#pragma unroll
    for (int g = 0; g < GMAX; ++g)
      if (g < G)
#pragma unroll
        for (int e = 0; e < DPL; ++e) red[(warp * GMAX + g) * D + lane * DPL + e] = acc[g][e];
    __syncthreads();
    for (int i = tid; i < G * D; i += kDecThreads) {
      const int g = i / D, dd = i % D;
      const float o = (red[(0 * GMAX + g) * D + dd] + red[(1 * GMAX + g) * D + dd]) +
                      (red[(2 * GMAX + g) * D + dd] + red[(3 * GMAX + g) * D + dd]);
      part_o[(((size_t)r * nq + hk * G + g) * NB + b) * D + dd] = o;
    }
    if (tid < G) {
      float mm = 0.f, ll = 0.f;  // m_run and l_run are equal in every thread
#pragma unroll
      for (int g = 0; g < GMAX; ++g) if (g == tid) { mm = m_run[g]; ll = l_run[g]; }
      float* ml = part_ml + (((size_t)r * nq + hk * G + tid) * NB + b) * 2;
      ml[0] = mm; ml[1] = ll;
    }
    __syncthreads();  // red (v_s) is staged into again by the next key block
  }
}

// ---------------------------------------------------------------------------
// The whole attention of a decode step in one launch: rotary encoding of the query
// and the new key, the write of the new key and value into their page, the split
// attention over the key blocks, and the merge of the key blocks' partials.
//
// Block (kv head, request, slot) as above.  Every block rotates its own copy of the
// group's queries (kept in float32).  The block that owns the key block holding the
// token's own position rotates the new key, stores key and value into the cache, and
// then reads them back like any other key.  After its last key block a block adds one
// to the counter of its (request, kv head); the block that brings the counter to the
// number of participating blocks merges all partials in ascending key-block order and
// writes the output, then clears the counter.  Nobody waits for anybody.
// qkv rows stay as the projection wrote them (unrotated).
// ---------------------------------------------------------------------------
template <typename T, int D, int GMAX>
__global__ void __launch_bounds__(kDecThreads, 4)
decode_attention_fused_kernel(const T* __restrict__ qkv, int q_row_stride, T* __restrict__ k_pages,
                              T* __restrict__ v_pages, int write_kv, const int* __restrict__ block_table,
                              int max_pages, int page_size, int num_pages, const int* __restrict__ q_start,
                              const int* __restrict__ ctx_len, const float* __restrict__ cos_t,
                              const float* __restrict__ sin_t, int table_len, int rot, T* __restrict__ out,
                              float* __restrict__ part_o, float* __restrict__ part_ml, int* __restrict__ counters,
                              int nq, int nkv, int G, float scale, int window, int KB, int NB, int* status,
                              unsigned long long* trace) {
  constexpr int DPL = D / 32;
  constexpr int CPK = D * (int)sizeof(T) / 16;   // 16-byte chunks per key or value row
  constexpr int EPC = 16 / (int)sizeof(T);       // elements per chunk
  __shared__ __align__(16) float q_s[GMAX][D];
  __shared__ float red_s[4][GMAX];
  __shared__ int last_s;
  extern __shared__ __align__(16) unsigned char dec_smem[];
  T (*k_s)[32][D] = reinterpret_cast<T (*)[32][D]>(dec_smem);                                  // [4][32][D]
  T (*v_s)[32][D] = reinterpret_cast<T (*)[32][D]>(dec_smem + (size_t)4 * 32 * D * sizeof(T)); // [4][32][D]
  // optional profiling: nanosecond stamps of this block's phases, [blocks, 8]
  auto stamp = [&](int slot) {
    if (trace && threadIdx.x == 0) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      trace[(((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * 8 + slot] = t;
    }
  };
  stamp(0);
  pdl_trigger();
  // Lengths, block tables and the keys and values of earlier tokens were all written
  // before the kernel in front of this one started, so they may be read at once.
  const int hk = blockIdx.x, r = blockIdx.y;
  const int pos = ctx_len[r] - 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (pos < 0 || pos / KB >= NB || (cos_t != nullptr && pos >= table_len)) {
    pdl_wait();
    if (tid == 0 && blockIdx.z == 0) atomicCAS(status, 0, KVB_STATUS_BAD_POSITION);
    return;
  }
  if ((int)blockIdx.z * KB > pos) return;   // no key block for this slot; it is not counted either
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int* table = block_table + (size_t)r * max_pages;
  const int half = rot >> 1;
  const bool rotary = cos_t != nullptr && rot > 0;

  // Requests the keys and values of the 128 positions from `base` on into shared memory;
  // the token's own position is left out when this step writes it (it is filled in below).
  // Returns this thread's own key's offset, -1 if it has none to read.
  auto request_tile = [&](int base, int k_end, bool skip_pos) -> long long {
    const int j = base + tid;
    long long off = -1;
    if (j < k_end && j >= lo && !(skip_pos && j == pos)) {
      const int lp = j / page_size;
      const int page = lp < max_pages ? table[lp] : -1;
      if (page < 0 || page >= num_pages) atomicCAS(status, 0, KVB_STATUS_UNMAPPED_PAGE);
      else off = (((long long)page * nkv + hk) * page_size + (j % page_size)) * D;
    }
#pragma unroll
    for (int i = 0; i < CPK; ++i) {
      const int c = i * 32 + lane;
      const int key = c / CPK, part = c % CPK;
      const long long oj = __shfl_sync(0xffffffffu, off, key);
      if (oj >= 0) {
        cp_async_16(reinterpret_cast<char*>(&k_s[warp][key][0]) + part * 16,
                    reinterpret_cast<const char*>(k_pages + oj) + part * 16);
        cp_async_16(reinterpret_cast<char*>(&v_s[warp][key][0]) + part * 16,
                    reinterpret_cast<const char*>(v_pages + oj) + part * 16);
      }
    }
    return off;
  };

  const int b_first = blockIdx.z;
  const int k_end_first = min(b_first * KB + KB, pos + 1);
  long long off = -1;
  const bool first_has_keys = b_first * KB + KB > lo;
  // A layer that reads another layer's cache finds the key and value of the token's own position
  // there: the owning layer wrote them earlier in this same step, several launches back.  Only the
  // wait below orders this kernel behind all of those, so a first tile that holds that position
  // is asked for after it.
  const bool own_key_from_this_step = !write_kv && pos >= b_first * KB && pos < b_first * KB + kDecThreads;
  if (first_has_keys && !own_key_from_this_step) off = request_tile(b_first * KB, k_end_first, write_kv != 0);

  pdl_wait();
  stamp(1);   // the kernel before this one has finished: its q, k, v rows may be read
  if (first_has_keys && own_key_from_this_step) off = request_tile(b_first * KB, k_end_first, false);
  const T* row = qkv + (size_t)q_start[r] * q_row_stride;
  // the group's queries, rotated (pairs (j, j + rot/2) of the first rot dims), scaled
  for (int i = tid; i < G * D; i += kDecThreads) {
    const int g = i / D, dd = i % D;
    const T* qh = row + (size_t)(hk * G + g) * D;
    float val;
    if (rotary && dd < rot) {
      const int j = dd < half ? dd : dd - half;
      const float c = cos_t[(size_t)pos * half + j], sn = sin_t[(size_t)pos * half + j];
      const float x1 = to_f32(qh[j]), x2 = to_f32(qh[j + half]);
      val = dd < half ? x1 * c - x2 * sn : x1 * sn + x2 * c;
    } else {
      val = to_f32(qh[dd]);
    }
    q_s[g][dd] = val * scale;
  }
  // The new key and value: the block that owns the key block of `pos` rotates the key,
  // stores both in the cache, and puts them into its shared-memory tile itself.
  const int b_star = pos / KB;
  const bool owner = write_kv && (b_star % (int)gridDim.z) == (int)blockIdx.z;
  // `pos` lies in the tile that was requested above: its key and value are put there directly
  const bool place_direct = owner && b_star == b_first && (pos - b_star * KB) < kDecThreads;
  bool own_ok = false;
  if (owner) {
    const int lp = pos / page_size;
    const int page = lp < max_pages ? table[lp] : -1;
    if (page < 0 || page >= num_pages) {
      if (tid == 0) atomicCAS(status, 0, KVB_STATUS_UNMAPPED_PAGE);
    } else {
      own_ok = true;
      const size_t dst = (((size_t)page * nkv + hk) * page_size + (pos % page_size)) * D;
      const T* kh = row + (size_t)(nq + hk) * D;
      const T* vh = row + (size_t)(nq + nkv + hk) * D;
      const int slot = (pos - b_star * KB) % kDecThreads;  // place of `pos` inside its 128-key pass
      for (int dd = tid; dd < D; dd += kDecThreads) {
        float val;
        if (rotary && dd < rot) {
          const int j = dd < half ? dd : dd - half;
          const float c = cos_t[(size_t)pos * half + j], sn = sin_t[(size_t)pos * half + j];
          const float x1 = to_f32(kh[j]), x2 = to_f32(kh[j + half]);
          val = dd < half ? x1 * c - x2 * sn : x1 * sn + x2 * c;
        } else {
          val = to_f32(kh[dd]);
        }
        const T kr = from_f32<T>(val);
        k_pages[dst + dd] = kr;
        v_pages[dst + dd] = vh[dd];
        if (place_direct) { k_s[slot >> 5][slot & 31][dd] = kr; v_s[slot >> 5][slot & 31][dd] = vh[dd]; }
      }
      if (!place_direct) __threadfence();  // it will be fetched from L2 by a later pass of this block
    }
  }
  __syncthreads();
  stamp(2);   // queries rotated, new key/value stored

  for (int b = b_first; b * KB <= pos && b < NB; b += gridDim.z) {
    const int k0 = b * KB;
    if (k0 + KB <= lo) continue;
    float m_run[GMAX], l_run[GMAX], acc[GMAX][DPL];
#pragma unroll
    for (int g = 0; g < GMAX; ++g) {
      m_run[g] = -CUDART_INF_F; l_run[g] = 0.f;
#pragma unroll
      for (int e = 0; e < DPL; ++e) acc[g][e] = 0.f;
    }
    const int k_end = min(k0 + KB, pos + 1);
    for (int base = k0; base < k_end; base += kDecThreads) {
      const bool prefetched = (b == b_first && base == k0);
      // Later tiles are requested here; by now the new key, if it falls into one of them,
      // is in the cache and is read like any other.
      if (!prefetched) off = request_tile(base, k_end, false);
      const int j_mine = base + tid;
      bool have = off >= 0;
      if (prefetched && place_direct && own_ok && j_mine == pos) have = true;   // the key this block placed itself
      cp_async_wait_all();
      __syncwarp();
      float s[GMAX];
#pragma unroll
      for (int g = 0; g < GMAX; ++g) s[g] = have ? 0.f : -CUDART_INF_F;
      if (have) {
        const T* k = &k_s[warp][lane][0];
#pragma unroll
        for (int c = 0; c < CPK; ++c) {
          const int cc = (c + lane) % CPK;                // each lane starts at another chunk: no bank conflicts
          float kf[8];
          if constexpr (sizeof(T) == 2) {
            Vec8<T>::load(k + cc * 8, kf);
#pragma unroll
            for (int g = 0; g < GMAX; ++g) {
              if (g < G) {
                const float4 qa = *reinterpret_cast<const float4*>(&q_s[g][cc * 8]);
                const float4 qb = *reinterpret_cast<const float4*>(&q_s[g][cc * 8 + 4]);
                float t = s[g];
                t = fmaf(qa.x, kf[0], t); t = fmaf(qa.y, kf[1], t); t = fmaf(qa.z, kf[2], t); t = fmaf(qa.w, kf[3], t);
                t = fmaf(qb.x, kf[4], t); t = fmaf(qb.y, kf[5], t); t = fmaf(qb.z, kf[6], t); t = fmaf(qb.w, kf[7], t);
                s[g] = t;
              }
            }
          } else {
            const float4 ka = *reinterpret_cast<const float4*>(k + cc * EPC);
#pragma unroll
            for (int g = 0; g < GMAX; ++g) {
              if (g < G) {
                const float4 qa = *reinterpret_cast<const float4*>(&q_s[g][cc * EPC]);
                float t = s[g];
                t = fmaf(qa.x, to_f32(ka.x), t); t = fmaf(qa.y, to_f32(ka.y), t);
                t = fmaf(qa.z, to_f32(ka.z), t); t = fmaf(qa.w, to_f32(ka.w), t);
                s[g] = t;
              }
            }
          }
        }
      }
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float wm = warp_max(g < G ? s[g] : -CUDART_INF_F);
        if (lane == 0) red_s[warp][g] = wm;
      }
      __syncthreads();
      float p[GMAX], corr[GMAX];
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float bm = fmaxf(fmaxf(red_s[0][g], red_s[1][g]), fmaxf(red_s[2][g], red_s[3][g]));
        const float m_new = fmaxf(m_run[g], bm);
        corr[g] = (m_run[g] == -CUDART_INF_F) ? 0.f : __expf(m_run[g] - m_new);
        p[g] = (have && g < G) ? __expf(s[g] - m_new) : 0.f;
        m_run[g] = m_new;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        const float ws = warp_sum(p[g]);
        if (lane == 0) red_s[warp][g] = ws;
      }
      __syncthreads();
#pragma unroll
      for (int g = 0; g < GMAX; ++g) {
        l_run[g] = l_run[g] * corr[g] + ((red_s[0][g] + red_s[1][g]) + (red_s[2][g] + red_s[3][g]));
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[g][e] *= corr[g];
      }
      const int n_here = min(32, k_end - (base + warp * 32));
      const unsigned have_mask = __ballot_sync(0xffffffffu, have);
      for (int jj = 0; jj < n_here; ++jj) {
        float pj[GMAX];
#pragma unroll
        for (int g = 0; g < GMAX; ++g) pj[g] = __shfl_sync(0xffffffffu, p[g], jj);
        if (!((have_mask >> jj) & 1u)) continue;
        float vf[DPL];
        const T* v = &v_s[warp][jj][lane * DPL];
        if constexpr (sizeof(T) == 2 && DPL == 2) {
          const unsigned w = *reinterpret_cast<const unsigned*>(v);
          vf[0] = __uint_as_float(w << 16); vf[1] = __uint_as_float(w & 0xffff0000u);
        } else if constexpr (sizeof(T) == 2 && DPL == 4) {
          const uint2 w = *reinterpret_cast<const uint2*>(v);
          vf[0] = __uint_as_float(w.x << 16); vf[1] = __uint_as_float(w.x & 0xffff0000u);
          vf[2] = __uint_as_float(w.y << 16); vf[3] = __uint_as_float(w.y & 0xffff0000u);
        } else {
#pragma unroll
          for (int e = 0; e < DPL; ++e) vf[e] = to_f32(v[e]);
        }
#pragma unroll
        for (int g = 0; g < GMAX; ++g)
          if (g < G)
#pragma unroll
            for (int e = 0; e < DPL; ++e) acc[g][e] = fmaf(pj[g], vf[e], acc[g][e]);
      }
      __syncthreads();   // red_s and the tiles are rewritten by the next pass
    }
    float* red = reinterpret_cast<float*>(dec_smem);
    static_assert(sizeof(T) * 32 >= sizeof(float) * GMAX, "the tiles must hold the warps' partial outputs");
#pragma unroll
    for (int g = 0; g < GMAX; ++g)
      if (g < G)
#pragma unroll
        for (int e = 0; e < DPL; ++e) red[(warp * GMAX + g) * D + lane * DPL + e] = acc[g][e];
    __syncthreads();
    for (int i = tid; i < G * D; i += kDecThreads) {
      const int g = i / D, dd = i % D;
      const float o = (red[(0 * GMAX + g) * D + dd] + red[(1 * GMAX + g) * D + dd]) +
                      (red[(2 * GMAX + g) * D + dd] + red[(3 * GMAX + g) * D + dd]);
      part_o[(((size_t)r * nq + hk * G + g) * NB + b) * D + dd] = o;
    }
    if (tid < G) {
      float mm = 0.f, ll = 0.f;
#pragma unroll
      for (int g = 0; g < GMAX; ++g) if (g == tid) { mm = m_run[g]; ll = l_run[g]; }
      float* ml = part_ml + (((size_t)r * nq + hk * G + tid) * NB + b) * 2;
      ml[0] = mm; ml[1] = ll;
    }
    __syncthreads();
  }
  stamp(3);   // key blocks done

  // ---- who is last merges
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int expected = min((int)gridDim.z, pos / KB + 1);
    const int old = atomicAdd(&counters[r * nkv + hk], 1);
    last_s = (old == expected - 1);
    if (last_s) counters[r * nkv + hk] = 0;   // ready for the next launch
  }
  __syncthreads();
  stamp(4);   // counted
  if (!last_s) return;
  __threadfence();
  // (max, sum) of every head and key block first, all requested at once; then the outputs
  const int b0 = lo / KB, b1 = pos / KB, nbk = b1 - b0 + 1;
  float* ml_s = reinterpret_cast<float*>(dec_smem);            // [G][nbk][2], nbk <= 64
  for (int i = tid; i < G * nbk * 2; i += kDecThreads) {
    const int g = i / (nbk * 2), rest = i % (nbk * 2);
    ml_s[i] = __ldcg(part_ml + ((size_t)r * nq + hk * G + g) * NB * 2 + (size_t)b0 * 2 + rest);
  }
  __syncthreads();
  for (int i = tid; i < G * D; i += kDecThreads) {
    const int g = i / D, dd = i % D;
    const float* mlg = ml_s + (size_t)g * nbk * 2;
    const float* po = part_o + (((size_t)r * nq + hk * G + g) * NB + b0) * D + dd;
    float M = -CUDART_INF_F;
    for (int b = 0; b < nbk; ++b) M = fmaxf(M, mlg[2 * b]);
    float L = 0.f, a = 0.f;
    for (int bb = 0; bb < nbk; bb += 8) {
      float x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = (bb + u < nbk) ? __ldcg(po + (size_t)(bb + u) * D) : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (bb + u < nbk) {
          const float f = __expf(mlg[2 * (bb + u)] - M);
          L += mlg[2 * (bb + u) + 1] * f;
          a += x[u] * f;
        }
      }
    }
    out[((size_t)q_start[r] * nq + hk * G + g) * D + dd] = from_f32<T>(L > 0.f ? a / L : 0.f);
  }
  stamp(5);   // merged
}

template <typename T, int D>
__global__ void decode_attention_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                const int* __restrict__ q_start, const int* __restrict__ ctx_len,
                                                T* __restrict__ out, int nq, int window, int KB, int NB,
                                                int* status) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, h = blockIdx.y;
  const int pos = ctx_len[r] - 1;
  if (pos < 0 || pos / KB >= NB) {  // a context beyond the key blocks the scratch was sized for
    if (threadIdx.x == 0) atomicCAS(status, 0, KVB_STATUS_BAD_POSITION);
    return;
  }
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int b0 = lo / KB, b1 = pos / KB;  // blocks that hold keys
  const float* ml = part_ml + ((size_t)r * nq + h) * NB * 2;
  const float* po = part_o + ((size_t)r * nq + h) * NB * D;
  float M = -CUDART_INF_F;
  for (int b = b0; b <= b1; ++b) M = fmaxf(M, ml[2 * b]);
  float L = 0.f;
  for (int b = b0; b <= b1; ++b) L += ml[2 * b + 1] * __expf(ml[2 * b] - M);
  T* o = out + ((size_t)q_start[r] * nq + h) * D;
  for (int dd = threadIdx.x; dd < D; dd += blockDim.x) {
    float a = 0.f;
    for (int b = b0; b <= b1; ++b) a += po[(size_t)b * D + dd] * __expf(ml[2 * b] - M);
    o[dd] = from_f32<T>(L > 0.f ? a / L : 0.f);
  }
}

template <typename T, int D, int GMAX>
static int launch_decode(const void* q, int q_row_stride, const void* k_pages, const void* v_pages,
                         const int* block_table, int max_pages, int page_size, int num_pages, const int* q_start,
                         const int* ctx_len, void* out, float* part_o, float* part_ml, int R, int nq, int nkv,
                         float scale, int window, int KB, int NB, int* status, cudaStream_t stream) {
  // about four blocks per SM in total, never more slots than key blocks
  int slots = (4 * kvb_sm_count() + nkv * R - 1) / (nkv * R);
  slots = slots < 1 ? 1 : (slots > NB ? NB : slots);
  dim3 grid(nkv, R, slots);
  const size_t smem = (size_t)4 * 32 * D * sizeof(T);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(decode_attention_split_kernel<T, D, GMAX>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  kvb_launch(decode_attention_split_kernel<T, D, GMAX>, grid, dim3(kDecThreads), smem, stream, (const T*)q,
             q_row_stride, (const T*)k_pages, (const T*)v_pages, block_table, max_pages, page_size, num_pages,
             q_start, ctx_len, part_o, part_ml, nq, nkv, nq / nkv, scale, window, KB, NB, status);
  kvb_launch(decode_attention_combine_kernel<T, D>, dim3(R, nq), dim3(D >= 64 ? 64 : 32), 0, stream,
             (const float*)part_o, (const float*)part_ml, q_start, ctx_len, (T*)out, nq, window, KB, NB, status);
  return kvb_launch_result();
}

// Returns 1 when (d, group) has a split kernel: d in {32, 64, 128}, group <= 8.
KVB_EXPORT int kvb_decode_attention_supported(int d, int group) {
  return (d == 32 || d == 64 || d == 128) && group >= 1 && group <= 8;
}

// One query token per request: token row q_start[r], position ctx_len[r]-1.
// Scratch: part_o [R, nq, NB, d] and part_ml [R, nq, NB, 2] float32, NB = key blocks
// of KB keys (KB a multiple of 128) covering the longest context the caller allows.
// Two launches.  Refuses what kvb_decode_attention_supported refuses, and R or NB > 65535.
KVB_EXPORT int kvb_decode_attention(const void* q, int q_row_stride, const void* k_pages, const void* v_pages,
                                    const int* block_table, int max_pages, int page_size, int num_pages,
                                    const int* q_start, const int* ctx_len, void* out, float* part_o,
                                    float* part_ml, int R, int nq, int nkv, int d, float scale, int window,
                                    int KB, int NB, int dtype, int* status, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (nkv < 1 || nq % nkv || !kvb_decode_attention_supported(d, nq / nkv) || KB % kDecThreads || NB < 1 ||
      R > 65535 || NB > 65535)
    return KVB_ERR_BAD_SIZE;
  const int G = nq / nkv;
#define KVB_DEC(T, D, GM)                                                                                  \
  return launch_decode<T, D, GM>(q, q_row_stride, k_pages, v_pages, block_table, max_pages, page_size,    \
                                 num_pages, q_start, ctx_len, out, part_o, part_ml, R, nq, nkv, scale,    \
                                 window, KB, NB, status, stream)
#define KVB_DEC_D(T, D) do { if (G <= 2) KVB_DEC(T, D, 2); else if (G <= 4) KVB_DEC(T, D, 4); else KVB_DEC(T, D, 8); } while (0)
#define KVB_DEC_T(T) do { if (d == 32) KVB_DEC_D(T, 32); else if (d == 64) KVB_DEC_D(T, 64); else KVB_DEC_D(T, 128); } while (0)
  if (dtype == KVB_BF16) KVB_DEC_T(__nv_bfloat16);
  if (dtype == KVB_F32) KVB_DEC_T(float);
  return KVB_ERR_BAD_DTYPE;
}

// ===========================================================================
// The same decode attention for callers that cannot allocate: the scratch between
// the split and the combine launch is a static device array of this library.
// Declared and documented in decode_attention_noalloc.h.
// ===========================================================================
#include "decode_attention_noalloc.h"

#include <mutex>

static __device__ __align__(256) float g_decode_noalloc_scratch[KVB_DECODE_NOALLOC_SCRATCH_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
float* g_noalloc_ptr[kMaxDevices] = {nullptr};  // device address of the array, per device ordinal

// In host code `g_decode_noalloc_scratch` is only a handle for the runtime, not an
// address a kernel could use; the device address has to be asked for, once per
// device, with that device current.
int noalloc_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return KVB_ERR_SCRATCH_SETUP;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_decode_noalloc_scratch);
    if (e != cudaSuccess) return (int)e;
    if (p == nullptr) return KVB_ERR_SCRATCH_SETUP;
    g_noalloc_ptr[dev] = static_cast<float*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}
}  // namespace

KVB_EXPORT unsigned long long kvb_decode_attention_noalloc_scratch_needed(int R, int nq, int NB, int d) {
  if (R < 0 || nq < 0 || NB < 0 || d < 0) return ~0ull;
  return (unsigned long long)R * nq * NB * (unsigned long long)(d + 2);
}

KVB_EXPORT const char* kvb_decode_attention_noalloc_error(int code) {
  switch (code) {
    case 0: return "ok";
    case KVB_ERR_BAD_DTYPE: return "unsupported dtype (0 = float32, 1 = bfloat16)";
    case KVB_ERR_BAD_SIZE:
      return "a size the decode kernel refuses (head size must be 32, 64 or 128, group size 1..8, KB a multiple of 128)";
    case KVB_ERR_SCRATCH_TOO_SMALL:
      return "R * nq * NB * (d + 2) exceeds the 4 Mi floats of built-in scratch; use kvb_decode_attention with "
             "caller-provided scratch, or fewer requests / key blocks per call";
    case KVB_ERR_SCRATCH_SETUP: return "the built-in scratch could not be located on the current device";
    default: return code > 0 ? "a CUDA runtime error (the code is a cudaError_t)" : "unknown error code";
  }
}

KVB_EXPORT int kvb_decode_attention_noalloc(const void* q, int q_row_stride, const void* k_pages,
                                            const void* v_pages, const int* block_table, int max_pages,
                                            int page_size, int num_pages, const int* q_start,
                                            const int* ctx_len, void* out, int R, int nq, int nkv, int d,
                                            float scale, int window, int KB, int NB, int dtype, int* status,
                                            cudaStream_t stream) {
  if (R <= 0) return 0;
  if (nq < 1 || NB < 1 || d < 1) return KVB_ERR_BAD_SIZE;
  const unsigned long long need = kvb_decode_attention_noalloc_scratch_needed(R, nq, NB, d);
  if (need > (unsigned long long)KVB_DECODE_NOALLOC_SCRATCH_FLOATS) return KVB_ERR_SCRATCH_TOO_SMALL;
  float* scratch = nullptr;
  const int rc = noalloc_scratch_for_current_device(&scratch);
  if (rc != 0) return rc;
  // Partial outputs first, then the (max, sum) pairs.  The array itself is aligned to 256 bytes;
  // the second offset, R * nq * NB * d floats, is a multiple of 16 bytes because the split kernel
  // takes head sizes 32, 64 and 128 only (any other d is refused by kvb_decode_attention below
  // before anything is launched), so d floats are always a multiple of 128 bytes.
  float* part_o = scratch;
  float* part_ml = scratch + (size_t)R * nq * NB * d;
  return kvb_decode_attention(q, q_row_stride, k_pages, v_pages, block_table, max_pages, page_size, num_pages,
                              q_start, ctx_len, out, part_o, part_ml, R, nq, nkv, d, scale, window, KB, NB,
                              dtype, status, stream);
}


template <typename T, int D, int GMAX>
static int launch_decode_fused(const void* qkv, int q_row_stride, void* k_pages, void* v_pages, int write_kv,
                               const int* block_table, int max_pages, int page_size, int num_pages,
                               const int* q_start, const int* ctx_len, const float* cos_t, const float* sin_t,
                               int table_len, int rot, void* out, float* part_o, float* part_ml, int* counters,
                               int R, int nq, int nkv, float scale, int window, int KB, int NB, int* status,
                               unsigned long long* trace, cudaStream_t stream) {
  int slots = (4 * kvb_sm_count() + nkv * R - 1) / (nkv * R);
  slots = slots < 1 ? 1 : (slots > NB ? NB : slots);
  dim3 grid(nkv, R, slots);
  const size_t smem = (size_t)2 * 4 * 32 * D * sizeof(T);   // a key tile and a value tile of 128 positions
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(decode_attention_fused_kernel<T, D, GMAX>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  kvb_launch(decode_attention_fused_kernel<T, D, GMAX>, grid, dim3(kDecThreads), smem, stream, (const T*)qkv,
             q_row_stride, (T*)k_pages, (T*)v_pages, write_kv, block_table, max_pages, page_size, num_pages,
             q_start, ctx_len, cos_t, sin_t, table_len, rot, (T*)out, part_o, part_ml, counters, nq, nkv, nq / nkv,
             scale, window, KB, NB, status, trace);
  return kvb_launch_result();
}

// The attention of a decode step in one launch (see decode_attention_fused_kernel).
// qkv: [T, (nq + 2 nkv) d] as the projection wrote it; request r's token is row q_start[r]
// at position ctx_len[r]-1.  write_kv = 0: the layer reads another layer's cache and
// writes nothing.  cos_t/sin_t: [table_len, rot/2] or nullptr for no rotation.
// Scratch: part_o [R, nq, NB, d], part_ml [R, nq, NB, 2] float32; counters [R * nkv] int32,
// zero on entry, left zero.  trace: nullptr, or [blocks, 8] uint64 phase stamps (profiling).
// Same size rules as kvb_decode_attention.
KVB_EXPORT int kvb_decode_attention_fused(const void* qkv, int q_row_stride, void* k_pages, void* v_pages,
                                          int write_kv, const int* block_table, int max_pages, int page_size,
                                          int num_pages, const int* q_start, const int* ctx_len,
                                          const float* cos_t, const float* sin_t, int table_len, int rot, void* out,
                                          float* part_o, float* part_ml, int* counters, int R, int nq, int nkv,
                                          int d, float scale, int window, int KB, int NB, int dtype, int* status,
                                          unsigned long long* trace, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (nkv < 1 || nq % nkv || !kvb_decode_attention_supported(d, nq / nkv) || KB % kDecThreads || NB < 1 ||
      R > 65535 || (rot & 1) || rot > d)
    return KVB_ERR_BAD_SIZE;
  const int G = nq / nkv;
#define KVB_DECF(T, D, GM)                                                                                   \
  return launch_decode_fused<T, D, GM>(qkv, q_row_stride, k_pages, v_pages, write_kv, block_table, max_pages, \
                                       page_size, num_pages, q_start, ctx_len, cos_t, sin_t, table_len, rot,  \
                                       out, part_o, part_ml, counters, R, nq, nkv, scale, window, KB, NB,     \
                                       status, trace, stream)
#define KVB_DECF_D(T, D) do { if (G <= 2) KVB_DECF(T, D, 2); else if (G <= 4) KVB_DECF(T, D, 4); else KVB_DECF(T, D, 8); } while (0)
#define KVB_DECF_T(T) do { if (d == 32) KVB_DECF_D(T, 32); else if (d == 64) KVB_DECF_D(T, 64); else KVB_DECF_D(T, 128); } while (0)
  if (dtype == KVB_BF16) KVB_DECF_T(__nv_bfloat16);
  if (dtype == KVB_F32) KVB_DECF_T(float);
  return KVB_ERR_BAD_DTYPE;
}
