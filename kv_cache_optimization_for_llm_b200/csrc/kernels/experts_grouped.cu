// The products of gated experts (experts.cu) over the tokens that chose them, for steps of many bfloat16 tokens.
//
//   * expert_lists_kernel: a block per expert writes the tokens that chose it, in their order, and each one's place
//     among them;
//   * gather_rows_kernel copies every token's row to its experts' (requests of four scattered rows by TMA, tile::gather4, took the
//     product 62 us more than tiles that lie together; the copy takes 8);
//   * grouped_kernel<FIRST>: gate and up products with the activation behind them.  A tile is 128 tokens of one expert x 128 features: 128 gate rows and the 128 up rows of the same
//     features are one operand of 256, so the epilogue has both in one lane of tensor memory.  The expert that every token uses
//     is more tiles of the same kind, its tokens read as they lie.  Results: the chosen experts' rows one behind the other,
//     and the shared expert's row per token;
//   * grouped_kernel<SECOND>: the chosen experts' rows times their second matrices, as float32 rows;
//   * join_rows_kernel: the shared expert's second product (made by the caller, float32) plus a token's rows, the lowest expert
//     first, rounded once.  (As the epilogue of that product, four lanes a row: 43 us with it, 15 and 11 apart.)
//
// The products are one persistent form: a block an SM of six warps (loader, issuer, four for the epilogue), tiles of 128 x 256, four
// stages of 64 k by TMA with the 128-byte swizzle, two accumulators in tensor memory.  What the experts' counts
// are is known on the device only: every block adds them up and finds its tiles in the sums, so the host waits for nothing
// and a captured step may route otherwise each time.
// Every sum follows the sizes and the expert's index, not the neighbours in the step.
// Measured (2048 tokens, width 2048, 32 experts of 256 features of which a token uses 4, a shared one of 2048; us): FIRST 71, SECOND 25, the
// shared second product 18, join 16, gather 8, lists 5; all products over all tokens with the activation kernel between them 195.  What
// bounds FIRST: the operands' way from L2 (48 KB per 64 k and SM, 0.7 us; 13 TB/s over the GPU), not the tensor pipe (0.27 us).
#include "limited_act.cuh"
#include "tc5.cuh"

namespace {

using namespace tc5;

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int kStages = 4, kABytes = BM * 128, kBBytes = BN * 128, kStageBytes = kABytes + kBBytes;
constexpr int kMaxExperts = 256, kMaxTop = 16;
enum { FIRST = 0, SECOND = 1 };
constexpr int kThreads = 192;
constexpr int pitch_of(int mode) { return mode == FIRST ? 20 : 36; }     // words between rows of a warp's 32 in shared memory

struct Params {
  const float* gate; int ld_gate;            // [T, >= E], 0: not chosen
  const float* shared_logit; int ld_s;       // [T] or nullptr
  const int* counts; const int* list;        // [E], [E][T]
  int T, E, H, F, S, top;
  float limit, shared_limit, alpha, offset;
  int weigh_output;
  __nv_bfloat16* act; __nv_bfloat16* shared_act;          // FIRST: [T top, F], [T, S]
  float* rows;                                            // SECOND: [T top, H]
  int* status;
};

struct alignas(16) Shared {
  unsigned long long full[kStages], empty[kStages], acc_full[2], acc_empty[2];
  unsigned tmem;
  int abort_flag;
  int base[kMaxExperts + 1];      // rows of the experts in front
  int tile[kMaxExperts + 1];      // tiles of 128 rows of the experts in front
};

__device__ __forceinline__ void tmem_ld32(unsigned taddr, float* v) {
  unsigned r[32];
  tmem_ld16(taddr, r);
  tmem_ld16(taddr + 16, r + 16);
  wait_ld();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<unsigned*>(&h);
}

__global__ void __launch_bounds__(512) expert_lists_kernel(const float* __restrict__ gate, int ld_gate, int T, int E,
                                                           int* __restrict__ counts, int* __restrict__ list, int* __restrict__ place) {
  __shared__ int warp_total[16];
  pdl_trigger();
  pdl_wait();
  const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int before = 0;
  for (int t0 = 0; t0 < T; t0 += 512) {
    const int t = t0 + threadIdx.x;
    const bool chosen = t < T && gate[(size_t)t * ld_gate + e] != 0.f;
    const unsigned votes = __ballot_sync(0xffffffffu, chosen);
    if (lane == 0) warp_total[warp] = __popc(votes);
    __syncthreads();
    int at = before + __popc(votes & ((1u << lane) - 1u)), all = 0;
#pragma unroll
    for (int w = 0; w < 16; ++w) {
      const int n = warp_total[w];
      if (w < warp) at += n;
      all += n;
    }
    if (chosen) {
      list[(size_t)e * T + at] = t;
      place[(size_t)t * E + e] = at;
    }
    before += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) counts[e] = before;
}

// Rows of the experts in front of each expert, by one warp: to[0 .. E]; tiles of 128 rows of them as well where wanted.
__device__ __forceinline__ void add_up(const int* __restrict__ counts, int E, int* to, int* tiles, int lane) {
  int rows = 0, cut = 0;
  for (int b = 0; b < E; b += 32) {
    const int n = b + lane < E ? counts[b + lane] : 0;
    int r = n, t = (n + BM - 1) / BM;
    for (int o = 1; o < 32; o <<= 1) {
      const int r2 = __shfl_up_sync(0xffffffffu, r, o), t2 = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) { r += r2; t += t2; }
    }
    if (b + lane < E) {
      to[b + lane + 1] = rows + r;
      if (tiles != nullptr) tiles[b + lane + 1] = cut + t;
    }
    rows += __shfl_sync(0xffffffffu, r, 31);
    cut += __shfl_sync(0xffffffffu, t, 31);
  }
  if (lane == 0) {
    to[0] = 0;
    if (tiles != nullptr) tiles[0] = 0;
  }
}

// A block per token: its row of x goes to each of its experts' rows, and their numbers into rows_of[t, 0 .. top), the lowest expert
// first (-1 behind the last).
__global__ void __launch_bounds__(128) gather_rows_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const float* __restrict__ gate,
                                                          int ld_gate, const int* __restrict__ counts, const int* __restrict__ place,
                                                          int E, int H, int top, __nv_bfloat16* __restrict__ xg, int* __restrict__ rows_of) {
  __shared__ int base[kMaxExperts + 1], mine[kMaxTop];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    add_up(counts, E, base, nullptr, lane);
    __syncwarp();
    int n = 0;
    for (int b = 0; b < E; b += 32) {
      const bool chosen = b + lane < E && gate[(size_t)t * ld_gate + b + lane] != 0.f;
      const unsigned votes = __ballot_sync(0xffffffffu, chosen);
      const int at = n + __popc(votes & ((1u << lane) - 1u));
      if (chosen && at < top) mine[at] = base[b + lane] + place[(size_t)t * E + b + lane];
      n += __popc(votes);
    }
    if (lane >= n && lane < top) mine[lane] = -1;
    __syncwarp();
    if (lane < top) rows_of[(size_t)t * top + lane] = mine[lane];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < H / 8; c += 128) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + c * 8);
    for (int j = 0; j < top; ++j)
      if (mine[j] >= 0) *reinterpret_cast<uint4*>(xg + (size_t)mine[j] * H + c * 8) = v;
  }
}

__global__ void __launch_bounds__(256) join_rows_kernel(const float* __restrict__ shared, const float* __restrict__ rows,
                                                        const int* __restrict__ rows_of, __nv_bfloat16* __restrict__ out, int H, int top) {
  pdl_trigger();
  pdl_wait();
  const size_t t = blockIdx.x;
  int row[kMaxTop];
#pragma unroll
  for (int j = 0; j < kMaxTop; ++j) row[j] = j < top ? rows_of[t * top + j] : -1;
  for (int c = threadIdx.x * 4; c < H; c += 1024) {
    float4 s = *reinterpret_cast<const float4*>(shared + t * H + c);
#pragma unroll
    for (int j = 0; j < kMaxTop; ++j)
      if (row[j] >= 0) {
        const float4 v = *reinterpret_cast<const float4*>(rows + (size_t)row[j] * H + c);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
    *reinterpret_cast<uint2*>(out + t * H + c) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
  }
}

// The expert whose tiles hold tile `m` (all lanes of a warp ask together): the last one that begins at or in front of it and has any.
__device__ __forceinline__ int expert_of(const Shared* sh, int E, int m, int lane) {
  int e = 0;
  for (int b = 0; b < E; b += 32)
    e += __popc(__ballot_sync(0xffffffffu, b + lane < E && sh->tile[b + lane + 1] <= m));
  return e;
}

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
grouped_kernel(const __grid_constant__ CUtensorMap map_own, const __grid_constant__ CUtensorMap map_all,
               const __grid_constant__ CUtensorMap map_w, const Params p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Shared* sh = reinterpret_cast<Shared*>(base + kStages * kStageBytes);
  float* staging = reinterpret_cast<float*>(sh + 1);
  volatile int* abort_flag = &sh->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&sh->acc_full[a], 1); mbar_init(&sh->acc_empty[a], 4); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&sh->tmem, 512);
  fence_before();
  __syncthreads();
  fence_after();
  const unsigned tmem = sh->tmem;
  pdl_trigger();
  pdl_wait();
  if (warp == 0) add_up(p.counts, p.E, sh->base, sh->tile, lane);
  __syncthreads();

  // tiles: the experts' first (rows of tokens outside, features inside), then the shared expert's
  const int routed_m = sh->tile[p.E];
  const int routed_n = MODE == FIRST ? p.F / 128 : (p.H + BN - 1) / BN;
  const int shared_m = (p.T + BM - 1) / BM;
  const int routed = routed_m * routed_n, total = routed + (MODE == SECOND ? 0 : shared_m * (p.S / 128));
  const int steps = ((MODE == FIRST ? p.H : p.F) + BK - 1) / BK;
  auto place_of = [&](int tile, int& m, int& n) {
    if (MODE == SECOND || tile < routed) { m = tile / routed_n; n = tile - m * routed_n; }
    else { n = (tile - routed) / shared_m; m = tile - routed - n * shared_m; }
  };
  bool failed = false;

  if (warp == 0) {
    int s = 0;
    unsigned parity = 1;      // a first pass over the ring waits for nothing
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const bool own = MODE == SECOND || tile < routed;
      int m, n;
      place_of(tile, m, n);
      const int e = own ? expert_of(sh, p.E, m, lane) : p.E;
      const int r0 = own ? sh->base[e] + (m - sh->tile[e]) * BM : m * BM;
      for (int k = 0; k < steps; ++k) {
        if (lane == 0) {
          if (!wait_or_abort(&sh->empty[s], parity, abort_flag)) { failed = true; break; }
          unsigned char* a_s = base + s * kStageBytes;
          mbar_expect_tx(&sh->full[s], kStageBytes);
          if (MODE == FIRST) {
            const int w0 = (own ? 2 * e * p.F : 2 * p.E * p.F) + n * 128;
            tma_load_2d(a_s + kABytes, &map_w, k * BK, w0, &sh->full[s]);
            tma_load_2d(a_s + kABytes + kBBytes / 2, &map_w, k * BK, w0 + (own ? p.F : p.S), &sh->full[s]);
          } else {
            const int col = e * p.F + k * BK;
            tma_load_2d(a_s + kABytes, &map_w, col, n * BN, &sh->full[s]);
            tma_load_2d(a_s + kABytes + kBBytes / 2, &map_w, col, n * BN + BN / 2, &sh->full[s]);
          }
          tma_load_2d(a_s, own ? &map_own : &map_all, k * BK, r0, &sh->full[s]);
        }
        if (++s == kStages) { s = 0; parity ^= 1u; }
      }
      failed = __shfl_sync(0xffffffffu, (int)failed, 0) != 0;
      if (failed) break;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const unsigned idesc = idesc_bf16(BM, BN);
      int s = 0, acc = 0;
      unsigned parity = 0, acc_parity = 1;
      for (int tile = blockIdx.x; tile < total && !failed; tile += gridDim.x) {
        if (!wait_or_abort(&sh->acc_empty[acc], acc_parity, abort_flag)) { failed = true; break; }
        fence_after();
        const unsigned d = tmem + acc * BN;
        for (int k = 0; k < steps; ++k) {
          if (!wait_or_abort(&sh->full[s], parity, abort_flag)) { failed = true; break; }
          fence_after();
          const unsigned a_addr = smem_u32(base + s * kStageBytes);
          const unsigned long long ad = smem_desc_sw128(a_addr), bd = smem_desc_sw128(a_addr + kABytes);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) umma_ss(d, ad + 2 * kk, bd + 2 * kk, idesc, (k | kk) ? 1u : 0u);
          umma_commit(&sh->empty[s]);
          if (++s == kStages) { s = 0; parity ^= 1u; }
        }
        if (!failed) umma_commit(&sh->acc_full[acc]);
        if (++acc == 2) { acc = 0; acc_parity ^= 1u; }
      }
    }
  } else {
    const int r = (warp & 3) * 32 + lane;                       // row of the tile
    const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16);
    int acc = 0;
    unsigned parity = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const bool own = MODE == SECOND || tile < routed;
      int m, n;
      place_of(tile, m, n);
      const int e = own ? expert_of(sh, p.E, m, lane) : p.E;
      const int i = (own ? m - sh->tile[e] : m) * BM + r;
      const bool there = i < (own ? sh->base[e + 1] - sh->base[e] : p.T);
      float w = 1.f, post = 1.f, lim = p.limit;
      if (MODE == FIRST) {
        if (own) {
          if (there) w = p.gate[(size_t)p.list[(size_t)e * p.T + i] * p.ld_gate + e];
          if (p.weigh_output) { post = w; w = 1.f; }
        } else {
          lim = p.shared_limit;
          if (there && p.shared_logit != nullptr) post = 1.0f / (1.0f + expf(-p.shared_logit[(size_t)i * p.ld_s]));
        }
      }
      float* mine = staging + (warp - 2) * 32 * pitch_of(MODE);
      if (!wait_or_abort(&sh->acc_full[acc], parity, abort_flag)) { failed = true; break; }
      fence_after();
      const unsigned cols = lanes + acc * BN;
      // Results go through shared memory, so that neighbouring lanes store neighbouring bytes of a row.
      if (MODE == FIRST) {
        const int first_row = i - lane, rows_there = (own ? sh->base[e + 1] - sh->base[e] : p.T) - first_row;
        __nv_bfloat16* to = own ? p.act + (size_t)(sh->base[e] + first_row) * p.F + n * 128 : p.shared_act + (size_t)first_row * p.S + n * 128;
        const int ld = own ? p.F : p.S;
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          float g[32], u[32];
          tmem_ld32(cols + c, g);
          tmem_ld32(cols + 128 + c, u);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            unsigned o[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              o[q] = pack_bf16(limited_one(g[j + 2 * q], u[j + 2 * q], w, lim, p.alpha, p.offset) * post,
                               limited_one(g[j + 2 * q + 1], u[j + 2 * q + 1], w, lim, p.alpha, p.offset) * post);
            *reinterpret_cast<uint4*>(mine + lane * 20 + j / 2) = make_uint4(o[0], o[1], o[2], o[3]);
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int row = 8 * q + (lane >> 2);
            if (row < rows_there)
              *reinterpret_cast<uint4*>(to + (size_t)row * ld + c + 8 * (lane & 3)) = *reinterpret_cast<const uint4*>(mine + row * 20 + 4 * (lane & 3));
          }
        }
      } else {
        const int first_row = i - lane, rows_there = sh->base[e + 1] - sh->base[e] - first_row;
        float* to = p.rows + (size_t)(sh->base[e] + first_row) * p.H + n * BN;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          float v[32];
          tmem_ld32(cols + c, v);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(mine + lane * 36 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
          __syncwarp();
          const int col = c + 4 * (lane & 7);
          if (n * BN + col < p.H)            // H is a multiple of 8
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const int row = 4 * q + (lane >> 3);
              if (row < rows_there)
                *reinterpret_cast<float4*>(to + (size_t)row * p.H + col) = *reinterpret_cast<const float4*>(mine + row * 36 + 4 * (lane & 7));
            }
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->acc_empty[acc]);
      if (++acc == 2) { acc = 0; parity ^= 1u; }
    }
  }
  if (failed) *abort_flag = 1;
  fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) atomicCAS(p.status, 0, KVB_STATUS_WAIT_TIMEOUT);
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let copies and products that may still run finish
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 512);
}

constexpr int smem_of(int mode) { return 1024 + kStages * kStageBytes + (int)sizeof(Shared) + 4 * 4 * 32 * pitch_of(mode); }
static_assert(smem_of(FIRST) <= 232448 && smem_of(SECOND) <= 232448, "shared memory of a block");

template <int MODE>
int launch(const CUtensorMap& own, const CUtensorMap& all, const CUtensorMap& w, const Params& p, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(grouped_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_of(MODE));
  if (e != cudaSuccess) return (int)e;
  e = kvb_launch(grouped_kernel<MODE>, dim3(kvb_sm_count()), dim3(kThreads), smem_of(MODE), stream, own, all, w, p);
  return e == cudaSuccess ? kvb_launch_result() : (int)e;
}

int bf16_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, long long ld, int box) {
  return make_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, rows, cols, ld * 2, box);
}

}  // namespace

// The chosen experts' part of a step: float32 rows [T top, H] of down_e act_e(x), expert after expert, and their numbers rows_of[t, 0 .. top), the
// lowest expert first, -1 behind the last; and shared_act [T, S], the activation of the expert that every token uses.
// x [T, H]; first [2 E F + 2 S, H]: per expert F gate rows and F up rows, then the shared expert's; down [H, >= E F] with rows ld_down apart,
// the experts' columns side by side.  gate [T, >= E] float32, 0 for an expert that was not chosen, at most `top` others a row.
// Scratch: lists E + 2 E T ints, xg T top H and act T top F bfloat16.  F and S multiples of 128, H of 8; everything on 16-byte
// boundaries.
KVB_EXPORT int kvb_experts_grouped(const void* x, int ldx, const void* first, const void* down, int ld_down, const float* gate,
                                   int ld_gate, const float* shared_logit, int ld_s, int T, int H, int E, int F, int S, int top,
                                   float limit, float shared_limit, float alpha, float offset, int weigh_output, int* lists, void* xg,
                                   void* act, void* shared_act, float* rows, int* rows_of, int* status, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H < 8 || (H & 7) || E < 1 || E > kMaxExperts || F < 128 || (F & 127) || S < 128 || (S & 127) || top < 1 || top > E || top > kMaxTop)
    return KVB_ERR_BAD_SIZE;
  if ((long long)T * top > 0x3fffffff || 2ll * E * F + 2ll * S > 0x3fffffff) return KVB_ERR_BAD_SIZE;
  if ((ldx & 7) || (ld_down & 7) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(first) |
      reinterpret_cast<uintptr_t>(down) | reinterpret_cast<uintptr_t>(xg) | reinterpret_cast<uintptr_t>(act) |
      reinterpret_cast<uintptr_t>(shared_act) | reinterpret_cast<uintptr_t>(rows)) & 15)) return KVB_ERR_ALIGN;
  Params p;
  p.gate = gate; p.ld_gate = ld_gate; p.shared_logit = shared_logit; p.ld_s = ld_s;
  int *counts = lists, *list = lists + E, *place = list + (size_t)E * T;
  p.counts = counts; p.list = list;
  p.T = T; p.E = E; p.H = H; p.F = F; p.S = S;
  p.limit = limit; p.shared_limit = shared_limit; p.alpha = alpha; p.offset = offset; p.weigh_output = weigh_output;
  p.act = (__nv_bfloat16*)act; p.shared_act = (__nv_bfloat16*)shared_act; p.rows = rows;
  p.status = status;
  CUtensorMap mx, mg, m1, ma, m2;
  int e;
  if ((e = bf16_map(&mx, x, T, H, ldx, BM)) || (e = bf16_map(&mg, xg, (long long)T * top, H, H, BM)) ||
      (e = bf16_map(&m1, first, 2ll * E * F + 2ll * S, H, H, 128)) || (e = bf16_map(&ma, act, (long long)T * top, F, F, BM)) ||
      (e = bf16_map(&m2, down, H, (long long)E * F, ld_down, 128)))
    return e;
  cudaError_t ce = kvb_launch(expert_lists_kernel, dim3(E), dim3(512), 0, stream, gate, ld_gate, T, E, counts, list, place);
  if (ce != cudaSuccess) return (int)ce;
  ce = kvb_launch(gather_rows_kernel, dim3(T), dim3(128), 0, stream, (const __nv_bfloat16*)x, ldx, gate, ld_gate, counts, place, E, H, top,
                  (__nv_bfloat16*)xg, rows_of);
  if (ce != cudaSuccess) return (int)ce;
  if ((e = launch<FIRST>(mg, mx, m1, p, stream))) return e;
  return launch<SECOND>(ma, ma, m2, p, stream);
}

// out[t] = shared[t] + the token's rows in their order, rounded once.  shared [T, H] float32 dense, out bfloat16 dense, H a multiple of 8.
KVB_EXPORT int kvb_experts_join(const float* shared, const float* rows, const int* rows_of, void* out, int T, int H, int top,
                                cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H < 8 || (H & 7) || top < 1 || top > kMaxTop) return KVB_ERR_BAD_SIZE;
  if ((reinterpret_cast<uintptr_t>(shared) | reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(out)) & 15) return KVB_ERR_ALIGN;
  cudaError_t ce = kvb_launch(join_rows_kernel, dim3(T), dim3(256), 0, stream, shared, rows, rows_of, (__nv_bfloat16*)out, H, top);
  return ce == cudaSuccess ? kvb_launch_result() : (int)ce;
}
