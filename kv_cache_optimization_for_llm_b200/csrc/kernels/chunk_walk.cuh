// A matrix memory per head with one decay per head and token, along a request's run of tokens, on tensor cores:
//
//   S_t = keep_t S_{t-1} + take_t k_t v_t^T   (S is N x Dv),     y_t = S_t^T q_t
//
// with q, k, v bfloat16 and everything else float32.  A block owns DVC value columns of one (request, head) and walks the
// run in pieces of 64 tokens.  Inside a piece (i, j its tokens, P_i the product of the decays up to i, S what it begins with):
//
//   y_i = P_i (S^T q_i) + sum_{j <= i} (q_i . k_j) (P_i / P_j) take_j v_j
//   S  <- P_63 S + sum_j (P_63 / P_j) take_j k_j v_j^T
//
// four products on mma.sync m16n8k16, the state in their accumulators for the whole run.  In each of them one operand is
// bfloat16 as it came; the other (the state, the weighed scores, the weighed values) is float32 and goes in as the sum of three
// bfloat16 numbers, which hold its 24 bits, so that the products are as exact as float32 ones.  Decays are kept as
// logarithms summed up in float64 and differences taken from pairs (high, low) of floats: a quotient P_i / P_j of two close
// tokens does not lose digits to a long run's sum.
//
// What bounds it: one piece is a chain of four products and three barriers (about 2 us for a block alone on its SM); a run is as many
// pieces one behind the other, and the heads' columns are dealt over the SMs.  Walking token by token in float32 instead was bound
// by the FMAs and the shared-memory loads that feed them, and took three launches (pieces side by side, a sweep over
// their states in memory, the pieces again): 64 heads of 128 x 64, runs of 1111 + 700 + 237 tokens about 700 us, now 118; 32 heads of
// 64 x 64, 2048 tokens about 260 us, now 125.
#pragma once

#include "common.cuh"

#include <math_constants.h>

namespace walk {

typedef __nv_bfloat16 bf16;

constexpr int kPiece = 64, kThreads = 128, kGateWarp = kThreads / 32, kBlock = kThreads + 32;      // a fifth warp makes the next piece's gates

enum Rule { SSD = 0, MLSTM = 1 };

struct Args {
  // bfloat16; head h reads q and k at (h / share) * N and v at h * Dv, rows ld apart (all three pointers at their first column)
  const bf16* q; const bf16* k; const bf16* v; int ld, share;
  // SSD: raw step sizes (bfloat16, rows ld_g apart), take = softplus(raw + bias), keep = exp(-exp(A_log) take), y += D v
  const bf16* dt; const float* dt_bias; const float* A_log; const float* D;
  // MLSTM: raw input gates, then raw forget gates (float32 [T, 2 H], rows ld_g apart), capped; y = S^T q / denominator
  const float* gates; const float* bi; const float* bf; float cap, q_scale;
  int ld_g;
  float* state; long long slot_stride;     // slot 0's [H][Dv][N]; MLSTM: behind it [H][Dv / 64][N] and [H][Dv / 64]
  float* y;                                // [T, H * Dv] float32
  const int* q_start; const int* req_start; const int* slots;
  int H, Dv, first;                        // requests first .. are walked
};

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm4(uint32_t* r, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldm4t(uint32_t* r, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldm2t(uint32_t* r, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(void* to, const void* from, bool inside) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_at(to)), "l"(from), "r"(inside ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t pair_of(bf16 x, bf16 y) {
  __nv_bfloat162 v;
  v.x = x; v.y = y;
  return *reinterpret_cast<uint32_t*>(&v);
}
// x and y as sums of three bfloat16 numbers each: p[0] + p[1] + p[2], the two side by side
__device__ __forceinline__ void split3(uint32_t* p, float x, float y) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
    p[i] = *reinterpret_cast<const uint32_t*>(&v);
    x -= __bfloat162float(v.x);
    y -= __bfloat162float(v.y);
  }
}

// bytes from row to row: an odd number of 16-byte chunks, so that eight rows' chunks lie in different banks
__host__ __device__ constexpr int pitch(int cols) { return (cols * 2 / 16 | 1) * 16; }

template <int RULE, int N, int DVC>
struct Layout {
  static constexpr int COLS = DVC + (RULE == MLSTM ? 8 : 0);     // MLSTM: the vector n is one more value column, of ones
  static constexpr int PN = pitch(N), PX = pitch(DVC), PC = pitch(COLS);
  static constexpr int K = 0;                                     // [2][64] rows of PN
  static constexpr int Q = K + 2 * kPiece * PN;                   // [64] rows of PN
  static constexpr int X = Q + kPiece * PN;                       // [2][64] rows of PX
  static constexpr int W = X + 2 * kPiece * PX;                   // [3][64] rows of PC: weighed values
  static constexpr int S = W + 3 * kPiece * PC;                   // [3][N] rows of PC: the state
  static constexpr int G = S + 3 * N * PC;                        // [2] gates
  static constexpr int bytes = G + 2 * (8 * kPiece + 4) * 4;
};

// A piece's gates: column j's and row i's logarithms as pairs, weights of the values, factor on the state's part, and
//   SSD:   scores' factor take_j;  MLSTM: exp(-m_i)
struct Gates {
  float col_hi[kPiece], col_lo[kPiece], row_hi[kPiece], row_lo[kPiece], weigh[kPiece], from[kPiece], aux[kPiece], unused[kPiece];
  float keep, m, pad[2];
};
static_assert(sizeof(Gates) == (8 * kPiece + 4) * 4, "as laid out");

__device__ __forceinline__ void block_barrier() { asm volatile("bar.sync 0, %0;" ::"n"(kBlock) : "memory"); }
__device__ __forceinline__ void walkers_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

__device__ __forceinline__ void as_pair(double x, float& hi, float& lo) {
  hi = (float)x;
  lo = isinf(hi) ? 0.f : (float)(x - (double)hi);
}
__device__ __forceinline__ double scan_sum(double v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += x;
  }
  return v;
}
__device__ __forceinline__ double scan_max(double v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double x = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = fmax(v, x);
  }
  return v;
}

__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// the raw gates of tokens `lane` and `lane + 32` of the piece that starts at token row c0 and ends before t1
template <int RULE>
__device__ __forceinline__ void raw_gates(const Args& p, int h, int c0, int t1, int lane, float (&raw)[4]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int t = c0 + lane + 32 * u;
    raw[2 * u] = raw[2 * u + 1] = 0.f;
    if (t < t1) {
      if (RULE == SSD) {
        raw[2 * u] = __bfloat162float(p.dt[(size_t)t * p.ld_g + h]);
      } else {
        raw[2 * u] = p.gates[(size_t)t * p.ld_g + h];
        raw[2 * u + 1] = p.gates[(size_t)t * p.ld_g + p.H + h];
      }
    }
  }
}

// One warp: from the raw gates to `g`.  m: MLSTM's maximum before the piece.
template <int RULE>
__device__ __forceinline__ void make_gates(const Args& p, int h, int nt, int lane, const float (&raw)[4], float m, Gates& g) {
  if (RULE == SSD) {
    const float rate = expf(p.A_log[h]), bias = p.dt_bias[h];
    float take[2];
    double c[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const bool in = lane + 32 * u < nt;                        // behind the run's end nothing decays and nothing comes in
      take[u] = in ? softplus(raw[2 * u] + bias) : 0.f;
      c[u] = scan_sum(in ? -(double)(rate * take[u]) : 0.0, lane);
    }
    c[1] += __shfl_sync(0xffffffffu, c[0], 31);
    const double total = __shfl_sync(0xffffffffu, c[1], 31);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u;
      as_pair(c[u], g.row_hi[i], g.row_lo[i]);
      g.col_hi[i] = -g.row_hi[i];
      g.col_lo[i] = -g.row_lo[i];
      g.weigh[i] = expf((float)(total - c[u])) * take[u];
      g.from[i] = expf((float)c[u]);
      g.aux[i] = take[u];
    }
    if (lane == 0) g.keep = expf((float)total);
  } else {
    const float bi = p.bi ? p.bi[h] : 0.f, bf_ = p.bf ? p.bf[h] : 0.f;
    double F[2], a[2], mu[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const bool in = lane + 32 * u < nt;
      const float gi = p.cap * tanhf((raw[2 * u] + bi) / p.cap);
      const float gf = log_sigmoid(p.cap * tanhf((raw[2 * u + 1] + bf_) / p.cap));
      F[u] = scan_sum(in ? (double)gf : 0.0, lane);
      if (u) F[1] += __shfl_sync(0xffffffffu, F[0], 31);
      a[u] = in ? (double)gi - F[u] : -INFINITY;                 // the input gate, seen from the piece's start
    }
    mu[0] = fmax(scan_max(a[0], lane), (double)m);               // the maximum, seen from the piece's start
    mu[1] = fmax(scan_max(a[1], lane), __shfl_sync(0xffffffffu, mu[0], 31));
    const double mu_end = __shfl_sync(0xffffffffu, mu[1], 31), F_end = __shfl_sync(0xffffffffu, F[1], 31);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u;
      as_pair(a[u], g.col_hi[i], g.col_lo[i]);
      as_pair(-mu[u], g.row_hi[i], g.row_lo[i]);
      g.weigh[i] = expf((float)(a[u] - mu_end));
      g.from[i] = expf((float)((double)m - mu[u]));
      g.aux[i] = expf((float)(-(F[u] + mu[u])));
    }
    if (lane == 0) {
      g.keep = expf((float)((double)m - mu_end));
      g.m = (float)(F_end + mu_end);
    }
  }
}

template <int RULE, int N, int DVC>
__global__ void __launch_bounds__(kBlock) walk_kernel(const Args p) {
  using L = Layout<RULE, N, DVC>;
  constexpr int MT = N / 64, NT = L::COLS / 8, NX = DVC / 8, KN = N / 16;      // MT: 16-row tiles of the state per warp
  extern __shared__ __align__(128) unsigned char sm[];
  Gates* gates = reinterpret_cast<Gates*>(sm + L::G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int slices = p.Dv / DVC, h = blockIdx.x / slices, col0 = blockIdx.x % slices * DVC, r = p.first + blockIdx.y;
  pdl_trigger();
  pdl_wait();
  const int t0 = p.q_start[r], t1 = p.q_start[r + 1];
  const bool fresh = p.req_start[r] == 0;
  float* slot = p.state + (size_t)p.slots[r] * p.slot_stride;
  const bf16* q = p.q + (size_t)(h / p.share) * N;
  const bf16* k = p.k + (size_t)(h / p.share) * N;
  const bf16* v = p.v + (size_t)h * p.Dv + col0;

  auto bring_rows = [&](unsigned char* to, int at, const bf16* from, int cols, int c0) {
    const int chunks = cols / 8;
    for (int x = tid; x < kPiece * chunks; x += kThreads) {
      const int i = x / chunks, c = x - i * chunks;
      const bool in = c0 + i < t1;
      copy16(to + i * at + c * 16, from + (size_t)(in ? c0 + i : t0) * p.ld + c * 8, in);
    }
  };
  auto bring = [&](int piece) {
    const int c0 = t0 + piece * kPiece;
    bring_rows(sm + L::K + (piece & 1) * kPiece * L::PN, L::PN, k, N, c0);
    bring_rows(sm + L::Q, L::PN, q, N, c0);
    bring_rows(sm + L::X + (piece & 1) * kPiece * L::PX, L::PX, v, DVC, c0);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  const int pieces = (t1 - t0 + kPiece - 1) / kPiece;
  const size_t splits = (size_t)(p.Dv / 64), at_n = (size_t)p.H * p.Dv * N + ((size_t)h * splits + col0 / 64) * N;
  const size_t at_m = (size_t)p.H * p.Dv * N + (size_t)p.H * splits * N + (size_t)h * splits + col0 / 64;
  if (warp == kGateWarp) {
    const float m0 = RULE == MLSTM && !fresh ? slot[at_m] : 0.f;
    if (RULE == MLSTM) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    float raw[4], m = m0;
    if (pieces > 0) raw_gates<RULE>(p, h, t0, t1, lane, raw);
    for (int piece = 0; piece < pieces; ++piece) {       // a piece's gates are made while the other warps walk the one before
      Gates& g = gates[piece & 1];
      const int c0 = t0 + piece * kPiece;
      make_gates<RULE>(p, h, min(kPiece, t1 - c0), lane, raw, m, g);
      if (piece + 1 < pieces) raw_gates<RULE>(p, h, c0 + kPiece, t1, lane, raw);
      __syncwarp();
      if (RULE == MLSTM) m = g.m;
      block_barrier();
    }
    if (RULE == MLSTM) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (pieces > 0 && lane == 0 && col0 % 64 == 0) slot[at_m] = m;
    }
    return;
  }

  // the state: rows (warp * MT + mt) * 16 + gq (+ 8), columns 8 nt + 2 tq (+ 1)
  float S[MT][NT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = (warp * MT + mt) * 16 + gq + (e >> 1) * 8, c = 8 * nt + 2 * tq + (e & 1);
        float x = 0.f;
        if (!fresh) {
          if (c < DVC) x = slot[((size_t)h * p.Dv + col0 + c) * N + n];
          else if (c == DVC) x = slot[at_n + n];
        }
        S[mt][nt][e] = x;
      }
  // MLSTM: the blocks of 64 value columns share n and m in the slot; nobody writes them before all have read
  if (RULE == MLSTM) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  auto put_state = [&]() {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t part[3];
          split3(part, S[mt][nt][2 * half], S[mt][nt][2 * half + 1]);
          unsigned char* to = sm + L::S + ((warp * MT + mt) * 16 + gq + 8 * half) * L::PC + (8 * nt + 2 * tq) * 2;
#pragma unroll
          for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(to + s * N * L::PC) = part[s];
        }
  };

  if (pieces > 0) bring(0);
  put_state();
  const int row = warp * 16 + gq;                        // this thread's tokens of a piece: row and row + 8
  for (int piece = 0; piece < pieces; ++piece) {
    const int c0 = t0 + piece * kPiece, b = piece & 1;
    const Gates& g = gates[b];
    const unsigned char* Ks = sm + L::K + b * kPiece * L::PN;
    const unsigned char* Xs = sm + L::X + b * kPiece * L::PX;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    block_barrier();                                     // rows, gates and the state's parts are there, the buffers before them free

    // weighed values, three parts each
    for (int x = tid; x < kPiece * NX; x += kThreads) {
      const int j = x / NX, c = x - j * NX;
      const uint4 in = *reinterpret_cast<const uint4*>(Xs + j * L::PX + c * 16);
      const uint32_t* w2 = reinterpret_cast<const uint32_t*>(&in);
      const float wj = g.weigh[j];
      uint4 out[3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t part[3];
        split3(part, __uint_as_float(w2[e] << 16) * wj, __uint_as_float(w2[e] & 0xffff0000u) * wj);
#pragma unroll
        for (int s = 0; s < 3; ++s) reinterpret_cast<uint32_t*>(&out[s])[e] = part[s];
      }
#pragma unroll
      for (int s = 0; s < 3; ++s) *reinterpret_cast<uint4*>(sm + L::W + (s * kPiece + j) * L::PC + c * 16) = out[s];
    }
    if (RULE == MLSTM && tid < kPiece) {
      uint32_t part[3];
      split3(part, g.weigh[tid], 0.f);
#pragma unroll
      for (int s = 0; s < 3; ++s)
        *reinterpret_cast<uint4*>(sm + L::W + (s * kPiece + tid) * L::PC + DVC * 2) = make_uint4(part[s], 0, 0, 0);
    }

    // q . k for the keys up to the warp's last token, and S^T q
    float G[8][4], acc[NT][4];
#pragma unroll
    for (int x = 0; x < 8; ++x) G[x][0] = G[x][1] = G[x][2] = G[x][3] = 0.f;
#pragma unroll
    for (int x = 0; x < NT; ++x) acc[x][0] = acc[x][1] = acc[x][2] = acc[x][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) {
      uint32_t a[4];
      ldm4(a, sm + L::Q + (warp * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
      for (int jt = 0; jt < 4; ++jt)
        if (jt <= warp) {
          uint32_t f[4];
          ldm4(f, Ks + (jt * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + (kk * 2 + (lane >> 3 & 1)) * 16);
          mma(G[2 * jt], a, f[0], f[1]);
          mma(G[2 * jt + 1], a, f[2], f[3]);
        }
#pragma unroll
      for (int s = 2; s >= 0; --s) {
        const unsigned char* Ss = sm + L::S + (s * N + kk * 16 + (lane & 15)) * L::PC;
#pragma unroll
        for (int nt = 0; nt + 1 < NT; nt += 2) {
          uint32_t f[4];
          ldm4t(f, Ss + (nt + (lane >> 4)) * 16);
          mma(acc[nt], a, f[0], f[1]);
          mma(acc[nt + 1], a, f[2], f[3]);
        }
        if (NT & 1) {
          uint32_t f[2];
          ldm2t(f, Ss + (NT - 1) * 16);
          mma(acc[NT - 1], a, f[0], f[1]);
        }
      }
    }
    walkers_barrier();                                   // the weighed values are there; q and the state's parts are free
    if (piece + 1 < pieces) bring(piece + 1);

    // the scores' weights, then their product with the values
    const float rh0 = g.row_hi[row], rl0 = g.row_lo[row], rh1 = g.row_hi[row + 8], rl1 = g.row_lo[row + 8];
    const float f0 = g.from[row], f1 = g.from[row + 8];
#pragma unroll
    for (int x = 0; x < NT; ++x) { acc[x][0] *= f0; acc[x][1] *= f0; acc[x][2] *= f1; acc[x][3] *= f1; }
#pragma unroll
    for (int jt = 0; jt < 4; ++jt)
      if (jt <= warp) {
        uint32_t part[3][4];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float* e = G[2 * jt + half];
          const int j = jt * 16 + half * 8 + 2 * tq;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float ch = g.col_hi[j + u], cl = g.col_lo[j + u], w = RULE == SSD ? g.aux[j + u] : 1.f;
            e[u] = j + u <= row ? e[u] * (expf((rh0 + ch) + (rl0 + cl)) * w) : 0.f;
            e[2 + u] = j + u <= row + 8 ? e[2 + u] * (expf((rh1 + ch) + (rl1 + cl)) * w) : 0.f;
          }
          uint32_t up[3], low[3];
          split3(up, e[0], e[1]);
          split3(low, e[2], e[3]);
#pragma unroll
          for (int s = 0; s < 3; ++s) { part[s][2 * half] = up[s]; part[s][2 * half + 1] = low[s]; }
        }
#pragma unroll
        for (int nt = 0; nt < NX; nt += 2) {
          uint32_t f[4];
          ldm4t(f, Xs + (jt * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
#pragma unroll
          for (int s = 2; s >= 0; --s) {
            mma(acc[nt], part[s], f[0], f[1]);
            mma(acc[nt + 1], part[s], f[2], f[3]);
          }
        }
        if (RULE == MLSTM) {
          const uint32_t ones = gq == 0 ? 0x3f803f80u : 0u;      // the column of ones
#pragma unroll
          for (int s = 2; s >= 0; --s) mma(acc[NT - 1], part[s], ones, ones);
        }
      }
    float den0 = 0.f, den1 = 0.f;
    if (RULE == MLSTM) {
      den0 = __shfl_sync(0xffffffffu, acc[NT - 1][0], lane & ~3);
      den1 = __shfl_sync(0xffffffffu, acc[NT - 1][2], lane & ~3);
      den0 = fmaxf(fabsf(den0 * p.q_scale), g.aux[row]) + 1e-6f;
      den1 = fmaxf(fabsf(den1 * p.q_scale), g.aux[row + 8]) + 1e-6f;
    }
    const float skip = RULE == SSD ? p.D[h] : 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = row + 8 * half;
      if (c0 + i < t1) {
        float* to = p.y + (size_t)(c0 + i) * p.H * p.Dv + (size_t)h * p.Dv + col0 + 2 * tq;
#pragma unroll
        for (int nt = 0; nt < NX; ++nt) {
          float2 o = make_float2(acc[nt][2 * half], acc[nt][2 * half + 1]);
          if (RULE == SSD) {
            const uint32_t x2 = *reinterpret_cast<const uint32_t*>(Xs + i * L::PX + (8 * nt + 2 * tq) * 2);
            o.x = fmaf(skip, __uint_as_float(x2 << 16), o.x);
            o.y = fmaf(skip, __uint_as_float(x2 & 0xffff0000u), o.y);
          } else {
            const float den = half ? den1 : den0;
            o.x = o.x * p.q_scale / den;
            o.y = o.y * p.q_scale / den;
          }
          *reinterpret_cast<float2*>(to + 8 * nt) = o;
        }
      }
    }

    // the state
    const float keep = g.keep;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[mt][nt][e] *= keep;
#pragma unroll
    for (int jj = 0; jj < kPiece / 16; ++jj) {
      uint32_t a[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
        ldm4t(a[mt], Ks + (jj * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + ((warp * MT + mt) * 2 + (lane >> 3 & 1)) * 16);
#pragma unroll
      for (int s = 2; s >= 0; --s) {
        const unsigned char* Ws = sm + L::W + (s * kPiece + jj * 16 + (lane & 15)) * L::PC;
#pragma unroll
        for (int nt = 0; nt + 1 < NT; nt += 2) {
          uint32_t f[4];
          ldm4t(f, Ws + (nt + (lane >> 4)) * 16);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            mma(S[mt][nt], a[mt], f[0], f[1]);
            mma(S[mt][nt + 1], a[mt], f[2], f[3]);
          }
        }
        if (NT & 1) {
          uint32_t f[2];
          ldm2t(f, Ws + (NT - 1) * 16);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) mma(S[mt][NT - 1], a[mt], f[0], f[1]);
        }
      }
    }
    if (piece + 1 < pieces) put_state();
  }
  if (RULE == MLSTM) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (pieces > 0) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int n = (warp * MT + mt) * 16 + gq + (e >> 1) * 8, c = 8 * nt + 2 * tq + (e & 1);
          if (c < DVC) slot[((size_t)h * p.Dv + col0 + c) * N + n] = S[mt][nt][e];
          else if (c == DVC && col0 % 64 == 0) slot[at_n + n] = S[mt][nt][e];
        }
  }
}

// Whether the walk takes these sizes and addresses: 64 or 128 state rows, whole blocks of 64 value columns, 16-byte rows.
static inline bool takes(int N, int Dv, const void* q, const void* k, const void* v, int ld) {
  return (N == 64 || N == 128) && Dv >= 64 && Dv % 64 == 0 && ld % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15) == 0;
}

template <int RULE, int N, int DVC>
static int launch(const Args& a, int R, cudaStream_t stream) {
  constexpr int smem = Layout<RULE, N, DVC>::bytes;
  cudaError_t e = cudaFuncSetAttribute(walk_kernel<RULE, N, DVC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.H * (a.Dv / DVC)), (unsigned)R);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (kvb_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (RULE == MLSTM) {                     // the blocks of 64 value columns of one head
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 64 / DVC;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  e = cudaLaunchKernelEx(&cfg, walk_kernel<RULE, N, DVC>, a);
  return e != cudaSuccess ? (int)e : kvb_launch_result();
}

// 32 value columns a block; 16 where that would leave SMs without one (a run's pieces follow one another, so that a block's time is
// the launch's time whatever its width).
template <int RULE, int N>
static int launch_width(const Args& a, int R, cudaStream_t stream) {
  if ((long long)a.H * (a.Dv / 32) * R * 8 < (long long)kvb_sm_count() * 7) return launch<RULE, N, 16>(a, R, stream);
  return launch<RULE, N, 32>(a, R, stream);
}

template <int RULE>
static int launch_any(const Args& a, int N, int R, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (R > 65535 || a.H < 1) return KVB_ERR_BAD_SIZE;
  return N == 64 ? launch_width<RULE, 64>(a, R, stream) : launch_width<RULE, 128>(a, R, stream);
}

}  // namespace walk
