// The matrix memories of chunk_walk.cuh with every product made for all pieces of all runs at once, in three launches.  What a piece of 64
// tokens adds to the state does not depend on the state, so the only thing that goes from piece to piece is S <- keep S + change:
//
//   1. changes   a block per (piece, head, 64 value columns): the piece's gates summed up and its change, sum_j w_j k_j v_j^T;
//   2. states    a thread per four numbers of a state goes through the run's pieces and leaves in each change's place the state
//                that the piece begins with;
//   3. results   a block per (piece, head, 64 value columns): y_i = P_i S^T q_i + sum_{j <= i} (q_i . k_j) (P_i / P_j) take_j v_j.
//
// The products are the walk's, operand for operand: bfloat16 ones as they came, float32 ones in three parts, sums over more than a
// block of 16 made from zero and added up by float32 instructions; values that are not finite are left out of them and make NaNs of
// their column from their token on.  MLSTM: weights in a change are seen from the piece's own largest gate, since the running maximum m is only
// known in the second launch, which scales the change by exp(own - max(own, m)) when it adds it.
//
// What bounds it: bytes between the launches (a state of 32 KB a piece and head at 128 x 64, written twice and read twice, mostly in L2)
// and latency: three blocks of nine warps an SM (72 registers; the results with two: 75 us instead of 62), where the walk has one block with a
// barrier a piece.  The gates are made once and left to the results (mlstm 31 -> 27 us).  32 heads of 64 x 64, 2048 tokens: changes 15, states
// 14, results 25 us, the walk in one launch 86.  64 heads of 128 x 64, runs of 1111 + 700 + 237 tokens: 35, 19, 62, the walk 121 (one run of 2048
// 115 / 182): there every head makes the scores of its group's keys and queries again, and the states' bytes count.
#pragma once

#include "chunk_walk.cuh"

namespace pieces {

using namespace walk;
using walk::Args;
using walk::Gates;

constexpr int kWorkers = 256, kAll = kWorkers + 32;        // eight warps for products, one for the gates
constexpr int kNever = kPiece;

__host__ __device__ constexpr int cols_of(int rule) { return 64 + (rule == MLSTM ? 1 : 0); }     // MLSTM: the vector n behind the values' columns

struct Scratch {
  // [unit][columns * N], unit = (piece * H + head) * splits + block of 64 columns: a piece's change, then the state it begins with.  In the order
  // in which the products' right operands hold it: 8 columns, 16 rows, lane (column lane / 4, rows 2 (lane % 4), + 1, + 8, + 9); the vector n as it is
  float* s;
  double2* sums;    // [piece * H + head]: the logarithm of the piece's decay; MLSTM: the largest gate seen from the piece's start
  float* m;         // [unit] MLSTM: the running maximum that the piece begins with
  unsigned char* gates;    // [piece * H + head] of gate_bytes: what the first launch's gates leave for the third
};

// SSD: the piece's gates.  MLSTM: a token's logarithms summed up, input gates seen from the piece's start and their running maxima, as doubles.
__host__ __device__ constexpr int gate_bytes(int rule) { return rule == SSD ? (int)sizeof(Gates) : 3 * kPiece * (int)sizeof(double); }
static_assert(sizeof(Gates) % 16 == 0, "copied in 16 bytes");

// Piece `at` of the step: its run, which of the run's pieces it is and the run's number of pieces; false: there are fewer.
__device__ __forceinline__ bool find_piece(const Args& p, int R, int at, int& r, int& local, int& n) {
  for (int i = 0; i < R; ++i) {
    n = (p.q_start[p.first + i + 1] - p.q_start[p.first + i] + kPiece - 1) / kPiece;
    if (at < n) {
      r = p.first + i;
      local = at;
      return true;
    }
    at -= n;
  }
  return false;
}

// 64 token rows from c0 on of `cols` columns, zero behind t1, by the block's workers
__device__ __forceinline__ void bring(unsigned char* to, int at, const bf16* from, int ld, int cols, int c0, int t1, int tid) {
  const int chunks = cols / 8;
  for (int x = tid; x < kPiece * chunks; x += kWorkers) {
    const int i = x / chunks, c = x - i * chunks;
    const bool in = c0 + i < t1;
    copy16(to + i * at + c * 16, from + (size_t)(in ? c0 + i : c0) * ld + c * 8, in);
  }
}

// The values that a thread brought: those that are not finite leave, the first such token of a column (and of any) is recorded.
__device__ __forceinline__ void look_at_values(unsigned char* Xs, int at, int* spoilt, int tid) {
  for (int x = tid; x < kPiece * 8; x += kWorkers) {
    const int j = x / 8, c = x - j * 8;
    uint4* where = reinterpret_cast<uint4*>(Xs + j * at + c * 16);
    const uint4 v = *where;
    if (not_finite(v.x) | not_finite(v.y) | not_finite(v.z) | not_finite(v.w)) {
      const uint32_t two[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (not_finite(two[e >> 1] >> 16 * (e & 1) & 0xffffu)) {
          atomicMin(spoilt + 1 + c * 8 + e, j);
          atomicMin(spoilt, j);
        }
      *where = make_uint4(finite_part(v.x), finite_part(v.y), finite_part(v.z), finite_part(v.w));
    }
  }
}

template <int RULE, int N>
struct ChangesLayout {
  static constexpr int PN = pitch(N), PX = pitch(64);
  static constexpr int K = 0;                                     // [64] rows of PN
  static constexpr int X = K + kPiece * PN;                       // [64] rows of PX
  static constexpr int W = X + kPiece * PX;                       // [3][64] rows of PX: weighed values
  static constexpr int G = W + 3 * kPiece * PX;                   // [64] weights
  static constexpr int V = G + kPiece * 4;                        // MLSTM: [256] parts of the vector's change
  static constexpr int F = V + (RULE == MLSTM ? kWorkers * 4 : 0);
  static constexpr int bytes = F + (1 + 64) * 4;
};

template <int RULE, int N>
__global__ void __launch_bounds__(kAll, 3) changes_kernel(const Args p, int R, const Scratch sc) {
  using L = ChangesLayout<RULE, N>;
  constexpr int COLS = cols_of(RULE), NT = N / 16;               // NT: 8-wide tiles of half the state's rows
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int splits = p.Dv / 64, h = blockIdx.x / splits, split = blockIdx.x - h * splits;
  int* spoilt = reinterpret_cast<int*>(sm + L::F);
  float* weigh = reinterpret_cast<float*>(sm + L::G);
  if (tid < 1 + 64) spoilt[tid] = kNever;
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  int r, local, n;
  if (!find_piece(p, R, blockIdx.y, r, local, n)) return;
  const int c0 = p.q_start[r] + local * kPiece, t1 = p.q_start[r + 1];
  const size_t unit = ((size_t)blockIdx.y * p.H + h) * splits + split;
  if (warp == 8) {
    float raw[4];
    raw_gates<RULE>(p, h, c0, t1, lane, raw);
    GateWarp<RULE> w;
    w.sums(p, h, min(kPiece, t1 - c0), lane, raw);
    const double c63 = __shfl_sync(0xffffffffu, w.c[1], 31);
    const double top = RULE == MLSTM ? __shfl_sync(0xffffffffu, w.top[1], 31) : 0.0;
#pragma unroll
    for (int u = 0; u < 2; ++u)
      weigh[lane + 32 * u] = RULE == SSD ? expf((float)(c63 - w.c[u])) * w.take[u] : expf((float)(w.a[u] - top));
    if (split == 0) {
      const size_t at = (size_t)blockIdx.y * p.H + h;
      if (lane == 0) sc.sums[at] = make_double2(c63, top);
      unsigned char* left = sc.gates + at * gate_bytes(RULE);
      if (RULE == SSD) {
        w.put(lane, 0.f, *reinterpret_cast<Gates*>(left));
      } else {
        double* to = reinterpret_cast<double*>(left) + lane;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          to[32 * u] = w.c[u];
          to[kPiece + 32 * u] = w.a[u];
          to[2 * kPiece + 32 * u] = w.top[u];
        }
      }
    }
  } else {
    bring(sm + L::K, L::PN, p.k + (size_t)(h / p.share) * N, p.ld, N, c0, t1, tid);
    bring(sm + L::X, L::PX, p.v + (size_t)h * p.Dv + split * 64, p.ld, 64, c0, t1, tid);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    look_at_values(sm + L::X, L::PX, spoilt, tid);
  }
  __syncthreads();
  if (warp < 8) {
    for (int x = tid; x < kPiece * 8; x += kWorkers) {             // weighed values, three parts each
      const int j = x / 8, c = x - j * 8;
      const uint4 in = *reinterpret_cast<const uint4*>(sm + L::X + j * L::PX + c * 16);
      const uint32_t* w2 = reinterpret_cast<const uint32_t*>(&in);
      const float wj = weigh[j];
      uint4 out[3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t part[3];
        split3(part, __uint_as_float(w2[e] << 16) * wj, __uint_as_float(w2[e] & 0xffff0000u) * wj);
#pragma unroll
        for (int u = 0; u < 3; ++u) reinterpret_cast<uint32_t*>(&out[u])[e] = part[u];
      }
#pragma unroll
      for (int u = 0; u < 3; ++u) *reinterpret_cast<uint4*>(sm + L::W + (u * kPiece + j) * L::PX + c * 16) = out[u];
    }
    if (RULE == MLSTM) {
      constexpr int kRuns = kWorkers / N, kTokens = kPiece / kRuns;
      const int i = tid % N, j0 = tid / N * kTokens;
      float sum = 0.f;
#pragma unroll 8
      for (int j = 0; j < kTokens; ++j)
        sum = fmaf(__bfloat162float(*reinterpret_cast<const bf16*>(sm + L::K + (j0 + j) * L::PN + i * 2)), weigh[j0 + j], sum);
      reinterpret_cast<float*>(sm + L::V)[tid] = sum;
    }
  }
  __syncthreads();
  if (warp == 8) return;
  float* to = sc.s + unit * COLS * N;
  // a warp's share: 16 columns, half the state's rows
  const int ct = warp >> 1, n0 = (warp & 1) * (N / 2);
  float d[NT][4];
#pragma unroll
  for (int x = 0; x < NT; ++x) d[x][0] = d[x][1] = d[x][2] = d[x][3] = 0.f;
#pragma unroll
  for (int jj = 0; jj < kPiece / 16; ++jj) {
    uint32_t a[3][4];
#pragma unroll
    for (int u = 0; u < 3; ++u)
      ldm4t(a[u], sm + L::W + (u * kPiece + jj * 16 + (lane & 7) + (lane >> 4) * 8) * L::PX + (ct * 2 + (lane >> 3 & 1)) * 16);
#pragma unroll
    for (int nt = 0; nt < NT; nt += 2) {
      uint32_t f[4];
      ldm4t(f, sm + L::K + (jj * 16 + (lane & 15)) * L::PN + (n0 / 8 + nt + (lane >> 4)) * 16);
      float t[2][4];
      mma0(t[0], a[2], f[0], f[1]);
      mma0(t[1], a[2], f[2], f[3]);
#pragma unroll
      for (int u = 1; u >= 0; --u) {
        mma(t[0], a[u], f[0], f[1]);
        mma(t[1], a[u], f[2], f[3]);
      }
      add4(d[nt], t[0]);
      add4(d[nt + 1], t[1]);
    }
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const bool bad = spoilt[1 + ct * 16 + gq + 8 * half] != kNever;
#pragma unroll
    for (int nt = 0; nt < NT; nt += 2)
      *reinterpret_cast<float4*>(to + (((2 * ct + half) * (N / 16) + (n0 / 8 + nt) / 2) * 32 + lane) * 4) =
          bad ? make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F)
              : make_float4(d[nt][2 * half], d[nt][2 * half + 1], d[nt + 1][2 * half], d[nt + 1][2 * half + 1]);
  }
  if (RULE == MLSTM && tid < N) {
    const float* part = reinterpret_cast<const float*>(sm + L::V) + tid;
    float sum = part[0];
#pragma unroll
    for (int x = 1; x < kWorkers / N; ++x) sum += part[x * N];
    to[64 * N + tid] = sum;
  }
}

// grid (columns * N / 4 / 256 rounded up, H * splits, R)
template <int RULE, int N>
__global__ void __launch_bounds__(256) states_kernel(const Args p, const Scratch sc) {
  constexpr int COLS = cols_of(RULE), AHEAD = 8;
  pdl_trigger();
  pdl_wait();
  const int splits = p.Dv / 64, h = blockIdx.y / splits, split = blockIdx.y - h * splits, r = p.first + blockIdx.z;
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (e >= COLS * N) return;
  int before = 0;
  for (int i = p.first; i < r; ++i) before += (p.q_start[i + 1] - p.q_start[i] + kPiece - 1) / kPiece;
  const int n = (p.q_start[r + 1] - p.q_start[r] + kPiece - 1) / kPiece;
  if (n == 0) return;
  const bool fresh = p.req_start[r] == 0;
  float* slot = p.state + (size_t)p.slots[r] * p.slot_stride;
  const size_t at_n = (size_t)p.H * p.Dv * N + ((size_t)h * splits + split) * N;
  const size_t at_m = (size_t)p.H * p.Dv * N + (size_t)p.H * splits * N + (size_t)h * splits + split;
  // where the four numbers lie in the slot (whose floats may start anywhere): two and two eight rows on, n's side by side
  const int of_lane = e / 4 & 31, kk = e / 128 % (N / 16), c = e / (8 * N) * 8 + (of_lane >> 2);
  const bool vector = e >= 64 * N;
  float* mine = slot + (vector ? at_n + (e - 64 * N) : ((size_t)h * p.Dv + split * 64 + c) * N + 16 * kk + 2 * (of_lane & 3));
  const int far = vector ? 2 : 8;
  float S[4];
#pragma unroll
  for (int x = 0; x < 4; ++x) S[x] = fresh ? 0.f : mine[(x & 1) + (x >> 1) * far];
  float m = RULE == MLSTM && !fresh ? slot[at_m] : 0.f;
  const size_t step = (size_t)p.H * splits * COLS * N;
  float* at = sc.s + (((size_t)before * p.H + h) * splits + split) * COLS * N + e;
  const double2* sums = sc.sums + (size_t)before * p.H + h;
  float* ms = sc.m + ((size_t)before * p.H + h) * splits + split;
  for (int s0 = 0; s0 < n; s0 += AHEAD) {
    float4 d[AHEAD];
    double2 g[AHEAD];
#pragma unroll
    for (int x = 0; x < AHEAD; ++x)
      if (s0 + x < n) {
        d[x] = *reinterpret_cast<const float4*>(at + (s0 + x) * step);
        g[x] = sums[(size_t)(s0 + x) * p.H];
      }
#pragma unroll
    for (int x = 0; x < AHEAD; ++x)
      if (s0 + x < n) {
        *reinterpret_cast<float4*>(at + (s0 + x) * step) = make_float4(S[0], S[1], S[2], S[3]);
        float keep;
        if (RULE == SSD) {
          keep = expf((float)g[x].x);
        } else {
          if (e == 0) ms[(size_t)(s0 + x) * p.H * splits] = m;
          const double top = fmax(g[x].y, (double)m);
          const float take = expf((float)(g[x].y - top));
          keep = expf((float)((double)m - top));
          m = (float)(g[x].x + top);
          d[x].x *= take; d[x].y *= take; d[x].z *= take; d[x].w *= take;
        }
        S[0] = fmaf(S[0], keep, d[x].x);
        S[1] = fmaf(S[1], keep, d[x].y);
        S[2] = fmaf(S[2], keep, d[x].z);
        S[3] = fmaf(S[3], keep, d[x].w);
      }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) mine[(x & 1) + (x >> 1) * far] = S[x];
}

template <int RULE, int N>
struct ResultsLayout {
  static constexpr int PN = pitch(N), PX = pitch(64);
  static constexpr int K = 0;                                     // [64] rows of PN
  static constexpr int Q = K + kPiece * PN;
  static constexpr int X = Q + kPiece * PN;                       // [64] rows of PX
  static constexpr int P = X + kPiece * PX;                       // [3][64] rows of PX: weighed scores, blocks on and below the diagonal
  static constexpr int G = P + 3 * kPiece * PX;                   // gates
  static constexpr int D = G + (int)sizeof(Gates);                // MLSTM: [3][64] the denominators' parts
  static constexpr int F = D + (RULE == MLSTM ? 3 * kPiece * 4 : 0);
  static constexpr int bytes = F + (1 + 64) * 4;
};

template <int RULE, int N>
__global__ void __launch_bounds__(kAll, 3) results_kernel(const Args p, int R, const Scratch sc) {
  using L = ResultsLayout<RULE, N>;
  constexpr int COLS = cols_of(RULE), KN = N / 16;
  extern __shared__ __align__(128) unsigned char sm[];
  Gates& g = *reinterpret_cast<Gates*>(sm + L::G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int splits = p.Dv / 64, h = blockIdx.x / splits, split = blockIdx.x - h * splits;
  int* spoilt = reinterpret_cast<int*>(sm + L::F);
  float* dens = reinterpret_cast<float*>(sm + L::D);
  if (tid < 1 + 64) spoilt[tid] = kNever;
  __syncthreads();
  pdl_trigger();
  pdl_wait();
  int r, local, n;
  if (!find_piece(p, R, blockIdx.y, r, local, n)) return;
  const int c0 = p.q_start[r] + local * kPiece, t1 = p.q_start[r + 1];
  const size_t unit = ((size_t)blockIdx.y * p.H + h) * splits + split;
  const float* from = sc.s + unit * COLS * N;
  // a warp's columns of the state as a right operand: column 8 warp + gq, rows 16 kk + 2 tq (+ 1, + 8, + 9)
  float4 S[KN];
  const unsigned char* left = sc.gates + ((size_t)blockIdx.y * p.H + h) * gate_bytes(RULE);
  if (warp == 8) {
    if (RULE == SSD) {
      for (int x = lane; x < (int)sizeof(Gates) / 16; x += 32) reinterpret_cast<uint4*>(&g)[x] = reinterpret_cast<const uint4*>(left)[x];
    } else {
      GateWarp<RULE> w;
      const double* of = reinterpret_cast<const double*>(left) + lane;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        w.c[u] = of[32 * u];
        w.a[u] = of[kPiece + 32 * u];
        w.top[u] = of[2 * kPiece + 32 * u];
      }
      w.put(lane, sc.m[unit], g);
    }
    if (RULE == MLSTM && lane == 0 && local == n - 1)
      p.state[(size_t)p.slots[r] * p.slot_stride + (size_t)p.H * p.Dv * N + (size_t)p.H * splits * N + (size_t)h * splits + split] = g.m;
  } else {
    bring(sm + L::K, L::PN, p.k + (size_t)(h / p.share) * N, p.ld, N, c0, t1, tid);
    bring(sm + L::Q, L::PN, p.q + (size_t)(h / p.share) * N, p.ld, N, c0, t1, tid);
    bring(sm + L::X, L::PX, p.v + (size_t)h * p.Dv + split * 64, p.ld, 64, c0, t1, tid);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) S[kk] = *reinterpret_cast<const float4*>(from + ((warp * KN + kk) * 32 + lane) * 4);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    look_at_values(sm + L::X, L::PX, spoilt, tid);
  }
  __syncthreads();
  if (warp < 8) {
    // Scores, two warps to a block of 16 rows: of the blocks of 16 keys up to the rows' own, low .. high - 1
    const int hw = warp >> 1, second = warp & 1, row = hw * 16 + gq;
    const int low = second ? (hw + 2) / 2 : 0, high = second ? hw + 1 : (hw + 2) / 2;
    float G[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) G[x][0] = G[x][1] = G[x][2] = G[x][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) {
      uint32_t a[4];
      ldm4(a, sm + L::Q + (hw * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
        if (low + jj < high) {
          uint32_t f[4];
          ldm4(f, sm + L::K + ((low + jj) * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + (kk * 2 + (lane >> 3 & 1)) * 16);
          float t[2][4];
          mma0(t[0], a, f[0], f[1]);
          mma0(t[1], a, f[2], f[3]);
          add4(G[2 * jj], t[0]);
          add4(G[2 * jj + 1], t[1]);
        }
    }
    const float rh0 = g.row_hi[row], rl0 = g.row_lo[row], rh1 = g.row_hi[row + 8], rl1 = g.row_lo[row + 8];
    const float r0 = g.rows[row], r1 = g.rows[row + 8];
    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
    for (int jj = 0; jj < 2; ++jj)
      if (low + jj < high) {
        const int jt = low + jj;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float* e = G[2 * jj + half];
          const int j = jt * 16 + half * 8 + 2 * tq;
          if (jt < hw) {
            const float2 w = *reinterpret_cast<const float2*>(g.cols + 8 * hw * (hw - 1) + j);
            e[0] *= r0 * w.x;
            e[1] *= r0 * w.y;
            e[2] *= r1 * w.x;
            e[3] *= r1 * w.y;
          } else {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const float ch = g.col_hi[j + u], cl = g.col_lo[j + u], w = RULE == SSD ? g.aux[j + u] : 1.f;
              e[u] = j + u <= row ? e[u] * (expf((rh0 + ch) + (rl0 + cl)) * w) : 0.f;
              e[2 + u] = j + u <= row + 8 ? e[2 + u] * (expf((rh1 + ch) + (rl1 + cl)) * w) : 0.f;
            }
          }
          if (RULE == MLSTM) {
            sum0 += e[0] + e[1];
            sum1 += e[2] + e[3];
          }
          uint32_t up[3], down[3];
          split3(up, e[0], e[1]);
          split3(down, e[2], e[3]);
#pragma unroll
          for (int u = 0; u < 3; ++u) {
            unsigned char* to = sm + L::P + (u * kPiece + row) * L::PX + j * 2;
            *reinterpret_cast<uint32_t*>(to) = up[u];
            *reinterpret_cast<uint32_t*>(to + 8 * L::PX) = down[u];
          }
        }
      }
    if (RULE == MLSTM) {                                 // the weighed scores' sums, and n . q, a quarter of the rows a thread
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        sum0 += __shfl_xor_sync(0xffffffffu, sum0, o);
        sum1 += __shfl_xor_sync(0xffffffffu, sum1, o);
      }
      if (tq == 0) {
        dens[second * kPiece + row] = sum0;
        dens[second * kPiece + row + 8] = sum1;
      }
      const int i = tid >> 2;
      float sum = 0.f;
#pragma unroll
      for (int x = 0; x < N / 32; ++x) {                 // chunks of eight rows: tid & 3, + 4, ..
        const int at = (x * 4 + (tid & 3)) * 8;
        const uint4 qs = *reinterpret_cast<const uint4*>(sm + L::Q + i * L::PN + at * 2);
        const float4 n0 = *reinterpret_cast<const float4*>(from + 64 * N + at), n1 = *reinterpret_cast<const float4*>(from + 64 * N + at + 4);
        const uint32_t* two = reinterpret_cast<const uint32_t*>(&qs);
        const float ns[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          sum = fmaf(__uint_as_float(two[y] << 16), ns[2 * y], sum);
          sum = fmaf(__uint_as_float(two[y] & 0xffff0000u), ns[2 * y + 1], sum);
        }
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if ((tid & 3) == 0) dens[2 * kPiece + i] = sum;
    }
  }
  __syncthreads();
  if (warp == 8) return;

  // a warp's eight columns of all 64 rows; S^T q first, 16 rows of the state after 16
  float accs[4][4];
#pragma unroll
  for (int rt = 0; rt < 4; ++rt) accs[rt][0] = accs[rt][1] = accs[rt][2] = accs[rt][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < KN; ++kk) {
    uint32_t b[2][3];
    split3(b[0], S[kk].x, S[kk].y);
    split3(b[1], S[kk].z, S[kk].w);
#pragma unroll
    for (int rt = 0; rt < 4; ++rt) {
      uint32_t a[4];
      ldm4(a, sm + L::Q + (rt * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
      float t[4];
      mma0(t, a, b[0][2], b[1][2]);
      mma(t, a, b[0][1], b[1][1]);
      mma(t, a, b[0][0], b[1][0]);
      add4(accs[rt], t);
    }
  }
  uint32_t v[4][2];
#pragma unroll
  for (int jt = 0; jt < 4; ++jt) ldm2t(v[jt], sm + L::X + (jt * 16 + (lane & 15)) * L::PX + warp * 16);
  const float skip = RULE == SSD ? p.D[h] : 0.f;
  const int col = 8 * warp + 2 * tq;
#pragma unroll
  for (int rt = 0; rt < 4; ++rt) {
    const float* acc = accs[rt];
    float own[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int jt = 0; jt <= rt; ++jt) {
      float t[4];
#pragma unroll
      for (int u = 2; u >= 0; --u) {
        uint32_t a[4];
        ldm4(a, sm + L::P + (u * kPiece + rt * 16 + (lane & 15)) * L::PX + (jt * 2 + (lane >> 4)) * 16);
        if (u == 2) mma0(t, a, v[jt][0], v[jt][1]);
        else mma(t, a, v[jt][0], v[jt][1]);
      }
      add4(own, t);
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = rt * 16 + gq + 8 * half;
      if (c0 + i >= t1) continue;
      const float f = g.from[i];
      float2 o = make_float2(fmaf(f, acc[2 * half], own[2 * half]), fmaf(f, acc[2 * half + 1], own[2 * half + 1]));
      if (RULE == SSD) {
        const uint32_t x2 = *reinterpret_cast<const uint32_t*>(sm + L::X + i * L::PX + col * 2);
        o.x = fmaf(skip, __uint_as_float(x2 << 16), o.x);
        o.y = fmaf(skip, __uint_as_float(x2 & 0xffff0000u), o.y);
      } else {
        float den = fmaf(f, dens[2 * kPiece + i], dens[i] + dens[kPiece + i]);
        den = fmaxf(fabsf(den * p.q_scale), g.aux[i]) + 1e-6f;
        o.x = o.x * p.q_scale / den;
        o.y = o.y * p.q_scale / den;
      }
      if (spoilt[1 + col] <= i) o.x = CUDART_NAN_F;
      if (spoilt[2 + col] <= i) o.y = CUDART_NAN_F;
      *reinterpret_cast<float2*>(p.y + (size_t)(c0 + i) * p.H * p.Dv + (size_t)h * p.Dv + split * 64 + col) = o;
    }
  }
}

// Bytes of scratch for runs of `tokens` in all, R of them: at most tokens / 64 + R pieces.
static long long scratch_bytes(int rule, long long tokens, int R, int H, int N, int Dv) {
  const long long pieces = tokens / kPiece + R;
  return pieces * H * ((Dv / 64) * (4ll * cols_of(rule) * N + 4) + (long long)sizeof(double2) + gate_bytes(rule)) + 64;
}

template <int RULE, int N>
static int launch_sized(const Args& a, int R, long long tokens, void* scratch, cudaStream_t stream) {
  const long long count = tokens / kPiece + R;
  const int splits = a.Dv / 64;
  if (count > 65535 || (long long)a.H * splits > 65535 || R > 65535) return KVB_ERR_BAD_SIZE;
  Scratch sc;
  sc.s = static_cast<float*>(scratch);
  sc.sums = reinterpret_cast<double2*>(sc.s + count * a.H * splits * cols_of(RULE) * N);
  sc.gates = reinterpret_cast<unsigned char*>(sc.sums + count * a.H);
  sc.m = reinterpret_cast<float*>(sc.gates + count * a.H * gate_bytes(RULE));
  const dim3 grid((unsigned)(a.H * splits), (unsigned)count);
  static OncePerDevice sized;
  cudaError_t e = sized(kvb_device(), [] {
    const cudaError_t first = cudaFuncSetAttribute(changes_kernel<RULE, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChangesLayout<RULE, N>::bytes);
    if (first != cudaSuccess) return first;
    return cudaFuncSetAttribute(results_kernel<RULE, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, ResultsLayout<RULE, N>::bytes);
  });
  if (e == cudaSuccess) e = kvb_launch(changes_kernel<RULE, N>, grid, dim3(kAll), ChangesLayout<RULE, N>::bytes, stream, a, R, sc);
  if (e == cudaSuccess)
    e = kvb_launch(states_kernel<RULE, N>, dim3((unsigned)((cols_of(RULE) * N / 4 + 255) / 256), (unsigned)(a.H * splits), (unsigned)R),
                   dim3(256), 0, stream, a, sc);
  if (e == cudaSuccess) e = kvb_launch(results_kernel<RULE, N>, grid, dim3(kAll), ResultsLayout<RULE, N>::bytes, stream, a, R, sc);
  return e == cudaSuccess ? kvb_launch_result() : (int)e;
}

// a.first .. a.first + R - 1: runs of `tokens` in all at most.  Sizes and addresses as the walk takes them; scratch on a 16-byte boundary.
template <int RULE>
static int launch(const Args& a, int N, int R, long long tokens, void* scratch, long long bytes, cudaStream_t stream) {
  if (R <= 0 || tokens <= 0) return 0;
  if (a.H < 1 || (reinterpret_cast<uintptr_t>(scratch) & 15) || scratch_bytes(RULE, tokens, R, a.H, N, a.Dv) > bytes) return KVB_ERR_BAD_SIZE;
  return N == 64 ? launch_sized<RULE, 64>(a, R, tokens, scratch, stream) : launch_sized<RULE, 128>(a, R, tokens, scratch, stream);
}

}  // namespace pieces
