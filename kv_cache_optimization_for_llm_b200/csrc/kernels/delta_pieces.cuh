// The gated delta rule of delta_walk.cuh with all that does not wait for the state made for every piece of every run at once, in three
// launches.  With the inverse T of a piece's I + A (see there), its corrections are
//
//   U = T R = U0 - W S,    U0 = T (beta v),    W = T (beta P k / |k|)
//
// so a walk over the pieces has two products left, U and the state's change:
//
//   1. prepare   a block per (piece, head): gates, key norms, A, its inverse, W (three bfloat16 parts) and U0;
//   2. chain     a block per (run, head, 16 or 32 value columns) walks the pieces: U = U0 - W S, S <- P_63 S + sum_j (P_63 / P_j) k_j u_j^T;
//                it leaves U and the state that every piece begins with;
//   3. results   a block per (piece, head, 32 columns): o_i = P_i S^T q_i + sum_{j <= i} (P_i / P_j) (q_i . k_j) u_j.
//
// The products are those of the walk, operand for operand: bfloat16 ones as they came, float32 ones in three parts, sums over more than a
// block of 16 added up by float32 instructions.  What is not finite is left out of them in the same way (first tokens of a piece whose
// key, gate or value is not finite are recorded, and results from such a token on, and the state, become NaNs at the end).
//
// What bounds it: the chain takes about 4300 cycles a piece of 32 columns (two barriers, and between them every warp's loads from shared
// memory, then every warp's products); the other two are latency, four blocks an SM.  32 heads of 64 x 64, runs of 1548 + 500 tokens: prepare
// 46, chain 56, results 31 us, the walk in one launch 206.  (A chain without barriers, a warp for 16 columns of the transposed state as a
// left operand in registers: 70 us, since one warp issues a product in 18 cycles however many are independent.)
#pragma once

#include "delta_walk.cuh"

namespace delta_pieces {

using namespace delta_walk;
using delta_walk::Args;
using delta_walk::Gates;

constexpr int kN = 64;                       // key size
constexpr int kNoToken = kPiece;             // "none" among a piece's tokens

struct Scratch {
  bf16* w;          // [unit][3][64][64], unit = piece * H + head, pieces counted over the runs
  float* u;         // [unit][64][Dv]: U0, then U
  float* s;         // [unit][64][Dv]: the state a piece begins with
  Gates* gates;     // [unit]
  int* spoilt;      // [unit][1 + Dv]: first token whose key or gates, whose value in that column, is not finite
};

// Piece `at` of the step: its run and which of the run's pieces it is; false: there are fewer.
__device__ __forceinline__ bool find_piece(const Args& p, int R, int at, int& r, int& local) {
  for (int i = 0; i < R; ++i) {
    const int n = (p.q_start[p.first + i + 1] - p.q_start[p.first + i] + kPiece - 1) / kPiece;
    if (at < n) {
      r = p.first + i;
      local = at;
      return true;
    }
    at -= n;
  }
  return false;
}
__device__ __forceinline__ int pieces_before(const Args& p, int r) {
  int n = 0;
  for (int i = p.first; i < r; ++i) n += (p.q_start[i + 1] - p.q_start[i] + kPiece - 1) / kPiece;
  return n;
}

struct PrepareLayout {
  // Four blocks an SM: of T and A the 16 x 16 blocks on and below the diagonal only, and the values wait in registers until A is done
  // with.  A block's rows are 48 bytes apart, so that eight of them lie in different banks.
  static constexpr int PN = pitch(kN), PT = pitch(kPiece), PB = 48, PD = 20, PV = pitch(64);
  static constexpr int BLOCK = 16 * PB;
  static constexpr int K = 0;                                     // [64] rows of PN
  static constexpr int T = K + kPiece * PN;                       // [3][10] blocks: the inverse, block (I, J) at I (I + 1) / 2 + J
  static constexpr int A = T + 3 * 10 * BLOCK;                    // [3][6] blocks: A below its diagonal blocks, (I, J) at I (I - 1) / 2 + J
  static constexpr int V = A;                                     // behind A: [64] rows of PV
  static constexpr int W = T;                                     // behind all of these: [3][64] rows of PT
  static constexpr int D = A + 3 * 6 * BLOCK;                     // [4][16] columns of PD floats
  static_assert(kPiece * PV <= 3 * 6 * BLOCK && 3 * kPiece * PT <= 3 * 16 * BLOCK, "what comes later fits what was there");
  static constexpr int G = D + 4 * 16 * PD * 4;
  static constexpr int F = G + (int)sizeof(Gates);                // [1 + Dv]
  static constexpr int bytes = F + (1 + 64) * 4;
};

__global__ void __launch_bounds__(kWalkers + 32) prepare_kernel(const Args p, int R, const Scratch sc) {
  using L = PrepareLayout;
  constexpr int KN = kN / 16;
  extern __shared__ __align__(128) unsigned char sm[];
  Gates& g = *reinterpret_cast<Gates*>(sm + L::G);
  int* spoilt = reinterpret_cast<int*>(sm + L::F);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int h = blockIdx.x;
  pdl_trigger();
  pdl_wait();
  int r, local;
  if (!find_piece(p, R, blockIdx.y, r, local)) return;
  const size_t unit = (size_t)blockIdx.y * p.H + h;
  const int c0 = p.q_start[r] + local * kPiece, t1 = p.q_start[r + 1];
  for (int i = tid; i < 1 + p.Dv; i += kWalkers + 32) spoilt[i] = kNoToken;
  unsigned char* Ks = sm + L::K;
  unsigned char* Ts = sm + L::T;
  bar<3, kWalkers + 32>();                         // `spoilt` is set up
  if (warp == 4) {
    // gates (as in the walk)
    const float rate = expf(p.head_rate[h]), dbias = p.decay_bias[h];
    double c[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u, t = c0 + i;
      float la = 0.f, be = 0.f;
      if (t < t1) {
        la = -(rate * softplus20(__bfloat162float(p.decay[(size_t)t * p.ld_decay + h]) + dbias));
        la = la < -200.f ? -200.f : la;
        be = sigmoid(__bfloat162float(p.beta[(size_t)t * p.ld_beta + h]));
        if (isnan(la + be)) {
          atomicMin(spoilt, i);
          la = be = 0.f;
        }
      }
      g.beta[i] = be;
      c[u] = scan_sum((double)la, lane);
    }
    c[1] += __shfl_sync(0xffffffffu, c[0], 31);
    const double total = __shfl_sync(0xffffffffu, c[1], 31), c15 = __shfl_sync(0xffffffffu, c[0], 15);
    const double c31 = __shfl_sync(0xffffffffu, c[0], 31), c47 = __shfl_sync(0xffffffffu, c[1], 15);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = lane + 32 * u;
      as_pair(c[u], g.hi[i], g.lo[i]);
      g.from[i] = expf((float)c[u]);
      g.weigh[i] = expf((float)(total - c[u]));
      g.rows[i] = expf((float)(c[u] - (u ? (lane < 16 ? c31 : c47) : c15)));
    }
    if (lane < 16) {
      g.cols[lane] = expf((float)(c15 - c[0]));
      g.cols[80 + lane] = expf((float)(c47 - c[1]));
    }
    g.cols[16 + lane] = expf((float)(c31 - c[0]));
    g.cols[48 + lane] = expf((float)(c47 - c[0]));
    if (lane == 0) g.keep = expf((float)total);
    bar<3, kWalkers + 32>();                       // the gates are there
    return;
  }
  const int ht = tid, hw = warp;
  uint4 values[4];
  {
    const bf16* k = p.k + (size_t)(h / p.share) * kN;
    const bf16* v = p.v + (size_t)h * p.Dv;
    const int chunks = kN / 8;
    for (int x = ht; x < kPiece * chunks; x += kWalkers) {
      const int i = x / chunks, c = x - i * chunks;
      const bool in = c0 + i < t1;
      copy16(Ks + i * L::PN + c * 16, k + (size_t)(in ? c0 + i : c0) * p.ld_k + c * 8, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // two threads a row of values: this one's chunks 4 (ht & 1) ..
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int i = ht >> 1, at = (ht & 1) * 4 + c;
      values[c] = make_uint4(0u, 0u, 0u, 0u);
      if (c0 + i < t1 && at * 8 < p.Dv) values[c] = *reinterpret_cast<const uint4*>(v + (size_t)(c0 + i) * p.ld_v + at * 8);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  bar<3, kWalkers + 32>();
  // norms of the keys, values that are not finite: two threads a row
  if (ht < 64) {
    unsigned char* from = Ks + ht * L::PN;
    float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < kN / 8; ++c) {
      const uint4 u = *reinterpret_cast<const uint4*>(from + c * 16);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = __uint_as_float(w[e] << 16), y = __uint_as_float(w[e] & 0xffff0000u);
        ss[e] = fmaf(x, x, ss[e]);
        ss[e] = fmaf(y, y, ss[e]);
      }
    }
    float sum = (ss[0] + ss[1]) + (ss[2] + ss[3]);
    if (!isfinite(sum)) {
      uint32_t bad = 0u;
      for (int c = 0; c < kN / 2; ++c) bad |= not_finite(reinterpret_cast<const uint32_t*>(from)[c]);
      if (bad) atomicMin(spoilt, ht);
      for (int c = 0; c < kN / 8; ++c) reinterpret_cast<uint4*>(from)[c] = make_uint4(0u, 0u, 0u, 0u);
      sum = CUDART_INF_F;
    }
    const float inv = 1.0f / sqrtf(sum + 1e-6f);
    g.kinv[ht] = inv;
    g.weigh[ht] *= inv;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t* w = reinterpret_cast<uint32_t*>(values + c);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t bad = not_finite(w[e]);
      if (bad) {
        const int at = 1 + ((ht & 1) * 4 + c) * 8 + 2 * e;
        if (bad & 0x8000u) atomicMin(spoilt + at, ht >> 1);
        if (bad & 0x80000000u) atomicMin(spoilt + at + 1, ht >> 1);
        w[e] = finite_part(w[e]);
      }
    }
  }
  bar<2, kWalkers>();
  float* Dg = reinterpret_cast<float*>(sm + L::D) + hw * 16 * L::PD;
  {                                                // rows 16 hw .. of A (as in the walk)
    float G[8][4];
#pragma unroll
    for (int x = 0; x < 8; ++x) G[x][0] = G[x][1] = G[x][2] = G[x][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) {
      uint32_t a[4];
      ldm4(a, Ks + (hw * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
      for (int jt = 0; jt < 4; ++jt)
        if (jt <= hw) {
          uint32_t f[4];
          ldm4(f, Ks + (jt * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + (kk * 2 + (lane >> 3 & 1)) * 16);
          float t[2][4];
          mma0(t[0], a, f[0], f[1]);
          mma0(t[1], a, f[2], f[3]);
          add4(G[2 * jt], t[0]);
          add4(G[2 * jt + 1], t[1]);
        }
    }
    const int row = hw * 16 + gq;
    const float h0 = g.hi[row], l0 = g.lo[row], h1 = g.hi[row + 8], l1 = g.lo[row + 8];
    const float w0 = g.beta[row] * g.kinv[row], w1 = g.beta[row + 8] * g.kinv[row + 8];
    const float r0 = w0 * g.rows[row], r1 = w1 * g.rows[row + 8];
#pragma unroll
    for (int x = 0; x < 8; ++x)
      if (x / 2 <= hw) {
        const int j = x * 8 + 2 * tq;
        if (x / 2 < hw) {
          const float2 f = *reinterpret_cast<const float2*>(g.cols + 8 * hw * (hw - 1) + j);
          const float cc0 = f.x * g.kinv[j], cc1 = f.y * g.kinv[j + 1];
          G[x][0] *= r0 * cc0;
          G[x][1] *= r0 * cc1;
          G[x][2] *= r1 * cc0;
          G[x][3] *= r1 * cc1;
          uint32_t up[3], low[3];
          split3(up, G[x][0], G[x][1]);
          split3(low, G[x][2], G[x][3]);
          unsigned char* to = sm + L::A + (hw * (hw - 1) / 2 + x / 2) * L::BLOCK + gq * L::PB + (j & 15) * 2;
#pragma unroll
          for (int u = 0; u < 3; ++u) {
            *reinterpret_cast<uint32_t*>(to + u * 6 * L::BLOCK) = up[u];
            *reinterpret_cast<uint32_t*>(to + u * 6 * L::BLOCK + 8 * L::PB) = low[u];
          }
        } else {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float ch = g.hi[j + u], cl = g.lo[j + u], w = g.kinv[j + u];
            G[x][u] *= w0 * w * expf((h0 - ch) + (l0 - cl));
            G[x][2 + u] *= w1 * w * expf((h1 - ch) + (l1 - cl));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = gq + (e >> 1) * 8, c = (j & 15) + (e & 1);
            Dg[c * L::PD + (i & 1) * 8 + (i >> 1)] = c < i ? G[x][e] : 0.f;
          }
        }
      }
  }
  __syncwarp();
  {                                                // the diagonal block's inverse (as in the walk)
    const int par = lane & 1, odd = lane >> 1 & 1;
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = 2 * e + par == (lane >> 1) ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 15; ++j) {
      const float u = __shfl_sync(0xffffffffu, x[j >> 1], (lane & ~1) | (j & 1));
      const float4* column = reinterpret_cast<const float4*>(Dg + j * L::PD + par * 8);
#pragma unroll
      for (int e = (j >> 1) & ~3; e < 8; e += 4) {
        const float4 a = column[e >> 2];
        x[e] = fmaf(-a.x, u, x[e]);
        x[e + 1] = fmaf(-a.y, u, x[e + 1]);
        x[e + 2] = fmaf(-a.z, u, x[e + 2]);
        x[e + 3] = fmaf(-a.w, u, x[e + 3]);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, odd ? x[e] : x[e + 1], 2);
      const float mine = odd ? x[e + 1] : x[e];
      uint32_t part[3];
      split3(part, odd ? other : mine, odd ? mine : other);
#pragma unroll
      for (int u = 0; u < 3; ++u)
        *reinterpret_cast<uint32_t*>(Ts + (u * 10 + hw * (hw + 3) / 2) * L::BLOCK + (2 * (e + odd) + par) * L::PB + (lane >> 1 & ~1) * 2) = part[u];
    }
  }
  bar<2, kWalkers>();
  {                                                // the blocks below it (as in the walk)
    auto mma6t = [&](float (*acc)[4], const uint32_t (*left)[4], const unsigned char* from, int part) {
      uint32_t f[3][4];
#pragma unroll
      for (int u = 0; u < 3; ++u) ldm4(f[u], from + u * part + ((lane & 7) + (lane >> 4) * 8) * L::PB + (lane >> 3 & 1) * 16);
      float t[2][4];
      mma0(t[0], left[2], f[0][0], f[0][1]);
      mma0(t[1], left[2], f[0][2], f[0][3]);
#pragma unroll
      for (int x = 1; x < 6; ++x) {
        const int o = x < 3 ? 2 : x < 5 ? 1 : 0, u = x < 3 ? x : x < 5 ? x - 3 : 0;
        mma(t[0], left[o - u], f[u][0], f[u][1]);
        mma(t[1], left[o - u], f[u][2], f[u][3]);
      }
      add4(acc[0], t[0]);
      add4(acc[1], t[1]);
    };
    uint32_t left[3][3][4];
#pragma unroll
    for (int u = 0; u < 3; ++u)
      ldm4t(left[0][u], Ts + (u * 10 + hw * (hw + 3) / 2) * L::BLOCK + ((lane & 7) + (lane >> 4) * 8) * L::PB + (lane >> 3 & 1) * 16);
#pragma unroll
    for (int d = 1; d < 4; ++d)
      if (hw + d < 4) {
        const int I = hw + d;
        float X[2][4] = {}, Y[2][4] = {};
#pragma unroll
        for (int e = 0; e < d; ++e) mma6t(X, left[e], sm + L::A + (I * (I - 1) / 2 + hw + e) * L::BLOCK, 6 * L::BLOCK);
        uint32_t x[3][4], y[3][4];
        left_parts(x, X, 1.f);
        mma6t(Y, x, Ts + I * (I + 3) / 2 * L::BLOCK, 10 * L::BLOCK);
        left_parts(y, Y, -1.f);
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          stm4t(y[u], Ts + (u * 10 + I * (I + 1) / 2 + hw) * L::BLOCK + ((lane & 7) + (lane >> 4) * 8) * L::PB + (lane >> 3 & 1) * 16);
          if (d < 3)
#pragma unroll
            for (int e = 0; e < 4; ++e) left[d][u][e] = y[u][e];
        }
      }
  }
  bar<2, kWalkers>();                              // T is whole, A is done with
#pragma unroll
  for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(sm + L::V + (ht >> 1) * L::PV + ((ht & 1) * 4 + c) * 16) = values[c];
  bar<2, kWalkers>();
  // Row blocks 0 and 3 hold five blocks of T between them, 1 and 2 as well: warp w takes the rows of block w for the even pairs of
  // columns and of block 3 - w for the odd ones.
  auto scaled = [&](uint32_t (*a)[4], int rb, int jt, bool keys) {      // block (rb, jt) of T, column j times beta_j (and P_j / |k_j|)
    uint32_t b[3][4];
#pragma unroll
    for (int u = 0; u < 3; ++u) ldm4(b[u], Ts + (u * 10 + rb * (rb + 1) / 2 + jt) * L::BLOCK + (lane & 15) * L::PB + (lane >> 4) * 16);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = jt * 16 + (e >> 1) * 8 + 2 * tq;
      float f0 = g.beta[j], f1 = g.beta[j + 1];
      if (keys) { f0 *= g.from[j] * g.kinv[j]; f1 *= g.from[j + 1] * g.kinv[j + 1]; }
      const float x = (__uint_as_float(b[0][e] << 16) + __uint_as_float(b[1][e] << 16)) + __uint_as_float(b[2][e] << 16);
      const float y = (__uint_as_float(b[0][e] & 0xffff0000u) + __uint_as_float(b[1][e] & 0xffff0000u)) + __uint_as_float(b[2][e] & 0xffff0000u);
      uint32_t part[3];
      split3(part, x * f0, y * f1);
#pragma unroll
      for (int u = 0; u < 3; ++u) a[u][e] = part[u];
    }
  };
  float W[2][2][2][4];                             // [turn][pair of 16 columns][8 columns]
#pragma unroll
  for (int turn = 0; turn < 2; ++turn) {
    const int rb = turn ? 3 - hw : hw;
    const int row = rb * 16 + gq;
    float (*acc)[2][4] = W[turn];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) acc[x][y][0] = acc[x][y][1] = acc[x][y][2] = acc[x][y][3] = 0.f;
    for (int jt = 0; jt <= rb; ++jt) {
      uint32_t a[3][4];
      scaled(a, rb, jt, true);
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int np = 2 * x + turn;
        uint32_t f[4];
        ldm4t(f, Ks + (jt * 16 + (lane & 15)) * L::PN + (np * 2 + (lane >> 4)) * 16);
        float t[2][4];
        mma0(t[0], a[2], f[0], f[1]);
        mma0(t[1], a[2], f[2], f[3]);
        mma(t[0], a[1], f[0], f[1]);
        mma(t[1], a[1], f[2], f[3]);
        mma(t[0], a[0], f[0], f[1]);
        mma(t[1], a[0], f[2], f[3]);
        add4(acc[x][0], t[0]);
        add4(acc[x][1], t[1]);
      }
    }
    // U0, two times 16 columns
    float d[2][2][4] = {};
    for (int jt = 0; jt <= rb; ++jt) {
      uint32_t a[3][4];
      scaled(a, rb, jt, false);
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (turn + 2 * x < p.Dv / 16) {
          uint32_t f[4];
          ldm4t(f, sm + L::V + (jt * 16 + (lane & 15)) * L::PV + ((turn + 2 * x) * 2 + (lane >> 4)) * 16);
          float t[2][4];
          mma0(t[0], a[2], f[0], f[1]);
          mma0(t[1], a[2], f[2], f[3]);
          mma(t[0], a[1], f[0], f[1]);
          mma(t[1], a[1], f[2], f[3]);
          mma(t[0], a[0], f[0], f[1]);
          mma(t[1], a[0], f[2], f[3]);
          add4(d[x][0], t[0]);
          add4(d[x][1], t[1]);
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
      if (turn + 2 * x < p.Dv / 16) {
        float* to = sc.u + (unit * kPiece + row) * p.Dv + (turn + 2 * x) * 16 + 2 * tq;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          *reinterpret_cast<float2*>(to + 8 * y) = make_float2(d[x][y][0], d[x][y][1]);
          *reinterpret_cast<float2*>(to + (size_t)8 * p.Dv + 8 * y) = make_float2(d[x][y][2], d[x][y][3]);
        }
      }
  }
  bar<2, kWalkers>();                              // nobody reads T any more
#pragma unroll
  for (int turn = 0; turn < 2; ++turn) {
    const int row = (turn ? 3 - hw : hw) * 16 + gq;
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int col = (2 * (2 * x + turn) + y) * 8 + 2 * tq;
          uint32_t up[3], low[3];
          split3(up, W[turn][x][y][0], W[turn][x][y][1]);
          split3(low, W[turn][x][y][2], W[turn][x][y][3]);
          unsigned char* to = sm + L::W + row * L::PT + col * 2;
#pragma unroll
          for (int u = 0; u < 3; ++u) {
            *reinterpret_cast<uint32_t*>(to + u * kPiece * L::PT) = up[u];
            *reinterpret_cast<uint32_t*>(to + (u * kPiece + 8) * L::PT) = low[u];
          }
        }
  }
  bar<2, kWalkers>();
  bf16* wg = sc.w + unit * 3 * kPiece * kN;
  for (int x = ht; x < 3 * kPiece * (kN / 8); x += kWalkers)
    *reinterpret_cast<uint4*>(wg + x * 8) = *reinterpret_cast<const uint4*>(sm + L::W + (x / 8) * L::PT + (x % 8) * 16);
  for (int x = ht; x < (int)sizeof(Gates) / 16; x += kWalkers)
    reinterpret_cast<uint4*>(sc.gates + unit)[x] = reinterpret_cast<const uint4*>(&g)[x];
  for (int x = ht; x < 1 + p.Dv; x += kWalkers) sc.spoilt[unit * (1 + p.Dv) + x] = spoilt[x];
}

// DVC value columns a block, a warp for 16 rows of 16 of them.
template <int DVC>
struct ChainLayout {
  static constexpr int PN = pitch(kN), PX = pitch(DVC), STAGES = 3;
  static constexpr int W = 0;                                     // [STAGES][3][64] rows of PN
  static constexpr int K = W + STAGES * 3 * kPiece * PN;          // [STAGES][64] rows of PN
  static constexpr int U = K + STAGES * kPiece * PN;              // [STAGES][64][DVC + 4] floats
  static constexpr int PU = DVC + 4;
  static constexpr int S = U + STAGES * kPiece * PU * 4;          // [3][64] rows of PX
  static constexpr int X = S + 3 * kN * PX;                       // [3][64] rows of PX: weighed corrections
  static constexpr int G = X + 3 * kPiece * PX;                   // [STAGES][68] floats: weigh, keep
  static constexpr int bytes = G + STAGES * 68 * 4;
};

template <int DVC>
__global__ void __launch_bounds__(DVC * 8) chain_kernel(const Args p, const Scratch sc) {
  using L = ChainLayout<DVC>;
  constexpr int THREADS = DVC * 8, KN = kN / 16;
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int slices = p.Dv / DVC, h = blockIdx.x / slices, col0 = blockIdx.x % slices * DVC, r = p.first + blockIdx.y;
  pdl_trigger();
  pdl_wait();
  const int t0 = p.q_start[r], t1 = p.q_start[r + 1], pieces = (t1 - t0 + kPiece - 1) / kPiece;
  if (pieces <= 0) return;
  const int base = pieces_before(p, r);
  float* slot = p.state + (size_t)p.slots[r] * p.slot_stride;
  const bf16* k = p.k + (size_t)(h / p.share) * kN;
  auto unit_of = [&](int piece) { return (size_t)(base + piece) * p.H + h; };
  auto bring = [&](int piece) {
    if (piece < pieces) {
      const int b = piece % L::STAGES, c0 = t0 + piece * kPiece;
      const size_t unit = unit_of(piece);
      const bf16* w = sc.w + unit * 3 * kPiece * kN;
      for (int x = tid; x < 3 * kPiece * (kN / 8); x += THREADS)
        copy16(sm + L::W + (b * 3 * kPiece + x / 8) * L::PN + (x % 8) * 16, w + x * 8, true);
      for (int x = tid; x < kPiece * (kN / 8); x += THREADS) {
        const bool in = c0 + x / 8 < t1;
        copy16(sm + L::K + (b * kPiece + x / 8) * L::PN + (x % 8) * 16, k + (size_t)(in ? c0 + x / 8 : t0) * p.ld_k + x % 8 * 8, in);
      }
      const float* u = sc.u + unit * kPiece * p.Dv + col0;
      for (int x = tid; x < kPiece * (DVC / 4); x += THREADS)
        copy16(sm + L::U + ((b * kPiece + x / (DVC / 4)) * L::PU + x % (DVC / 4) * 4) * 4, u + (size_t)(x / (DVC / 4)) * p.Dv + x % (DVC / 4) * 4, true);
      if (tid < 17)
        copy16(sm + L::G + (b * 68 + tid * 4) * 4, reinterpret_cast<const float*>(sc.gates + unit) + (tid < 16 ? offsetof(Gates, weigh) / 4 + tid * 4 : offsetof(Gates, keep) / 4), true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  bring(0);
  bring(1);
  const int rb = warp & 3, cb = warp >> 2;               // 16 tokens (and 16 rows of the state), 16 columns
  const bool fresh = p.req_start[r] == 0;
  float S[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = rb * 16 + gq + (e >> 1) * 8, c = cb * 16 + 8 * nt + 2 * tq + (e & 1);
      S[nt][e] = fresh ? 0.f : slot[((size_t)h * p.Dv + col0 + c) * kN + n];
    }
  auto put = [&](int at, int row, int nt, float x, float y) {
    uint32_t part[3];
    split3(part, x, y);
    unsigned char* to = sm + at + row * L::PX + (cb * 16 + 8 * nt + 2 * tq) * 2;
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(to + s * kPiece * L::PX) = part[s];
  };
  const int row = rb * 16 + gq;
  auto barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); };
  for (int piece = 0; piece < pieces; ++piece) {
    const int b = piece % L::STAGES;
    const size_t unit = unit_of(piece);
    float* sg = sc.s + (unit * kN + row) * p.Dv + col0 + cb * 16 + 2 * tq;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {                     // the state this piece begins with: for the products, and for the results
      put(L::S, row, nt, S[nt][0], S[nt][1]);
      put(L::S, row + 8, nt, S[nt][2], S[nt][3]);
      *reinterpret_cast<float2*>(sg + 8 * nt) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(sg + (size_t)8 * p.Dv + 8 * nt) = make_float2(S[nt][2], S[nt][3]);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    barrier();                                           // this piece has arrived, the state is there; the last piece's stage is free
    bring(piece + 2);
    const float* g = reinterpret_cast<const float*>(sm + L::G) + b * 68;
    // a key without weight adds nothing; one that is not finite has none, and must not meet the zeros it is multiplied with
    if (tid < kPiece && g[tid] == 0.f)
      for (int c = 0; c < kN / 8; ++c) *reinterpret_cast<uint4*>(sm + L::K + (b * kPiece + tid) * L::PN + c * 16) = make_uint4(0u, 0u, 0u, 0u);
    // U = U0 - W S
    float acc[2][4];
#pragma unroll
    for (int x = 0; x < 2; ++x) acc[x][0] = acc[x][1] = acc[x][2] = acc[x][3] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) {
      uint32_t a[3][4], f[3][4];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        ldm4(a[s], sm + L::W + ((b * 3 + s) * kPiece + rb * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
        ldm4t(f[s], sm + L::S + (s * kN + kk * 16 + (lane & 15)) * L::PX + (cb * 2 + (lane >> 4)) * 16);
      }
      float t[2][4];
      mma0(t[0], a[2], f[0][0], f[0][1]);
      mma0(t[1], a[2], f[0][2], f[0][3]);
#pragma unroll
      for (int x = 1; x < 6; ++x) {
        const int o = x < 3 ? 2 : x < 5 ? 1 : 0, s = x < 3 ? x : x < 5 ? x - 3 : 0;
        mma(t[0], a[o - s], f[s][0], f[s][1]);
        mma(t[1], a[o - s], f[s][2], f[s][3]);
      }
      add4(acc[0], t[0]);
      add4(acc[1], t[1]);
    }
    {
      const float w0 = g[row], w1 = g[row + 8];
      const float* u0 = reinterpret_cast<const float*>(sm + L::U) + (b * kPiece + row) * L::PU + cb * 16 + 2 * tq;
      float* ug = sc.u + (unit * kPiece + row) * p.Dv + col0 + cb * 16 + 2 * tq;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float2 x = *reinterpret_cast<const float2*>(u0 + 8 * nt), y = *reinterpret_cast<const float2*>(u0 + 8 * L::PU + 8 * nt);
        const float a0 = x.x - acc[nt][0], a1 = x.y - acc[nt][1], b0 = y.x - acc[nt][2], b1 = y.y - acc[nt][3];
        put(L::X, row, nt, w0 * a0, w0 * a1);
        put(L::X, row + 8, nt, w1 * b0, w1 * b1);
        *reinterpret_cast<float2*>(ug + 8 * nt) = make_float2(a0, a1);
        *reinterpret_cast<float2*>(ug + (size_t)8 * p.Dv + 8 * nt) = make_float2(b0, b1);
      }
    }
    barrier();
    // S <- keep S + sum_j k_j (weigh_j u_j)^T
    const float keep = g[64];
    float d[2][4];
#pragma unroll
    for (int jj = 0; jj < kPiece / 16; ++jj) {
      uint32_t a[4];
      ldm4t(a, sm + L::K + (b * kPiece + jj * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + (rb * 2 + (lane >> 3 & 1)) * 16);
      float t[2][4];
#pragma unroll
      for (int s = 2; s >= 0; --s) {
        uint32_t f[4];
        ldm4t(f, sm + L::X + (s * kPiece + jj * 16 + (lane & 15)) * L::PX + (cb * 2 + (lane >> 4)) * 16);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (s == 2) mma0(t[c], a, f[2 * c], f[2 * c + 1]);
          else mma(t[c], a, f[2 * c], f[2 * c + 1]);
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) d[c][e] = jj == 0 ? t[c][e] : d[c][e] + t[c][e];
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[c][e] = fmaf(S[c][e], keep, d[c][e]);
  }
  // What is not finite: from the first such token on results are NaNs, and so is the state.  A piece's entries become those of everything up to it.
  __shared__ int lost[1 + DVC];
  if (tid <= DVC) {
    const int at = tid == 0 ? 0 : col0 + tid;
    bool any = false;
    for (int piece = 0; piece < pieces; ++piece) {
      int* entry = sc.spoilt + unit_of(piece) * (1 + p.Dv) + at;
      const bool here = *entry != kNoToken;
      if (any) *entry = 0;
      any |= here;
    }
    lost[tid] = any;
  }
  __syncthreads();
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = rb * 16 + gq + (e >> 1) * 8, c = cb * 16 + 8 * nt + 2 * tq + (e & 1);
      slot[((size_t)h * p.Dv + col0 + c) * kN + n] = lost[0] || lost[1 + c] ? CUDART_NAN_F : S[nt][e];
    }
}

// A block makes 32 columns of one (piece, head): a warp for 16 tokens.
struct ResultsLayout {
  static constexpr int PN = pitch(kN);
  static constexpr int K = 0;
  static constexpr int Q = K + kPiece * PN;
  static constexpr int G = Q + kPiece * PN;
  static constexpr int S = G + (int)sizeof(Gates);                // [3][64] rows of pitch(32), then U the same
  static constexpr int PX = pitch(32);
  static constexpr int U = S + 3 * kN * PX;
  static constexpr int bytes = U + 3 * kPiece * PX;
};

__global__ void __launch_bounds__(kWalkers) results_kernel(const Args p, int R, const Scratch sc) {
  using L = ResultsLayout;
  constexpr int KN = kN / 16, NX = 4;                    // 32 columns a block
  extern __shared__ __align__(128) unsigned char sm[];
  Gates& g = *reinterpret_cast<Gates*>(sm + L::G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int slices = p.Dv / 32, h = blockIdx.x / slices, col0 = blockIdx.x % slices * 32;
  pdl_trigger();
  pdl_wait();
  int r, local;
  if (!find_piece(p, R, blockIdx.y, r, local)) return;
  const size_t unit = (size_t)blockIdx.y * p.H + h;
  const int c0 = p.q_start[r] + local * kPiece, t1 = p.q_start[r + 1];
  {
    const bf16* q = p.q + (size_t)(h / p.share) * kN;
    const bf16* k = p.k + (size_t)(h / p.share) * kN;
    for (int x = tid; x < kPiece * (kN / 8); x += kWalkers) {
      const int i = x / 8, c = x % 8;
      const bool in = c0 + i < t1;
      copy16(sm + L::K + i * L::PN + c * 16, k + (size_t)(in ? c0 + i : c0) * p.ld_k + c * 8, in);
      copy16(sm + L::Q + i * L::PN + c * 16, q + (size_t)(in ? c0 + i : c0) * p.ld_q + c * 8, in);
    }
    for (int x = tid; x < (int)sizeof(Gates) / 16; x += kWalkers)
      copy16(sm + L::G + x * 16, reinterpret_cast<const unsigned char*>(sc.gates + unit) + x * 16, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // the state and the corrections, in parts
    const float* from[2] = {sc.s + unit * kN * p.Dv + col0, sc.u + unit * kPiece * p.Dv + col0};
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int x = tid + (i & 3) * kWalkers;
      v[i] = *reinterpret_cast<const float4*>(from[i >> 2] + (size_t)(x >> 3) * p.Dv + (x & 7) * 4);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int x = tid + (i & 3) * kWalkers;
      uint32_t lo[3], hi[3];
      split3(lo, v[i].x, v[i].y);
      split3(hi, v[i].z, v[i].w);
      unsigned char* to = sm + (i >> 2 ? L::U : L::S) + (x >> 3) * L::PX + (x & 7) * 8;
#pragma unroll
      for (int s = 0; s < 3; ++s) *reinterpret_cast<uint2*>(to + s * kPiece * L::PX) = make_uint2(lo[s], hi[s]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  if (tid < 64) {                                        // a query's norm a thread; a key that is not finite was left out
    unsigned char* from = sm + L::Q + tid * L::PN;
    float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < kN / 8; ++c) {
      const uint4 u = *reinterpret_cast<const uint4*>(from + c * 16);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = __uint_as_float(w[e] << 16), y = __uint_as_float(w[e] & 0xffff0000u);
        ss[e] = fmaf(x, x, ss[e]);
        ss[e] = fmaf(y, y, ss[e]);
      }
    }
    float sum = (ss[0] + ss[1]) + (ss[2] + ss[3]);
    if (!isfinite(sum)) {
      uint32_t bad = 0u;
      for (int c = 0; c < kN / 2; ++c) bad |= not_finite(reinterpret_cast<const uint32_t*>(from)[c]);
      if (!bad)                                          // (a query that is not finite spoils its own row only)
        for (int c = 0; c < kN / 8; ++c) reinterpret_cast<uint4*>(from)[c] = make_uint4(0u, 0u, 0u, 0u);
      sum = CUDART_INF_F;
    }
    g.qinv[tid] = rsqrtf((float)kN) / sqrtf(sum + 1e-6f);
  } else {
    const int i = tid - 64;
    if (!(g.kinv[i] > 0.f))                              // its norm was beyond float32's range, or a part of it not finite
      for (int c = 0; c < kN / 8; ++c) *reinterpret_cast<uint4*>(sm + L::K + i * L::PN + c * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  const unsigned char *Ks = sm + L::K, *Qs = sm + L::Q;
  float G[8][4], accq[NX][4];
#pragma unroll
  for (int x = 0; x < 8; ++x) G[x][0] = G[x][1] = G[x][2] = G[x][3] = 0.f;
#pragma unroll
  for (int x = 0; x < NX; ++x) accq[x][0] = accq[x][1] = accq[x][2] = accq[x][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < KN; ++kk) {
    uint32_t aq[4];
    ldm4(aq, Qs + (warp * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
    for (int nt = 0; nt < NX; nt += 2) {
      float t[2][4];
#pragma unroll
      for (int s = 2; s >= 0; --s) {
        uint32_t f[4];
        ldm4t(f, sm + L::S + (s * kN + kk * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
        if (s == 2) {
          mma0(t[0], aq, f[0], f[1]);
          mma0(t[1], aq, f[2], f[3]);
        } else {
          mma(t[0], aq, f[0], f[1]);
          mma(t[1], aq, f[2], f[3]);
        }
      }
      add4(accq[nt], t[0]);
      add4(accq[nt + 1], t[1]);
    }
#pragma unroll
    for (int jt = 0; jt < 4; ++jt)
      if (jt <= warp) {
        uint32_t f[4];
        ldm4(f, Ks + (jt * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + (kk * 2 + (lane >> 3 & 1)) * 16);
        mma(G[2 * jt], aq, f[0], f[1]);
        mma(G[2 * jt + 1], aq, f[2], f[3]);
      }
  }
  const int row = warp * 16 + gq;
  const float from0 = g.from[row], from1 = g.from[row + 8];
#pragma unroll
  for (int x = 0; x < NX; ++x) { accq[x][0] *= from0; accq[x][1] *= from0; accq[x][2] *= from1; accq[x][3] *= from1; }
  const float h0 = g.hi[row], l0 = g.lo[row], h1 = g.hi[row + 8], l1 = g.lo[row + 8], r0 = g.rows[row], r1 = g.rows[row + 8];
#pragma unroll
  for (int jt = 0; jt < 4; ++jt)
    if (jt <= warp) {
      uint32_t a[3][4];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float* e = G[2 * jt + half];
        const int j = jt * 16 + half * 8 + 2 * tq;
        if (jt < warp) {
          const float2 f = *reinterpret_cast<const float2*>(g.cols + 8 * warp * (warp - 1) + j);
          const float w0 = f.x * g.kinv[j], w1 = f.y * g.kinv[j + 1];
          e[0] *= r0 * w0;
          e[1] *= r0 * w1;
          e[2] *= r1 * w0;
          e[3] *= r1 * w1;
        } else {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float ch = g.hi[j + u], cl = g.lo[j + u], w = g.kinv[j + u];
            e[u] = j + u <= row ? e[u] * (expf((h0 - ch) + (l0 - cl)) * w) : 0.f;
            e[2 + u] = j + u <= row + 8 ? e[2 + u] * (expf((h1 - ch) + (l1 - cl)) * w) : 0.f;
          }
        }
        uint32_t up[3], low[3];
        split3(up, e[0], e[1]);
        split3(low, e[2], e[3]);
#pragma unroll
        for (int s = 0; s < 3; ++s) { a[s][2 * half] = up[s]; a[s][2 * half + 1] = low[s]; }
      }
#pragma unroll
      for (int nt = 0; nt < NX; nt += 2) {
        uint32_t f[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s) ldm4t(f[s], sm + L::U + (s * kPiece + jt * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
        float t[2][4];
        mma0(t[0], a[2], f[0][0], f[0][1]);
        mma0(t[1], a[2], f[0][2], f[0][3]);
#pragma unroll
        for (int x = 1; x < 6; ++x) {
          const int o = x < 3 ? 2 : x < 5 ? 1 : 0, s = x < 3 ? x : x < 5 ? x - 3 : 0;
          mma(t[0], a[o - s], f[s][0], f[s][1]);
          mma(t[1], a[o - s], f[s][2], f[s][3]);
        }
        add4(accq[nt], t[0]);
        add4(accq[nt + 1], t[1]);
      }
    }
  const int* spoilt = sc.spoilt + unit * (1 + p.Dv);
  const int whole = spoilt[0];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int i = row + 8 * half;
    if (c0 + i < t1) {
      const float f = g.qinv[i];
      float* to = p.o + (size_t)(c0 + i) * p.H * p.Dv + (size_t)h * p.Dv + col0 + 2 * tq;
#pragma unroll
      for (int nt = 0; nt < NX; ++nt) {
        const int* col = spoilt + 1 + col0 + 8 * nt + 2 * tq;
        *reinterpret_cast<float2*>(to + 8 * nt) = make_float2(min(whole, col[0]) <= i ? CUDART_NAN_F : accq[nt][2 * half] * f,
                                                              min(whole, col[1]) <= i ? CUDART_NAN_F : accq[nt][2 * half + 1] * f);
      }
    }
  }
}

// Bytes of scratch for steps of `tokens` in R runs: at most tokens / 64 + R pieces.
static long long scratch_bytes(long long tokens, int R, int H, int Dv) {
  const long long units = (tokens / kPiece + R) * H;
  return units * (3ll * kPiece * kN * 2 + 2ll * kPiece * Dv * 4 + (long long)sizeof(Gates) + (1 + Dv) * 4) + 64;
}

static bool takes_pieces(const Args& a, int N) { return N == kN && a.Dv <= 64 && delta_walk::takes(a, N); }

static int launch(const Args& a, int R, long long tokens, void* scratch, cudaStream_t stream) {
  const long long pieces = tokens / kPiece + R, units = pieces * a.H;
  if (R <= 0) return 0;
  if (R > 65535 || pieces > 65535 || !takes_pieces(a, kN) || scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 15)) return KVB_ERR_BAD_SIZE;
  static_assert(sizeof(Gates) % 16 == 0, "copied in 16 bytes");
  Scratch sc;
  sc.w = static_cast<bf16*>(scratch);
  sc.u = reinterpret_cast<float*>(sc.w + units * 3 * kPiece * kN);
  sc.s = sc.u + units * kPiece * a.Dv;
  sc.gates = reinterpret_cast<Gates*>(sc.s + units * kPiece * a.Dv);
  sc.spoilt = reinterpret_cast<int*>(sc.gates + units);
  constexpr int prep = PrepareLayout::bytes;
  cudaError_t e = cudaFuncSetAttribute(prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, prep);
  if (e == cudaSuccess) e = kvb_launch(prepare_kernel, dim3((unsigned)a.H, (unsigned)pieces), dim3(kWalkers + 32), prep, stream, a, R, sc);
  if (e != cudaSuccess) return (int)e;
  // 16 value columns a block, 32 where that still gives (nearly) every SM a block
  if ((long long)a.H * (a.Dv / 32) * R * 5 < (long long)kvb_sm_count() * 4) {
    e = cudaFuncSetAttribute(chain_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChainLayout<16>::bytes);
    if (e == cudaSuccess) e = kvb_launch(chain_kernel<16>, dim3((unsigned)(a.H * (a.Dv / 16)), (unsigned)R), dim3(128), ChainLayout<16>::bytes, stream, a, sc);
  } else {
    e = cudaFuncSetAttribute(chain_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChainLayout<32>::bytes);
    if (e == cudaSuccess) e = kvb_launch(chain_kernel<32>, dim3((unsigned)(a.H * (a.Dv / 32)), (unsigned)R), dim3(256), ChainLayout<32>::bytes, stream, a, sc);
  }
  if (e != cudaSuccess) return (int)e;
  e = cudaFuncSetAttribute(results_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ResultsLayout::bytes);
  if (e == cudaSuccess) e = kvb_launch(results_kernel, dim3((unsigned)(a.H * (a.Dv / 32)), (unsigned)pieces), dim3(kWalkers), ResultsLayout::bytes, stream, a, R, sc);
  return e == cudaSuccess ? kvb_launch_result() : (int)e;
}

}  // namespace delta_pieces
