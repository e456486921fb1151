// The gated delta rule with one decay per head and token, along a request's run of tokens, on tensor cores:
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q          (k, q unit vectors, q also times N^-1/2)
//
// A block owns DVC value columns of one (request, head) and walks the run in pieces of 64 tokens.  With P_i the product of a
// piece's decays up to token i and S what the piece begins with, the corrections u of the piece solve
//
//   (I + A) U = R,    A_ij = beta_i (P_i / P_j) (k_i . k_j)  for j < i,    R_i = beta_i (v_i - P_i S^T k_i)
//
// and  o_i = P_i S^T q_i + sum_{j <= i} (P_i / P_j) (q_i . k_j) u_j,    S <- P_63 S + sum_j (P_63 / P_j) k_j u_j^T.
//
// A does not depend on the state: four helper warps fetch the next piece's rows and make the inverse of I + A for it (its diagonal
// blocks of 16 by elimination in float32, two lanes a column, the blocks below them by products), a ninth warp makes its gates, while
// four walking warps do this piece's products on mma.sync.  As in
// chunk_walk.cuh keys and queries go in as they came (their norms are factors per token) and every float32 operand as the
// sum of three bfloat16 numbers; where both are float32 (inverse and right side, weighed scores and corrections) six of
// the nine products are made, the others lie below 2^-24 (with eight of them no error changed).  Every sum over more than one 16 x 16
// block is added up by float32 instructions (mma0 there says why).
// Measured against 64 bits, runs of 64 to 4096 tokens: the state is two to three times as close as token by token where it forgets
// slowly (5e-6 against 1e-5 of its norm), and like it at the floor of a dozen roundings where it forgets quickly (1e-7 to 3e-7); keys that
// are nearly the same cost up to 1.6 times the scan's error there (2.2e-7 against 1.4e-7).
//
// Zero times an infinity is a NaN, and the products above hold zeros in the place of all later tokens.  So what is not finite is left out
// of them: a key, or a gate that is a NaN, makes its head's results NaN from its token on, a value its column's, and what stands in
// front of it is as it would be without it.  (Sums of finite numbers beyond float32's range are not told apart like this.)
//
// What bounds it: latency, about 10500 cycles a piece, for walkers (three steps of products with a barrier behind each) and helpers
// (rows, norms, A, its inverse) alike.  Walking token by token in float32 is a chain of 64 steps of two dot products each: 32 heads
// of 64 x 64, runs of 1548 + 500 tokens 474 us, now 197 (176 with all sums in one chain of accumulations; twice that with the whole inverse by
// elimination).  Long runs of keys of 64 take three launches instead: delta_pieces.cuh.
#pragma once

#include "chunk_walk.cuh"

namespace delta_walk {

using namespace walk;

constexpr int kWalkers = 128, kAll = 2 * kWalkers + 32;      // walkers, helpers, one warp for the gates

struct Args {
  const bf16* q; int ld_q;            // head h reads q and k at (h / share) * N, v at h * Dv
  const bf16* k; int ld_k;
  const bf16* v; int ld_v;
  int share;
  const bf16* decay; int ld_decay; const float* decay_bias; const float* head_rate;     // [T, H], [H], [H]
  const bf16* beta; int ld_beta;                                                        // [T, H], before the sigmoid
  float* state; long long slot_stride;                                                  // slot 0's [H][Dv][N]
  float* o;                                                                             // [T, H * Dv] float32
  const int* q_start; const int* req_start; const int* slots;
  int H, Dv, first;
};

struct Gates {
  float hi[kPiece], lo[kPiece];       // log P_i as a pair
  float from[kPiece];                 // P_i
  float beta[kPiece], kinv[kPiece], qinv[kPiece];
  float weigh[kPiece];                // P_63 / P_j / |k_j|
  float rows[kPiece], cols[96];       // P_i / P_j = rows[i] cols[8 I (I - 1) + j] for i in the I-th 16 tokens and j before them, by way of
                                      // the last token before these: neither factor exceeds one
  float keep, pad[3];
};

template <int N, int DVC>
struct Layout {
  static constexpr int PN = pitch(N), PX = pitch(DVC), PT = pitch(kPiece);
  static constexpr int STAGES = N == 64 ? 3 : 2;                  // three where they fit: rows are fetched a round before the helpers need them
  static constexpr int PD = 20;                                   // floats per column of a diagonal block: eight even rows, eight odd ones
  static constexpr int K = 0;                                     // [STAGES][64] rows of PN
  static constexpr int Q = K + STAGES * kPiece * PN;              // [STAGES][64] rows of PN
  static constexpr int V = Q + STAGES * kPiece * PN;              // [STAGES][64] rows of PX
  static constexpr int S = V + STAGES * kPiece * PX;              // [3][N] rows of PX
  static constexpr int R = S + 3 * N * PX;                        // [3][64] rows of PX: right sides
  static constexpr int U = R + 3 * kPiece * PX;                   // [3][64]: corrections
  static constexpr int W = U + 3 * kPiece * PX;                   // [3][64]: weighed corrections
  static constexpr int T = W + 3 * kPiece * PX;                   // [2][3][64] rows of PT: the inverse
  static constexpr int A = T + 2 * 3 * kPiece * PT;               // [3][64] rows of PT: A left of its diagonal blocks
  static constexpr int D = A + 3 * kPiece * PT;                   // [4][16] columns of PD floats: A's diagonal blocks
  static constexpr int G = D + 4 * 16 * PD * 4;                   // [3] gates
  static constexpr int F = G + 3 * (int)sizeof(Gates);            // first tokens of the run that are not finite: any, whole head, [DVC] columns
  static constexpr int bytes = F + (2 + DVC) * 4;
};

__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus20(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ void stm4t(const uint32_t* r, void* p) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
               ::"r"(smem_at(p)), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
// two 16 x 8 accumulators side by side, times `sign`, as a 16 x 16 left operand in three parts
__device__ __forceinline__ void left_parts(uint32_t (*to)[4], const float (*d)[4], float sign) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t up[3], low[3];
    split3(up, sign * d[half][0], sign * d[half][1]);
    split3(low, sign * d[half][2], sign * d[half][3]);
#pragma unroll
    for (int s = 0; s < 3; ++s) { to[s][2 * half] = up[s]; to[s][2 * half + 1] = low[s]; }
  }
}
template <int ID, int THREADS> __device__ __forceinline__ void bar() { asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory"); }

template <int N, int DVC>
__global__ void __launch_bounds__(kAll) delta_walk_kernel(const Args p) {
  using L = Layout<N, DVC>;
  constexpr int MT = N / 64, NX = DVC / 8, KN = N / 16;
  extern __shared__ __align__(128) unsigned char sm[];
  Gates* gates = reinterpret_cast<Gates*>(sm + L::G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, tq = lane & 3;
  const int slices = p.Dv / DVC, h = blockIdx.x / slices, col0 = blockIdx.x % slices * DVC, r = p.first + blockIdx.y;
  pdl_trigger();
  pdl_wait();
  const int t0 = p.q_start[r], t1 = p.q_start[r + 1];
  // Round s: the gates of piece s, the rows of piece s (of s - 1 with two stages), the inverse of piece s - 1, the walk over piece s - 2.
  const int pieces = (t1 - t0 + kPiece - 1) / kPiece, rounds = pieces > 0 ? pieces + 2 : 0;
  float* slot = p.state + (size_t)p.slots[r] * p.slot_stride;
  int* spoilt = reinterpret_cast<int*>(sm + L::F);
  constexpr int kNever = 0x7fffffff;
  auto spoil = [&](int which, int token) {
    atomicMin(spoilt + which, token);
    atomicMin(spoilt, token);
  };

  if (warp == 8) {
    // ------------------------------------------------------------ gates
    const float rate = expf(p.head_rate[h]), dbias = p.decay_bias[h];
    for (int i = lane; i < 2 + DVC; i += 32) spoilt[i] = kNever;
    __syncwarp();
    for (int s = 0; s < rounds; ++s) {
      if (s < pieces) {
        Gates& g = gates[s % 3];
        double c[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = lane + 32 * u, t = t0 + s * kPiece + i;
          float la = 0.f, be = 0.f;                      // behind the run's end nothing decays
          if (t < t1) {
            la = -(rate * softplus20(__bfloat162float(p.decay[(size_t)t * p.ld_decay + h]) + dbias));
            la = la < -200.f ? -200.f : la;              // (exp(-200) is zero in float32, and sums of -200 lose nothing)
            be = sigmoid(__bfloat162float(p.beta[(size_t)t * p.ld_beta + h]));
            if (isnan(la + be)) {
              spoil(1, s * kPiece + i);
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
          g.rows[i] = expf((float)(c[u] - (u ? (lane < 16 ? c31 : c47) : c15)));                 // (unused in the first 16)
        }
        if (lane < 16) {
          g.cols[lane] = expf((float)(c15 - c[0]));
          g.cols[80 + lane] = expf((float)(c47 - c[1]));
        }
        g.cols[16 + lane] = expf((float)(c31 - c[0]));
        g.cols[48 + lane] = expf((float)(c47 - c[0]));
        if (lane == 0) g.keep = expf((float)total);
      }
      bar<0, kAll>();
    }
    return;
  }

  if (warp >= 4) {
    // ------------------------------------------------------------ helpers
    const int ht = tid - kWalkers, hw = warp - 4;
    const bf16* q = p.q + (size_t)(h / p.share) * N;
    const bf16* k = p.k + (size_t)(h / p.share) * N;
    const bf16* v = p.v + (size_t)h * p.Dv + col0;
    const float q_scale = rsqrtf((float)N);
    auto rows = [&](unsigned char* to, int at, const bf16* from, int ld, int cols, int c0) {
      const int chunks = cols / 8;
      for (int x = ht; x < kPiece * chunks; x += kWalkers) {
        const int i = x / chunks, c = x - i * chunks;
        const bool in = c0 + i < t1;
        copy16(to + i * at + c * 16, from + (size_t)(in ? c0 + i : t0) * ld + c * 8, in);
      }
    };
    auto bring = [&](int piece) {
      const int c0 = t0 + piece * kPiece, b = piece % L::STAGES;
      rows(sm + L::K + b * kPiece * L::PN, L::PN, k, p.ld_k, N, c0);
      rows(sm + L::Q + b * kPiece * L::PN, L::PN, q, p.ld_q, N, c0);
      rows(sm + L::V + b * kPiece * L::PX, L::PX, v, p.ld_v, DVC, c0);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // acc += left (16 x 16) * the transpose of the 16 x 16 block at `from`, both in three parts: the six products that count
    auto mma6t = [&](float (*acc)[4], const uint32_t (*left)[4], const unsigned char* from) {
      uint32_t f[3][4];
#pragma unroll
      for (int u = 0; u < 3; ++u) ldm4(f[u], from + (u * kPiece + (lane & 7) + (lane >> 4) * 8) * L::PT + (lane >> 3 & 1) * 16);
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
    for (int s = 0; s < rounds; ++s) {
      if (L::STAGES == 3 && s < pieces) bring(s);
      if (s >= 1 && s <= pieces) {
        const int piece = s - 1, b = piece % L::STAGES;
        Gates& g = gates[piece % 3];
        unsigned char* Ks = sm + L::K + b * kPiece * L::PN;
        unsigned char* Ts = sm + L::T + (piece & 1) * 3 * kPiece * L::PT;
        if (L::STAGES == 2) {
          bring(piece);
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          bar<2, kWalkers>();
        }
        {                                                // a row's norm a thread: keys, then queries
          const int i = ht & 63;
          unsigned char* from = (ht < 64 ? Ks : sm + L::Q + b * kPiece * L::PN) + i * L::PN;
          float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int c = 0; c < N / 8; ++c) {
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
          if (!isfinite(sum)) {                          // a row that is not finite, or squares beyond float32's range (the unit vector is zero then)
            uint32_t bad = 0u;
            for (int c = 0; c < N / 2; ++c) bad |= not_finite(reinterpret_cast<const uint32_t*>(from)[c]);
            if (bad && ht < 64) spoil(1, piece * kPiece + i);
            if (!bad || ht < 64)                         // (a query that is not finite spoils its own row only)
              for (int c = 0; c < N / 8; ++c) reinterpret_cast<uint4*>(from)[c] = make_uint4(0u, 0u, 0u, 0u);
            sum = CUDART_INF_F;                          // (its factor is zero)
          }
          if (ht < 64) {
            const float inv = 1.0f / sqrtf(sum + 1e-6f);
            g.kinv[i] = inv;
            g.weigh[i] *= inv;
          } else {
            g.qinv[i] = q_scale / sqrtf(sum + 1e-6f);
          }
        }
        bar<2, kWalkers>();
        float* Dg = reinterpret_cast<float*>(sm + L::D) + hw * 16 * L::PD;
        {                                                // rows 16 hw .. of A: bfloat16 parts left of the diagonal block, the block itself as floats
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
                const float c0 = f.x * g.kinv[j], c1 = f.y * g.kinv[j + 1];
                G[x][0] *= r0 * c0;
                G[x][1] *= r0 * c1;
                G[x][2] *= r1 * c0;
                G[x][3] *= r1 * c1;
              } else {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const float ch = g.hi[j + u], cl = g.lo[j + u], w = g.kinv[j + u];
                  G[x][u] *= w0 * w * expf((h0 - ch) + (l0 - cl));
                  G[x][2 + u] *= w1 * w * expf((h1 - ch) + (l1 - cl));
                }
              }
              if (x / 2 < hw) {
                uint32_t up[3], low[3];
                split3(up, G[x][0], G[x][1]);
                split3(low, G[x][2], G[x][3]);
                unsigned char* to = sm + L::A + row * L::PT + j * 2;
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                  *reinterpret_cast<uint32_t*>(to + u * kPiece * L::PT) = up[u];
                  *reinterpret_cast<uint32_t*>(to + (u * kPiece + 8) * L::PT) = low[u];
                }
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int i = gq + (e >> 1) * 8, c = (j & 15) + (e & 1);
                  Dg[c * L::PD + (i & 1) * 8 + (i >> 1)] = c < i ? G[x][e] : 0.f;
                }
              }
            }
        }
        __syncwarp();
        {                                                // the diagonal block's inverse: lanes 2 m and 2 m + 1 hold column m's even and odd rows
          const int par = lane & 1, odd = lane >> 1 & 1;
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = 2 * e + par == (lane >> 1) ? 1.f : 0.f;
#pragma unroll
          for (int j = 0; j < 15; ++j) {
            const float u = __shfl_sync(0xffffffffu, x[j >> 1], (lane & ~1) | (j & 1));
            const float4* column = reinterpret_cast<const float4*>(Dg + j * L::PD + par * 8);
#pragma unroll
            for (int e = (j >> 1) & ~3; e < 8; e += 4) { // rows up to j itself are zero in A
              const float4 a = column[e >> 2];
              x[e] = fmaf(-a.x, u, x[e]);
              x[e + 1] = fmaf(-a.y, u, x[e + 1]);
              x[e + 2] = fmaf(-a.z, u, x[e + 2]);
              x[e + 3] = fmaf(-a.w, u, x[e + 3]);
            }
          }
#pragma unroll
          for (int e = 0; e < 8; e += 2) {               // of two neighbouring columns the first writes the even e, the second the odd ones
            const float other = __shfl_xor_sync(0xffffffffu, odd ? x[e] : x[e + 1], 2);
            const float mine = odd ? x[e + 1] : x[e];
            uint32_t part[3];
            split3(part, odd ? other : mine, odd ? mine : other);
#pragma unroll
            for (int u = 0; u < 3; ++u)
              *reinterpret_cast<uint32_t*>(Ts + (u * kPiece + hw * 16 + 2 * (e + odd) + par) * L::PT + (hw * 16 + (lane >> 1 & ~1)) * 2) = part[u];
          }
        }
        bar<2, kWalkers>();
        // The blocks below it, T_IJ = -T_II (sum over K from J to I - 1 of A_IK T_KJ) for J = hw, transposed: every product's result is
        // the next one's left operand as it lies in the registers.
        uint32_t left[3][3][4];                          // T_KJ^T, K = hw + the first index
#pragma unroll
        for (int u = 0; u < 3; ++u)
          ldm4t(left[0][u], Ts + (u * kPiece + hw * 16 + (lane & 7) + (lane >> 4) * 8) * L::PT + (hw * 2 + (lane >> 3 & 1)) * 16);
#pragma unroll
        for (int d = 1; d < 4; ++d)
          if (hw + d < 4) {
            const int I = hw + d;
            float X[2][4] = {}, Y[2][4] = {};
#pragma unroll
            for (int e = 0; e < d; ++e) mma6t(X, left[e], sm + L::A + I * 16 * L::PT + (hw + e) * 32);
            uint32_t x[3][4], y[3][4];
            left_parts(x, X, 1.f);
            mma6t(Y, x, Ts + I * 16 * L::PT + I * 32);
            left_parts(y, Y, -1.f);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
              stm4t(y[u], Ts + (u * kPiece + I * 16 + (lane & 7) + (lane >> 4) * 8) * L::PT + (hw * 2 + (lane >> 3 & 1)) * 16);
              if (d < 3)
#pragma unroll
                for (int e = 0; e < 4; ++e) left[d][u][e] = y[u][e];
            }
          }
      }
      if (L::STAGES == 3) asm volatile("cp.async.wait_group 0;" ::: "memory");
      bar<0, kAll>();                                    // the walkers are done with the piece before; this one is ready
    }
    return;
  }

  // -------------------------------------------------------------- walkers
  const bool fresh = p.req_start[r] == 0;
  float S[MT][NX][4];                                    // rows (warp * MT + mt) * 16 + gq (+ 8), columns 8 nt + 2 tq (+ 1)
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < NX; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = (warp * MT + mt) * 16 + gq + (e >> 1) * 8, c = 8 * nt + 2 * tq + (e & 1);
        S[mt][nt][e] = fresh ? 0.f : slot[((size_t)h * p.Dv + col0 + c) * N + n];
      }
  auto put = [&](int at, int rows, int row, int nt, float x, float y) {      // two neighbouring columns of a row, in three parts
    uint32_t part[3];
    split3(part, x, y);
    unsigned char* to = sm + at + row * L::PX + (8 * nt + 2 * tq) * 2;
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(to + s * rows * L::PX) = part[s];
  };
  auto put_state = [&]() {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NX; ++nt) {
        put(L::S, N, (warp * MT + mt) * 16 + gq, nt, S[mt][nt][0], S[mt][nt][1]);
        put(L::S, N, (warp * MT + mt) * 16 + gq + 8, nt, S[mt][nt][2], S[mt][nt][3]);
      }
  };
  // acc += a (three parts, one 16 x 16 tile) * the three parts at `from`, rows jt * 16 ..: the six products that count
  auto mma6 = [&](float (*acc)[4], const uint32_t (*a)[4], int from, int jt) {
#pragma unroll
    for (int nt = 0; nt < NX; nt += 2) {
      uint32_t f[3][4];
#pragma unroll
      for (int s = 0; s < 3; ++s) ldm4t(f[s], sm + from + (s * kPiece + jt * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
      float t[2][4];
      mma0(t[0], a[2], f[0][0], f[0][1]);
      mma0(t[1], a[2], f[0][2], f[0][3]);
#pragma unroll
      for (int x = 1; x < 6; ++x) {
        const int o = x < 3 ? 2 : x < 5 ? 1 : 0, s = x < 3 ? x : x < 5 ? x - 3 : 0;
        mma(t[0], a[o - s], f[s][0], f[s][1]);
        mma(t[1], a[o - s], f[s][2], f[s][3]);
      }
      add4(acc[nt], t[0]);
      add4(acc[nt + 1], t[1]);
    }
  };
  if (pieces > 0) {
    put_state();
    bar<0, kAll>();
    bar<0, kAll>();                                      // the first piece is ready
  }
  const int row = warp * 16 + gq;                        // this thread's tokens of a piece: row and row + 8
  for (int piece = 0; piece < pieces; ++piece) {
    const int c0 = t0 + piece * kPiece, b = piece % L::STAGES;
    const Gates& g = gates[piece % 3];
    const unsigned char* Ks = sm + L::K + b * kPiece * L::PN;
    const unsigned char* Qs = sm + L::Q + b * kPiece * L::PN;
    const unsigned char* Vs = sm + L::V + b * kPiece * L::PX;
    float G[8][4], accq[NX][4], acck[NX][4];
#pragma unroll
    for (int x = 0; x < 8; ++x) G[x][0] = G[x][1] = G[x][2] = G[x][3] = 0.f;
#pragma unroll
    for (int x = 0; x < NX; ++x) {
      accq[x][0] = accq[x][1] = accq[x][2] = accq[x][3] = 0.f;
      acck[x][0] = acck[x][1] = acck[x][2] = acck[x][3] = 0.f;
    }
#pragma unroll
    for (int kk = 0; kk < KN; ++kk) {
      uint32_t aq[4], ak[4];
      ldm4(aq, Qs + (warp * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
      ldm4(ak, Ks + (warp * 16 + (lane & 15)) * L::PN + (kk * 2 + (lane >> 4)) * 16);
#pragma unroll
      for (int nt = 0; nt < NX; nt += 2) {
        float tk[2][4], tq4[2][4];
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          uint32_t f[4];
          ldm4t(f, sm + L::S + (s * N + kk * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
          if (s == 2) {
            mma0(tk[0], ak, f[0], f[1]);
            mma0(tk[1], ak, f[2], f[3]);
            mma0(tq4[0], aq, f[0], f[1]);
            mma0(tq4[1], aq, f[2], f[3]);
          } else {
            mma(tk[0], ak, f[0], f[1]);
            mma(tk[1], ak, f[2], f[3]);
            mma(tq4[0], aq, f[0], f[1]);
            mma(tq4[1], aq, f[2], f[3]);
          }
        }
        add4(acck[nt], tk[0]);
        add4(acck[nt + 1], tk[1]);
        add4(accq[nt], tq4[0]);
        add4(accq[nt + 1], tq4[1]);
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
    const float from0 = g.from[row], from1 = g.from[row + 8];
    {
      const float f0 = from0 * g.kinv[row], f1 = from1 * g.kinv[row + 8], b0 = g.beta[row], b1 = g.beta[row + 8];
#pragma unroll
      for (int nt = 0; nt < NX; ++nt) {
        uint32_t v0 = *reinterpret_cast<const uint32_t*>(Vs + row * L::PX + (8 * nt + 2 * tq) * 2);
        uint32_t v1 = *reinterpret_cast<const uint32_t*>(Vs + (row + 8) * L::PX + (8 * nt + 2 * tq) * 2);
        if (not_finite(v0) | not_finite(v1)) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (not_finite(v0 >> 16 * e & 0xffffu)) spoil(2 + 8 * nt + 2 * tq + e, piece * kPiece + row);
            if (not_finite(v1 >> 16 * e & 0xffffu)) spoil(2 + 8 * nt + 2 * tq + e, piece * kPiece + row + 8);
          }
          v0 = finite_part(v0);
          v1 = finite_part(v1);
        }
        put(L::R, kPiece, row, nt, b0 * fmaf(-f0, acck[nt][0], __uint_as_float(v0 << 16)),
            b0 * fmaf(-f0, acck[nt][1], __uint_as_float(v0 & 0xffff0000u)));
        put(L::R, kPiece, row + 8, nt, b1 * fmaf(-f1, acck[nt][2], __uint_as_float(v1 << 16)),
            b1 * fmaf(-f1, acck[nt][3], __uint_as_float(v1 & 0xffff0000u)));
      }
    }
    bar<1, kWalkers>();

    // the corrections
#pragma unroll
    for (int x = 0; x < NX; ++x) acck[x][0] = acck[x][1] = acck[x][2] = acck[x][3] = 0.f;
#pragma unroll
    for (int jt = 0; jt < 4; ++jt)
      if (jt <= warp) {
        uint32_t a[3][4];
#pragma unroll
        for (int s = 0; s < 3; ++s)
          ldm4(a[s], sm + L::T + (((piece & 1) * 3 + s) * kPiece + warp * 16 + (lane & 15)) * L::PT + (jt * 2 + (lane >> 4)) * 16);
        mma6(acck, a, L::R, jt);
      }
    {
      const float w0 = g.weigh[row], w1 = g.weigh[row + 8];
#pragma unroll
      for (int nt = 0; nt < NX; ++nt) {
        put(L::U, kPiece, row, nt, acck[nt][0], acck[nt][1]);
        put(L::U, kPiece, row + 8, nt, acck[nt][2], acck[nt][3]);
        put(L::W, kPiece, row, nt, w0 * acck[nt][0], w0 * acck[nt][1]);
        put(L::W, kPiece, row + 8, nt, w1 * acck[nt][2], w1 * acck[nt][3]);
      }
    }
    bar<1, kWalkers>();

    // the read-outs
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
        mma6(accq, a, L::U, jt);
      }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = row + 8 * half;
      if (c0 + i < t1) {
        const float f = g.qinv[i];
        float* to = p.o + (size_t)(c0 + i) * p.H * p.Dv + (size_t)h * p.Dv + col0 + 2 * tq;
#pragma unroll
        for (int nt = 0; nt < NX; ++nt)
          *reinterpret_cast<float2*>(to + 8 * nt) = make_float2(accq[nt][2 * half] * f, accq[nt][2 * half + 1] * f);
        if (spoilt[0] <= piece * kPiece + i)
          for (int c = 0; c < 2 * NX; ++c)
            if (min(spoilt[1], spoilt[2 + c / 2 * 8 + 2 * tq + (c & 1)]) <= piece * kPiece + i) to[c / 2 * 8 + (c & 1)] = CUDART_NAN_F;
      }
    }

    // the state
    const float keep = g.keep;
#pragma unroll
    for (int nt = 0; nt < NX; nt += 2) {
      float d[MT][2][4];
#pragma unroll
      for (int jj = 0; jj < kPiece / 16; ++jj) {
        uint32_t a[MT][4];
        float t[MT][2][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
          ldm4t(a[mt], Ks + (jj * 16 + (lane & 7) + (lane >> 4) * 8) * L::PN + ((warp * MT + mt) * 2 + (lane >> 3 & 1)) * 16);
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          uint32_t f[4];
          ldm4t(f, sm + L::W + (s * kPiece + jj * 16 + (lane & 15)) * L::PX + (nt + (lane >> 4)) * 16);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              if (s == 2) mma0(t[mt][c], a[mt], f[2 * c], f[2 * c + 1]);
              else mma(t[mt][c], a[mt], f[2 * c], f[2 * c + 1]);
            }
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[mt][c][e] = jj == 0 ? t[mt][c][e] : d[mt][c][e] + t[mt][c][e];
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[mt][nt + c][e] = fmaf(S[mt][nt + c][e], keep, d[mt][c][e]);
    }
    if (piece + 1 < pieces) put_state();
    bar<0, kAll>();
  }
  if (pieces > 0) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < NX; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int n = (warp * MT + mt) * 16 + gq + (e >> 1) * 8, c = 8 * nt + 2 * tq + (e & 1);
          slot[((size_t)h * p.Dv + col0 + c) * N + n] = min(spoilt[1], spoilt[2 + c]) != kNever ? CUDART_NAN_F : S[mt][nt][e];
        }
  }
}

static inline bool takes(const Args& a, int N) {
  return (N == 64 || N == 128) && a.Dv >= 32 && a.Dv % 32 == 0 && ((a.ld_q | a.ld_k | a.ld_v) & 7) == 0 &&
         ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
}

template <int N, int DVC>
static int launch(const Args& a, int R, cudaStream_t stream) {
  constexpr int smem = Layout<N, DVC>::bytes;
  static_assert(smem <= 227 * 1024, "one block's shared memory");
  cudaError_t e = cudaFuncSetAttribute(delta_walk_kernel<N, DVC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  kvb_launch(delta_walk_kernel<N, DVC>, dim3((unsigned)(a.H * (a.Dv / DVC)), (unsigned)R), dim3(kAll), smem, stream, a);
  return kvb_launch_result();
}

// 16 value columns a block, 32 where that still gives (nearly) every SM a block: one block fits an SM, and its time is the run's
// whatever its width.  A state of 128 rows leaves room for 16 only.
static int launch_any(const Args& a, int N, int R, cudaStream_t stream) {
  if (R <= 0) return 0;
  if (R > 65535 || a.H < 1 || !takes(a, N)) return KVB_ERR_BAD_SIZE;
  if (N == 128) return launch<128, 16>(a, R, stream);
  if ((long long)a.H * (a.Dv / 32) * R * 5 < (long long)kvb_sm_count() * 4) return launch<64, 16>(a, R, stream);
  return launch<64, 32>(a, R, stream);
}

}  // namespace delta_walk
