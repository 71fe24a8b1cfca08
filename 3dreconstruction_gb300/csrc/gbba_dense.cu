// Dense Cholesky solve of the reduced camera system S z = rhs.
//
// Replaces DenseSchurComplementSolver::SolveReducedLinearSystem (Eigen LLT,
// 3rdparty/ceres/internal/ceres/schur_complement_solver.cc:180-222) and the
// CXSparse factorisation the reference configures (:316-340): S is dense for
// the workloads here (every camera pair is covisible), so a blocked dense
// factorisation on the GPU is the right tool.
//
// Layout: S is n_pad x n_pad row-major (n_pad = round_up(n, 64)); only the
// lower triangle is read.  Padding rows/columns carry the identity, so every
// 64x64 tile is full and no kernel needs bounds checks.
//
// Algorithm (right-looking, block size 64, one launch sequence per panel k):
//   panel : S_kk = L_kk L_kk^T (by every CTA), y_k = L_kk^-1 b_k,
//           L_ik = S_ik L_kk^-T and b_i -= L_ik y_k for i > k
//   syrk  : S_ij -= L_ik L_jk^T for k < j <= i (trailing update)
// then the backward substitution L^T x = y, right-looking by block rows:
//   trsv_bwd(k): x_k = L_kk^-T y_k; y_j -= L_kj^T x_k for j < k.
// A non-positive pivot sets *flag (LINEAR_SOLVER_FAILURE in ceres terms).
// FP32: k_panel32 and k_syrk_tc or k_syrk_wide; FP64: k_panel64 and
// k_syrk_split; both: k_trsv_bwd.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <type_traits>

#include "gbba_internal.h"
#include "gbba_pivot.cuh"
#include "gbba_umma.cuh"

namespace gbba {

constexpr int NB = 64;

// Two padded 64x64 tiles (plus a few vectors) live in dynamic shared memory:
// 66.5 KB in FP64, above the 48 KB static limit (the backward substitution).
template <typename T>
__device__ __forceinline__ T (*tile_at(int i))[NB + 1] {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<T(*)[NB + 1]>(smem_raw + (size_t)i * NB * (NB + 1) * sizeof(T));
}
template <typename T>
__device__ __forceinline__ T* vec_at(int i) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<T*>(smem_raw + (size_t)2 * NB * (NB + 1) * sizeof(T) + (size_t)i * NB * sizeof(T));
}
template <typename T>
constexpr size_t dense_smem_bytes() { return (size_t)2 * NB * (NB + 1) * sizeof(T) + 2 * NB * sizeof(T); }

// Copy the 64x64 tile at src (row stride ld) into a padded shared tile.  All
// of a thread's global loads are issued before its shared stores so that
// their latencies overlap.
template <typename T>
__device__ __forceinline__ void load_tile(T (*dst)[NB + 1], const T* __restrict__ src, int64_t ld, int tid) {
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::n, PER_ROW = NB / W, ITER = NB * PER_ROW / 256;
  V v[ITER];
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = tid + it * 256, r = idx / PER_ROW, c = (idx % PER_ROW) * W;
    v[it] = *reinterpret_cast<const V*>(src + r * ld + c);
  }
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = tid + it * 256, r = idx / PER_ROW, c = (idx % PER_ROW) * W;
    const T* e = reinterpret_cast<const T*>(&v[it]);
#pragma unroll
    for (int w = 0; w < W; ++w) dst[r][c + w] = e[w];
  }
}

// Reciprocal of a pivot.  Single precision uses the fast hardware reciprocal
// (__fdividef, within 2 ulp for normal pivots): it sits on the elimination's
// critical path, and the FP32 factor only feeds LM steps whose acceptance is
// decided on the FP64 cost.
__device__ __forceinline__ float pivot_rcp(float d) { return __fdividef(1.0f, d); }

// Panel kb (FP32): the diagonal tile's factor and inverse, and one 64 x 64
// tile of the block column below it per CTA:
//   (with upd) S_kk -= P P^T and S_ib,kb -= L_ib,kb-1 P^T, P = L_kb,kb-1 (the
//              previous panel's update of this block column)
//   S_kk = L_kk L_kk^T, y_kb = L_kk^-1 b_kb,
//   L_ib,kb = S_ib,kb L_kk^-T,  b_ib -= L_ib,kb y_kb
//   (with ops) the tile's TF32 operands of the trailing update (k_syrk_tc).
// Every CTA factors the diagonal tile itself: that costs no time (the chain of
// pivots bounds it) and saves a kernel and its hand-over per panel.  S_kk and
// b_kb stay as they are (other CTAs may still have to read them): L_kk^-1 goes
// to Linv, y_kb to y.  A grid of one CTA without a tile serves the last panel.
//
// Warps 0..7 factor the tile in shared memory, four 16-column panels p
// (offset o = 16p):
//   1. warps 0..3: the 16 x 16 diagonal block, outer-product LDL^T with the
//      same row operations applied to an identity block (its inverse).  Of
//      the 16 columns l at pivot j, those right of j take the elimination of
//      the block, the others that of the identity (its row j ends at column
//      j); warp w holds columns w, w + 4, w + 8, w + 12 of all rows and a
//      pivot's column is passed on through shared memory, one barrier of the
//      four warps per pivot;
//   2. panel solve  L_ip = A_ip L_pp^-T  for the rows below;
//   3. trailing update  A_il -= L_ip L_lp^T  inside the tile.
// Warps 8..15 apply the previous panel's update to the CTA's own tile first,
// then form row p of 16 x 16 blocks of L^-1 as soon as diagonal block p is
// factored, Li_pJ = -Li_pp sum_{K=J..p-1} L_pK Li_KJ, beside steps 2, 3 and the
// next block's pivots.  All warps then multiply by L_kk^-T.
// A non-positive (or non-finite) pivot is replaced by 1 and sets *flag.
// Medium workload (94 panels): 22 us a panel, against 25 + 10 us for a
// diagonal kernel (one warp per block, pivots by shuffles) and a panel kernel.
constexpr int kPanel32Threads = 512;
constexpr int kTileLd = NB + 4;  // 16-byte aligned rows
constexpr int kTileF = NB * kTileLd;
constexpr size_t kPanel32Smem = sizeof(float) * (5 * (size_t)kTileF + 3 * 256 + 256 + 2 * NB);
// Operands of the TF32 trailing update, per 64 x 64 tile: [hi, lo][32 columns]
// of 64 rows x 128 bytes in 128-byte swizzle.
constexpr int kOpsPiece = 64 * 32;
constexpr int kOpsTile = 4 * kOpsPiece;

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// acc(4 x 4) += X Y^T over 64 columns, rows ty + 16 i of X and tx + 16 j of Y
// (tiles of row stride kTileLd: a quarter warp's 16-byte loads touch all banks).
__device__ __forceinline__ void tile_xyt(const float* X, const float* Y, int ty, int tx, float acc[4][4]) {
#pragma unroll 4
  for (int k4 = 0; k4 < NB; k4 += 4) {
    float x[4][4], y[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ld4<float>(X + (ty + 16 * i) * kTileLd + k4, x[i]);
      ld4<float>(Y + (tx + 16 * i) * kTileLd + k4, y[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][j] += x[i][k] * y[j][k];
  }
}
// One or two 64 x 64 tiles (row stride ld) into shared memory by 256 threads,
// all loads in flight at once.
__device__ __forceinline__ void load_tiles32(float* d0, const float* __restrict__ s0, float* d1,
                                             const float* __restrict__ s1, int64_t ld, int t) {
  float v[2][4][4];
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int64_t at = ((t + it * 256) >> 4) * ld + (t & 15) * 4;
    ld4<float>(s0 + at, v[0][it]);
    if (s1) ld4<float>(s1 + at, v[1][it]);
  }
#pragma unroll
  for (int it = 0; it < 4; ++it) {
    const int at = ((t + it * 256) >> 4) * kTileLd + (t & 15) * 4;
    st4<float>(d0 + at, v[0][it]);
    if (s1) st4<float>(d1 + at, v[1][it]);
  }
}

__global__ void __launch_bounds__(kPanel32Threads) k_panel32(float* __restrict__ S, int64_t ld, int kb, int nb,
                                                             float* __restrict__ Linv_all, float* __restrict__ b,
                                                             float* __restrict__ y, float* __restrict__ ops,
                                                             int* __restrict__ flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* A = reinterpret_cast<float*>(smem_raw);  // [64][kTileLd]: S_kk, overwritten by L_kk
  float* Li = A + kTileF;                         // [64][kTileLd]: L_kk^-1
  float* P = Li + kTileF;                         // [64][kTileLd]: L_kb,kb-1
  float* T1 = P + kTileF;                         // [64][kTileLd]: L_ib,kb-1, then L_ib,kb
  float* T2 = T1 + kTileF;                        // [64][kTileLd]: S_ib,kb
  float* scr = T2 + kTileF;                       // [3][16][16] products of the inverse blocks
  float* cb = scr + 3 * 256;                      // [16][16] the pivots' columns
  float* yb = cb + 256;                           // [64] b_kb
  float* yv = yb + NB;                            // [64] y_kb
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t off = (int64_t)kb * NB;
  const int64_t ib = kb + 1 + blockIdx.x;
  const bool has_tile = ib < nb;
  const bool upd = kb > 0;
  const int64_t r0 = ib * NB;
  // barriers; one of its own per diagonal block (an arrival must not run ahead
  // into a phase that the other side has not entered)
  enum { kBarA = 1, kBarDiag = 2, kBarB = 3, kBarStage = 4 /* .. 7 */ };
  if (tid < 256) {
    load_tiles32(A, S + off * ld + off, P, upd ? S + off * ld + off - NB : nullptr, ld, tid);
    if (tid < NB) yb[tid] = b[off + tid];
    if (upd) {
      __syncthreads();  // P is read by all
      const int ty = tid >> 4, tx = tid & 15;
      float acc[4][4] = {};
      tile_xyt(P, P, ty, tx, acc);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) A[(ty + 16 * i) * kTileLd + tx + 16 * j] -= acc[i][j];
    }
    bar_sync(kBarA, 256);
    for (int p = 0; p < 4; ++p) {
      const int o = 16 * p;
      // ---- 1. diagonal 16 x 16 block
      if (warp < 4) {
        const int r = lane & 15;
        const int l0 = warp + 4 * (lane >> 4), l1 = l0 + 8;  // this lane's columns of row r
        float a0 = A[(o + r) * kTileLd + o + l0], a1 = A[(o + r) * kTileLd + o + l1];
        float e0 = r == l0 ? 1.f : 0.f, e1 = r == l1 ? 1.f : 0.f;
        if (l0 == 0) cb[r] = a0;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          bar_sync(kBarDiag, 128);
          const float* col = cb + 16 * j;
          float d = col[j];
          const float cr = col[r], c0 = col[l0], c1 = col[l1];
          const float f0 = __shfl_sync(0xffffffffu, e0, j + (lane & 16)), f1 = __shfl_sync(0xffffffffu, e1, j + (lane & 16));
          if (!(d > 0.f && d - d == 0.f)) {  // non-positive, NaN or infinite pivot
            d = 1.f;
            if (tid == 0) {
              cb[17 * j] = 1.f;
              atomicExch(flag, 1);
            }
          }
          const float m = r > j ? cr * pivot_rcp(d) : 0.f;
          auto column = [&](int l, float& av, float& ev, float cl, float fl) {
            const bool right = l > j;
            const float v = fmaf(-m, right ? cl : fl, right ? av : ev);
            av = right ? v : av;
            ev = right ? ev : v;
            if (l == j + 1) cb[16 * (j + 1) + r] = av;
          };
          if (j + 1 < 8) {  // the next pivot's column first
            column(l0, a0, e0, c0, f0);
            column(l1, a1, e1, c1, f1);
          } else {
            column(l1, a1, e1, c1, f1);
            column(l0, a0, e0, c0, f0);
          }
        }
        bar_sync(kBarDiag, 128);
        // L_pp = L_u D^1/2, L_pp^-1 = D^-1/2 L_u^-1
        const float sd = sqrtf(cb[17 * r]), rs = 1.f / sd;
        const float rl0 = __shfl_sync(0xffffffffu, rs, l0), rl1 = __shfl_sync(0xffffffffu, rs, l1);
        A[(o + r) * kTileLd + o + l0] = l0 < r ? a0 * rl0 : (l0 == r ? sd : 0.f);
        A[(o + r) * kTileLd + o + l1] = l1 < r ? a1 * rl1 : (l1 == r ? sd : 0.f);
        Li[(o + r) * kTileLd + o + l0] = l0 <= r ? e0 * rs : 0.f;
        Li[(o + r) * kTileLd + o + l1] = l1 <= r ? e1 * rs : 0.f;
      }
      bar_sync(kBarA, 256);
      bar_arrive(kBarStage + p, kPanel32Threads);  // warps 8..15 take row p of L^-1
      if (p == 3) break;
      // ---- 2. panel solve: rows o+16..63, L_ic = sum_k A_ik Li_pp[c][k]
      const int rows = NB - o - 16;
      float pv[3];
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int idx = tid + u * 256;
        pv[u] = 0.f;
        if (idx < rows * 16) {
          const int i = o + 16 + (idx >> 4), c = idx & 15;
          float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k4 = 0; k4 < 16; k4 += 4) {
            float av[4], lv[4];
            ld4<float>(A + i * kTileLd + o + k4, av);
            ld4<float>(Li + (o + c) * kTileLd + o + k4, lv);
#pragma unroll
            for (int k = 0; k < 4; ++k) s4[k] += av[k] * lv[k];
          }
          pv[u] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
        }
      }
      __syncwarp();  // a row's 16 values are read by its half warp only
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int idx = tid + u * 256;
        if (idx < rows * 16) A[(o + 16 + (idx >> 4)) * kTileLd + o + (idx & 15)] = pv[u];
      }
      bar_sync(kBarA, 256);
      // ---- 3. trailing update inside the tile, a lower 16 x 16 block at a time
      {
        const int r = tid >> 4, c = tid & 15;
#pragma unroll
        for (int I = 1; I < 4; ++I)
#pragma unroll
          for (int J = 1; J <= I; ++J) {
            if (J <= p || I <= p) continue;
            const float* x = A + (16 * I + r) * kTileLd + o;
            const float* z = A + (16 * J + c) * kTileLd + o;
            float acc = 0.f;
#pragma unroll
            for (int k4 = 0; k4 < 16; k4 += 4) {
              float xv[4], zv[4];
              ld4<float>(x + k4, xv);
              ld4<float>(z + k4, zv);
#pragma unroll
              for (int k = 0; k < 4; ++k) acc += xv[k] * zv[k];
            }
            A[(16 * I + r) * kTileLd + 16 * J + c] -= acc;
          }
      }
      bar_sync(kBarA, 256);
    }
  } else {
    const int t = tid - 256, ty = t >> 4, tx = t & 15;
    if (has_tile) load_tiles32(T2, S + r0 * ld + off, T1, upd ? S + r0 * ld + off - NB : nullptr, ld, t);
    if (upd) {
      __syncthreads();
      if (has_tile) {
        float acc[4][4] = {};
        tile_xyt(T1, P, ty, tx, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) T2[(ty + 16 * i) * kTileLd + tx + 16 * j] -= acc[i][j];
      }
    }
    // the blocks of L^-1 above the diagonal
    for (int idx = t; idx < NB * NB; idx += 256)
      if ((idx & 63) >> 4 > idx >> 10) Li[(idx >> 6) * kTileLd + (idx & 63)] = 0.f;
    for (int I = 0; I < 4; ++I) {
      bar_sync(kBarStage + I, kPanel32Threads);
      // T_IJ = sum_{K=J}^{I-1} L_IK Li_KJ, then Li_IJ = -Li_II T_IJ
      for (int J = 0; J < I; ++J) {
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        for (int K = J; K < I; ++K) {
          const float* ar = A + (16 * I + ty) * kTileLd + 16 * K;
#pragma unroll
          for (int k4 = 0; k4 < 16; k4 += 4) {
            float av[4];
            ld4<float>(ar + k4, av);
#pragma unroll
            for (int k = 0; k < 4; ++k) s4[k] += av[k] * Li[(16 * K + k4 + k) * kTileLd + 16 * J + tx];
          }
        }
        scr[(J << 8) + t] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      }
      bar_sync(kBarB, 256);
      for (int J = 0; J < I; ++J) {
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        const float* lr = Li + (16 * I + ty) * kTileLd + 16 * I;
#pragma unroll
        for (int k4 = 0; k4 < 16; k4 += 4) {
          float lv[4];
          ld4<float>(lr + k4, lv);
#pragma unroll
          for (int k = 0; k < 4; ++k) s4[k] += lv[k] * scr[(J << 8) + (k4 + k) * 16 + tx];
        }
        Li[(16 * I + ty) * kTileLd + 16 * J + tx] = -((s4[0] + s4[1]) + (s4[2] + s4[3]));
      }
      bar_sync(kBarB, 256);
    }
  }
  __syncthreads();
  // y = L^-1 b (4 threads per row); L^-1 and y out; L_ib,kb = S_ib,kb L^-T into T1
  if (tid < 256) {
    const int r = tid >> 2, q = tid & 3;
    float v = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) v += Li[r * kTileLd + 16 * q + c] * yb[16 * q + c];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if (q == 0) {
      yv[r] = v;
      if (blockIdx.x == 0) y[off + r] = v;
    }
  }
  if (blockIdx.x == 0) {
    float* Lo = Linv_all + (int64_t)kb * NB * NB;
    for (int idx = tid; idx < NB * NB / 4; idx += kPanel32Threads) {
      float v[4];
      ld4<float>(Li + (idx >> 4) * kTileLd + (idx & 15) * 4, v);
      st4<float>(Lo + 4 * idx, v);
    }
  }
  if (!has_tile) return;
  {
    const int ty = tid >> 4, tx = tid & 15;  // rows ty, ty + 32; columns tx + 16 j
    float acc[2][4] = {};
#pragma unroll 4
    for (int k4 = 0; k4 < NB; k4 += 4) {
      float x[2][4], z[4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ld4<float>(T2 + (ty + 32 * i) * kTileLd + k4, x[i]);
#pragma unroll
      for (int j = 0; j < 4; ++j) ld4<float>(Li + (tx + 16 * j) * kTileLd + k4, z[j]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[i][j] += x[i][k] * z[j][k];
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) T1[(ty + 32 * i) * kTileLd + tx + 16 * j] = acc[i][j];
  }
  __syncthreads();
  for (int idx = tid; idx < NB * NB / 4; idx += kPanel32Threads) {
    const int r = idx >> 4, c4 = idx & 15;
    float v[4];
    ld4<float>(T1 + r * kTileLd + 4 * c4, v);
    st4<float>(S + (r0 + r) * ld + off + 4 * c4, v);
    if (ops) {
      float hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        hi[e] = umma::tf32_round(v[e]);
        lo[e] = v[e] - hi[e];
      }
      float* d = ops + ib * kOpsTile + (c4 >> 3) * kOpsPiece + r * 32 + (((c4 & 7) ^ (r & 7)) << 2);
      st4<float>(d, hi);
      st4<float>(d + 2 * kOpsPiece, lo);
    }
  }
  // b_ib -= L y: 4 threads per row, 16 columns each
  if (tid < 256) {
    const int r = tid >> 2, q = tid & 3;
    float s4 = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) s4 += T1[r * kTileLd + 16 * q + c] * yv[16 * q + c];
    s4 += __shfl_xor_sync(0xffffffffu, s4, 1);
    s4 += __shfl_xor_sync(0xffffffffu, s4, 2);
    if (q == 0) b[r0 + r] -= s4;
  }
}

// Trailing update over 128 x 128 output tiles (2 x 2 tiles of 64):
// S_IJ -= L_Ik L_Jk^T, K = 64 (panel kb).  blockIdx.x enumerates the lower
// triangle of 128-tiles over the 64-tiles first..nb-1; at the matrix edge a
// 128-tile holds one 64-tile row or column (the missing half is zero-filled
// and not stored), and the quarter of a diagonal 128-tile above the diagonal
// is not stored.  Operands are staged k-major (X^T, row stride 132) so that a
// thread's 8 rows and 8 columns at one k are 16-byte shared loads; thread
// (ty, tx) owns rows 8ty..8ty+7 x columns 8tx..8tx+7 of the output tile.
constexpr int kWideLd = 2 * NB + 4;
template <typename T>
constexpr size_t wide_smem_bytes() { return (size_t)2 * NB * kWideLd * sizeof(T); }

template <typename T>
__device__ __forceinline__ void load_panel_t(T* __restrict__ dst, const T* __restrict__ S, int64_t ld, int64_t row0,
                                             int64_t col0, int valid_rows, int tid) {
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::n, ITER = 2 * NB * NB / W / 256;
  V v[ITER];
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = tid + it * 256, kv = idx / (2 * NB), r = idx % (2 * NB);
    if (r < valid_rows) v[it] = *reinterpret_cast<const V*>(S + (row0 + r) * ld + col0 + kv * W);
    else {
      T* z = reinterpret_cast<T*>(&v[it]);
#pragma unroll
      for (int w = 0; w < W; ++w) z[w] = T(0);
    }
  }
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = tid + it * 256, kv = idx / (2 * NB), r = idx % (2 * NB);
    const T* e = reinterpret_cast<const T*>(&v[it]);
#pragma unroll
    for (int w = 0; w < W; ++w) dst[(kv * W + w) * kWideLd + r] = e[w];
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_syrk_wide(T* __restrict__ S, int64_t ld, int kb, int first, int nb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* XiT = reinterpret_cast<T*>(smem_raw);
  T* XjT = XiT + NB * kWideLd;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int64_t t = blockIdx.x;
  int64_t R = (int64_t)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((R + 1) * (R + 2) / 2 <= t) ++R;
  while (R * (R + 1) / 2 > t) --R;
  const int64_t C = t - R * (R + 1) / 2;
  const int64_t ib0 = first + 2 * R, jb0 = first + 2 * C;
  const int rows_i = ib0 + 1 < nb ? 2 * NB : NB, rows_j = jb0 + 1 < nb ? 2 * NB : NB;
  const int64_t c0 = (int64_t)kb * NB;
  load_panel_t<T>(XiT, S, ld, ib0 * NB, c0, rows_i, tid);
  load_panel_t<T>(XjT, S, ld, jb0 * NB, c0, rows_j, tid);
  __syncthreads();
  // rows {4ty+i, 64+4ty+i} x columns {4tx+j, 64+4tx+j}: the 16-byte shared
  // loads of a quarter warp cover 128 contiguous bytes (no bank conflicts)
  T acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = T(0);
#pragma unroll 4
  for (int k = 0; k < NB; ++k) {
    T xa[8], xb[8];
    ld4<T>(XiT + k * kWideLd + ty * 4, xa);
    ld4<T>(XiT + k * kWideLd + NB + ty * 4, xa + 4);
    ld4<T>(XjT + k * kWideLd + tx * 4, xb);
    ld4<T>(XjT + k * kWideLd + NB + tx * 4, xb + 4);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] += xa[i] * xb[j];
  }
#pragma unroll
  for (int qi = 0; qi < 2; ++qi)
#pragma unroll
    for (int qj = 0; qj < 2; ++qj) {
      const int64_t rb = ib0 + qi, cb = jb0 + qj;
      if (rb >= nb || cb >= nb || rb < cb) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        T* p = S + (rb * NB + ty * 4 + i) * ld + cb * NB + tx * 4;
        T v[4];
        ld4<T>(p, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] -= acc[4 * qi + i][4 * qj + j];
        st4<T>(p, v);
      }
    }
}

// The same trailing update on the tensor cores (FP32 path): one CTA per 128 x
// 64 output (two row tiles I >= J and the column tile J), acc = L_I L_J^T over
// the panel's 64 columns by tcgen05 kind::tf32 MMAs in 3xTF32 (FP32 accuracy),
// accumulated in tensor memory; the epilogue subtracts it from S.  The
// operands' hi and lo parts were laid out by k_panel32 (once per tile instead
// of once per output tile) and arrive by bulk copies; S's rows are loaded while
// they do.  Two CTAs share an SM, so that one's copies and epilogue run beside
// the other's.  Bound by S's traffic: the medium workload's first update moves
// 144 MB of S and takes 40 us (91 us with 128 x 128 tiles that split their
// own operands).
// A bounded wait that runs out sets *flag = 6 (the step is then rejected) and
// the tile is left alone.
struct TcSmem {  // 1024-byte aligned (kTcSmem leaves room for it)
  float a[4][2 * kOpsPiece];  // [hi, lo][32 columns], the two row tiles one after the other
  float b[4][kOpsPiece];
  uint64_t load_bar, mma_bar;
  uint32_t tmem_base, fail;
};
constexpr size_t kTcSmem = sizeof(TcSmem) + 1024;
constexpr int kSyrkTcThreads = 256;
__global__ void __launch_bounds__(kSyrkTcThreads, 2) k_syrk_tc(float* __restrict__ S, int64_t ld, int j0, int nb,
                                                               const float* __restrict__ ops, int* __restrict__ flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TcSmem& g = *reinterpret_cast<TcSmem*>(smem_raw + ((1024 - (umma::smem_addr(smem_raw) & 1023)) & 1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // CTA t: column tile jb = j0, j0 + 1, ... with ceil((nb - jb) / 2) pairs of row tiles each
  int jb = j0, t = blockIdx.x;
  while (t >= (nb - jb + 1) / 2) {
    t -= (nb - jb + 1) / 2;
    ++jb;
  }
  const int ib = jb + 2 * t;
  const bool two = ib + 1 < nb;
  if (tid == 0) {
    umma::mbar_init(&g.load_bar, 1);
    umma::mbar_init(&g.mma_bar, 1);
    g.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    constexpr uint32_t kBytes = kOpsPiece * 4;
    const float* pa = ops + ib * (int64_t)kOpsTile;
    const float* pb = ops + jb * (int64_t)kOpsTile;
    umma::mbar_expect(&g.load_bar, (two ? 12 : 8) * kBytes);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      umma::bulk_load(g.a[p], pa + p * kOpsPiece, kBytes, &g.load_bar);
      if (two) umma::bulk_load(g.a[p] + kOpsPiece, pa + kOpsTile + p * kOpsPiece, kBytes, &g.load_bar);
      umma::bulk_load(g.b[p], pb + p * kOpsPiece, kBytes, &g.load_bar);
    }
  }
  if (warp == 0) {
    __syncwarp();
    umma::tmem_alloc(&g.tmem_base, 64);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tm = g.tmem_base;
  // S: thread t takes 16-byte pieces t, t + 256, ... of the rows (16 a row)
  float* out = S + (int64_t)ib * NB * ld + (int64_t)jb * NB + 4 * (tid & 15);
  const int rows = two ? 2 * NB : NB;
  float4 x[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int r = (tid >> 4) + 16 * e;
    if (r < rows) x[e] = *reinterpret_cast<const float4*>(out + (int64_t)r * ld);
  }
  if (tid == 0) {
    constexpr uint32_t idesc = umma::idesc_tf32(128, 64);
    const uint64_t da = umma::smem_desc_sw128(umma::smem_addr(g.a[0]));
    const uint64_t db = umma::smem_desc_sw128(umma::smem_addr(g.b[0]));
    constexpr uint32_t kA = sizeof(g.a[0]) / 16, kB = sizeof(g.b[0]) / 16;
    const bool ok = umma::mbar_wait(&g.load_bar, 0);
    if (ok) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {  // 8 columns: piece k / 4, 32 bytes each
        const uint32_t ca = (k >> 2) * kA + 2 * (k & 3), cb = (k >> 2) * kB + 2 * (k & 3);
        umma::mma_tf32(tm, da + 2 * kA + ca, db + cb, idesc, k != 0);  // lo hi
        umma::mma_tf32(tm, da + ca, db + 2 * kB + cb, idesc, 1);       // hi lo
        umma::mma_tf32(tm, da + ca, db + cb, idesc, 1);                // hi hi
      }
    }
    umma::mma_commit(&g.mma_bar);
    if (!umma::mbar_wait(&g.mma_bar, 0) || !ok) g.fail = 1;
  }
  __syncthreads();  // one thread polls, the others wait here
  const bool ok = g.fail == 0;
  umma::fence_after_sync();
  if (ok) {
    // accumulator rows (a tensor-memory lane each) through shared memory to
    // the threads that hold S's pieces
    constexpr int kLd = NB + 4;
    float* acc = g.a[0];
    {
      float v[32];
      const int r = 32 * (warp & 3) + lane, c0 = 32 * (warp >> 2);
      umma::tmem_ld32(tm + ((uint32_t)(32 * (warp & 3)) << 16) + c0, v);
#pragma unroll
      for (int e = 0; e < 32; e += 4) st4<float>(acc + r * kLd + c0 + e, v + e);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int r = (tid >> 4) + 16 * e;
      if (r >= rows) continue;
      float v[4];
      ld4<float>(acc + r * kLd + 4 * (tid & 15), v);
      x[e].x -= v[0];
      x[e].y -= v[1];
      x[e].z -= v[2];
      x[e].w -= v[3];
      *reinterpret_cast<float4*>(out + (int64_t)r * ld) = x[e];
    }
  } else if (tid == 0) {
    atomicExch(flag, 6);
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tm, 64);
}

// Backward substitution of block row kb: x_k = L_kk^-T y_k in every CTA, then
// y_j -= L_kj^T x_k in CTA j.  kBlocks: Linv_all holds k_panel64's tiles as they
// are (inverses of the diagonal 16 x 16 blocks, L below them), and x_k is
// substituted by those blocks instead of taken from the inverse of the tile.
template <typename T, bool kBlocks = false>
__global__ void __launch_bounds__(256) k_trsv_bwd(const T* __restrict__ S, int64_t ld, int kb, const T* __restrict__ Linv_all,
                                                  T* __restrict__ b, T* __restrict__ x) {
  T(*Li)[NB + 1] = tile_at<T>(0);
  T* yk = vec_at<T>(0);
  T* xk = vec_at<T>(1);
  const int tid = threadIdx.x;
  const int64_t k0 = (int64_t)kb * NB;
  // the next block row's kernel may start now (programmatic dependent
  // launch): it touches b only after its griddepcontrol.wait
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  load_tile<T>(Li, Linv_all + (int64_t)kb * NB * NB, NB, tid);
  const int jb = blockIdx.x;
  const int c = tid & (NB - 1), q = tid >> 6;
  // this block's column of L_kj^T (written by the factorisation, complete
  // before the backward substitution began) is loaded before the wait
  T v[NB / 4];
  if (jb != kb) {
    const T* col = S + (k0 + q) * ld + (int64_t)jb * NB + c;
#pragma unroll
    for (int t = 0; t < NB / 4; ++t) v[t] = col[(int64_t)(4 * t) * ld];
  }
  // y_k and the b entries this kernel updates were written by the previous
  // block row's kernel: wait for it, and read b through L2
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (tid < NB) yk[tid] = __ldcg(b + k0 + tid);
  __syncthreads();
  if constexpr (kBlocks) {
    // 16 lanes a row of the block: the rows below it, then its inverse
    const int i = tid >> 4, l = tid & 15;
#pragma unroll
    for (int I = 3; I >= 0; --I) {
      T s = T(0);
#pragma unroll
      for (int K = I + 1; K < 4; ++K) s = fma(Li[16 * K + l][16 * I + i], xk[16 * K + l], s);
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (l == 0) yk[16 * I + i] -= s;
      __syncthreads();
      s = l >= i ? Li[16 * I + l][16 * I + i] * yk[16 * I + l] : T(0);
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (l == 0) xk[16 * I + i] = s;
      __syncthreads();
    }
  } else {
    if (tid < NB) {
      T s = T(0);
#pragma unroll 16
      for (int r = 0; r < NB; ++r) s += Li[r][tid] * yk[r];  // L^-1 is lower: zeros for r < tid
      xk[tid] = s;
    }
    __syncthreads();
  }
  if (jb == kb) {
    if (tid < NB) x[k0 + tid] = xk[tid];
    return;
  }
  // y_j -= L_kj^T x_k : thread (q, c) sums rows q, q+4, ... of column c;
  // consecutive threads read consecutive columns of a row (coalesced)
  T s = T(0);
#pragma unroll
  for (int t = 0; t < NB / 4; ++t) s += v[t] * xk[q + 4 * t];
  T* part = &Li[0][0];  // L_kk^-1 is no longer needed
  __syncthreads();
  part[q * NB + c] = s;
  __syncthreads();
  if (tid < NB)
    b[(int64_t)jb * NB + tid] = __ldcg(b + (int64_t)jb * NB + tid) -
                                (part[tid] + part[NB + tid] + part[2 * NB + tid] + part[3 * NB + tid]);
}

// ---------------------------------------------------------------- FP64 factorisation
// GB300 issues two FP64 FMAs a clock per multiprocessor, so in FP64 a 64 x 64
// x 64 tile product takes 66 us on one SM.  The FP64 path therefore
//   - splits a panel over all SMs (k_panel64: the diagonal tile factored by
//     every CTA, at no cost in time, with 16 rows of the panel per CTA);
//   - keeps the trailing update off the FP64 pipe (k_syrk_split): the products
//     are formed exactly on the tensor cores from FP16 digits.
// Factorisation and solve, against 64 x 64 tiles on the FP64 pipe: n = 114
// 0.14 ms (0.40), n = 1,806 2.2 ms (7.9), n = 2,388 3.2 ms (11.7), n = 5,988
// 17.4 ms (81.5); backward error the same (5.6e-16 at n = 2,388).
//
// Digits (error-free transformation of Ozaki, Ogita, Oishi and Rump, "Error-
// free transformations of matrix multiplication", 2012): row i of the panel is
// scaled by 2^e_i, its largest |l_ik| 2^e_i in [1/2, 1), and rounded to 62
// fractional bits, q = sum_p d_p 2^(56 - 8 p) with eight balanced digits
// |d_p| <= 128.  The digit products of equal weight p + q = g, g = 0..7, are
// summed in one FP32 accumulator each: at most 8 products of 64 terms of at
// most 2^14, so every partial sum is an integer of at most 2^23, exact in
// FP32.  The eight sums make a 62-bit integer with integer arithmetic.  Left out
// are the products of weight 8 and more, seven pairs of digits of 64 terms of
// at most 2^14 each: at most 2^-53.2 max_k |l_ik| max_k |l_jk| a panel, and about
// 2^-59 of it when the digits' signs are random.  The two maxima are at most
// sqrt(S_ii S_jj), so normwise this is within the rounding of a Cholesky
// factorisation in FP64; an entry whose rows have their large values in
// different columns keeps that absolute error, where an FMA would round each
// of its small products relative to itself.
constexpr int kDigits = 8;
constexpr int kDigitTile = 64 * 64;                            // one digit of a 64 x 64 tile (8 KB of FP16)
constexpr size_t kTileDigitBytes = (size_t)kDigits * kDigitTile * 2;

// Panel kb: [L_kk; L_ik] of the diagonal tile and of this CTA's rows below it,
// y_kb = L_kk^-1 b_kb, b_i -= L_ik y_kb and the digits of the rows.  L_kk with
// its diagonal 16 x 16 blocks inverted goes to the tile's place in Linv, y_kb
// to y: S_kk and b_kb stay as they are, other CTAs may still have to read them.  CTA j holds the rows
// row0 + j R .. + R - 1 (row0 = 64 (kb + 1), R a multiple of 16; the grid has
// at least one CTA, which may hold no rows) under a copy of the diagonal tile
// and the row b_kb^T, and factors them together, 16 columns at a time:
//   1. warps 0..3, one per scheduler (each holds a quarter of the SM's FP64
//      lanes): the 16 x 16 diagonal block, LDL^T with the row operations
//      applied to an identity block (its inverse).  Of the 16 columns l at
//      pivot j, those right of j take the elimination of the block, the
//      others that of the identity (its row j ends at column j); warp w holds
//      columns w, w + 4, w + 8, w + 12 and passes a pivot's column on through
//      shared memory, with one barrier of the four warps per pivot;
//   2. L_ip = A_ip L_pp^-T for all rows below (a thread takes columns j and
//      15 - j of a row: 17 products for the two, whatever j);
//   3. A_il -= L_ip L_lp^T for the columns to the right.
// Bound by FP64: about 100,000 FMAs for 16 rows (25 us at two a clock) and the
// chain of 64 pivots (0.4 us each: reciprocal, multiplier, update).  nblk (4,
// less in the last tile) is the number of 16-column blocks that hold
// unknowns; the padding behind them is the identity already.
// n = 2,388 (38 panels): 55 us a panel, against 199 + 134 us for a diagonal
// kernel and one 64 x 64 tile per CTA.
// 512 threads of 72 registers: no two CTAs of a panel share an SM (its FP64
// pipe), and one of them leaves the registers for one CTA of the bulk update.
constexpr int kPanelThreads = 512;
constexpr int kPanelLd = 66;
constexpr int kPanelMaxRows = 64;
inline size_t panel64_smem(int R) { return sizeof(double) * ((size_t)(64 + R + 1) * kPanelLd + 4 * 16 * 18 + 256); }
__global__ void __maxnreg__(72) k_panel64(double* __restrict__ S, int64_t ld, int kb, int R,
                                                           int nblk, double* __restrict__ Linv_all,
                                                           double* __restrict__ b, double* __restrict__ y,
                                                           int32_t* __restrict__ ex, __half* __restrict__ digits,
                                                           int* __restrict__ flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = reinterpret_cast<double*>(smem_raw);         // rows 0..63 tile, 64..64+R-1 rows, 64+R: b^T
  double* Li = A + (size_t)(64 + R + 1) * kPanelLd;        // [4][16][18] inverses of the diagonal blocks
  double* cb = Li + 4 * 16 * 18;                           // [16][16] the pivots' columns
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t off = (int64_t)kb * NB;
  const int64_t row0 = off + NB + (int64_t)blockIdx.x * R;
  const int rows = (int)max((int64_t)0, min((int64_t)R, ld - row0));  // a multiple of 16
  const int nr = 64 + rows;                                           // rows without b^T
  for (int idx = tid; idx < nr * 32; idx += kPanelThreads) {
    const int r = idx >> 5, c = (idx & 31) * 2;
    const double2 v = *reinterpret_cast<const double2*>(S + (r < 64 ? off + r : row0 + r - 64) * ld + off + c);
    *reinterpret_cast<double2*>(A + r * kPanelLd + c) = v;
  }
  double* yb = A + nr * kPanelLd;
  if (tid < 64) yb[tid] = b[off + tid];
  __syncthreads();
  for (int p = 0; p < nblk; ++p) {
    const int o = 16 * p;
    double* Lp = Li + p * 16 * 18;
    if (warp < 4) {
      const int r = lane & 15;
      const int l0 = warp + 4 * (lane >> 4), l1 = l0 + 8;  // this lane's columns of row r
      double a0 = A[(o + r) * kPanelLd + o + l0], a1 = A[(o + r) * kPanelLd + o + l1];
      double e0 = r == l0 ? 1.0 : 0.0, e1 = r == l1 ? 1.0 : 0.0;
      if (l0 == 0) cb[r] = a0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const double* col = cb + 16 * j;
        double d = col[j];
        const double cr = col[r], c0 = col[l0], c1 = col[l1];
        const double f0 = __shfl_sync(0xffffffffu, e0, j + (lane & 16)), f1 = __shfl_sync(0xffffffffu, e1, j + (lane & 16));
        if (!positive_finite(d)) {  // non-positive, NaN or infinite pivot
          d = 1.0;
          if (tid == 0) {
            cb[17 * j] = 1.0;
            atomicExch(flag, 1);
          }
        }
        const double m = r > j ? -cr * rcp_series(d) : 0.0;
        // the next pivot's column first: the other warps wait for it
        auto column = [&](int l, double& av, double& ev, double cl, double fl) {
          const bool right = l > j;
          const double v = fma(m, right ? cl : fl, right ? av : ev);
          av = right ? v : av;
          ev = right ? ev : v;
          if (l == j + 1) cb[16 * (j + 1) + r] = av;
        };
        if (j + 1 < 8) {
          column(l0, a0, e0, c0, f0);
          column(l1, a1, e1, c1, f1);
        } else {
          column(l1, a1, e1, c1, f1);
          column(l0, a0, e0, c0, f0);
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      // L_pp = L_u D^1/2, L_pp^-1 = D^-1/2 L_u^-1
      double sd, rs;
      sqrt_newton(cb[17 * r], sd, rs);
      const double rl0 = __shfl_sync(0xffffffffu, rs, l0), rl1 = __shfl_sync(0xffffffffu, rs, l1);
      A[(o + r) * kPanelLd + o + l0] = l0 < r ? a0 * rl0 : (l0 == r ? sd : 0.0);
      A[(o + r) * kPanelLd + o + l1] = l1 < r ? a1 * rl1 : (l1 == r ? sd : 0.0);
      Lp[r * 18 + l0] = l0 <= r ? e0 * rs : 0.0;
      Lp[r * 18 + l1] = l1 <= r ? e1 * rs : 0.0;
    }
    __syncthreads();
    // rows below the block, and b^T: columns j and 15 - j per thread
    {
      const int j = tid & 7, first = o + 16, total = nr + 1 - first;
      const double* l0 = Lp + j * 18;
      const double* l1 = Lp + (15 - j) * 18;
      for (int i0 = 0; i0 < total; i0 += 4 * (kPanelThreads / 8)) {
        double s0[4], s1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * (kPanelThreads / 8) + (tid >> 3);
          s0[u] = s1[u] = 0.0;
          if (i >= total) continue;
          const double* ar = A + (first + i) * kPanelLd + o;
          double acc = 0.0;
#pragma unroll
          for (int s = 0; s < 17; ++s) {
            const bool lo = s <= j;
            const int k = lo ? s : s - j - 1;
            if (s == j + 1) {
              s0[u] = acc;
              acc = 0.0;
            }
            acc = fma(ar[k], lo ? l0[k] : l1[k], acc);
          }
          s1[u] = acc;
        }
        // a row's 16 values are read by the eight threads of its quarter warp only
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = i0 + u * (kPanelThreads / 8) + (tid >> 3);
          if (i >= total) continue;
          double* ar = A + (first + i) * kPanelLd + o;
          ar[j] = s0[u];
          ar[15 - j] = s1[u];
        }
      }
    }
    __syncthreads();
    if (p + 1 < nblk) {
      // columns to the right: the tile's lower 4 x 4 blocks, then the rows and b^T
      const int m = 48 - o, nbk = m / 4, ntri = nbk * (nbk + 1) / 2 * 16, total = ntri + (rows + 1) * m;
      const double* base = A + o;
      for (int t = tid; t < total; t += kPanelThreads) {
        int i, l;
        if (t < ntri) {
          const int blk = t >> 4;
          int bi = (int)((sqrtf(8.0f * (float)blk + 1.0f) - 1.0f) * 0.5f);
          while ((bi + 1) * (bi + 2) / 2 <= blk) ++bi;
          while (bi * (bi + 1) / 2 > blk) --bi;
          i = o + 16 + 4 * bi + ((t >> 2) & 3);
          l = o + 16 + 4 * (blk - bi * (bi + 1) / 2) + (t & 3);
        } else {
          const int u = t - ntri;
          i = 64 + u / m;
          l = o + 16 + u % m;
        }
        const double* x = base + i * kPanelLd;
        const double* y = base + l * kPanelLd;
        double s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const double2 xv = *reinterpret_cast<const double2*>(x + k), yv = *reinterpret_cast<const double2*>(y + k);
          s0 = fma(xv.x, yv.x, s0);
          s1 = fma(xv.y, yv.y, s1);
        }
        A[i * kPanelLd + l] -= s0 + s1;
      }
      __syncthreads();
    }
  }
  if (blockIdx.x == 0) {  // every CTA holds the same factor of the tile
    double* Lo = Linv_all + (int64_t)kb * NB * NB;
    for (int idx = tid; idx < 64 * 64; idx += kPanelThreads) {
      const int r = idx >> 6, c = idx & 63, p = r >> 4;
      double v = 0.0;
      if (p != (c >> 4)) v = c < r ? A[r * kPanelLd + c] : 0.0;
      else v = p < nblk ? Li[(p * 16 + (r & 15)) * 18 + (c & 15)] : (r == c ? 1.0 : 0.0);
      Lo[idx] = v;
    }
    if (tid < 64) y[off + tid] = yb[tid];
  }
  // this CTA's rows of L, their digits and b_i -= L_i y
  for (int idx = tid; idx < rows * 32; idx += kPanelThreads) {
    const int r = idx >> 5, c = (idx & 31) * 2;
    *reinterpret_cast<double2*>(S + (row0 + r) * ld + off + c) =
        *reinterpret_cast<const double2*>(A + (64 + r) * kPanelLd + c);
  }
  for (int idx = tid; idx < rows * 8; idx += kPanelThreads) {
    const int r = idx >> 3, k8 = idx & 7;
    const int64_t i = row0 + r;
    const double* x = A + (64 + r) * kPanelLd + 8 * k8;
    // the row's exponent from its largest entry (its eight threads are a
    // quarter warp); rows whose entries are not finite belong to a failed
    // factorisation and take any value
    double big = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) big = fmax(big, fabs(x[k]));
    const unsigned mask = __activemask();
#pragma unroll
    for (int w = 1; w < 8; w <<= 1) big = fmax(big, __shfl_xor_sync(mask, big, w));
    int xp = 0;
    if (big > 0.0 && big < CUDART_INF) frexp(big, &xp);  // big < 2^xp
    if (k8 == 0) ex[i] = -xp;
    unsigned long long q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double lim = 4611686018427387392.0;  // below 2^62
      const double v = fmin(fmax(scalbn(x[k], 62 - xp), -lim), lim);
      q[k] = ((unsigned long long)__double2ll_rn(v) + 0x0080808080808080ull) ^ 0x8000000000000000ull;
    }
    // digit p of the tile of row i: rows of 128 bytes in 128-byte swizzle
    __half* dst = digits + (i >> 6) * (kDigits * (int64_t)kDigitTile) + (i & 63) * 64 + ((k8 ^ (int)(i & 7)) * 8);
    const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1024 + 128
#pragma unroll
    for (int p = 0; p < kDigits; ++p) {
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // 1024 + byte has the bits 0x6400 | byte
        const uint32_t u = 0x64006400u | (uint32_t)((q[2 * k] >> (56 - 8 * p)) & 0xff) |
                           ((uint32_t)((q[2 * k + 1] >> (56 - 8 * p)) & 0xff) << 16);
        const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&u), bias);
        w[k] = *reinterpret_cast<const uint32_t*>(&v);
      }
      *reinterpret_cast<uint4*>(dst + p * kDigitTile) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  for (int r = tid >> 2; r < rows; r += kPanelThreads / 4) {  // rows is a multiple of 16: whole warps
    const int q = tid & 3;
    const double* x = A + (64 + r) * kPanelLd + q;
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 64; c += 4) s = fma(x[c], yb[q + c], s);
    const unsigned mask = __activemask();
    s += __shfl_xor_sync(mask, s, 1);
    s += __shfl_xor_sync(mask, s, 2);
    if (q == 0) b[row0 + r] -= s;
  }
}

// Trailing update of panel kb on the tensor cores from the panel's digits:
// S_IJ -= L_I L_J^T for the 64-column tiles J >= j0 and the row tiles I >= J,
// one CTA per two row tiles and N of a tile's columns.  The eight sums of
// digit products take N accumulator columns each; the operands arrive by bulk
// copies with a barrier per digit, so that the MMAs start on the first.  The
// epilogue makes each output's eight sums one FP64 number with integer
// arithmetic and spends one FP64 instruction on it instead of 64.
// N = 16 for the block column that the next panel waits for (four CTAs per
// pair of tiles, a short epilogue: 11 us).  N = 32 for the bulk: its 160 KB of
// operands leave room for a CTA of the next panel on the same SM, which runs
// on the FP64 pipe meanwhile (with N = 64 and 192 KB the two take turns:
// 4.2 ms against 3.2 ms for n = 2,388).
// A bounded wait that runs out sets *flag = 6 (the step is then rejected).
template <int N>
struct SplitSmem {  // 1024-byte aligned (split_smem_bytes leaves room for it)
  __half a[kDigits][2 * kDigitTile];
  __half b[kDigits][N * 64];
  uint64_t load_bar[kDigits], mma_bar;
  uint32_t tmem_base, fail;
  int32_t col_ex[N];
};
template <int N>
constexpr size_t split_smem_bytes() { return sizeof(SplitSmem<N>) + 1024; }
// v 2^e (rounded to nearest) without FP64 instructions; zero below the normal range.
__device__ __forceinline__ double scaled_integer(long long v, int e) {
  const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  const int n = __clzll((long long)m);
  const int ef = 1023 + 63 - n + e;  // exponent field
  if (m == 0 || ef < 1) return 0.0;
  // the rounded mantissa's leading one (and a carry out of it) adds to the field below it
  const unsigned long long bits = ((unsigned long long)(ef - 1) << 52) + (((m << n) >> 11) + (((m << n) >> 10) & 1));
  return __longlong_as_double((long long)(bits | ((unsigned long long)v & 0x8000000000000000ull)));
}
constexpr int kSplitThreads = 256;
constexpr int kBulkN = 32;
template <int N>
__global__ void __maxnreg__(112) k_syrk_split(double* __restrict__ S, int64_t ld, int j0, int nb,
                                                              const __half* __restrict__ digits,
                                                              const int32_t* __restrict__ ex, int* __restrict__ flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SplitSmem<N>& g = *reinterpret_cast<SplitSmem<N>*>(smem_raw + ((1024 - (umma::smem_addr(smem_raw) & 1023)) & 1023));
  constexpr int kCols = 8 * N;    // accumulator columns
  constexpr int C = N / 2;        // output columns per thread
  constexpr int CH = C > 16 ? 16 : C;  // of which loaded at a time
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // CTA t: column tile jb = j0, j0 + 1, ... with ceil((nb - jb) / 2) pairs of row tiles each
  int jb = j0, t = blockIdx.x / (64 / N);
  const int cj = (blockIdx.x % (64 / N)) * N;  // first column inside the tile
  while (t >= (nb - jb + 1) / 2) {
    t -= (nb - jb + 1) / 2;
    ++jb;
  }
  const int ib = jb + 2 * t;
  const bool two = ib + 1 < nb;
  if (tid == 0) {
#pragma unroll
    for (int p = 0; p < kDigits; ++p) umma::mbar_init(&g.load_bar[p], 1);
    umma::mbar_init(&g.mma_bar, 1);
    g.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const __half* da = digits + ib * (kDigits * (int64_t)kDigitTile);
    const __half* db = digits + jb * (kDigits * (int64_t)kDigitTile) + cj * 64;
    constexpr uint32_t kBytes = kDigitTile * 2, kBytesB = N * 64 * 2;
#pragma unroll
    for (int p = 0; p < kDigits; ++p) {
      umma::mbar_expect(&g.load_bar[p], (two ? 2 * kBytes : kBytes) + kBytesB);
      umma::bulk_load(g.a[p], da + p * kDigitTile, kBytes, &g.load_bar[p]);
      if (two) umma::bulk_load(g.a[p] + kDigitTile, da + (kDigits + p) * (int64_t)kDigitTile, kBytes, &g.load_bar[p]);
      umma::bulk_load(g.b[p], db + p * kDigitTile, kBytesB, &g.load_bar[p]);
    }
  }
  if (tid >= 64 && tid < 64 + N) g.col_ex[tid - 64] = ex[(int64_t)jb * NB + cj + tid - 64];
  if (warp == 0) {
    __syncwarp();
    umma::tmem_alloc(&g.tmem_base, kCols);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tm = g.tmem_base;
  // this thread's outputs: a row of the pair of tiles, half of the columns
  const int r = 32 * (warp & 3) + lane, c0 = C * (warp >> 2);
  const bool mine = r < 64 || two;  // uniform over a warp
  const int64_t row = (int64_t)ib * NB + r;
  double* out = S + row * ld + (int64_t)jb * NB + cj + c0;
  double x[CH];  // the first ones are loaded while the operands arrive
  auto load = [&](int h) {
#pragma unroll
    for (int c = 0; c < CH; c += 2) {
      const double2 w = *reinterpret_cast<const double2*>(out + h + c);
      x[c] = w.x;
      x[c + 1] = w.y;
    }
  };
  int ei = 0;
  if (mine) {
    ei = ex[row];
    load(0);
  }
  if (tid == 0) {
    constexpr uint32_t idesc = umma::idesc_f16(128, N);
    // descriptors advance by (bytes / 16)
    const uint64_t da = umma::smem_desc_sw128(umma::smem_addr(g.a[0]));
    const uint64_t db = umma::smem_desc_sw128(umma::smem_addr(g.b[0]));
    constexpr uint32_t kStepA = sizeof(g.a[0]) / 16, kStepB = sizeof(g.b[0]) / 16;
    bool ok = true;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) {  // digit weights p + q = s: N accumulator columns each
      ok = umma::mbar_wait(&g.load_bar[s], 0) && ok;
      if (!ok) continue;
#pragma unroll
      for (int p = 0; p <= s; ++p)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma::mma_f16(tm + N * s, da + (p * kStepA + 2 * k), db + ((s - p) * kStepB + 2 * k), idesc, (p | k) != 0);
    }
    umma::mma_commit(&g.mma_bar);
    if (!umma::mbar_wait(&g.mma_bar, 0) || !ok) g.fail = 1;
  }
  // one thread polls, the others wait at the barrier: 256 polling threads
  // take the shared memory's bandwidth from the copies (16 us against 9)
  __syncthreads();
  const bool ok = g.fail == 0;
  umma::fence_after_sync();
  if (ok) {
    if (mine) {
      const uint32_t lanes = tm + ((uint32_t)(32 * (warp & 3)) << 16) + c0;
#pragma unroll 1
      for (int h = 0; h < C; h += CH) {
        if (h) load(h);
#pragma unroll
        for (int c8 = 0; c8 < CH; c8 += 8) {
          uint32_t v[kDigits][8];
#pragma unroll
          for (int s = 0; s < kDigits; ++s) umma::tmem_ld8(lanes + N * s + h + c8, v[s]);
          umma::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            int d[kDigits];
#pragma unroll
            for (int s = 0; s < kDigits; ++s) d[s] = __float2int_rn(__uint_as_float(v[s][c]));
            // sum_s d_s 2^(-12 - 8 s) in units of 2^-56, |sum| < 64
            long long sum = 0;
#pragma unroll
            for (int s = 0; s < 6; ++s) sum = sum * 256 + d[s];
            sum = sum * 16 + ((d[6] * 256 + d[7] + 2048) >> 12);
            x[c8 + c] -= scaled_integer(sum, -56 - ei - g.col_ex[c0 + h + c8 + c]);
          }
        }
#pragma unroll
        for (int c = 0; c < CH; c += 2) *reinterpret_cast<double2*>(out + h + c) = make_double2(x[c], x[c + 1]);
      }
    }
  } else if (tid == 0) {
    atomicExch(flag, 6);
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tm, kCols);
}

// Every tile's L^-1 (the backward substitution reads it) from k_panel64's
// tiles, in place: the off-diagonal 16 x 16 blocks by increasing distance from
// the diagonal, Li_IJ = -Li_II sum_{K=J..I-1} L_IK Li_KJ, one CTA per tile.
// Off the panel chain, all tiles at once.
__global__ void __launch_bounds__(256) k_tile_inverse(double* __restrict__ Linv_all) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* L = reinterpret_cast<double*>(smem_raw);  // [64][66]
  double* Li = L + 64 * kPanelLd;                   // [64][66]
  double* scr = Li + 64 * kPanelLd;                 // [3][16][16]
  const int tid = threadIdx.x;
  double* G = Linv_all + (int64_t)blockIdx.x * NB * NB;
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int r = idx >> 6, c = idx & 63;
    const double v = G[idx];
    L[r * kPanelLd + c] = v;  // its diagonal blocks are not read
    Li[r * kPanelLd + c] = (r >> 4) == (c >> 4) ? v : 0.0;
  }
  __syncthreads();
  const int r = tid >> 4, c = tid & 15;
#pragma unroll
  for (int dist = 1; dist < 4; ++dist) {
    // a thread's blocks and each block's 16-term pieces are independent chains
    double sum[3][3];
#pragma unroll
    for (int J = 0; J < 4 - dist; ++J)
#pragma unroll
      for (int K = 0; K < dist; ++K) sum[J][K] = 0.0;
#pragma unroll 4
    for (int k = 0; k < 16; ++k)
#pragma unroll
      for (int J = 0; J < 4 - dist; ++J)
#pragma unroll
        for (int K = 0; K < dist; ++K)
          sum[J][K] = fma(L[(16 * (J + dist) + r) * kPanelLd + 16 * (J + K) + k],
                          Li[(16 * (J + K) + k) * kPanelLd + 16 * J + c], sum[J][K]);
#pragma unroll
    for (int J = 0; J < 4 - dist; ++J) {
      double s = sum[J][0];
#pragma unroll
      for (int K = 1; K < dist; ++K) s += sum[J][K];
      scr[J * 256 + tid] = s;
    }
    __syncthreads();
#pragma unroll
    for (int J = 0; J < 4 - dist; ++J) sum[J][0] = 0.0;
#pragma unroll 4
    for (int k = 0; k < 16; ++k)
#pragma unroll
      for (int J = 0; J < 4 - dist; ++J)
        sum[J][0] = fma(Li[(16 * (J + dist) + r) * kPanelLd + 16 * (J + dist) + k], scr[J * 256 + k * 16 + c], sum[J][0]);
#pragma unroll
    for (int J = 0; J < 4 - dist; ++J) Li[(16 * (J + dist) + r) * kPanelLd + 16 * J + c] = -sum[J][0];
    __syncthreads();
  }
  for (int idx = tid; idx < 64 * 64; idx += 256) G[idx] = Li[(idx >> 6) * kPanelLd + (idx & 63)];
}
constexpr size_t kTileInverseSmem = sizeof(double) * (2 * 64 * kPanelLd + 3 * 256);

// Bytes of the factorisation's workspace: the operands of two panels (the
// trailing update of a panel runs beside the next; FP64: digits and their
// rows' exponents), and y.
size_t dense_cholesky_work_bytes(int64_t n_pad, bool fp64) {
  if (!fp64) return 2 * (size_t)(n_pad / NB) * kOpsTile * sizeof(float) + (size_t)n_pad * sizeof(float);
  return 2 * (size_t)(n_pad / NB) * kTileDigitBytes + (size_t)n_pad * (sizeof(double) + 2 * sizeof(int32_t));
}

// Opt the kernels into their dynamic shared memory (once per device and type;
// called before any stream capture).
template <typename T>
void dense_cholesky_prepare() {
  static PerDeviceOnce once;
  once.run([] {
    const int sm = (int)dense_smem_bytes<T>();
    GBBA_CUDA(cudaFuncSetAttribute(k_trsv_bwd<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    GBBA_CUDA(cudaFuncSetAttribute(k_trsv_bwd<T, std::is_same<T, double>::value>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
    if constexpr (std::is_same<T, float>::value) {
      GBBA_CUDA(cudaFuncSetAttribute(k_panel32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanel32Smem));
      GBBA_CUDA(cudaFuncSetAttribute(k_syrk_wide<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)wide_smem_bytes<T>()));
      GBBA_CUDA(cudaFuncSetAttribute(k_syrk_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem));
    } else {
      GBBA_CUDA(cudaFuncSetAttribute(k_panel64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)panel64_smem(kPanelMaxRows)));
      GBBA_CUDA(cudaFuncSetAttribute(k_syrk_split<kBulkN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)split_smem_bytes<kBulkN>()));
      GBBA_CUDA(cudaFuncSetAttribute(k_syrk_split<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)split_smem_bytes<16>()));
      GBBA_CUDA(cudaFuncSetAttribute(k_tile_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kTileInverseSmem));
    }
  });
}

// Launch on the panel chain at the device's greatest stream priority (the
// attribute is kept when the launch is captured into a graph), so that the
// panel's CTAs are scheduled ahead of the trailing update's.
//
// With pdl the launch may begin while the previous kernel on the stream is
// still running (programmatic dependent launch): the kernel must execute
// griddepcontrol.wait before it touches anything the previous kernel writes.
template <typename... Exp, typename... Act>
void launch_hi(gbba_handle* h, bool pdl, void (*k)(Exp...), unsigned grid, unsigned block, size_t smem,
               cudaStream_t st, Act... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributePriority;
  at[0].val.priority = h->prio_hi;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 2 : 1;
  GBBA_CUDA(cudaLaunchKernelEx(&cfg, k, args...));
  count_launch(h);
}

// Solve S x = b (S -> L below the diagonal tiles, b is used up); x receives
// the solution.
//
// Right-looking, 64-wide panels, look-ahead by one panel.  Per step k the
// call's stream runs panel(k+1), which applies panel k's update to block
// column k+1 itself and factors it, while the side stream applies panel k's
// update to block columns k+2...  The two touch disjoint tiles; the call's
// stream waits for the side stream's step k-1 before step k (that step wrote
// block column k+1 and read the operands that panel k+1 replaces), and the
// side stream starts step k once panel k is solved.  The side stream is joined
// back before the backward substitution, so the sequence can be captured.
// tensor: the trailing update on the tensor cores (k_syrk_tc) or on the FP32
// pipes (k_syrk_wide).
static void dense_cholesky_solve_fp32(gbba_handle* h, float* S, int64_t n_pad, float* b, float* x, float* Linv_all,
                                      void* work, int* flag, cudaStream_t st, bool tensor) {
  const int nb = (int)(n_pad / NB);
  dense_cholesky_prepare<float>();
  float* const ops[2] = {static_cast<float*>(work), static_cast<float*>(work) + (int64_t)nb * kOpsTile};
  float* y = ops[1] + (int64_t)nb * kOpsTile;
  bool side_pending = false;
  for (int k = -1; k + 1 < nb; ++k) {
    const int rem = nb - k - 1;  // tiles in block column k+1, diagonal included
    if (side_pending) {
      GBBA_CUDA(cudaStreamWaitEvent(st, h->ev_side, 0));
      side_pending = false;
    }
    if (k >= 0 && rem > 1) {
      GBBA_CUDA(cudaEventRecord(h->ev_main, st));
      GBBA_CUDA(cudaStreamWaitEvent(h->side, h->ev_main, 0));
      if (tensor) {
        int64_t ctas = 0;
        for (int j = k + 2; j < nb; ++j) ctas += (nb - j + 1) / 2;
        k_syrk_tc<<<(unsigned)ctas, kSyrkTcThreads, kTcSmem, h->side>>>(S, n_pad, k + 2, nb, ops[k & 1], flag);
      } else {
        const int64_t tw = rem / 2;  // 128-tiles per side over the 64-tiles k+2..nb-1
        k_syrk_wide<float><<<(unsigned)(tw * (tw + 1) / 2), 256, wide_smem_bytes<float>(), h->side>>>(S, n_pad, k,
                                                                                                      k + 2, nb);
      }
      check_launch(h);
      GBBA_CUDA(cudaEventRecord(h->ev_side, h->side));
      side_pending = true;
    }
    launch_hi(h, false, k_panel32, (unsigned)std::max(1, rem - 1), kPanel32Threads, kPanel32Smem, st, S, n_pad, k + 1,
              nb, Linv_all, b, y, tensor ? ops[(k + 1) & 1] : nullptr, flag);
  }
  if (side_pending) GBBA_CUDA(cudaStreamWaitEvent(st, h->ev_side, 0));
  // backward substitution: each block row's kernel starts while the previous
  // one finishes (programmatic dependent launch; the first one waits fully)
  for (int kb = nb - 1; kb >= 0; --kb)
    launch_hi(h, kb != nb - 1, k_trsv_bwd<float, false>, (unsigned)(kb + 1), 256, dense_smem_bytes<float>(), st,
              (const float*)S, n_pad, kb, (const float*)Linv_all, y, x);
}

// FP64: the same look-ahead with the kernels above.  Per step k the call's
// stream runs panel k, then panel k's update of block column k+1; the side
// stream updates block columns k+2.. meanwhile.  The call's stream waits for
// the side stream's step k-1 before step k's update (both write block column
// k+1; the digits of panel k+1 then replace those of panel k-1).
static void dense_cholesky_solve_fp64(gbba_handle* h, double* S, int64_t n, int64_t n_pad, double* b, double* x,
                                      double* Linv_all, void* work, int* flag, cudaStream_t st) {
  const int nb = (int)(n_pad / NB);
  dense_cholesky_prepare<double>();
  __half* digits[2];
  digits[0] = static_cast<__half*>(work);
  digits[1] = digits[0] + nb * kTileDigitBytes / 2;
  double* y = reinterpret_cast<double*>(digits[1] + nb * kTileDigitBytes / 2);
  int32_t* const exps[2] = {reinterpret_cast<int32_t*>(y + n_pad), reinterpret_cast<int32_t*>(y + n_pad) + n_pad};
  bool side_pending = false;
  for (int k = 0; k < nb; ++k) {
    const int64_t below = (int64_t)(nb - k - 1) * NB;
    // rows per CTA: 16, more when that would put two CTAs on an SM (they
    // share its FP64 pipe, and each factors the diagonal tile)
    const int R = (int)std::min<int64_t>(kPanelMaxRows, std::max<int64_t>(1, ceil_div(below, 16 * (int64_t)h->sm_count)) * 16);
    const int nblk = k + 1 < nb ? 4 : (int)ceil_div(std::max<int64_t>(n - (int64_t)k * NB, 1), 16);
    launch_hi(h, false, k_panel64, (unsigned)std::max<int64_t>(1, ceil_div(below, R)), kPanelThreads, panel64_smem(R),
              st, S, n_pad, k, R, nblk, Linv_all, b, y, exps[k & 1], digits[k & 1], flag);
    if (k + 1 == nb) break;
    if (k + 2 < nb) {
      GBBA_CUDA(cudaEventRecord(h->ev_main, st));
      GBBA_CUDA(cudaStreamWaitEvent(h->side, h->ev_main, 0));
    }
    if (side_pending) GBBA_CUDA(cudaStreamWaitEvent(st, h->ev_side, 0));
    launch_hi(h, false, k_syrk_split<16>, (unsigned)((nb - k) / 2 * 4), kSplitThreads, split_smem_bytes<16>(), st, S, n_pad, k + 1,
              nb, (const __half*)digits[k & 1], (const int32_t*)exps[k & 1], flag);
    side_pending = k + 2 < nb;
    if (side_pending) {
      int64_t ctas = 0;
      for (int j = k + 2; j < nb; ++j) ctas += (nb - j + 1) / 2;
      k_syrk_split<kBulkN><<<(unsigned)(ctas * (64 / kBulkN)), kSplitThreads, split_smem_bytes<kBulkN>(), h->side>>>(S, n_pad, k + 2, nb, digits[k & 1],
                                                                                  exps[k & 1], flag);
      check_launch(h);
      GBBA_CUDA(cudaEventRecord(h->ev_side, h->side));
    }
  }
  if (side_pending) GBBA_CUDA(cudaStreamWaitEvent(st, h->ev_side, 0));
  // The inverses of all tiles cost 27 us once, substitution by 16-column blocks
  // about half a microsecond more in each step of the chain of block rows.  10
  // iterations with the blocks and with the inverses: 1 tile 2.93 and 3.17 ms, 4
  // tiles 5.29 and 5.48, 8 tiles 8.07 and 8.22, 12 tiles 11.96 and 12.11, 20 tiles
  // 18.31 and 18.45; by that slope the sides meet at some 45 tiles.  The line is
  // short of it: larger systems keep the rounding of the inverses.
  const bool blocks = nb <= 8;
  if (!blocks) {
    k_tile_inverse<<<(unsigned)nb, 256, kTileInverseSmem, st>>>(Linv_all);
    check_launch(h);
  }
  for (int kb = nb - 1; kb >= 0; --kb)
    launch_hi(h, kb != nb - 1, blocks ? k_trsv_bwd<double, true> : k_trsv_bwd<double, false>, (unsigned)(kb + 1), 256,
              dense_smem_bytes<double>(), st, (const double*)S, n_pad, kb, (const double*)Linv_all, y, x);
}

// n: unknowns of S (n_pad with the padding); work: dense_cholesky_work_bytes.
template <typename T>
void dense_cholesky_solve(gbba_handle* h, T* S, int64_t n, int64_t n_pad, T* b, T* x, T* Linv_all, void* work,
                          int* flag, cudaStream_t st) {
  if constexpr (std::is_same<T, double>::value)
    dense_cholesky_solve_fp64(h, S, n, n_pad, b, x, Linv_all, work, flag, st);
  else
    dense_cholesky_solve_fp32(h, S, n_pad, b, x, Linv_all, work, flag, st, h->factor_tensor);
}

template void dense_cholesky_prepare<double>();
template void dense_cholesky_prepare<float>();
template void dense_cholesky_solve<double>(gbba_handle*, double*, int64_t, int64_t, double*, double*, double*, void*,
                                           int*, cudaStream_t);
template void dense_cholesky_solve<float>(gbba_handle*, float*, int64_t, int64_t, float*, float*, float*, void*, int*,
                                          cudaStream_t);

}  // namespace gbba
