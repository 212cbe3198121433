// Overlap factorisation (once per structure): S = L L^T and X = L^-T, the
// first step of sygvd (reference src/lapack/sygvd.cu:223-313), as one kernel
// on a CTA or a thread block cluster per structure.
//
// 64 x 64 blocks throughout.  Cholesky, left-looking, one block column at a
// time: the diagonal block's owner forms S_JJ - sum_k L_Jk L_Jk^T, factors it
// in shared memory and inverts the factor (X_JJ = L_JJ^-T); then every block
// below forms S_IJ - sum_k L_Ik L_Jk^T and solves with L_JJ^T by substitution,
// which gives L_IJ.  (Multiplied by the inverse X_JJ instead, L L^T - S grows by
// the condition of L_JJ: with functions in pairs 3e-6 apart, 138 of them, the
// residual of H C = S C w was 4.3e-7 of the largest |w|, by substitution 1.3e-10.)
// The inverse by block diagonals: X_rc = -X_rr sum_{k=r+1..c} L_kr^T X_kc,
// every block of a diagonal independent.  The products run on the FP64 tensor
// instruction; a block's terms are added in the order of k whichever CTA owns
// it (block row I belongs to CTA I mod C), so the bits do not depend on the
// cluster size.
//
// What bounds it: the diagonal blocks are a serial chain (two barriers and a
// reciprocal square root per column); everything else is matrix products.  The
// former kernels updated 16 columns at a time with scalar FMAs on one CTA per
// structure and re-read the finished part from L2 for every group.
#include <cooperative_groups.h>

#include "tb_common.cuh"
#include "tb_kernels.h"

namespace tb {

namespace {

constexpr int kB = kFactorBlock;     // 64
constexpr int kP = kB + 4;           // row stride of shared blocks: 4 mod 16, conflict-free fragments
constexpr int kSlab = 16;            // k values staged per round
constexpr int kT = 256;
static_assert(kB == 64, "eight warps of 16 x 32");

extern __shared__ __align__(16) double factor_sm[];

struct Cluster {
  int rank, size;
  __device__ __forceinline__ void sync() const {
    __syncwarp();
    if (size == 1) __syncthreads();
    else cooperative_groups::this_cluster().sync();
    __syncwarp();
  }
};

__device__ __forceinline__ void cp8(double* smem, const double* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 8 : 0;  // the rest of the 8 bytes is zero-filled
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}
// D = A B + D for one 8 x 8 x 4 step (lane l = 4 g + t: A[g][t], B[t][g], D[g][2t], D[g][2t+1])
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// A warp's 16 x 32 part of a 64 x 64 block, as 2 x 4 fragments.
struct Acc {
  double d[2][4][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) d[x][y][0] = d[x][y][1] = 0.0;
  }
};

// acc += A B over k0 <= k < k1 with both operands in global memory, through a
// two-stage ring of slabs: A(k, i) = A[k sak + i sai] for i < na, B(k, j) =
// B[k n + j] for j < nb.  kA: A's rows are contiguous in k (sai = n, sak = 1),
// else in i.  As, Bs: 2 x kSlab x kP.
template <bool kA>
__device__ __forceinline__ void block_product(Acc& acc, const double* A, int na, const double* B, int nb, int n, int k0,
                                              int k1, double* As, double* Bs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 1) * 16, wc = (warp & 1) * 32;
  auto stage = [&](int buf, int ks) {
    double* as = As + buf * kSlab * kP;
    double* bs = Bs + buf * kSlab * kP;
#pragma unroll
    for (int r = 0; r < kSlab * kB / kT; ++r) {
      if (kA) {
        const int kk = tid & 15, i = (tid >> 4) + 16 * r;
        const bool v = ks + kk < k1 && i < na;
        cp8(as + kk * kP + i, v ? A + (long long)i * n + ks + kk : A, v);
      } else {
        const int i = tid & 63, kk = (tid >> 6) + 4 * r;
        const bool v = ks + kk < k1 && i < na;
        cp8(as + kk * kP + i, v ? A + (long long)(ks + kk) * n + i : A, v);
      }
      const int j = tid & 63, kk = (tid >> 6) + 4 * r;
      const bool v = ks + kk < k1 && j < nb;
      cp8(bs + kk * kP + j, v ? B + (long long)(ks + kk) * n + j : B, v);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  if (k0 < k1) stage(0, k0);
  int buf = 0;
  for (int ks = k0; ks < k1; ks += kSlab, buf ^= 1) {
    if (ks + kSlab < k1) {
      stage(buf ^ 1, ks + kSlab);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const double* as = As + buf * kSlab * kP;
    const double* bs = Bs + buf * kSlab * kP;
#pragma unroll
    for (int k4 = 0; k4 < kSlab; k4 += 4) {
      double af[2], bf[4];
#pragma unroll
      for (int x = 0; x < 2; ++x) af[x] = as[(k4 + t) * kP + wr + 8 * x + g];
#pragma unroll
      for (int y = 0; y < 4; ++y) bf[y] = bs[(k4 + t) * kP + wc + 8 * y + g];
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) dmma(acc.d[x][y][0], acc.d[x][y][1], af[x], bf[y]);
    }
    __syncthreads();
  }
}

// acc += A B for two 64 x 64 blocks in shared memory (row stride kP), A[i][k]
// and B[k][j].
__device__ __forceinline__ void shared_product(Acc& acc, const double* A, const double* B) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 1) * 16, wc = (warp & 1) * 32;
#pragma unroll 4
  for (int k4 = 0; k4 < kB; k4 += 4) {
    double af[2], bf[4];
#pragma unroll
    for (int x = 0; x < 2; ++x) af[x] = A[(wr + 8 * x + g) * kP + k4 + t];
#pragma unroll
    for (int y = 0; y < 4; ++y) bf[y] = B[(k4 + t) * kP + wc + 8 * y + g];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) dmma(acc.d[x][y][0], acc.d[x][y][1], af[x], bf[y]);
  }
}

// f(i, j, value) for every entry of the warp's part of the block
template <typename F>
__device__ __forceinline__ void each(const Acc& acc, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 1) * 16, wc = (warp & 1) * 32;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int h = 0; h < 2; ++h) f(wr + 8 * x + g, wc + 8 * y + 2 * t + h, acc.d[x][y][h]);
}

// 64 x 64 block at G (row stride n, nr x nc of it valid) into shared memory, zero elsewhere
__device__ __forceinline__ void load_block(double* T, const double* G, int n, int nr, int nc) {
#pragma unroll 4
  for (int r = 0; r < kB * kB / kT; ++r) {
    const int x = threadIdx.x + kT * r, i = x >> 6, j = x & 63;
    T[i * kP + j] = (i < nr && j < nc) ? G[(long long)i * n + j] : 0.0;
  }
}

// X T = the 64 x 64 block in T solved for X = T L^-T by substitution, L the lower
// factor whose transpose is in Y (Y[k][j] = L[j][k], j >= k), inv[q] = 1 / L_qq;
// row stride kP.  Warp w takes the rows 8w .. 8w + 7 alone: eight columns at a
// time, lane (g, t) holding columns 2t and 2t + 1 of row g, then their part of
// the columns beyond on the tensor instruction (56 of them, against 128 for a
// product with L^-T).  f(i, j, value) for every entry.
template <typename F>
__device__ __forceinline__ void solve_block(const double* T, const double* Y, const double* inv, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const double2* Tr = reinterpret_cast<const double2*>(T + (8 * warp + g) * kP + 2 * t);
  double d0[8], d1[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const double2 v = Tr[4 * c];
    d0[c] = v.x;
    d1[c] = v.y;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double2 l = *reinterpret_cast<const double2*>(Y + (8 * c + q) * kP + 8 * c + 2 * t);
      const double x = __shfl_sync(0xffffffffu, (q & 1 ? d1[c] : d0[c]) * inv[8 * c + q], (lane & ~3) | (q >> 1));
      d0[c] = 2 * t == q ? x : (2 * t > q ? d0[c] - x * l.x : d0[c]);
      d1[c] = 2 * t + 1 == q ? x : (2 * t + 1 > q ? d1[c] - x * l.y : d1[c]);
    }
    if (c == 7) break;
    double a[2];  // the eight columns as two left operands
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int src = (lane & ~3) | ((4 * s + t) >> 1);
      const double x0 = __shfl_sync(0xffffffffu, d0[c], src), x1 = __shfl_sync(0xffffffffu, d1[c], src);
      a[s] = -((t & 1) ? x1 : x0);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int e = c + 1; e < 8; ++e) dmma(d0[e], d1[e], a[s], Y[(8 * c + 4 * s + t) * kP + 8 * e + g]);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    f(8 * warp + g, 8 * c + 2 * t, d0[c]);
    f(8 * warp + g, 8 * c + 2 * t + 1, d1[c]);
  }
}

// Cholesky of the m x m block in T (lower triangle used) in place, right-looking
// with one barrier per column: column q stays as it is while the rest is
// updated with its scaled entries (lane group i = tid / 4 on row i) and is
// scaled at the end.  inv[q] = 1 / L_qq.  Returns false (in every thread) when
// a pivot is not positive.
__device__ __forceinline__ bool factor_diag(double* T, double* inv, int m) {
  const int i = threadIdx.x >> 2, sub = threadIdx.x & 3;
  bool ok = true;
  for (int q = 0; q < m; ++q) {
    const double d = T[q * kP + q];
    ok &= d > 0.0;
    const double r = d > 0.0 ? 1.0 / sqrt(d) : 1.0;
    if (threadIdx.x == 0) inv[q] = r;
    if (i > q && i < m) {
      const double li = T[i * kP + q] * r;
#pragma unroll 4
      for (int j = q + 1 + sub; j <= i; j += 4) T[i * kP + j] -= li * (T[j * kP + q] * r);
    }
    __syncthreads();
  }
  for (int q = sub; q <= i && i < m; q += 4) T[i * kP + q] = q == i ? sqrt(T[i * kP + q]) : T[i * kP + q] * inv[q];
  __syncthreads();
  return ok;
}

// X = L^-T of the m x m lower factor in T: column c (four lanes) by backward
// substitution from row c up; zero below the diagonal of X's m x m part (row
// stride kP).
__device__ __forceinline__ void invert_diag(const double* T, const double* inv, int m, double* X) {
  const int c = threadIdx.x >> 2, sub = threadIdx.x & 3;
  for (int r = m - 1; r >= 0; --r) {
    double s = 0.0;
    if (r < c && c < m)
      for (int k = r + 1 + sub; k <= c; k += 4) s += T[k * kP + r] * X[k * kP + c];
    __syncwarp();
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (sub == 0) X[r * kP + c] = r > c ? 0.0 : (r == c ? inv[r] : -s * inv[r]);
    __syncwarp();
  }
  __syncthreads();
}

}  // namespace

__global__ void __launch_bounds__(kT, 2) k_factor(DevBatch B, const double* __restrict__ S, double* __restrict__ Wb,
                                                  double* __restrict__ Xb, int* __restrict__ status, int ncoop) {
  unsigned csize, crank;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int cid = (int)(blockIdx.x / csize);
  const bool coop = cid < ncoop;
  const Cluster cl{coop ? (int)crank : 0, coop ? (int)csize : 1};
  const int slot = coop ? cid : ncoop + (cid - ncoop) * (int)csize + (int)crank;
  if (slot >= B.nmol) return;
  const int m = B.order ? B.order[slot] : slot;
  if (status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (on_library(B, n)) return;
  const long long mo = B.moff[m];
  const double* s = S + mo;
  double* W = Wb + mo;  // W[k][i] = L[i][k], i >= k
  double* X = Xb + mo;
  double* T = factor_sm;           // kB x kP
  double* Y = T + kB * kP;         // kB x kP
  double* As = Y + kB * kP;        // 2 x kSlab x kP
  double* Bs = As + 2 * kSlab * kP;
  __shared__ double inv[kB];
  __shared__ int bad;              // set in every CTA of the cluster
  const int nb = (n + kB - 1) / kB;
  if (threadIdx.x == 0) bad = 0;
  cl.sync();
  for (int J = 0; J < nb; ++J) {
    const int j0 = J * kB, mj = min(kB, n - j0);
    Acc acc;
    if (J % cl.size == cl.rank) {
      acc.zero();
      block_product<false>(acc, W + j0, mj, W + j0, mj, n, 0, j0, As, Bs);
      each(acc, [&](int i, int j, double v) {
        T[i * kP + j] = (i < mj && j <= i) ? s[(long long)(j0 + j) * n + j0 + i] - v : 0.0;
      });
      __syncthreads();
      const bool ok = factor_diag(T, inv, mj);
      if (!ok && threadIdx.x < cl.size) {
        if ((int)threadIdx.x == cl.rank) bad = 1;
        else *cooperative_groups::this_cluster().map_shared_rank(&bad, threadIdx.x) = 1;
      }
      invert_diag(T, inv, mj, Y);
      for (int x = threadIdx.x; x < mj * mj; x += kT) {
        const int k = x / mj, i = x - k * mj;
        if (!TB_GUARD(1, (long long)(j0 + k) * n + j0 + i, 0, (long long)n * n)) continue;
        if (i >= k) W[(long long)(j0 + k) * n + j0 + i] = T[i * kP + k];
        X[(long long)(j0 + k) * n + j0 + i] = Y[k * kP + i];
      }
    }
    cl.sync();
    if (bad) break;
    bool have = false;  // L_JJ^T in Y and the reciprocals of its diagonal
    for (int I = J + 1; I < nb; ++I) {
      if (I % cl.size != cl.rank) continue;
      const int i0 = I * kB, mi = min(kB, n - i0);
      if (!have) {
        load_block(Y, W + (long long)j0 * n + j0, n, mj, mj);
        if (threadIdx.x < mj) inv[threadIdx.x] = X[(long long)(j0 + threadIdx.x) * n + j0 + threadIdx.x];
      }
      have = true;
      acc.zero();
      block_product<false>(acc, W + i0, mi, W + j0, mj, n, 0, j0, As, Bs);
      each(acc, [&](int i, int j, double v) {
        T[i * kP + j] = (i < mi && j < mj) ? s[(long long)(j0 + j) * n + i0 + i] - v : 0.0;
      });
      __syncthreads();
      solve_block(T, Y, inv, [&](int i, int j, double v) {
        if (i < mi && j < mj && TB_GUARD(2, (long long)(j0 + j) * n + i0 + i, 0, (long long)n * n) &&
            TB_GUARD(3, (long long)(i0 + i) * n + j0 + j, 0, (long long)n * n)) {
          W[(long long)(j0 + j) * n + i0 + i] = v;
          X[(long long)(i0 + i) * n + j0 + j] = 0.0;  // below the diagonal
        }
      });
      __syncthreads();  // T is rewritten
    }
    cl.sync();
  }
  if (bad) {
    if (threadIdx.x == 0 && cl.rank == 0) status[m] = kStNotSpd;
    return;
  }
  for (int d = 1; d < nb; ++d) {
    for (int r = 0; r + d < nb; ++r) {
      if (r % cl.size != cl.rank) continue;
      const int r0 = r * kB, c0 = (r + d) * kB, mc = min(kB, n - c0);
      Acc acc;
      acc.zero();
      block_product<true>(acc, W + (long long)r0 * n, kB, X + c0, mc, n, r0 + kB, c0 + mc, As, Bs);
      each(acc, [&](int i, int j, double v) { T[i * kP + j] = v; });
      load_block(Y, X + (long long)r0 * n + r0, n, kB, kB);
      __syncthreads();
      acc.zero();
      shared_product(acc, Y, T);
      each(acc, [&](int i, int j, double v) {
        if (j < mc && TB_GUARD(4, (long long)(r0 + i) * n + c0 + j, 0, (long long)n * n))
          X[(long long)(r0 + i) * n + c0 + j] = -v;
      });
      __syncthreads();
    }
    cl.sync();
  }
}

cudaError_t launch_factor(const FactorPlan& P, const DevBatch& B, const double* S, double* W, double* X, int* status,
                          cudaStream_t st) {
  const int C = P.c.cluster, groups = P.c.ncoop + (P.count - P.c.ncoop + C - 1) / C;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(groups * C));
  cfg.blockDim = dim3(kT);
  cfg.dynamicSmemBytes = factor_smem_bytes();
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = C > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_factor, B, S, W, X, status, P.c.ncoop);
}

TB_OOB_EXPORT(oob_factor)

size_t factor_smem_bytes() { return (2 * (size_t)kB * kP + 4 * kSlab * kP) * sizeof(double); }

}  // namespace tb
