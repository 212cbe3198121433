// Batched FP64 dense linear algebra for uneven structure sizes:
//  * k_gemm: C = alpha op(A) diag(ks) op(B) + beta C over a tile list;
//  * k_syev_jacobi: eigenproblems of the smallest structures (others: tb_syev.cu).
// Together with k_factor (tb_factor.cu) these give sygvd (itype 1, jobz 'V'; reference src/lapack/sygvd.h:4-23):
// H C = S C e  <=>  (X^T H X) Z = Z e, C = X Z.
#include "tb_common.cuh"
#include "tb_kernels.h"

namespace tb {

// ------------------------------------------------------------ batched GEMM
// C_m = alpha * op(A_m) * diag(ks_m) * op(B_m) + beta * C_m for every tile in
// the list (structure, tile row, tile col).  Square n_m x n_m operands with
// leading dimension n_m at offset moff[m]; K = kdim[m] if kdim != NULL.
// op(B) may gather its columns through perm (eigenvector reordering).
// `shape` skips known zeros and redundant tiles: kGemmKUpToJ (op(B) upper
// triangular: only k < the tile's last column), kGemmKUpToI (op(A) lower
// triangular: k < its last row), kGemmKFromI (op(A) upper triangular: k >=
// its first row), kGemmSym (C symmetric: tiles below the diagonal are
// skipped, and each element of the upper triangle is computed once and also
// written to its mirror).
// TILE x TILE tiles (64 or 32) on the FP64 tensor instruction
// mma.sync.m8n8k4.f64: four warps, each owning a quarter of the tile as
// (TILE/16) x (TILE/16) fragments of 8 x 8.  K slabs of 16 are staged by
// cp.async in a two-stage ring (zero fill past the matrix edge); the shared
// tiles are padded by 4 doubles so the 64-bit fragment loads of a half-warp
// hit 16 distinct bank pairs.  Every output element accumulates over k in the
// same order (slabs starting at multiples of 16, then the four k-steps of the
// instruction) whatever the tile; the k ranges that only one tile size skips
// hold exact zeros of the triangular operand, which leave a sum unchanged.
// So the two tile sizes give the same bits, and the autotuner picks the tile
// per structure size (k_gemm: 64, k_gemm32: 32).
constexpr int GK = 16;
static_assert(kGemmThreads == 128, "k_gemm assumes four warps");

namespace {
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 8 : 0;  // bytes read; the rest of the 8 is zero-filled
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
// D = A B + D for one 8 x 8 x 4 step.  Lane l = 4 g + t holds A[g][t], B[t][g]
// and D[g][2t], D[g][2t+1].
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <int GT>
__device__ __forceinline__ void gemm_body(const DevBatch& B, const int4* __restrict__ tiles, int ntiles,
                                          const double* __restrict__ Ab, int ta, const double* __restrict__ Bb,
                                          int tb_, const int* __restrict__ perm, const double* __restrict__ ks,
                                          const int* __restrict__ kdim, double* __restrict__ Cb, double alpha,
                                          double beta, const int* __restrict__ active, int shape) {
  constexpr int GP = GT + 4, FX = GT / 16;  // padded row; fragments per warp and dimension
  constexpr int RA = GT / 8;                // slab elements of op(A) (and of op(B)) per thread
  constexpr int TSH = GT == 64 ? 6 : 5;     // log2(GT)
  __shared__ __align__(16) double As[2][GK][GP];
  __shared__ __align__(16) double Bs[2][GK][GP];
  __shared__ __align__(16) double Ks[2][GK];
  __shared__ int colS[GT];  // columns of op(B) for this tile (through perm)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tg = lane & 3;                          // fragment coordinates
  const int wr = (warp >> 1) * (GT / 2), wc = (warp & 1) * (GT / 2);  // this warp's quarter of the tile
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int4 tl = tiles[t];
    const int m = tl.x;
    if (active && !active[m]) continue;
    if ((shape & kGemmSym) && tl.z < tl.y) continue;
    const int n = B.ooff[m + 1] - B.ooff[m];
    // the reduction length never leaves [0, n], whatever kdim holds
    const int K = kdim ? min(max(kdim[m], 0), n) : n;
    const long long mo = B.moff[m];
    const long long vo = B.ooff[m];
    const double* A = Ab + mo;
    const double* Bm = Bb + mo;
    const int* pm = perm ? perm + vo : nullptr;
    const double* kv = ks ? ks + vo : nullptr;
    const int i0 = tl.y * GT, j0 = tl.z * GT;
    int klo = 0, khi = K;
    if (shape & kGemmKUpToJ) khi = min(khi, j0 + GT);
    if (shape & kGemmKUpToI) khi = min(khi, i0 + GT);
    if (shape & kGemmKFromI) klo = min(i0, K);
    double acc[FX][FX][2];
#pragma unroll
    for (int a = 0; a < FX; ++a)
#pragma unroll
      for (int b = 0; b < FX; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    __syncthreads();  // colS and the ring of the previous tile are free
    if (tid < GT) colS[tid] = pm ? (j0 + tid < n ? pm[j0 + tid] : 0) : j0 + tid;
    __syncthreads();
    // Element r of a slab for this thread:
    //   op(A) not transposed: kk = tid & 15, ii = (tid >> 4) + 8 r;  transposed: ii = tid & (GT-1), kk = (tid >> log2 GT) + (128/GT) r
    //   op(B) not transposed: jj = tid & (GT-1), kb = (tid >> log2 GT) + (128/GT) r;  transposed: kb = tid & 15, jj = (tid >> 4) + 8 r
    const int lo16 = tid & 15, hi8 = tid >> 4, loT = tid & (GT - 1), hiT = tid >> TSH;
    constexpr int SK = kGemmThreads / GT;  // k step of the transposed loads
    auto issue = [&](int buf, int k0) {
      if (!ta) {
        const int gk = k0 + lo16;
#pragma unroll
        for (int r = 0; r < RA; ++r) {
          const int gi = i0 + hi8 + 8 * r;
          const bool v = gi < n && gk < K;
          cp_async8(&As[buf][lo16][hi8 + 8 * r], v ? A + (long long)gi * n + gk : A, v);
        }
      } else {
        const int gi = i0 + loT;
#pragma unroll
        for (int r = 0; r < RA; ++r) {
          const int gk = k0 + hiT + SK * r;
          const bool v = gi < n && gk < K;
          cp_async8(&As[buf][hiT + SK * r][loT], v ? A + (long long)gk * n + gi : A, v);
        }
      }
      if (!tb_) {
        const bool vj = j0 + loT < n;
        const int col = colS[loT];
#pragma unroll
        for (int r = 0; r < RA; ++r) {
          const int gk = k0 + hiT + SK * r;
          const bool v = vj && gk < K;
          cp_async8(&Bs[buf][hiT + SK * r][loT], v ? Bm + (long long)gk * n + col : Bm, v);
        }
      } else {
        const int gk = k0 + lo16;
#pragma unroll
        for (int r = 0; r < RA; ++r) {
          const int jj = hi8 + 8 * r;
          const bool v = j0 + jj < n && gk < K;
          cp_async8(&Bs[buf][lo16][jj], v ? Bm + (long long)colS[jj] * n + gk : Bm, v);
        }
      }
      if (kv && tid < GK) cp_async8(&Ks[buf][tid], k0 + tid < K ? kv + k0 + tid : kv, k0 + tid < K);
      cp_async_commit();
    };
    const int nk = khi > klo ? (khi - klo + GK - 1) / GK : 0;
    if (nk > 0) issue(0, klo);
    for (int kt = 0; kt < nk; ++kt) {
      const int cur = kt & 1;
      if (kt + 1 < nk) {
        issue(cur ^ 1, klo + (kt + 1) * GK);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      if (kv) {  // diag(ks) between the factors: scale the slab of op(B) once
        for (int e = tid; e < GK * GT; e += kGemmThreads) Bs[cur][e / GT][e % GT] *= Ks[cur][e / GT];
        __syncthreads();
      }
#pragma unroll
      for (int k4 = 0; k4 < GK; k4 += 4) {
        double af[FX], bf[FX];
#pragma unroll
        for (int x = 0; x < FX; ++x) af[x] = As[cur][k4 + tg][wr + 8 * x + g];
#pragma unroll
        for (int y = 0; y < FX; ++y) bf[y] = Bs[cur][k4 + tg][wc + 8 * y + g];
#pragma unroll
        for (int x = 0; x < FX; ++x)
#pragma unroll
          for (int y = 0; y < FX; ++y) dmma(acc[x][y][0], acc[x][y][1], af[x], bf[y]);
      }
      __syncthreads();  // buffer cur is refilled two slabs later
    }
#pragma unroll
    for (int x = 0; x < FX; ++x) {
      const int gi = i0 + wr + 8 * x + g;
      if (gi >= n) continue;
#pragma unroll
      for (int y = 0; y < FX; ++y) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int gj = j0 + wc + 8 * y + 2 * tg + h;
          if (gj >= n) continue;
          // symmetric result: the upper triangle is computed and mirrored, so
          // no element depends on which tile it fell in
          if ((shape & kGemmSym) && gi > gj) continue;
          if (!TB_GUARD(8, (long long)gi * n + gj, 0, (long long)n * n)) continue;
          double* c = Cb + mo + (long long)gi * n + gj;
          const double r = beta == 0.0 ? alpha * acc[x][y][h] : alpha * acc[x][y][h] + beta * (*c);
          *c = r;
          if ((shape & kGemmSym) && gi != gj) Cb[mo + (long long)gj * n + gi] = r;
        }
      }
    }
  }
}
}  // namespace

__global__ void __launch_bounds__(kGemmThreads) k_gemm(DevBatch B, const int4* __restrict__ tiles, int ntiles,
                                                       const double* __restrict__ Ab, int ta,
                                                       const double* __restrict__ Bb, int tb_,
                                                       const int* __restrict__ perm, const double* __restrict__ ks,
                                                       const int* __restrict__ kdim, double* __restrict__ Cb,
                                                       double alpha, double beta, const int* __restrict__ active,
                                                       int shape) {
  gemm_body<64>(B, tiles, ntiles, Ab, ta, Bb, tb_, perm, ks, kdim, Cb, alpha, beta, active, shape);
}

__global__ void __launch_bounds__(kGemmThreads) k_gemm32(DevBatch B, const int4* __restrict__ tiles, int ntiles,
                                                         const double* __restrict__ Ab, int ta,
                                                         const double* __restrict__ Bb, int tb_,
                                                         const int* __restrict__ perm, const double* __restrict__ ks,
                                                         const int* __restrict__ kdim, double* __restrict__ Cb,
                                                         double alpha, double beta, const int* __restrict__ active,
                                                         int shape) {
  gemm_body<32>(B, tiles, ntiles, Ab, ta, Bb, tb_, perm, ks, kdim, Cb, alpha, beta, active, shape);
}

TB_OOB_EXPORT(oob_linalg)

}  // namespace tb
