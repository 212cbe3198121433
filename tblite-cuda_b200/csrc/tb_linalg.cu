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

// ------------------------------------------------ small structures: one-warp Jacobi
// Cyclic Jacobi (Jacobi 1846; the parallel tournament ordering of Brent and
// Luk 1985) for structures of at most 32 AOs, one warp per structure, the
// matrix and the rotation accumulator in shared memory (33-double pitch).
// A round applies n/2 disjoint rotations: lane t forms the rotation of pair t
// (symmetric Schur: tau = (a_qq - a_pp)/(2 a_pq), t = sign(tau)/(|tau| +
// sqrt(1 + tau^2)), c = 1/sqrt(1 + t^2), s = t c, which zeroes a_pq in
// J^T A J), then lane k updates row k of every pair's two columns (A J, V J)
// and column k of every pair's two rows (J^T A).  Sweeps stop when the
// off-diagonal norm is below 1e-14 of the Frobenius norm (at most 50 sweeps,
// else TB_EIGEN_FAILED).  A one-CTA eigensolver spends most of its 256
// threads' time waiting at barriers on such small matrices; a warp per
// structure runs eight times as many structures per SM.
__global__ void __launch_bounds__(kJacobiWarps * 32) k_syev_jacobi(DevBatch B, double* __restrict__ Ab,
                                                                  double* __restrict__ Zb,
                                                                  double* __restrict__ wout,
                                                                  int* __restrict__ perm, int* __restrict__ status,
                                                                  const int* __restrict__ active,
                                                                  const int* __restrict__ list, int nlist) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int li = blockIdx.x * kJacobiWarps + warp;
  if (li >= nlist) return;
  const int m = list[li];
  if ((active && !active[m]) || status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (n > kJacobiMaxN) return;
  constexpr int P = kJacobiPitch;
  extern __shared__ double jac_smem[];
  double* a = jac_smem + (size_t)warp * 2 * kJacobiMaxN * P;  // n x n, pitch P
  double* v = a + kJacobiMaxN * P;
  __shared__ double rot_c[kJacobiWarps][kJacobiMaxN / 2], rot_s[kJacobiWarps][kJacobiMaxN / 2];
  __shared__ int rot_p[kJacobiWarps][kJacobiMaxN / 2], rot_q[kJacobiWarps][kJacobiMaxN / 2];
  const long long mo = B.moff[m], vo = B.ooff[m];
  const double* A = Ab + mo;
  if (lane < n)
    for (int j = 0; j < n; ++j) {
      a[lane * P + j] = 0.5 * (A[(long long)lane * n + j] + A[(long long)j * n + lane]);
      v[lane * P + j] = lane == j ? 1.0 : 0.0;
    }
  __syncwarp();
  const int nn = n + (n & 1);  // players; index n (odd n) sits out
  double fro = 0.0;
  if (lane < n)
    for (int j = 0; j < n; ++j) fro += a[lane * P + j] * a[lane * P + j];
  fro = warp_sum(fro);
  bool conv = n <= 1;
  for (int sweep = 0; sweep < 50 && !conv; ++sweep) {
    double off = 0.0;
    if (lane < n)
      for (int j = 0; j < n; ++j)
        if (j != lane) off += a[lane * P + j] * a[lane * P + j];
    off = warp_sum(off);
    if (off <= 1e-28 * fro) { conv = true; break; }
    for (int r = 0; r < nn - 1; ++r) {
      if (lane < nn / 2) {
        int p = lane == 0 ? r : (r + lane) % (nn - 1);
        int q = lane == 0 ? nn - 1 : (r - lane + nn - 1) % (nn - 1);
        if (p > q) { const int x = p; p = q; q = x; }
        double c = 1.0, s = 0.0;
        if (q < n) {
          const double apq = a[p * P + q];
          if (apq != 0.0) {
            const double tau = (a[q * P + q] - a[p * P + p]) / (2.0 * apq);
            const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
            c = 1.0 / sqrt(1.0 + t * t);
            s = t * c;
          }
        }
        rot_p[warp][lane] = p;
        rot_q[warp][lane] = q < n ? q : p;  // the sitting-out pair becomes the identity
        rot_c[warp][lane] = c;
        rot_s[warp][lane] = q < n ? s : 0.0;
      }
      __syncwarp();
      // columns: A <- A J and V <- V J, lane k on row k
      if (lane < n)
        for (int t = 0; t < nn / 2; ++t) {
          const int p = rot_p[warp][t], q = rot_q[warp][t];
          if (p == q) continue;
          const double c = rot_c[warp][t], s = rot_s[warp][t];
          const double akp = a[lane * P + p], akq = a[lane * P + q];
          a[lane * P + p] = c * akp - s * akq;
          a[lane * P + q] = s * akp + c * akq;
          const double vkp = v[lane * P + p], vkq = v[lane * P + q];
          v[lane * P + p] = c * vkp - s * vkq;
          v[lane * P + q] = s * vkp + c * vkq;
        }
      __syncwarp();
      // rows: A <- J^T A, lane k on column k
      if (lane < n)
        for (int t = 0; t < nn / 2; ++t) {
          const int p = rot_p[warp][t], q = rot_q[warp][t];
          if (p == q) continue;
          const double c = rot_c[warp][t], s = rot_s[warp][t];
          const double apk = a[p * P + lane], aqk = a[q * P + lane];
          a[p * P + lane] = c * apk - s * aqk;
          a[q * P + lane] = s * apk + c * aqk;
        }
      __syncwarp();
    }
  }
  if (!conv) {
    if (lane == 0) status[m] = kStEigenFailed;
    return;
  }
  // eigenvector i (column i of v) as row i of Z; ascending order by rank (ties by index)
  double* Z = Zb + mo;
  if (lane < n && TB_GUARD(10, (long long)lane * n + n - 1, 0, (long long)n * n)) {
    for (int k = 0; k < n; ++k) Z[(long long)lane * n + k] = v[k * P + lane];
    const double di = a[lane * P + lane];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = a[j * P + j];
      rank += (dj < di || (dj == di && j < lane)) ? 1 : 0;
    }
    perm[vo + rank] = lane;
    wout[vo + rank] = di;
  }
}

}  // namespace tb
