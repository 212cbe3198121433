// Batched FP64 dense linear algebra for uneven structure sizes:
//  * k_gemm: C = alpha op(A) diag(ks) op(B) + beta C over a tile list;
//  * k_reduce_f32: the mixed form's FP32 reduction to tridiagonal form and Q;
//    FP64 eigensolver: tb_syev.cu, and k_syev_jacobi here.
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

// ------------------------------------------------------------ eigensolver
// FP32 reduction of the mixed form's eigensolve (FP64: tb_syev.cu) of A (n x n,
// row-major, overwritten), one CTA of 256 threads per structure:
//  1. Householder tridiagonalisation in panels (tridiagonalise): within a
//     panel the trailing block keeps its value from the panel start, each
//     step forms its product with one read-only walk (colwalk, row segments)
//     and corrects it with the panel's pairs; the panel-closing walk
//     (panel_walk) applies the rank-2 width update fused with the next
//     product.  Reflector k is kept in row k of A.
//  2. Zc = Q^T accumulated backwards in compact-WY blocks of kQBlock
//     reflectors (form_q).
// The tridiagonal problem and the product with Q go through k_syev's divide
// and conquer: implicit QL on one CTA, a serial chain of rotations applied to
// FP32 vectors, was more than half of the eigensolve (9.1 ms of a launch over
// 64 clusters of 48..384 AOs), and FP32 merges cost an SCF iteration.
namespace {

// Tridiagonalisation panel: reflectors per panel (2 panel n <= ring) and rows
// per load batch of the panel-closing walk; a panel of one (each step's update
// fused with the next product) is as fast as a wider one in FP32.
template <typename T> struct PanelCfg;
template <> struct PanelCfg<float> { static constexpr int width = 1, batch = 12; };
// Read-only Householder walk (colwalk): the warps form kWalkRowGroups row
// groups (interleaved rows) times nw / kWalkRowGroups column groups; a lane
// holds `cols` columns (32 apart) of its group's strip and loads `rows` rows
// of them before using any, so a warp reads whole row segments (contiguous
// for DRAM) with cols * rows loads in flight per lane.
constexpr int kWalkRowGroups = 4;
template <typename T> struct WalkCfg { static constexpr int cols = 3, rows = 4; };
static_assert(PanelCfg<float>::width <= kRing, "panel exceeds the ring");
constexpr int kQBlock = 16;     // reflectors per compact-WY block of the Q accumulation

__device__ inline float tb_sqrt(float x) { return sqrtf(x); }

template <typename T>
__device__ inline T block_sum_syev(T v, T* red) { return block_sum(v, red); }

// Householder reflector of row k: x = A[k][k+1..n-1] -> tau[k], e[k] and v
// (v[0] = 1), written to `v` and back into row k.
template <typename T>
__device__ void reflector(T* A, int n, int k, T* v, T* tau, T* e, T* red, T* sh) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int mm = n - k - 1;
  T* rowk = A + (long long)k * n + k + 1;
  T part = T(0);
  for (int i = 1 + tid; i < mm; i += nt) part += rowk[i] * rowk[i];
  const T sigma = block_sum_syev(part, red);
  if (tid == 0) {
    const T alpha = rowk[0];
    if (sigma == T(0)) {
      tau[k] = T(0); e[k] = alpha; sh[0] = T(0); sh[1] = T(0);
    } else {
      const T r = tb_sqrt(alpha * alpha + sigma);
      const T beta = alpha <= T(0) ? r : -r;
      tau[k] = (beta - alpha) / beta;
      e[k] = beta;
      sh[0] = tau[k];
      sh[1] = T(1) / (alpha - beta);
    }
  }
  __syncthreads();
  const T scal = sh[1];
  const bool refl = sh[0] != T(0);
  for (int i = tid; i < mm; i += nt) {
    const T x = i == 0 ? T(1) : (refl ? rowk[i] * scal : T(0));
    v[i] = x;
    if (refl) rowk[i] = x;
  }
  __syncthreads();
}

// Rows of a walk over an nm-column block are split in two halves (separate
// threads, partial sums added at the end) when that shortens the slowest
// thread's walk by more than an eighth: it walks ceil(nm/nt) whole columns,
// or ceil(2nm/nt) halves.  True for nm <= nt/2 (idle warps otherwise) and for
// the ranges of nm where a last partial round of whole columns would run.
__device__ inline bool walk_split(int nm, int nt) {
  const int whole = (nm + nt - 1) / nt * nm, halves = (2 * nm + nt - 1) / nt * ((nm + 1) >> 1);
  return 8 * halves < 7 * whole;
}

// Read-only walk over the square block r0..r0+nm-1 (rows and columns) of a
// row-major matrix M: out_c = scale * sum_r M[r][c] x_{r-r0}.  Row group g
// (warps g, g + kWalkRowGroups, ...) sums rows g, g + kWalkRowGroups, ... into
// its own partial vector (group 0: out, groups 1..3: p1, p2, p3, nm entries
// each, distinct from x and out); the partials are added at the end in a fixed
// order, so the result is deterministic.  Needs a multiple of kWalkRowGroups
// warps.  Kept out of line (as is panel_walk) so that its load registers are
// allocated apart from the rest of the eigensolver.
template <typename T>
__device__ __noinline__ void colwalk(const T* M, int n, int r0, int nm, const T* x, T* out, T scale, T* p1, T* p2,
                                     T* p3) {
  constexpr int kJ = WalkCfg<T>::cols, kR = WalkCfg<T>::rows, kG = kWalkRowGroups;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int ncg = (nt >> 5) / kG, rg = warp % kG, cg = warp / kG;
  const int strip = 32 * kJ * ncg;  // columns per pass
  T* mine = rg == 0 ? out : (rg == 1 ? p1 : (rg == 2 ? p2 : p3));
  const T* Mb = M + (long long)r0 * n + r0;
  for (int c0 = 0; c0 < nm; c0 += strip) {
    const int cb = c0 + cg * 32 * kJ + lane;
    T acc[kJ];
#pragma unroll
    for (int j = 0; j < kJ; ++j) acc[j] = T(0);
    for (int rb = rg; rb < nm; rb += kG * kR) {
      T q[kR][kJ];
#pragma unroll
      for (int u = 0; u < kR; ++u)
#pragma unroll
        for (int j = 0; j < kJ; ++j) {
          const int r = rb + kG * u, c = cb + 32 * j;
          q[u][j] = (r < nm && c < nm) ? Mb[(long long)r * n + c] : T(0);
        }
#pragma unroll
      for (int u = 0; u < kR; ++u) {
        const int r = rb + kG * u;
        const T xr = r < nm ? x[r] : T(0);
#pragma unroll
        for (int j = 0; j < kJ; ++j) acc[j] += q[u][j] * xr;
      }
    }
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
      const int c = cb + 32 * j;
      if (c < nm) mine[c] = acc[j];
    }
  }
  __syncthreads();
  for (int c = tid; c < nm; c += nt) out[c] = scale * (((out[c] + p1[c]) + p2[c]) + p3[c]);
}

// Closing walk of a tridiagonalisation panel over rows and columns
// r0..r0+nm-1 (both relative to the matrix origin, the block is square):
// M -= sum_i PV_i PW_i^T + PW_i PV_i^T over the panel's pairs (absolute
// index), and out_c = scale * sum_r M_new[r][c] x_{r-r0}.  One thread per
// column (or column half, see walk_split) keeps its column's pair entries in
// registers.
template <typename T>
__device__ __noinline__ void panel_walk(T* M, int n, int r0, int nm, const T* PV, const T* PW, const T* x, T* out,
                                        T scale, T* part) {
  constexpr int kPanel = PanelCfg<T>::width, kPanelBatch = PanelCfg<T>::batch;
  const int tid = threadIdx.x, nt = blockDim.x;
  const bool split = walk_split(nm, nt);
  const int half = split ? (nm + 1) >> 1 : nm, nunit = split ? 2 * nm : nm;
  for (int un = tid; un < nunit; un += nt) {
    const int h = un >= nm, jj = h ? un - nm : un;
    const int rb = h ? half : 0, re = h ? nm : half;
    const int c = r0 + jj;
    T vc[kPanel], wc[kPanel];
#pragma unroll
    for (int i = 0; i < kPanel; ++i) {
      vc[i] = PV[(long long)i * n + c];
      wc[i] = PW[(long long)i * n + c];
    }
    T acc = T(0);
    for (int i0 = rb; i0 < re; i0 += kPanelBatch) {
      T q[kPanelBatch];
#pragma unroll
      for (int u = 0; u < kPanelBatch; ++u)
        q[u] = (i0 + u < re) ? M[(long long)(r0 + i0 + u) * n + c] : T(0);
#pragma unroll
      for (int u = 0; u < kPanelBatch; ++u) {
        if (i0 + u < re) {
          const int rr = r0 + i0 + u;
          T y = q[u];
#pragma unroll
          for (int i = 0; i < kPanel; ++i) y -= PV[(long long)i * n + rr] * wc[i] + PW[(long long)i * n + rr] * vc[i];
          M[(long long)rr * n + c] = y;
          acc += y * x[i0 + u];
        }
      }
    }
    if (h) part[jj] = acc;
    else out[jj] = split ? acc : scale * acc;
  }
  if (split) {
    __syncthreads();
    for (int jj = tid; jj < nm; jj += nt) out[jj] = scale * (out[jj] + part[jj]);
  }
}

// Phase 1 of k_reduce_f32: A (n x n, symmetric, row-major) is reduced to
// tridiagonal form in place; reflector k is stored in row k of A from column
// k+1 on (leading 1), its scale in tau[k], the off-diagonal in e.  Out of line
// so that its registers are allocated apart from the later phases.
template <typename T>
__device__ __noinline__ void tridiagonalise(T* A, int n, T* e, T* tau, T* v, T* vn, T* p, T* w, T* d, T* ring,
                                            T* red, T* sh) {
  const int tid = threadIdx.x, nt = blockDim.x;
  // tridiagonalisation in panels of PanelCfg<T>::width reflectors.  Within a
  // panel the trailing block keeps its value A0 from the panel start; step k
  // forms p = tau A0 v and corrects it with the open pairs (v_i, w_i):
  // A = A0 - sum_i (v_i w_i^T + w_i v_i^T).  Only the row that yields the next
  // reflector is brought up to date; the block itself is rewritten once, when
  // the panel closes, fused with the next step's product.
  if (n < 3) return;
  {
    const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    constexpr int kPanel = PanelCfg<T>::width;
    T* PV = ring;               // kPanel x n: v_i of the open panel (absolute index)
    T* PW = ring + kPanel * n;  // kPanel x n: w_i
    __shared__ T dots[2 * kPanel];
    const int nref = n - 2;     // reflectors 0 .. n-3
    reflector(A, n, 0, v, tau, e, red, sh);
    // p0 = tau0 * A[1..][1..] v0
    colwalk<T>(A, n, 1, n - 1, v, p, tau[0], w, d, vn);
    __syncthreads();
    int np = 0;  // pairs in the open panel
    for (int k = 0; k < nref; ++k) {
      const int mm = n - k - 1, b0 = k + 1;
      const T tk = tau[k];
      if (np > 0) {  // dots[i] = w_i . v, dots[np + i] = v_i . v over the block, one warp per dot
        for (int q = wid; q < 2 * np; q += nw) {
          const T* src = (q < np ? PW + (long long)q * n : PV + (long long)(q - np) * n) + b0;
          T acc = T(0);
          for (int j = lane; j < mm; j += 32) acc += src[j] * v[j];
          acc = warp_sum(acc);
          if (lane == 0) dots[q] = acc;
        }
        __syncthreads();
      }
      // p = tau (A0 v - sum_i v_i (w_i.v) + w_i (v_i.v)); w = p - (tau/2)(p.v) v
      T part = T(0);
      for (int j = tid; j < mm; j += nt) {
        T pj = p[j];
        for (int i = 0; i < np; ++i)
          pj -= tk * (PV[(long long)i * n + b0 + j] * dots[i] + PW[(long long)i * n + b0 + j] * dots[np + i]);
        p[j] = pj;
        part += pj * v[j];
      }
      const T pv = block_sum_syev(part, red);
      const T kk = T(0.5) * tk * pv;
      for (int j = tid; j < mm; j += nt) {
        PV[(long long)np * n + b0 + j] = v[j];
        PW[(long long)np * n + b0 + j] = p[j] - kk * v[j];
      }
      ++np;
      __syncthreads();
      // row r = k+1 (columns r..n-1) brought up to date; the last step also row n-1's diagonal
      const int r = k + 1;
      if (r == nref) {
        for (int c = r + tid; c < n; c += nt) {
          T x = A[(long long)r * n + c];
          for (int i = 0; i < np; ++i)
            x -= PV[(long long)i * n + r] * PW[(long long)i * n + c] + PW[(long long)i * n + r] * PV[(long long)i * n + c];
          A[(long long)r * n + c] = x;
        }
        if (tid == 0) {
          T x = A[(long long)(n - 1) * n + n - 1];
          for (int i = 0; i < np; ++i) x -= T(2) * PV[(long long)i * n + n - 1] * PW[(long long)i * n + n - 1];
          A[(long long)(n - 1) * n + n - 1] = x;
        }
        __syncthreads();
      }
      if (r < nref) {
        // the updated row goes straight into reflector r (as `reflector` does from A): the
        // diagonal back to A, the rest through vn, then the reflector (or, for a zero tail,
        // the row itself) back into row r
        const int mr = n - r - 1;
        T part2 = T(0);
        for (int c = r + tid; c < n; c += nt) {
          T x = A[(long long)r * n + c];
          for (int i = 0; i < np; ++i)
            x -= PV[(long long)i * n + r] * PW[(long long)i * n + c] + PW[(long long)i * n + r] * PV[(long long)i * n + c];
          if (c == r) {
            A[(long long)r * n + r] = x;
          } else {
            vn[c - r - 1] = x;
            if (c > r + 1) part2 += x * x;
          }
        }
        const T sigma = block_sum_syev(part2, red);  // synchronises
        if (tid == 0) {
          const T alpha = vn[0];
          if (sigma == T(0)) {
            tau[r] = T(0); e[r] = alpha; sh[0] = T(0); sh[1] = T(0);
          } else {
            const T rr = tb_sqrt(alpha * alpha + sigma);
            const T beta = alpha <= T(0) ? rr : -rr;
            tau[r] = (beta - alpha) / beta;
            e[r] = beta;
            sh[0] = tau[r];
            sh[1] = T(1) / (alpha - beta);
          }
        }
        __syncthreads();
        {
          const T scal = sh[1];
          const bool refl = sh[0] != T(0);
          T* rowr = A + (long long)r * n + r + 1;
          for (int i = tid; i < mr; i += nt) {
            const T u = vn[i];
            const T x = i == 0 ? T(1) : (refl ? u * scal : T(0));
            vn[i] = x;
            rowr[i] = refl ? x : u;
          }
          __syncthreads();
        }
        if (np == kPanel) {  // close the panel: A -= V W^T + W V^T on the block, fused with p_r = tau_r A vn
          panel_walk<T>(A, n, r + 1, n - r - 1, PV, PW, vn, p, tau[r], w);
          np = 0;
        } else {  // p_r = tau_r A0 vn
          colwalk<T>(A, n, r + 1, n - r - 1, vn, p, tau[r], w, d, v);  // v is in PV already
        }
        __syncthreads();
      }
      T* t = v; v = vn; vn = t;
    }
  }
}

// Phase 2 of k_reduce_f32: Z = Q^T from the reflectors left in A and tau by
// tridiagonalise.  ring: kQBlock x n of shared memory.  Out of line like phase 1.
template <typename T>
__device__ __noinline__ void form_q(const T* A, T* Z, int n, const T* tau, T* ring) {
  const int tid = threadIdx.x, nt = blockDim.x;
  // Zc = Q^T (row c of Zc = column c of Q), Q = H_0 H_1 ... H_{n-3},
  // accumulated backwards in blocks of kQBlock reflectors in compact WY form:
  // H_k0 ... H_k1 = I - V T V^T (V = [v_k0 .. v_k1], T upper triangular), so
  // Zc <- Zc H_k1 ... H_k0 = Zc - (Zc V) T^T V^T on rows and columns >= k0+1.
  // Each row of that block is read twice and written once per block instead of
  // once per reflector.  V is staged in shared memory (the rotation ring is not
  // in use yet); one warp per row: partial dots of the row with the kQBlock
  // reflectors, a warp reduction, T^T applied by kQBlock lanes, then the update.
  for (int i = tid >> 5; i < n; i += nt >> 5)
    for (int j = tid & 31; j < n; j += 32) Z[(long long)i * n + j] = i == j ? T(1) : T(0);
  __syncthreads();
  {
    const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    __shared__ T Ts[kQBlock][kQBlock];          // T of the block
    __shared__ T yv[kQBlock][kQBlock];          // V^T V (upper part)
    __shared__ T wps[kEigThreads / 32][kQBlock];  // per warp: (row . V) T^T
    T* Vs = ring;                               // kQBlock x m, m <= n - 1
    const int nref = n - 2;
    for (int k1 = nref - 1; k1 >= 0; k1 -= kQBlock) {
      const int k0 = k1 - kQBlock + 1 > 0 ? k1 - kQBlock + 1 : 0, bb = k1 - k0 + 1;
      const int c0 = k0 + 1, m = n - c0;
      // Vs[j][cc] = v_{k0+j}[c0 + cc]: row k0+j of A from column k0+j+1 (which holds 1), zero before
      for (int e = tid; e < kQBlock * m; e += nt) {
        const int j = e / m, cc = e - j * m, c = c0 + cc;
        Vs[e] = (j < bb && c >= k0 + j + 1) ? A[(long long)(k0 + j) * n + c] : T(0);
      }
      __syncthreads();
      for (int pq = wid; pq < kQBlock * kQBlock; pq += nw) {
        const int j = pq / kQBlock, i = pq - j * kQBlock;
        if (j >= i || i >= bb) continue;  // warp-uniform
        T acc = T(0);
        for (int cc = lane; cc < m; cc += 32) acc += Vs[j * m + cc] * Vs[i * m + cc];
        acc = warp_sum(acc);
        if (lane == 0) yv[j][i] = acc;
      }
      __syncthreads();
      if (tid < kQBlock) {  // T column by column, lane r: T[i][i] = tau, T[0:i][i] = -tau T[0:i][0:i] (V^T v_i)[0:i]
        const int r = tid;
        for (int i = 0; i < kQBlock; ++i) {
          const T ti = i < bb ? tau[k0 + i] : T(0);
          T x = T(0);
          if (i < bb) {
            if (r == i) {
              x = ti;
            } else if (r < i) {
              T sacc = T(0);
              for (int q = r; q < i; ++q) sacc += Ts[r][q] * yv[q][i];
              x = -ti * sacc;
            }
          }
          Ts[r][i] = x;
          __syncwarp(0xffffu);
        }
      }
      __syncthreads();
      for (int r = c0 + wid; r < n; r += nw) {
        T* zr = Z + (long long)r * n + c0;
        T acc[kQBlock];
#pragma unroll
        for (int j = 0; j < kQBlock; ++j) acc[j] = T(0);
        for (int cc = lane; cc < m; cc += 32) {
          const T z = zr[cc];
#pragma unroll
          for (int j = 0; j < kQBlock; ++j) acc[j] += z * Vs[j * m + cc];
        }
#pragma unroll
        for (int j = 0; j < kQBlock; ++j) acc[j] = warp_sum(acc[j]);
        if (lane < kQBlock) {  // (row . V) T^T, entry lane
          T x = T(0);
#pragma unroll
          for (int q = 0; q < kQBlock; ++q) x += acc[q] * Ts[lane][q];
          wps[wid][lane] = x;
        }
        __syncwarp();
        T wp[kQBlock];
#pragma unroll
        for (int j = 0; j < kQBlock; ++j) wp[j] = wps[wid][j];
        for (int cc = lane; cc < m; cc += 32) {
          T z = zr[cc];
#pragma unroll
          for (int j = 0; j < kQBlock; ++j) z -= wp[j] * Vs[j * m + cc];
          zr[cc] = z;
        }
        __syncwarp();
      }
      __syncthreads();
    }
  }

}

}  // namespace

// Structures of kDcMin+ AOs: reflectors and Q in FP32; Q^T (in FP64) into Zd, the
// diagonal and off-diagonal into the first 2n entries of the scratch Sd, from
// where k_syev takes the tridiagonal problem.
__global__ void __launch_bounds__(kEigThreads, 4) k_reduce_f32(DevBatch B, float* __restrict__ Ab,
                                                            float* __restrict__ Zb, double* __restrict__ Zd,
                                                            double* __restrict__ Sd, const int* __restrict__ status,
                                                            const int* __restrict__ active) {
  const int m = B.order ? B.order[blockIdx.x] : blockIdx.x;  // largest structures first
  if (active && !active[m]) return;
  if (status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (on_library(B, n) || n < kDcMin) return;
  const long long mo = B.moff[m];
  float* A = Ab + mo;
  float* Z = Zb + mo;
  extern __shared__ __align__(16) float reduce_sm[];
  float* d = reduce_sm;  // n
  float* e = d + n;      // n
  float* tau = e + n;    // n
  float* v = tau + n;    // n
  float* vn = v + n;     // n
  float* p = vn + n;     // n
  float* w = p + n;      // n
  float* ring = w + n;   // kQBlock x n
  __shared__ float red[kEigThreads / 32];
  __shared__ float sh[4];
  const int tid = threadIdx.x, nt = blockDim.x;
  // symmetrise
  for (int i = tid >> 5; i < n; i += nt >> 5)
    for (int j = i + 1 + (tid & 31); j < n; j += 32) {
      const float s = 0.5f * (A[(long long)i * n + j] + A[(long long)j * n + i]);
      A[(long long)i * n + j] = s;
      A[(long long)j * n + i] = s;
    }
  for (int i = tid; i < n; i += nt) { e[i] = 0.0f; tau[i] = 0.0f; }
  __syncthreads();
  // d: scratch until the end
  tridiagonalise<float>(A, n, e, tau, v, vn, p, w, d, ring, red, sh);
  for (int i = tid; i < n; i += nt) {
    Sd[mo + i] = A[(long long)i * n + i];
    Sd[mo + n + i] = i == n - 2 ? A[(long long)i * n + n - 1] : e[i];
  }
  form_q<float>(A, Z, n, tau, ring);
  __syncthreads();
  for (int i = tid >> 5; i < n; i += nt >> 5)
    for (int j = tid & 31; j < n; j += 32) Zd[mo + (long long)i * n + j] = Z[(long long)i * n + j];
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
