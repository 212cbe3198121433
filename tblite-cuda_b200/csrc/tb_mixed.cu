// Mixed-precision form of the SCF iteration.
//
// Each structure runs in one of two phases (MolState::phase):
//  * mixed (0): the contractions F' = X^T F X, C = X V and P = C f C^T are
//    TF32x3 split-precision tensor-core GEMMs accumulated in FP32 on
//    FP64-stored operands (k_gemm_tc, tb_tc.cu);
//  * FP64 (1): entered once the mixed phase meets the (loosened) convergence
//    test; the same contractions as FP64 GEMMs.  A structure retires only
//    after at least two FP64 iterations and the full-accuracy convergence test.
// In both phases the eigensolve is the FP64 one (tb_syev.cu; Q and the merges
// on the FP64 tensor instruction), in the mixed phase on F' averaged with its
// transpose.  It is faster here than the FP32 reduction with an FP64 refinement
// step of its pairs that it replaced: 64 clusters of 48..384 AOs took 6.9 ms, 0.6
// ms of refinement and 8 N^3 flops of FP64 GEMMs an iteration, and 3.5 ms in FP64
// on clusters of CTAs.  Structures on the library path keep cuSOLVER's FP32
// eigensolver in the mixed phase (vectors orthogonal to about n * 1e-7) and
// one FP64 refinement step of its pairs: Ogita-Aishima iterative refinement
// (T. Ogita, K. Aishima, Japan J. Indust. Appl. Math. 35 (2018) 1007-1035,
// algorithm RefSyEv).  Fermi level, Fock build, Mulliken analysis, energies and
// Broyden mixing are FP64 throughout.
// The kernels here follow the batch conventions of tb_linalg.cu: tile lists of
// (structure, tile row, tile col), per-structure masks, row-major N x N blocks
// at moff[m].
#include "tb_common.cuh"
#include "tb_kernels.h"

namespace tb {

namespace {
constexpr int MT = 64;
}  // namespace

// lo[m] = active and in the mixed phase; hi[m] = active and in the FP64 phase;
// ll[m] / li[m] = lo[m] and on the library / in-house eigensolver.
__global__ void k_phase_masks(DevBatch B, const int* __restrict__ active, const int* __restrict__ phase,
                              int* __restrict__ lo, int* __restrict__ hi, int* __restrict__ ll,
                              int* __restrict__ li) {
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < B.nmol; m += gridDim.x * blockDim.x) {
    const int a = active[m], low = a && phase[m] == 0;
    const int lib = on_library(B, B.ooff[m + 1] - B.ooff[m]);
    lo[m] = low;
    hi[m] = a && phase[m] != 0;
    ll[m] = low && lib;
    li[m] = low && !lib;
  }
}

// F' <- (F' + F'^T) / 2 of the masked structures.  The two triangles of a
// TF32x3 product differ in its last bits (about 1e-7 of the norm); the eigensolvers
// read one of them, both, or their mean, and get the same symmetric matrix this
// way.  A CTA takes a 64 x 64 tile on or above the diagonal and its mirror image,
// as 32 x 32 blocks through shared memory so that rows are read and written whole.
__global__ void k_symmetrize(DevBatch B, const int4* __restrict__ tiles, int ntiles, double* __restrict__ F,
                             const int* __restrict__ mask) {
  __shared__ double up[32][33], low[32][33];
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int4 tl = tiles[t];
    const int m = tl.x;
    if (!mask[m] || tl.z < tl.y) continue;
    const int n = B.ooff[m + 1] - B.ooff[m];
    double* f = F + B.moff[m];
    for (int q = 0; q < 4; ++q) {
      const int i0 = tl.y * MT + 32 * (q >> 1), j0 = tl.z * MT + 32 * (q & 1);
      if (i0 > j0 || j0 >= n) continue;
      __syncthreads();
      for (int e = threadIdx.x; e < 32 * 32; e += blockDim.x) {
        const int r = e / 32, c = e % 32;
        if (i0 + r < n && j0 + c < n) up[r][c] = f[(long long)(i0 + r) * n + j0 + c];
        if (j0 + r < n && i0 + c < n) low[r][c] = f[(long long)(j0 + r) * n + i0 + c];
      }
      __syncthreads();
      for (int e = threadIdx.x; e < 32 * 32; e += blockDim.x) {
        const int r = e / 32, c = e % 32;
        if (i0 + r < n && j0 + c < n) f[(long long)(i0 + r) * n + j0 + c] = 0.5 * (up[r][c] + low[c][r]);
        if (j0 + r < n && i0 + c < n) f[(long long)(j0 + r) * n + i0 + c] = 0.5 * (up[c][r] + low[r][c]);
      }
    }
  }
}

// Af = (float) F' for the masked structures, tile by tile.
__global__ void k_to_f32(DevBatch B, const int4* __restrict__ tiles, int ntiles, const double* __restrict__ F,
                         float* __restrict__ Af, const int* __restrict__ mask) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int4 tl = tiles[t];
    const int m = tl.x;
    if (!mask[m]) continue;
    const int n = B.ooff[m + 1] - B.ooff[m];
    const long long mo = B.moff[m];
    for (int e = threadIdx.x; e < MT * MT; e += blockDim.x) {
      const int i = tl.y * MT + e / MT, j = tl.z * MT + e % MT;
      if (i < n && j < n) Af[mo + (long long)i * n + j] = (float)F[mo + (long long)i * n + j];
    }
  }
}

// V[i][j] = Zf[perm[j]][i] in FP64: eigenvector j (ascending) as column j.
__global__ void k_gather_vectors(DevBatch B, const int4* __restrict__ tiles, int ntiles, const float* __restrict__ Zf,
                                 const int* __restrict__ perm, double* __restrict__ V, const int* __restrict__ mask) {
  __shared__ float tile[32][33];
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int4 tl = tiles[t];
    const int m = tl.x;
    if (!mask[m]) continue;
    const int n = B.ooff[m + 1] - B.ooff[m];
    const long long mo = B.moff[m];
    const int* pm = perm + B.ooff[m];
    // the 64 x 64 tile as four 32 x 32 transposes
    for (int q = 0; q < 4; ++q) {
      const int i0 = tl.y * MT + 32 * (q >> 1), j0 = tl.z * MT + 32 * (q & 1);
      __syncthreads();
      for (int e = threadIdx.x; e < 32 * 32; e += blockDim.x) {
        const int jj = e / 32, ii = e % 32;  // row perm[j0+jj] of Zf read along i (coalesced)
        const int j = j0 + jj, i = i0 + ii;
        tile[jj][ii] = (j < n && i < n) ? Zf[mo + (long long)pm[j] * n + i] : 0.0f;
      }
      __syncthreads();
      for (int e = threadIdx.x; e < 32 * 32; e += blockDim.x) {
        const int ii = e / 32, jj = e % 32;
        const int i = i0 + ii, j = j0 + jj;
        if (i < n && j < n) V[mo + (long long)i * n + j] = (double)tile[jj][ii];
      }
    }
  }
}

// One refinement step, coefficient part, one CTA per masked structure.
// In: G = V^T V and Sm = V^T A V (FP64).
//  1. lambda_i = Sm_ii / G_ii, delta = 2 (||Sm - diag(lambda)||_F +
//     max|lambda| ||I - G||_F) (Frobenius norms bound the published 2-norms
//     from above, so delta is conservative);
//  2. E (overwrites G) with R = I - G:
//       E_ij = (Sm_ij + lambda_j R_ij) / (lambda_j - lambda_i)  if |lambda_j - lambda_i| > delta
//            = R_ij / 2                                          otherwise (and on the diagonal).
// The caller then forms V + V E.  Refined eigenvalues go to w.  Pairs closer than
// delta keep a rotation among themselves, which leaves the density unchanged.
__global__ void __launch_bounds__(256) k_oa_step(DevBatch B, double* __restrict__ G, const double* __restrict__ Sm,
                                                 double* __restrict__ w, const int* __restrict__ mask) {
  const int m = blockIdx.x;
  if (!mask[m]) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  const long long mo = B.moff[m];
  double* g = G + mo;
  const double* s = Sm + mo;
  double* lam = w + B.ooff[m];
  __shared__ double red[32];
  __shared__ double sh_amax;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = nt >> 5;

  // ---- 1. lambda and delta
  double amax = 0.0;
  for (int i = tid; i < n; i += nt) {
    const double l = s[(long long)i * n + i] / g[(long long)i * n + i];
    lam[i] = l;
    amax = fmax(amax, fabs(l));
  }
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (lane == 0) red[wid] = amax;
  __syncthreads();  // also publishes lam
  if (tid == 0) {
    double a = 0.0;
    for (int k = 0; k < nw; ++k) a = fmax(a, red[k]);
    sh_amax = a;
  }
  __syncthreads();
  double so = 0.0, rr = 0.0;
  for (long long e = tid; e < (long long)n * n; e += nt) {
    const int i = (int)(e / n), j = (int)(e - (long long)i * n);
    const double r = (i == j ? 1.0 : 0.0) - g[e];
    const double d = i == j ? s[e] - lam[i] : s[e];
    so += d * d;
    rr += r * r;
  }
  so = block_sum(so, red);
  rr = block_sum(rr, red);
  const double delta = 2.0 * (sqrt(so) + sh_amax * sqrt(rr));

  // ---- 2. E into G
  for (long long e = tid; e < (long long)n * n; e += nt) {
    const int i = (int)(e / n), j = (int)(e - (long long)i * n);
    const double r = (i == j ? 1.0 : 0.0) - g[e];
    const double gap = lam[j] - lam[i];
    double x;
    if (i != j && fabs(gap) > delta) x = (s[e] + lam[j] * r) / gap;
    else x = 0.5 * r;
    g[e] = x;
  }
}

}  // namespace tb
