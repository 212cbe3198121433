// FP64 symmetric eigensolver for structures of kDcMin+ AOs (k_syev): one CTA
// or one thread block cluster per structure, the same bits either way.
//
//  1. Householder tridiagonalisation in panels of kPanel reflectors
//     (tridiag_tiles): within a panel the trailing block keeps its value from
//     the panel start, each step forms its product with one read-only walk of
//     the upper triangle and corrects it with the panel's pairs; the
//     panel-closing walk applies the rank-2 kPanel update on the FP64 tensor
//     instruction, fused with the next product.
//  2. Zc = Q^T accumulated backwards in compact-WY blocks (form_q).
//  3. Tridiagonal eigenproblem by divide and conquer (dc_solve).
//  4. Ascending order by rank (ties by index).
// Together with k_factor and k_gemm this is sygvd (reference
// src/lapack/sygvd.h:4-23).
//
// Work is cut into units whose boundaries and order of additions depend on
// the matrix order alone (row/column tiles of the walks, 64-row tiles of Q,
// 64 x 64 tiles of the merge products, teams of four lanes per secular root),
// never on how many warps share them.  So a structure gives the same bits on
// one CTA (a large batch: 296 structures resident on 148 SMs, throughput) and
// on a cluster of 2..16 (a few structures: latency).  The CTAs of a cluster keep
// identical copies of the vectors (d, e, tau, v, p, w, the panel) in their
// shared memory and repeat the O(n) arithmetic on them; only the units are
// divided, their results exchanged through global memory (walk partials, Z,
// merge blocks) or the peers' shared memory (roots, recomputed z), with one
// cluster barrier per Householder step and three per shared merge.
#include <cooperative_groups.h>

#include "tb_common.cuh"
#include "tb_kernels.h"

namespace tb {

namespace {

constexpr double kEps = 2.220446049250313e-16;
constexpr double kSqrt2 = 1.4142135623730951;
constexpr int kPanel = 8;    // reflectors per tridiagonalisation panel
constexpr int kQBlock = 16;  // reflectors per compact-WY block of the Q accumulation
constexpr int kWarps = kEigThreads / 32;
static_assert(kEigThreads == 256, "the tile shapes below assume eight warps");
static_assert(kPanel <= kRing, "panel exceeds the shared-memory ring");

// The kernels' dynamic shared memory.  The out-of-line functions take offsets
// into it, not pointers: through a generic pointer every access is a generic
// load, several cycles slower on the chains that bound a step.
extern __shared__ __align__(16) double syev_sm[];
__device__ __forceinline__ int sm_off(const double* p) { return (int)(p - syev_sm); }

// ------------------------------------------------------------ CTAs of one structure
struct Group {
  int rank, size;  // this CTA's rank in the structure's cluster; size 1: a CTA of its own
};

// Barrier over the group's CTAs; what they wrote before it (global and peers'
// shared memory) is visible after it.  The warp is brought together first: the
// cluster barrier by itself lets the lanes of a warp that has diverged (the
// four-lane teams leave their loops one by one) arrive and go on separately,
// and a warp-wide instruction after it (mma.sync, a block barrier) is then
// executed by part of a warp, which is an illegal instruction.
__device__ __forceinline__ void group_sync(const Group& g) {
  __syncwarp();
  if (g.size == 1) __syncthreads();
  else cooperative_groups::this_cluster().sync();
  __syncwarp();
}

// *p = v in the shared memory of CTA r of the group (the same variable there)
__device__ __forceinline__ void put_at(double* p, double v, const Group& g, int r) {
  if (r == g.rank) {
    *p = v;
  } else {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    unsigned ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
  }
}
__device__ __forceinline__ void put_at(int* p, int v, const Group& g, int r) {
  if (r == g.rank) {
    *p = v;
  } else {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    unsigned ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
  }
}

// D = A B + D for one 8 x 8 x 4 step.  Lane l = 4 g + t holds A[g][t], B[t][g]
// and D[g][2t], D[g][2t+1].  Volatile: without it the compiler may sink the
// instruction into a branch that only some lanes take (a guarded store of its
// result), where a warp-wide instruction hangs.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Block-wide sum in a fixed order with one barrier.  The caller alternates
// between two `red` buffers of kWarps entries: a buffer is rewritten only
// after the barrier of the call in between, by when everyone has read it.
__device__ __forceinline__ double block_sum_once(double v, double* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) t += red[w];
  return t;
}

// 1/x for the divide-and-conquer inner loops: the hardware reciprocal
// estimate (rcp.approx.ftz.f64) refined by two Newton-Raphson steps for
// f(r) = 1/r - x, r <- r + r (1 - x r), each squaring the relative error;
// within a few units in the last place, not correctly rounded.  x = 0 gives
// inf and |x| = inf gives 0, as 1/x does (the refinement is NaN there).
__device__ __forceinline__ double dc_rcp(double x) {
  double r0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r0) : "d"(x));
  double r = fma(r0, fma(-x, r0, 1.0), r0);
  r = fma(r, fma(-x, r, 1.0), r);
  return r == r ? r : r0;
}

// ------------------------------------------------------------ 1. tridiagonalisation
// Tiles of a walk over an nm x nm block, upper triangle: row tiles of 2^RS
// rows, column strips of 2^CS; unit (I, J) exists where the strip's last
// column reaches the tile's first row.  A unit adds its column products
// (entries on and above the diagonal) into col[I][c] and its row products
// (entries above the diagonal) into row[J][r] of the scratch, each written
// once, and p is their sum in a fixed order.  Wider tiles for larger blocks
// keep at most 38 column and 10 row partials per entry (every CTA of a group
// reads them all).  Coarser tiles (32 x 32, 32 x 64, 64 x 128) left most warps
// of a cluster without a unit: 138 AOs alone 1.03 ms against 0.87, 384 3.40
// against 2.87, 722 10.2 against 8.2, for 3% on a batch of one CTA each.
constexpr int kWalk1 = 224, kWalk2 = 448;  // 16 x 32, 16 x 64, above: 32 x 128
static_assert(kSyevNarrowMaxN == kWalk2 + 1, "k_syev has no walk of the third shape");
__host__ __device__ constexpr int parts(int nm, int shift) { return (nm + (1 << shift) - 1) >> shift; }

// Position in the unit list of one warp: units are numbered strip by strip.
template <int RS>
struct Units {
  int cs, nI, nJ, J = 0, base = 0;
  __device__ __forceinline__ Units(int nm, int cshift) : cs(cshift), nI(parts(nm, RS)), nJ(parts(nm, cshift)) {}
  // row tile of unit u (>= the previous one's); -1 past the last
  __device__ __forceinline__ int seek(int u) {
    for (;;) {
      const int cnt = min(nI, parts((J + 1) << cs, RS));
      if (u - base < cnt) return u - base;
      base += cnt;
      if (++J >= nJ) return -1;
    }
  }
};

// Read-only walk: partials of M x over the upper triangle of the block at Mb
// (nm x nm, row stride n).  A warp reads whole row segments (32 Q contiguous
// entries), U rows of them before using any (U Q loads in flight per lane).
// The row sums of eight rows are reduced on the FP64 tensor instruction: with
// lane l's products of row i as the 4 x 8 operand B_i (entry [l % 4][l / 4])
// and A_i the matrix with ones in row i only, sum_i A_i B_i holds eight partial
// sums of row i in its row i; one addition and two exchanges finish them (the
// same sums by exchanges alone took four times the instructions, and the walk
// is bound by its instructions when three CTAs share an SM).  U changes no
// sum's order.
template <int RS, int CS, int U>
__device__ __noinline__ void walk_read(const double* Mb, int n, int nm, int xo, double* part, int gw, int ngw) {
  constexpr int Q = 1 << (CS - 5);
  static_assert(U % 8 == 0, "rows are reduced in eights");
  const double* x = syev_sm + xo;
  const int lane = threadIdx.x & 31, g = lane >> 2;
  Units<RS> un(nm, CS);
  double* col = part;
  double* row = part + (long long)un.nI * nm;
  for (int u = gw;; u += ngw) {
    __syncwarp();
    const int I = un.seek(u);
    if (I < 0) return;
    const int c0 = un.J << CS, rbeg = I << RS;
    const int rend = min(min(nm, rbeg + (1 << RS)), c0 + (1 << CS));
    double xs[Q], acc[Q];
    int cc[Q];  // column, -1 past the block
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      const int c = c0 + lane + 32 * j;
      cc[j] = c < nm ? c : -1;
      xs[j] = c < nm ? x[c] : 0.0;
      acc[j] = 0.0;
    }
    double* rowp = row + (long long)un.J * nm;
    for (int rb = rbeg; rb < rend; rb += U) {
      double a[U][Q];
      const double* Mr = Mb + (long long)rb * n + c0 + lane;
      // one comparison per entry everywhere: a second copy of this code for the
      // sub-blocks wholly above the diagonal cost a branch per row (11%)
#pragma unroll
      for (int i = 0; i < U; ++i) {
#pragma unroll
        for (int j = 0; j < Q; ++j) a[i][j] = cc[j] - rb >= i ? Mr[32 * j] : 0.0;
        Mr += n;
      }
      double v[U];  // lane's products of each row
#pragma unroll
      for (int i = 0; i < U; ++i) {
        // (rows past the block hold zeros; x is finite there)
        const double xr = x[rb + i];
        v[i] = 0.0;
#pragma unroll
        for (int j = 0; j < Q; ++j) {
          acc[j] += a[i][j] * xr;
          if (cc[j] - rb > i) v[i] += a[i][j] * xs[j];
        }
      }
      double s0[U / 4], s1[U / 4];  // two chains (even and odd rows) per eight rows
#pragma unroll
      for (int k = 0; k < U / 4; ++k) s0[k] = s1[k] = 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k < U / 8; ++k) dmma(s0[2 * k + (i & 1)], s1[2 * k + (i & 1)], g == i ? 1.0 : 0.0, v[8 * k + i]);
#pragma unroll
      for (int k = 0; k < U / 8; ++k) {
        double t = (s0[2 * k] + s1[2 * k]) + (s0[2 * k + 1] + s1[2 * k + 1]);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        const int r = rb + 8 * k + g;
        if ((lane & 3) == 0 && r < nm && TB_GUARD(1, rowp - part + r, 0, (long long)n * n / 2)) rowp[r] = t;
      }
      TB_GUARD_CONVERGE();
    }
#pragma unroll
    for (int j = 0; j < Q; ++j)
      if (cc[j] >= 0 && TB_GUARD(2, (long long)I * nm + cc[j], 0, (long long)n * n / 2))
        col[(long long)I * nm + cc[j]] = acc[j];
  }
}

// Panel-closing walk over the same units: with the
// panel's pairs as K = [PV; PW] and L = [PW; PV] (16 x n, absolute index), the
// upper triangle is updated as M -= K^T L on 16 x 16 sub-tiles of the FP64
// tensor instruction (accumulators initialised from M, stored back), and the
// partials of M_new x are formed from the same fragments.  NB sub-tiles of a
// 16-column block are loaded before the first is used.
template <int RS, int NB>
__device__ __noinline__ void walk_close(double* Mb, int n, int r0, int nm, int CS, int pvo, int xo, double* part, int gw,
                                        int ngw) {
  const double *PV = syev_sm + pvo, *PW = PV + kPanel * n, *x = syev_sm + xo;
  constexpr int RB = 1 << (RS - 4);
  static_assert(RB % NB == 0, "sub-tiles per load round");
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  Units<RS> un(nm, CS);
  double* col = part;
  double* row = part + (long long)un.nI * nm;
  for (int u = gw;; u += ngw) {
    __syncwarp();
    const int I = un.seek(u);
    if (I < 0) return;
    const int J = un.J, c0 = J << CS, rbeg = I << RS;
    double rp[RB][2];
#pragma unroll
    for (int i = 0; i < RB; ++i) rp[i][0] = rp[i][1] = 0.0;
    for (int cw = c0; cw < min(nm, c0 + (1 << CS)); cw += 16) {
      double cs[4] = {0.0, 0.0, 0.0, 0.0};  // column sums, index 2y + h
      double xc[4];
      int cx[4];  // column, -1 past the block
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = cw + 8 * (k >> 1) + 2 * t + (k & 1);
        cx[k] = c < nm ? c : -1;
        xc[k] = c < nm ? x[c] : 0.0;
      }
      double* M0 = Mb + (long long)(rbeg + g) * n + cw + 2 * t;
#pragma unroll
      for (int rb0 = 0; rb0 < RB; rb0 += NB) {
        double d[NB][2][4];
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
          for (int xx = 0; xx < 2; ++xx) {
            const int r = rbeg + 16 * (rb0 + i) + 8 * xx + g;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              d[i][xx][k] = cx[k] >= r ? M0[(long long)(16 * (rb0 + i) + 8 * xx) * n + 8 * (k >> 1) + (k & 1)] : 0.0;
          }
        // (rows and columns past the block take its last one's pairs: their
        // entries are neither stored nor added)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const double* Lc = (ks < 2 ? PW : PV) + (4 * (ks & 1) + t) * n + r0;
          const double* Kr = (ks < 2 ? PV : PW) + (4 * (ks & 1) + t) * n + r0;
          double b[2];
#pragma unroll
          for (int y = 0; y < 2; ++y) b[y] = Lc[min(cw + 8 * y + g, nm - 1)];
#pragma unroll
          for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int xx = 0; xx < 2; ++xx) {
              const double a = -Kr[min(rbeg + 16 * (rb0 + i) + 8 * xx + g, nm - 1)];
#pragma unroll
              for (int y = 0; y < 2; ++y) dmma(d[i][xx][2 * y], d[i][xx][2 * y + 1], a, b[y]);
            }
        }
        // store the upper entries, drop the others from the products
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
          for (int xx = 0; xx < 2; ++xx) {
            const int r = rbeg + 16 * (rb0 + i) + 8 * xx + g;
            const double xr = x[min(r, nm - 1)];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const double z = d[i][xx][k];
              if (cx[k] >= r && TB_GUARD(3, (long long)(r0 + r) * n + r0 + cx[k], 0, (long long)n * n)) {
                M0[(long long)(16 * (rb0 + i) + 8 * xx) * n + 8 * (k >> 1) + (k & 1)] = z;
                cs[k] += z * xr;
              }
              if (cx[k] > r) rp[rb0 + i][xx] += z * xc[k];
            }
          }
        TB_GUARD_CONVERGE();
      }
      // column sums over the eight row lanes g (lane bits 4, 3, 2): lane bit 4
      // ends with y, bit 3 with h
      {
        const bool u16 = lane & 16, u8 = lane & 8;
        const double s0 = u16 ? cs[0] : cs[2], s1 = u16 ? cs[1] : cs[3];
        const double k0 = (u16 ? cs[2] : cs[0]) + __shfl_xor_sync(0xffffffffu, s0, 16);
        const double k1 = (u16 ? cs[3] : cs[1]) + __shfl_xor_sync(0xffffffffu, s1, 16);
        const double s = u8 ? k0 : k1;
        double k = (u8 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, s, 8);
        k += __shfl_xor_sync(0xffffffffu, k, 4);
        const int c = cw + (u16 ? 8 : 0) + 2 * t + (u8 ? 1 : 0);
        if (!(lane & 4) && c < nm && TB_GUARD(4, (long long)I * nm + c, 0, (long long)n * n / 2))
          col[(long long)I * nm + c] = k;
        TB_GUARD_CONVERGE();
      }
    }
#pragma unroll
    for (int rbk = 0; rbk < RB; ++rbk) {  // row sums over the four column lanes t
      const bool u1 = lane & 1;
      double k = (u1 ? rp[rbk][1] : rp[rbk][0]) +
                 __shfl_xor_sync(0xffffffffu, u1 ? rp[rbk][0] : rp[rbk][1], 1);
      k += __shfl_xor_sync(0xffffffffu, k, 2);
      const int r = rbeg + 16 * rbk + (u1 ? 8 : 0) + g;
      if (!(lane & 2) && r < nm && TB_GUARD(5, row - part + (long long)J * nm + r, 0, (long long)n * n / 2))
        row[(long long)J * nm + r] = k;
      TB_GUARD_CONVERGE();
    }
  }
}

// Sum of entry c's partials: column tiles I with rows I <= c, then the strips
// with columns beyond c.  Every load is issued before `between` runs and the
// first addition follows it.
template <int RS, int CS, int NI, int NJ, typename F>
__device__ __forceinline__ double walk_gather(const double* part, int nm, int c, F between) {
  const int ni = (c >> RS) + 1, j0 = (c + 1) >> CS, nj = parts(nm, CS) - j0;  // strips whose last column is > c
  const double* col = part + c;
  const double* row = col + (long long)(parts(nm, RS) + j0) * nm;
  double a[NI], b[NJ];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    a[i] = i < ni ? *col : 0.0;
    col += nm;
  }
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    b[j] = j < nj ? *row : 0.0;
    row += nm;
  }
  between();
  double t = 0.0;
#pragma unroll
  for (int i = 0; i < NI; ++i) t += a[i];
#pragma unroll
  for (int j = 0; j < NJ; ++j) t += b[j];
  return t;
}
template <bool W, typename F>
__device__ __forceinline__ double walk_gather(const double* part, int nm, int c, F between) {
  if (nm <= kWalk1) return walk_gather<4, 5, parts(kWalk1, 4), parts(kWalk1, 5)>(part, nm, c, between);
  if (nm <= kWalk2) return walk_gather<4, 6, parts(kWalk2, 4), parts(kWalk2, 6)>(part, nm, c, between);
  if constexpr (!W) return 0.0;  // (the two-CTA kernel takes orders up to kWalk2 + 1: less code, 3% in a batch)
  else return walk_gather<5, 7, parts(kSyevMaxN, 5), parts(kSyevMaxN, 7)>(part, nm, c, between);
}

// A (n x n, upper triangle used, row-major) to tridiagonal form: reflector k
// (leading 1) in row k of A from column k+1 on, its scale in tau[k], the
// diagonal in d, the off-diagonal in e; d, e and tau complete in every CTA.
// gs: n^2 doubles of scratch for the walk partials, two halves: a CTA may write a
// step's partials while a slower one still gathers the step before's.
template <bool W>
__device__ __forceinline__ void tridiag_tiles(double* A, int n, double* d, double* e, double* tau, double* v, double* vn,
                                           double* p, double* w, double* ring, double* gs, const Group g) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gw = g.rank + g.size * wid, ngw = g.size * kWarps;
  double* PV = ring;               // kPanel x n: v_i of the open panel (absolute index)
  double* PW = ring + kPanel * n;  // kPanel x n: w_i
  __shared__ double dots[2][2 * kPanel], red[2][kWarps], s_alpha;
  // the walks read up to 31 entries of x past the block (against zeros): keep what
  // follows v and vn finite
  for (int i = tid; i < n; i += kEigThreads) v[i] = vn[i] = p[i] = w[i] = 0.0;
  __syncthreads();
  const int half = n * n / 2;
  const int nref = n - 2;  // reflectors 0 .. n-3
  int np = 0;              // pairs in the open panel
  for (int r = 0;; ++r) {
    // row r brought up to date with pair r-1 (formed here from the last walk)
    const int mm = n - r;  // columns r .. n-1, entry j = column r + j
    double part2 = 0.0;
    if (r == 0) {
      for (int j = tid; j < mm; j += kEigThreads) {
        const double x = A[j];
        if (j == 0) d[0] = x;
        else if (j == 1) s_alpha = x;
        else { vn[j - 1] = x; part2 += x * x; }
      }
    } else {
      const double tk = tau[r - 1];
      double* rowr = A + (long long)r * n + r;
      const double* dot = dots[r & 1];
      double part = 0.0;
      for (int j = tid; j < mm; j += kEigThreads) {
        const double raw = rowr[j];
        // the open pairs' part of p and of row r, while the partials arrive
        double cp = 0.0, cx = 0.0;
        const double sum = walk_gather<W>(gs + ((r - 1) & 1) * half, mm, j, [&]() {
          for (int i = 0; i < np; ++i) {
            const double pv = PV[i * n + r + j], pw = PW[i * n + r + j];
            cp += pv * dot[i] + pw * dot[kPanel + i];
            cx += PV[i * n + r] * pw + PW[i * n + r] * pv;
          }
        });
        const double pj = tk * (sum - cp);
        p[j] = pj;
        w[j] = raw - cx;
        part += pj * v[j];
      }
      // reflector r-1 into row r-1: every CTA has read that row's old values
      // before the last group barrier
      if (g.size == 1 || (r - 1) % g.size == g.rank)
        for (int j = tid; j < mm; j += kEigThreads)
          if (TB_GUARD(6, (long long)(r - 1) * n + r + j, 0, (long long)n * n)) A[(long long)(r - 1) * n + r + j] = v[j];
      const double kk = 0.5 * tk * block_sum_once(part, red[0]);
      const double w0 = p[0] - kk;  // v[0] = 1
      for (int j = tid; j < mm; j += kEigThreads) {
        const double vj = v[j], wj = p[j] - kk * vj, x = w[j] - (wj + w0 * vj);
        PV[np * n + r + j] = vj;
        PW[np * n + r + j] = wj;
        if (j == 0) d[r] = x;
        else if (j == 1) s_alpha = x;
        else { vn[j - 1] = x; part2 += x * x; }
      }
      ++np;
    }
    const double sigma = block_sum_once(part2, red[1]);
    const double alpha = s_alpha;
    if (r == nref) {  // the last 2 x 2 block
      if (tid == 0) {
        e[r] = alpha;
        double x = A[(long long)(n - 1) * n + n - 1];
        for (int i = 0; i < np; ++i) x -= 2.0 * PV[i * n + n - 1] * PW[i * n + n - 1];
        d[n - 1] = x;
      }
      break;
    }
    // reflector r: v_new = (1, x / (alpha - beta)), beta = -sign(alpha) |(alpha, x)|,
    // tau = (beta - alpha) / beta = 1 + |alpha| / |beta|; every thread the same
    // scalars, from one reciprocal square root and one refined reciprocal
    const int mr = n - r - 1;
    double scal = 0.0, tr = 0.0, beta = alpha;
    if (sigma != 0.0) {
      const double s2 = alpha * alpha + sigma, ri = rsqrt(s2), rr = s2 * ri;
      beta = alpha <= 0.0 ? rr : -rr;
      tr = 1.0 + fabs(alpha) * ri;
      scal = copysign(dc_rcp(fabs(alpha) + rr), -beta);
    }
    if (tid == 0) { tau[r] = tr; e[r] = beta; vn[0] = 1.0; }
    for (int i = 1 + tid; i < mr; i += kEigThreads) vn[i] *= scal;
    __syncthreads();
    // products with the new reflector over rows and columns r+1 .. n-1
    double* Mb = A + (long long)(r + 1) * n + r + 1;
    double* out = gs + (r & 1) * half;
    if (np == kPanel) {
      if (mr <= kWalk2) walk_close<4, 1>(Mb, n, r + 1, mr, mr <= kWalk1 ? 5 : 6, sm_off(PV), sm_off(vn), out, gw, ngw);
      else if constexpr (W) walk_close<5, 2>(Mb, n, r + 1, mr, 7, sm_off(PV), sm_off(vn), out, gw, ngw);
      np = 0;
    } else {
      if (mr <= kWalk1) walk_read<4, 5, 16>(Mb, n, mr, sm_off(vn), out, gw, ngw);
      else if (mr <= kWalk2) walk_read<4, 6, 16>(Mb, n, mr, sm_off(vn), out, gw, ngw);
      else if constexpr (W) walk_read<5, 7, 16>(Mb, n, mr, sm_off(vn), out, gw, ngw);
      // the next step's w_i . v and v_i . v, one warp each, in every CTA; the
      // last warps of the group first (the walk's units start at warp 0).  Two
      // buffers: a CTA one step behind may still read the other
      double* dot = dots[(r + 1) & 1];
      for (int q = ngw - 1 - gw; q < 2 * np; q += ngw) {
        const double* src = (q < np ? PW + q * n : PV + (q - np) * n) + r + 1;
        double acc = 0.0;
        for (int j = lane; j < mr; j += 32) acc += src[j] * vn[j];
        acc = warp_sum(acc);
        if (lane < g.size) put_at(dot + (q < np ? q : kPanel + q - np), acc, g, lane);
      }
    }
    group_sync(g);
    double* s = v; v = vn; vn = s;
  }
  group_sync(g);  // A's reflectors are written; the partials have been read
}

// ------------------------------------------------------------ 2. Q
// One compact-WY block applied to eight rows of Z by one warp, on the FP64
// tensor instruction: with Zt the rows row0..row0+7 (lane (g, t) = (lane / 4,
// lane % 4) owns row row0 + g) and columns c0..n-1 (m of them) of Z, Vs the
// block's reflectors (kQBlock x m, shared memory, row stride mp) and Ts its T:
//   Wm = Zt Vs^T, Wt = Wm T^T, Zt -= Wt Vs.
// Wm and Wt (8 x kQBlock) stay in registers -- an accumulator becomes the next
// product's left operand by exchanges among the four lanes of a row -- so the
// warps share nothing but Vs and Ts and meet no barrier inside a block.  U
// steps of four columns are loaded before the first is used.
template <int U>
__device__ __forceinline__ void formq_rows(double* Z, int n, int row0, int c0, int m, const double* Vs, int mp,
                                           const double (*Ts)[kQBlock + 4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int r = row0 + g;
  const bool valid = r >= c0 && r < n;
  double* zr = Z + (long long)r * n + c0;
  double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};  // Wm[g][8y + 2t], Wm[g][8y + 2t + 1]
  const double* Vg = Vs + g * mp + t;
  int k0 = 0;
  for (; k0 + 4 * U <= m; k0 += 4 * U) {
    __syncwarp();
    double z[U];
#pragma unroll
    for (int u = 0; u < U; ++u) z[u] = valid ? zr[k0 + 4 * u + t] : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int y = 0; y < 2; ++y) dmma(a0[y], a1[y], z[u], Vg[8 * y * mp + k0 + 4 * u]);
  }
  for (; k0 < m; k0 += 16) {  // the rest, four steps at a time (past column m: zeros times zeros)
    __syncwarp();
    double z[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) z[u] = (valid && k0 + 4 * u + t < m) ? zr[k0 + 4 * u + t] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const double b = k0 + 4 * u + t < m ? Vg[8 * y * mp + k0 + 4 * u] : 0.0;
        dmma(a0[y], a1[y], z[u], b);
      }
  }
  // left-operand fragment s (columns 4s + t) of an 8 x 16 accumulator
  auto left = [&](const double* d0, const double* d1, int s) {
    const int src = (lane & ~3) | ((4 * (s & 1) + t) >> 1);
    const double x0 = __shfl_sync(0xffffffffu, d0[s >> 1], src), x1 = __shfl_sync(0xffffffffu, d1[s >> 1], src);
    return (t & 1) ? x1 : x0;
  };
  double w0[2] = {0.0, 0.0}, w1[2] = {0.0, 0.0};  // Wt
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const double a = left(a0, a1, s);
#pragma unroll
    for (int y = 0; y < 2; ++y) dmma(w0[y], w1[y], a, Ts[8 * y + g][4 * s + t]);
  }
  double wf[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) wf[s] = -left(w0, w1, s);
  const double* Vt = Vs + t * mp + g;
  constexpr int V = U / 2;  // 8-column fragments per round
  int ct = 0;
  for (; ct + 8 * V <= m; ct += 8 * V) {
    __syncwarp();
    double d0[V], d1[V];
#pragma unroll
    for (int y = 0; y < V; ++y) {
      const int c = ct + 8 * y + 2 * t;
      d0[y] = valid ? zr[c] : 0.0;
      d1[y] = valid ? zr[c + 1] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int y = 0; y < V; ++y) dmma(d0[y], d1[y], wf[s], Vt[4 * s * mp + ct + 8 * y]);
    if (valid)
#pragma unroll
      for (int y = 0; y < V; ++y) {
        const int c = ct + 8 * y + 2 * t;
        if (!TB_GUARD(7, (long long)r * n + c0 + c + 1, 0, (long long)n * n)) continue;
        zr[c] = d0[y];
        zr[c + 1] = d1[y];
      }
  }
  for (; ct < m; ct += 16) {
    __syncwarp();
    double d0[2], d1[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int c = ct + 8 * y + 2 * t;
      d0[y] = (valid && c < m) ? zr[c] : 0.0;
      d1[y] = (valid && c + 1 < m) ? zr[c + 1] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const double b = ct + 8 * y + g < m ? Vt[4 * s * mp + ct + 8 * y] : 0.0;
        dmma(d0[y], d1[y], wf[s], b);
      }
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int c = ct + 8 * y + 2 * t;
      if (valid && c < m && TB_GUARD(8, (long long)r * n + c0 + c, 0, (long long)n * n)) zr[c] = d0[y];
      if (valid && c + 1 < m && TB_GUARD(8, (long long)r * n + c0 + c + 1, 0, (long long)n * n)) zr[c + 1] = d1[y];
    }
  }
}

// Zc = Q^T (row c of Zc = column c of Q), Q = H_0 H_1 ... H_{n-3}, accumulated
// backwards in blocks of kQBlock reflectors in compact WY form: H_k0 ... H_k1
// = I - V T V^T (V = [v_k0 .. v_k1], T upper triangular), so
// Zc <- Zc H_k1 ... H_k0 = Zc - (Zc V) T^T V^T on rows and columns >= k0+1.
// Every row of Zc is transformed independently of the others: warp gw of the
// group's ngw takes the rows of the 8-row groups gw, gw + ngw, ... throughout,
// and the CTAs never wait for one another; each forms V and T of the block
// itself.  vbuf: 20 n elements of shared memory.
template <bool W>
__device__ __forceinline__ void form_q(const double* A, double* Z, int n, const double* tau, double* vbuf,
                                    const Group grp) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = lane >> 2, t = lane & 3;
  const int gw = grp.rank + grp.size * wid, ngw = grp.size * kWarps;
  for (int q = gw; 8 * q < n; q += ngw)
    for (int i = 8 * q; i < min(n, 8 * q + 8); ++i)
      for (int j = lane; j < n; j += 32) Z[(long long)i * n + j] = i == j ? 1.0 : 0.0;
  __shared__ double Ts[kQBlock][kQBlock + 4];  // T of the block (rows padded against bank conflicts)
  __shared__ double yv[2][3][64];              // V V^T: fragments (0,0), (0,1), (1,1) of 8 x 8, two halves of the columns
  double* Vs = vbuf;
  const int nref = n - 2;
  for (int k1 = nref - 1; k1 >= 0; k1 -= kQBlock) {
    const int k0 = k1 - kQBlock + 1 > 0 ? k1 - kQBlock + 1 : 0, bb = k1 - k0 + 1;
    const int c0 = k0 + 1, m = n - c0;
    const int mp = m + ((20 - (m & 15)) & 15);  // row stride 4 mod 16: conflict-free fragments of both kinds
    __syncthreads();  // Vs and Ts of the previous block have been read
    // Vs[j][cc] = v_{k0+j}[c0 + cc]: row k0+j of A from column k0+j+1 (which holds 1), zero before
    for (int j = wid; j < kQBlock; j += kWarps) {
      const double* Ar = A + (long long)(k0 + j) * n + c0;
#pragma unroll 4
      for (int cc = lane; cc < m; cc += 32) Vs[j * mp + cc] = (j < bb && cc >= j) ? Ar[cc] : 0.0;
    }
    __syncthreads();
    if (wid < 6) {  // fragment (fa, fb) of V V^T over one half of the columns, one warp each
      const int half = wid / 3, f = wid % 3, fa = f == 2, fb = f > 0;
      const int steps = (m + 3) / 4, kb = half ? 4 * ((steps + 1) / 2) : 0, ke = half ? m : min(m, 4 * ((steps + 1) / 2));
      double y0[2] = {0.0, 0.0}, y1[2] = {0.0, 0.0};
      for (int k = kb; k < ke; k += 8) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = k + 4 * h + t;
          const double a = kk < ke ? Vs[(8 * fa + g) * mp + kk] : 0.0, b = kk < ke ? Vs[(8 * fb + g) * mp + kk] : 0.0;
          dmma(y0[h], y1[h], a, b);
        }
      }
      yv[half][f][8 * g + 2 * t] = y0[0] + y0[1];
      yv[half][f][8 * g + 2 * t + 1] = y1[0] + y1[1];
    }
    __syncthreads();
    if (tid < kQBlock) {  // T[i][i] = tau, T[0:i][i] = -tau T[0:i][0:i] (V^T v_i)[0:i]; lane r: row r
      const int r = tid;
      double acc[kQBlock];
#pragma unroll
      for (int i = 0; i < kQBlock; ++i) acc[i] = 0.0;
#pragma unroll
      for (int q = 0; q < kQBlock; ++q) {
        const double tq = q < bb ? tau[k0 + q] : 0.0;
        const double x = q == r ? tq : (q > r ? -tq * acc[q] : 0.0);
        Ts[r][q] = x;
#pragma unroll
        for (int i = q + 1; i < kQBlock; ++i) {
          const int f = (q >> 3) + (i >> 3), xy = 8 * (q & 7) + (i & 7);
          acc[i] += x * (yv[0][f][xy] + yv[1][f][xy]);
        }
      }
    }
    __syncthreads();
    for (int q = (c0 >> 3) + ((gw - (c0 >> 3)) % ngw + ngw) % ngw; 8 * q < n; q += ngw)
      formq_rows<W ? 32 : 16>(Z, n, 8 * q, c0, m, Vs, mp, Ts);
  }
}

// ------------------------------------------------------------ 3. divide and conquer (Cuppen)
// Tridiagonal T (d, e) = diag(T_left, T_right) + rho v v^T torn at every node
// of a halving tree down to leaves of at most kDcLeaf rows; the eigenvector
// matrix G of each node (rows = eigenvectors in T's index space, an m x m
// diagonal block of an n x n buffer) is built bottom-up by rank-one merges:
//  * z = [last column of G_left ; sign(e) * first column of G_right], of norm
//    sqrt(2) (columns of orthogonal matrices) and left so: divided by its norm,
//    which rounds the same way in every merge, the rank-one term came out short
//    by up to 0.8 eps (dense matrices of 256 rows lost 0.65 eps of their
//    Frobenius norm); eigenvalues sorted;
//  * deflation (tolerance 8 eps max(|delta|max, 2 rho), 2 rho = rho |z|^2):
//    entries with sqrt(2) rho |z_i| below it keep their eigenpair; adjacent close pairs
//    are rotated so that one z entry vanishes (LAPACK dlaed2's two tests);
//  * roots of the secular equation 1 + rho sum z_i^2 / (delta_i - lambda) = 0
//    by bracketed two-pole rational interpolation (Bunch, Nielsen and Sorensen
//    1978), each root kept as (nearest pole, offset) so that delta_i - lambda
//    keeps full relative accuracy;
//  * z recomputed from the roots (Gu and Eisenstat 1994) so the eigenvectors
//    w_j = z_i / (delta_i - lambda_j) are orthogonal to working accuracy;
//  * G_node = W G_children as a tiled product.
// Finally Zc <- G Zc (Zc = Q^T), and the eigenvalues are left in d.
// kDcMin, kDcK, kDcBs, kDcTileElems and dc_ws_elems (tb_kernels.h): the
// workspace starts at tau and runs to the end of the dynamic shared memory,
// which syev_smem_bytes sizes so that every structure of kDcMin+ rows has it.
//
// The roots, the recomputed z and the norms are each formed by a team of four
// lanes (terms sub, sub + 4, ..., combined by two exchanges): a root's chain of
// passes over the k terms is four times shorter than with one thread, and a
// group's CTAs take every size-th root.

template <int T = 4>
__device__ __forceinline__ double team_sum(double v, unsigned mask) {
  if constexpr (T == 4) {
    v += __shfl_xor_sync(mask, v, 1);
    v += __shfl_xor_sync(mask, v, 2);
  }
  return v;
}
__device__ __forceinline__ double team_mul(double v, unsigned mask) {
  v *= __shfl_xor_sync(mask, v, 1);
  v *= __shfl_xor_sync(mask, v, 2);
  return v;
}

// Root j of 1 + rho sum_i z_i^2 / (dl_i - lambda) = 0 (dl strictly ascending,
// rho > 0): lambda = dl[*o] + *tau, by the T (4 or 1) lanes of `mask` (sub 0..T-1).
// The two poles p = min(j, k-2) and p+1 beside the root are treated apart: the
// start solves the equation with the other terms frozen at the interval's
// middle (for the last root, half way to its upper bound), each step replaces
// the terms up to p and those beyond by one pole each with the same value and
// slope; a step out of the bracket bisects it.  An accepted root takes the Newton
// step of its last evaluation: below the acceptance bound (8 eps of the terms)
// the iterates still lie to one side.
template <int T>
__device__ __forceinline__ void secular_root(int j, int k, const double* dl, const double* z, double rho, int sub, unsigned mask,
                             int* o_out, double* tau_out) {
  if (k == 1) {
    *o_out = 0;
    *tau_out = rho * z[0] * z[0];
    return;
  }
  const bool last = j == k - 1;
  const int p = last ? k - 2 : j;
  const double del = dl[p + 1] - dl[p], zp = z[p] * z[p], zq = z[p + 1] * z[p + 1];
  double top = 0.0;  // last root: upper bound of lambda - dl[k-1]
  if (last) {
    for (int i = sub; i < k; i += T) top += z[i] * z[i];
    top = rho * team_sum<T>(top, mask);
  }
  const double mid = 0.5 * (last ? top : del);  // from dl[j]
  double c = 0.0;  // the other terms at mid, plus 1 / rho
#pragma unroll 4
  for (int i = sub; i < k; i += T) {
    const double q = z[i] * z[i] * dc_rcp((dl[i] - dl[j]) - mid);
    c += i == p || i == p + 1 ? 0.0 : q;
  }
  c = dc_rcp(rho) + team_sum<T>(c, mask);
  int o = j;
  double lo = 0.0, hi = mid, tau;
  const double rm = dc_rcp(mid);
  if (!last && c + (zq - zp) * rm >= 0.0) {  // root in the lower half: x from dl[p], c x^2 - a x + b = 0
    const double a = c * del + zp + zq, b = zp * del, sq = sqrt(fmax(a * a - 4.0 * b * c, 0.0));
    tau = a > 0.0 ? 2.0 * b * dc_rcp(a + sq) : (a - sq) * dc_rcp(2.0 * c);
  } else {  // x from dl[p + 1]: c x^2 + a x - b = 0, negative below it, positive past the last
    const double a = c * del - zp - zq, b = zq * del, sq = sqrt(fmax(a * a + 4.0 * b * c, 0.0));
    if (last) {
      hi = top;
      tau = a > 0.0 ? 2.0 * b * dc_rcp(a + sq) : (sq - a) * dc_rcp(2.0 * c);
    } else {
      o = j + 1;
      lo = -mid;
      hi = 0.0;
      tau = a < 0.0 ? 2.0 * b * dc_rcp(a - sq) : -(a + sq) * dc_rcp(2.0 * c);
    }
  }
  if (!(tau > lo && tau < hi)) tau = 0.5 * (lo + hi);
  const double base = dl[o];
  for (int it = 0; it < 100; ++it) {
    double psi = 0.0, phi = 0.0, dpsi = 0.0, dphi = 0.0;
    // (one loop without branches: four terms' chains overlap)
#pragma unroll 4
    for (int i = sub; i < k; i += T) {
      const double r = dc_rcp((dl[i] - base) - tau);
      const double q = z[i] * z[i] * r, dq = q * r;
      const bool left = i <= p;
      psi += left ? q : 0.0; dpsi += left ? dq : 0.0;
      phi += left ? 0.0 : q; dphi += left ? 0.0 : dq;
    }
    psi = rho * team_sum<T>(psi, mask); phi = rho * team_sum<T>(phi, mask);
    dpsi = rho * team_sum<T>(dpsi, mask); dphi = rho * team_sum<T>(dphi, mask);
    const double f = 1.0 + psi + phi;
    const double err = kEps * (8.0 * (fabs(psi) + fabs(phi)) + 3.0 + fabs(tau) * (dpsi + dphi));
    if (fabs(f) <= err) {
      const double tn = tau - f * dc_rcp(dpsi + dphi);
      if (tn > lo && tn < hi) tau = tn;
      break;
    }
    if (f < 0.0) lo = tau; else hi = tau;
    if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi))) break;
    // psi ~ c1 + s1 / (a - eta), phi ~ c2 + s2 / (b - eta)
    const double a = (dl[p] - base) - tau, b = (dl[p + 1] - base) - tau;
    const double s1 = dpsi * a * a, c1 = psi - dpsi * a, s2 = dphi * b * b, c2 = phi - dphi * b;
    const double C = 1.0 + c1 + c2;
    const double Bq = C * (a + b) + s1 + s2;
    const double sq = sqrt(fmax(Bq * Bq - 4.0 * C * a * b * f, 0.0));
    const double q = Bq >= 0.0 ? 0.5 * (Bq + sq) : 0.5 * (Bq - sq);
    double tn = tau + a * b * f * dc_rcp(q);
    if (!(tn > lo && tn < hi)) tn = tau + q * dc_rcp(C);
    if (!(tn > lo && tn < hi)) tn = 0.5 * (lo + hi);
    tau = tn;
  }
  *o_out = o;
  *tau_out = tau;
}

// Out[(r0 + j) ld + c0 + c] = sum_i gen(j, i) In[(srow ? srow[i] : i) ld + c0 + c]
// for j < nrow, c < ncol, i < kdim, the group's CTAs taking every size-th of
// the 64 x 64 output tiles (numbered from first); slabs of kDcK staged in
// shared memory (Wt: 64 x kDcK, Bt: kDcK x 64 with padded rows), the next
// slab (its loads and generated entries) fetched into registers while the
// current one is multiplied on the FP64 tensor instruction (each warp a
// 16 x 32 block as 2 x 4 fragments of 8 x 8).
template <typename Gen>
__device__ void dc_gemm(int nrow, int kdim, int ncol, Gen gen, const double* In, const int* srow, double* Out, int r0,
                        int c0, int ld, double* Wt, double* Bt, const Group g, int first = 0) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, gl = lane >> 2, tg = lane & 3;
  const int wrow = (warp >> 1) * 16, wcol = (warp & 1) * 32;  // this warp's block of the tile
  int idx = first;
  for (int j0 = 0; j0 < nrow; j0 += 64) {
    for (int cb = 0; cb < ncol; cb += 64, ++idx) {
      if (g.size > 1 && idx % g.size != g.rank) continue;
      double acc[2][4], acc2[2][4];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = acc2[a][b] = 0.0;
      constexpr int kPer = 64 * kDcK / kEigThreads;  // slab entries per thread
      double wr[kPer], br[kPer];
      auto fetch = [&](int i0) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const int x = tid + u * kEigThreads;
          const int jj = x / kDcK, kk = x - jj * kDcK, j = j0 + jj, i = i0 + kk;
          wr[u] = (j < nrow && i < kdim) ? gen(j, i) : 0.0;
          const int kb = x >> 6, cc = x & 63, ib = i0 + kb;
          br[u] = (ib < kdim && cb + cc < ncol) ? In[(long long)(srow ? srow[ib] : ib) * ld + c0 + cb + cc] : 0.0;
        }
      };
      fetch(0);
      for (int i0 = 0; i0 < kdim; i0 += kDcK) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const int x = tid + u * kEigThreads;
          Wt[x] = wr[u];
          Bt[(x >> 6) * kDcBs + (x & 63)] = br[u];
        }
        __syncthreads();
        if (i0 + kDcK < kdim) fetch(i0 + kDcK);
#pragma unroll
        for (int k4 = 0; k4 < kDcK; k4 += 4) {
          double af[2], bf[4];
#pragma unroll
          for (int x = 0; x < 2; ++x) af[x] = Wt[(wrow + 8 * x + gl) * kDcK + k4 + tg];
#pragma unroll
          for (int y = 0; y < 4; ++y) bf[y] = Bt[(k4 + tg) * kDcBs + wcol + 8 * y + gl];
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) dmma(acc[x][y], acc2[x][y], af[x], bf[y]);
        }
        __syncthreads();
      }
      // fragment (x, y): rows wrow + 8x + gl, columns wcol + 8y + 2 tg + {0, 1}
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int j = j0 + wrow + 8 * x + gl;
        if (j >= nrow) continue;
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          const int c = cb + wcol + 8 * y + 2 * tg;
          if (c < ncol && TB_GUARD(11, (long long)(r0 + j) * ld + c0 + c, 0, (long long)ld * ld))
            Out[(long long)(r0 + j) * ld + c0 + c] = acc[x][y];
          if (c + 1 < ncol && TB_GUARD(11, (long long)(r0 + j) * ld + c0 + c + 1, 0, (long long)ld * ld))
            Out[(long long)(r0 + j) * ld + c0 + c + 1] = acc2[x][y];
        }
      }
    }
  }
}

// One merge of the node [lo, hi) torn at t by the CTAs of g: children's G
// blocks in Gi (the node's diagonal block), eigenvalues in d[lo, hi) of every
// CTA.  The rows lo..hi-1 of V (columns vc0 .. vc0+vcols-1; V = Gi itself, or
// the children's eigenvectors already applied to Zc) are combined into the
// same rows of Out and the merged eigenvalues written to d[lo, hi) of every
// CTA.  V is overwritten.  ws: dc_ws_elems(hi - lo) doubles.
template <bool W>
__device__ __noinline__ void dc_merge(int dofs, int eofs, int n, int ld, int lo, int t, int hi, double* Gi, double* V,
                                      int vc0, int vcols, double* Out, int wofs, const Group g) {
  double *d = syev_sm + dofs, *ws = syev_sm + wofs;
  const double* e = syev_sm + eofs;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gw = g.rank * kWarps + wid, ngw = g.size * kWarps;
  const int m = hi - lo;
  double* delta = ws;          // m: sorted eigenvalues (rotated pairs updated)
  double* zs = delta + m;      // m: sorted z
  double* dl = zs + m;         // k: non-deflated delta
  double* zl = dl + m;         // k: their z, then the recomputed z
  double* tv = zl + m;         // k: root offsets
  double* inrm = tv + m;       // k: 1 / |w_j|
  double* rc = inrm + m;       // rotations: cosine
  double* rsn = rc + m;        //            sine
  double* Wt = rsn + m;
  double* Bt = Wt + 64 * kDcK;
  int* rowof = reinterpret_cast<int*>(Wt + kDcTileElems);  // m: row of sorted entry s
  int* flg = rowof + m;   // m: deflated
  int* ndl = flg + m;     // m: sorted index of the k non-deflated, then of the deflated
  int* rp = ndl + m;      // rotations: rows
  int* rq = rp + m;
  int* ori = rq + m;      // k: root origin (index into dl)
  int* srow = ori + m;    // k: row of non-deflated entry
  __shared__ int s_k, s_nrot;
  const double ev = e[t - 1];
  const double rho = fabs(ev), sg = ev >= 0.0 ? 1.0 : -1.0;
  // children's blocks are diagonal sub-blocks: clear the rest of the node's block
  if (V == Gi)
    for (int r = lo + gw; r < hi; r += ngw)
      for (int c = (r < t ? t : lo) + lane; c < (r < t ? hi : t); c += 32) Gi[(long long)r * ld + c] = 0.0;
  // z (in rc until the rotations are formed)
  for (int r = lo + tid; r < hi; r += kEigThreads) {
    const double z = r < t ? Gi[(long long)r * ld + t - 1] : sg * Gi[(long long)r * ld + t];
    rc[r - lo] = z;
    rowof[r - lo] = r;  // valid rows even where non-finite eigenvalues leave ranks unset below
    delta[r - lo] = zs[r - lo] = 0.0;
  }
  __syncthreads();
  // rank sort of the eigenvalues (ties by index)
  for (int r = lo + tid; r < hi; r += kEigThreads) {
    const double dr = d[r];
    int rank = 0;
    for (int q = lo; q < hi; ++q) {
      const double dq = d[q];
      rank += (dq < dr || (dq == dr && q < r)) ? 1 : 0;
    }
    rowof[rank] = r;
    delta[rank] = dr;
    zs[rank] = rc[r - lo];
  }
  __syncthreads();
  if (tid < 32) {  // deflation scan and compaction, warp 0
    double dmax = 0.0;
    for (int s = lane; s < m; s += 32) dmax = fmax(dmax, fabs(delta[s]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    const double tol = 8.0 * kEps * fmax(dmax, 2.0 * rho);
    int kc = 0;  // entries with a z of their own, in order (in ndl)
    for (int s0 = 0; s0 < m; s0 += 32) {
      const int s = s0 + lane;
      const bool keep = s < m && !(kSqrt2 * rho * fabs(zs[s]) <= tol);
      if (s < m) flg[s] = keep ? 0 : 1;
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (keep) ndl[kc + __popc(bal & ((1u << lane) - 1u))] = s;
      kc += __popc(bal);
    }
    __syncwarp();
    // close pair (a, s) of neighbours: the rotation zeroing z_a (c = z_s / tau, sn = -z_a / tau,
    // tau = |(z_a, z_s)|) deflates when |(d_s - d_a) c sn| <= tol, tested as
    // |d_s - d_a| |z_a z_s| <= tol tau^2 without the square root
    auto close_pair = [&](int q) {
      const int a = ndl[q - 1], s = ndl[q];
      const double za = zs[a], zb = zs[s];
      return fabs(delta[s] - delta[a]) * fabs(za * zb) <= tol * (za * za + zb * zb);
    };
    // A rotation changes its second entry, so only the next pair: 32 pairs are
    // tested at once, and one again after the rotation before it.  (One lane
    // testing all in order is a chain of dependent shared-memory reads: with it
    // a 384-AO structure took 2.49 ms, now 2.38, 722 AOs 7.27 and 7.06 ms, 1024
    // clusters of 48..384 AOs 17.8 and 17.6 ms.)
    int nrot = 0;
    for (int q0 = 0; q0 < kc; q0 += 32) {
      const int q = q0 + lane;
      unsigned hits = __ballot_sync(0xffffffffu, q > 0 && q < kc && close_pair(q));
      while (hits) {
        const int b = __ffs(hits) - 1;
        hits &= hits - 1;
        if (lane == 0) {
          const int a = ndl[q0 + b - 1], s = ndl[q0 + b];
          const double za = zs[a], zb = zs[s], tau = sqrt(za * za + zb * zb);
          const double c = zb / tau, sn = -za / tau;
          rp[nrot] = rowof[a]; rq[nrot] = rowof[s]; rc[nrot] = c; rsn[nrot] = sn;
          zs[s] = tau; zs[a] = 0.0;
          const double da = delta[a], ds = delta[s];
          delta[a] = da * c * c + ds * sn * sn;
          delta[s] = da * sn * sn + ds * c * c;
          flg[a] = 1;
        }
        ++nrot;
        __syncwarp();
        if (b < 31 && q0 + b + 1 < kc) {
          const unsigned bit = 2u << b;
          hits = close_pair(q0 + b + 1) ? hits | bit : hits & ~bit;
        }
        __syncwarp();
      }
    }
    if (lane == 0) s_nrot = nrot;
    __syncwarp();
    // non-deflated entries first, then the deflated ones, each in order
    int k = 0;
    for (int s0 = 0; s0 < m; s0 += 32) {
      const int s = s0 + lane;
      const bool keep = s < m && !flg[s];
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int pos = k + __popc(bal & ((1u << lane) - 1u));
        ndl[pos] = s; dl[pos] = delta[s]; zl[pos] = zs[s]; srow[pos] = rowof[s];
      }
      k += __popc(bal);
    }
    int q = k;
    for (int s0 = 0; s0 < m; s0 += 32) {
      const int s = s0 + lane;
      const bool defl = s < m && flg[s];
      const unsigned bal = __ballot_sync(0xffffffffu, defl);
      if (defl) ndl[q + __popc(bal & ((1u << lane) - 1u))] = s;
      q += __popc(bal);
    }
    if (lane == 0) s_k = k;
  }
  __syncthreads();
  const int k = s_k, nrot = s_nrot;
  // close-pair rotations on the rows, one thread per column, in order (a group
  // first waits until its CTAs have read z and cleared their rows)
  if (nrot > 0 && g.size > 1) group_sync(g);
  for (int c = vc0 + g.rank * kEigThreads + tid; c < vc0 + vcols; c += g.size * kEigThreads)
    for (int q = 0; q < nrot; ++q) {
      double* pa = V + (long long)rp[q] * ld + c;
      double* pb = V + (long long)rq[q] * ld + c;
      const double a = *pa, b = *pb;
      *pa = rc[q] * a + rsn[q] * b;
      *pb = rc[q] * b - rsn[q] * a;
    }
  // teams of four lanes: roots, recomputed z, norms
  const int sub = lane & 3, team = tid >> 2, gteam = g.rank + g.size * team, nteam = g.size * (kEigThreads / 4);
  const unsigned mask = 0xfu << (lane & ~3);
  for (int j = gteam; j < k; j += nteam) {
    int o;
    double tj;
    secular_root<4>(j, k, dl, zl, rho, sub, mask, &o, &tj);
    for (int r = sub; r < g.size; r += 4) {
      put_at(ori + j, o, g, r);
      put_at(tv + j, tj, g, r);
    }
  }
  group_sync(g);  // (brings the teams of a warp together again)
  // z of the k poles, recomputed from the roots (Gu and Eisenstat: every ratio
  // in (0, 1]); the new entry keeps the old one's sign, so a lane of the team
  // that reads it late reads the same sign
  for (int i = gteam; i < k; i += nteam) {
    const double di = dl[i];
    double prod = 1.0;
#pragma unroll 4
    for (int j = sub; j < k - 1; j += 4)  // root j over pole j, from the entry's own pole on j + 1
      prod *= ((dl[ori[j]] - di) + tv[j]) * dc_rcp(dl[j + (j >= i)] - di);
    prod = team_mul(prod, mask) * (((dl[ori[k - 1]] - di) + tv[k - 1]) / rho);
    const double z = copysign(sqrt(fmax(prod, 0.0)), zl[i]);
    for (int r = sub; r < g.size; r += 4) put_at(zl + i, z, g, r);
  }
  group_sync(g);
  // W formed once (row stride n) instead of once per 64-column tile of the
  // product, where Gi has a free k x k block: at the root all of Gi is free
  // once z has been read; below it, rows lo.. of Gi beside the node's block
  // (columns hi.. or ..lo) belong to no node of this level
  double* Wb = nullptr;
  if (V != Gi) Wb = Gi;
  else if (hi + k <= n) Wb = Gi + (long long)lo * ld + hi;
  else if (lo >= k) Wb = Gi + (long long)lo * ld + (lo - k);
  // norms: of this CTA's rows of W (rows gw, gw + ngw, ...), of all rows where
  // every tile generates its own
  const int r0w = g.rank * kWarps;
  const int nq = !Wb ? k : (k > r0w ? kWarps * ((k - r0w + ngw - 1) / ngw) : 0);
  for (int q = team; q < nq; q += kEigThreads / 4) {
    const int j = Wb ? (q / kWarps) * ngw + r0w + q % kWarps : q;
    if (j >= k) continue;
    const double bj = dl[ori[j]], tj = tv[j];
    double s = 0.0;
#pragma unroll 4
    for (int i = sub; i < k; i += 4) {
      const double w = zl[i] * dc_rcp((dl[i] - bj) - tj);
      s += w * w;
    }
    s = team_sum(s, mask);
    if (sub == 0) inrm[j] = 1.0 / sqrt(s);
  }
  __syncwarp();
  __syncthreads();
  // roots: Out rows lo .. lo+k-1; deflated: rows lo+k .. hi-1 copied
  auto wgen = [&](int j, int i) { return zl[i] * dc_rcp((dl[i] - dl[ori[j]]) - tv[j]) * inrm[j]; };
  if (Wb) {
    for (int j = gw; j < k; j += ngw)
      for (int i = lane; i < k; i += 32)
        if (TB_GUARD(12, Wb - Gi + (long long)j * ld + i, 0, (long long)n * ld)) Wb[(long long)j * ld + i] = wgen(j, i);
    group_sync(g);
    dc_gemm(k, k, vcols, [&](int j, int i) { return Wb[(long long)j * ld + i]; }, V, srow, Out, lo, vc0, ld, Wt, Bt, g);
  } else {
    dc_gemm(k, k, vcols, wgen, V, srow, Out, lo, vc0, ld, Wt, Bt, g);
  }
  for (int q = gw; q < m - k; q += ngw) {
    const double* src = V + (long long)rowof[ndl[k + q]] * ld;
    double* dst = Out + (long long)(lo + k + q) * ld;
    for (int c = vc0 + lane; c < vc0 + vcols; c += 32)
      if (TB_GUARD(13, dst - Out + c, 0, (long long)n * ld)) dst[c] = src[c];
  }
  __syncthreads();
  for (int j = tid; j < m; j += kEigThreads) d[lo + j] = j < k ? dl[ori[j]] + tv[j] : delta[ndl[j]];
  group_sync(g);
}

constexpr int kDcLeaf = 24;  // leaves of the merge tree: at most this many rows, solved by one warp

// Workspace of a leaf of s rows: W (rows and columns rounded up to fours, zero
// past s; row stride leaf_ldw(s)), six vectors, the rotations' cosines and sines, and 8 s ints.
__host__ __device__ constexpr int leaf_pad(int s) { return (s + 3) / 4 * 4; }
__host__ __device__ constexpr int leaf_ldw(int s) { return leaf_pad(s) + 2; }
__host__ __device__ constexpr int leaf_ws(int s) { return leaf_pad(s) * leaf_ldw(s) + 12 * s + 2; }
static_assert(leaf_ws(kDcLeaf) <= dc_ws_elems<double>(kDcMin), "leaf workspace exceeds the divide-and-conquer workspace");

// Leaf [lo0, lo0+s) of the tree (s <= S <= 32) by one warp: the same divide
// and conquer down to single rows, every node of a level at once -- lane r is
// row r of its node (its pole, root and row of W) and column r of the
// eigenvector block, which it holds in registers, so a level costs what its
// largest merge costs on one lane per row.  (Implicit QL, a serial chain of
// some 500 rotations of 130 cycles for 24 rows, took ten times as long.)
// Close-pair rotations enter as factors of W.  Eigenvalues to d[lo0, lo0+s),
// the block to G's diagonal block (row stride ld).
template <int S>
__device__ __noinline__ void dc_leaf(int dofs, int eofs, int lo0, int s, int wofs, double* G, int ld) {
  double *d = syev_sm + dofs, *ws = syev_sm + wofs;
  const double* e = syev_sm + eofs;
  const int lane = threadIdx.x & 31, ldw = leaf_ldw(s), sp = leaf_pad(s);
  double* W = ws;
  double* z = W + sp * ldw;
  double* zs = z + s;      // sorted
  double* delta = zs + s;  // sorted eigenvalues
  double* dl = delta + s;  // per node from its lo on: the k not deflated
  double* zl = dl + s;
  double* tv = zl + s;
  double* rc = tv + s;     // rotations
  double* rsn = rc + s;
  int* rowof = reinterpret_cast<int*>(rsn + s);
  int* srow = rowof + s;
  int* ndl = srow + s;
  int* ori = ndl + s;
  int* rp = ori + s;
  int* rq = rp + s;
  int* fl = rq + s;    // per node at its lo: deflated entries (bits), rotations
  int* nr = fl + s;
  const bool row = lane < s;
  const unsigned below = (1u << lane) - 1u;
  double g[S];
#pragma unroll
  for (int r = 0; r < S; ++r) g[r] = r == lane ? 1.0 : 0.0;
  // every boundary inside the leaf is torn at some level
  double dr = 0.0;
  if (row) dr = d[lo0 + lane] - (lane > 0 ? fabs(e[lo0 + lane - 1]) : 0.0) - (lane < s - 1 ? fabs(e[lo0 + lane]) : 0.0);
  int depth = 0;
  while ((1 << depth) < s) ++depth;
  for (int dep = depth - 1; dep >= 0; --dep) {
    int lo = 0, hi = s;
    for (int l = 0; l < dep; ++l) {
      const int mid = (lo + hi) >> 1;
      if (lane >= mid) lo = mid; else hi = mid;
    }
    const int m = hi - lo, t = (lo + hi) >> 1, j = lane - lo;
    const bool act = row && m >= 2;
    const unsigned node = m >= 32 ? 0xffffffffu : (((1u << (m & 31)) - 1u) << lo);
    const double ev = act ? e[lo0 + t - 1] : 0.0, rho = fabs(ev), sg = ev >= 0.0 ? 1.0 : -1.0;
    // z: the columns beside the tear publish their node's rows
    if (act && (lane == t - 1 || lane == t)) {
      const int ra = lane == t ? t : lo, rz = lane == t ? hi : t;
      const double f = lane == t ? sg : 1.0;
#pragma unroll
      for (int r = 0; r < S; ++r)
        if (r >= ra && r < rz) z[r] = f * g[r];
    }
    __syncwarp();
    int rank = lane;
    const double zr = act ? z[lane] : 0.0;
    if (act) delta[lane] = dr;  // unsorted, for the ranks
    __syncwarp();
    if (act) {
      rank = lo;
      for (int q = lo; q < hi; ++q) {
        const double dq = delta[q];
        rank += (dq < dr || (dq == dr && q < lane)) ? 1 : 0;
      }
    }
    __syncwarp();
    if (act) {
      rowof[lane] = lane;  // valid rows even where non-finite values leave ranks unset
      delta[lane] = zs[lane] = 0.0;
    }
    __syncwarp();
    if (act) {
      rowof[rank] = lane;
      delta[rank] = dr;
      zs[rank] = zr;
    }
    __syncwarp();
    if (act && j == 0) {  // deflation scan of the node, in order (the tests of dc_merge)
      double dmax = 0.0;
      for (int i = lo; i < hi; ++i) dmax = fmax(dmax, fabs(delta[i]));
      const double tol = 8.0 * kEps * fmax(dmax, 2.0 * rho);
      unsigned f = 0;
      int n = 0, prev = -1;
      double za = 0.0, da = 0.0;
      for (int i = lo; i < hi; ++i) {
        double zb = zs[i], db = delta[i];
        if (kSqrt2 * rho * fabs(zb) <= tol) { f |= 1u << i; continue; }
        if (prev >= 0) {
          const double t2 = za * za + zb * zb;
          if (fabs(db - da) * fabs(za * zb) <= tol * t2) {
            const double tau = sqrt(t2), c = zb / tau, sn = -za / tau;
            rp[lo + n] = rowof[prev]; rq[lo + n] = rowof[i]; rc[lo + n] = c; rsn[lo + n] = sn; ++n;
            delta[prev] = da * c * c + db * sn * sn;
            db = da * sn * sn + db * c * c;
            delta[i] = db;
            zb = tau;
            zs[i] = tau;
            zs[prev] = 0.0;
            f |= 1u << prev;
          }
        }
        prev = i; za = zb; da = db;
      }
      fl[lo] = (int)f;
      nr[lo] = n;
    }
    __syncwarp();
    int k = 0, nrot = 0;
    if (act) {  // not deflated first, then the deflated, each in order
      const unsigned defl = (unsigned)fl[lo] & node, keep = node & ~defl;
      nrot = nr[lo];
      k = __popc(keep);
      if ((keep >> lane) & 1u) {
        const int pos = lo + __popc(keep & below);
        dl[pos] = delta[lane]; zl[pos] = zs[lane]; srow[pos] = rowof[lane];
      } else {
        ndl[lo + k + __popc(defl & below)] = lane;
      }
    }
    __syncwarp();
    if (j < k) {
      int o;
      double tj;
      secular_root<1>(j, k, dl + lo, zl + lo, rho, 0, 0u, &o, &tj);
      ori[lane] = o;
      tv[lane] = tj;
    }
    __syncwarp();
    double znew = 0.0;
    if (j < k) {  // Gu and Eisenstat
      const double di = dl[lane];
      double prod = ((dl[lo + ori[lo + k - 1]] - di) + tv[lo + k - 1]) / rho;
#pragma unroll 4
      for (int q = 0; q < k - 1; ++q)  // root q over pole q, or past the pole itself q + 1
        prod *= ((dl[lo + ori[lo + q]] - di) + tv[lo + q]) * dc_rcp(dl[lo + q + (q >= j)] - di);
      znew = copysign(sqrt(fmax(prod, 0.0)), zl[lane]);
    }
    __syncwarp();
    if (j < k) zl[lane] = znew;
    __syncwarp();
    if (lane < sp) {  // row `lane` of W
      double2* Wz = reinterpret_cast<double2*>(W + lane * ldw);
      for (int c = 0; c < sp / 2; ++c) Wz[c] = make_double2(0.0, 0.0);
    }
    if (row) {
      double* Wr = W + lane * ldw;
      if (j < k) {
        const double bj = dl[lo + ori[lane]], tj = tv[lane];
        double nn = 0.0;
#pragma unroll 4
        for (int i = 0; i < k; ++i) {
          const double w = zl[lo + i] * dc_rcp((dl[lo + i] - bj) - tj);
          Wr[srow[lo + i]] = w;
          nn += w * w;
        }
        const double inv = 1.0 / sqrt(nn);
#pragma unroll 4
        for (int i = lo; i < hi; ++i) Wr[i] *= inv;  // (the node's deflated columns hold 0)
        dr = bj + tj;
      } else if (act) {
        Wr[rowof[ndl[lane]]] = 1.0;
        dr = delta[ndl[lane]];
      } else {
        Wr[lane] = 1.0;
      }
      for (int q = nrot - 1; q >= 0; --q) {
        const int pa = rp[lo + q], pb = rq[lo + q];
        const double a = Wr[pa], b = Wr[pb];
        Wr[pa] = rc[lo + q] * a - rsn[lo + q] * b;
        Wr[pb] = rsn[lo + q] * a + rc[lo + q] * b;
      }
    }
    __syncwarp();
    // column `lane` of W G, in parts of 24 or 16 rows: the first of two parts
    // waits in its place in G, so that a part and g fit the registers
    constexpr int kPart = S <= 24 ? S : (S + 1) / 2;
    double gn[kPart];
    double* Gc = G + (long long)lo0 * ld + lo0 + lane;
#pragma unroll
    for (int r0 = 0; r0 < S; r0 += kPart) {
#pragma unroll
      for (int q0 = 0; q0 < kPart; q0 += 4) {
        if (r0 + q0 < sp) {  // four rows at a time; W holds zeros past s
          double b[4][2] = {};
#pragma unroll
          for (int c0 = 0; c0 < S; c0 += 4) {
            if (c0 < sp) {
#pragma unroll
              for (int c = c0; c < c0 + 4; c += 2)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const double2 w = *reinterpret_cast<const double2*>(W + (r0 + q0 + q) * ldw + c);
                  b[q][0] += w.x * g[c];
                  b[q][1] += w.y * g[c + 1];
                }
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) gn[q0 + q] = b[q][0] + b[q][1];
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) gn[q0 + q] = 0.0;
        }
      }
      if (r0 + kPart < S && row)
#pragma unroll
        for (int q = 0; q < kPart; ++q)
          if (r0 + q < s) Gc[(long long)(r0 + q) * ld] = gn[q];
    }
#pragma unroll
    for (int q = 0; q < kPart; ++q) g[S - kPart + q] = gn[q];
#pragma unroll
    for (int q = 0; q < S - kPart; ++q) g[q] = (row && q < s) ? Gc[(long long)q * ld] : 0.0;
    __syncwarp();
  }
  if (row) {
    d[lo0 + lane] = dr;
#pragma unroll
    for (int r = 0; r < S; ++r)
      if (r < s && TB_GUARD(14, (long long)(lo0 + r) * ld + lo0 + lane, 0, (long long)ld * ld))
        G[(long long)(lo0 + r) * ld + lo0 + lane] = g[r];
  }
  __syncwarp();
}

// Node b of depth dep of the halving tree: [lo, hi); *plen = its parent's size.
__device__ inline void dc_node(int n, int dep, int b, int* lo_out, int* hi_out, int* plen) {
  int lo = 0, hi = n, pl = n + 1;
  for (int l = 0; l < dep; ++l) {
    const int mid = (lo + hi) >> 1;
    pl = hi - lo;
    if ((b >> (dep - 1 - l)) & 1) lo = mid; else hi = mid;
  }
  *lo_out = lo; *hi_out = hi; *plen = pl;
}

// Eigenvalues (d, in every CTA) and eigenvector rows (Zc <- G Zc) of the
// tridiagonal (d, e) by the merge tree with leaves of at most S rows (n > S);
// G0, G1 and Z are n x n with row stride ld, ws dc_ws_elems(n), lws lws_cap
// elements for the leaves (even address).  A level with at least as many nodes as CTAs gives each CTA
// whole merges (no barriers between CTAs inside them), the levels above share
// every merge.
template <bool W, int S>
__device__ void dc_solve(double* d, double* e, double* Z, double* G0, double* G1, int n, int ld, double* ws,
                         double* lws, long long lws_cap, const Group g) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const Group alone{0, 1};
  int depth = 0;  // nodes at this depth have at most S rows
  while (((n + (1 << depth) - 1) >> depth) > S) ++depth;
  // tear every internal node (rho = |e[t-1]| off both neighbours)
  for (int dep = 0; dep < depth; ++dep) {
    for (int b = tid; b < (1 << dep); b += kEigThreads) {
      int lo, hi, pl;
      dc_node(n, dep, b, &lo, &hi, &pl);
      if (hi - lo <= S) continue;
      const int t = (lo + hi) >> 1;
      const double rho = fabs(e[t - 1]);
      d[t - 1] -= rho;  // nodes of one depth are disjoint
      d[t] -= rho;
    }
    __syncthreads();
  }
  group_sync(g);  // every CTA's d is torn before a peer writes a leaf's eigenvalues there
  // as many leaf warps as the workspace holds blocks for the largest leaf: of the
  // deepest level or, where a node of exactly S rows one level up is one, S
  const int deepest = (n + (1 << depth) - 1) >> depth;
  const int lsize = leaf_ws(depth > 0 && (n >> (depth - 1)) <= S ? S : deepest);
  const int lw = (int)min((long long)kWarps, lws_cap / lsize);
  for (int dep = depth; dep >= 0; --dep) {
    double* Gi = ((depth - dep - 1) & 1) ? G1 : G0;
    double* Go = ((depth - dep) & 1) ? G1 : G0;
    // leaves of this depth, one warp each
    for (int b = g.rank + g.size * wid; wid < lw && b < (1 << dep); b += g.size * lw) {
      int lo, hi, pl;
      dc_node(n, dep, b, &lo, &hi, &pl);
      if (hi - lo < 1 || hi - lo > S || pl <= S) continue;
      if (!TB_GUARD(15, leaf_ws(hi - lo), 0, lsize + 1) || !TB_GUARD(16, (wid + 1) * lsize, 0, lws_cap + 1)) continue;
      dc_leaf<S>(sm_off(d), sm_off(e), lo, hi - lo, sm_off(lws) + wid * lsize, Go, ld);
      for (int r = 0; g.size > 1 && r < g.size; ++r)
        if (r != g.rank && lane < hi - lo) put_at(d + lo + lane, d[lo + lane], g, r);
    }
    if (dep > 0) {
      const bool whole = (1 << dep) >= g.size;
      if (whole) __syncthreads();  // the leaf blocks in ws have been read
      else group_sync(g);
      for (int b = 0; b < (1 << dep); ++b) {
        if (whole && b % g.size != g.rank) continue;
        int lo, hi, pl;
        dc_node(n, dep, b, &lo, &hi, &pl);
        if (hi - lo <= S) continue;
        dc_merge<W>(sm_off(d), sm_off(e), n, ld, lo, (lo + hi) >> 1, hi, Gi, Gi, lo, hi - lo, Go, sm_off(ws),
                    whole ? alone : g);
        if (whole)
          for (int r = 0; r < g.size; ++r)
            if (r != g.rank)
              for (int i = lo + tid; i < hi; i += kEigThreads) put_at(d + i, d[i], g, r);
      }
      group_sync(g);
    } else {
      // root: Y = diag(G_left, G_right) Zc into the free buffer, then the
      // merge combines rows of Y straight into Zc
      group_sync(g);
      const int t = n >> 1;
      double* Wt = ws;
      double* Bt = Wt + 64 * kDcK;
      int first = 0;  // tiles of the first product, so that the second's continue the round
      for (int h = 0; h < 2; ++h) {
        const int lc = h ? t : 0, sz = h ? n - t : t;
        dc_gemm(sz, sz, n, [&](int j, int i) { return Gi[(long long)(lc + j) * ld + lc + i]; }, Z + (long long)lc * ld,
                nullptr, Go, lc, 0, ld, Wt, Bt, g, first);
        first = ((sz + 63) / 64) * ((n + 63) / 64);
      }
      group_sync(g);
      dc_merge<W>(sm_off(d), sm_off(e), n, ld, 0, t, n, Gi, Go, 0, n, Z, sm_off(ws), g);
    }
  }
}

// ------------------------------------------------------------ small structures
// Structures below kDcMin AOs, one CTA each, wholly in registers and shared
// memory: such a matrix is a few thousand entries, so a Householder step costs
// what its chain of reductions and barriers costs.  Lane group r = tid / 4
// holds row r, lane sub = tid % 4 of it the columns 8i + 2 sub + {0, 1} (the
// operands shared by all rows are then read from shared memory 16 bytes at a
// time without conflicts).  Every warp repeats the step's scalars on its own
// copy of the vectors, so a step has one barrier (the exchange of p = A v).
// The eigenvectors of the tridiagonal come from dc_solve with leaves of at most
// kSmallLeaf rows (24 AOs: 0.14 ms as one leaf of a warp, 0.10 as two and a
// merge by the CTA), all buffers in shared memory.
static_assert(kEigThreads / 4 >= kDcMin, "four lanes per row");

__device__ __forceinline__ void small_reduce(const double* A, int n, int ld, double* V, double* d, double* e, double* tau,
                                          double* ws) {
  // per warp: reflectors k and k-1 and w; shared: p and row k+1, two buffers each
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, r = tid >> 2, sub = tid & 3;
  double* vS = ws + 192 * wid;  // [2][64]
  double* wS = vS + 128;
  double* pS = ws + 192 * kWarps;  // [2][64]
  double* rowS = pS + 128;         // [2][64]
  __shared__ double s_last;        // row n-1's diagonal
  double a[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int c = 8 * (i >> 1) + 2 * sub + (i & 1);
    a[i] = (r < n && c < n) ? A[(long long)r * n + c] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) vS[lane + 32 * i] = 0.0;
  if (r == n - 1)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (8 * (i >> 1) + 2 * sub + (i & 1) == n - 1) s_last = a[i];
  double x0 = lane < n ? A[lane] : 0.0, x1 = lane + 32 < n ? A[lane + 32] : 0.0;  // row k at columns lane, lane + 32
  __syncthreads();
  for (int k = 0;; ++k) {
    if (wid == 0 && lane == (k & 31)) d[k] = k < 32 ? x0 : x1;
    if (k == n - 1) break;
    const int c1 = k + 1;
    const double alpha = __shfl_sync(0xffffffffu, c1 < 32 ? x0 : x1, c1 & 31);
    double* v = vS + 64 * (k & 1);
    const double* vp = vS + 64 * (c1 & 1);
    if (k == n - 2) {  // the last diagonal: the rows in registers carry every pair but the last
      if (tid == 0) e[k] = alpha;
      x0 = x1 = s_last - 2.0 * vp[n - 1] * wS[n - 1];
      continue;
    }
    // reflector k (as in tridiag_tiles)
    const double sigma = warp_sum((lane > c1 ? x0 * x0 : 0.0) + (lane + 32 > c1 ? x1 * x1 : 0.0));
    double scal = 0.0, tk = 0.0, beta = alpha;
    if (sigma != 0.0) {
      const double s2 = alpha * alpha + sigma, ri = rsqrt(s2), rr = s2 * ri;
      beta = alpha <= 0.0 ? rr : -rr;
      tk = 1.0 + fabs(alpha) * ri;
      scal = copysign(dc_rcp(fabs(alpha) + rr), -beta);
    }
    if (tid == 0) { e[k] = beta; tau[k] = tk; }
    const double v0 = lane == c1 ? 1.0 : (lane > c1 ? x0 * scal : 0.0);
    const double v1 = lane + 32 == c1 ? 1.0 : (lane + 32 > c1 ? x1 * scal : 0.0);
    v[lane] = v0;
    v[lane + 32] = v1;
    __syncwarp();
    // the previous pair applied to the rows, and p = A v
    const double vr = vp[r], wr = wS[r];
    double p = 0.0, q = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (8 * i >= n) break;
      const int c = 8 * i + 2 * sub;
      const double2 vv = *reinterpret_cast<const double2*>(v + c);
      const double2 pp = *reinterpret_cast<const double2*>(vp + c);
      const double2 ww = *reinterpret_cast<const double2*>(wS + c);
      a[2 * i] -= vr * ww.x + wr * pp.x;
      a[2 * i + 1] -= vr * ww.y + wr * pp.y;
      p += a[2 * i] * vv.x;
      q += a[2 * i + 1] * vv.y;
    }
    p += q;
    p += __shfl_xor_sync(0xffffffffu, p, 1);
    p += __shfl_xor_sync(0xffffffffu, p, 2);
    double* pb = pS + 64 * (k & 1);
    double* rb = rowS + 64 * (k & 1);
    if (sub == 0) pb[r] = p;
    if (r == c1)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<double2*>(rb + 8 * i + 2 * sub) = make_double2(a[2 * i], a[2 * i + 1]);
    if (k == n - 3 && r == n - 1)
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (8 * (i >> 1) + 2 * sub + (i & 1) == n - 1) s_last = a[i];
    __syncthreads();
    if (wid == 0) {  // reflector k, for the eigenvectors
      if (lane < n) V[k * ld + lane] = v0;
      if (lane + 32 < n) V[k * ld + lane + 32] = v1;
    }
    const double p0 = lane > k ? tk * pb[lane] : 0.0, p1 = lane + 32 > k ? tk * pb[lane + 32] : 0.0;
    const double kk = 0.5 * tk * warp_sum(p0 * v0 + p1 * v1);
    const double w0 = p0 - kk * v0, w1 = p1 - kk * v1;
    const double wn = __shfl_sync(0xffffffffu, c1 < 32 ? w0 : w1, c1 & 31);
    x0 = rb[lane] - (w0 + wn * v0);  // v is 1 at c1
    x1 = rb[lane + 32] - (w1 + wn * v1);
    __syncwarp();  // every lane has read the previous w
    wS[lane] = w0;
    wS[lane + 32] = w1;
    __syncwarp();
  }
}

// Z = Q^T (as form_q) from the reflectors in V: row r in the registers of its
// four lanes, so the rows meet nothing but their own two exchanges per reflector.
__device__ __forceinline__ void small_q(const double* V, int n, int ld, const double* tau, double* Z) {
  const int tid = threadIdx.x, r = tid >> 2, sub = tid & 3;
  double z[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) z[i] = 8 * (i >> 1) + 2 * sub + (i & 1) == r ? 1.0 : 0.0;
  for (int k = n - 3; k >= 0; --k) {
    const double* v = V + k * ld + 2 * sub;
    double p = 0.0, q = 0.0, u[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      u[2 * i] = u[2 * i + 1] = 0.0;
      if (8 * i < n) {
        const double2 vv = *reinterpret_cast<const double2*>(v + 8 * i);
        u[2 * i] = 8 * i + 2 * sub < n ? vv.x : 0.0;  // past the row: whatever follows it
        u[2 * i + 1] = 8 * i + 2 * sub + 1 < n ? vv.y : 0.0;
      }
      p += z[2 * i] * u[2 * i];
      q += z[2 * i + 1] * u[2 * i + 1];
    }
    p += q;
    p += __shfl_xor_sync(0xffffffffu, p, 1);
    p += __shfl_xor_sync(0xffffffffu, p, 2);
    p *= tau[k];
#pragma unroll
    for (int i = 0; i < 16; ++i) z[i] -= p * u[i];
  }
  if (r < n)
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int c = 8 * (i >> 1) + 2 * sub + (i & 1);
      if (c < n) Z[r * ld + c] = z[i];
    }
}

// Structures of kDcMin+ AOs (those below: k_syev_small).  The grid is ncoop groups
// of C CTAs (C = the cluster size), each on one structure (the first ncoop of
// B.order), then CTAs with a structure each, C to a cluster.
template <bool W>
__device__ __forceinline__ void syev_structure(const DevBatch& B, double* __restrict__ Ab, double* __restrict__ Zb,
                                               double* __restrict__ Sb, double* __restrict__ wout,
                                               int* __restrict__ perm, int* __restrict__ status,
                                               const int* __restrict__ active, int ncoop) {
  unsigned csize, crank;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int cid = (int)(blockIdx.x / csize);
  const bool coop = cid < ncoop;
  const Group g{coop ? (int)crank : 0, coop ? (int)csize : 1};
  const int slot = coop ? cid : ncoop + (cid - ncoop) * (int)csize + (int)crank;
  if (slot >= B.nmol) return;
  const int m = B.order ? B.order[slot] : slot;  // largest structures first
  // (the tests below read the same words in every CTA of a group)
  if (active && !active[m]) return;
  if (status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (on_library(B, n) || n < kDcMin) return;
  const long long mo = B.moff[m], vo = B.ooff[m];
  double* A = Ab + mo;
  double* Z = Zb + mo;
  double* Sc = Sb + mo;
  double* d = syev_sm;     // n
  double* e = d + n;       // n
  double* tau = e + n;     // n
  double* v = tau + n;     // n
  double* vn = v + n;      // n
  double* p = vn + n;      // n
  double* w = p + n;       // n
  double* ring = w + n;    // 2 kRing n
  __shared__ int q_fail;
  const int tid = threadIdx.x;

  if (B.trid_max > 0 && n >= B.trid_min && n >= kTridMin && n <= B.trid_max) {
    // tridiagonalised in shared memory by k_trid_smem: reflectors in A's rows,
    // d | e | tau in the first 3n entries of the scratch slice
    for (int i = tid; i < n; i += kEigThreads) {
      d[i] = Sc[i];
      e[i] = i < n - 1 ? Sc[n + i] : 0.0;
      tau[i] = i < n - 2 ? Sc[2 * n + i] : 0.0;
    }
    group_sync(g);
  } else {
    tridiag_tiles<W>(A, n, d, e, tau, v, vn, p, w, ring, Sc, g);
  }
  form_q<W>(A, Z, n, tau, v, g);
  group_sync(g);  // Z is complete, A and the scratch are free

  unsigned dyn_bytes;
  asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
  const long long ws_cap = (long long)(dyn_bytes / sizeof(double)) - 2LL * n;
  if (tid == 0) { q_fail = 0; e[n - 1] = 0.0; }
  __syncthreads();
  dc_solve<W, kDcLeaf>(d, e, Z, A, Sc, n, n, tau, tau, ws_cap, g);  // (tau: at an even element)
  for (int i = tid; i < n; i += kEigThreads)
    if (!(fabs(d[i]) < 1e30)) q_fail = 1;  // non-finite input
  __syncthreads();
  if (q_fail) {
    if (tid == 0 && g.rank == 0) status[m] = kStEigenFailed;  // k_fermi retires the structure
    return;
  }
  // ascending order by rank (ties by index)
  for (int i = g.rank * kEigThreads + tid; i < n; i += g.size * kEigThreads) {
    const double di = d[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = d[j];
      rank += (dj < di || (dj == di && j < i)) ? 1 : 0;
    }
    if (!TB_GUARD(9, rank, 0, n)) continue;
    perm[vo + rank] = i;
    wout[vo + rank] = di;
  }
}

}  // namespace

// Two CTAs per SM (128 registers) for batches that fill the GPU with a CTA per
// structure of at most kWalk2 + 1 AOs, one CTA per SM with whole units in
// registers for clusters and larger orders.  Both run
// the same arithmetic in the same order.  (Three CTAs per SM at 80 registers
// spilled in the walks and held 16 loads in flight per lane instead of 32:
// 444 structures of 300 AOs took 4.1 ms of an SM each against 3.9.  Where two fall
// short is between one wave of two and one of three to an SM: 300 structures of 66
// AOs take 0.99 ms, 444 of them 1.11, the former kernel at three to an SM 0.91 and
// 0.93; of 96 AOs 1.48 and 1.69 against 1.58 and 1.61; up to 296 and beyond 444
// structures two are faster, up to 1.6 times.)
__global__ void __launch_bounds__(kEigThreads, 2) k_syev(DevBatch B, double* __restrict__ Ab, double* __restrict__ Zb,
                                                         double* __restrict__ Sb, double* __restrict__ wout,
                                                         int* __restrict__ perm, int* __restrict__ status,
                                                         const int* __restrict__ active, int ncoop) {
  syev_structure<false>(B, Ab, Zb, Sb, wout, perm, status, active, ncoop);
}
__global__ void __launch_bounds__(kEigThreads, 1) k_syev_wide(DevBatch B, double* __restrict__ Ab,
                                                              double* __restrict__ Zb, double* __restrict__ Sb,
                                                              double* __restrict__ wout, int* __restrict__ perm,
                                                              int* __restrict__ status,
                                                              const int* __restrict__ active, int ncoop) {
  syev_structure<true>(B, Ab, Zb, Sb, wout, perm, status, active, ncoop);
}

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
// jacobi_warp: structure list[li] by this warp, on its 2 kJacobiMaxN rows of `a`.
__device__ __noinline__ void jacobi_warp(const DevBatch& B, const double* __restrict__ Ab, double* __restrict__ Zb,
                                         double* __restrict__ wout, int* __restrict__ perm,
                                         int* __restrict__ status, const int* __restrict__ active,
                                         const int* __restrict__ list, int nlist, int li) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (li >= nlist) return;
  const int m = list[li];
  if ((active && !active[m]) || status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (n > kJacobiMaxN) return;
  constexpr int P = kJacobiPitch;
  double* a = syev_sm + (size_t)warp * 2 * kJacobiMaxN * P;  // n x n, pitch P
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

__global__ void __launch_bounds__(kJacobiWarps * 32) k_syev_jacobi(DevBatch B, const double* __restrict__ Ab,
                                                                  double* __restrict__ Zb,
                                                                  double* __restrict__ wout,
                                                                  int* __restrict__ perm, int* __restrict__ status,
                                                                  const int* __restrict__ active,
                                                                  const int* __restrict__ list, int nlist) {
  jacobi_warp(B, Ab, Zb, wout, perm, status, active, list, nlist, blockIdx.x * kJacobiWarps + (threadIdx.x >> 5));
}

// Structures of B.order from position `first` on, one CTA each.
__global__ void __launch_bounds__(kEigThreads, 2) k_syev_small(DevBatch B, const double* __restrict__ Ab,
                                                               double* __restrict__ Zb, double* __restrict__ wout,
                                                               int* __restrict__ perm, int* __restrict__ status,
                                                               const int* __restrict__ active, int first,
                                                               const int* __restrict__ jlist, int njac) {
  const int slot = first + (int)blockIdx.x;
  if (slot >= B.nmol) {  // the CTAs past the structures: one-warp Jacobi
    const int warp = threadIdx.x >> 5;
    if (warp < kJacobiWarps)
      jacobi_warp(B, Ab, Zb, wout, perm, status, active, jlist, njac, (slot - B.nmol) * kJacobiWarps + warp);
    return;
  }
  const int m = B.order ? B.order[slot] : slot;
  if ((active && !active[m]) || status[m] != kStOk) return;
  const int n = B.ooff[m + 1] - B.ooff[m];
  if (on_library(B, n) || n >= kDcMin || n <= B.jacobi_max) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, ld = small_ld(n);
  double* ws = syev_sm;                               // small_ws_elems(n)
  double* G0 = ws + small_ws_elems(n);                // n x ld: reflectors, then merge blocks
  double* G1 = G0 + n * ld;
  double* Z = G1 + n * ld;
  double* d = Z + n * ld;
  double* e = d + n;
  double* tau = e + n;
  __shared__ int q_fail;
  const long long mo = B.moff[m], vo = B.ooff[m];
  small_reduce(Ab + mo, n, ld, G0, d, e, tau, ws);
  if (tid == 0) { e[n - 1] = 0.0; q_fail = 0; }
  __syncthreads();
  small_q(G0, n, ld, tau, Z);
  __syncthreads();
  if (n > kSmallLeaf) {
    // the leaves' workspace: ws or, since the deepest level's blocks go to G0, G1
    const bool big = n * ld > small_ws_elems(n);
    dc_solve<false, kSmallLeaf>(d, e, Z, G0, G1, n, ld, ws, big ? G1 : ws, big ? n * ld : small_ws_elems(n),
                                Group{0, 1});
  } else {
    if (wid == 0) dc_leaf<kSmallLeaf>(sm_off(d), sm_off(e), 0, n, sm_off(ws), G0, ld);
    __syncthreads();
  }
  for (int i = tid; i < n; i += kEigThreads)
    if (n > 1 && !isfinite(d[i])) q_fail = 1;  // non-finite input (one row is its own eigenvalue, whatever it holds)
  __syncthreads();
  if (q_fail) {
    if (tid == 0) status[m] = kStEigenFailed;  // k_fermi retires the structure
    return;
  }
  double* Zg = Zb + mo;
  for (int r = wid; r < n; r += kWarps)
    for (int c = lane; c < n; c += 32) {
      double x = 0.0;
      if (n > kSmallLeaf) x = Z[r * ld + c];
      else
        for (int i = 0; i < n; ++i) x += G0[r * ld + i] * Z[i * ld + c];
      Zg[(long long)r * n + c] = x;
    }
  for (int i = tid; i < n; i += kEigThreads) {
    const double di = d[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double dj = d[j];
      rank += (dj < di || (dj == di && j < i)) ? 1 : 0;
    }
    if (!TB_GUARD(9, rank, 0, n)) continue;
    perm[vo + rank] = i;
    wout[vo + rank] = di;
  }
}

TB_OOB_EXPORT(oob_syev)

cudaError_t launch_syev(const SyevPlan& P, const DevBatch& B, double* A, double* Z, double* Sb, double* w, int* perm,
                        int* status, const int* active, cudaStream_t st, int64_t* launches, const int* jlist,
                        int njac) {
  cudaError_t e = cudaSuccess;
  const size_t smem = syev_smem_bytes(P.nmax > 1 ? P.nmax : 1);
  if (P.n64 > 0 && P.nmax >= kDcMin) {
    DevBatch Bs = B;
    Bs.nmol = P.n64;  // the kernel's bound on its position in the order
    const int C = P.c.cluster;
    const int groups = P.c.ncoop + (P.n64 - P.c.ncoop + C - 1) / C;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(groups * C));
    cfg.blockDim = dim3(kEigThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, P.c.wide ? k_syev_wide : k_syev, Bs, A, Z, Sb, w, perm, status, active, P.c.ncoop);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  if (P.nsmall > 0) {
    // in the order, the small structures follow n64 (with no order, anywhere)
    const int first = B.order ? P.n64 : 0;
    // The Jacobi structures ride along in CTAs of four: a launch of their own
    // lasts as long as one of them (400 molecules of 6..60 AOs: 9 launches of
    // 0.125 ms after 9 of 0.236 ms, now 9 of 0.259).  Alone they take the smaller
    // CTAs, three to an SM (4000 of 6 AOs 0.77 ms against 3.16 on one CTA each).
    const int nj = (njac + kJacobiWarps - 1) / kJacobiWarps;
    size_t smem_small = small_smem_bytes(P.small_max);
    if (njac > 0 && jacobi_smem_bytes() > smem_small) smem_small = jacobi_smem_bytes();
    k_syev_small<<<B.nmol - first + nj, kEigThreads, smem_small, st>>>(B, A, Z, w, perm, status, active, first, jlist,
                                                                       njac);
    e = cudaGetLastError();
    if (launches) ++*launches;
  } else if (njac > 0) {
    k_syev_jacobi<<<(njac + kJacobiWarps - 1) / kJacobiWarps, kJacobiWarps * 32, jacobi_smem_bytes(), st>>>(
        B, A, Z, w, perm, status, active, jlist, njac);
    e = cudaGetLastError();
    if (launches) ++*launches;
  }
  return e;
}

}  // namespace tb
