// How batches are spread over CTAs and thread block clusters: host code only,
// from the structures' sizes and modelled times.
#include <algorithm>
#include <cmath>
#include <functional>

#include "tb_kernels.h"

namespace tb {

namespace {
// Time of one structure of n AOs on a group of C CTAs, in ms: what each CTA
// repeats or waits for (the steps' barriers, gathers and scalars, a merge's
// sort and scan), plus what they divide.  Measured on one structure alone with
// one CTA per SM, at 138, 384, 722, 1196 AOs: 1.1, 7.8, 41, 156 ms on one CTA;
// 0.85, 4.8, 23, 84 on two; 0.72, 3.3, 13.5, 47 on four; 0.75, 2.6, 9.0, 29 on
// eight; 0.74, 2.5, 7.2, 20 on sixteen.
double syev_ms(double n, int C) {
  const double serial = n * (4.6e-3 + 2.05e-6 * n), shared = n * n * (6.6e-6 + 8.55e-8 * n);
  return serial + shared / C;
}
}  // namespace

// The combination with the shortest modelled span.  A span is list scheduling of
// the order (largest first) over as many clusters as the GPU holds at once
// (kCap: cudaOccupancyMaxActiveClusters on a B200, one and two CTAs per SM) for
// every cluster size and a geometric set of splits into cluster and one-CTA
// structures.  Two CTAs on an SM slow each other (kSlowTwo), and the narrower
// kernel alone is slower (kSlowNarrow): 148 structures of 150, 300 and 384 AOs take
// 1.31, 5.31 and 9.19 ms wide, 1.46, 5.70 and 9.94 narrow (1.07 to 1.11 times), 296
// of them 1.95, 8.02 and 14.1 (1.49 to 1.54 times, all in step; 1.42 is for uneven
// batches: 400 clusters of 48..384 AOs on one CTA each take 10.8 ms, modelled 11.2).
// By plan: 400 clusters 8.1 ms (on two), 128 4.5 (8.9 on one, 5.8 on two), 48 chains
// of 122..1196 AOs 33.5 (on eight; 165 on one).  Where one CTA
// per structure is within 3% of the CTAs' total work, or more than 592 structures
// could gain half a millisecond at most, no clusters are tried: they repeat work,
// and the search takes about as long on the host (0.8 ms for the factorisation of
// 1024 structures).  (The number alone is no such rule: with clusters for at most
// 592 structures, 8 chains of 602 AOs with 640 of 66..120 took 175 ms a call, now
// 62; a chain of 1196 with 600 of 66 AOs, in-house, 981 and 165; 620 clusters of
// 66..384 AOs 136 either way.)
ClusterChoice choose_clusters(const int* sizes, int first, int last, double (*ms)(double, int), bool two_per_sm,
                              bool one_per_sm) {
  ClusterChoice best;
  std::vector<double> busy;  // finish times of the clusters in flight (a heap)
  auto schedule = [&](int cap, int C, int k, double slow, double limit) {
    if (last - first == 1) return slow * ms(sizes[first], C);
    busy.clear();
    double end = 0.0;
    for (int i = first; i < last && end < limit;) {
      const bool coop = C > 1 && i < k;
      double t = slow * ms(sizes[i], coop ? C : 1);
      i += coop ? 1 : C;
      if ((int)busy.size() == cap) {
        std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
        t += busy.back();
        busy.pop_back();
      }
      busy.push_back(t);
      std::push_heap(busy.begin(), busy.end(), std::greater<double>());
      end = std::max(end, t);
    }
    return end;
  };
  constexpr int kCap[2][5] = {{148, 74, 33, 15, 7}, {296, 148, 71, 33, 14}};
  constexpr double kSlowTwo = 1.42, kSlowNarrow = 1.1;
  const int cnt = last - first;
  best.span = 1e300;
  // what no plan can undercut: the one-CTA times over the CTAs (clusters only add work)
  double least = 0.0;
  for (int i = first; i < last; ++i) least += ms(sizes[i], 1);
  least *= std::min(kSlowTwo / kCap[1][0], 1.0 / kCap[0][0]);
  for (int per = two_per_sm ? 2 : 1; per >= (one_per_sm ? 1 : 2); --per)
    for (int c = 0; c < 5; ++c) {
      const int C = 1 << c;
      if (C > 1 && (0.97 * best.span <= least || (cnt > 4 * 148 && best.span - least < 0.5))) break;
      for (int k = cnt; k >= 1; k = k > 1 ? (3 * k) / 4 : 0) {
        const int items = C > 1 ? k + (cnt - k + C - 1) / C : cnt;
        const double slow = per == 1 ? 1.0 : items > kCap[0][c] ? kSlowTwo : kSlowNarrow;
        const double t = schedule(kCap[per - 1][c], C, first + k, slow, best.span);
        if (t < 0.97 * best.span) best = {C, C > 1 ? first + k : 0, per == 1, t};
        if (C == 1) break;
      }
    }
  return best;
}

void SyevPlan::build(const int* sizes, int count, int lib_above, int jacobi_max) {
  *this = SyevPlan();
  int first = 0;  // structures of the library path lead the order and exit at once
  for (int i = 0; i < count; ++i) {
    const int n = sizes[i];
    if (lib_above != 0 && n > lib_above) { first = n64 = i + 1; continue; }
    nmax = n > nmax ? n : nmax;
    if (n >= kDcMin) n64 = i + 1;
    else if (n > jacobi_max) { ++nsmall; small_max = std::max(small_max, n); }
  }
  if (n64 > first)
    c = choose_clusters(sizes, first, n64, syev_ms, nmax <= kSyevNarrowMaxN, true);
}

// The k largest structures go to cuSOLVER, the rest to the batched in-house
// solvers, with k minimising the modelled time of one SCF iteration's eigensolve:
//   sum_{i<k} t_lib(N_i) + span(N_k, N_{k+1}, ...)
// (library calls run one after another, then k_syev runs the rest).  k stops at
// the first structure below kLibMinN: alone, 256 AOs take 1.4 ms in-house and 2.3
// in cuSOLVER, 384 AOs 2.4 and 3.9, and in a batch the calls add up while the
// in-house structures run beside one another.  So every k leaves the structures
// below 64 AOs in-house; k_syev_small's time for them is a constant of the sum and left out.
int choose_lib_above(std::vector<int> sizes, const SolverModel& M) {
  std::sort(sizes.begin(), sizes.end(), std::greater<int>());
  const int nmol = (int)sizes.size();
  int k0 = 0;
  while (k0 < nmol && sizes[k0] > kSyevMaxN) ++k0;
  if (k0 == nmol) return -1;
  int last = k0;  // the first that is not offered
  while (last < nmol && sizes[last] >= kLibMinN) ++last;
  const int step = std::max(1, (last - k0) / 64);  // at most 65 plans (2 ms each for 2000 structures)
  double lib_sum = 0.0, best = 1e300;  // (the k0 structures above the in-house limit count the same for every k)
  int best_k = k0;
  for (int k = k0; lib_sum < best;) {
    SyevPlan rest;
    rest.build(sizes.data() + k, nmol - k, 0, 0);
    const double in_t = 1e-3 * rest.c.span * M.scale;
    if (lib_sum + in_t < best) { best = lib_sum + in_t; best_k = k; }
    if (k == last) break;
    for (const int end = std::min(last, k + step); k < end; ++k) lib_sum += M.lib256 + M.lib_slope * (sizes[k] - 256);
  }
  if (best_k == nmol) return -1;
  return best_k == k0 ? kSyevMaxN : sizes[best_k];
}

namespace {
// Time of one structure of n AOs on C CTAs, in ms: a diagonal block and the
// two barriers of its column, and the products the CTAs divide.
double factor_ms(double n, int C) { return 0.03 * std::ceil(n / kFactorBlock) + 8.0e-9 * n * n * n / C; }
}  // namespace

void FactorPlan::build(const int* sizes, int nstructures, int lib_above) {
  *this = FactorPlan();
  count = nstructures;
  int first = 0;  // structures of the library path lead the order and exit at once
  while (first < count && lib_above != 0 && sizes[first] > lib_above) ++first;
  if (first < count) c = choose_clusters(sizes, first, count, factor_ms, true, false);
}

}  // namespace tb
