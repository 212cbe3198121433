"""CPU: the host-side plans (tb_plan.cu), compiled into a program that launches nothing.

The plans of one structure allocate nothing, since tb_sygvd_noalloc makes them
at a C entry.  The automatic choice sends a structure to cuSOLVER, whose calls run one after
another, only where that shortens the modelled eigensolve; small structures
beside a large one stay with the batched solvers.  Model coefficients as
measured on a B200."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tblite-cuda_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <iostream>
#include <string>
#include "tb_plan.cu"
extern int allocations;
int main() {
  {  // the plans of one structure, as tb_sygvd_noalloc makes them
    tb::SyevPlan p;
    tb::FactorPlan f;
    const int before = allocations;
    for (int n = 1; n <= 256; ++n) {
      p.build(&n, 1, 0, 0);
      f.build(&n, 1, 0);
    }
    std::printf("%d\n", allocations - before);
  }
  tb::SolverModel M;
  tb::SyevPlan p, q;
  const int m1 = 256, m2 = 512;
  p.build(&m1, 1, 0, 0);
  q.build(&m2, 1, 0, 0);
  M.lib256 = 2.3321e-3;
  M.lib_slope = (12.1454e-3 - 2.3321e-3) / 768;
  M.scale = 500.0 * (1.37712e-3 / p.c.span + 3.61923e-3 / q.c.span);
  int n;
  while (std::cin >> n) {
    std::vector<int> s(n);
    for (int& x : s) std::cin >> x;
    std::sort(s.begin(), s.end(), std::greater<int>());
    tb::SyevPlan P;
    P.build(s.data(), n, tb::kSyevMaxN, 0);
    std::printf("%d %d %d %d %.6f\n", tb::choose_lib_above(s, M), P.c.cluster, P.c.ncoop, (int)P.c.wide, P.c.span);
  }
}
"""

COUNT = r"""
#include <cstdlib>
#include <new>
int allocations = 0;
void* operator new(std::size_t n) {
  ++allocations;
  return std::malloc(n);
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cu").write_text(PROGRAM)
    (d / "count.cpp").write_text(COUNT)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", CSRC, str(d / "plan.cu"), str(d / "count.cpp"), "-o",
                    str(d / "plan")], check=True, capture_output=True, timeout=300)

    def run(sizes):
        out = subprocess.run([str(d / "plan")], input=f"{len(sizes)} " + " ".join(map(str, sizes)), text=True,
                             capture_output=True, timeout=60, check=True).stdout.split()
        assert out.pop(0) == "0"  # allocations of a plan for one structure
        return dict(lib_above=int(out[0]), cluster=int(out[1]), ncoop=int(out[2]), wide=int(out[3]),
                    span=float(out[4]))

    return run


@pytest.mark.parametrize("large, small", [
    ([1000], [6 + 6 * (i % 10) for i in range(100)]),
    ([1190], [20 + i for i in range(50)]),
    ([1190], [62, 68, 74]),
    ([1100], [6 + i % 55 for i in range(200)]),
    ([1196], [50] * 50),
    ([600], [66] * 700),
    ([1400], [50] * 20),
    ([1400, 1300, 700], [383, 300, 6]),
])
def test_small_structures_stay_in_house_beside_large_ones(plan, large, small):
    lib = plan(large + small)["lib_above"]
    assert lib >= max(small)  # what has more AOs goes to the library
    assert lib >= 0


def test_a_single_large_structure_beside_small_ones_goes_to_the_library(plan):
    for large, small in ((1000, [6 + 6 * (i % 10) for i in range(100)]), (1190, list(range(20, 70))),
                         (1190, [62, 68, 74])):
        assert max(small) <= plan([large] + small)["lib_above"] < large


@pytest.mark.parametrize("sizes, expect", [([300], 1216), ([384] * 8, 1216), ([6] * 50, 1216), ([1217], -1),
                                           ([1300, 2000], -1), ([2000, 60], 1216)])
def test_ends_of_the_range(plan, sizes, expect):
    assert plan(sizes)["lib_above"] == expect


@pytest.mark.parametrize("large, small", [([1196], 66), ([1000] * 10, 66), ([384], 100)])
def test_a_few_large_structures_keep_their_clusters_in_any_number_of_small_ones(plan, large, small):
    # ten more small structures add little to a plan whose span is its large ones'
    spans = [plan(large + [small] * k)["span"] for k in (560, 580, 590, 600, 620)]
    assert max(spans) <= 1.1 * min(spans)
    assert plan(large + [small] * 600)["cluster"] > 1


def test_waves_of_like_structures_take_one_cta_each(plan):
    assert plan([6 * (11 + i * 53 // 899) for i in range(900)])["cluster"] == 1
    assert plan([100] * 5000 + [384])["cluster"] == 1


def test_batches_of_the_narrow_kernel(plan):
    # what tests/test_gpu_syev_groups.py compares with structures alone, which take the wide one
    from test_gpu_syev_groups import NARROW_LARGE, narrow_sizes
    one, two = plan(narrow_sizes(900)), plan(narrow_sizes(700))
    assert (one["wide"], one["cluster"]) == (0, 1)
    assert (two["wide"], two["cluster"]) == (0, 2) and two["ncoop"] > len(NARROW_LARGE)
    assert plan([449, 448, 225, 224] * 74)["wide"] == 0
    for n in NARROW_LARGE + [449, 448, 225, 224]:
        assert plan([n])["wide"] == 1
