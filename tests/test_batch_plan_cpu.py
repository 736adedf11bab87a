"""The choice of a batch's wide jobs (csrc/batch_plan.h, compiled alone for the
CPU): what it costs beside sorting the jobs, and that it is as good as trying
each number with every job simulated."""
import os
import subprocess

from conftest import REPO

CODE = r"""
#include "batch_plan.h"
#include <chrono>
#include <cmath>
#include <cstdio>
#include <random>
using Jobs = std::vector<long long>;
static double end_of(const Jobs& s, int pairs, int k) {  // the k first on two pairs of SMs each, the others in order
  std::vector<double> free(pairs, 0.0);
  double end = 0;
  for (int q = 0; q < (int)s.size(); ++q) {
    if (q < k) {
      free[2 * q] = free[2 * q + 1] = 0.74 * s[q];
      end = std::max(end, 0.74 * s[q]);
      continue;
    }
    auto at = std::min_element(free.begin(), free.end());
    *at += (double)s[q];
    end = std::max(end, *at);
  }
  return end;
}
int main() {
  std::mt19937_64 rng(1);
  double worst = 0;
  for (int t = 0; t < 400; ++t) {
    Jobs s(2 + rng() % 500);
    std::uniform_real_distribution<> u(5.0, 5.0 + (rng() % 900) / 100.0);
    for (auto& x : s) x = (long long)std::exp(u(rng));
    if (t % 3 == 0)
      for (size_t k = 0; k < rng() % 4 && k < s.size(); ++k) s[k] *= 5;
    std::sort(s.rbegin(), s.rend());
    const int pairs = 76, got = vnm::wide_jobs(s, 152);
    const double plain = end_of(s, pairs, 0);
    double best = plain;
    for (int k = 1; k < (int)s.size() && 4 * k <= pairs; ++k) best = std::min(best, end_of(s, pairs, k));
    if (best >= 0.9 * plain) best = plain;  // not worth it
    worst = std::max(worst, end_of(s, pairs, got) / best);
  }
  Jobs s(50000);
  std::uniform_real_distribution<> u(4.0, 10.0);
  for (auto& x : s) x = (long long)std::exp(u(rng));
  const auto t0 = std::chrono::steady_clock::now();
  std::sort(s.rbegin(), s.rend());
  const auto t1 = std::chrono::steady_clock::now();
  const int got = vnm::wide_jobs(s, 152);
  const auto t2 = std::chrono::steady_clock::now();
  std::printf("%f %d %f\n", worst, got, std::chrono::duration<double>(t2 - t1) / std::chrono::duration<double>(t1 - t0));
}
"""


def test_choice_of_wide_jobs(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(CODE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(REPO, "vnm-graph-reordering_gb300", "csrc"),
                    "-o", str(exe), str(src)], check=True)
    worst, got, share = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    # a gain below 10 % is left
    assert float(worst) <= 1 / 0.9
    assert int(got) == 0 and float(share) < 1.0, share
