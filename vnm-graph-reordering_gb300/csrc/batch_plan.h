// Which jobs of a batch run on wider clusters: host arithmetic only.
#pragma once
#include <algorithm>
#include <functional>
#include <vector>

namespace vnm {

// How many of a batch's jobs (entries in descending order) to run on clusters
// of 4 blocks when the others run on 2.  A job's time goes with its entries
// (0.135 us each on 2 blocks) and is about 0.74 of that on 4, measured on R-MAT
// at 2:8 and taken for every M; the others start in order wherever two SMs come free, and the number with the
// earliest end is taken, within half of the SMs and where it gains at least 10
// %.  (256 R-MAT matrices, 256-8192 rows: the largest job alone took all of the
// 24.8 ms that the batch takes with 2 blocks for all; 19.2 ms so, at 2:4 11.9
// and 8.8.)
// The GPU waits for the answer, so it takes a small part of the time of sorting
// the jobs: the starts are simulated for the jobs above a 16th of an even share
// of the work (what is left fills the SMs evenly), for the numbers that the
// work itself and the largest jobs leave a chance, and not at all where the
// largest is below a ninth, as the plain order then ends within 10 % of what
// any order could (all jobs simulated for each number: 2.9 ms of 76 at 50000
// matrices of 64 rows).
inline int wide_jobs(const std::vector<long long>& sizes, int num_sms) {
  const int n = (int)sizes.size(), pairs = num_sms / 2;
  if (n < 2 || pairs < 1) return 0;
  double rest = 0;
  for (const long long s : sizes) rest += (double)s;
  double work = rest;  // of the SM pairs, with the jobs so far wide
  const double share = work / pairs;
  int heads = 0;
  for (; heads < n && 16.0 * (double)sizes[heads] > share; ++heads) rest -= (double)sizes[heads];
  int best = 0;
  double best_end = 0;
  std::vector<double> ends;  // when each pair of SMs comes free: a heap, earliest on top
  for (int k = 0; k < n && 4 * k <= pairs && 9.0 * (double)sizes[k > 0 ? k - 1 : 0] > share; ++k) {
    const double limit = best_end * (best == 0 ? 0.9 : 1.0);
    if (k > 0) {
      work += (2 * 0.74 - 1) * (double)sizes[k - 1];
      if (std::max(work / pairs, (double)sizes[k]) >= limit) continue;  // no end is earlier
    }
    ends.assign(pairs, 0.0);
    double end = 0, busy = rest;
    for (int q = 0; q < k; ++q) {
      const double t = 0.74 * (double)sizes[q];
      ends[2 * q] = ends[2 * q + 1] = t;
      end = std::max(end, t);
      busy += 2 * t;
    }
    std::make_heap(ends.begin(), ends.end(), std::greater<double>());
    for (int q = k; q < heads; ++q) {
      std::pop_heap(ends.begin(), ends.end(), std::greater<double>());
      ends.back() += (double)sizes[q];
      end = std::max(end, ends.back());
      busy += (double)sizes[q];
      std::push_heap(ends.begin(), ends.end(), std::greater<double>());
    }
    end = std::max(end, busy / pairs);
    if (k == 0 || end < limit) {
      best = k;
      best_end = end;
    }
  }
  return best;
}

}  // namespace vnm
