// chip_plan.h -- host: how cases are split into clusters of the on-chip engine.
#pragma once
#include <algorithm>
#include <functional>
#include <vector>

#include "chip_engine.h"

namespace acs {

struct PlanCase {
  int nx, ny, pitch;
  bool scalars;
  bool ok;   // its constants and porosity suit the on-chip arithmetic
  int want;  // CTAs that the caller asks for (0: none)
};
struct ChipPlan {
  std::vector<int> k;  // CTAs of every case's on-chip cluster, 0 where the cluster engine takes the case
  double us = 0.0;     // modelled time of a pseudo-iteration of all cases on chip (0: not all fit)
};

// Shared memory of one CTA when a case runs on chip in clusters of K (0: it does not fit).
inline size_t chip_bytes(const PlanCase& c, int K, bool phys) {
  if (!c.ok) return 0;
  const size_t s = sizeof(double) * (size_t)chip_layout(c.nx, c.ny, c.pitch, K, c.scalars, phys).total;
  return s <= (size_t)CHIP_MAX_SMEM ? s : 0;
}

// Whether a case runs on chip depends on the case and the device only, so a split that the caller asks for
// changes no result: it is the size asked for where the case fits in that, else the next larger one that it
// fits in, else its largest.  (Left to the cluster engine, a 102 x 102 FAST case asked into 4 CTAs had other
// roundings and about four times the time per pseudo-iteration.)  The other cases get the split with the
// smallest modelled time of one pseudo-iteration of all cases: a case in K CTAs takes
// CHIP_T0 + CHIP_T1 * (nodes of its largest strip), and the device runs as many clusters of K at once as its
// GPCs hold (on a B200 15 of 9 CTAs, 11 of 10, 7 of 11 to 16).  resident(K): that number; sizes that the
// device cannot hold at all (0: fewer SMs, or a share of the device) are left out, and a case that only fits
// in such a size goes to the cluster engine.
inline ChipPlan plan_chip(const std::vector<PlanCase>& cases, bool fast, const std::function<int(int)>& resident) {
  const int n = (int)cases.size();
  ChipPlan p;
  p.k.assign(n, 0);
  int slots[17], asked[17] = {};
  auto res = [&](int K) {
    if (!asked[K]) slots[K] = resident(K);
    asked[K] = 1;
    return slots[K];
  };
  std::vector<std::vector<int>> sizes(n);  // cluster sizes that take the case, ascending
  std::vector<int> todo;
  bool free_split = false;  // some case's split is the plan's own
  for (int c = 0; c < n; ++c) {
    const int kmax = std::max(1, std::min(16, (cases[c].ny + 1) / 4));
    for (int K = 1; K <= kmax; ++K)
      if (chip_bytes(cases[c], K, false) && res(K) > 0) sizes[c].push_back(K);
    if (!sizes[c].empty()) todo.push_back(c);
    free_split |= !sizes[c].empty() && !cases[c].want;
  }
  if (todo.empty()) return p;
  // the smallest size of case c that is at least what is asked for (by the caller, else K), else its largest
  auto at_least = [&](int c, int K) {
    auto it = std::lower_bound(sizes[c].begin(), sizes[c].end(), cases[c].want ? cases[c].want : K);
    return it == sizes[c].end() ? sizes[c].back() : *it;
  };
  const double t0 = fast ? CHIP_T0_FAST : CHIP_T0_EXACT, t1 = fast ? CHIP_T1_FAST : CHIP_T1_EXACT;
  double best = 0.0;
  int best_k = 0;
  for (int K = 1; K <= (free_split ? 16 : 1); ++K) {
    int kk = 0;
    std::vector<double> t;
    for (int c : todo) {
      const int k = at_least(c, K);
      kk = std::max(kk, k);
      t.push_back((t0 + t1 * cases[c].nx * ((cases[c].ny + 1 + k - 1) / k)) * (cases[c].scalars ? 1.0 : 0.6));
    }
    // longest first onto the slot that is free first
    std::sort(t.begin(), t.end(), std::greater<double>());
    std::vector<double> busy(std::min((size_t)res(kk), t.size()), 0.0);
    for (double x : t) {
      std::pop_heap(busy.begin(), busy.end(), std::greater<double>());
      busy.back() += x;
      std::push_heap(busy.begin(), busy.end(), std::greater<double>());
    }
    const double end = *std::max_element(busy.begin(), busy.end());
    if (!best_k || end < best) {
      best = end;
      best_k = K;
    }
  }
  for (int c : todo) p.k[c] = at_least(c, best_k);
  if ((int)todo.size() == n) p.us = best;
  return p;
}

}  // namespace acs
