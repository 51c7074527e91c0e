// Cluster sizes of the resident kernel (resident.cu) and how the resident
// classes of one batch share the SMs between them.
#pragma once

#include <algorithm>
#include <cstddef>
#include <limits>
#include <vector>

namespace qpb {

// One cluster size of a side: CTAs per start, and the time of an iteration
// while every start is resident (RAAR, measured on one B200).
struct ClusterSize {
  int ctas;
  double us;
};

// Sizes of a side, smallest first; empty for a side without a resident kernel.
inline std::vector<ClusterSize> cluster_sizes(int side) {
  switch (side) {
    case 64: return {{1, 3.4}, {2, 3.0}, {4, 2.3}, {8, 2.05}};
    case 128: return {{2, 10.9}, {4, 6.3}, {8, 4.4}, {16, 3.8}};
    case 256: return {{8, 11.1}, {16, 7.5}};
    default: return {};
  }
}

// A class's starts, and the clusters of each of its sizes (in the order of
// cluster_sizes) that the device runs at once.
struct ClusterClaim {
  int side;
  int starts;
  std::vector<int> room;
};

// CTAs per start for classes whose launches run beside each other. Each class
// for itself would take the largest clusters it fits (resident_cluster), and
// classes that do so together run one after another: 4 starts each of 64, 128
// and 256 square took 12.5 us an iteration, with 8, 16 and 16 CTAs a start
// 160 of 148 SMs. Of all combinations this takes the one with the shortest
// iteration: the slowest class's where all clusters fit beside each other,
// else that plus the work of all classes spread over the SMs (the bound for
// launches that start as others end); among equals the one whose classes take
// least time together. Measured times per class and size decide that, so a
// class gives up SMs where it loses least.
inline std::vector<int> share_clusters(const std::vector<ClusterClaim>& claims, int sms) {
  std::vector<std::vector<ClusterSize>> sizes;
  for (const ClusterClaim& c : claims) sizes.push_back(cluster_sizes(c.side));
  std::vector<std::size_t> pick(claims.size(), 0);
  std::vector<int> best(claims.size(), 0);
  double best_us = std::numeric_limits<double>::infinity(), best_together = 0.0;
  for (;;) {
    double longest = 0.0, work = 0.0, together = 0.0;
    long long ctas = 0;
    bool fits = true;
    for (std::size_t k = 0; k < claims.size(); ++k) {
      const ClusterSize s = sizes[k][pick[k]];
      const long long taken = static_cast<long long>(claims[k].starts) * s.ctas;
      ctas += taken;
      longest = std::max(longest, s.us);
      work += static_cast<double>(taken) * s.us;
      together += s.us;
      // clusters as large as this one or larger take the same places
      long long clusters = 0;
      for (std::size_t j = 0; j < claims.size(); ++j) {
        if (sizes[j][pick[j]].ctas >= s.ctas) clusters += claims[j].starts;
      }
      fits = fits && clusters <= claims[k].room[pick[k]];
    }
    fits = fits && ctas <= sms;
    const double us = fits ? longest : longest + work / sms;
    if (us < best_us || (us == best_us && together < best_together)) {
      best_us = us;
      best_together = together;
      for (std::size_t k = 0; k < claims.size(); ++k) best[k] = sizes[k][pick[k]].ctas;
    }
    std::size_t k = 0;  // the next combination
    while (k < claims.size() && ++pick[k] == sizes[k].size()) pick[k++] = 0;
    if (k == claims.size()) return best;
  }
}

}  // namespace qpb
