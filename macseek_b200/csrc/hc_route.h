// Which kernel a hyper-connection step takes (hc_step.cu), as plain host code.
#pragma once
#include <algorithm>

namespace msb {

constexpr int kHcRanks = 16;                       // blocks of a cluster
constexpr int kHcThreadsMax = 960;                 // 6 row groups x (5120 / 16 / 2) column pairs

struct HcRoute { int tokens, clusters; };          // per round of a cluster; tokens 0: the ticket kernel

// fit1, fit4: clusters of the kernels for 1 and 4 tokens per round that the device runs at once.  16 blocks are more than every
// device must be able to place together: 0 where it cannot.
inline HcRoute hc_route(int D, int n, bool aligned8, int fit1, int fit4) {
  // whole warps of column pairs in every block of a cluster, 8-byte aligned vectors
  if (D % (64 * kHcRanks) || D / (2 * kHcRanks) * 6 > kHcThreadsMax || !aligned8) return {0, 0};
  if (n <= fit1) return {1, n};
  if (fit4 <= 0) return {0, 0};
  return {4, std::min(fit4, (n + 3) / 4)};         // 4 tokens per round once every cluster that fits has one
}

}  // namespace msb
