// Which kernel a log-softmax and a sampling top-k take (sample.cu), as plain host code.
#pragma once
#include <algorithm>

namespace msb {

// Estimates in us, fitted to a B200 (1 to 256 rows of 64 to 300000; the chosen form is at most a few per cent slower than the
// other).  A wave of clusters of 8 blocks, about a tenth of the SMs at once, takes 4.3 whatever the row is as long as its eighth
// lies in registers; a block per row takes 0.28 per 1024 values, and more once blocks share an SM.
//   us, clusters / block per row:  1 x 8000 4.7 / 4.2   1 x 12000 4.7 / 5.0   16 x 24000 9.0 / 7.6   16 x 32000 9.0 / 9.8
//                                  64 x 65536 23 / 21   64 x 129280 26 / 44   256 x 8000 77 / 7
inline bool log_softmax_by_cluster(int rows, int V, int sms) {
  const int at_once = std::max(1, sms / 10);
  const double clusters = 0.4 + 4.3 * ((rows + at_once - 1) / at_once);
  const double block = (2.1 + 0.28 * V / 1024) * (1.0 + std::max(0, rows - sms / 2) / 128.0);
  return clusters < block;
}

// The sampling top-k: a cluster of 8 blocks per row that keeps the logits in registers, or groups of blocks and a last block's finish.
// Times in us for k = 64, groups / clusters (12 clusters run at once, more rows take another wave):
//   1 x 17000 17.3 / 8.7   1 x 129280 16.0 / 9.8   1 x 160000 18.2 / 12.7   12 x 129280 20.3 / 12.1   16 x 129280 23.9 / 17.6
//   32 x 17000 24.5 / 18.5   32 x 129280 32.9 / 25.5   64 x 17000 27.9 / 28.7   64 x 32000 25.4 / 29.5   64 x 129280 49.7 / 41.0
// (one logit of 129280 7.2 / 7.2).  Short rows end within the groups' first block or two; they were not tried with clusters.
constexpr int kTopkClusterMinV = 16385, kTopkClusterMaxV = 163840;      // 40 registers per thread
inline bool topk_by_cluster(int rows, int V) {
  return V >= kTopkClusterMinV && V <= kTopkClusterMaxV && (rows <= 32 || (rows <= 64 && V >= 65000));
}

}  // namespace msb
