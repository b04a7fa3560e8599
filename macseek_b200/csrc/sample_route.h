// Which kernel a log-softmax takes (sample.cu), as plain host code.
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

}  // namespace msb
