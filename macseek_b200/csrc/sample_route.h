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
// Estimates in us, fitted to 710 calls of 1 to 100 rows of 16385 to 163840 on a B200 (the other form is 7 % faster in one of them, 4 % in
// another): 15 clusters run at once and a wave takes the longer the more registers a thread holds, and where the blocks' parts do
// not start on a cache line; the groups pay for every block beyond one per SM and, from two logits on, for a last block's search.
//   us, groups / clusters, k = 1:  1 x 65536 6.7 / 4.9    1 x 129280 6.7 / 7.1    16 x 32000 6.9 / 9.8    32 x 32000 9.3 / 14.2   48 x 131072 30.3 / 26.6
//                         k = 16:  1 x 140000 9.6 / 10.0  18 x 22000 10.4 / 10.7  32 x 48000 14.6 / 16.0  48 x 131072 33.8 / 28.2
//                         k = 64:  1 x 16385 15.7 / 7.9   1 x 129280 15.7 / 9.8   32 x 22000 23.9 / 18.1  64 x 129280 51.1 / 40.0
// Longer rows do not fit in registers; shorter ones and more rows are the groups'.
constexpr int kTopkClusterMinV = 16385, kTopkClusterMaxV = 163840;      // 40 registers per thread
inline bool topk_by_cluster(int rows, int V, int k = 64) {
  if (V < kTopkClusterMinV || V > kTopkClusterMaxV || rows > (V >= 65000 ? 64 : 32)) return false;
  const int waves = (rows + 14) / 15, blocks = rows * ((V + 4095) / 4096);
  const double odd = V % 256 ? 1.0 : 0.0;                    // parts of V / 8 that start within a line
  const double wave = V <= 65536 ? 1.7 + (4.0 + 0.1 * odd) * waves : V <= 131072 ? 1.4 + (6.5 + 0.7 * odd) * waves      // 16, 32,
                                                                                 : 1.6 + (7.2 + 0.8 * odd) * waves;     // 40 registers
  const double clusters = wave + k / 64.0 * (2.0 + 0.9 * waves);
  const double groups = (blocks <= 148 ? 7.5 : 5.9 + 0.0165 * blocks) + (k == 1 ? 0.0 : 1.2 + 0.1 * k + 0.16 * std::max(0, k - 32));
  return clusters < groups;
}
// How many granule maxima may reach the cluster form's threshold before its search ends.  Of 129 granules of 128 normal values (16385
// logits) 128 reach a bound that 630 values reach, too many for the list (256): the exact selection followed, 24.5 us for
// 64 of 16385.  At 80 of them it is 125 values and 7.9 us.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr unsigned topk_enough(unsigned k) { return k > 32u ? k + k / 4u : 2u * k > 32u ? 2u * k : 32u; }

}  // namespace msb
