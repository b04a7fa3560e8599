// Which kernel a projection of two tokens takes (matvec.cu), as plain host code.
#pragma once

namespace msb {

// The tensor-core kernel decodes a weight for up to 4 tokens, so from 3 tokens on it is always the faster one (1.1 to 2.9 times over
// 512 to 32768 rows of 1024 to 12288).  With two the other kernel, two columns per pass, ends sooner
//  - when there are so few rows that most SMs have no tile of 16 and the others a long row each (512 x 12288 Q8_0: 7.2 us against
//    10.5; IQ1_S rows are short enough throughout),
//  - on many rows of some widths.  The lines are those of the times (us, two columns / tensor cores, 16384 rows, 20000 for 1792 and
//    7168): IQ1_S 8192 25.1 / 27.2, 12288 58 / 41; IQ2_XXS 4096 14.5 / 16.9, 6144 25 / 25; Q6_K 1792 11.3 / 16.0, 2048 8.8 / 11.2,
//    4096 16.9 / 16.4, 7168 39 / 54, 8192 42 / 46; Q8_0 1536 7.4 / 9.0, 4096 24 / 18; Q5_K 1024 8.6 / 9.0, 12288 69 / 75.  IQ4_NL,
//    whose decoding costs the two-column kernel most: nowhere.
inline bool two_tokens_by_mma(int t, int rows, int cols, int sms) {
  enum { kQ8_0 = 8, kQ5_K = 13, kQ6_K = 14, kIQ2_XXS = 16, kIQ1_S = 19 };
  const int tiles = (rows + 15) / 16;
  if (2 * tiles < sms && t != kIQ1_S && cols > tiles * (t == kQ6_K || t == kIQ2_XXS ? 256 : 160)) return false;
  if (rows < 4096) return true;
  switch (t) {
    case kIQ1_S:
    case kIQ2_XXS: return rows < 8192 || (cols != 4096 && cols != 8192);
    case kQ6_K: return cols <= 1536 || (cols >= 2304 && cols <= 6144) || (cols > 8192 && cols < 12288);
    case kQ8_0: return cols >= 2048;
    case kQ5_K: return cols >= 1536 && cols < 12288;
    default: return true;
  }
}

}  // namespace msb
