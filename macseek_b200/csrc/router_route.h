// Which kernel selects the experts of n tokens (router.cu), as plain host code.
#pragma once

namespace msb {

// A block per token, whose threads all score, or a warp per token.  64 registers a thread: 8 blocks of 128 run on an SM, 1184 on a B200's
// 148; of the warp form's blocks (4 tokens) an SM has one more every 592 tokens, and the fourth, from 1777 on, costs what a second
// wave of the other form does.
//   us of the selection and a small kernel between, warp / block:
//     E 384   1 token 6.5 / 4.4   999 8.5 / 6.4   1184 8.6 / 6.5   1280 9.8 / 9.9   1776 9.9 / 10.1   2048 11.2 / 10.2   2300 11.3 / 11.6
//     E 64    1       4.3 / 3.6   999 5.5 / 4.9   1184 5.6 / 4.9   1280 6.5 / 7.2   1776 6.6 / 7.4    2048 7.6 / 7.5     2300 7.6 / 8.8
//     E 16    1184    4.6 / 4.2   1280 5.2 / 5.8  2048 6.0 / 6.1   8192, E 384: 27.2 / 28.7
// A few blocks more than run at once begin as the first end (E 384, 1190 tokens: 9.5 / 8.5).
inline bool router_block_per_token(int n, int E) { return E >= 48 ? n <= 1192 || (n > 1776 && n <= 2048) : n <= 1184; }

}  // namespace msb
