// Which kernel multiplies 9 to 16 tokens by the decode stream.  A plain function, so that a host program can check it.
#pragma once

#include <stdint.h>

// True: the GEMV with two tiles of 8 tokens.  False: the tensor-core kernel.  K: inputs; tiles: 16-row tiles of the launch; ctas:
// CTAs of that GEMV that run at once (two an SM without weight multipliers, one with them); M: tokens.
// The GEMV gives a row tile to one CTA, so its time is rounds of tiles times K, plus 2.5 us; the tensor-core kernel splits K
// over a cluster and needs about 4 us for its start and its end.  Measured over 256 to 17408 inputs and 16 to 17408 rows, with
// and without multipliers, 9 to 16 tokens, weights from HBM and from L2: the line is 0.4 % behind the faster one on average, 9 % at
// worst without multipliers, 19 with.  us, GEMV and tensor cores, 9 tokens from HBM unless said:
//   one round     1024 x 4096 3.2, 6.0; 4096 x 2048 4.7, 6.0; 6144 x 4096 6.6, 8.3 and with 16 tokens 7.5, 8.4; 11264 x 4096 with
//                 16 tokens 11.6, 10.9; few rows, which a cluster splits best: 6144 x 1024 with 16 tokens 6.6, 5.5
//   two rounds    1024 x 8192 4.4, 6.1; 4096 x 8192 8.4, 9.0; 5120 x 8192 from L2 9.0, 9.4; 256 x 8192 from L2 4.0, 3.2 (a single
//                 slice of K: no cluster, nothing to hand over)
//   three rounds  1024 x 12288 6.2, 4.9
// Groups of 128 and 256 inputs need a half and a quarter of the folds: 6144 x 4096 in groups of 256 5.5, 7.5; 5120 x 8192 7.8, 8.7;
// 11264 x 2048 with 16 tokens in groups of 128 6.6, 7.7.  Weight multipliers cost the tensor-core kernel more.
inline bool rq_gemv_takes_16(int64_t K, int64_t tiles, int64_t ctas, int64_t M, int group, bool has_k) {
    const int64_t any_m = group == 64 ? 4096 : 6144;      // inputs up to which the number of tokens makes no difference
    if (tiles > 2 * ctas) return false;
    if (tiles > ctas) return K > 256 && K <= any_m;
    if (K <= any_m) return true;
    if (tiles < 64) return false;
    const int64_t many = group == 64 ? 96 : group == 128 ? 192 : 144, few = group == 64 ? (has_k ? 80 : 64) : group == 128 ? 112 : 80;
    return K * M <= 1024 * (tiles >= 128 ? many : few);
}
