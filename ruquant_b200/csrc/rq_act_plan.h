// Host rules of the activation quantizer's launches.  Plain functions, so that a host program can check them.
#pragma once

#include <stdint.h>

// The widest cluster that RQ_TUNE_ACT_CMAX allows: the power of two in 1 .. 8 that is not above what it asks for.
inline int rq_act_cluster_cap(int asked) {
    int c = 8;
    while (c > 1 && c > asked) c >>= 1;
    return c;
}

// CTAs of a token's cluster, at most cap (1: no cluster): two units of work for each, and all M clusters running at once.
// at_once[2], [4] and [8]: clusters of so many CTAs that fit on the device.
inline int rq_act_cluster(int cap, int units, int64_t M, const int * at_once) {
    int c = cap;
    while (c > 1 && (units < 2 * c || M > at_once[c])) c >>= 1;
    return c;
}

// Whether M tokens of K inputs, a CTA each, take CTAs of 256 threads rather than 128 (Paley orders that have both forms).  While
// the tokens are few the phases are latency, which more warps shorten; and as SMs come free of the kernel ahead, the CTAs that
// start first fill them up: six of 128 threads to an SM where three of 256 would leave tokens for the next.  Nodes of 5120 rows, us
// with 128 and with 256 threads, several in a row:
//   250 tokens  3072 21.9, 20.1   5120 32.2, 28.9   6144 39.6, 34.4   11264 62.1, 58.6
//   444         3072 24.3, 22.4   5120 35.6, 31.6   6144 43.0, 37.1   11264 69.7, 65.2   15360 99.0, 98.0
//   512          768 12.7, 14.1   3072 24.5, 24.8    5120 35.6, 34.4    6144 43.2, 40.6   11264 71.5, 73.8
//   592         3072 25.9, 26.4   5120 37.8, 37.7   6144 46.0, 44.4   11264 77.1, 80.0   15360 124, 130
//   1024        3072 40.4, 42.9   5120 60.1, 63.2   6144 73.7, 75.6   11264 128, 131     15360 191, 205
inline bool rq_act_256(int p, int64_t K, int64_t M, int sms) { return M <= (p <= 20 && K >= 4096 ? 4 : 3) * (int64_t) sms; }
