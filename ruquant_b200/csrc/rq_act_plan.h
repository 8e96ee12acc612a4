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
