// How rq_gemm_w4_kernel divides tensor memory, and which barrier an accumulator set completes on.  Plain constants, so that the
// host compiler can check the barriers' rule as well.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define RQ_HD __host__ __device__
#else
#define RQ_HD
#endif

constexpr uint32_t RQ_W4_TMEM_COLS = 512;
constexpr int RQ_W4_FOLD_TEAMS = 2;             // fold warps take every second accumulator set
constexpr int RQ_W4_M_STAGES = 4;               // stages of the multiplier ring, one per slice of 256 inputs

// runs of a step, A buffers of a step each, accumulator sets of a step each (SR * nt columns); nt: tokens covered
RQ_HD constexpr int rq_w4_sr(int nt) { return nt <= 32 ? 4 : 2; }
RQ_HD constexpr int rq_w4_na(int) { return 4; }
RQ_HD constexpr uint32_t rq_w4_d_col(int nt) { return (uint32_t) (rq_w4_na(nt) * rq_w4_sr(nt) * 16); }
RQ_HD constexpr int rq_w4_nd(int nt) { return (int) (RQ_W4_TMEM_COLS - rq_w4_d_col(nt)) / (rq_w4_sr(nt) * nt); }
// groups of an accumulator set, and sets per slice, with gsteps runs of 64 inputs per activation group
RQ_HD constexpr int rq_w4_set_groups(int nt, int gsteps) { return rq_w4_sr(nt) >= gsteps ? rq_w4_sr(nt) / gsteps : 1; }
RQ_HD constexpr int rq_w4_slice_sets(int nt, int gsteps) { return 4 / gsteps / rq_w4_set_groups(nt, gsteps); }

// Barriers that tell the fold warps of a finished set: set s completes phase s / bars of barrier s % bars.  A wait names a phase by
// its parity alone, so whoever waits must have seen the phase before end: were there as many barriers as buffers where these are
// odd in number (64 tokens: 3), a team would meet a barrier at every second phase, and its wait could be satisfied by the
// phase before the other team's, whose completion nothing orders before.  An even number gives every barrier to one team.
RQ_HD constexpr int rq_w4_full_bars(int nt) { return rq_w4_nd(nt) % RQ_W4_FOLD_TEAMS == 0 ? rq_w4_nd(nt) : RQ_W4_FOLD_TEAMS * rq_w4_nd(nt); }
