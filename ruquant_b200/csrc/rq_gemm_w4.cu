// Batch-width contraction on the tensor cores, straight from the int4 decode stream: tcgen05.mma with the weights as the
// A operand in tensor memory and the accumulators beside it.
//
// Why: up to 64 tokens the node is bound by reading the weights once (K*N/2 bytes), but the decode GEMV's register MMAs
// and per-token folds cannot keep up with HBM above a handful of tokens, and above 16 it reads the stream again for every
// 16 tokens.  Here 128 weight rows are the MMA's M (tensor-memory lanes) and all tokens of the call its N, so the stream
// is read once whatever the number of tokens; a group's sums cost 2 MMAs.
//
// Pipeline of one CTA (640 threads, one CTA per SM):
//   warp 0      weight producer: one TMA box of 128 rows x 256 inputs (8 pieces of 2 KB) per ring stage.  The
//               weights do not depend on the preceding kernel: the ring fills before griddepcontrol.wait.
//   warp 3      activation producer: TMA boxes of NT tokens x 128 inputs (128B swizzle) into a ring of their own.
//   warp 2      multipliers: transposes m_g of every token into [group][token] words of a small ring.
//   warps 4-11  unpack: a thread owns a weight row; 8 words give the row's 64 inputs of a run, three instructions turn a word
//               into eight int8 16*c, tcgen05.st puts them into tensor memory as the A operand.
//               (Through shared memory the unpacked operand would be written and read again: 256 cycles of shared-memory
//               bandwidth per 128 x 128 weights, which arrive from HBM every 356.)
//   warp 1      MMA issue, kind::i8, D = 128 * S_g (int32), one accumulator per activation group.
//   warps 12-19 fold: warps 12-15 the even accumulator sets, 16-19 the odd ones; a thread owns a row and all tokens: total += (m_g * D) >> 11 (rq_common.cuh), or with weight
//               multipliers (k * m_g * (D >> 7)) >> 4; then y = ((float(total) * 16) * u) * s_w.
// The tensor pipe needs 28 cycles for a run of 64 inputs and 16 tokens (64 for 64 tokens): what a hand-over between the roles
// costs (an arrival, a wait that wakes up, a fence: 50 to 150 cycles) decides, so the roles hand over steps of SR runs.
// Handing over single runs the kernel took 530 cycles a run whatever the number of tokens.
// Registers move from the control and unpack warps to the fold warps, which hold totals, sums and the next multipliers.
// Few row tiles: a cluster of CTAs splits K; integer sums are exact in any order.  Every CTA pushes its partial totals into
// the shared memory of the CTA that owns the token, one cluster barrier, and the owner adds and stores.
// Measured, the four contractions of a 5120-wide decoder layer launched back to back (170 MB of codes, 26 us at the copy rate):
// 59 us at 16 tokens (the register-MMA kernel: 87), 73 at 32 (174 in two passes), 108 at 64 (344 in four); one launch of
// 5120 x 34816 runs at 3.7 TB/s at 16 tokens and is bound by the hand-overs between the roles and about 4 us of start and end,
// at 64 tokens by the integer folds (1.9 TB/s).
// Every wait is bounded as in the other kernels: on expiry the waiter raises a CTA-wide abort flag, every role leaves its
// loop, copies in flight are drained, tensor memory is released and a status word is set.
#include <cuda.h>

#include <stdlib.h>

#include <mutex>
#include <type_traits>

#include "rq_common.cuh"
#include "rq_gemm_w4_plan.h"

namespace {

constexpr int ROWS = 128;                       // weight rows per CTA tile
constexpr int SLICE = 256;                      // inputs per ring stage
constexpr int RUNS = SLICE / 64;                // 64-input runs per stage
constexpr uint32_t W_BYTES = ROWS * SLICE / 2;  // 16 KB of codes per stage
constexpr uint32_t SUB_BYTES = W_BYTES / 8;     // the part of one 16-row tile of the decode stream (a row of the TMA box)
constexpr int THREADS = 640;
constexpr int UNPACK_WARPS = 8;
constexpr int MS = RQ_W4_M_STAGES;
constexpr uint32_t TMEM_COLS = RQ_W4_TMEM_COLS;
constexpr int MAX_SPLIT = 8;
constexpr long long WAIT_CYCLES = 2000000000ll;

constexpr int MAX_BUFS = 8, MAX_STAGES = 9;
// Two rings: a weight slot is free as soon as it is unpacked, an activation slot when the MMAs have read it, steps later (in one
// ring the weights would hold their slots as long: at 16 tokens half of the ring was not in flight)
__host__ __device__ constexpr int w_stages_of(int nt) { return nt <= 32 ? 9 : nt <= 48 ? 7 : 5; }
__host__ __device__ constexpr int b_stages_of(int nt) { return nt <= 16 ? 6 : nt <= 32 ? 5 : 4; }
__host__ __device__ constexpr uint32_t b_bytes_of(int nt) { return (uint32_t) nt * SLICE; }
__host__ __device__ constexpr uint32_t ring_bytes_of(int nt) { return w_stages_of(nt) * W_BYTES + b_stages_of(nt) * b_bytes_of(nt); }
__host__ __device__ constexpr uint32_t m_bytes_of(int nt) { return (uint32_t) (MS * RUNS * nt * 4); }
// totals the two fold warps of a quarter exchange: nt tokens of 128 rows
__host__ __device__ constexpr uint32_t swap_bytes_of(int nt) { return (uint32_t) nt * ROWS * 4; }
// partial totals pushed by the cluster's CTAs: split * ceil(nt / split) tokens of 128 rows
__host__ __device__ constexpr uint32_t part_bytes_of(int nt) { return (uint32_t) (nt + MAX_SPLIT - 1) * ROWS * 4; }
__host__ __device__ constexpr uint32_t smem_bytes_of(int nt) { return ring_bytes_of(nt) + m_bytes_of(nt) + part_bytes_of(nt) + swap_bytes_of(nt) + 1024; }

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return (uint32_t) __cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// bounded wait: false when the barrier did not flip within WAIT_CYCLES or another role already gave up
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int * abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t i = 1;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63u) == 0u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > WAIT_CYCLES) { *abort_flag = 1; return false; }
        }
    }
}
// the same for a whole warp: all lanes leave with the same answer
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int * abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap * map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// K-major tile of NT rows x 128 bytes, 128B swizzle (rows of 128 bytes, atoms of 8 rows 1024 bytes apart): start address
// >> 4 [0,14), stride byte offset >> 4 [32,46), descriptor version 1 [46,48), SWIZZLE_128B = 2 [61,64)
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    return (uint64_t) ((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t) (1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::i8: D = s32 (2 at [4,6)), A and B signed int8 (1 at [7,10) and [10,13)), N >> 3 at [17,23), M >> 4 at [24,29)
__host__ __device__ constexpr uint32_t idesc_of(int nt) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (nt >> 3) << 17) | ((uint32_t) (ROWS >> 4) << 24);
}
// A from tensor memory (128 lanes x 8 columns of 4 bytes), B from shared memory; called by a converged warp
template <int NT>
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, int acc) {
    asm volatile("{\n\t.reg .pred pe, p;\n\telect.sync _|pe, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t@pe tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc_of(NT)), "r"(acc) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred pe;\n\telect.sync _|pe, 0xffffffff;\n\t@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" :: "r"(bar) : "memory");
}

// 16 or 32 columns of this thread's lane
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t taddr, const uint32_t (&v)[N]) {
    if constexpr (N == 16)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                     :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                     "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                     :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[N - 16]), "r"(v[N - 15]),
                        "r"(v[N - 14]), "r"(v[N - 13]), "r"(v[N - 12]), "r"(v[N - 11]), "r"(v[N - 10]), "r"(v[N - 9]), "r"(v[N - 8]),
                        "r"(v[N - 7]), "r"(v[N - 6]), "r"(v[N - 5]), "r"(v[N - 4]), "r"(v[N - 3]), "r"(v[N - 2]), "r"(v[N - 1]) : "memory");
}
// N columns (a multiple of 8) of this thread's lane, requested; complete after tmem_ld_wait
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, int (&v)[N]) {
#pragma unroll
    for (int c = 0; c < N; c += 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[c]), "=r"(v[c + 1]), "=r"(v[c + 2]), "=r"(v[c + 3]), "=r"(v[c + 4]), "=r"(v[c + 5]), "=r"(v[c + 6]), "=r"(v[c + 7])
                     : "r"(taddr + c) : "memory");
}
// completes this thread's tensor-memory loads; the values are threaded through so that no use moves above the wait
template <int N>
__device__ __forceinline__ void tmem_ld_wait(int (&v)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < N; c += 8)
        asm volatile("" : "+r"(v[c]), "+r"(v[c + 1]), "+r"(v[c + 2]), "+r"(v[c + 3]), "+r"(v[c + 4]), "+r"(v[c + 5]), "+r"(v[c + 6]), "+r"(v[c + 7]));
}

struct W4Job {
    const float * sw;
    const int8_t * wk;      // [N][K/64] or null
    float * y;
    float * y_more[RQ_MAX_RANKS - 1];
    int64_t ldy;
    int N;
    int n_more;
};
struct W4Params {
    W4Job job[RQ_MAX_WEIGHTS];
    int tile_start[RQ_MAX_WEIGHTS + 1];     // in tiles of 128 rows
    int n_jobs;
    const int32_t * msh;    // [M][K/G]
    const float * u;
    int32_t * status;
    int K, M, G;
    int split;              // CTAs of a cluster that share a row tile (slices of K)
};

__device__ __forceinline__ int job_of_tile(const W4Params & prm, int tile) {
    int w = 0;
#pragma unroll
    for (int i = 1; i < RQ_MAX_WEIGHTS; ++i) if (i < prm.n_jobs && tile >= prm.tile_start[i]) w = i;
    return w;
}

struct __align__(8) W4Shared {
    uint64_t full_w[MAX_STAGES], empty_w[MAX_STAGES], full_b[MAX_STAGES], empty_b[MAX_STAGES];
    uint64_t a_full[MAX_BUFS], a_empty[MAX_BUFS];
    uint64_t d_full[MAX_BUFS], d_empty[MAX_BUFS];
    uint64_t m_full[MS], m_empty[MS];
    float u[64];
    int fold_ok[4][2];
    uint32_t tmem_base;
    int abort_flag;
};

// NT: tokens covered, a multiple of 16 (the MMA's N).  HAS_K: weight multipliers.
template <int NT, bool HAS_K>
__global__ void __launch_bounds__(THREADS, 1)
rq_gemm_w4_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w0,
                  const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_w2, const W4Params prm) {
    constexpr int W_STAGES = w_stages_of(NT), B_STAGES = b_stages_of(NT);
    constexpr int CG = NT <= 16 ? 4 : NT <= 32 ? 2 : 1;      // groups a fold warp takes at a time (up to 64 sums)
    constexpr int SR = rq_w4_sr(NT), NA = rq_w4_na(NT), ND = rq_w4_nd(NT), NF = rq_w4_full_bars(NT);
    static_assert(NA <= MAX_BUFS && ND <= MAX_BUFS && NF <= MAX_BUFS, "barriers");
    static_assert(NF % RQ_W4_FOLD_TEAMS == 0 && MS % RQ_W4_FOLD_TEAMS == 0, "a fold warp meets every phase of a barrier that it waits on");
    extern __shared__ uint8_t smem_raw[];
    __shared__ W4Shared sh;
    const uint32_t raw = smem_u32(smem_raw), ring = (raw + 1023u) & ~1023u;
    uint8_t * ring_p = smem_raw + (ring - raw);
    int * m_ring = reinterpret_cast<int *>(ring_p + ring_bytes_of(NT));          // [MS][RUNS][NT]
    int * part = reinterpret_cast<int *>(ring_p + ring_bytes_of(NT) + m_bytes_of(NT));      // [split][tokens of this CTA][ROWS]
    int * swap = part + part_bytes_of(NT) / 4;      // [NT][ROWS]
    const int warp = __shfl_sync(0xffffffffu, (int) (threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int K = prm.K, M = prm.M, ng64 = K >> 6;
    const int split = prm.split, rank = split > 1 ? (int) (blockIdx.x % split) : 0;
    const int tiles = prm.tile_start[prm.n_jobs], first = (int) blockIdx.x / split, stride = (int) gridDim.x / split;
    const int nsl = K / SLICE, sl0 = nsl * rank / split, sl1 = nsl * (rank + 1) / split, n_sl = sl1 - sl0;
    const int gsteps = prm.G >> 6, gps = RUNS / gsteps;       // runs per activation group, groups per slice
    const int dgroups = rq_w4_set_groups(NT, gsteps), dsets = gps / dgroups;      // groups of an accumulator set, sets per slice
    volatile int * abort_flag = &sh.abort_flag;

    if (threadIdx.x == 0) rq_trace(prm.status, 0x5c);
    if (threadIdx.x == 0) {
        for (int s = 0; s < W_STAGES; ++s) { mbar_init(smem_u32(&sh.full_w[s]), 1); mbar_init(smem_u32(&sh.empty_w[s]), UNPACK_WARPS); }
        for (int s = 0; s < B_STAGES; ++s) { mbar_init(smem_u32(&sh.full_b[s]), 1); mbar_init(smem_u32(&sh.empty_b[s]), 1); }
        for (int b = 0; b < NA; ++b) { mbar_init(smem_u32(&sh.a_full[b]), UNPACK_WARPS); mbar_init(smem_u32(&sh.a_empty[b]), 1); }
        for (int b = 0; b < ND; ++b) mbar_init(smem_u32(&sh.d_empty[b]), 4);
        for (int b = 0; b < NF; ++b) mbar_init(smem_u32(&sh.d_full[b]), 1);
        for (int b = 0; b < MS; ++b) { mbar_init(smem_u32(&sh.m_full[b]), 1); mbar_init(smem_u32(&sh.m_empty[b]), 4 * dsets); }
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&sh.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (split > 1) cluster_arrive();          // this CTA has started: its shared memory may be written by the others
    const uint32_t tmem_base = sh.tmem_base;

    // the block is launched with 96 registers a thread: 128 x 40 + 256 x 72 + 256 x 144 of its 640 x 96
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;" ::: "memory");
    if (warp == 0) {
        // ---- weights: a box of 8 16-row tiles x 256 inputs per stage (tiles beyond the weight's last one arrive as zeros)
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = first; tile < tiles && ok; tile += stride) {
                const int wi = job_of_tile(prm, tile);
                const CUtensorMap * map = wi == 0 ? &tmap_w0 : wi == 1 ? &tmap_w1 : &tmap_w2;
                const int sub0 = (tile - prm.tile_start[wi]) * 8;
                for (int sl = 0; sl < n_sl; ++sl, ++it) {
                    const uint32_t s = it % W_STAGES;
                    if (!mbar_wait(smem_u32(&sh.empty_w[s]), ((it / W_STAGES) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    const uint32_t bar = smem_u32(&sh.full_w[s]);
                    mbar_expect_tx(bar, W_BYTES);
                    tma_load_2d(ring + s * W_BYTES, map, bar, (sl0 + sl) * SLICE, sub0);
                }
            }
            if (*abort_flag) {      // let every copy that was issued land before the CTA's shared memory goes away
                for (uint32_t k = it > (uint32_t) W_STAGES ? it - W_STAGES : 0; k < it; ++k) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(smem_u32(&sh.full_w[k % W_STAGES]), (k / W_STAGES) & 1u) && clock64() - t0 < WAIT_CYCLES) { }
                }
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        // ---- activations (written by the preceding kernel): two boxes of NT tokens x 128 inputs per stage
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = first; tile < tiles && ok; tile += stride) {
                for (int sl = 0; sl < n_sl; ++sl, ++it) {
                    const uint32_t s = it % B_STAGES;
                    if (!mbar_wait(smem_u32(&sh.empty_b[s]), ((it / B_STAGES) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                    const uint32_t bar = smem_u32(&sh.full_b[s]), dst = ring + W_STAGES * W_BYTES + s * b_bytes_of(NT);
                    mbar_expect_tx(bar, b_bytes_of(NT));
                    tma_load_2d(dst, &tmap_x, bar, (sl0 + sl) * SLICE, 0);
                    tma_load_2d(dst + b_bytes_of(NT) / 2, &tmap_x, bar, (sl0 + sl) * SLICE + 128, 0);
                }
            }
            if (*abort_flag) {
                for (uint32_t k = it > (uint32_t) B_STAGES ? it - B_STAGES : 0; k < it; ++k) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(smem_u32(&sh.full_b[k % B_STAGES]), (k / B_STAGES) & 1u) && clock64() - t0 < WAIT_CYCLES) { }
                }
            }
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---- multipliers: gps per token and slice, transposed into [group][token]; tokens beyond M get 0
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t it = 0;
        bool ok = true;
        for (int t = lane; t < NT; t += 32) sh.u[t] = t < M ? __ldg(prm.u + t) : 0.0f;      // (seen by whoever waits for the first slot)
        const int n_ag = nsl * gps;
        for (int tile = first; tile < tiles && ok; tile += stride) {
            for (int sl = 0; sl < n_sl; ++sl, ++it) {
                const uint32_t s = it % MS;
                int4 q[(NT + 31) / 32];
#pragma unroll
                for (int h = 0; h < (NT + 31) / 32; ++h) {      // (requested before the slot is free: a trip to L2 each)
                    const int tok = h * 32 + lane;
                    q[h] = make_int4(0, 0, 0, 0);
                    if (tok < M) {
                        const int32_t * p = prm.msh + (size_t) tok * n_ag + (size_t) (sl0 + sl) * gps;
                        if (gps == 4) q[h] = __ldg(reinterpret_cast<const int4 *>(p));
                        else if (gps == 2) { const int2 v = __ldg(reinterpret_cast<const int2 *>(p)); q[h].x = v.x; q[h].y = v.y; }
                        else q[h].x = __ldg(p);
                    }
                }
                if (!mbar_wait_warp(smem_u32(&sh.m_empty[s]), ((it / MS) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                int * d = m_ring + s * (RUNS * NT);
#pragma unroll
                for (int h = 0; h < (NT + 31) / 32; ++h) {
                    const int tok = h * 32 + lane;
                    if (tok < NT) {
                        d[tok] = q[h].x;
                        d[NT + tok] = q[h].y;
                        d[2 * NT + tok] = q[h].z;
                        d[3 * NT + tok] = q[h].w;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh.m_full[s]));
            }
        }
    } else if (warp == 1) {
        // ---- MMA issue.  The runs per group are a constant of the loop: with a running count deciding, per run, the accumulator and
        // whether it starts anew, an instruction took 57 cycles to issue instead of 14.
        auto issue = [&](auto gsc) {
            constexpr int GS = decltype(gsc)::value;
            uint32_t s = 0, ph = 0;               // ring slot and its phase
            uint32_t ab = 0, aph = 0;             // A buffer
            uint32_t db = 0, dph = 1;             // accumulator buffer
            uint32_t fb = 0;                      // barrier its set completes on
            const uint64_t db0 = umma_desc(ring + W_STAGES * W_BYTES);
            for (int tile = first; tile < tiles; tile += stride) {
                for (int sl = 0; sl < n_sl; ++sl) {
                    if (!mbar_wait_warp(smem_u32(&sh.full_b[s]), ph, abort_flag)) return;
                    const uint64_t bs = db0 + (uint64_t) ((s * b_bytes_of(NT)) >> 4);
#pragma unroll
                    for (int st = 0; st < RUNS / SR; ++st) {
                        // (a set holds a step's groups, or one group that spans two steps)
                        if ((st * SR) % GS == 0 && !mbar_wait_warp(smem_u32(&sh.d_empty[db]), dph, abort_flag)) return;
                        if (!mbar_wait_warp(smem_u32(&sh.a_full[ab]), aph, abort_flag)) return;
                        tc_fence_after();
                        const uint32_t a = tmem_base + ab * (SR * 16), d = tmem_base + rq_w4_d_col(NT) + db * (SR * NT);
#pragma unroll
                        for (int i = 0; i < SR; ++i) {
                            const int r = st * SR + i;
                            // run r: box r / 2, 64 bytes into the swizzled row for odd runs, 32 bytes per instruction
                            const uint64_t b = bs + (uint64_t) (((r >> 1) * (b_bytes_of(NT) / 2) + (r & 1) * 64) >> 4);
                            umma_ts<NT>(d + (i / GS) * NT, a + i * 16, b, r % GS != 0 ? 1 : 0);
                            umma_ts<NT>(d + (i / GS) * NT, a + i * 16 + 8, b + 2, 1);
                        }
                        umma_commit(smem_u32(&sh.a_empty[ab]));
                        if (++ab == NA) { ab = 0; aph ^= 1u; }
                        if ((st * SR + SR) % GS == 0) {
                            umma_commit(smem_u32(&sh.d_full[NF == ND ? db : fb]));
                            if (NF != ND && ++fb == NF) fb = 0;
                            if (++db == ND) { db = 0; dph ^= 1u; }
                        }
                    }
                    umma_commit(smem_u32(&sh.empty_b[s]));
                    if (++s == (uint32_t) B_STAGES) { s = 0; ph ^= 1u; }
                }
            }
        };
        if (gsteps == 1) issue(std::integral_constant<int, 1>{});
        else if (gsteps == 2) issue(std::integral_constant<int, 2>{});
        else issue(std::integral_constant<int, 4>{});
    }
    } else if (warp < 4 + UNPACK_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;" ::: "memory");
        // ---- unpack: warps 4-7 the first half of a step's runs, warps 8-11 the second; a warp's quarter of the 128 rows is fixed
        // by its index
        const int q = warp & 3, set = (warp - 4) >> 2;
        const int row = q * 32 + lane, gid = row & 7;
        const uint32_t src0 = ring + (uint32_t) (row >> 4) * SUB_BYTES + (uint32_t) set * (SR / 2 * 512) + (uint32_t) (row & 8);
        const uint32_t off[4] = { (uint32_t) rq_w4_slot(gid, 0) * 16, (uint32_t) rq_w4_slot(gid, 1) * 16, (uint32_t) rq_w4_slot(gid, 2) * 16,
                                  (uint32_t) rq_w4_slot(gid, 3) * 16 };
        const uint32_t lane_base = tmem_base + ((uint32_t) (q * 32) << 16) + (uint32_t) set * (SR / 2 * 16);
        uint32_t s = 0, ph = 0, ab = 0, aph = 1;
        bool ok = true;
        for (int tile = first; tile < tiles && ok; tile += stride) {
            for (int sl = 0; sl < n_sl && ok; ++sl) {
                if (!mbar_wait_warp(smem_u32(&sh.full_w[s]), ph, abort_flag)) { ok = false; break; }
#pragma unroll
                for (int st = 0; st < RUNS / SR; ++st) {
                    uint32_t v[SR * 8];
#pragma unroll
                    for (int i = 0; i < SR / 2; ++i)
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v[i * 16 + 4 * t + 1]), "=r"(v[i * 16 + 4 * t + 3])
                                         : "r"(src0 + s * W_BYTES + (uint32_t) (st * SR + i) * 512 + off[t]));
#pragma unroll
                    for (int i = 0; i < SR * 8; i += 2) {          // low nibbles: inputs 16*i' of column 4t + i' even, high: odd
                        v[i] = (v[i + 1] << 4) & 0xF0F0F0F0u;
                        v[i + 1] &= 0xF0F0F0F0u;
                    }
                    if (!mbar_wait_warp(smem_u32(&sh.a_empty[ab]), aph, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    tmem_st(lane_base + ab * (SR * 16), v);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh.a_full[ab]));
                    if (++ab == NA) { ab = 0; aph ^= 1u; }
                }
                if (!ok) break;
                if (lane == 0) mbar_arrive(smem_u32(&sh.empty_w[s]));      // (after the __syncwarp of the last step: all lanes have read)
                if (++s == (uint32_t) W_STAGES) { s = 0; ph ^= 1u; }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 144;" ::: "memory");
        // ---- fold
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int q = warp & 3, h = (warp - 4 - UNPACK_WARPS) >> 2, row = q * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t) (q * 32) << 16) + rq_w4_d_col(NT);
        const bool fmt_ok = prm.status == nullptr || prm.status[1] == RQ_FMT_I8;
        if (!fmt_ok && threadIdx.x == (4 + UNPACK_WARPS) * 32) atomicExch(prm.status, 2);
        uint32_t gset = 0, it = 0;            // accumulator sets and slices, all tiles
        bool ok = true;
        for (int tile = first; tile < tiles && ok; tile += stride) {
            const int wi = job_of_tile(prm, tile);
            const W4Job & jb = prm.job[wi];
            const int n = (tile - prm.tile_start[wi]) * ROWS + row;
            const float s_w = n < jb.N ? __ldg(jb.sw + n) : 0.0f;
            const int8_t * kp = nullptr;
            if (HAS_K) kp = jb.wk + (size_t) (n < jb.N ? n : 0) * ng64 + (size_t) sl0 * RUNS;
            int tot[NT];
#pragma unroll
            for (int i = 0; i < NT; ++i) tot[i] = 0;
            for (int sl = 0; sl < n_sl && ok; ++sl, ++it) {
                const uint32_t ms = it % MS;
                const int * mrow = m_ring + ms * (RUNS * NT);
                for (int ds = 0; ds < dsets; ++ds, ++gset) {
                    if ((int) (gset & 1u) != h) continue;
                    uint32_t k4 = 0;
                    if (HAS_K) k4 = __ldg(reinterpret_cast<const uint32_t *>(kp) + sl);      // four multipliers, one per run
                    if (!mbar_wait_warp(smem_u32(&sh.m_full[ms]), (it / MS) & 1u, abort_flag)) { ok = false; break; }
                    const uint32_t db = gset % ND;
                    if (!mbar_wait_warp(smem_u32(&sh.d_full[gset % NF]), (gset / NF) & 1u, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    for (int g = 0; g < dgroups; g += CG) {
                        int v[CG][NT];
#pragma unroll
                        for (int c = 0; c < CG; ++c) if (c == 0 || g + c < dgroups) tmem_ld(lane_base + db * (SR * NT) + (g + c) * NT, v[c]);
#pragma unroll
                        for (int c = 0; c < CG; ++c) tmem_ld_wait(v[c]);
                        if (g + CG >= dgroups) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(smem_u32(&sh.d_empty[db]));
                        }
#pragma unroll
                        for (int c = 0; c < CG; ++c) {
                            if (c > 0 && g + c >= dgroups) break;
                            const int gg = ds * dgroups + g + c;             // group of the slice
                            // (groups of 128 and 256 come with one multiplier for all their runs: the last run's)
                            const int k = HAS_K ? (int) ((k4 >> (8 * (gg * gsteps + gsteps - 1))) & 0xFFu) : 1;
#pragma unroll
                            for (int t = 0; t < NT; t += 4) {
                                const int4 m = *reinterpret_cast<const int4 *>(mrow + gg * NT + t);
                                const int mm[4] = { m.x, m.y, m.z, m.w };
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    if (HAS_K) tot[t + i] += (k * mm[i] * (v[c][t + i] >> 7)) >> 4;
                                    else       tot[t + i] += (mm[i] * v[c][t + i]) >> RQ_FOLD_SHIFT;
                                }
                            }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh.m_empty[ms]));
                }
            }
            // The two warps of a quarter hold totals of different inputs: warp h keeps the tokens of its half and takes the
            // other's totals for them through shared memory.
            constexpr int HALF = NT / 2;
#pragma unroll
            for (int i = 0; i < HALF; ++i) swap[((1 - h) * HALF + i) * ROWS + row] = h ? tot[i] : tot[HALF + i];
            sh.fold_ok[q][h] = ok ? 1 : 0;         // (all lanes write the same; a warp that gave up still meets its partner)
            asm volatile("bar.sync %0, 64;" :: "r"(1 + q) : "memory");
            ok = sh.fold_ok[q][0] != 0 && sh.fold_ok[q][1] != 0;
            if (!ok) break;
#pragma unroll
            for (int i = 0; i < HALF; ++i) tot[i] = (h ? tot[HALF + i] : tot[i]) + swap[(h * HALF + i) * ROWS + row];
            const int tok0 = h * HALF;
            if (split > 1) {
                // token t belongs to CTA t % split: the partial total goes into its shared memory, slot (this CTA, t / split)
                cluster_wait();           // (every CTA of the cluster has started; one tile per cluster)
                const int own = (NT + split - 1) / split;
                int slot = tok0 / split, to = tok0 - slot * split;
                const uint32_t at = smem_u32(part) + (uint32_t) (rank * own * ROWS + row) * 4u;
#pragma unroll
                for (int i = 0; i < HALF; ++i) {
                    asm volatile("st.shared::cluster.b32 [%0], %1;" :: "r"(map_to_cta(at + (uint32_t) (slot * ROWS * 4), (uint32_t) to)), "r"(tot[i]) : "memory");
                    if (++to == split) { to = 0; ++slot; }
                }
            } else {
                if (n < jb.N && fmt_ok) {
                    float * y = jb.y + (size_t) tok0 * jb.ldy + n;
                    const int64_t ldy = jb.ldy;
                    const int more = jb.n_more;
#pragma unroll
                    for (int i = 0; i < HALF; ++i) {
                        if (tok0 + i < M) {
                            const float v = __fmul_rn(__fmul_rn(__fmul_rn((float) tot[i], 16.0f), sh.u[tok0 + i]), s_w);
                            y[(size_t) i * ldy] = v;
                            for (int d = 0; d < more; ++d) jb.y_more[d][(size_t) (tok0 + i) * ldy + n] = v;
                        }
                    }
                }
                asm volatile("bar.sync %0, 64;" :: "r"(1 + q) : "memory");      // (both have read before the next tile's exchange)
            }
        }
        if (split > 1 && !ok) cluster_wait();      // (given up before the push: the barrier's phases stay in step)
    }

    tc_fence_before();
    __syncthreads();
    if (split > 1) {
        if (warp < 4 + UNPACK_WARPS) cluster_wait();
        __syncwarp();
        cluster_arrive();
        asm volatile("griddepcontrol.wait;" ::: "memory");      // (returns at once; some of these threads have not waited yet)
        const int tile = first, wi = job_of_tile(prm, tile);
        const W4Job & jb = prm.job[wi];
        const int row = threadIdx.x & (ROWS - 1), n = (tile - prm.tile_start[wi]) * ROWS + row, own = (NT + split - 1) / split;
        const bool live = n < jb.N && !*abort_flag && (prm.status == nullptr || prm.status[1] == RQ_FMT_I8);
        const float s_w = live ? __ldg(jb.sw + n) : 0.0f;
        cluster_wait();           // all partial totals of this CTA's tokens are here
        if (live) {
            for (int o = (int) (threadIdx.x / ROWS); o * split + rank < M; o += THREADS / ROWS) {
                const int tok = o * split + rank;
                int total = 0;
                for (int r = 0; r < split; ++r) total += part[(r * own + o) * ROWS + row];
                const float v = __fmul_rn(__fmul_rn(__fmul_rn((float) total, 16.0f), sh.u[tok]), s_w);
                jb.y[(size_t) tok * jb.ldy + n] = v;
                for (int d = 0; d < jb.n_more; ++d) jb.y_more[d][(size_t) tok * jb.ldy + n] = v;
            }
        }
    }
    if (threadIdx.x == 0 && sh.abort_flag && prm.status != nullptr) atomicExch(prm.status, 1);
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

template <int NT, bool HAS_K>
cudaError_t configure_w4() {
    return cudaFuncSetAttribute(rq_gemm_w4_kernel<NT, HAS_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem_bytes_of(NT));
}

template <int NT, bool HAS_K>
cudaError_t launch_w4(const CUtensorMap & tx, const CUtensorMap (&tw)[RQ_MAX_WEIGHTS], const W4Params & prm, int sms, cudaStream_t stream) {
    const int tiles = prm.tile_start[prm.n_jobs];
    const int clusters = prm.split > 1 ? tiles : (tiles < sms ? tiles : sms);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (clusters * prm.split));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes_of(NT);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    static const int pdl = getenv("RQ_NO_PDL") ? 0 : 1;      // read once
    attr[0].val.programmaticStreamSerializationAllowed = pdl;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned) prm.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, rq_gemm_w4_kernel<NT, HAS_K>, tx, tw[0], tw[1], tw[2], prm);
}

// clusters of c CTAs that run at the same time (every variant takes an SM to itself, so one stands for all)
cudaError_t clusters_that_fit(int c, int * n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (c * 148));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes_of(64);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned) c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(n, rq_gemm_w4_kernel<64, false>, &cfg);
}

}  // namespace

cudaError_t rq_configure_gemm_w4() {
    cudaError_t e;
    if ((e = configure_w4<16, false>()) != cudaSuccess) return e;
    if ((e = configure_w4<32, false>()) != cudaSuccess) return e;
    if ((e = configure_w4<48, false>()) != cudaSuccess) return e;
    if ((e = configure_w4<64, false>()) != cudaSuccess) return e;
    if ((e = configure_w4<16, true>()) != cudaSuccess) return e;
    if ((e = configure_w4<32, true>()) != cudaSuccess) return e;
    if ((e = configure_w4<48, true>()) != cudaSuccess) return e;
    return configure_w4<64, true>();
}

// M <= 64 tokens of int8 activations (RQ_FMT_I8); all jobs share the activation and the weight-multiplier mode
cudaError_t rq_launch_gemm_w4(const rq_gemv_job * jobs, int n_jobs, int64_t K, const int8_t * a8, const int32_t * msh,
                              const float * u, int64_t M, int G, int32_t * status, cudaStream_t stream) {
    if (n_jobs < 1 || n_jobs > RQ_MAX_WEIGHTS || M < 1 || M > 64) return cudaErrorInvalidValue;
    // first use on a device (normally rq_w4a4_prepare's, outside stream capture); several host threads may get here at once
    static std::mutex mu;
    static int sm_count[64] = {}, max_clusters[64][MAX_SPLIT + 1] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int sms;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (sm_count[dev] == 0) {
            if ((e = rq_configure_gemm_w4()) != cudaSuccess) return e;
            int n = 0;
            if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
            for (int c = 2; c <= MAX_SPLIT; ++c) if ((e = clusters_that_fit(c, &max_clusters[dev][c])) != cudaSuccess) return e;
            sm_count[dev] = n;
        }
        sms = sm_count[dev];
    }
    W4Params prm = {};
    prm.n_jobs = n_jobs;
    for (int i = 0; i < n_jobs; ++i) {
        W4Job & jb = prm.job[i];
        jb.sw = jobs[i].sw; jb.wk = jobs[i].wk; jb.y = jobs[i].y; jb.ldy = jobs[i].ldy; jb.N = (int) jobs[i].N;
        jb.n_more = jobs[i].n_more;
        for (int d = 0; d < jobs[i].n_more; ++d) jb.y_more[d] = jobs[i].y_more[d];
        prm.tile_start[i + 1] = prm.tile_start[i] + (int) ((jobs[i].N + ROWS - 1) / ROWS);
    }
    prm.msh = msh; prm.u = u; prm.status = status; prm.K = (int) K; prm.M = (int) M; prm.G = G;
    // K is split while that puts more SMs to work: as many CTAs per row tile as let all clusters run at once (clusters stay
    // inside a GPC, so fewer fit than the SM count suggests)
    const int tiles = prm.tile_start[n_jobs], nsl = (int) (K / SLICE);
    int split = MAX_SPLIT;
    while (split > 1 && (split > nsl || max_clusters[dev][split] < tiles)) --split;
    prm.split = split;
    const int nt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 48 ? 48 : 64;
    alignas(64) CUtensorMap tx, tw[RQ_MAX_WEIGHTS];
    for (int i = 0; i < RQ_MAX_WEIGHTS; ++i) {
        const rq_gemv_job & jb = jobs[i < n_jobs ? i : 0];
        if (rq_encode_tmap_w4(&tw[i], jb.w4, K, (jb.N + 15) / 16) != 0) return cudaErrorInvalidValue;
    }
    if (rq_encode_tmap_i8(&tx, a8, K, M, nt) != 0) return cudaErrorInvalidValue;
    const bool has_k = jobs[0].wk != nullptr;
    switch (nt) {
        case 16: return has_k ? launch_w4<16, true>(tx, tw, prm, sms, stream) : launch_w4<16, false>(tx, tw, prm, sms, stream);
        case 32: return has_k ? launch_w4<32, true>(tx, tw, prm, sms, stream) : launch_w4<32, false>(tx, tw, prm, sms, stream);
        case 48: return has_k ? launch_w4<48, true>(tx, tw, prm, sms, stream) : launch_w4<48, false>(tx, tw, prm, sms, stream);
        default: return has_k ? launch_w4<64, true>(tx, tw, prm, sms, stream) : launch_w4<64, false>(tx, tw, prm, sms, stream);
    }
}
