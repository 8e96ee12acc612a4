// Prefill-width contraction on the sm_100a tensor cores: tcgen05.mma with the accumulator in tensor memory, operands
// staged by TMA, and the reference's per-group fold done by the epilogue warps straight out of tensor memory while the
// tensor pipe works on the next group.
//
// Why the accumulator leaves tensor memory every G inputs: the reference shifts each group's term right by 4 before
// the int32 sum (ggml_vec_dot_w4a4_a4, ggml/src/ggml-cpu/quants.c in patches/llama.cpp-ruquant.patch:173), which is
// not linear, so groups cannot be accumulated together.  Two operand formats:
//   F8  (weights without multipliers, the usual case): A = e4m3 byte of (q - z_g) [M][K], B = e4m3 byte of c [N][K],
//       tcgen05.mma kind::f8f6f4 with fp32 accumulators, which hold S_g exactly (sums of products of small integers);
//       the fold (m_g * S_g) >> 4 is ONE round-down FMA per output on a running total kept in [2^23, 2^24).
//   I8  (weights with multipliers k): A = int8 8*(q - z_g), B = int8 k*c, kind::i8, D = 8*k*S_g, term = (D * m_g) >> 7.
// Tokens are the MMA's M rows (TMEM lanes), weight rows its N columns: an epilogue thread owns one token, so m_g is
// one register per group.
//
// CTA = 128 tokens x BN = 256 weight rows (fewer where that fills the chip better).  Warp 0 lane 0: TMA producer over a ring of
// 128-input K slices (128B swizzle).  Warp 1: TMEM allocation and MMA issue into two accumulator buffers.  Warps 4-11: fold +
// final fp32 epilogue y = ((float(total) * 16) * u) * s_w.
//
// What bounds the kernel, per 64 inputs and 256 rows: the MMAs take 257 cycles, tensor memory delivers the 32 K sums in 186, the
// folds need 256 cycles of the fp32 pipe, and the port of shared memory 384: 24 KB of operands written by the copies and read
// by the MMAs at 128 bytes a cycle.  It runs at about 600 (389 us for 4096 tokens x 5120 x 17408, 1875 TOPS; 458 before); with
// the folds compiled out at 460.  The rest is the epilogue warps' own: the first load of a group (its barrier is looked at one
// piece ahead: 5 to 12 %), the look at the totals (3 %), the multipliers (3 %), the final scaling and store (7 %).
// Pairs of CTAs (cta_group::2, half of the weight rows staged by each, 256 cycles of the shared-memory port) were 3 to 6 %
// slower at 512 and 4096 tokens and take twice the tokens per unit: their releases and commits cross the pair, and with two
// buffers that loop sets the pace.  Two MMAs of 128 rows with buffers of their own read the tokens twice (449 cycles): 2 % slower.
// PUSH (N-sharded ranks): warps 2 and 3 copy every finished unit from this GPU's output into the other ranks' copies
// (peer stores), so that no folding warp ever waits for NVLink.
// Every wait is bounded: on expiry the waiter raises a CTA-wide abort flag and a status word in global memory,
// everyone leaves the pipeline, outstanding TMA transactions are drained and tensor memory is released.
#include <cuda.h>

#include <stdlib.h>

#include <mutex>
#include <type_traits>

#include "rq_common.cuh"

namespace {

constexpr int BM = 128, BK = 128;
constexpr int TC_THREADS = 384;
// A tile has BN = 32 * NQ weight rows, NQ = 4, 5, 6 or 8; an epilogue warp folds half of them
constexpr int BUF_COLS = 256;                       // tensor memory of an accumulator buffer
constexpr int STAGES = 4;
constexpr uint32_t A_BYTES = BM * BK;
__host__ __device__ constexpr uint32_t bh_bytes_of(int nq) { return (uint32_t) nq * 16 * BK; }      // half a tile of weight rows
__host__ __device__ constexpr uint32_t stage_bytes_of(int nq) { return A_BYTES + 2u * bh_bytes_of(nq); }
constexpr uint32_t STAGING_BYTES = 8 * 32 * 32 * 4;      // a 32 x 32 fp32 transposition tile per epilogue warp
__host__ __device__ constexpr uint32_t smem_bytes_of(int nq) { return STAGES * stage_bytes_of(nq) + STAGING_BYTES + 1024; }   // + alignment slack
constexpr long long WAIT_CYCLES = 2000000000ll;                // about a second at B200 clocks
constexpr uint32_t TMEM_COLS = 512;

__device__ __forceinline__ uint32_t smem_u32(const void * p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
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

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap * map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 :: "r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// lane 0's arrival as a predicated instruction: no branch, no reconvergence around it
__device__ __forceinline__ void mbar_arrive_lane0(uint32_t bar, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" :: "r"(bar), "r"(lane) : "memory");
}
// K-major operand tile in the canonical 128B-swizzled layout TMA writes: rows of 128 bytes, 8-row atoms 1024 bytes
// apart.  Fields: start address >> 4 [0,14), leading byte offset >> 4 [16,30) (unused for swizzled K-major, 1),
// stride byte offset >> 4 [32,46), descriptor version 1 [46,48), layout type SWIZZLE_128B = 2 [61,64).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    return (uint64_t) ((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t) (1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::i8: D = s32 (2 at [4,6)), A and B signed int8 (1 at [7,10) and [10,13)), both
// K-major (0 at 15, 16), N >> 3 at [17,23), M >> 4 at [24,29)
// kind::f8f6f4: D = f32 (1 at [4,6)), A and B e4m3 (0 at [7,10) and [10,13)), K-major, same N and M fields
__host__ __device__ constexpr uint32_t idesc_of(bool f8, int n) {
    return (f8 ? (1u << 4) : ((2u << 4) | (1u << 7) | (1u << 10))) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (BM >> 4) << 24);
}

// One instruction of K = 32: 128 tokens x N weight rows.  Called by the whole (converged) warp with warp-uniform operands; one
// elected lane issues.
template <bool F8, int N>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, int acc) {
    if (F8) asm volatile("{\n\t.reg .pred pe, p;\n\telect.sync _|pe, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t@pe tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                         :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc_of(true, N)), "r"(acc) : "memory");
    else    asm volatile("{\n\t.reg .pred pe, p;\n\telect.sync _|pe, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t@pe tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                         :: "r"(tmem_d), "l"(da), "l"(db), "r"(idesc_of(false, N)), "r"(acc) : "memory");
}
// the commits, like the MMAs, are called by the whole warp and issued by one elected lane
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("{\n\t.reg .pred pe;\n\telect.sync _|pe, 0xffffffff;\n\t@pe tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, int (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                   "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                   "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                 : "r"(taddr) : "memory");
}
// 16 columns, into the first half of the buffer
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int (&v)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr) : "memory");
}
template <int W>
__device__ __forceinline__ void tmem_ld_piece(uint32_t taddr, int (&v)[32]) {
    if constexpr (W == 32) tmem_ld32(taddr, v);
    else tmem_ld16(taddr, v);
}
// completes this thread's outstanding tensor-memory loads; the values are threaded through as read-write operands
// so that no use of them can be scheduled above the wait
__device__ __forceinline__ void tmem_ld_wait(int (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                   "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
                   "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :: "memory");
}

// integer path (weights k*c, activations 8*(q - z)): D = 8*k*S, term = (D * m) >> 7: one integer multiply and one
// shift-add per output per group (measured on B200: 50+ outputs per clock per SM, against 30 for a high multiply-add)
template <int BASE, int W, int HC>
__device__ __forceinline__ void fold_i8(int (&tot)[HC], const int (&v)[32], int mm) {
#pragma unroll
    for (int i = 0; i < W; ++i) tot[BASE + i] += (v[i] * mm) >> 7;
}

// fp8 path: D = S exactly (fp32 accumulation of products of small integers).  The running total lives in a float
// kept inside [2^23, 2^24), where the spacing of floats is 1: a round-down fused multiply-add
//     t <- fma.rm(S, m/16, t)
// adds floor(S*m/16) = (m*S) >> 4 exactly (S*m/16 has at most 21 + 4 significant bits below 2^23, the sum is rounded
// once, downwards, to an integer) -- the reference's shifted term in ONE instruction.  Two neighbouring columns share
// a 64-bit register pair and one packed instruction (fma.rm.f32x2): half the issue slots of the scalar form.
constexpr int FOLD_MAGIC_BITS = 0x4B480000;      // 2^23 + 2^22 + 2^19
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, uint32_t & lo, uint32_t & hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
template <int BASE, int W, int HP>
__device__ __forceinline__ void fold_f8(uint64_t (&tf)[HP], const int (&v)[32], uint64_t mf2) {
#pragma unroll
    for (int i = 0; i < W / 2; ++i)
        asm("fma.rm.f32x2 %0, %1, %2, %0;" : "+l"(tf[BASE / 2 + i]) : "l"(pack2((uint32_t) v[2 * i], (uint32_t) v[2 * i + 1])), "l"(mf2));
}
// Re-centring.  A float in the window is 2^23 + mantissa with mantissa = 4.5 * 2^20 + t, t the running total since the last
// re-centring.  Every CHECK_INPUTS inputs a warp looks whether all its totals have t in [-2^19, 2^19), that is bits 22..20 of the
// mantissa = 100: an AND and an OR over the totals, a logic operation each per output.  With the activations and weights of a
// model they always have.  Otherwise these bits, a digit in 0..7, move into an unsigned byte of a packed carry word and are set
// to 4.  Bounds: a group of G inputs adds at most 255 * (G*8*15) / 16 in magnitude, 2.94 M per 1536 inputs, on top of t in
// [-2^19, 2^19): the mantissa stays inside [4 * 2^20 - 2.94 M, 5 * 2^20 + 2.94 M), within [0, 2^23); K <= 32768 has at most 32
// re-centrings (groups of 256 are looked at every 1024 inputs, the nearest multiple of four groups), so a byte holds at most
// 32 * 7 = 224.  At the end
//     total = (sum of digits - 4 * number of re-centrings) * 2^20 + (float - 12.5 * 2^20),
// the last term being t, whatever its size.  (Moving the digits every 1536 inputs without looking cost 10 % of the kernel.)
constexpr int CHECK_INPUTS = 1536;
// The carry words live in shared memory between re-centrings (the per-warp tile that later stages the transposed
// store; word w of lane l at w * 32 + l: conflict-free) -- the registers they would take are the difference between a
// fold loop that fits and one that spills.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
// Integer instructions run at half the rate of the FMAs on this part, so the re-centring counts them: byte 2 of each
// of four floats (mantissa bits 16..23) is gathered with three byte permutes, one shift and one mask turn the four
// bytes into the four digits, already packed as the carry word wants them; one logic op per float resets the digit.
template <int HP>
__device__ __forceinline__ bool totals_centred(const uint64_t (&tf)[HP]) {
    uint32_t all = 0xffffffffu, any = 0u;
#pragma unroll
    for (int i = 0; i < HP; ++i) {
        uint32_t lo, hi;
        unpack2(tf[i], lo, hi);
        all &= lo & hi;
        any |= lo | hi;
    }
    return __all_sync(0xffffffffu, (all & 0x00400000u) != 0u && (any & 0x00300000u) == 0u);
}
template <int HP>
__device__ __forceinline__ void recenter(uint64_t (&tf)[HP], uint32_t * carry_smem) {
    const uint32_t base = smem_u32(carry_smem);
#pragma unroll
    for (int i = 0; i < HP / 2; ++i) {          // carry word i: columns 4i .. 4i+3 = pairs 2i, 2i+1
        uint32_t w[4];
        unpack2(tf[2 * i], w[0], w[1]);
        unpack2(tf[2 * i + 1], w[2], w[3]);
        const uint32_t g = prmt(prmt(w[0], w[1], 0x0062u), prmt(w[2], w[3], 0x0062u), 0x5410u);
        const uint32_t cw = (g >> 4) & 0x07070707u;
        // a reduction without a return value: nothing waits for shared memory here (a load-add-store chain per word
        // would, the fold leaves no registers to batch the loads)
        asm volatile("red.shared.add.u32 [%0], %1;" :: "r"(base + (uint32_t) (i * 128)), "r"(cw) : "memory");
        // the digits are reset on the 64-bit pairs where they live: two logic ops per pair on its own halves -- taking the
        // halves apart, changing them and packing them again cost four register moves per pair on top
        tf[2 * i] = (tf[2 * i] & 0xFF8FFFFFFF8FFFFFull) | 0x0040000000400000ull;
        tf[2 * i + 1] = (tf[2 * i + 1] & 0xFF8FFFFFFF8FFFFFull) | 0x0040000000400000ull;
    }
}

// Up to three weights that share the activation (q/k/v, gate/up) are one launch: their row tiles form one list, so that a
// narrow weight's few tiles do not leave most of the chip idle for a launch of their own.
struct TcJob {
    const float * sw;
    float * y;
    float * y_more[RQ_MAX_RANKS - 1];   // further copies of the output (other ranks' buffers, peer-mapped), same layout
    int64_t ldy;
    int N;
    int n_more;
    int vec;                            // 16-byte stores are safe: ldy % 4 == 0 and every destination 16-byte aligned
};
struct TcParams {
    TcJob job[RQ_MAX_WEIGHTS];
    int tile_start[RQ_MAX_WEIGHTS + 1]; // in tiles of 32 * NQ weight rows
    int n_jobs;
    const int32_t * msh;
    const float * u;
    int32_t * status;
    int K, M, G;
};

__device__ __forceinline__ int job_of_tile(const TcParams & prm, int tile) {
    int w = 0;
#pragma unroll
    for (int i = 1; i < RQ_MAX_WEIGHTS; ++i) if (i < prm.n_jobs && tile >= prm.tile_start[i]) w = i;
    return w;
}

struct __align__(8) TcShared {
    uint64_t full[STAGES], empty[STAGES];
    uint64_t tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
    int abort_flag;
    unsigned int units_stored;          // PUSH: epilogue warps that have stored a unit, summed over units (8 per unit)
};

// F8 = true: multipliers all 1, operands are e4m3 bytes of c and (q - z), fp8 MMA with fp32 accumulators, float fold.
// F8 = false: weight multipliers present, B holds int8 k*c, A int8 8*(q - z), integer MMA and integer fold.
// The kernel is persistent: CTA c takes work units c, c + stride, ... where unit v = n_tile * m_tiles + m_tile -- token tiles
// fastest, so the CTAs running at one time share their weight slices in L2.  Slots, phases and
// accumulator buffers are running counters that carry over from one unit to the next: the MMAs of the next unit start
// while the epilogue warps still scale and store the previous one.
template <bool F8, bool PUSH, int NQ>
__global__ void __launch_bounds__(TC_THREADS, 1)
rq_gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b0, const __grid_constant__ CUtensorMap tmap_b1,
                  const __grid_constant__ CUtensorMap tmap_b2, const TcParams prm) {
    constexpr int BN = 32 * NQ, HC = 16 * NQ;            // weight rows of a tile, columns of an epilogue warp
    constexpr uint32_t BH_BYTES = bh_bytes_of(NQ);
    static_assert(!PUSH || NQ == 8, "the pushing warps carry rows of 256 columns");
    constexpr uint32_t STAGE_BYTES = stage_bytes_of(NQ);
    extern __shared__ uint8_t smem_raw[];
    __shared__ TcShared sh;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    // (the warp index through a shuffle from lane 0: the compiler then knows that it, and every tensor-memory and barrier
    // address derived from it, is the same in all lanes, and keeps them in uniform registers)
    const int warp = __shfl_sync(0xffffffffu, (int) (threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int n_ks = prm.K / BK;          // ring slices of 128 inputs
    const int gsteps = prm.G / 64;        // 64-input steps per activation group: 1, 2 or 4
    const int n_ag = prm.K / prm.G;       // activation groups
    const int m_tiles = (prm.M + BM - 1) / BM, units = m_tiles * prm.tile_start[prm.n_jobs];
    const int first = (int) blockIdx.x, stride = (int) gridDim.x;
    volatile int * abort_flag = &sh.abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&sh.full[s]), 1); mbar_init(smem_u32(&sh.empty[s]), 1); }
        // an accumulator buffer is free when the 8 epilogue warps have arrived
        for (int b = 0; b < 2; ++b) { mbar_init(smem_u32(&sh.tmem_full[b]), 1); mbar_init(smem_u32(&sh.tmem_empty[b]), 8); }
        sh.abort_flag = 0;
        sh.units_stored = 0;
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
    const uint32_t tmem_base = sh.tmem_base;

    // warps 0-3 (TMA, MMA, two idle) give registers back; the two epilogue warpgroups take them
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;" ::: "memory");
    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;              // slices issued, all units
            bool ok = true;
            // the weights do not depend on the kernel ahead (the quantizer): those of the first slices are asked for before the wait
            uint32_t early = 0;
            for (int v = first; v < units && ok; v += stride) {
                const int n_tile = v / m_tiles, m_tile = v - n_tile * m_tiles;
                const int wi = job_of_tile(prm, n_tile), brow = (n_tile - prm.tile_start[wi]) * BN;
                const CUtensorMap * tmap_b = wi == 0 ? &tmap_b0 : wi == 1 ? &tmap_b1 : &tmap_b2;
                auto load_b = [&](uint32_t s, int ks) {
                    const uint32_t dst = ring + s * STAGE_BYTES + A_BYTES, bar = smem_u32(&sh.full[s]);
                    mbar_expect_tx(bar, STAGE_BYTES);
                    tma_load_2d(dst, tmap_b, bar, ks * BK, brow);
                    tma_load_2d(dst + BH_BYTES, tmap_b, bar, ks * BK, brow + BN / 2);
                };
                if (v == first) {
                    for (; early < (uint32_t) STAGES && early < (uint32_t) n_ks; ++early) load_b(early, (int) early);
                    asm volatile("griddepcontrol.wait;" ::: "memory");
                }
                for (int ks = 0; ks < n_ks; ++ks, ++it) {
                    const uint32_t s = it % STAGES;
                    if (it >= early) {
                        if (!mbar_wait(smem_u32(&sh.empty[s]), ((it / STAGES) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
                        load_b(s, ks);
                    }
                    tma_load_2d(ring + s * STAGE_BYTES, &tmap_a, smem_u32(&sh.full[s]), ks * BK, m_tile * BM);
                }
            }
            if (*abort_flag) {
                // drain: every slice that was issued must land before the CTA's shared memory is given back
                for (uint32_t k = it > (uint32_t) STAGES ? it - STAGES : 0; k < it; ++k) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(smem_u32(&sh.full[k % STAGES]), (k / STAGES) & 1u) && clock64() - t0 < WAIT_CYCLES) { }
                }
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the loop with warp-uniform values (descriptors and addresses then live in the uniform
        // datapath) and elects a lane at each MMA and commit.
        const uint64_t da0 = umma_desc(ring), db0 = umma_desc(ring + A_BYTES);
        uint32_t s = 0, ph = 0;               // ring slot and its phase
        bool ok = true;
        auto wait = [&](uint64_t * bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, abort_flag)); };
        auto done_slice = [&]() {
            umma_commit(smem_u32(&sh.empty[s]));
            if (++s == (uint32_t) STAGES) { s = 0; ph ^= 1u; }
        };
        if (gsteps == 1) {
            // groups of 64 inputs (the usual case): group h of a slice goes to buffer h, nothing but the phase is left to
            // compute (an MMA takes 14 cycles to issue, 57 when a running count decides its accumulator and whether it starts it)
            uint32_t aph = 1;
            for (int v = first; v < units && ok; v += stride) {
                for (int ks = 0; ks < n_ks && ok; ++ks, aph ^= 1u) {
                    if (!wait(&sh.full[s], ph)) { ok = false; break; }
                    const uint64_t so = (uint64_t) ((s * STAGE_BYTES) >> 4);
                    const uint64_t da = da0 + so, db = db0 + so;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (!wait(&sh.tmem_empty[h], aph)) { ok = false; break; }
                        tc_fence_after();
                        umma<F8, BN>(tmem_base + h * BUF_COLS, da + h * 4, db + h * 4, 0);          // bytes >> 4 inside the swizzled row
                        umma<F8, BN>(tmem_base + h * BUF_COLS, da + h * 4 + 2, db + h * 4 + 2, 1);
                        umma_commit(smem_u32(&sh.tmem_full[h]));
                    }
                    if (ok) done_slice();
                }
            }
        } else {
            // wider groups are whole slices
            const int spg = gsteps >> 1;
            uint32_t gcount = 0;                  // accumulator groups issued, all units
            int sg = 0;                           // slices of the current group already issued
            for (int v = first; v < units && ok; v += stride) {
                for (int ks = 0; ks < n_ks; ++ks) {
                    const uint32_t buf = gcount & 1u;
                    if (!wait(&sh.full[s], ph) || (sg == 0 && !wait(&sh.tmem_empty[buf], ((gcount >> 1) & 1u) ^ 1u))) { ok = false; break; }
                    tc_fence_after();
                    const uint64_t so = (uint64_t) ((s * STAGE_BYTES) >> 4);
                    const uint64_t da = da0 + so, db = db0 + so;
#pragma unroll
                    for (int i = 0; i < 4; ++i) umma<F8, BN>(tmem_base + buf * BUF_COLS, da + 2 * i, db + 2 * i, sg == 0 && i == 0 ? 0 : 1);
                    if (++sg == spg) { umma_commit(smem_u32(&sh.tmem_full[buf])); sg = 0; ++gcount; }
                    done_slice();
                }
            }
        }
    } else if (PUSH && prm.job[0].n_more > 0) {
        // Warps 2 and 3 carry the finished units to the other ranks.  The epilogue warps store a unit into this GPU's
        // output only; these two warps read it back (from L2) and store it into every other rank's copy.  Peer stores
        // drain at NVLink speed -- a quarter of a unit's fold time per destination at best -- and a warp that waits for
        // them cannot fold: issued by the epilogue warps they added their whole duration to the kernel.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int pw = warp - 2;
        const TcJob & jb = prm.job[0];           // (one weight per pushing launch)
        const bool fmt_ok = prm.status == nullptr || prm.status[1] == (F8 ? RQ_FMT_E4M3 : RQ_FMT_I8);
        volatile unsigned int * stored = &sh.units_stored;
        unsigned int k = 0;
        // (a wrong activation format: the epilogue warps store nothing and count nothing, so there is nothing to wait for)
        for (int v = first; v < units && fmt_ok; v += stride, ++k) {
            bool ok = true;
            const long long t0 = clock64();
            while (*stored < 8u * (k + 1u)) {          // bounded, like every wait of this kernel
                if (*abort_flag) { ok = false; break; }
                if (clock64() - t0 > WAIT_CYCLES) { *abort_flag = 1; ok = false; break; }
                __nanosleep(256);
            }
            if (!__all_sync(0xffffffffu, ok)) break;
            __threadfence();
            const int n_tile = v / m_tiles, m_tile = v - n_tile * m_tiles;
            const int row0 = m_tile * BM, col = n_tile * BN + (pw * 32 + lane) * 4;      // 64 lanes x 4 columns = a unit's row
            const int rows = prm.M - row0 < BM ? prm.M - row0 : BM;
            if (jb.vec && col + 3 < jb.N) {
                // four rows of loads in flight per lane (eight, with registers taken from the epilogue warps, changed
                // nothing: 0.494 against 0.497 ms for the 4096 x 17408 node on 4 GPUs -- the peer stores set the pace, about
                // 3.4 GB/s per SM whichever warps issue them)
                for (int r = 0; r < rows; r += 4) {
                    float4 q[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (r + u < rows) q[u] = __ldcg(reinterpret_cast<const float4 *>(jb.y + (size_t) (row0 + r + u) * jb.ldy + col));
                    for (int d = 0; d < jb.n_more; ++d) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (r + u < rows) *reinterpret_cast<float4 *>(jb.y_more[d] + (size_t) (row0 + r + u) * jb.ldy + col) = q[u];
                    }
                }
            } else if (col < jb.N) {
                for (int r = 0; r < rows; ++r) {
                    const size_t at = (size_t) (row0 + r) * jb.ldy + col;
                    float q[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) q[u] = col + u < jb.N ? __ldcg(jb.y + at + u) : 0.0f;
                    for (int d = 0; d < jb.n_more; ++d) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (col + u < jb.N) jb.y_more[d][at + u] = q[u];
                    }
                }
            }
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;" ::: "memory");
        const int e = warp - 4, quarter = warp & 3, half = e >> 2;
        uint32_t lane_base = tmem_base + ((uint32_t) (quarter * 32) << 16) + (uint32_t) (half * HC);
        // (opaque to the compiler from here on: it would otherwise rebuild the address from the warp index -- seven integer
        // instructions -- in front of every tensor-memory load instead of keeping it in a register)
        asm volatile("" : "+r"(lane_base));
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // the quantizer records the format it wrote: refuse to multiply the wrong one
        const bool fmt_ok = prm.status == nullptr || prm.status[1] == (F8 ? RQ_FMT_E4M3 : RQ_FMT_I8);
        const uint32_t empty_bar0 = smem_u32(&sh.tmem_empty[0]), full_bar0 = smem_u32(&sh.tmem_full[0]);
        // groups between two looks at the totals: a multiple of four (the loop below walks four groups at a time)
        const int check_every = prm.G >= 256 ? 4 : CHECK_INPUTS / prm.G;
        const bool fast4 = (n_ag & 3) == 0;            // the unit's groups come in fours; then a token's multipliers are 16-byte aligned, too
        float * stg = reinterpret_cast<float *>(smem_raw + (ring - smem_u32(smem_raw)) + STAGES * STAGE_BYTES) + e * 1024;
        uint32_t * carry_smem = reinterpret_cast<uint32_t *>(stg) + lane;
        uint32_t gcount = 0;              // accumulator groups folded (all units)
        bool ok = true;
        RQ_CYC_DECL(c_tfull);
        RQ_CYC_DECL(c_epi);
        RQ_CYC_DECL(c_hold);
        RQ_CYC_DECL(c_rec);
        RQ_CYC_DECL(c_fin);
        RQ_CYC_DECL(c_tail);
        RQ_CYC_BEGIN(c_epi);
        for (int v = first; v < units && ok; v += stride) {
            const int n_tile = v / m_tiles, m_tile = v - n_tile * m_tiles;
            const int row = m_tile * BM + quarter * 32 + lane;
            const bool row_ok = row < prm.M;
            // rows beyond M: zeros from the TMA, folded with token 0's multipliers and never stored
            const int32_t * mrow = prm.msh + (size_t) (row_ok ? row : 0) * n_ag;
            // (kept in registers for the unit: rebuilt from the lane index they cost a dozen integer instructions per load)
            asm volatile("" : "+l"(mrow));
            // the multipliers of four groups at a time
            auto load_m4 = [&](int ag) -> int4 {
                if (fast4) return __ldg(reinterpret_cast<const int4 *>(mrow + ag));
                int4 r = make_int4(0, 0, 0, 0);
                r.x = __ldg(mrow + ag);
                if (ag + 1 < n_ag) r.y = __ldg(mrow + ag + 1);
                if (ag + 2 < n_ag) r.z = __ldg(mrow + ag + 2);
                if (ag + 3 < n_ag) r.w = __ldg(mrow + ag + 3);
                return r;
            };
            int tot[F8 ? 1 : HC];
            uint64_t tf[F8 ? HC / 2 : 1];
            if (F8) {
#pragma unroll
                for (int i = 0; i < HC / 2; ++i) tf[F8 ? i : 0] = pack2((uint32_t) FOLD_MAGIC_BITS, (uint32_t) FOLD_MAGIC_BITS);
            } else {
#pragma unroll
                for (int i = 0; i < HC; ++i) tot[F8 ? 0 : i] = 0;
            }
            int since = 0, n_rec = 0;
            int4 mcur = load_m4(0);
            // Software pipeline over 32-column pieces of the accumulator: the tensor-memory load of piece c+1 is in flight
            // while piece c folds, and the first piece of the NEXT group is requested (its barrier permitting) before the
            // last piece of this group folds, so a warp never sits out a whole load latency.
            int va[32], vb[32];
            RQ_CYC_BEGIN(c_tfull);
            if (!__all_sync(0xffffffffu, mbar_wait(full_bar0 + (gcount & 1u) * 8u, (gcount >> 1) & 1u, abort_flag))) { ok = false; break; }
            RQ_CYC_END(c_tfull);
            tc_fence_after();
            tmem_ld32(lane_base + (gcount & 1u) * BUF_COLS, va);
            for (int ag = 0; ag < n_ag && ok; ag += 4) {
                const int mq[4] = { mcur.x, mcur.y, mcur.z, mcur.w };
                if (ag + 4 < n_ag) mcur = load_m4(ag + 4);
                const int cnt = n_ag - ag < 4 ? n_ag - ag : 4;
                // the unit's last groups: what its final scaling reads (u, and four row units a lane) is asked for now, so that it comes
                // from L1 then
                if (ag + 4 >= n_ag) {
                    const int wj = job_of_tile(prm, n_tile), c0 = (n_tile - prm.tile_start[wj]) * BN + half * HC + lane * 4;
                    float t0, t1 = 0.0f;
                    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(t0) : "l"(prm.u + (row_ok ? row : 0)));
                    if (lane * 4 < HC && c0 < prm.job[wj].N) asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(t1) : "l"(prm.job[wj].sw + c0));
                }
                // One group.  FAST: the unit's groups come in fours (always with groups of 64 inputs), so the accumulator
                // buffer and the barrier phase of group j of the four are known when the code is compiled, up to the
                // phase p0 the four start with -- the integer instructions that would derive them from the running
                // count run at half rate and hold the issue port.
                auto group = [&](auto jc, auto fc, uint32_t p0) {
                    constexpr int J = decltype(jc)::value;
                    constexpr bool FAST = decltype(fc)::value;
                    const uint32_t buf = FAST ? (uint32_t) (J & 1) : (gcount & 1u);
                    const uint32_t t0 = lane_base + buf * BUF_COLS;
                    uint64_t mf2 = 0;
                    if constexpr (F8) mf2 = pack2((uint32_t) mq[J], (uint32_t) mq[J]);      // f32 bits of m / 16, twice
                    const int mm = mq[J];
                    RQ_CYC_BEGIN(c_hold);
                    // pieces of 32 columns, the last one 16 wide when NQ is odd; piece 0 of group J is in va or vb by the number
                    // of pieces before it (four groups hold an even number)
                    auto pieces = [&](auto & self, auto pc, int (&cur)[32], int (&nxt)[32]) {
                        constexpr int P = decltype(pc)::value, W = HC - 32 * P < 32 ? HC - 32 * P : 32;
                        constexpr bool LAST = 32 * (P + 1) >= HC;
                        // the first look at the next group's barrier goes out ahead of the wait for this piece
                        const bool more = FAST ? (J < 3 || ag + 4 < n_ag) : (ag + J + 1 < n_ag);
                        const uint32_t nbuf = FAST ? (uint32_t) ((J + 1) & 1) : ((gcount + 1u) & 1u);
                        const uint32_t nph = FAST ? (p0 ^ (uint32_t) (((J + 1) >> 1) & 1)) : (((gcount + 1u) >> 1) & 1u);
                        bool ready = false;
                        if (LAST && more) ready = mbar_try_wait(full_bar0 + nbuf * 8u, nph);
                        tmem_ld_wait(cur);
                        if constexpr (!LAST) {
                            tmem_ld_piece<(HC - 32 * (P + 1) < 32 ? HC - 32 * (P + 1) : 32)>(t0 + 32 * (P + 1), nxt);
                            if constexpr (F8) fold_f8<32 * P, W>(tf, cur, mf2); else fold_i8<32 * P, W>(tot, cur, mm);
                            self(self, std::integral_constant<int, P + 1>{}, nxt, cur);
                        } else {
                            // the accumulator is in registers: hand the buffer back before the last piece is folded
                            tc_fence_before();
                            __syncwarp();
                            mbar_arrive_lane0(empty_bar0 + buf * 8u, lane);
                            RQ_CYC_END(c_hold);
                            RQ_CYC_BEGIN(c_tail);
                            ++gcount;
                            if (more) {
                                // the loads are warp-collective: leave the loop together or not at all
                                RQ_CYC_BEGIN(c_tfull);
                                if (!__all_sync(0xffffffffu, ready)) ok = __all_sync(0xffffffffu, mbar_wait(full_bar0 + nbuf * 8u, nph, abort_flag));
                                RQ_CYC_END(c_tfull);
                                if (ok) {
                                    tc_fence_after();
                                    tmem_ld32(lane_base + nbuf * BUF_COLS, nxt);
                                }
                            }
                            if constexpr (F8) fold_f8<32 * P, W>(tf, cur, mf2); else fold_i8<32 * P, W>(tot, cur, mm);
                        }
                    };
                    if constexpr ((J * ((HC + 31) / 32)) & 1) pieces(pieces, std::integral_constant<int, 0>{}, vb, va);
                    else                                      pieces(pieces, std::integral_constant<int, 0>{}, va, vb);
                    RQ_CYC_END(c_tail);
                };
                if (fast4) {
                    uint32_t p0 = (gcount >> 1) & 1u;
                    asm volatile("" : "+r"(p0));           // (likewise: one value per four groups, not three instructions per use)
                    if (ok) group(std::integral_constant<int, 0>{}, std::true_type{}, p0);
                    if (ok) group(std::integral_constant<int, 1>{}, std::true_type{}, p0);
                    if (ok) group(std::integral_constant<int, 2>{}, std::true_type{}, p0);
                    if (ok) group(std::integral_constant<int, 3>{}, std::true_type{}, p0);
                } else {
                    if (0 < cnt && ok) group(std::integral_constant<int, 0>{}, std::false_type{}, 0u);
                    if (1 < cnt && ok) group(std::integral_constant<int, 1>{}, std::false_type{}, 0u);
                    if (2 < cnt && ok) group(std::integral_constant<int, 2>{}, std::false_type{}, 0u);
                    if (3 < cnt && ok) group(std::integral_constant<int, 3>{}, std::false_type{}, 0u);
                }
                if constexpr (F8) {
                    since += cnt;
                    if (since >= check_every) {          // (after the unit's last groups as well: the final conversion does not need it)
                        RQ_CYC_BEGIN(c_rec);
                        since = 0;
                        if (!totals_centred(tf)) {
                            if (n_rec == 0) {                   // (the previous unit's store ended with a warp barrier)
#pragma unroll
                                for (int i = 0; i < HC / 4; ++i) carry_smem[i * 32] = 0u;
                            }
                            recenter(tf, carry_smem);
                            ++n_rec;
                        }
                        RQ_CYC_END(c_rec);
                    }
                }
            }
            if (!ok) break;
            if (!fmt_ok) {
                if (lane == 0 && prm.status != nullptr) atomicExch(prm.status, 2);
                continue;
            }
            RQ_CYC_BEGIN(c_fin);
            {
                // Final scaling y = ((float(total) * 16) * u) * s_w and the store.  A thread owns a token's 128 outputs,
                // but a row-per-thread store would scatter 16-byte pieces over 32 rows: the warp transposes 32 x 32
                // pieces through shared memory (16-byte chunks XOR-swizzled by row, conflict-free both ways), after which
                // eight lanes write 128 contiguous bytes of a row and apply s_w, which is per column.
                // (total * 16) * u as ONE multiply by 16u: the factor 16 is exact on either side (u = R / 3825 with R a
                // finite float difference cannot overflow times 16), so the product is rounded once, from the same real
                const float ut16 = __fmul_rn(row_ok ? __ldg(prm.u + row) : 0.0f, 16.0f);
                const int jj = lane & 7, rsub = lane >> 3;
                // Shared-memory addresses of the transposition, kept in registers (opaque to the compiler, which would
                // otherwise rebuild each from the warp and lane indices -- a dozen integer instructions -- at every access):
                // this lane's row for the stores with its swizzle term, and for the loads row rsub with the term of
                // (row, 16-byte chunk jj); rows it8*4 + rsub differ from it by 512 bytes per step and, in the swizzle, by
                // the bit of it8's parity.
                uint32_t st_addr = smem_u32(stg) + (uint32_t) lane * 128u, st_x = (uint32_t) (lane & 7) << 4;
                uint32_t ld_addr = smem_u32(stg) + (uint32_t) rsub * 128u, ld_x = (uint32_t) (jj ^ rsub) << 4;
                asm volatile("" : "+r"(st_addr), "+r"(st_x), "+r"(ld_addr), "+r"(ld_x));
                const int wi = job_of_tile(prm, n_tile);
                const TcJob & jb = prm.job[wi];
                const int N = jb.N;
                const bool vec = jb.vec != 0, sw_vec = (reinterpret_cast<uintptr_t>(jb.sw) & 15) == 0;
                // first of this lane's four columns of piece c (beyond N: nothing there to store)
                auto piece_col = [&](int c) -> int { return c * 32 + jj * 4 < HC ? (n_tile - prm.tile_start[wi]) * BN + half * HC + c * 32 + jj * 4 : N; };
                // float(total) without integer conversions (they run at a quarter of the FMA rate).  Without re-centrings it is what
                // the float holds beyond 12.5 * 2^20, one exact subtraction.  Otherwise the carry words come back into registers (before
                // the tile is reused), the digit byte becomes the mantissa of 2^23 + digit with one byte permute, both parts are made
                // floats by exact subtractions, and one fused multiply-add forms digit * 2^20 + low with the single round-to-nearest an
                // int -> float conversion of the total would make.  Every re-centring moved a digit that stood for digit - 4 units of
                // 2^20 and left 4 behind.  (The float itself is 12.5 * 2^20 plus the rest: the 12 goes into the digit's subtrahend.)
                const float dsub = 8388608.0f + (float) (4 * n_rec + 12);
                if (F8 && n_rec > 0) {
#pragma unroll
                    for (int i = 0; i < HC / 4; ++i) {
                        const uint32_t carry = carry_smem[i * 32];
                        uint32_t w[4];
                        unpack2(tf[F8 ? 2 * i : 0], w[0], w[1]);
                        unpack2(tf[F8 ? 2 * i + 1 : 0], w[2], w[3]);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const float df = __fsub_rn(__uint_as_float(prmt(carry, 0x4B000000u, 0x7650u | (uint32_t) k)), dsub);
                            w[k] = __float_as_uint(__fmaf_rn(df, 1048576.0f, __fsub_rn(__uint_as_float(w[k]), 524288.0f)));
                        }
                        tf[F8 ? 2 * i : 0] = pack2(w[0], w[1]);
                        tf[F8 ? 2 * i + 1 : 0] = pack2(w[2], w[3]);
                    }
                    __syncwarp();
                } else if (F8) {
#pragma unroll
                    for (int i = 0; i < HC / 2; ++i)
                        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(tf[F8 ? i : 0]) : "l"(pack2(0xCB480000u, 0xCB480000u)));      // -(12.5 * 2^20)
                }
                {
                // the row units of all column pieces, requested before anything else: one load latency per unit
                float sc[(HC + 31) / 32][4];
#pragma unroll
                for (int c = 0; c < (HC + 31) / 32; ++c) {
                    const int ncol = piece_col(c);
                    if (sw_vec && ncol + 3 < N) {
                        const float4 q = __ldg(reinterpret_cast<const float4 *>(jb.sw + ncol));
                        sc[c][0] = q.x; sc[c][1] = q.y; sc[c][2] = q.z; sc[c][3] = q.w;
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k) sc[c][k] = ncol + k < N ? __ldg(jb.sw + ncol + k) : 0.0f;
                    }
                }
#pragma unroll
                for (int c = 0; c < (HC + 31) / 32; ++c) {
#pragma unroll
                    for (int j = 0; j < 8 && c * 32 + j * 4 < HC; ++j) {
                        const int i = c * 32 + j * 4;
                        float f[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            float totalf;
                            if constexpr (F8) {
                                uint32_t w[2];
                                unpack2(tf[F8 ? (i + k) >> 1 : 0], w[0], w[1]);
                                totalf = __uint_as_float(w[k & 1]);
                            } else {
                                totalf = (float) tot[F8 ? 0 : i + k];
                            }
                            f[k] = __fmul_rn(totalf, ut16);
                        }
                        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                                     :: "r"(st_addr + (st_x ^ (uint32_t) (j << 4))), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
                    }
                    __syncwarp();
                    const int ncol = piece_col(c);
                    float * yrow = jb.y + (size_t) (m_tile * BM + quarter * 32 + rsub) * jb.ldy + ncol;      // row rsub; + 4 rows per step
#pragma unroll
                    for (int it8 = 0; it8 < 8; ++it8) {
                        const int grow = m_tile * BM + quarter * 32 + it8 * 4 + rsub;
                        float4 q;       // row it8*4 + rsub, chunk jj ^ (row & 7) = jj ^ rsub ^ 4*(it8 & 1)
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w)
                                     : "r"(ld_addr + (uint32_t) (it8 * 512) + (ld_x ^ (uint32_t) ((it8 & 1) << 6))) : "memory");
                        const float o0 = __fmul_rn(q.x, sc[c][0]), o1 = __fmul_rn(q.y, sc[c][1]), o2 = __fmul_rn(q.z, sc[c][2]), o3 = __fmul_rn(q.w, sc[c][3]);
                        if (grow < prm.M) {
                            // this GPU's buffer; N-sharded ranks get their copies from warps 2 and 3
                            float * yr = yrow + (size_t) (it8 * 4) * jb.ldy;
                            if (vec && ncol + 3 < N) {
                                *reinterpret_cast<float4 *>(yr) = make_float4(o0, o1, o2, o3);
                            } else {
                                if (ncol < N) yr[0] = o0;
                                if (ncol + 1 < N) yr[1] = o1;
                                if (ncol + 2 < N) yr[2] = o2;
                                if (ncol + 3 < N) yr[3] = o3;
                            }
                        }
                    }
                    __syncwarp();
                }
                }
            }
            if constexpr (PUSH) {
                // the unit is in this GPU's output: let the pushing warps see it
                __threadfence();
                __syncwarp();
                if (lane == 0) atomicAdd(&sh.units_stored, 1u);
            }
            RQ_CYC_END(c_fin);
        }
        RQ_CYC_END(c_epi);
        if (warp == 4 && lane == 0) { RQ_CYC_REPORT(prm.status, 0x45, c_tfull); RQ_CYC_REPORT(prm.status, 0x46, c_epi); RQ_CYC_REPORT(prm.status, 0x49, c_hold);
                                      RQ_CYC_REPORT(prm.status, 0x4a, c_rec); RQ_CYC_REPORT(prm.status, 0x4b, c_fin); RQ_CYC_REPORT(prm.status, 0x4c, c_tail); }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && sh.abort_flag && prm.status != nullptr) atomicExch(prm.status, 1);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

typedef CUresult (*encode_fn_t)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_fn_t get_encode() {
    // resolved once; the initialisation of a function-local static is thread-safe
    static const encode_fn_t fn = []() -> encode_fn_t {
        void * p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            return reinterpret_cast<encode_fn_t>(p);
        }
        return nullptr;
    }();
    return fn;
}

}  // namespace

int rq_encode_tmap_i8(void * tmap_out, const void * base, int64_t K, int64_t rows, int box_rows) {
    encode_fn_t fn = get_encode();
    if (fn == nullptr) return -1;
    alignas(64) CUtensorMap map;
    const cuuint64_t dims[2] = { (cuuint64_t) K, (cuuint64_t) rows };
    const cuuint64_t strides[1] = { (cuuint64_t) K };       // bytes between rows
    const cuuint32_t box[2] = { (cuuint32_t) BK, (cuuint32_t) box_rows };
    const cuuint32_t estr[2] = { 1, 1 };
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -1;
    memcpy(tmap_out, &map, sizeof(map));
    return 0;
}

// the int4 decode stream as rows of 16-row tiles (K * 8 bytes each), boxes of 8 tiles x 256 inputs (2 KB), not swizzled
int rq_encode_tmap_w4(void * tmap_out, const void * base, int64_t K, int64_t tiles) {
    encode_fn_t fn = get_encode();
    if (fn == nullptr) return -1;
    alignas(64) CUtensorMap map;
    const cuuint64_t dims[2] = { (cuuint64_t) K, (cuuint64_t) tiles };       // in 8-byte elements
    const cuuint64_t strides[1] = { (cuuint64_t) K * 8 };
    const cuuint32_t box[2] = { 256, 8 };
    const cuuint32_t estr[2] = { 1, 1 };
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return -1;
    memcpy(tmap_out, &map, sizeof(map));
    return 0;
}

template <bool F8, bool PUSH, int NQ>
static cudaError_t configure_tc() {
    return cudaFuncSetAttribute(rq_gemm_tc_kernel<F8, PUSH, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes_of(NQ));
}
template <bool F8>
static cudaError_t configure_tc_all() {
    cudaError_t e;
    if ((e = configure_tc<F8, true, 8>()) != cudaSuccess) return e;
    if ((e = configure_tc<F8, false, 8>()) != cudaSuccess) return e;
    if ((e = configure_tc<F8, false, 6>()) != cudaSuccess) return e;
    if ((e = configure_tc<F8, false, 5>()) != cudaSuccess) return e;
    return configure_tc<F8, false, 4>();
}

cudaError_t rq_configure_gemm_tc() {
    // fp8 operands (no weight multipliers) or int8
    const cudaError_t e = configure_tc_all<false>();
    return e != cudaSuccess ? e : configure_tc_all<true>();
}

struct TcMaps { alignas(64) CUtensorMap a, b[RQ_MAX_WEIGHTS]; };

template <bool F8, bool PUSH, int NQ>
static cudaError_t launch_tc(const TcMaps & t, const TcParams & prm, int workers, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) workers);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem_bytes_of(NQ);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    static const int pdl = getenv("RQ_NO_PDL") ? 0 : 1;      // read once
    attr[0].val.programmaticStreamSerializationAllowed = pdl;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, rq_gemm_tc_kernel<F8, PUSH, NQ>, t.a, t.b[0], t.b[1], t.b[2], prm);
}

template <bool F8>
static cudaError_t launch_tc_any(const TcMaps & t, const TcParams & prm, int nq, bool push, int workers, cudaStream_t stream) {
    if (push) return launch_tc<F8, true, 8>(t, prm, workers, stream);
    switch (nq) {
        case 4:  return launch_tc<F8, false, 4>(t, prm, workers, stream);
        case 5:  return launch_tc<F8, false, 5>(t, prm, workers, stream);
        case 6:  return launch_tc<F8, false, 6>(t, prm, workers, stream);
        default: return launch_tc<F8, false, 8>(t, prm, workers, stream);
    }
}

cudaError_t rq_launch_gemm_tc(const rq_gemm_job * jobs, int n_jobs, int fmt, int64_t K, const int8_t * a8, const int32_t * msh, const float * u,
                              int64_t M, int G, int32_t * status, cudaStream_t stream) {
    if (n_jobs < 1 || n_jobs > RQ_MAX_WEIGHTS) return cudaErrorInvalidValue;
    // first use on a device (normally rq_w4a4_prepare's, outside stream capture); several host threads may get here at once
    static std::mutex mu;
    static bool configured[64] = {};
    static int sm_count[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int sms;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!configured[dev]) {
            e = rq_configure_gemm_tc();
            if (e != cudaSuccess) return e;
            e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
            if (e != cudaSuccess) return e;
            configured[dev] = true;
        }
        sms = sm_count[dev] > 0 ? sm_count[dev] : 148;
    }
    const bool f8 = fmt == RQ_FMT_E4M3;
    const int m_tiles = (int) ((M + BM - 1) / BM);
    bool push = false;
    for (int i = 0; i < n_jobs; ++i) push = push || jobs[i].n_more > 0;
    if (push && n_jobs > 1) return cudaErrorInvalidValue;

    // Weight rows per tile: the widest tile costs least per row (the 128 x 64 token operand and every hand-over are shared by
    // more columns), but a launch takes whole rounds of one unit per SM, and one of 5120 rows and 512 tokens has 80 units of
    // 256 rows for 148 SMs.  The narrower tile is taken where it saves more rounds than its rounds are dearer per row.  Time of a
    // round with 256, 192, 160 and 128 rows, fp8 operands, the last of three full rounds, us: K = 4096 23.5, 20.0, 18.2, 16.3; 11264
    // 54, 46, 41, 38; 17408 84, 76, 62, 56; in groups of 256 11264 41, 33, 31, 28.  Integer operands in groups of 256: 11264 44, 34, 32,
    // 29, in about the same proportion; in groups of 64, where their fold of two instructions per sum weighs more, narrow tiles are
    // cheaper: 4096 37, 27, 25, 22; 11264 97, 68, 60, 55; 17408 159, 111, 97, 84.
    static const int rows_nq[4] = { 8, 6, 5, 4 }, cost[2][4] = { { 105, 75, 68, 54 }, { 82, 70, 64, 57 } };
    const bool even = f8 || G > 64;
    int nq = 8, units = 0;
    long best = 0;
    for (int c = 0; c < (push ? 1 : 4); ++c) {
        int tiles = 0;
        for (int i = 0; i < n_jobs; ++i) tiles += (int) ((jobs[i].N + 32 * rows_nq[c] - 1) / (32 * rows_nq[c]));
        const int n = tiles * m_tiles;
        const long time = (long) ((n + sms - 1) / sms) * cost[even][c];
        if (c == 0 || time < best) { best = time; nq = rows_nq[c]; units = n; }
    }

    TcMaps t;
    if (rq_encode_tmap_i8(&t.a, a8, K, M, BM) != 0) return cudaErrorInvalidValue;
    TcParams prm = {};
    prm.n_jobs = n_jobs;
    prm.msh = msh; prm.u = u; prm.status = status;
    prm.K = (int) K; prm.M = (int) M; prm.G = G;
    for (int i = 0; i < n_jobs; ++i) {
        TcJob & jb = prm.job[i];
        const rq_gemm_job & in = jobs[i];
        jb.sw = in.sw; jb.y = in.y; jb.ldy = in.ldy; jb.N = (int) in.N; jb.n_more = in.n_more;
        // 16-byte stores only when every destination allows them (a peer's buffer may be aligned differently from ours)
        bool vec = (in.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(in.y) & 15) == 0;
        for (int d = 0; d < in.n_more; ++d) {
            jb.y_more[d] = in.y_more[d];
            vec = vec && (reinterpret_cast<uintptr_t>(in.y_more[d]) & 15) == 0;
        }
        jb.vec = vec ? 1 : 0;
        prm.tile_start[i + 1] = prm.tile_start[i] + (int) ((in.N + 32 * nq - 1) / (32 * nq));
        // (the map made with the weight has boxes of half a tile of 256 rows)
        if (nq == 8) memcpy(&t.b[i], in.tmap_w8, sizeof(t.b[i]));
        else if (rq_encode_tmap_i8(&t.b[i], in.w8, K, in.N, 16 * nq) != 0) return cudaErrorInvalidValue;
    }
    for (int i = n_jobs; i < RQ_MAX_WEIGHTS; ++i) t.b[i] = t.b[0];
    const int workers = units < sms ? units : sms;           // one CTA per SM: the ring takes its whole shared memory
    return f8 ? launch_tc_any<true>(t, prm, nq, push, workers, stream) : launch_tc_any<false>(t, prm, nq, push, workers, stream);
}
