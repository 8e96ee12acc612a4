// Weight quantizer on the GPU: rows of fp32 -> rows of 144-byte W4A4 / W4A4H blocks, bit-identical to the reference's
// CPU quantizer (quantize_row_w4a4_ref / quantize_row_w4a4h_ref, rq_quantize_row_w, rq_scale_search, rq_pack in
// patches/llama.cpp-ruquant.patch:2489-2580, 2681-2710 of the reference).  Not on the MUL_MAT path: it makes the
// path's input (model conversion, test and benchmark tensors) without the CPU's 0.5 ms per row.
//
// Bit-parity contract
//   scale search  per row (or per block of 256 / per 64 inputs with weight groups): amax = max |x|; thirteen candidates
//                 s_r = (amax * (1.0f - 0.025f * r)) / 7.0f; for each, err_r = sum over the inputs IN ORDER, in double, of
//                 e*e with e = (double)(q*s) - (double)x, q = clamp(rintf(x / s), -8, 7); the first smallest err wins.
//                 The sum's order is part of the result (it decides which candidate wins a near-tie).
//                 The multiply and the add of err += e*e are separate roundings (the reference is built without fused
//                 multiply-add contraction on its baseline x86-64 target).
//   weight groups smax = max of the group scales, v = smax / 15, k_g = clamp(rintf(s_g / v), 1, 15), codes with k_g * v;
//                 header d = v, sum = 1<<30 | k_b (per block) or 3<<29 | k0 | k1<<4 | k2<<8 | k3<<12 (per 64 inputs).
//   no groups     header d = s, sum = the row's code sum.
//   pad[0] = row length K (W4A4) or Hadamard length n (W4A4H), pad[1] = 0 (activation clip unset).
// W4A4H rows are rotated first by the activation path's own rotation kernel (same operations, same order).
#include <math.h>

#include "rq_common.cuh"
#include "rq_act_dev.cuh"

namespace {

constexpr int CAND = 13;

__device__ __forceinline__ float candidate_scale(float amax, int r) {
    return __fdiv_rn(__fmul_rn(amax, __fsub_rn(1.0f, __fmul_rn(0.025f, (float) r))), 7.0f);
}
__device__ __forceinline__ float code_of(float x, float s) {
    return fminf(fmaxf(rintf(__fdiv_rn(x, s)), -8.0f), 7.0f);
}

// rint(x / s) as the reference rounds it, from t = x * inv with inv = 1 / s rounded: t is within 2e-6 of the rounded quotient
// (|x / s| <= 10.01), so the two round to the same code unless t is that close to a half -- then the division decides.
__device__ __forceinline__ float code_near(float x, float s, float inv) {
    constexpr float MAGIC = 12582912.0f;          // 1.5 * 2^23: the sum rounds t to the nearest even integer
    const float t = __fmul_rn(x, inv);
    const float r = __fsub_rn(__fadd_rn(t, MAGIC), MAGIC);
    // (an infinite or NaN t fails the comparison as well)
    if (fabsf(__fsub_rn(t, r)) < 0.49999f) return fminf(fmaxf(r, -8.0f), 7.0f);
    return code_of(x, s);
}

// Weight groups: one half-warp per (row, group): lanes 0..12 each walk the group's inputs for one candidate; lanes of a
// half-warp read the same address (a broadcast), consecutive iterations the next float of the same 32-byte sector.
// sg[row * ng + g] receives the winning scale (0 for an all-zero group).
// e = q*s - x is exact in fp32: with s in [2^E, 2^(E+1)) both terms are multiples of 2^(E-24) and |e| <= s/2 when |q| = 1,
// multiples of 2^(E-23) with |e| < 1.01 * s/2 when |q| > 1, multiples of 2^(E-21) with |e| < 3.01 s beyond the last code, and
// q = 0 gives -x: never more than 24 bits.  Its square is exact in double, so one fused multiply-add rounds as the
// reference's separate multiply and add do.
__global__ void __launch_bounds__(256) rq_wsearch_kernel(const float * __restrict__ x, int64_t ldx, int64_t n_rows, int K, int gs,
                                                         float * __restrict__ sg) {
    const int ng = K / gs;
    const int64_t unit = ((int64_t) blockIdx.x * blockDim.x + threadIdx.x) >> 4;     // (row, group) index
    const int r = threadIdx.x & 15;
    const bool live = unit < n_rows * ng;
    const int64_t row = live ? unit / ng : 0;
    const int g = live ? (int) (unit - row * ng) : 0;
    const float * xg = x + row * ldx + (int64_t) g * gs;

    // amax: every lane of the half-warp takes a stride-16 share, then a max over the 16 lanes (exact in any order)
    float amax = 0.0f;
    for (int i = r; i < gs; i += 16) amax = fmaxf(amax, fabsf(__ldg(xg + i)));
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));

    double err = INFINITY;
    float s = 0.0f;
    if (amax > 0.0f && r < CAND) {
        s = candidate_scale(amax, r);
        const float inv = __fdiv_rn(1.0f, s);
        err = 0.0;
        for (int i = 0; i < gs; i += 4) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(xg + i));
            const float v[4] = { q.x, q.y, q.z, q.w };
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double e = (double) __fsub_rn(__fmul_rn(code_near(v[k], s, inv), s), v[k]);
                err = __fma_rn(e, e, err);
            }
        }
    }
    // the first smallest error: walk the candidates in order, as the reference's loop does
    double best_err = INFINITY;
    float best_s = 0.0f;
    const int base = (threadIdx.x & 31) & 16;
    for (int c = 0; c < CAND; ++c) {
        const double ec = __shfl_sync(0xffffffffu, err, base + c);
        const float sc = __shfl_sync(0xffffffffu, s, base + c);
        if (ec < best_err) { best_err = ec; best_s = sc; }
    }
    if (live && r == 0) sg[unit] = amax > 0.0f ? best_s : 0.0f;
}

// packed pairs of floats: one instruction for two values
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float & lo, float & hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }

// One scale per row: a CTA holds the row in shared memory, finds the scale, packs the codes.
//
// The reference's 13 error sums are sequential double sums, but all that is used of them is which is the smallest.  So the
// sums are formed first in fp32, in parallel: A_r = sum d^2, d = t - clamp(rint(t)), t = x * (1 / s_r).  Bounds, in units of
// s_r: d differs from the reference's (q s - x) / s by at most 2.9e-6 (t from x / s: 1.2e-6 for |x / s| <= 10, the
// reference's rounded quotient: 6e-7, the distance to the nearest code counts twice; its rounded product q s: 4.8e-7), so the
// norms sqrt(sum) differ by at most ETA * sqrt(K) with ETA = 4e-6; the fp32 sum of K / 256 terms a lane and 10 levels of tree
// adds a relative (K / 256 + 10) * 2^-24 at most, half of that in the norm.  Candidates whose interval
// s_r * (sqrt(A_r) +- bound) reaches below the smallest upper end are summed again exactly as the reference sums them; mostly
// that is one and nothing is left to do.  Rows outside the range of the bounds (NaN, infinity, 2^+-40) take the exact sums of
// all 13.
// Bound by issue: per input and candidate five packed half instructions and two clamps.  Converting 17408 rows of 5120 (the
// rotation included) takes 405 us; 2267 with a thread per (row, candidate) that walked the sequential sum (a division, two
// conversions and three double operations per input) and a second pass that read the rows again to pack them.
constexpr int WROW_THREADS = 128, EXACT_CHUNK = 64;
__global__ void __launch_bounds__(WROW_THREADS) rq_wrow_kernel(const float * __restrict__ x, int64_t ldx, int K, int pad0, rq_block * __restrict__ out) {
    extern __shared__ __align__(16) float xs[];
    __shared__ double e2[CAND][EXACT_CHUNK];
    __shared__ float red[WROW_THREADS / 32][16], cand_s[16], cand_inv[16];
    __shared__ int red_i[WROW_THREADS / 32];
    __shared__ float win_s;
    __shared__ unsigned contested_s;
    __shared__ uint64_t row_bar;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t row = blockIdx.x;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((uint32_t) __cvta_generic_to_shared(&row_bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const float * xr = x + row * ldx;

    rq_act_dev::bulk_load_row(xs, xr, K, &row_bar, tid, WROW_THREADS, nullptr);      // (nowhere to report to: copied again if it does not land)

    float amax = 0.0f;
    for (int i = tid; i < K / 4; i += WROW_THREADS) {
        const float4 q = reinterpret_cast<const float4 *>(xs)[i];
        amax = fmaxf(fmaxf(fmaxf(amax, fabsf(q.x)), fmaxf(fabsf(q.y), fabsf(q.z))), fabsf(q.w));
    }
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) red[warp][0] = amax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < WROW_THREADS / 32; ++w) amax = fmaxf(amax, red[w][0]);
    __syncthreads();

    float s = 0.0f;
    if (amax > 0.0f) {
        if (tid < 16) {
            const float c = candidate_scale(amax, tid < CAND ? tid : 0);
            cand_s[tid] = c;
            cand_inv[tid] = __fdiv_rn(1.0f, c);
        }
        __syncthreads();
        unsigned contested = (1u << CAND) - 1u;
        if (amax > 9.0e-13f && amax < 1.0e12f) {
            uint64_t acc[CAND];
            float inv[CAND];
#pragma unroll
            for (int c = 0; c < CAND; ++c) { acc[c] = 0; inv[c] = cand_inv[c]; }
            const uint64_t magic = pack2(12582912.0f, 12582912.0f), unmagic = pack2(-12582912.0f, -12582912.0f), minus1 = pack2(-1.0f, -1.0f);
            for (int i = tid; i < K / 4; i += WROW_THREADS) {
                const float4 q = reinterpret_cast<const float4 *>(xs)[i];
                const uint64_t v[2] = { pack2(q.x, q.y), pack2(q.z, q.w) };
#pragma unroll
                for (int c = 0; c < CAND; ++c) {
                    const uint64_t inv2 = pack2(inv[c], inv[c]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint64_t t = mul2(v[h], inv2);
                        float r0, r1;
                        unpack2(add2(add2(t, magic), unmagic), r0, r1);
                        const uint64_t d = fma2(pack2(fminf(fmaxf(r0, -8.0f), 7.0f), fminf(fmaxf(r1, -8.0f), 7.0f)), minus1, t);
                        acc[c] = fma2(d, d, acc[c]);
                    }
                }
            }
            // 16 sums over 32 lanes: every step halves the number of sums a lane carries
            float a[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                float lo = 0.0f, hi = 0.0f;
                if (c < CAND) unpack2(acc[c < CAND ? c : 0], lo, hi);
                a[c] = __fadd_rn(lo, hi);
            }
#pragma unroll
            for (int n = 8, o = 16; n > 0; n >>= 1, o >>= 1) {
                const bool upper = (lane & o) != 0;
#pragma unroll
                for (int c = 0; c < n; ++c) {
                    const float give = upper ? a[c] : a[c + n], keep = upper ? a[c + n] : a[c];
                    a[c] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, o));
                }
            }
            a[0] = __fadd_rn(a[0], __shfl_xor_sync(0xffffffffu, a[0], 1));
            if ((lane & 1) == 0) red[warp][lane >> 1] = a[0];      // lane bits 4..1 are the bits of the sum's index, high to low
            __syncthreads();
            if (warp == 0) {
                float lo = INFINITY, hi = INFINITY;
                bool sane = true;
                if (lane < CAND) {
                    float sum = 0.0f;
#pragma unroll
                    for (int w = 0; w < WROW_THREADS / 32; ++w) sum = __fadd_rn(sum, red[w][lane]);
                    const float norm = __fsqrt_rn(sum), rel = (float) (K / 256 + 16) * 6.0e-8f, eta = 4.0e-6f * __fsqrt_rn((float) K);
                    lo = cand_s[lane] * (norm - norm * rel - eta);
                    hi = cand_s[lane] * (norm + norm * rel + eta);
                    sane = hi < INFINITY;             // (a NaN among the inputs)
                }
                float least = hi;
                for (int o = 16; o > 0; o >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
                const unsigned mask = __ballot_sync(0xffffffffu, lane < CAND && lo <= least);
                const bool all_sane = __all_sync(0xffffffffu, sane);
                if (lane == 0) contested_s = all_sane ? mask : (1u << CAND) - 1u;
            }
            __syncthreads();
            contested = contested_s;
        }
        if ((contested & (contested - 1u)) != 0u) {
            // the reference's own sums for the contested candidates: the squares of a chunk in parallel, then a lane per candidate
            // adds them in order
            double err = lane < CAND && ((contested >> lane) & 1u) ? 0.0 : (double) INFINITY;
            for (int i0 = 0; i0 < K; i0 += EXACT_CHUNK) {
                for (int k = tid; k < CAND * EXACT_CHUNK; k += WROW_THREADS) {
                    const int c = k / EXACT_CHUNK, i = k % EXACT_CHUNK;
                    if ((contested >> c) & 1u) {
                        const float v = xs[i0 + i], sc = cand_s[c];
                        const double e = __dsub_rn((double) __fmul_rn(code_of(v, sc), sc), (double) v);
                        e2[c][i] = __dmul_rn(e, e);
                    }
                }
                __syncthreads();
                if (warp == 0 && lane < CAND && ((contested >> lane) & 1u)) {
#pragma unroll 16
                    for (int i = 0; i < EXACT_CHUNK; ++i) err = __dadd_rn(err, e2[lane][i]);
                }
                __syncthreads();
            }
            if (warp == 0) {      // the first smallest error, as the reference's loop finds it
                double best_err = INFINITY;
                float best_s = 0.0f;
                for (int c = 0; c < CAND; ++c) {
                    const double ec = __shfl_sync(0xffffffffu, err, c);
                    if (ec < best_err) { best_err = ec; best_s = cand_s[c]; }
                }
                if (lane == 0) win_s = best_s;
            }
        } else if (tid == 0) {
            win_s = cand_s[__ffs(contested) - 1];
        }
        __syncthreads();
        s = win_s;
    }

    // codes: a thread packs whole words of 8
    rq_block * yr = out + row * (K / RQ_BLOCK_CODES);
    const float inv = s > 0.0f ? __fdiv_rn(1.0f, s) : 0.0f;
    int code_sum = 0;
    for (int w = tid; w < K / 8; w += WROW_THREADS) {
        const float4 a = reinterpret_cast<const float4 *>(xs)[2 * w], b = reinterpret_cast<const float4 *>(xs)[2 * w + 1];
        const float v[8] = { a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w };
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = s > 0.0f ? (int) code_near(v[j], s, inv) : 0;
            code_sum += c;
            word |= (uint32_t) (c & 0xF) << (4 * j);
        }
        yr[w >> 5].qs[w & 31] = word;
    }
    for (int o = 16; o > 0; o >>= 1) code_sum += __shfl_xor_sync(0xffffffffu, code_sum, o);
    if (lane == 0) red_i[warp] = code_sum;
    __syncthreads();
    int row_sum = 0;
#pragma unroll
    for (int w = 0; w < WROW_THREADS / 32; ++w) row_sum += red_i[w];
    for (int b = tid; b < K / RQ_BLOCK_CODES; b += WROW_THREADS) {
        yr[b].d = s;
        yr[b].sum = row_sum;
        yr[b].pad[0] = pad0;
        yr[b].pad[1] = 0;
    }
}

// Weight groups, one CTA per row: group multipliers, codes, headers.
__global__ void __launch_bounds__(256) rq_wpack_kernel(const float * __restrict__ x, int64_t ldx, int K, int gs, int pad0,
                                                       const float * __restrict__ sg, rq_block * __restrict__ out) {
    __shared__ float red[8];
    __shared__ float unit_s;
    const int64_t row = blockIdx.x;
    const int tid = threadIdx.x, ng = K / gs;
    const float * xr = x + row * ldx;
    const float * sr = sg + row * ng;
    rq_block * yr = out + row * (K / RQ_BLOCK_CODES);

    float smax = 0.0f;
    for (int g = tid; g < ng; g += blockDim.x) smax = fmaxf(smax, sr[g]);
    for (int o = 16; o > 0; o >>= 1) smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    if ((tid & 31) == 0) red[tid >> 5] = smax;
    __syncthreads();
    if (tid == 0) {
        float v = 0.0f;
        for (int i = 0; i < (int) (blockDim.x >> 5); ++i) v = fmaxf(v, red[i]);
        unit_s = __fdiv_rn(v, 15.0f);
    }
    __syncthreads();
    const float unit = unit_s;
    auto mult = [&](int g) -> float { return unit > 0.0f ? fminf(fmaxf(rintf(__fdiv_rn(sr[g], unit)), 1.0f), 15.0f) : 1.0f; };
    // a thread packs whole words of 8 codes
    for (int w = tid; w < K / 8; w += blockDim.x) {
        const float s = __fmul_rn((float) (int) mult((w * 8) / gs), unit);
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = s > 0.0f ? (int) code_of(xr[w * 8 + j], s) : 0;
            word |= (uint32_t) (c & 0xF) << (4 * j);
        }
        yr[w >> 5].qs[w & 31] = word;
    }
    for (int b = tid; b < K / RQ_BLOCK_CODES; b += blockDim.x) {
        auto m = [&](int g) -> uint32_t { return (uint32_t) (int) mult(g); };
        yr[b].d = unit;
        yr[b].sum = gs == RQ_BLOCK_CODES ? (int32_t) (1u << 30 | m(b))
                                         : (int32_t) (3u << 29 | m(4 * b) | m(4 * b + 1) << 4 | m(4 * b + 2) << 8 | m(4 * b + 3) << 12);
        yr[b].pad[0] = pad0;
        yr[b].pad[1] = 0;
    }
}

}  // namespace

// x: [n_rows][K] fp32 rows ldx apart, already rotated for W4A4H.  wgroup: 0, 256 or 64.  sg: n_rows * (K / gs) floats
// of scratch (gs = K without weight groups).  pad0: what the headers' pad[0] records.
cudaError_t rq_launch_wquant(const float * x, int64_t ldx, int64_t n_rows, int64_t K, int wgroup, int pad0, float * sg,
                             rq_block * out, cudaStream_t stream) {
    if (wgroup == 0) {
        const size_t smem = (size_t) K * sizeof(float);
        if (smem > 40 * 1024) {       // beyond what a kernel may use unasked; a property of the current device's copy of the kernel
            const cudaError_t e = cudaFuncSetAttribute(rq_wrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RQ_MAX_K * (int) sizeof(float));
            if (e != cudaSuccess) return e;
        }
        rq_wrow_kernel<<<(unsigned) n_rows, WROW_THREADS, smem, stream>>>(x, ldx, (int) K, pad0, out);
        return cudaGetLastError();
    }
    const int64_t threads = n_rows * (K / wgroup) * 16;
    rq_wsearch_kernel<<<(unsigned) ((threads + 255) / 256), 256, 0, stream>>>(x, ldx, n_rows, (int) K, wgroup, sg);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    rq_wpack_kernel<<<(unsigned) n_rows, 256, 0, stream>>>(x, ldx, (int) K, wgroup, pad0, sg, out);
    return cudaGetLastError();
}
