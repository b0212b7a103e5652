// C[M,N] = A[M,K] * W[N,K]^T in bfloat16 on the 5th-generation tensor cores.
//
// tcgen05.mma (kind::f16; cta_group::1 with 128 x BN x 16 per instruction, and for most
// products of many tokens cta_group::2 with 256 x BN x 16 over a pair of SMs, see
// gemm_tc_pair_kernel) issued by one elected lane, operands staged in shared memory by TMA
// (128-byte swizzle, K-major), accumulators in tensor memory, read back with tcgen05.ld
// for the epilogue.
// The reference has no dense tensor-core product: its linears are 4-bit codebook
// GEMVs (runtime/cuda/codebook_gemv.cu:86-114) with a fixed-order second stage
// for determinism (:178-184); the same rule holds here (no atomics anywhere).
//
// Two orientations:
//   tokens >  128: the 128 lanes of a tile are tokens, its BN columns weight rows; single SMs, pairs of SMs or a cluster
//                  that cuts a tile's K, and the tile's width, by the least of the fitted costs in choose_form
//   tokens <= 128: swapped, the 128 lanes are weight rows and the BN columns are the
//                  tokens (BN = 16..128), so a decode step streams every weight
//                  once through full-height MMA tiles whatever the batch size
// and optional split-K (small N, large K): each split writes 32-bit partials to
// scratch and tb_splitk_reduce adds them in split order.
//
// Roles per CTA (320 threads): warp 0 issues TMA loads, warp 1 owns tensor memory
// and issues the MMAs, warps 2..9 are the epilogue (a warp reads the 32 lanes of
// tensor memory that its index modulo 4 selects; the two warps of a quarter take
// the chunks of columns in turn).  The kernel is persistent: a
// CTA walks its share of the work items; two accumulator stages let the epilogue
// of one item overlap the MMAs of the next.
//
// Every wait on an mbarrier is bounded.  A wait that runs out records a code in
// the error word, and all roles leave their loops, wait (bounded) for TMA loads
// still in flight, free the tensor memory and return.  tb_gemm_tc_error() reads
// and clears the word.
//
// Sizes: K must be a multiple of 8 elements and A, W 16-byte aligned (TMA strides);
// anything else is refused and the caller falls back to the FMA kernel.
#include "common.cuh"
#include "tcgen05.cuh"
#include <stdlib.h>

TB_EXPORT_ERROR()

#define BM 128
#define BK 64
#define EPI_WARPS 8                      // two warps for each quarter of the tensor memory's lanes
#define GEMM_THREADS (64 + 32 * EPI_WARPS)

__device__ int g_gemm_error = 0;

// ---------------------------------------------------------------------------
struct GemmParams {
    int rows_p, rows_q, K;           // P: the 128-lane operand, Q: the BN-column operand
    int tiles_p, tiles_q, splits, kb_per_split, kblocks;
    void* out; long long ld_out;     // C as [tokens, weight rows], row stride ld_out
    float* partial;                  // [splits][tokens][weight rows] when splits > 1
    float cap;
    float scale;                     // the output times this (1 for a plain product); after the cap, never with it
    int act;                         // gated epilogue: 0 gelu_tanh, 1 silu, 2 clamped_swish (only with GATED kernels)
    float limit;                     // clamped_swish: both branches are bounded by it
    int unary;                       // plain epilogues: 0 nothing, 1 every output becomes relu(v)^2, 2 v Phi(v) (never on partial sums)
    // Grouped products: a tile of tokens (128 rows, or the BN of swapped tiles) multiplies the weight rows of its group
    // tile_group[tile], which start at row tile_group[tile] * group_rows of the weight operand; a negative entry: the tile
    // is not in use and nobody touches it.
    const int* tile_group;
    int group_rows;
    int staged;                      // the rows of C are made of whole 16-byte pieces: chunks of 32 columns are stored through shared memory
    int cluster;                     // gemm_tc_split_kernel: CTAs that share a tile's K
    const float* row_scale;          // grouped products: the sums of token row r times row_scale[r], before the activation; or null
};

// Gated epilogue.  The weight rows are interleaved in blocks of 16: [gate 0..15 | up 0..15 | gate 16..31 | ...],
// so that a gate and its up value always meet in one epilogue thread (token-major tiles: columns j and j + 16
// of a 32-column chunk) or in one warp (swapped tiles: lanes l and l + 16).  The output has half the width:
// out[token][16 b + j] = act(gate) * up, computed on the 32-bit accumulators
// (the reference's gelu_mul_k does this as a kernel of its own, runtime/cuda/codebook_gemv.cu:531-537).
// The result is rounded to bfloat16, so tanh and the logistic function are taken through the fast exponential
// and division (relative error near 2^-21): 0.5 (1 + tanh(y)) = 1 / (1 + e^(-2y)).
// clamped_swish: g' = min(g, L), u' = clamp(u, -L, L), g' / (1 + e^(-1.702 g')) * (u' + 1).
// That error grows with the gate, to 2^-19 at -30, and below -87.3, where the divisor passes 2^126, the quotient is 0.  Act 3
// (EXACT, the grouped products of experts): silu by expf and a true quotient, the function of the experts' other kernels.
template <bool EXACT>
__device__ __forceinline__ float gated(float g, float u, int act, float limit) {
    if (EXACT && act == 3) return g / (1.0f + expf(-g)) * u;
    if (act == 2) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit) + 1.0f;
    }
    const float y = act == 0 ? 1.5957691216f * (g + 0.044715f * g * g * g) : (act == 2 ? 1.702f * g : g);     // 2 sqrt(2/pi) (g + 0.044715 g^3)
    return __fdividef(g, 1.0f + __expf(-y)) * u;
}

// Shared-memory budget.  Many tokens (tiles are reused, the tensor cores are the limit): as many stages as an SM
// holds.  Few tokens (swapped tiles, a stream of weights) and a short stream: half of an SM, so that the next
// product's CTAs already sit beside this one's, fetch their tensor maps and fill their stages with weights while this
// one drains; the two kernels together keep as many bytes in flight as one with the whole SM.  A long stream (WIDE:
// the host asks for it from TB_WIDE_FROM_BYTES of weights on) takes the whole SM: its own bytes in flight count for
// more than the overlap with its neighbours.  Measured, decode steps at context 2,048 with every small product on
// the whole SM against half: 2B shape 2.5 % slower at batch 8, 9B shape 2 % faster, 27B shape 5 % faster; with 32 to
// 128 tokens the whole SM is never slower (9B shape at batch 64: 4 % faster).
#ifndef TB_SWAP_KB
#define TB_SWAP_KB 108
#endif
#ifndef TB_WIDE_FROM_BYTES
#define TB_WIDE_FROM_BYTES (128 << 20)
#endif
#ifndef TB_SWAP_HALF_UPTO
#define TB_SWAP_HALF_UPTO 16
#endif
#define EPI_STAGE_BYTES (32 * 128)       // an epilogue warp's 32 rows of a 32-column chunk, on their way through shared memory
template <int BN, bool SWAP, bool WIDE = false> struct Cfg {
    static constexpr int STAGE_BYTES = BM * BK * 2 + BN * BK * 2;
    static constexpr int BUDGET = (!SWAP ? 192 : (!WIDE && BN <= TB_SWAP_HALF_UPTO) ? TB_SWAP_KB : 200) * 1024;
    static constexpr int STAGES_RAW = BUDGET / STAGE_BYTES;
    static constexpr int STAGES = STAGES_RAW > 10 ? 10 : STAGES_RAW;
    static constexpr int ACC_COLS = BN < 32 ? 32 : BN <= 128 ? BN : 256;       // columns of one accumulator stage
    static constexpr int TMEM_COLS = 2 * ACC_COLS;                   // a power of two >= 32
    static constexpr int EPI = SWAP ? 0 : EPI_WARPS * EPI_STAGE_BYTES;
    static constexpr int EPI_OFF = STAGES * STAGE_BYTES + 256 /* barriers */;
    static constexpr int SMEM = EPI_OFF + EPI + 1024 /* alignment */;
};

// The exact gelu, v Phi(v), for an output that is rounded to bfloat16.  The tail Q(t) = 1 - Phi(t), t = |v|, is half of
// erfc(t / sqrt 2), which formula 7.1.26 of Abramowitz and Stegun, Handbook of Mathematical Functions, gives as a
// polynomial in 1 / (1 + p t / sqrt 2) times e^(-t^2 / 2) (error at most 1.5e-7).
__device__ __forceinline__ float gelu_exact(float v) {
    const float x = fabsf(v) * 0.70710678f;
    const float k = __fdividef(1.0f, fmaf(0.3275911f, x, 1.0f));
    float q = fmaf(1.061405429f, k, -1.453152027f);
    q = fmaf(q, k, 1.421413741f);
    q = fmaf(q, k, -0.284496736f);
    q = fmaf(q, k, 0.254829592f);
    q = 0.5f * q * k * __expf(-x * x);
    return v * (v < 0.f ? q : 1.0f - q);
}

// Epilogue of token-major tiles: the thread holds CH consecutive columns (weight rows q0 .. q0 + CH - 1) of token prow.
// What a plain epilogue does to one output before the scale: the cap, then the unary activation.
__device__ __forceinline__ float pointwise(float v, const GemmParams& p) {
    if (p.cap > 0.f) v = softcap_f(v, p.cap);
    if (p.unary == 1) { v = fmaxf(v, 0.f); v *= v; }
    else if (p.unary == 2) v = gelu_exact(v);
    return v;
}

template <typename TOut, bool GATED, int CH, bool EXACT = false>
__device__ __forceinline__ void store_token_major(const uint32_t* r, int prow, int q0, int sp, const GemmParams& p) {
    static_assert(!GATED || CH == 32, "a gate and its up value lie 16 columns apart");
    if (GATED) {
        // 32 columns = 16 gates then their 16 ups: 16 outputs at column q0 / 2
        if (prow < p.rows_p && q0 < p.rows_q) {
            bf16* dst = (bf16*)p.out + (size_t)prow * p.ld_out + (q0 >> 1);
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                const float v0 = gated<EXACT>(__uint_as_float(r[j]), __uint_as_float(r[j + 16]), p.act, p.limit);
                const float v1 = gated<EXACT>(__uint_as_float(r[j + 1]), __uint_as_float(r[j + 17]), p.act, p.limit);
                __nv_bfloat162 h2 = __floats2bfloat162_rn(v0, v1);
                w[j >> 1] = *(uint32_t*)&h2;
            }
            if ((((uintptr_t)dst) & 15) == 0) {
                *(uint4*)dst = make_uint4(w[0], w[1], w[2], w[3]);
                *(uint4*)(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) *(uint32_t*)(dst + 2 * j) = w[j];
            }
        }
    } else {
        // tokens on lanes (prow), weight rows on columns (q0 + j): a thread writes a row segment
        if (prow < p.rows_p) {
            if (p.splits > 1) {
                float* dst = p.partial + ((size_t)sp * p.rows_p + prow) * p.rows_q + q0;
#pragma unroll
                for (int j = 0; j < CH; j++) if (q0 + j < p.rows_q) dst[j] = __uint_as_float(r[j]);
            } else {
                TOut* dst = (TOut*)p.out + (size_t)prow * p.ld_out + q0;
                const bool vec = (q0 + CH <= p.rows_q) && ((((uintptr_t)dst) & 15) == 0);
                if (vec && sizeof(TOut) == 2) {
#pragma unroll
                    for (int j = 0; j < CH; j += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            float v0 = __uint_as_float(r[j + 2 * e]), v1 = __uint_as_float(r[j + 2 * e + 1]);
                            v0 = pointwise(v0, p); v1 = pointwise(v1, p);
                            v0 *= p.scale; v1 *= p.scale;
                            __nv_bfloat162 h2 = __floats2bfloat162_rn(v0, v1);
                            w[e] = *(uint32_t*)&h2;
                        }
                        *(uint4*)((bf16*)dst + j) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                } else if (vec) {
#pragma unroll
                    for (int j = 0; j < CH; j += 4) {
                        float4 v = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                               __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
                        v.x = pointwise(v.x, p); v.y = pointwise(v.y, p); v.z = pointwise(v.z, p); v.w = pointwise(v.w, p);
                        v.x *= p.scale; v.y *= p.scale; v.z *= p.scale; v.w *= p.scale;
                        *(float4*)((float*)dst + j) = v;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < CH; j++) if (q0 + j < p.rows_q) {
                        float v = __uint_as_float(r[j]);
                        v = pointwise(v, p);
                        dst[j] = from_f<TOut>(v * p.scale);
                    }
                }
            }
        }
    }
}


// The same 32 columns of a warp's 32 rows, rows of whole 16-byte pieces, through 4 KB of shared memory: a row's piece of a
// chunk then leaves as whole sectors, 8 (float), 4 or 2 lanes side by side.  Written by the thread that holds the row, 16
// bytes a lane, every store touches 32 lines and the SM takes a line a cycle: a tile of 128 x 256 floats took 11.9 us so,
// 3.3 this way (the product of 2,048 tokens x 2,304 x 2,048: 25.7 -> 18.2 us).  Pieces are swizzled against bank conflicts.
template <typename TOut, bool GATED, bool EXACT = false>
__device__ __forceinline__ void store_staged(const uint32_t* r, uint8_t* stage, int lane, int row0, int q0, const GemmParams& p) {
    constexpr int RB = GATED ? 32 : 32 * (int)sizeof(TOut), U = RB / 16;
    auto f = [](int row) { return U == 8 ? row & 7 : U == 4 ? (row >> 1) & 3 : (row >> 2) & 1; };
#pragma unroll
    for (int u = 0; u < U; u++) {
        uint32_t w[4];
        if (GATED) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int j = u * 8 + e * 2;
                __nv_bfloat162 h2 = __floats2bfloat162_rn(gated<EXACT>(__uint_as_float(r[j]), __uint_as_float(r[j + 16]), p.act, p.limit),
                                                          gated<EXACT>(__uint_as_float(r[j + 1]), __uint_as_float(r[j + 17]), p.act, p.limit));
                w[e] = *(uint32_t*)&h2;
            }
        } else if (sizeof(TOut) == 2) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int j = u * 8 + e * 2;
                __nv_bfloat162 h2 = __floats2bfloat162_rn(pointwise(__uint_as_float(r[j]), p) * p.scale, pointwise(__uint_as_float(r[j + 1]), p) * p.scale);
                w[e] = *(uint32_t*)&h2;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) w[e] = __float_as_uint(pointwise(__uint_as_float(r[u * 4 + e]), p) * p.scale);
        }
        *(uint4*)(stage + lane * RB + ((u ^ f(lane)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    __syncwarp();
    const int c0 = GATED ? q0 >> 1 : q0;
#pragma unroll
    for (int i = 0; i < U; i++) {
        const int idx = i * 32 + lane, row = idx / U, u = idx % U;
        const uint4 v = *(const uint4*)(stage + row * RB + ((u ^ f(row)) << 4));
        if (row0 + row < p.rows_p)
            *(uint4*)((uint8_t*)p.out + ((size_t)(row0 + row) * p.ld_out + c0) * sizeof(TOut) + u * 16) = v;
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// The two warps that feed a product (one issues the copies, one the MMAs) run a short loop per k-block, and a chain of
// dependent instructions in it is paid per k-block whatever the tile.  With one thread of a diverged warp, a stage index
// modulo the number of stages, 64-bit descriptors made per MMA and a look at the abort flag, an SM spent 620 cycles a
// k-block for tiles 128, 192 and 256 columns wide alike, although the MMAs need 256 to 512; with 32-bit addresses, a
// counted stage and stepped descriptors 547; with the whole warp in the loop and one elected lane issuing 414, 430 and
// 512 (a pair of SMs at 256 x 256: 576 before, 512 now, which is the MMAs' own time).
// ---------------------------------------------------------------------------
struct Ring {                            // the stage that comes next, and the phase of its barriers
    uint32_t s = 0, ph = 0;
    template <int STAGES> __device__ __forceinline__ void step() { if (++s == STAGES) { s = 0; ph ^= 1; } }
};
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tile_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// The same for data that a step reads once, the first to leave L2: the weights.  A decode step streams more of them than L2
// holds (2B shape: 156 MB a layer), and what went with them were the small kernels between the products: their
// instructions, the partial sums, keys and values.  Step of one sequence, 2B shape: 1,585 -> 1,450 us.  With many tokens
// several CTAs read a weight tile, but at about the same time (tiles of tokens are the inner index of a launch's order), and
// what the next launches read again is tokens.
__device__ __forceinline__ uint64_t once_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void tile_load_once(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "l"(policy) : "memory");
}
__device__ __forceinline__ void tile_load_pair_once(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int c0, int c1, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(dst), "l"((uint64_t)map), "r"(cluster_bar), "r"(c0), "r"(c1), "l"(policy) : "memory");
}
__device__ __forceinline__ void tile_load_pair(uint32_t dst, const CUtensorMap* map, uint32_t cluster_bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(cluster_bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void commit_to_pair(uint32_t bar) {
    asm volatile("{\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\t"
                 "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair_lh(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t ab_hi, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 ad, bd;\n\t"
        "mov.b64 ad, {%1, %3};\n\t"
        "mov.b64 bd, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], ad, bd, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(ab_hi), "r"(idesc), "r"(acc) : "memory");
}
// One k-block: BK / 16 MMAs from the stage whose A starts at a_lo (low half of its descriptor), then the commit that frees it.
template <bool PAIR>
__device__ __forceinline__ void issue_kblock(uint32_t d_addr, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t acc, uint32_t empty) {
#pragma unroll
    for (int k = 0; k < BK / UMMA_K; k++) {
        const uint32_t step = k * (UMMA_K * 2 / 16);
        if (PAIR) umma_bf16_pair_lh(d_addr, a_lo + step, b_lo + step, hi, idesc, k ? 1u : acc);
        else umma_bf16_lh(d_addr, a_lo + step, b_lo + step, hi, idesc, k ? 1u : acc);
    }
    if (PAIR) commit_to_pair(empty); else commit_to(empty);
}

// GROUPED: see GemmParams::tile_group.
template <int BN, bool SWAP, typename TOut, bool GATED, bool WIDE, bool GROUPED>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q, GemmParams p) {
    pdl_launch_dependents();
    using C = Cfg<BN, SWAP, WIDE>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE_BYTES);
    uint64_t* full = bars;                       // [STAGES]
    uint64_t* empty = bars + C::STAGES;          // [STAGES]
    uint64_t* acc_full = bars + 2 * C::STAGES;   // [2]
    uint64_t* acc_empty = acc_full + 2;          // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 32) { tma_prefetch_map(&map_p); tma_prefetch_map(&map_q); }
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], EPI_WARPS); }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int n_items = p.tiles_p * p.tiles_q * p.splits;
    // item -> (tile_q, tile_p, split): the tiles that share a Q tile (prefill: a weight
    // tile; swapped: the tokens) run side by side
    auto decode = [&](int item, int& tp, int& tq, int& sp) {
        sp = item % p.splits; item /= p.splits;
        tp = item % p.tiles_p; tq = item / p.tiles_p;
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        const uint32_t sm0 = smem_u32(smem), full0 = smem_u32(full), empty0 = smem_u32(empty);
        uint32_t it = 0;
        const uint64_t policy = once_policy();
        auto w_load = [&](uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
            tile_load_once(dst, map, bar, c0, c1, policy);
        };
        Ring ring;
        bool ok = true, waited = false;
        // the tile that holds weights: the 128-lane operand when swapped, else the BN-column one
        const CUtensorMap* wmap = SWAP ? &map_p : &map_q;
        const CUtensorMap* amap = SWAP ? &map_q : &map_p;
        constexpr int W_OFF = SWAP ? 0 : BM * BK * 2, A_OFF = SWAP ? BM * BK * 2 : 0;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            int tp, tq, sp; decode(item, tp, tq, sp);
            const int kb0 = sp * p.kb_per_split, kb1 = min(p.kblocks, kb0 + p.kb_per_split);
            int w_row = SWAP ? tp * BM : tq * BN;
            const int a_row = SWAP ? tq * BN : tp * BM;
            if constexpr (GROUPED) {
                // the table of groups is the preceding kernel's work: nothing is fetched before it is there
                if (!waited) { pdl_wait(); waited = true; }
                const int g = p.tile_group[SWAP ? tq : tp];
                if (g < 0) continue;               // a tile past the last one in use: all three roles leave it out
                w_row += g * p.group_rows;
            }
            int kb = kb0;
            if (!waited) {
                // Weights do not depend on the kernel before this one: start streaming them into the
                // (still empty) stages at once, and only then wait for that kernel, whose output is
                // the activation operand.
                const int pre = min(kb1 - kb0, C::STAGES);
                if (elected())
                    for (int j = 0; j < pre; j++) {
                        bar_expect(full0 + 8 * j, C::STAGE_BYTES);
                        w_load(sm0 + j * C::STAGE_BYTES + W_OFF, wmap, full0 + 8 * j, (kb0 + j) * BK, w_row);
                    }
                pdl_wait();
                waited = true;
                if (elected())
                    for (int j = 0; j < pre; j++)
                        tile_load(sm0 + j * C::STAGE_BYTES + A_OFF, amap, full0 + 8 * j, (kb0 + j) * BK, a_row);
                __syncwarp();
                it = pre; kb = kb0 + pre;
                ring.s = pre % C::STAGES; ring.ph = pre / C::STAGES;
            }
            for (; kb < kb1; kb++, it++) {
                if (!warp_wait(empty0 + 8 * ring.s, ring.ph ^ 1, abort_flag)) { ok = false; break; }
                const uint32_t st = sm0 + ring.s * C::STAGE_BYTES, bar = full0 + 8 * ring.s;
                if (elected()) {
                    bar_expect(bar, C::STAGE_BYTES);
                    w_load(st + W_OFF, wmap, bar, kb * BK, w_row);
                    tile_load(st + A_OFF, amap, bar, kb * BK, a_row);
                }
                ring.step<C::STAGES>();
            }
        }
        if (!ok && lane == 0) {
            if (!*abort_flag) { atomicExch(&g_gemm_error, 1); *abort_flag = 1; }
            // loads already issued still land in this CTA's shared memory: wait for them
            for (uint32_t back = 1; back <= (uint32_t)C::STAGES && back <= it; back++) {
                const uint32_t j = it - back;
                mbar_wait(&full[j % C::STAGES], (j / C::STAGES) & 1);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        constexpr uint32_t idesc = instr_desc(BN);
        const uint64_t desc0 = smem_desc(smem_u32(smem));
        const uint32_t lo0 = desc_lo(desc0), hi = desc_hi(desc0), full0 = smem_u32(full), empty0 = smem_u32(empty);
        const uint32_t acc_full0 = smem_u32(acc_full), acc_empty0 = smem_u32(acc_empty);
        uint32_t tile_it = 0;
        Ring ring;
        bool ok = true;
        if (GROUPED) pdl_wait();      // the table of groups is the preceding kernel's work
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            int tp, tq, sp; decode(item, tp, tq, sp);
            if (GROUPED && p.tile_group[SWAP ? tq : tp] < 0) continue;
            const int kb0 = sp * p.kb_per_split, kb1 = min(p.kblocks, kb0 + p.kb_per_split);
            const int a = tile_it & 1; const uint32_t aph = (tile_it >> 1) & 1;
            tile_it++;
            if (!warp_wait(acc_empty0 + 8 * a, aph ^ 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d_addr = tmem_base + a * C::ACC_COLS;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!warp_wait(full0 + 8 * ring.s, ring.ph, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a_lo = lo0 + ring.s * (C::STAGE_BYTES / 16);
                if (elected()) issue_kblock<false>(d_addr, a_lo, a_lo + BM * BK * 2 / 16, hi, idesc, kb > kb0, empty0 + 8 * ring.s);
                ring.step<C::STAGES>();
            }
            if (ok && elected()) commit_to(acc_full0 + 8 * a);     // the accumulator is complete
        }
        if (!ok && lane == 0 && !*abort_flag) { atomicExch(&g_gemm_error, 2); *abort_flag = 1; }
        __syncwarp();
    } else {
        // ---------------- epilogue: warps 2..9 ----------------
        const int quarter = warp & 3;                  // the TMEM lanes this warp may read
        const int turn = (warp - 2) >> 2;              // the two warps of a quarter take the chunks of columns in turn
        pdl_wait();                                    // the output may still be read by the kernel before
        uint32_t tile_it = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            int tp, tq, sp; decode(item, tp, tq, sp);
            if (GROUPED && p.tile_group[SWAP ? tq : tp] < 0) continue;
            const int a = tile_it & 1; const uint32_t aph = (tile_it >> 1) & 1;
            tile_it++;
            // the decision must be the same in every lane: tcgen05.ld is a warp-wide instruction
            const bool mine = !*abort_flag && mbar_wait(&acc_full[a], aph);
            if (!__all_sync(0xffffffffu, mine)) { ok = false; break; }
            tc_fence_after();
            const int prow = tp * BM + quarter * 32 + lane;            // row of P this thread holds
            const uint32_t t_addr = tmem_base + a * C::ACC_COLS + ((uint32_t)(quarter * 32) << 16);
            constexpr int CH = BN >= 32 ? 32 : 16;
#pragma unroll 1
            for (int c0 = turn * CH; c0 < BN; c0 += (EPI_WARPS / 4) * CH) {
                uint32_t r[CH];
                if (CH == 32) tmem_ld32(t_addr + c0, r); else tmem_ld16(t_addr + c0, r);
                tmem_ld_wait();
                const int q0 = tq * BN + c0;                           // first row of Q in this chunk
                if (GROUPED && SWAP && p.row_scale != nullptr) {
#pragma unroll
                    for (int j = 0; j < CH; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * p.row_scale[q0 + j]);
                }
                if constexpr (!SWAP) {
                    if (GROUPED && p.row_scale != nullptr) {
                        const float f = prow < p.rows_p ? p.row_scale[prow] : 0.f;
#pragma unroll
                        for (int j = 0; j < CH; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) * f);
                    }
                    if (CH == 32 && p.staged && (GATED ? q0 < p.rows_q : q0 + CH <= p.rows_q))
                        store_staged<TOut, GATED, GROUPED>(r, smem + C::EPI_OFF + (warp - 2) * EPI_STAGE_BYTES, lane, prow - lane, q0, p);
                    else store_token_major<TOut, GATED, CH, GROUPED>(r, prow, q0, sp, p);
                } else if (GATED && SWAP) {
                    // Lanes 0..15 hold gates, lanes 16..31 the ups of the same 16 features.  Two tokens a round: the
                    // lower lanes hand over their gates of the second token and get the ups of the first, so that each
                    // half of the warp computes and stores one token.
                    const bool low = lane < 16;
                    const int feat = ((prow >> 5) << 4) + (lane & 15);
#pragma unroll
                    for (int j = 0; j < CH; j += 2) {
                        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(low ? r[j + 1] : r[j]), 16);
                        const float g = low ? __uint_as_float(r[j]) : got;
                        const float u = low ? got : __uint_as_float(r[j + 1]);
                        const int tok = q0 + j + (low ? 0 : 1);
                        if (tok < p.rows_q && prow < p.rows_p)
                            ((bf16*)p.out)[(size_t)tok * p.ld_out + feat] = __float2bfloat16_rn(gated<GROUPED>(g, u, p.act, p.limit));
                    }
                } else {
                    // weight rows on lanes (prow), tokens on columns (q0 + j): lanes write neighbours
                    if (prow < p.rows_p) {
#pragma unroll
                        for (int j = 0; j < CH; j++) {
                            const int tok = q0 + j;
                            if (tok >= p.rows_q) break;
                            float v = __uint_as_float(r[j]);
                            if (p.splits > 1) {
                                p.partial[((size_t)sp * p.rows_q + tok) * p.rows_p + prow] = v;
                            } else {
                                v = pointwise(v, p);
                                ((TOut*)p.out)[(size_t)tok * p.ld_out + prow] = from_f<TOut>(v * p.scale);
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[a]);
        }
        if (!ok && !*abort_flag && lane == 0) { atomicExch(&g_gemm_error, 3); *abort_flag = 1; }
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// ---------------------------------------------------------------------------
// The same product for many tokens on a pair of SMs (cta_group::2): a cluster of two CTAs owns a tile of 256 tokens
// by BN weight rows.  Each CTA copies its 128 tokens of A and its half of the tile's weight rows into its own shared
// memory; a lane of the even CTA issues MMAs of 256 x BN x 16 that read A and half of B from each CTA and leave
// each CTA's 128 tokens of the result in its own tensor memory.  With BN = 256 a k-block of 64 then costs an SM 32 KB of shared
// memory and of copies instead of 48 KB: on one SM a 128 x 256 tile reads and refills its operands faster than the
// shared memory delivers them, which is what bounds the single-CTA kernel above.
//
// Barriers: both CTAs' copies count their bytes on the leader's `full` barrier (the leader expects both shares);
// a commit arrives on `empty` and `acc_full` at the same offset in both CTAs; the epilogue warps of both CTAs arrive
// on the leader's `acc_empty`.  All waits on these are bounded as above.  The two cluster barriers (after set-up,
// before the tensor memory is given back) are not: every path reaches them, since every loop before them ends.
// ---------------------------------------------------------------------------
template <int BN_> struct PairCfg {
    static constexpr int BN = BN_, HALF = BN / 2;
    static constexpr int STAGE_BYTES = BM * BK * 2 + HALF * BK * 2;       // per CTA
    static constexpr int STAGES = 192 * 1024 / STAGE_BYTES;
    static constexpr int ACC_COLS = 256, TMEM_COLS = 2 * ACC_COLS;
    static constexpr int EPI_OFF = STAGES * STAGE_BYTES + 256 /* barriers */;
    static constexpr int SMEM = EPI_OFF + EPI_WARPS * EPI_STAGE_BYTES + 1024 /* alignment */;
};

template <int BN, typename TOut, bool GATED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q, GemmParams p) {
    pdl_launch_dependents();
    using C = PairCfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE_BYTES);
    uint64_t* full = bars;                       // [STAGES], the leader's is used
    uint64_t* empty = bars + C::STAGES;          // [STAGES], each CTA's own
    uint64_t* acc_full = bars + 2 * C::STAGES;   // [2], each CTA's own
    uint64_t* acc_empty = acc_full + 2;          // [2], the leader's is used
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();     // 0: the leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

    if (threadIdx.x == 32) { tma_prefetch_map(&map_p); tma_prefetch_map(&map_q); }
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 2 * EPI_WARPS); }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc_pair(tmem_slot, C::TMEM_COLS);
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int n_items = p.tiles_p * p.tiles_q * p.splits;
    auto decode = [&](int item, int& tp, int& tq, int& sp) {
        sp = item % p.splits; item /= p.splits;
        tp = item % p.tiles_p; tq = item / p.tiles_p;
    };
    constexpr int A_OFF = 0, W_OFF = BM * BK * 2;

    if (warp == 0) {
        // ---------------- TMA producer, in both CTAs ----------------
        const uint32_t lead_full = cluster_addr(&full[0], 0);
        const uint32_t sm0 = smem_u32(smem), full0 = smem_u32(full), empty0 = smem_u32(empty);
        uint32_t it = 0;
        const uint64_t policy = once_policy();
        Ring ring;
        bool ok = true, waited = false;
        for (int item = pair; item < n_items && ok; item += n_pairs) {
            int tp, tq, sp; decode(item, tp, tq, sp);
            const int kb0 = sp * p.kb_per_split, kb1 = min(p.kblocks, kb0 + p.kb_per_split);
            const int a_row = tp * 256 + (int)rank * BM, w_row = tq * C::BN + (int)rank * C::HALF;
            int kb = kb0;
            if (!waited) {
                // weights first, then the wait for the kernel before this one, then its output
                const int pre = min(kb1 - kb0, C::STAGES);
                if (elected())
                    for (int j = 0; j < pre; j++) {
                        if (rank == 0) bar_expect(full0 + 8 * j, 2 * C::STAGE_BYTES);
                        tile_load_pair_once(sm0 + j * C::STAGE_BYTES + W_OFF, &map_q, lead_full + 8 * j, (kb0 + j) * BK, w_row, policy);
                    }
                pdl_wait();
                waited = true;
                if (elected())
                    for (int j = 0; j < pre; j++)
                        tile_load_pair(sm0 + j * C::STAGE_BYTES + A_OFF, &map_p, lead_full + 8 * j, (kb0 + j) * BK, a_row);
                __syncwarp();
                it = pre; kb = kb0 + pre;
                ring.s = pre % C::STAGES; ring.ph = pre / C::STAGES;
            }
            for (; kb < kb1; kb++, it++) {
                if (!warp_wait(empty0 + 8 * ring.s, ring.ph ^ 1, abort_flag)) { ok = false; break; }
                const uint32_t st = sm0 + ring.s * C::STAGE_BYTES, bar = lead_full + 8 * ring.s;
                if (elected()) {
                    if (rank == 0) bar_expect(full0 + 8 * ring.s, 2 * C::STAGE_BYTES);
                    tile_load_pair_once(st + W_OFF, &map_q, bar, kb * BK, w_row, policy);
                    tile_load_pair(st + A_OFF, &map_p, bar, kb * BK, a_row);
                }
                ring.step<C::STAGES>();
            }
        }
        if (!ok && lane == 0) {
            if (!*abort_flag) { atomicExch(&g_gemm_error, 4); *abort_flag = 1; }
            // the leader's barriers count both CTAs' copies: wait for those already issued
            if (rank == 0)
                for (uint32_t back = 1; back <= (uint32_t)C::STAGES && back <= it; back++) {
                    const uint32_t j = it - back;
                    mbar_wait(&full[j % C::STAGES], (j / C::STAGES) & 1);
                }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer, in the leader ----------------
        if (rank == 0) {
            constexpr uint32_t idesc = instr_desc_pair(C::BN);
            const uint64_t desc0 = smem_desc(smem_u32(smem));
            const uint32_t lo0 = desc_lo(desc0), hi = desc_hi(desc0), full0 = smem_u32(full), empty0 = smem_u32(empty);
            const uint32_t acc_full0 = smem_u32(acc_full), acc_empty0 = smem_u32(acc_empty);
            uint32_t tile_it = 0;
            Ring ring;
            bool ok = true;
            for (int item = pair; item < n_items && ok; item += n_pairs, tile_it++) {
                int tp, tq, sp; decode(item, tp, tq, sp);
                const int kb0 = sp * p.kb_per_split, kb1 = min(p.kblocks, kb0 + p.kb_per_split);
                const int a = tile_it & 1; const uint32_t aph = (tile_it >> 1) & 1;
                if (!warp_wait(acc_empty0 + 8 * a, aph ^ 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_addr = tmem_base + a * C::ACC_COLS;
                for (int kb = kb0; kb < kb1; kb++) {
                    if (!warp_wait(full0 + 8 * ring.s, ring.ph, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_lo = lo0 + ring.s * (C::STAGE_BYTES / 16);
                    // the commit frees the stage in both CTAs
                    if (elected()) issue_kblock<true>(d_addr, a_lo, a_lo + W_OFF / 16, hi, idesc, kb > kb0, empty0 + 8 * ring.s);
                    ring.step<C::STAGES>();
                }
                if (ok && elected()) commit_to_pair(acc_full0 + 8 * a);    // the accumulator is complete in both CTAs
            }
            if (!ok && lane == 0 && !*abort_flag) { atomicExch(&g_gemm_error, 5); *abort_flag = 1; }
            __syncwarp();
        }
    } else {
        // ---------------- epilogue: warps 2..9 of both CTAs ----------------
        const int quarter = warp & 3;
        const int turn = (warp - 2) >> 2;
        const uint32_t lead_acc_empty = cluster_addr(&acc_empty[0], 0);
        pdl_wait();
        uint32_t tile_it = 0;
        bool ok = true;
        for (int item = pair; item < n_items && ok; item += n_pairs, tile_it++) {
            int tp, tq, sp; decode(item, tp, tq, sp);
            const int a = tile_it & 1; const uint32_t aph = (tile_it >> 1) & 1;
            const bool mine = !*abort_flag && mbar_wait(&acc_full[a], aph);
            if (!__all_sync(0xffffffffu, mine)) { ok = false; break; }
            tc_fence_after();
            const int prow = tp * 256 + (int)rank * BM + quarter * 32 + lane;
            const uint32_t t_addr = tmem_base + a * C::ACC_COLS + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int c0 = turn * 32; c0 < C::BN; c0 += (EPI_WARPS / 4) * 32) {
                uint32_t r[32];
                tmem_ld32(t_addr + c0, r);
                tmem_ld_wait();
                const int q0 = tq * C::BN + c0;
                if (p.staged && (GATED ? q0 < p.rows_q : q0 + 32 <= p.rows_q))
                    store_staged<TOut, GATED>(r, smem + C::EPI_OFF + (warp - 2) * EPI_STAGE_BYTES, lane, prow - lane, q0, p);
                else store_token_major<TOut, GATED, 32>(r, prow, q0, sp, p);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead_acc_empty + 8 * a);
        }
        if (!ok && !*abort_flag && lane == 0) { atomicExch(&g_gemm_error, 6); *abort_flag = 1; }
    }

    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    if (warp == 1) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
}

// ---------------------------------------------------------------------------
// Many tokens, but fewer tiles than SMs and a long K: a cluster of S CTAs owns one tile of 128 tokens by BN weight rows
// and each takes a share of K.  The shares meet in distributed shared memory: chunk c (32 columns) of the tile belongs to
// CTA c mod S; the others write their sums of it into that CTA's stages (idle by then), and the owner adds them in the
// order of K and runs the epilogue, so that every epilogue works (also those that need the whole sum), nothing passes
// through memory, and the result does not depend on which CTA was late.
// ---------------------------------------------------------------------------
template <int BN, typename TOut, bool GATED>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tc_split_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_q, GemmParams p) {
    pdl_launch_dependents();
    using C = Cfg<BN, false>;
    constexpr int CHUNKS = BN / 32;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE_BYTES);
    uint64_t* full = bars;                       // [STAGES]
    uint64_t* empty = bars + C::STAGES;          // [STAGES]
    uint64_t* acc_full = bars + 2 * C::STAGES;
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = p.cluster, ks = (int)cluster_ctarank();

    if (threadIdx.x == 32) { tma_prefetch_map(&map_p); tma_prefetch_map(&map_q); }
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(tmem_slot, BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int tile = blockIdx.x / S, tp = tile % p.tiles_p, tq = tile / p.tiles_p;
    const int kb0 = ks * p.kblocks / S, n_kb = (ks + 1) * p.kblocks / S - kb0;      // S <= kblocks: every share has work
    const int quarter = warp & 3, turn = (warp - 2) >> 2;
    const uint32_t t_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);

    if (warp == 0) {
        const int a_row = tp * BM, w_row = tq * BN;
        const int pre = min(n_kb, C::STAGES);
        const uint32_t sm0 = smem_u32(smem), full0 = smem_u32(full), empty0 = smem_u32(empty);
        bool ok = true;
        const uint64_t policy = once_policy();
        // weights first, then the wait for the kernel before this one, then its output
        if (elected())
            for (int j = 0; j < pre; j++) {
                bar_expect(full0 + 8 * j, C::STAGE_BYTES);
                tile_load_once(sm0 + j * C::STAGE_BYTES + BM * BK * 2, &map_q, full0 + 8 * j, (kb0 + j) * BK, w_row, policy);
            }
        pdl_wait();
        if (elected())
            for (int j = 0; j < pre; j++) tile_load(sm0 + j * C::STAGE_BYTES, &map_p, full0 + 8 * j, (kb0 + j) * BK, a_row);
        __syncwarp();
        Ring ring;
        ring.s = pre % C::STAGES; ring.ph = pre / C::STAGES;
        int it = pre;
        for (; it < n_kb; it++) {
            if (!warp_wait(empty0 + 8 * ring.s, ring.ph ^ 1, abort_flag)) { ok = false; break; }
            const uint32_t st = sm0 + ring.s * C::STAGE_BYTES, bar = full0 + 8 * ring.s;
            if (elected()) {
                bar_expect(bar, C::STAGE_BYTES);
                tile_load_once(st + BM * BK * 2, &map_q, bar, (kb0 + it) * BK, w_row, policy);
                tile_load(st, &map_p, bar, (kb0 + it) * BK, a_row);
            }
            ring.step<C::STAGES>();
        }
        if (!ok && lane == 0) {
            if (!*abort_flag) { atomicExch(&g_gemm_error, 7); *abort_flag = 1; }
            for (int back = 1; back <= C::STAGES && back <= it; back++) {
                const uint32_t j = it - back;
                mbar_wait(&full[j % C::STAGES], (j / C::STAGES) & 1);
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc(BN);
        const uint64_t desc0 = smem_desc(smem_u32(smem));
        const uint32_t lo0 = desc_lo(desc0), hi = desc_hi(desc0), full0 = smem_u32(full), empty0 = smem_u32(empty);
        Ring ring;
        bool ok = true;
        for (int it = 0; it < n_kb; it++) {
            if (!warp_wait(full0 + 8 * ring.s, ring.ph, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t a_lo = lo0 + ring.s * (C::STAGE_BYTES / 16);
            if (elected()) issue_kblock<false>(tmem_base, a_lo, a_lo + BM * BK * 2 / 16, hi, idesc, it > 0, empty0 + 8 * ring.s);
            ring.step<C::STAGES>();
        }
        if (ok && elected()) commit_to(smem_u32(acc_full));
        if (!ok && lane == 0 && !*abort_flag) { atomicExch(&g_gemm_error, 8); *abort_flag = 1; }
    } else {
        pdl_wait();                                    // the output may still be read by the kernel before
        // the decision must be the same in every lane: tcgen05.ld is a warp-wide instruction
        const bool mine = !*abort_flag && mbar_wait(acc_full, 0);
        if (!__all_sync(0xffffffffu, mine) && !*abort_flag && lane == 0) { atomicExch(&g_gemm_error, 9); *abort_flag = 1; }
    }
    tc_fence_before();
    cluster_sync();                                    // every share is complete and no CTA's stages are in use any more
    tc_fence_after();
    const int row = quarter * 32 + lane;
    if (warp >= 2) {
        for (int c = turn; c < CHUNKS; c += EPI_WARPS / 4) {
            const int owner = c % S;
            if (owner == ks) continue;
            uint32_t r[32];
            tmem_ld32(t_addr + c * 32, r);
            tmem_ld_wait();
            // [chunk of the owner][share, without the owner's][column][row]
            const uint32_t dst = cluster_addr(smem, owner) + ((((c / S) * (S - 1) + (ks < owner ? ks : ks - 1)) * 32) * BM + row) * 4;
#pragma unroll
            for (int j = 0; j < 32; j++) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(dst + j * BM * 4), "r"(r[j]) : "memory");
        }
    }
    tc_fence_before();
    cluster_sync();                                    // all sums are where they are added; nobody touches another CTA any more
    tc_fence_after();
    if (warp >= 2) {
        const float* sums = (const float*)smem;
        for (int c = turn; c < CHUNKS; c += EPI_WARPS / 4) {
            if (c % S != ks) continue;
            uint32_t r[32];
            tmem_ld32(t_addr + c * 32, r);
            tmem_ld_wait();
            const float* src = sums + (size_t)(c / S) * (S - 1) * 32 * BM + row;
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = 0.f;
            for (int s = 0; s < S; s++) {
                const float* from = src + (size_t)(s < ks ? s : s - 1) * 32 * BM;
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] += s == ks ? __uint_as_float(r[j]) : from[j * BM];
            }
#pragma unroll
            for (int j = 0; j < 32; j++) r[j] = __float_as_uint(v[j]);
            const int q0 = tq * BN + c * 32;
            if (p.staged && (GATED ? q0 < p.rows_q : q0 + 32 <= p.rows_q))
                store_staged<TOut, GATED>(r, smem + C::EPI_OFF + (warp - 2) * EPI_STAGE_BYTES, lane, tp * BM + quarter * 32, q0, p);
            else store_token_major<TOut, GATED, 32>(r, tp * BM + row, q0, 0, p);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, BN);
}

// partial[splits][rows][cols] summed in split order, then cap and conversion.
template <typename TOut>
__global__ void splitk_reduce_kernel(const float* __restrict__ partial, TOut* __restrict__ out, int rows, int cols,
                                     long long ld_out, int splits, float cap, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)rows * cols;
    if (i >= n) return;
    float s = 0.f;
    for (int k = 0; k < splits; k++) s += partial[(size_t)k * n + i];
    if (cap > 0.f) s = softcap_f(s, cap);
    out[(i / cols) * ld_out + (i % cols)] = from_f<TOut>(s * scale);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// rows x K bf16 matrix with row stride ld (elements); box = box_rows x 64 elements, 128-byte swizzle.
static int make_map(CUtensorMap* m, const void* base, long long rows, long long K, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return tb_refuse("gemm_tc: the driver does not provide cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return tb_refuse("gemm_tc: cuTensorMapEncodeTiled failed with %d", (int)r);
    return 0;
}

static int g_sms = 0;

template <int BN, bool SWAP, typename TOut, bool GATED = false, bool WIDE = false, bool GROUPED = false>
static int launch(const CUtensorMap& mp, const CUtensorMap& mq, const GemmParams& p, cudaStream_t stream) {
    using C = Cfg<BN, SWAP, WIDE>;
    static bool attr_set = false;
    auto kern = gemm_tc_kernel<BN, SWAP, TOut, GATED, WIDE, GROUPED>;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return (int)e;
        attr_set = true;
    }
    const int items = p.tiles_p * p.tiles_q * p.splits;
    const int grid = items < g_sms ? items : g_sms;
    tb_launch(kern, dim3(grid), dim3(GEMM_THREADS), C::SMEM, stream, mp, mq, p);
    return tb_launch_status();
}

// Many-token products on pairs of SMs: 0 never, 1 whenever the shape allows, 2 where it pays.  The environment
// variable TRAPETUM_GEMM_PAIR sets the start value (for profiling one kernel on every shape).
static int pair_policy_from_env() {
    const char* e = getenv("TRAPETUM_GEMM_PAIR");
    return (e && e[0] >= '0' && e[0] <= '2' && !e[1]) ? e[0] - '0' : 2;
}
static int g_pair = pair_policy_from_env();
static int g_pair_clusters = 0;

// Sets that policy (for comparisons and tests); returns the previous setting.
extern "C" int tb_gemm_tc_set_pair(int mode) { const int was = g_pair; g_pair = mode < 0 ? 0 : mode > 2 ? 2 : mode; return was; }

// Which form a product of many tokens takes: the one whose time, by a cost fitted to timed launches, is least.
//   time = launch + rounds * (round + k-blocks * kblock)      and not less than      launch - 2 + padded operations / rate
// with a round being as many tiles as the device runs at once.  In microseconds; 249 products of 130 to 3,500 tokens with
// the 2B, 9B, 27B and a medium model's matrices, weights from memory, in a graph: the form picked takes 0.7 % longer than
// the best on the mean and 8 % at most, and 13 % less than single SMs and pairs with tiles of 256 alone.  The k-block's
// time is the MMAs' (128 cycles for 256 x 256 x 16) from 192 columns a pair on, below that the copies'; the rate is what
// the power cap leaves.  A cluster of two to four CTAs on one tile's K pays where there are few tiles: 384 tokens x 2,304
// x 9,216: 63 us on single SMs at first, 35 with the loops as they are now, 23 with K cut in two.
struct TileForm { bool pair; int bn, cluster; };
static TileForm choose_form(int M, int N, int kblocks, int sms) {
    struct Cost { bool pair; int bn, cluster; double launch, round, kblock, rate; };
    static const Cost costs[] = {{false, 128, 1, 4.0, 0.9, 0.212, 1.30e9}, {false, 256, 1, 5.0, 0.5, 0.342, 1.50e9},
                                 {true, 128, 1, 5.0, 0.8, 0.167, 1.45e9},  {true, 192, 1, 6.5, 0.5, 0.227, 1.62e9},
                                 {true, 224, 1, 7.5, 0.9, 0.254, 1.68e9},  {true, 256, 1, 6.0, 1.0, 0.289, 1.68e9},
                                 {false, 128, 2, 1.5, 5.0, 0.230, 1.30e9}, {false, 128, 3, 1.5, 5.0, 0.230, 1.30e9},
                                 {false, 128, 4, 1.5, 5.0, 0.230, 1.30e9}, {false, 256, 3, 1.7, 7.7, 0.375, 1.50e9},
                                 {false, 256, 4, 1.7, 7.7, 0.375, 1.50e9}};
    TileForm best = {false, 128, 1};
    double least = 1e30;
    for (const Cost& c : costs) {
        const bool pairs_only = g_pair == 1 && N >= 256;
        if (c.pair ? (g_pair == 0 || N < 256) : pairs_only) continue;
        if (c.bn > 128 && N < 256) continue;
        if (c.cluster > 1 && 2 * c.cluster > kblocks) continue;
        const long long bm = c.pair ? 256 : BM, tiles = ((M + bm - 1) / bm) * ((N + c.bn - 1) / c.bn);
        // SMs are handed out a GPC at a time: of these kernels, one CTA an SM, the runtime reports 74 clusters of two, 45 of
        // three and 33 of four at once on a B200's 148 SMs.  (Elsewhere in proportion: an estimate in a cost, not a limit.)
        const long long slots = c.pair || c.cluster == 2 ? sms / 2 : c.cluster == 1 ? sms : c.cluster == 3 ? sms * 45 / 148 : sms * 33 / 148;
        const double rounds = (double)((tiles + slots - 1) / (slots > 0 ? slots : 1));
        const double busy = rounds * (c.round + (kblocks + c.cluster - 1) / c.cluster * c.kblock);
        const double power = 2.0 * bm * c.bn * BK * (double)tiles * kblocks / c.rate - 2.0;
        const double t = c.launch + (busy > power ? busy : power);
        if (t < least) { least = t; best = {c.pair, c.bn, c.cluster}; }
    }
    return best;
}

// That choice for a product of M > 128 tokens on a device of `sms` SMs: 1000 * CTAs per tile + columns, + 100000 for pairs.
extern "C" int tb_gemm_tc_form(int M, int N, int K, int sms) {
    const TileForm f = choose_form(M, N, (K + BK - 1) / BK, sms);
    return (f.pair ? 100000 : 0) + 1000 * f.cluster + f.bn;
}

template <int BN, typename TOut, bool GATED>
static int launch_pair(const CUtensorMap& mp, const CUtensorMap& mq, const GemmParams& p, cudaStream_t stream) {
    using C = PairCfg<BN>;
    static bool attr_set = false;
    auto kern = gemm_tc_pair_kernel<BN, TOut, GATED>;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return (int)e;
        attr_set = true;
    }
    if (!g_pair_clusters) {
        // how many pairs the device runs at once (an SM without a free neighbour takes none)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * (g_sms / 2)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = C::SMEM;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) { cudaGetLastError(); n = g_sms / 2; }
        g_pair_clusters = n < g_sms / 2 ? n : g_sms / 2;
    }
    const int items = p.tiles_p * p.tiles_q * p.splits;
    const int pairs = items < g_pair_clusters ? items : g_pair_clusters;
    tb_launch(kern, dim3(2 * pairs), dim3(GEMM_THREADS), C::SMEM, stream, mp, mq, p);
    return tb_launch_status();
}

template <int BN, typename TOut, bool GATED>
static int launch_split(const CUtensorMap& mp, const CUtensorMap& mq, const GemmParams& p, cudaStream_t stream) {
    using C = Cfg<BN, false>;
    static bool attr_set = false;
    auto kern = gemm_tc_split_kernel<BN, TOut, GATED>;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
        if (e != cudaSuccess) return (int)e;
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.tiles_p * p.tiles_q * p.cluster); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = C::SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kern, mp, mq, p);
    return tb_launch_status();
}

extern "C" int tb_gemm_tc_takes(const void* A, const void* W, int M, int N, int K, long long lda, long long ldw) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if (K % 8 || lda % 8 || ldw % 8) return 0;
    if (((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return 0;
    return 1;
}

extern "C" long long tb_gemm_tc_scratch_floats(int M, int N, int splits) {
    return splits > 1 ? (long long)splits * M * N : 0;
}

// How many K splits a small-token product should use so that about one CTA per SM streams weights.
extern "C" int tb_gemm_tc_splits(int M, int N, int K, int sms) {
    if (M > BM) return 1;
    const int tiles = (N + BM - 1) / BM;
    const int kblocks = (K + BK - 1) / BK;
    if (tiles * 2 > sms) return 1;
    int s = sms / tiles;
    if (s > kblocks / 2) s = kblocks / 2;          // at least two k-blocks per split
    if (s > 16) s = 16;
    if (s < 1) s = 1;
    const int per = (kblocks + s - 1) / s;
    return (kblocks + per - 1) / per;              // every split non-empty
}

// The split count a call really uses: every split gets the same number of k-blocks and none is empty.
extern "C" int tb_gemm_tc_effective_splits(int K, int splits) {
    const int kblocks = (K + BK - 1) / BK;
    if (splits < 1) splits = 1;
    if (splits > kblocks) splits = kblocks;
    const int per = (kblocks + splits - 1) / splits;
    return (kblocks + per - 1) / per;
}

// reduce = 0 with splits > 1: leave the partial sums in `scratch` ([splits][M][N]) for the consumer to add.
// out_scale: the output times this number (1: a plain product; not with a cap, not on partial sums that are left).
// act_limit: the limit of the gated activation 2 (clamped_swish).
static int gemm_tc_run(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K,
                       long long lda, long long ldw, long long ldc, float softcap, int splits, float* scratch,
                       int reduce, int gated_act, float act_limit, float out_scale, int unary, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (unary < 0 || unary > 2) return tb_refuse("gemm_tc: unknown unary activation %d", unary);
    if (unary && (gated_act >= 0 || softcap > 0.f)) return tb_refuse("gemm_tc: a unary activation goes with neither a gate nor a cap");
    if (unary) splits = 1;                           // the activation is not linear: no partial sums
    if (!tb_gemm_tc_takes(A, W, M, N, K, lda, ldw))
        return tb_refuse("gemm_tc: needs K, lda, ldw multiples of 8 and 16-byte aligned operands "
                         "(M=%d N=%d K=%d lda=%lld ldw=%lld)", M, N, K, lda, ldw);
    if (c_dtype != TB_F32 && c_dtype != TB_BF16) return tb_refuse("gemm_tc: unknown output dtype %d", c_dtype);
    if (!g_sms) {
        int dev = 0; cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 148;
    }
    const int kblocks = (K + BK - 1) / BK;
    if (splits < 1) splits = 1;
    if (splits > kblocks) splits = kblocks;
    int per = (kblocks + splits - 1) / splits;
    splits = (kblocks + per - 1) / per;
    if (splits > 1 && scratch == nullptr) return tb_refuse("gemm_tc: split-K needs scratch");
    const bool gated = gated_act >= 0;
    if (gated) {
        if (gated_act > 2) return tb_refuse("gemm_tc: unknown gated activation %d", gated_act);
        if (gated_act == 2 && !(act_limit > 0.f)) return tb_refuse("gemm_tc: clamped_swish needs a positive limit");
        if (N % 32) return tb_refuse("gemm_tc: the gated epilogue needs a multiple of 32 weight rows, got %d", N);
        if (c_dtype != TB_BF16) return tb_refuse("gemm_tc: the gated epilogue writes bfloat16");
        if (softcap > 0.f) return tb_refuse("gemm_tc: the gated epilogue takes no soft cap");
        splits = 1; per = kblocks;                   // the activation is not linear: no partial sums
    }

    const bool swap = M <= BM;
    const bool wide = (long long)N * K * 2 >= (long long)TB_WIDE_FROM_BYTES;
    TileForm form = {false, 128, 1};
    if (swap) form.bn = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
    else if (splits > 1) form.bn = N >= 256 ? 256 : 128;               // the caller's own split of K
    else form = choose_form(M, N, kblocks, g_sms);
    const int bn = form.bn;
    const bool pair = form.pair;

    GemmParams p;
    p.tile_group = nullptr; p.group_rows = 0; p.row_scale = nullptr;
    p.cluster = form.cluster;
    p.staged = splits == 1 && C != nullptr && ((uintptr_t)C & 15) == 0 && (ldc * (c_dtype == TB_BF16 ? 2 : 4)) % 16 == 0;
    p.K = K; p.kblocks = kblocks; p.splits = splits; p.kb_per_split = per;
    p.out = C; p.ld_out = ldc; p.partial = scratch; p.cap = splits > 1 ? 0.f : softcap;
    p.act = gated ? gated_act : 0;
    p.limit = act_limit;
    p.unary = unary;
    if (out_scale != 1.0f && (softcap > 0.f || gated || (splits > 1 && !reduce)))
        return tb_refuse("gemm_tc: an output scale goes with neither a cap, a gated epilogue nor partial sums");
    p.scale = splits > 1 ? 1.0f : out_scale;
    CUtensorMap mp, mq;
    if (swap) {
        p.rows_p = N; p.rows_q = M;
        if (make_map(&mp, W, N, K, ldw, BM) || make_map(&mq, A, M, K, lda, bn)) return -1;
    } else {
        p.rows_p = M; p.rows_q = N;
        if (make_map(&mp, A, M, K, lda, BM) || make_map(&mq, W, N, K, ldw, pair ? bn / 2 : bn)) return -1;
    }
    p.tiles_p = (p.rows_p + (pair ? 256 : BM) - 1) / (pair ? 256 : BM);
    p.tiles_q = (p.rows_q + bn - 1) / bn;

    int st;
#define OUT3(FN, ...) (gated ? FN<__VA_ARGS__, bf16, true>(mp, mq, p, stream) : c_dtype == TB_BF16 ? FN<__VA_ARGS__, bf16, false>(mp, mq, p, stream) : FN<__VA_ARGS__, float, false>(mp, mq, p, stream))
    if (swap) {
        // a long stream of weights: the kernel's own bytes in flight count for more than the overlap with its
        // neighbours, so it takes the whole SM
        if (bn == 16) st = wide && gated ? launch<16, true, bf16, true, true>(mp, mq, p, stream)
                           : wide && c_dtype == TB_F32 ? launch<16, true, float, false, true>(mp, mq, p, stream) : OUT3(launch, 16, true);
        else st = bn == 32 ? OUT3(launch, 32, true) : bn == 64 ? OUT3(launch, 64, true) : OUT3(launch, 128, true);
    } else if (p.cluster > 1) st = bn == 256 ? OUT3(launch_split, 256) : OUT3(launch_split, 128);
    else if (pair) st = bn == 256 ? OUT3(launch_pair, 256) : bn == 224 ? OUT3(launch_pair, 224) : bn == 192 ? OUT3(launch_pair, 192) : OUT3(launch_pair, 128);
    else st = bn == 256 ? OUT3(launch, 256, false) : OUT3(launch, 128, false);
#undef OUT3
    if (st) return st;
    if (splits > 1 && reduce) {
        const size_t n = (size_t)M * N;
        const unsigned blocks = (unsigned)((n + 255) / 256);
        if (c_dtype == TB_BF16)
            tb_launch(splitk_reduce_kernel<bf16>, dim3(blocks), dim3(256), 0, stream, scratch, (bf16*)C, M, N, ldc, splits, softcap, out_scale);
        else
            tb_launch(splitk_reduce_kernel<float>, dim3(blocks), dim3(256), 0, stream, scratch, (float*)C, M, N, ldc, splits, softcap, out_scale);
        st = tb_launch_status();
    }
    return st;
}

// Grouped products: C[m, :] = A[m, :] W_g^T for the group g = tile_group[m / tile] of the tile of rows that holds row m (tile: 128,
// or 16, 32 or 64 where groups have few rows: swapped tiles, every group's weights streamed once per tile).
// W holds `groups` matrices of N rows each, one after the other ([groups * N, K]); rows of A are ordered so that every
// tile belongs to one group.  gated_act >= 0: the gated epilogue on rows interleaved per group (N = 2 x the
// output's width, bfloat16 out); else a plain product into C (bfloat16 or float32).  tile_group: device memory,
// [ceil(M / tile)] group numbers in [0, groups), or -1 for a tile that is not in use (its rows of C are not written).
// unary: an activation of experts without a gate branch (0: none); row_scale [M] or null: a number per row of A that multiplies
// its sums before any activation.
extern "C" int tb_gemm_tc_grouped_tiles(const void* A, const void* W, void* C, int c_dtype, int M, int N, int groups, int K,
                                        long long lda, long long ldw, long long ldc, const int* tile_group, int gated_act,
                                        int unary, const float* row_scale, int tile, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || groups <= 0) return 0;
    if (unary < 0 || unary > 2 || (unary && gated_act >= 0)) return tb_refuse("gemm_tc_grouped: unary activation %d (with gate %d)", unary, gated_act);
    if (!tb_gemm_tc_takes(A, W, M, N, K, lda, ldw))
        return tb_refuse("gemm_tc_grouped: needs K, lda, ldw multiples of 8 and 16-byte aligned operands");
    if (c_dtype != TB_F32 && c_dtype != TB_BF16) return tb_refuse("gemm_tc_grouped: unknown output dtype %d", c_dtype);
    if (tile_group == nullptr) return tb_refuse("gemm_tc_grouped: no table of groups");
    if ((long long)groups * N > 2147483647LL) return tb_refuse("gemm_tc_grouped: %d groups of %d rows", groups, N);
    const bool gated = gated_act >= 0;
    if (gated && ((gated_act > 1 && gated_act != 3) || N % 32 || c_dtype != TB_BF16))
        return tb_refuse("gemm_tc_grouped: the gated epilogue (gelu_tanh, silu or exact silu) needs a multiple of 32 weight rows and writes bfloat16");
    if (tile != 16 && tile != 32 && tile != 64 && tile != 128) return tb_refuse("gemm_tc_grouped: tiles of %d rows", tile);
    if (!g_sms) {
        int dev = 0; cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 148;
    }
    const bool swap = tile < BM;
    const int bn = swap ? tile : N >= 256 ? 256 : 128;
    GemmParams p;
    p.tile_group = tile_group; p.group_rows = N; p.row_scale = row_scale;
    p.K = K; p.kblocks = (K + BK - 1) / BK; p.splits = 1; p.kb_per_split = p.kblocks;
    p.out = C; p.ld_out = ldc; p.partial = nullptr; p.cap = 0.f; p.scale = 1.0f;
    p.act = gated ? gated_act : 0; p.limit = 0.f; p.unary = unary;
    p.cluster = 1; p.staged = ((uintptr_t)C & 15) == 0 && (ldc * (c_dtype == TB_BF16 ? 2 : 4)) % 16 == 0;
    CUtensorMap mp, mq;
#define OUT3(...) (gated ? launch<__VA_ARGS__, bf16, true, true, true>(mp, mq, p, stream) : c_dtype == TB_BF16 ? launch<__VA_ARGS__, bf16, false, true, true>(mp, mq, p, stream) : launch<__VA_ARGS__, float, false, true, true>(mp, mq, p, stream))
    if (swap) {
        p.rows_p = N; p.rows_q = M;
        if (make_map(&mp, W, (long long)groups * N, K, ldw, BM) || make_map(&mq, A, M, K, lda, bn)) return -1;
        p.tiles_p = (N + BM - 1) / BM;
        p.tiles_q = (M + bn - 1) / bn;
        return bn == 16 ? OUT3(16, true) : bn == 32 ? OUT3(32, true) : OUT3(64, true);
    }
    p.rows_p = M; p.rows_q = N;
    if (make_map(&mp, A, M, K, lda, BM) || make_map(&mq, W, (long long)groups * N, K, ldw, bn)) return -1;
    p.tiles_p = (M + BM - 1) / BM;
    p.tiles_q = (N + bn - 1) / bn;
    return bn == 256 ? OUT3(256, false) : OUT3(128, false);
#undef OUT3
}

extern "C" int tb_gemm_tc_ex(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K,
                             long long lda, long long ldw, long long ldc, float softcap, int splits, float* scratch,
                             int reduce, int gated_act, float act_limit, float out_scale, cudaStream_t stream) {
    return gemm_tc_run(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, softcap, splits, scratch, reduce, gated_act, act_limit, out_scale, 0, stream);
}

// The plain product whose every output becomes relu(v)^2 (unary = 1) or v Phi(v) (2): a feed-forward without a gate branch.
extern "C" int tb_gemm_tc_unary(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K,
                                long long lda, long long ldw, long long ldc, int unary, cudaStream_t stream) {
    return gemm_tc_run(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, 0.f, 1, nullptr, 0, -1, 0.f, 1.0f, unary, stream);
}

extern "C" int tb_gemm_tc(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K,
                          long long lda, long long ldw, long long ldc, float softcap, int splits, float* scratch,
                          int reduce, int gated_act, cudaStream_t stream) {
    if (gated_act > 1) return tb_refuse("gemm_tc: gated activation %d needs its parameter (tb_gemm_tc_ex)", gated_act);
    return tb_gemm_tc_ex(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, softcap, splits, scratch, reduce, gated_act, 0.f, 1.0f, stream);
}

// out[rows][cols] = sum over splits, in order, of partial[s][rows][cols] (32-bit).
extern "C" int tb_sum_partials(const float* partial, float* out, int rows, int cols, int splits, cudaStream_t stream) {
    const size_t n = (size_t)rows * cols;
    if (n == 0) return 0;
    if (splits < 1) return tb_refuse("sum_partials: splits=%d", splits);
    tb_launch(splitk_reduce_kernel<float>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream,
              partial, out, rows, cols, (long long)cols, splits, 0.f, 1.0f);
    return tb_launch_status();
}

// Reads and clears the error word (0 = no wait ran out).  Synchronises the device.
extern "C" int tb_gemm_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(int));
    return v;
}
