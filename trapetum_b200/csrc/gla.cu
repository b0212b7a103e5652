// Gated linear attention: everything between the input products and the output product.
//
// Per head, with key channels d and value channels v, for the tokens of a sequence in order:
//     S[d][v] <- decay_t[d] * S[d][v] + k_t[d] * v_t[v];      o_t[v] = sum_d S[d][v] * q_t[d]
// where decay_t[d] = sigmoid(z_t[d])^(1/tau) and z_t = A2 (A1 x_t) + bias (a product of low rank).
// Then every head's o_t is divided by its root mean square over v (+ eps inside the root), multiplied
// by a weight shared by the heads and by silu(g_t).
//
//   tb_gla_decay      z from the 32-bit partial sums of A1 x, the decay as exp(-softplus(-z) / tau)
//   tb_gla_scan       the recurrence; the state S of every sequence lives in a 32-bit row addressed by
//                     slot, is read at the start of the step's tokens and written back at their end,
//                     so a step of whole prompts and a step of one token each are the same kernel
//   tb_gla_gate_norm  the unit norm, the weight (if any) and the gate; output in the activations' dtype
//
// With head_decay the decay is a constant per head (retention); there is then no decay matrix and no tb_gla_decay.
//
// 32-bit throughout: z, the decay, the state, o and the norm.  q, k, v and g arrive in the activations'
// dtype (they are products) and are widened on the way in.
//
// The scan: one CTA = 64 value channels of one head of one sequence (or of a chunk in time of it), eight warps
// that each own an eighth of the key channels; a thread keeps its part of two columns of S in registers.  q, k
// and the decay of eight tokens at a time are staged in shared memory (every thread of a warp reads the same
// 16-byte word: a broadcast that serves both columns), the next eight are on their way through registers
// meanwhile; the warps' partial outputs of a tile meet in shared memory once per tile.
//
//   tb_gla_blocks     decay, recurrence, norm and gate of whole prompts in bfloat16, on tensor cores (see "Prompts in
//                     blocks" below)
#include "common.cuh"

TB_EXPORT_ERROR()

struct GlaArgs {
    const void* proj; long long proj_stride;          // [T] rows of q (H*D), k (H*D), v (H*V), g (H*V)
    const float* a1; int a1_splits; long long a1_split_stride; int rank;   // [splits][T][rank]
    const float* a2; const float* a2_bias;            // [H*D][rank], [H*D]
    float inv_tau, q_scale;
    const float* norm_w; float eps;                   // [V]
    float* state; long long state_stride;             // [slots][H*D*V]
    const int* seq_start; const int* token_seq; const int* slot_ids;
    float* decay;                                     // [T][H*D] scratch
    float* y;                                         // [T][H*V] scratch
    void* out;                                        // [T][H*V]
    int heads, D, V, batch, n_tokens;
    // long prompts cut into chunks in time that run side by side (0 chunks: one CTA walks a whole sequence)
    float* chunk_state;                               // [batch][n_chunks][H*D*V]: a chunk's end state from zero, then its start state
    float* chunk_decay;                               // [batch][n_chunks][H*D]: the product of the chunk's decays
    int chunk_len, n_chunks;
    const float* head_decay;                          // [H] or null: the decay of every key channel and token of a head
    int log2_decay;                                   // tb_gla_decay leaves log2 of the decay, no less than -150 (a factor of 0)
};

// The argument block's size, for the Python mirror's check.
extern "C" int tb_gla_args_bytes() { return (int)sizeof(GlaArgs); }

constexpr int GLA_DECAY_TOK = 8;

// 8 tokens and 256 channels per CTA: a thread owns a channel, keeps the sums in registers and reads its row of A2 once, in
// 16-byte pieces where it may.  With 32 tokens a CTA and a word a load, 2,048 tokens of 1,024 channels took 15.9 us: few
// warps, each with 32 chains of exponential and logarithm one after another.
__global__ void __launch_bounds__(256) gla_decay_kernel(GlaArgs a) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float low_s[];    // [8][rank]: A1 x of these tokens
    const int t0 = blockIdx.x * GLA_DECAY_TOK, nt = min(GLA_DECAY_TOK, a.n_tokens - t0);
    const int HD = a.heads * a.D;
    pdl_wait();
    for (int i = threadIdx.x; i < GLA_DECAY_TOK * a.rank; i += blockDim.x) {
        const int tt = i / a.rank, r = i % a.rank;
        float v = 0.f;
        if (tt < nt)
            for (int s = 0; s < a.a1_splits; s++) v += a.a1[(size_t)s * a.a1_split_stride + (size_t)(t0 + tt) * a.rank + r];
        low_s[i] = v;
    }
    __syncthreads();
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= HD) return;
    float z[GLA_DECAY_TOK];
    const float bias = a.a2_bias[c];
#pragma unroll
    for (int tt = 0; tt < GLA_DECAY_TOK; tt++) z[tt] = 0.f;
    const float* w = a.a2 + (size_t)c * a.rank;
    if (a.rank % 4 == 0 && ((uintptr_t)a.a2 & 15) == 0) {
        for (int r = 0; r < a.rank; r += 4) {
            const float4 wr = *(const float4*)(w + r);
#pragma unroll
            for (int tt = 0; tt < GLA_DECAY_TOK; tt++) {
                const float4 l = *(const float4*)(low_s + tt * a.rank + r);
                z[tt] = fmaf(wr.x, l.x, z[tt]); z[tt] = fmaf(wr.y, l.y, z[tt]); z[tt] = fmaf(wr.z, l.z, z[tt]); z[tt] = fmaf(wr.w, l.w, z[tt]);
            }
        }
    } else {
        for (int r = 0; r < a.rank; r++) {
            const float wr = w[r];
#pragma unroll
            for (int tt = 0; tt < GLA_DECAY_TOK; tt++) z[tt] = fmaf(wr, low_s[tt * a.rank + r], z[tt]);
        }
    }
#pragma unroll
    for (int tt = 0; tt < GLA_DECAY_TOK; tt++) {
        if (tt >= nt) break;
        const float x = -(z[tt] + bias);               // log sigmoid(z) = -softplus(-z)
        const float sp = x > 20.f ? x : log1pf(expf(x));
        if (a.log2_decay) {
            const float l = -sp * a.inv_tau * 1.44269504f;
            a.decay[(size_t)(t0 + tt) * HD + c] = l < -150.f ? -150.f : l;     // (NaN stays)
        } else {
            a.decay[(size_t)(t0 + tt) * HD + c] = expf(-sp * a.inv_tau);
        }
    }
}

constexpr int GLA_TT = 8;          // tokens per tile
constexpr int GLA_WARPS = 8;       // slices of the key channels

// MODE 0: a sequence from the state its slot holds to the state it leaves there, with outputs.
// MODE 1: a chunk from a zero state, without outputs: its end state and the product of its decays (for the fold).
// MODE 2: a chunk from the start state the fold left, with outputs; the last chunk leaves the sequence's state.
constexpr int GLA_VT = 64;         // value channels per CTA: two per thread, so that a word of q, k or the decay serves two updates

template <typename T, int DPT, int MODE>
__global__ void __launch_bounds__(GLA_WARPS * 32, 2) gla_scan_kernel(GlaArgs a) {
    pdl_launch_dependents();
    constexpr int DP = DPT * GLA_WARPS;                // key channels, padded
    constexpr int PER = (GLA_TT * DP + GLA_WARPS * 32 - 1) / (GLA_WARPS * 32);   // staged (token, channel) places per thread
    __shared__ __align__(16) float q_s[GLA_TT][DP], k_s[GLA_TT][DP], d_s[GLA_TT][DP];
    __shared__ float v_s[GLA_TT][GLA_VT];
    __shared__ float part_s[GLA_TT][GLA_WARPS][GLA_VT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = blockIdx.y;
    const int b = MODE == 0 ? blockIdx.z : blockIdx.z / a.n_chunks;
    const int chunk = MODE == 0 ? 0 : blockIdx.z % a.n_chunks;
    const int D = a.D, V = a.V, HD = a.heads * D, HV = a.heads * V;
    const int v0 = blockIdx.x * GLA_VT;
    const int vc[2] = {v0 + lane, v0 + lane + 32};
    const bool v_ok[2] = {vc[0] < V, vc[1] < V};
    pdl_wait();
    int s0 = a.seq_start[b], s1 = a.seq_start[b + 1];
    const int seq_end = s1;
    if (MODE != 0) { s0 = min(s1, s0 + chunk * a.chunk_len); s1 = min(s1, s0 + a.chunk_len); }
    float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)h * D * V;
    float* cst = MODE == 0 ? nullptr : a.chunk_state + ((size_t)b * a.n_chunks + chunk) * a.heads * D * V + (size_t)h * D * V;
    float S[2][DPT], P[MODE == 1 ? DPT : 1];
#pragma unroll
    for (int j = 0; j < DPT; j++) {
        const int d = warp * DPT + j;
        const float* from = MODE == 2 ? cst : st;
#pragma unroll
        for (int c = 0; c < 2; c++) S[c][j] = (MODE != 1 && d < D && v_ok[c]) ? from[(size_t)d * V + vc[c]] : 0.f;
        if (MODE == 1) P[j] = 1.f;
    }
    const T* proj = (const T*)a.proj;
    // a tile's q, k, decay and v travel through registers: the next tile's loads are in flight while this one is computed
    float rq[PER], rk[PER], rd[PER], rv[2];
    auto fetch = [&](int t0) {
        const int nt = min(GLA_TT, s1 - t0);
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = threadIdx.x + u * GLA_WARPS * 32;
            const int tt = i / DP, d = i % DP;
            rq[u] = 0.f; rk[u] = 0.f; rd[u] = 1.f;
            if (i < GLA_TT * DP && tt < nt && d < D) {
                const T* row = proj + (size_t)(t0 + tt) * a.proj_stride;
                if (MODE != 1) rq[u] = to_f<T>(row[h * D + d]) * a.q_scale;
                rk[u] = to_f<T>(row[HD + h * D + d]);
                rd[u] = a.head_decay != nullptr ? a.head_decay[h] : a.decay[(size_t)(t0 + tt) * HD + h * D + d];
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {                  // 8 tokens x 64 channels = 2 per thread
            const int i = threadIdx.x + u * GLA_WARPS * 32;
            const int tt = i / GLA_VT, c = v0 + i % GLA_VT;
            rv[u] = (tt < nt && c < V) ? to_f<T>(proj[(size_t)(t0 + tt) * a.proj_stride + 2 * HD + h * V + c]) : 0.f;
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = threadIdx.x + u * GLA_WARPS * 32;
            if (i < GLA_TT * DP) { (&q_s[0][0])[i] = rq[u]; (&k_s[0][0])[i] = rk[u]; (&d_s[0][0])[i] = rd[u]; }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) (&v_s[0][0])[threadIdx.x + u * GLA_WARPS * 32] = rv[u];
    };
    if (s0 < s1) { fetch(s0); stash(); }
    __syncthreads();
    for (int t0 = s0; t0 < s1; t0 += GLA_TT) {
        const int nt = min(GLA_TT, s1 - t0);
        const bool more = t0 + GLA_TT < s1;
        if (more) fetch(t0 + GLA_TT);
        for (int tt = 0; tt < nt; tt++) {
            const float va = v_s[tt][lane], vb = v_s[tt][lane + 32];
            float acc_a = 0.f, acc_b = 0.f;
            if constexpr (DPT % 4 == 0) {
                const float4* d4 = reinterpret_cast<const float4*>(&d_s[tt][warp * DPT]);
                const float4* k4 = reinterpret_cast<const float4*>(&k_s[tt][warp * DPT]);
                const float4* q4 = reinterpret_cast<const float4*>(&q_s[tt][warp * DPT]);
#pragma unroll
                for (int j4 = 0; j4 < DPT / 4; j4++) {
                    const float4 dd = d4[j4], kk = k4[j4];
                    const float dv[4] = {dd.x, dd.y, dd.z, dd.w}, kv[4] = {kk.x, kk.y, kk.z, kk.w};
                    float qv[4] = {0.f, 0.f, 0.f, 0.f};
                    if (MODE != 1) { const float4 qq = q4[j4]; qv[0] = qq.x; qv[1] = qq.y; qv[2] = qq.z; qv[3] = qq.w; }
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int j = j4 * 4 + e;
                        S[0][j] = fmaf(dv[e], S[0][j], kv[e] * va);
                        S[1][j] = fmaf(dv[e], S[1][j], kv[e] * vb);
                        if (MODE == 1) P[j] *= dv[e];
                        else { acc_a = fmaf(S[0][j], qv[e], acc_a); acc_b = fmaf(S[1][j], qv[e], acc_b); }
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < DPT; j++) {
                    const int d = warp * DPT + j;
                    const float dec = d_s[tt][d], kk = k_s[tt][d];
                    S[0][j] = fmaf(dec, S[0][j], kk * va);
                    S[1][j] = fmaf(dec, S[1][j], kk * vb);
                    if (MODE == 1) P[j] *= dec;
                    else { acc_a = fmaf(S[0][j], q_s[tt][d], acc_a); acc_b = fmaf(S[1][j], q_s[tt][d], acc_b); }
                }
            }
            if (MODE != 1) { part_s[tt][warp][lane] = acc_a; part_s[tt][warp][lane + 32] = acc_b; }
        }
        __syncthreads();                               // every warp is done with the tile; the partial outputs are complete
        if (MODE != 1) {
            const int tt = warp;                       // 8 warps = the tile's 8 tokens
            if (tt < nt) {
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    float o = 0.f;
#pragma unroll
                    for (int w = 0; w < GLA_WARPS; w++) o += part_s[tt][w][lane + 32 * c];
                    if (v_ok[c]) a.y[(size_t)(t0 + tt) * HV + h * V + vc[c]] = o;
                }
            }
        }
        if (more) stash();
        __syncthreads();                               // the next tile is in shared memory; the partial outputs are free again
    }
    if (MODE == 2 && s1 != seq_end) return;            // only the chunk that holds the sequence's end leaves its state
    if (MODE == 2 && s0 == s1 && chunk != 0) return;   // (an empty chunk after the end: the one before it did)
#pragma unroll
    for (int j = 0; j < DPT; j++) {
        const int d = warp * DPT + j;
        float* to = MODE == 1 ? cst : st;
#pragma unroll
        for (int c = 0; c < 2; c++)
            if (d < D && v_ok[c]) to[(size_t)d * V + vc[c]] = S[c][j];
        if (MODE == 1 && d < D && blockIdx.x == 0 && lane == 0)
            a.chunk_decay[((size_t)b * a.n_chunks + chunk) * a.heads * D + (size_t)h * D + d] = P[j];
    }
}

// Start states of the chunks from their end states: S_start[0] = the slot's state, S_start[c+1] = P_c S_start[c] + E_c,
// element by element; chunk_state[c] is turned from E_c into S_start[c] in place.
__global__ void gla_fold_kernel(GlaArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int D = a.D, V = a.V;
    const long long per = (long long)a.heads * D * V;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= per * a.batch) return;
    const int b = (int)(i / per);
    const long long e = i % per;                      // (h, d, v)
    const long long hd = e / V;                       // h * D + d
    float S = a.state[(size_t)a.slot_ids[b] * a.state_stride + e];
    float* cs = a.chunk_state + (size_t)b * a.n_chunks * per + e;
    const float* cd = a.chunk_decay + (size_t)b * a.n_chunks * a.heads * D + hd;
    for (int c0 = 0; c0 < a.n_chunks; c0 += 8) {       // eight chunks' end states and decays on their way together
        float E[8], P[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const bool in = c0 + u < a.n_chunks;
            E[u] = in ? cs[(size_t)(c0 + u) * per] : 0.f;
            P[u] = in ? cd[(size_t)(c0 + u) * a.heads * D] : 1.f;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (c0 + u < a.n_chunks) {
                cs[(size_t)(c0 + u) * per] = S;
                S = fmaf(P[u], S, E[u]);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// Prompts in blocks (bfloat16; D up to 128, V up to 256).  A CTA owns a head of a chunk of a sequence, a warp 16 value
// channels, whose state S^T [16 v][D] stays in registers, as accumulators of mma.sync lie, while the CTA walks the
// chunk 16 tokens at a time.  With c_i[d] the sum of the log2 decays from the block's start through token i:
//     o_i = S^T (q_i 2^c_i) + sum_{j <= i} P_ij v_j,     P_ij = sum_d q_i[d] k_j[d] 2^(c_i - c_j)   (32-bit FMA)
//     S^T <- S^T 2^c_15 + sum_j v_j (k_j 2^(c_15 - c_j))^T
// No exponent is positive, so nothing overflows whatever the decays.  v is a bfloat16 number; S, P and the decayed q and k
// are 32-bit and enter as sums of three bfloat16 numbers each (of S times q the six products above 2^-24 are taken).  A tensor
// core's sums are cut off, so a block's are made apart from the state; decays come from ex2 of summed logs.  Against 64 bits
// the state of 2,048 tokens stands 1.5e-7 off (the recurrence 2.1e-6; with decays of about 0.6 a token 0.7e-7 and 0.5e-7).
// The sums c are made in 64 bits and kept as two 32-bit numbers.  Long prompts: a first launch (OUT false) leaves the sums of
// every chunk but a sequence's last, gla_block_fold_kernel turns them into start states, the second launch (OUT true) writes
// the outputs, normed and gated: the CTA holds the head.
// A non-finite v is seen by its own token and later ones only, as in the recurrence; what it leaves in the state is NaN to the
// next block's outputs (an infinity has no three parts).
// Prompts of 1,500 and 548 tokens, 8 heads of 128 x 256, all of ops.gla, passes back to back: 141.7 us (the recurrence in chunks,
// its norm a launch of its own: 453; there the chunks of the shorter prompt leave SMs idle too).  A block takes 9.6 us of its CTA: shared
// memory (14 of 18 thousand cycles), then issue slots; the products are a quarter of the tensor pipe.
// ---------------------------------------------------------------------------------------------------------
constexpr int GB = 16;                                // tokens of a block

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;                     // 0 source bytes: the 16 destination bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *(uint32_t*)&h;
}
// Two 32-bit numbers as sums of three bfloat16 numbers each: the remainders are exact, the last one holds what is left.
__device__ __forceinline__ void split3(float x, float y, uint32_t* part) {
    part[0] = pack2(x, y);
    x -= __uint_as_float(part[0] << 16); y -= __uint_as_float(part[0] & 0xffff0000u);
    part[1] = pack2(x, y);
    part[2] = pack2(x - __uint_as_float(part[1] << 16), y - __uint_as_float(part[1] & 0xffff0000u));
}
__device__ __forceinline__ void split3(float x, bf16* hi, int step) {      // to hi[0], hi[step], hi[2 step]
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const bf16 h = __float2bfloat16_rn(x);
        hi[k * step] = h;
        x -= __bfloat162float(h);
    }
}
// A sign bit of the result is set where one of two bfloat16 numbers is infinite or NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t v) { return (v & 0x7f807f80u) + 0x00800080u; }
__device__ __forceinline__ float exp2_fast(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

// Shared memory of a CTA, in bytes from its start.
template <int DP>
struct BlockSmem {
    static constexpr int RP = DP * 2 + 16;            // bytes of a row of D bfloat16 numbers (no bank conflicts)
    static constexpr int FP = DP + 16;                // floats of a row of D 32-bit numbers (two rows' 64 bytes side by side in the banks)
    static constexpr int k3 = 0;                      // [3][16][RP] decayed keys
    static constexpr int q3 = k3 + 3 * GB * RP;       // [3][16][RP] decayed queries
    static constexpr int qf = q3 + 3 * GB * RP;       // [16][FP] q, k, c (two numbers) in 32 bits
    static constexpr int kf = qf + GB * FP * 4;
    static constexpr int ch = kf + GB * FP * 4;
    static constexpr int cl = ch + GB * FP * 4;
    static constexpr int p3 = cl + GB * FP * 4;       // [3][16][48 bytes] the weights P
    static constexpr int full = p3 + 3 * GB * 48;     // [DP] 2^c_15
    static constexpr int pair = full + DP * 4;        // [120] (i, j) of the pairs i > j
    static constexpr int v = pair + 256;              // [2][16][V * 2 + 16] values, then [3][16][V * 2 + 16] gates
    static __host__ __device__ int o(int V) { return v + 5 * GB * (V * 2 + 16); }      // [16][V + 4] floats
    static __host__ __device__ int bytes(int V) { return o(V) + GB * (V + 4) * 4; }
};

// OUT: outputs, from the start states or (a sequence of one chunk) the slot's state; else a chunk's own sum and decays.
// NU: groups of eight key channels that a warp prepares.
template <int DP, int NU, bool OUT>
__global__ void __launch_bounds__(512, 1) gla_block_kernel(GlaArgs a) {
    pdl_launch_dependents();
    typedef BlockSmem<DP> L;
    constexpr int RP = L::RP, FP = L::FP, KS = DP / 16;
    extern __shared__ __align__(128) uint8_t sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.x, D = a.D, V = a.V, HD = a.heads * D, HV = a.heads * V;
    const int b = blockIdx.y / a.n_chunks, chunk = blockIdx.y % a.n_chunks;
    const int VP = V * 2 + 16;                        // bytes of a row of values
    uint8_t* pair = sm + L::pair;
    if (OUT && tid < 120) {                     // pair u: i (i - 1) / 2 + j
        int i = 1;
        while ((i + 1) * i / 2 <= tid) i++;
        pair[2 * tid] = i; pair[2 * tid + 1] = tid - i * (i - 1) / 2;
    }
    for (int e = tid; e < (3 * GB * RP * 2) / 4; e += blockDim.x) ((uint32_t*)sm)[e] = 0u;      // channels past D stay zero
    for (int e = tid; e < (4 * GB * FP); e += blockDim.x) ((float*)(sm + L::qf))[e] = 0.f;
    for (int e = tid; e < 3 * GB * 12; e += blockDim.x) ((uint32_t*)(sm + L::p3))[e] = 0u;      // and so does P above the diagonal
    pdl_wait();
    const int s0 = a.seq_start[b], len = a.seq_start[b + 1] - s0;
    const int c0 = chunk * a.chunk_len, n = min(a.chunk_len, len - c0);
    if (n <= 0 || (!OUT && c0 + n == len)) return;
    const bool last = c0 + n == len;
    const int slot = s0 / a.chunk_len + b + chunk;    // a sequence's chunks lie from slot floor(seq_start / chunk_len) + b on
    float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)h * D * V;
    float* cst = a.chunk_state + ((size_t)slot * a.heads + h) * D * V;
    const int v0 = warp * 16;
    // this thread's part of S^T: rows v0 + g and v0 + g + 8, columns 8 m + 2 t and 8 m + 2 t + 1
    float S[DP / 8][4];
#pragma unroll
    for (int m = 0; m < DP / 8; m++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int d = m * 8 + 2 * t + (e & 1);
            S[m][e] = (OUT && d < D) ? (len > a.chunk_len ? cst : st)[(size_t)d * V + v0 + g + (e >> 1) * 8] : 0.f;
        }
    const bf16* proj = (const bf16*)a.proj + (size_t)(s0 + c0) * a.proj_stride;
    const float* decay = a.decay + (size_t)(s0 + c0) * HD + (size_t)h * D;
    // thread (channel of eight a warp, four tokens) prepares channel d of tokens 4 tg .. 4 tg + 3
    const int tg = lane >> 3, dsub = lane & 7;
    constexpr int UNITS = DP / 8;
    float rq[NU][4], rk[NU][4], rl[NU][4];            // the next block's, on their way
    auto fetch = [&](int u2, int t0) {
        const int unit = warp + u2 * nwarp, d = unit * 8 + dsub;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int tt = t0 + tg * 4 + e;
            const bool in = unit < UNITS && d < D && tt < n;
            rq[u2][e] = (OUT && in) ? __bfloat162float(proj[(size_t)tt * a.proj_stride + h * D + d]) * a.q_scale : 0.f;
            rk[u2][e] = in ? __bfloat162float(proj[(size_t)tt * a.proj_stride + HD + h * D + d]) : 0.f;
            rl[u2][e] = in ? decay[(size_t)tt * HD + d] : 0.f;
        }
    };
    double chunk_log[NU];                             // without OUT: the sum over the chunk (of channel d, in every token group)
#pragma unroll
    for (int u2 = 0; u2 < NU; u2++) chunk_log[u2] = 0.0;
    auto put = [&](int u2) {
        const int unit = warp + u2 * nwarp, d = unit * 8 + dsub;
        double c[4];
        c[0] = rl[u2][0]; c[1] = c[0] + rl[u2][1]; c[2] = c[1] + rl[u2][2]; c[3] = c[2] + rl[u2][3];
        double before = c[3];                         // inclusive sum over the token groups, then without this one
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += up;
        }
        const double all = __shfl_sync(0xffffffffu, before, 24 + dsub);
        before -= c[3];
        if (!OUT) chunk_log[u2] += all;
        if (unit >= UNITS || d >= D) return;
        if (tg == 0) ((float*)(sm + L::full))[d] = exp2_fast((float)all);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int tt = tg * 4 + e;
            const double ce = before + c[e];
            split3(rk[u2][e] * exp2_fast((float)(all - ce)), (bf16*)(sm + L::k3 + tt * RP) + d, GB * RP / 2);
            if (OUT) {
                const float hi = (float)ce;
                split3(rq[u2][e] * exp2_fast(hi), (bf16*)(sm + L::q3 + tt * RP) + d, GB * RP / 2);
                ((float*)(sm + L::qf))[tt * FP + d] = rq[u2][e];
                ((float*)(sm + L::kf))[tt * FP + d] = rk[u2][e];
                ((float*)(sm + L::ch))[tt * FP + d] = hi;
                ((float*)(sm + L::cl))[tt * FP + d] = (float)(ce - (double)hi);
            }
        }
    };
    auto load_v = [&](int t0) {                       // values, and the gates for when their outputs are there
        const int blk = t0 / GB;
        for (int c = tid; c < GB * V / 8; c += blockDim.x) {
            const int r = c / (V / 8), k = (c % (V / 8)) * 8;
            const bool ok = t0 + r < n;
            const bf16* src = proj + (ok ? (size_t)(t0 + r) * a.proj_stride + 2 * HD + h * V + k : 0);
            cp_async16(sm + L::v + (blk & 1) * GB * VP + r * VP + k * 2, src, ok);
            if (OUT) cp_async16(sm + L::v + (2 + blk % 3) * GB * VP + r * VP + k * 2, ok ? src + HV : src, ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // outputs of a block whose o lies in shared memory: a warp takes a token
    float* so = (float*)(sm + L::o(V));
    auto finish = [&](int t0) {
        for (int tt = warp; tt < GB && t0 + tt < n; tt += nwarp) {
            const size_t tok = (size_t)(s0 + c0 + t0 + tt);
            const uint8_t* gp = sm + L::v + (2 + t0 / GB % 3) * GB * VP + tt * VP;
            const int v8 = lane * 8;
            float y[8];
            uint4 gv = make_uint4(0, 0, 0, 0);
            float ss = 0.f;
            if (v8 < V) {
                gv = *(const uint4*)(gp + v8 * 2);
                *(float4*)y = *(const float4*)(so + tt * (V + 4) + v8);
                *(float4*)(y + 4) = *(const float4*)(so + tt * (V + 4) + v8 + 4);
#pragma unroll
                for (int e = 0; e < 8; e++) ss = fmaf(y[e], y[e], ss);
            }
            const float r = 1.f / sqrtf(warp_sum(ss) / (float)V + a.eps);
            if (v8 < V) {
                const uint32_t gu[4] = {gv.x, gv.y, gv.z, gv.w};
                uint32_t out[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float g0 = __uint_as_float(gu[e] << 16), g1 = __uint_as_float(gu[e] & 0xffff0000u);
                    const float w0 = a.norm_w != nullptr ? a.norm_w[v8 + 2 * e] : 1.f, w1 = a.norm_w != nullptr ? a.norm_w[v8 + 2 * e + 1] : 1.f;
                    out[e] = pack2(y[2 * e] * r * w0 * (g0 / (1.f + expf(-g0))), y[2 * e + 1] * r * w1 * (g1 / (1.f + expf(-g1))));
                }
                *(uint4*)((bf16*)a.out + tok * HV + (size_t)h * V + v8) = make_uint4(out[0], out[1], out[2], out[3]);
            }
        }
    };
    __syncthreads();                                  // the zeros are there
    load_v(0);
#pragma unroll
    for (int u2 = 0; u2 < NU; u2++) { fetch(u2, 0); put(u2); }
    int buf = 0;
    for (int t0 = 0; t0 < n; t0 += GB, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                              // this block's rows are there; so is the last block's o
        const bool more = t0 + GB < n;
        if (more) {
            load_v(t0 + GB);
#pragma unroll
            for (int u2 = 0; u2 < NU; u2++) fetch(u2, t0 + GB);
        }
        float o[2][4];
        uint32_t vt[4];                               // v^T: 16 channels x 16 tokens
        ldsm_x4_t(smem_addr(sm + L::v + buf * GB * VP + ((lane >> 4) * 8 + (lane & 7)) * VP + (v0 + ((lane >> 3) & 1) * 8) * 2), vt);
        if (OUT) {
            if (t0 > 0) finish(t0 - GB);
        }
        // the two halves of the work on FMA and tensor pipes, in opposite order in every other warp
        for (int half = 0; half < 2; half++) {
            if (((half ^ warp) & 1) == 0) {
                if (OUT) {
                    // ---- P: four threads a pair i > j (16 channels a step between them), two a token's own product
                    for (int u = tid; u < 512; u += blockDim.x) {
                        const bool own = u >= 480;
                        const int i = own ? (u - 480) >> 1 : pair[(u >> 2) * 2], j = own ? i : pair[(u >> 2) * 2 + 1];
                        const int part = own ? u & 1 : u & 3;
                        const float* qi = (const float*)(sm + L::qf) + i * FP;
                        const float* kj = (const float*)(sm + L::kf) + j * FP;
                        float s = 0.f;
                        if (own) {
                            for (int d = part * 4; d < DP; d += 8) {
                                const float4 x = *(const float4*)(qi + d), y = *(const float4*)(kj + d);
                                s = fmaf(x.x, y.x, s); s = fmaf(x.y, y.y, s); s = fmaf(x.z, y.z, s); s = fmaf(x.w, y.w, s);
                            }
                        } else {
                            const float* hi = (const float*)(sm + L::ch);
                            const float* lo = (const float*)(sm + L::cl);
#pragma unroll 2
                            for (int d = part * 4; d < DP; d += 16) {
                                const float4 x = *(const float4*)(qi + d), y = *(const float4*)(kj + d);
                                const float4 ih = *(const float4*)(hi + i * FP + d), jh = *(const float4*)(hi + j * FP + d);
                                const float4 il = *(const float4*)(lo + i * FP + d), jl = *(const float4*)(lo + j * FP + d);
                                s = fmaf(x.x * y.x, exp2_fast((ih.x - jh.x) + (il.x - jl.x)), s);
                                s = fmaf(x.y * y.y, exp2_fast((ih.y - jh.y) + (il.y - jl.y)), s);
                                s = fmaf(x.z * y.z, exp2_fast((ih.z - jh.z) + (il.z - jl.z)), s);
                                s = fmaf(x.w * y.w, exp2_fast((ih.w - jh.w) + (il.w - jl.w)), s);
                            }
                        }
                        s += __shfl_xor_sync(0xffffffffu, s, 1);
                        if (!own) s += __shfl_xor_sync(0xffffffffu, s, 2);      // (the same in every lane of a warp)
                        if (part == 0) split3(s, (bf16*)(sm + L::p3 + i * 48) + j, GB * 24);
                    }
                }
                continue;
            }
            if (OUT) {
                // ---- o^T [16 v][16 tokens] from the state before the block
#pragma unroll
                for (int x = 0; x < 2; x++) { o[x][0] = o[x][1] = o[x][2] = o[x][3] = 0.f; }
#pragma unroll
                for (int ks = 0; ks < KS; ks++) {
                    uint32_t s3[4][3], f[3][4], A[3][4];
                    split3(S[2 * ks][0], S[2 * ks][1], s3[0]); split3(S[2 * ks][2], S[2 * ks][3], s3[1]);
                    split3(S[2 * ks + 1][0], S[2 * ks + 1][1], s3[2]); split3(S[2 * ks + 1][2], S[2 * ks + 1][3], s3[3]);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
#pragma unroll
                        for (int e = 0; e < 4; e++) A[k][e] = s3[e][k];
                        ldsm_x4(smem_addr(sm + L::q3 + k * GB * RP + ((lane >> 4) * 8 + (lane & 7)) * RP + (ks * 16 + ((lane >> 3) & 1) * 8) * 2), f[k]);
                    }
#pragma unroll
                    for (int sum = 2; sum >= 0; sum--)
#pragma unroll
                        for (int k = 0; k <= sum; k++) { mma_bf16(o[0], A[k], f[sum - k][0], f[sum - k][1]); mma_bf16(o[1], A[k], f[sum - k][2], f[sum - k][3]); }
                }
            }
            // ---- the state after the block
            const float* full = (const float*)(sm + L::full);
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                float u[2][4];                        // (a product's sums are cut off, not rounded: the state is not added to in them)
#pragma unroll
                for (int e = 0; e < 4; e++) u[0][e] = u[1][e] = 0.f;
#pragma unroll
                for (int k = 2; k >= 0; k--) {
                    uint32_t f[4];
                    ldsm_x4_t(smem_addr(sm + L::k3 + k * GB * RP + (((lane >> 3) & 1) * 8 + (lane & 7)) * RP + (ks * 16 + (lane >> 4) * 8) * 2), f);
                    mma_bf16(u[0], vt, f[0], f[1]);
                    mma_bf16(u[1], vt, f[2], f[3]);
                }
#pragma unroll
                for (int x = 0; x < 2; x++) {
                    const float2 w = *(const float2*)(full + ks * 16 + x * 8 + 2 * t);
                    float* s = S[2 * ks + x];
                    s[0] = fmaf(s[0], w.x, u[x][0]); s[1] = fmaf(s[1], w.y, u[x][1]);
                    s[2] = fmaf(s[2], w.x, u[x][2]); s[3] = fmaf(s[3], w.y, u[x][3]);
                }
            }
        }
        __syncthreads();                              // P is there; the block's q, k and decays have been read
        if (more) {
#pragma unroll
            for (int u2 = 0; u2 < NU; u2++) put(u2);
        }
        if (OUT) {
            if (__any_sync(0xffffffffu, ((not_finite(vt[0]) | not_finite(vt[1]) | not_finite(vt[2]) | not_finite(vt[3])) & 0x80008000u) != 0)) {
                // a weight of 0 times such a value of a later token would be NaN: token by token, up to the output's own
#pragma unroll 1
                for (int j = 0; j < GB; j++) {
                    const int from = (lane & ~3) | ((j & 7) >> 1);
                    const uint32_t a0 = __shfl_sync(0xffffffffu, j < 8 ? vt[0] : vt[2], from), a1 = __shfl_sync(0xffffffffu, j < 8 ? vt[1] : vt[3], from);
                    const float vj[2] = {__uint_as_float((j & 1) ? a0 & 0xffff0000u : a0 << 16), __uint_as_float((j & 1) ? a1 & 0xffff0000u : a1 << 16)};
#pragma unroll
                    for (int x = 0; x < 2; x++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int i = x * 8 + 2 * t + (e & 1);
                            const bf16* p = (const bf16*)(sm + L::p3 + i * 48) + j;
                            if (j <= i) o[x][e] = fmaf(__bfloat162float(p[0]) + (__bfloat162float(p[GB * 24]) + __bfloat162float(p[2 * GB * 24])), vj[e >> 1], o[x][e]);
                        }
                }
            } else {
#pragma unroll
            for (int k = 2; k >= 0; k--) {
                uint32_t f[4];
                ldsm_x4(smem_addr(sm + L::p3 + k * GB * 48 + ((lane >> 4) * 8 + (lane & 7)) * 48 + ((lane >> 3) & 1) * 16), f);
                mma_bf16(o[0], vt, f[0], f[1]);
                mma_bf16(o[1], vt, f[2], f[3]);
            }
            }
#pragma unroll
            for (int x = 0; x < 2; x++)
#pragma unroll
                for (int e = 0; e < 4; e++) so[(x * 8 + 2 * t + (e & 1)) * (V + 4) + v0 + g + (e >> 1) * 8] = o[x][e];
        }
    }
    if (OUT) {
        __syncthreads();
        finish((n - 1) / GB * GB);
        if (!last) return;
    } else if (tg == 0) {
#pragma unroll
        for (int u2 = 0; u2 < NU; u2++) {
            const int unit = warp + u2 * nwarp, d = unit * 8 + dsub;
            if (unit < UNITS && d < D) a.chunk_decay[((size_t)slot * a.heads + h) * D + d] = exp2_fast((float)chunk_log[u2]);
        }
    }
    float* to = OUT ? st : cst;
#pragma unroll
    for (int m = 0; m < DP / 8; m++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int d = m * 8 + 2 * t + (e & 1);
            if (d < D) to[(size_t)d * V + v0 + g + (e >> 1) * 8] = S[m][e];
        }
}

// Every chunk's own sum becomes the state before the chunk (sequences of one chunk keep theirs in the slot).
__global__ void __launch_bounds__(256) gla_block_fold_kernel(GlaArgs a) {
    pdl_launch_dependents();
    const int b = blockIdx.y, V = a.V;
    const size_t per = (size_t)a.heads * a.D * V;
    const size_t e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= per) return;
    const int hd = (int)(e / V);                      // h * D + d
    pdl_wait();
    const int s0 = a.seq_start[b], len = a.seq_start[b + 1] - s0, n = (len + a.chunk_len - 1) / a.chunk_len, slot = s0 / a.chunk_len + b;
    if (n <= 1) return;
    const float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + e;
    float4 s = make_float4(st[0], st[1], st[2], st[3]);
    float* E = a.chunk_state + (size_t)slot * per + e;
    const float* P = a.chunk_decay + (size_t)slot * a.heads * a.D + hd;
    for (int c0 = 0; c0 < n; c0 += 8) {               // eight chunks' sums on their way together; the last one has none
        float4 x[8]; float p[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (c0 + u < n - 1) { x[u] = *(const float4*)(E + (c0 + u) * per); p[u] = P[(size_t)(c0 + u) * a.heads * a.D]; }
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (c0 + u < n) {
                *(float4*)(E + (c0 + u) * per) = s;
                if (c0 + u < n - 1) { s.x = fmaf(p[u], s.x, x[u].x); s.y = fmaf(p[u], s.y, x[u].y); s.z = fmaf(p[u], s.z, x[u].z); s.w = fmaf(p[u], s.w, x[u].w); }
            }
    }
}

template <typename T, typename TO>
__global__ void gla_gate_norm_kernel(GlaArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= (long long)a.n_tokens * a.heads) return;
    const int t = (int)(item / a.heads), h = (int)(item % a.heads);
    const int V = a.V, HV = a.heads * V, HD = a.heads * a.D;
    const float* y = a.y + (size_t)t * HV + (size_t)h * V;
    float sq = 0.f;
    for (int v = lane; v < V; v += 32) sq = fmaf(y[v], y[v], sq);
    const float r = 1.f / sqrtf(warp_sum(sq) / (float)V + a.eps);
    const T* g = (const T*)a.proj + (size_t)t * a.proj_stride + 2 * HD + HV + (size_t)h * V;
    TO* o = (TO*)a.out + (size_t)t * HV + (size_t)h * V;
    for (int v = lane; v < V; v += 32) {
        const float gv = to_f<T>(g[v]);
        o[v] = from_f<TO>(y[v] * r * (a.norm_w != nullptr ? a.norm_w[v] : 1.f) * (gv / (1.f + expf(-gv))));
    }
}

static int check(const GlaArgs& a) {
    if (a.heads <= 0 || a.D <= 0 || a.V <= 0 || (a.rank <= 0 && a.head_decay == nullptr)) return tb_refuse("gla: heads=%d D=%d V=%d rank=%d", a.heads, a.D, a.V, a.rank);
    if (a.D > 256) return tb_refuse("gla: %d key channels per head; the scan keeps up to 256", a.D);
    if (a.heads > 65535 || a.batch > 65535) return tb_refuse("gla: %d heads x %d sequences exceed one launch", a.heads, a.batch);
    return 0;
}

extern "C" int tb_gla_decay(const GlaArgs* args, cudaStream_t stream) {
    if (args->n_tokens <= 0) return 0;
    if (check(*args)) return -1;
    if (args->rank > 256) return tb_refuse("gla: a decay of rank %d; the kernel takes up to 256", args->rank);
    const int HD = args->heads * args->D;
    tb_launch(gla_decay_kernel, dim3((args->n_tokens + GLA_DECAY_TOK - 1) / GLA_DECAY_TOK, (HD + 255) / 256), dim3(256),
              (size_t)GLA_DECAY_TOK * args->rank * sizeof(float), stream, *args);
    return tb_launch_status();
}

extern "C" int tb_gla_scan(const GlaArgs* args, int dtype, cudaStream_t stream) {
    if (args->n_tokens <= 0 || args->batch <= 0) return 0;
    if (check(*args)) return -1;
    const GlaArgs& a = *args;
    int dpt = 1;
    while (dpt * GLA_WARPS < a.D) dpt <<= 1;
    const bool chunks = a.n_chunks > 1;
    if (chunks && (a.chunk_len <= 0 || a.chunk_state == nullptr || a.chunk_decay == nullptr || (long long)a.batch * a.n_chunks > 65535))
        return tb_refuse("gla: %d chunks of %d tokens need their scratch (and batch x chunks <= 65535)", a.n_chunks, a.chunk_len);
    dim3 grid((a.V + GLA_VT - 1) / GLA_VT, a.heads, chunks ? a.batch * a.n_chunks : a.batch);
#define GLA_SCAN_M(N, M) TB_DISPATCH_1(dtype, T, tb_launch(gla_scan_kernel<T, N, M>, dim3(grid), dim3(GLA_WARPS * 32), 0, stream, a))
#define GLA_SCAN(N) do { if (mode == 0) GLA_SCAN_M(N, 0); else if (mode == 1) GLA_SCAN_M(N, 1); else GLA_SCAN_M(N, 2); } while (0)
    for (int pass = 0; pass < (chunks ? 3 : 1); pass++) {
        if (chunks && pass == 1) {
            const long long n = (long long)a.batch * a.heads * a.D * a.V;
            tb_launch(gla_fold_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, a);
        } else {
            const int mode = chunks ? (pass == 0 ? 1 : 2) : 0;
            switch (dpt) {
            case 1: GLA_SCAN(1); break;
            case 2: GLA_SCAN(2); break;
            case 4: GLA_SCAN(4); break;
            case 8: GLA_SCAN(8); break;
            case 16: GLA_SCAN(16); break;
            default: GLA_SCAN(32); break;
            }
        }
        const int st = tb_launch_status();
        if (st) return st;
    }
    return 0;
}

// How a step of whole prompts is cut in time: chunks of at least 64 tokens, as many as fill the GPU once (two CTAs an SM)
// and no more, so that no CTA waits for a second round.
extern "C" int tb_gla_plan(int heads, int V, int batch, int max_seq_len, int sms, int* chunk_len) {
    const long long ctas = (long long)((V + GLA_VT - 1) / GLA_VT) * heads * batch;
    int want = (int)((2LL * sms) / ctas);
    int most = max_seq_len / 64;
    if (want > most) want = most;
    if (want <= 1) { *chunk_len = 0; return 1; }
    int len = (max_seq_len + want - 1) / want;
    len = (len + GLA_TT - 1) / GLA_TT * GLA_TT;
    *chunk_len = len;
    return (max_seq_len + len - 1) / len;
}

// dtype: of the gate's columns; out_dtype: of the output.
extern "C" int tb_gla_gate_norm(const GlaArgs* args, int dtype, int out_dtype, cudaStream_t stream) {
    if (args->n_tokens <= 0) return 0;
    if (check(*args)) return -1;
    const long long items = (long long)args->n_tokens * args->heads;
    if (dtype == out_dtype) {
        TB_DISPATCH_1(dtype, T, tb_launch(gla_gate_norm_kernel<T, T>, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, *args));
    } else if (dtype == TB_F32 && out_dtype == TB_BF16) {
        tb_launch(gla_gate_norm_kernel<float, bf16>, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, *args);
    } else return tb_refuse("gla: gate dtype %d, output dtype %d", dtype, out_dtype);
    return tb_launch_status();
}

// Whether the block form takes these sizes: bfloat16, rows in whole 16-byte pieces, every warp's 16 value channels whole,
// at least half as many warps as groups of eight key channels.
extern "C" int tb_gla_blocks_takes(int dtype, int D, int V) {
    return dtype == TB_BF16 && D >= 8 && D <= 128 && D % 8 == 0 && V >= 16 && V <= 256 && V % 16 == 0 && (D <= 64 ? 8 : 16) <= 2 * (V / 16);
}

// Tokens per chunk: the length whose rounds of CTAs (one a SM) take least, in the time of a token of the second launch (0.6 us):
// a token costs a third of that in the first launch, a CTA's start and end 23 and 20, the fold 13.
extern "C" int tb_gla_blocks_chunk(int heads, int batch, int n_tokens, int max_seq_len, int sms) {
    auto rounds = [&](long long ctas) { return (double)((ctas + sms - 1) / sms); };
    int best = (max_seq_len + GB - 1) / GB * GB;
    double least = rounds((long long)heads * batch) * (best + 23);
    for (int len = 2 * GB; len < max_seq_len; len += GB) {
        const long long chunks = (long long)batch * ((max_seq_len + len - 1) / len), most = n_tokens / len + batch;
        const double cost = rounds(heads * (chunks < most ? chunks : most)) * (1.33 * len + 43) + 13;
        if (cost < least) { least = cost; best = len; }
    }
    return best;
}

// Scratch slots of a step: every sequence's chunks lie from slot floor(seq_start / chunk_len) + its index on.
extern "C" int tb_gla_blocks_slots(int batch, int n_tokens, int chunk_len) { return n_tokens / chunk_len + batch; }

template <int DP, int NU>
static int run_blocks(const GlaArgs& a, cudaStream_t stream) {
    const int smem = BlockSmem<DP>::bytes(a.V);
    const dim3 grid(a.heads, a.batch * a.n_chunks), block(a.V * 2);
    auto launch = [&](void (*kern)(GlaArgs)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BlockSmem<DP>::bytes(256));
        if (e != cudaSuccess) return (int)e;
        tb_launch(kern, grid, block, smem, stream, a);
        return tb_launch_status();
    };
    if (a.n_chunks == 1) return launch(gla_block_kernel<DP, NU, true>);
    int st = launch(gla_block_kernel<DP, NU, false>);
    if (st) return st;
    const long long quads = (long long)a.heads * a.D * a.V / 4;
    tb_launch(gla_block_fold_kernel, dim3((unsigned)((quads + 255) / 256), a.batch), dim3(256), 0, stream, a);
    st = tb_launch_status();
    if (st) return st;
    return launch(gla_block_kernel<DP, NU, true>);
}

// n_chunks: of the longest sequence; chunk_state [slots][heads * D * V] and chunk_decay [slots][heads * D] if more than one.
extern "C" int tb_gla_blocks(const GlaArgs* args, int dtype, cudaStream_t stream) {
    GlaArgs a = *args;
    if (a.n_tokens <= 0 || a.batch <= 0) return 0;
    if (check(a)) return -1;
    if (!tb_gla_blocks_takes(dtype, a.D, a.V) || a.head_decay != nullptr || a.rank > 256)
        return tb_refuse("gla: the block form takes bfloat16, D up to 128 and V up to 256 in whole pieces, got D=%d V=%d", a.D, a.V);
    if (((uintptr_t)a.proj & 15) || a.proj_stride % 8 || ((uintptr_t)a.out & 15) || ((uintptr_t)a.chunk_state & 15))
        return tb_refuse("gla: the block form needs 16-byte aligned rows");
    if (a.chunk_len < GB || a.chunk_len % GB || a.n_chunks < 1 || (long long)a.batch * a.n_chunks > 65535 ||
        (a.n_chunks > 1 && (a.chunk_state == nullptr || a.chunk_decay == nullptr)))
        return tb_refuse("gla: %d chunks of %d tokens need their scratch (and batch x chunks <= 65535)", a.n_chunks, a.chunk_len);
    a.log2_decay = 1;
    int st = tb_gla_decay(&a, stream);
    if (st) return st;
    const bool one = a.V / 16 >= (a.D <= 64 ? 8 : 16);
    if (a.D <= 64) return one ? run_blocks<64, 1>(a, stream) : run_blocks<64, 2>(a, stream);
    return one ? run_blocks<128, 1>(a, stream) : run_blocks<128, 2>(a, stream);
}
