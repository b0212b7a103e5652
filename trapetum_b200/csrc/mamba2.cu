// A selective state-space mixer (the Mamba-2 recurrence) between its input and output products.
//
// The input product gives a row [z: inner | xBC: channels] per token in the compute dtype and the step sizes
// [dt: heads] in 32-bit (they enter an exponential), inner = heads * P, channels = inner + 2 * groups * N.
// Three kernels:
//
//   tb_mamba2_conv       u = silu(bias + sum_j w[c][j] * in[t - (taps-1) + j][c]) over the token's own sequence,
//                        rows before the step's first token come from the sequence's state (zeros at its start);
//                        then the state takes the last taps-1 inputs.  One token per sequence: one launch does both.
//   tb_mamba2_scan       per head h (group g = h / (heads / groups)), with dt = softplus(dt_raw + dt_bias):
//                          S <- exp(-exp(A_log[h]) dt) S + dt * x_t B_t^T      S is [P][N]
//                          y_t = S C_t + D[h] x_t
//                        sequential over a sequence's tokens, S read from and written back to the state.  Where few
//                        long prompts would leave most SMs idle, a prompt is cut into chunks: one launch runs the
//                        recurrence of every chunk but the last from zero and keeps its end state and the product of
//                        its decays, a second launch starts every chunk from what the chunks before it left
//                        (S_c = D_(c-1) S_(c-1) + E_(c-1), folded by the chunk itself) and writes y.  Twice the
//                        arithmetic, chunks times the parallelism; the same sums in another order.
//   tb_mamba2_chunks     the same for prompts in bfloat16, as matrix products over chunks of 128 tokens (mma.sync; see
//                        "Prompts as products" below)
//   tb_mamba2_gate_norm  out = groupnorm(y * silu(z)) * w, the norm over `norm_groups` equal parts of a row.
//
// The state of a sequence is one 32-bit row: [heads][P][N] of S, then [taps-1][channels] of conv inputs
// (oldest first).  The convolution and its silu work on the compute dtype's values with 32-bit sums; softplus,
// the decay, S, y and the gated norm are 32-bit throughout.
#include "common.cuh"

TB_EXPORT_ERROR()

__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

struct Mamba2Args {
    const void* proj; long long proj_stride;      // [tokens][inner + channels], compute dtype
    const float* dt; long long dt_stride;          // [tokens][heads], the step sizes before bias and softplus,
    int dt_splits; long long dt_split_stride;      // as dt_splits partial sums (added in split order)
    int heads, P, N, groups, taps, norm_groups;
    const void* conv_w; const void* conv_b;        // [channels][taps], [channels]   (weights' dtype)
    const void* dt_bias; const void* A_log; const void* D;   // [heads]
    const void* norm_w;                            // [inner]
    float eps;
    float* state; long long state_stride;          // [slots][state_stride]
    const int* seq_start; const int* token_seq; const int* slot_ids;
    void* xbc;                                     // [tokens][channels], compute dtype (conv output)
    float* y;                                      // [tokens][inner]
    void* out;                                     // [tokens][inner], compute dtype
    int batch, n_tokens;
    // a long prompt cut into chunks that run side by side (see mamba2_scan_kernel): end states [batch][n_chunks][heads*P*N],
    // decay products [batch][n_chunks][heads], tokens per chunk (a multiple of the tile), chunks per sequence
    float* chunk_state; float* chunk_decay; int chunk_len; int n_chunks;
};

// The argument block's size, for the Python mirror's check.
extern "C" int tb_mamba2_args_bytes() { return (int)sizeof(Mamba2Args); }

// ---------------------------------------------------------------------------------------------------------
template <typename T, typename TW>
__global__ void mamba2_conv_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int inner = a.heads * a.P, ch = inner + 2 * a.groups * a.N;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t = blockIdx.x;
    if (c >= ch) return;
    const int b = a.token_seq[t];
    const int i = t - a.seq_start[b];                               // the token's index among the step's tokens of its sequence
    const float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)a.heads * a.P * a.N;
    const T* in = (const T*)a.proj + inner + c;
    const TW* w = (const TW*)a.conv_w + (size_t)c * a.taps;
    float acc = to_f<TW>(((const TW*)a.conv_b)[c]);
    for (int j = 0; j < a.taps; j++) {
        const int d = i - (a.taps - 1) + j;                          // index among the step's tokens; negative: from the state
        const float v = d >= 0 ? to_f<T>(in[(size_t)(t - (a.taps - 1) + j) * a.proj_stride])
                               : st[(size_t)(a.taps - 1 + d) * ch + c];
        acc += to_f<TW>(w[j]) * v;
    }
    ((T*)a.xbc)[(size_t)t * ch + c] = from_f<T>(silu_f(acc));
}

// Four taps in bfloat16: a thread takes four neighbouring channels of eight tokens in a row, whose inputs are on their way
// together, 8 bytes a load: 18 us for 2,048 tokens x 4,352 channels, cold (a thread per number: 76; eight channels a thread,
// whose registers leave half the warps: 26; its 36 MB are 5.4).
__device__ __forceinline__ void unpack4(const uint2& v, float* f) {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *(uint32_t*)&h;
}
template <int CONV_TOK>
__global__ void __launch_bounds__(128, 6) mamba2_conv4_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    const int inner = a.heads * a.P, ch = inner + 2 * a.groups * a.N;
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    const int t0 = blockIdx.x * CONV_TOK, nt = min(CONV_TOK, a.n_tokens - t0);
    if (c >= ch) return;
    float w[4][4], bias[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float4 x = *(const float4*)((const float*)a.conv_w + (size_t)(c + e) * 4);
        w[e][0] = x.x; w[e][1] = x.y; w[e][2] = x.z; w[e][3] = x.w;
        bias[e] = ((const float*)a.conv_b)[c + e];
    }
    pdl_wait();
    int b = a.token_seq[t0], i = t0 - a.seq_start[b];
    const bf16* in = (const bf16*)a.proj + inner + c;
    uint2 rows[CONV_TOK + 3];                        // tokens t0 - 3 .. t0 + 7 (earlier ones only of the same sequence)
#pragma unroll
    for (int r = 0; r < CONV_TOK + 3; r++) {
        rows[r] = make_uint2(0, 0);
        if (r < 3 ? i >= 3 - r : r - 3 < nt) rows[r] = *(const uint2*)(in + (size_t)(t0 + r - 3) * a.proj_stride);
    }
    float h[3][4];                                   // the three inputs before the token
    auto from_state = [&](int k, int row) {          // h[k] from row `row` of the sequence's state
        const float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)a.heads * a.P * a.N + (size_t)row * ch + c;
#pragma unroll
        for (int e = 0; e < 4; e++) h[k][e] = st[e];
    };
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (i >= 3 - k) unpack4(rows[k], h[k]);
        else from_state(k, k + i);                   // index i - 3 + k < 0: row 3 + (i - 3 + k) of the state
    }
#pragma unroll
    for (int r = 0; r < CONV_TOK; r++) {
        if (r >= nt) break;
        if (r > 0) {
            const int nb = a.token_seq[t0 + r];
            if (nb != b) {                           // the next sequence's first token
                b = nb;
#pragma unroll
                for (int k = 0; k < 3; k++) from_state(k, k);
            }
        }
        float cur[4], acc[4];
        unpack4(rows[r + 3], cur);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            acc[e] = bias[e] + w[e][0] * h[0][e];
            acc[e] += w[e][1] * h[1][e];
            acc[e] += w[e][2] * h[2][e];
            acc[e] = silu_f(acc[e] + w[e][3] * cur[e]);
            h[0][e] = h[1][e]; h[1][e] = h[2][e]; h[2][e] = cur[e];
        }
        *(uint2*)((bf16*)a.xbc + (size_t)(t0 + r) * ch + c) = make_uint2(pack2(acc[0], acc[1]), pack2(acc[2], acc[3]));
    }
}

// After a step of several tokens: the state keeps the last taps-1 inputs of each sequence.  One thread owns a
// (sequence, channel) column and shifts it in ascending order, so the update is safe in place.
template <typename T>
__global__ void mamba2_conv_state_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int inner = a.heads * a.P, ch = inner + 2 * a.groups * a.N;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int b = blockIdx.x;
    if (c >= ch) return;
    const int s0 = a.seq_start[b], n = a.seq_start[b + 1] - s0, keep = a.taps - 1;
    float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)a.heads * a.P * a.N;
    const T* in = (const T*)a.proj + inner + c;
    for (int j = 0; j < keep; j++) {
        const int d = n - keep + j;                                  // index among the step's tokens
        st[(size_t)j * ch + c] = d >= 0 ? to_f<T>(in[(size_t)(s0 + d) * a.proj_stride]) : st[(size_t)(j + n) * ch + c];
    }
}

// One token per sequence: convolution and state shift by the thread that owns the column.
template <typename T, typename TW>
__global__ void mamba2_conv_step_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int inner = a.heads * a.P, ch = inner + 2 * a.groups * a.N;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int b = blockIdx.x;                                        // token b belongs to sequence b
    if (c >= ch) return;
    const int keep = a.taps - 1;
    float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)a.heads * a.P * a.N;
    const TW* w = (const TW*)a.conv_w + (size_t)c * a.taps;
    const float cur = to_f<T>(((const T*)a.proj)[(size_t)b * a.proj_stride + inner + c]);
    float acc = to_f<TW>(((const TW*)a.conv_b)[c]);
    for (int j = 0; j < keep; j++) {
        const float v = st[(size_t)j * ch + c];
        acc += to_f<TW>(w[j]) * v;
        if (j > 0) st[(size_t)(j - 1) * ch + c] = v;
    }
    acc += to_f<TW>(w[keep]) * cur;
    if (keep > 0) st[(size_t)(keep - 1) * ch + c] = cur;
    ((T*)a.xbc)[(size_t)b * ch + c] = from_f<T>(silu_f(acc));
}

// ---------------------------------------------------------------------------------------------------------
// The recurrence.  A CTA owns (sequence, head, PT values of P): thread (pl, ns) keeps the states S[p][n] of two
// neighbouring p with n = (k * 8 + ns) * 4 + e (k < NV, e < 4) in registers, so that the eight threads of a pair read
// B and C of a token as eight neighbouring 16-byte words of shared memory (no bank conflict) and use each word for
// both p.  B, C,
// x, dt and the decay of TT tokens at a time are staged in shared memory; the next tile's values are requested into
// registers before this tile's steps run, so that the loads' latency hides behind the recurrence.  A thread's parts of
// the 2 TT outputs stay in registers and are added over the eight threads once per tile, off the dependency chain, by
// a butterfly in which every thread hands over half of what it holds at each of the three stages.
#define SCAN_NS 8
#define SCAN_TT 16
#define SCAN_PP 2

template <typename T> struct Chunk8;                                 // eight neighbouring values of the compute dtype
template <> struct Chunk8<bf16> {
    uint4 v;
    __device__ __forceinline__ void load(const bf16* p) { v = *(const uint4*)p; }
    __device__ __forceinline__ void zero() { v = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void store(float* d) const {
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float f[8];
#pragma unroll
        for (int i = 0; i < 4; i++) { f[2 * i] = __uint_as_float(u[i] << 16); f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
        *(float4*)d = make_float4(f[0], f[1], f[2], f[3]);
        *(float4*)(d + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
};
template <> struct Chunk8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = *(const float4*)p; b = *(const float4*)(p + 4); }
    __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void store(float* d) const { *(float4*)d = a; *(float4*)(d + 4) = b; }
};

// VEC8: N is a multiple of 8 and the rows of B and C start on 16-byte boundaries.
// MODE 0: a whole sequence per CTA.  MODE 1: a chunk from zero (the first chunk: from the sequence's state, of which it
// also leaves a copy in the last chunk's slot, which is otherwise unused), end state and decay product kept, no y;
// the last chunk of a sequence does nothing.  MODE 2: a chunk from the folded states of the chunks before it, y
// written; the last chunk writes the sequence's state (only it reads it in this launch: a sequence of one chunk).
template <typename T, typename TW, int NV, int PT, bool VEC8, int MODE>
__global__ void __launch_bounds__(SCAN_NS * PT / SCAN_PP) mamba2_scan_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    constexpr int NP = NV * 32;                                      // padded state size (zeros beyond N)
    constexpr int THREADS = SCAN_NS * PT / SCAN_PP;
    constexpr int CHUNKS = SCAN_TT * 2 * NP / 8;                     // 8-value chunks of B and C in a tile
    constexpr int CPT = (CHUNKS + THREADS - 1) / THREADS;            // chunks a thread fetches
    constexpr int XPT = SCAN_TT * PT / THREADS;                      // x values a thread fetches (4)
    extern __shared__ __align__(16) float sh[];                      // [TT][NP] B, [TT][NP] C, [TT][PT] x, [TT][2] dt and decay
    const int N = a.N, P = a.P, H = a.heads;
    const int inner = H * P, ch = inner + 2 * a.groups * N;
    const int b = MODE == 0 ? blockIdx.z : blockIdx.z / a.n_chunks, chunk = MODE == 0 ? 0 : blockIdx.z % a.n_chunks;
    const int h = blockIdx.y, p0 = blockIdx.x * PT;
    const int g = h / (H / a.groups);
    const int ns = threadIdx.x % SCAN_NS, pl = threadIdx.x / SCAN_NS;
    const int p = p0 + pl * SCAN_PP;                                 // this thread's first p
    float* sB = sh;
    float* sC = sh + SCAN_TT * NP;
    float* sx = sC + SCAN_TT * NP;
    float* sdt = sx + SCAN_TT * PT;
    const float A = -expf(to_f<TW>(((const TW*)a.A_log)[h]));
    const float Dh = to_f<TW>(((const TW*)a.D)[h]);
    const float dtb = to_f<TW>(((const TW*)a.dt_bias)[h]);
    pdl_wait();
    int s0 = a.seq_start[b], s1 = a.seq_start[b + 1];
    bool last = true;
    if (MODE != 0) {                                                 // this CTA's chunk of the sequence
        const int end = s1;
        s0 += chunk * a.chunk_len;
        if (s0 >= end) return;                                       // (the same in every thread)
        s1 = min(end, s0 + a.chunk_len);
        last = s1 == end;
        if (MODE == 1 && last) return;
    }
    float* S = a.state + (size_t)a.slot_ids[b] * a.state_stride + (size_t)h * P * N;
    const size_t hpn = (size_t)H * P * N;
    float* E = MODE == 0 ? nullptr : a.chunk_state + (size_t)b * a.n_chunks * hpn + (size_t)h * P * N;   // chunk 0's slot, this head
    float s[SCAN_PP][NV][4];
    auto each = [&](auto&& f) {                                      // f(j, k, e, offset in [P][N]) for the states this thread owns
#pragma unroll
        for (int j = 0; j < SCAN_PP; j++)
#pragma unroll
            for (int k = 0; k < NV; k++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int n = (k * SCAN_NS + ns) * 4 + e;
                    if (p + j < P && n < N) f(j, k, e, (size_t)(p + j) * N + n);
                }
    };
#pragma unroll
    for (int j = 0; j < SCAN_PP; j++)
#pragma unroll
        for (int k = 0; k < NV; k++)
#pragma unroll
            for (int e = 0; e < 4; e++) s[j][k][e] = 0.f;
    if (MODE == 0 || (MODE == 2 && chunk == 0 && last)) {
        each([&](int j, int k, int e, size_t o) { s[j][k][e] = S[o]; });
    } else if (MODE == 1) {
        if (chunk == 0) each([&](int j, int k, int e, size_t o) { s[j][k][e] = S[o]; E[(size_t)(a.n_chunks - 1) * hpn + o] = S[o]; });
    } else if (chunk == 0) {
        each([&](int j, int k, int e, size_t o) { s[j][k][e] = E[(size_t)(a.n_chunks - 1) * hpn + o]; });
    } else {
        for (int c = 0; c < chunk; c++) {                            // the first chunk's end state holds the sequence's state already
            const float d = c == 0 ? 0.f : a.chunk_decay[((size_t)b * a.n_chunks + c) * H + h];
            const float* Ec = E + (size_t)c * hpn;
            each([&](int j, int k, int e, size_t o) { s[j][k][e] = d * s[j][k][e] + Ec[o]; });
        }
    }
    float decay = 1.f;
    const T* xbc = (const T*)a.xbc;

    Chunk8<T> pre[VEC8 ? CPT : 1];
    float pre_x[XPT], pre_dt = 0.f;
    auto fetch = [&](int tb) {                                       // the tile that starts at token tb, into registers
        const int nt = min(SCAN_TT, s1 - tb);
        if (VEC8) {
#pragma unroll
            for (int l = 0; l < CPT; l++) {
                const int c = threadIdx.x + l * THREADS;
                const int tt = c / (2 * NP / 8), r = c % (2 * NP / 8);
                const int n8 = (r % (NP / 8)) * 8;
                pre[l].zero();
                if (c < CHUNKS && tt < nt && n8 < N)
                    pre[l].load(xbc + (size_t)(tb + tt) * ch + inner + g * N + (r >= NP / 8 ? a.groups * N : 0) + n8);
            }
        }
#pragma unroll
        for (int l = 0; l < XPT; l++) {
            const int i = threadIdx.x + l * THREADS;
            const int tt = i / PT, pp = p0 + i % PT;
            pre_x[l] = (tt < nt && pp < P) ? to_f<T>(xbc[(size_t)(tb + tt) * ch + h * P + pp]) : 0.f;
        }
        if (threadIdx.x < nt) {
            const float* q = a.dt + (size_t)(tb + threadIdx.x) * a.dt_stride + h;
            pre_dt = q[0];
            for (int sp = 1; sp < a.dt_splits; sp++) pre_dt += q[(size_t)sp * a.dt_split_stride];
        }
    };
    auto commit = [&](int tb) {                                      // registers (or, without VEC8, memory) to shared memory
        const int nt = min(SCAN_TT, s1 - tb);
        if (VEC8) {
#pragma unroll
            for (int l = 0; l < CPT; l++) {
                const int c = threadIdx.x + l * THREADS;
                const int tt = c / (2 * NP / 8), r = c % (2 * NP / 8);
                if (c < CHUNKS) pre[l].store((r >= NP / 8 ? sC : sB) + tt * NP + (r % (NP / 8)) * 8);
            }
        } else {
            for (int i = threadIdx.x; i < nt * NP; i += THREADS) {
                const int tt = i / NP, n = i % NP;
                const T* row = xbc + (size_t)(tb + tt) * ch + inner + g * N;
                sB[i] = n < N ? to_f<T>(row[n]) : 0.f;
                sC[i] = n < N ? to_f<T>(row[a.groups * N + n]) : 0.f;
            }
        }
#pragma unroll
        for (int l = 0; l < XPT; l++) sx[threadIdx.x + l * THREADS] = pre_x[l];
        if (threadIdx.x < nt) {
            const float dt = softplus_f(pre_dt + dtb);
            sdt[2 * threadIdx.x] = dt;
            sdt[2 * threadIdx.x + 1] = expf(A * dt);
        }
    };

    if (s0 < s1) fetch(s0);
    for (int tb = s0; tb < s1; tb += SCAN_TT) {
        const int nt = min(SCAN_TT, s1 - tb);
        __syncthreads();                                             // the last tile's steps have read shared memory
        commit(tb);
        __syncthreads();
        if (tb + SCAN_TT < s1) fetch(tb + SCAN_TT);
        float yp[SCAN_TT * SCAN_PP];                                 // yp[tt * 2 + j]: this thread's part of y of token tt, p + j
#pragma unroll
        for (int tt = 0; tt < SCAN_TT; tt++) {
            yp[2 * tt] = yp[2 * tt + 1] = 0.f;
            if (tt < nt) {                                           // the same in every thread of the CTA
                const float dec = sdt[2 * tt + 1], dt = sdt[2 * tt];
                if (MODE == 1) decay *= dec;
                const float dx0 = dt * sx[tt * PT + pl * SCAN_PP], dx1 = dt * sx[tt * PT + pl * SCAN_PP + 1];
                const float4* Bt = (const float4*)(sB + tt * NP);
                const float4* Ct = (const float4*)(sC + tt * NP);
                float y0[4] = {0.f, 0.f, 0.f, 0.f}, y1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < NV; k++) {
                    const float4 bv = Bt[k * SCAN_NS + ns], cv = Ct[k * SCAN_NS + ns];
                    const float bb[4] = {bv.x, bv.y, bv.z, bv.w}, cc[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        s[0][k][e] = dec * s[0][k][e] + dx0 * bb[e]; y0[e] += s[0][k][e] * cc[e];
                        s[1][k][e] = dec * s[1][k][e] + dx1 * bb[e]; y1[e] += s[1][k][e] * cc[e];
                    }
                }
                yp[2 * tt] = (y0[0] + y0[1]) + (y0[2] + y0[3]);
                yp[2 * tt + 1] = (y1[0] + y1[1]) + (y1[2] + y1[3]);
            }
        }
        if (MODE != 1) {                                             // (end states only: no outputs)
        // the eight threads of a pair add their parts: at each stage a thread keeps one half of its values and hands
        // the other to its partner; thread ns ends with the sums of tokens 2 ns and 2 ns + 1, both p
#pragma unroll
        for (int o = SCAN_NS / 2, half = SCAN_TT * SCAN_PP / 2; o > 0; o >>= 1, half >>= 1) {
            const bool up = (ns & o) != 0;
#pragma unroll
            for (int i = 0; i < SCAN_TT * SCAN_PP / 2; i++) {
                if (i < half) {
                    const float keep = up ? yp[i + half] : yp[i];
                    const float send = up ? yp[i] : yp[i + half];
                    yp[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int tt = 2 * ns + (r >> 1), j = r & 1;
            if (tt < nt && p + j < P)
                a.y[(size_t)(tb + tt) * inner + h * P + p + j] = yp[r] + Dh * sx[tt * PT + pl * SCAN_PP + j];
        }
        }
    }
    if (MODE == 1) {
        each([&](int j, int k, int e, size_t o) { E[(size_t)chunk * hpn + o] = s[j][k][e]; });
        if (blockIdx.x == 0 && threadIdx.x == 0) a.chunk_decay[((size_t)b * a.n_chunks + chunk) * H + h] = decay;
    } else if (last) {
        each([&](int j, int k, int e, size_t o) { S[o] = s[j][k][e]; });
    }
}

// ---------------------------------------------------------------------------------------------------------
// Prompts as products (bfloat16, N up to 128).  With the step sizes dt, the log2 decays l = max(A dt log2 e, -300) and
// their running sums c within a chunk of 128 tokens, S the state before it:
//     y_i = sum_{j <= i} (C_i . B_j) 2^(c_i - c_j) dt_j x_j  +  2^(c_i) S C_i  +  D x_i
//     S'  = 2^(c_last) S + sum_j 2^(c_last - c_j) dt_j x_j B_j^T
// in three launches: each chunk's own sum E, the states before the chunks (a scan over chunks, element by element), the
// outputs; sequences of one chunk take part in the last one only.  x, B and C are bfloat16 numbers; what meets them (the weighted scores, the weighted x, the state) is 32-bit and
// enters as the sum of three bfloat16 numbers, 24 bits.  A tensor core's sums are cut off, so 16 terms at a time are added up in
// them and those sums outside; decays come from ex2 of summed logs.  Against 64 bits the state of 2,048 tokens stands 0.97e-7 off
// (the recurrence 0.96e-7; with decays near 1, 1.1e-7 and 5.1e-7), the outputs 0.97e-7 (0.91e-7; 1.4e-7 and 4.8e-7).  The
// running sums are kept as two 32-bit numbers (c_i - c_j of near tokens keeps its digits); a decay below 2^-300 is 0 in any
// product.  A non-finite x is seen by its own token and later ones only, as in the recurrence; what it leaves in the state is
// NaN to the next chunk's outputs (an infinity has no three parts).
// 2,048 tokens, 64 heads of 64 x 128: 31 + 20 + 56 us cold (the recurrence in chunks: 167 + 235; both before the sums of 16 terms,
// which take 3 % more); the tensor pipe and the three-way splits share the time of the third launch.  All of ops.mamba2, passes
// back to back: 489 -> 136.8 us.
// ---------------------------------------------------------------------------------------------------------
constexpr int MC = 128, MCT = 256;                    // tokens of a chunk, threads
constexpr int MP = 64, MXPITCH = MP * 2 + 16;         // values of P a CTA takes; bytes of a shared row of them (no bank conflicts)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;                     // 0 source bytes: the 16 destination bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int K> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }
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
// A product's sums are cut off, not rounded, so what comes of 16 terms is added up outside of the products.
__device__ __forceinline__ void set0(float (*u)[4]) {
#pragma unroll
    for (int e = 0; e < 4; e++) u[0][e] = u[1][e] = 0.f;
}
// Two 32-bit numbers as sums of three bfloat16 numbers each: the remainders are exact, the last one holds what is left.
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack2(x, y);
    x -= __uint_as_float(hi << 16); y -= __uint_as_float(hi & 0xffff0000u);
    mid = pack2(x, y);
    lo = pack2(x - __uint_as_float(mid << 16), y - __uint_as_float(mid & 0xffff0000u));
}
__device__ __forceinline__ float exp2_fast(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// A sign bit of the result is set where one of two bfloat16 numbers is infinite or NaN.
__device__ __forceinline__ uint32_t not_finite(uint32_t v) { return (v & 0x7f807f80u) + 0x00800080u; }
// What two numbers' three parts add up to: the number in the low halves, in the high halves.
__device__ __forceinline__ float low3(const uint32_t* p) { return __uint_as_float(p[0] << 16) + (__uint_as_float(p[1] << 16) + __uint_as_float(p[2] << 16)); }
__device__ __forceinline__ float high3(const uint32_t* p) {
    return __uint_as_float(p[0] & 0xffff0000u) + (__uint_as_float(p[1] & 0xffff0000u) + __uint_as_float(p[2] & 0xffff0000u));
}

struct ChunkPlace { int t0, n, c, b, slot; bool alone; };   // first token, tokens, index in its sequence, sequence, scratch slot, its sequence's only one
// A sequence's chunks lie from slot floor(seq_start / 128) + b on, which leaves every sequence enough of them.
__device__ __forceinline__ ChunkPlace chunk_place(const Mamba2Args& a, int z) {
    ChunkPlace p;
    p.b = z / a.n_chunks; p.c = z % a.n_chunks;
    const int s0 = a.seq_start[p.b], s1 = a.seq_start[p.b + 1];
    p.t0 = s0 + p.c * MC; p.n = min(MC, s1 - p.t0); p.slot = s0 / MC + p.b + p.c;
    p.alone = a.n_chunks == 1 || s1 - s0 <= MC;       // (without chunks nothing looks for scratch, whatever the lengths)
    return p;
}

// dt and the running sums of the log2 decays of a chunk's tokens (past its end: no step, no decay) into shared memory.
__device__ __forceinline__ void chunk_decays(const Mamba2Args& a, const ChunkPlace& p, int h, float* sdt, float2* scum, double* red) {
    const int tid = threadIdx.x, lane = tid & 31;
    double l = 0.0;
    if (tid < MC) {
        float dt = 0.f;
        if (tid < p.n) {
            const float* q = a.dt + (size_t)(p.t0 + tid) * a.dt_stride + h;
            dt = q[0];
            for (int sp = 1; sp < a.dt_splits; sp++) dt += q[(size_t)sp * a.dt_split_stride];
            dt = softplus_f(dt + ((const float*)a.dt_bias)[h]);
            l = fmax((double)-expf(((const float*)a.A_log)[h]) * (double)dt * 1.4426950408889634, -300.0);
        }
        sdt[tid] = dt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, l, o);
            if (lane >= o) l += up;
        }
        if (lane == 31) red[tid >> 5] = l;
    }
    __syncthreads();
    if (tid < MC) {
        for (int w = 0; w < tid >> 5; w++) l += red[w];
        const float hi = (float)l;
        scum[tid] = make_float2(hi, (float)(l - (double)hi));
    }
    __syncthreads();
}

// n rows of COLS bfloat16 columns, of which `cols` exist, into padded shared rows; up to the next multiple of 16, rows of zeros.
template <int COLS>
__device__ __forceinline__ void load_chunk(uint8_t* dst, const bf16* src, long long stride, int n, int cols) {
    constexpr int CPR = COLS / 8, PITCH = COLS * 2 + 16;
#pragma unroll 4
    for (int c = threadIdx.x; c < (n + 15) / 16 * 16 * CPR; c += MCT) {
        const int r = c / CPR, k = (c % CPR) * 8;
        const bool ok = r < n && k < cols;
        cp_async16(dst + r * PITCH + k * 2, src + (ok ? (size_t)r * stride + k : 0), ok);
    }
}

// sum_j w_j x_j B_j^T of a chunk's n tokens.  Warp w: 16 rows of P, half of N, in accumulators.
template <int NP>
__device__ __forceinline__ void chunk_sum(const uint8_t* sB, const uint8_t* sx, const float* w, int n, float (*acc)[4]) {
    constexpr int BPITCH = NP * 2 + 16, NT = NP / 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 3;
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * (NP / 2);
#pragma unroll
    for (int j = 0; j < NT; j++) { acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f; }
    const int steps = (n + 15) / 16;
    for (int kk = 0; kk < steps; kk++) {
        const float2 wa = *(const float2*)(w + kk * 16 + 2 * t), wb = *(const float2*)(w + kk * 16 + 2 * t + 8);
        uint32_t x[4], hi[4], mid[4], lo[4];
        ldsm_x4_t(smem_addr(sx + (kk * 16 + (lane >> 4) * 8 + (lane & 7)) * MXPITCH + (m0 + ((lane >> 3) & 1) * 8) * 2), x);
#pragma unroll
        for (int e = 0; e < 4; e++)
            split3(__uint_as_float(x[e] << 16) * (e < 2 ? wa.x : wb.x), __uint_as_float(x[e] & 0xffff0000u) * (e < 2 ? wa.y : wb.y), hi[e], mid[e], lo[e]);
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
            uint32_t f[4];
            ldsm_x4_t(smem_addr(sB + (kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * BPITCH + (n0 + j * 8 + (lane >> 4) * 8) * 2), f);
            float u[2][4];
            set0(u);
            mma_bf16(u[0], lo, f[0], f[1]); mma_bf16(u[1], lo, f[2], f[3]);
            mma_bf16(u[0], mid, f[0], f[1]); mma_bf16(u[1], mid, f[2], f[3]);
            mma_bf16(u[0], hi, f[0], f[1]); mma_bf16(u[1], hi, f[2], f[3]);
#pragma unroll
            for (int e = 0; e < 4; e++) { acc[j][e] += u[0][e]; acc[j + 1][e] += u[1][e]; }
        }
    }
}

// E = sum_j 2^(c_last - c_j) dt_j x_j B_j^T: 64 values of P of one head, all N, of a sequence of several chunks.
template <int NP>
__global__ void __launch_bounds__(MCT) mamba2_chunk_sum_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    constexpr int BPITCH = NP * 2 + 16, NT = NP / 16;  // 8-column pieces a warp
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* sB = smem;                               // [128][BPITCH]
    uint8_t* sx = sB + MC * BPITCH;                   // [128][MXPITCH]
    float2* scum = (float2*)(sx + MC * MXPITCH);      // [128]
    float* sdt = (float*)(scum + MC);                 // [128], then the weights
    __shared__ double red[4];
    const int h = blockIdx.y, p0 = blockIdx.x * MP, N = a.N, P = a.P;
    const int inner = a.heads * P, ch = inner + 2 * a.groups * N, g_of = h / (a.heads / a.groups);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    pdl_wait();
    const ChunkPlace pl = chunk_place(a, blockIdx.z);
    if (pl.n <= 0 || pl.alone) return;
    const bf16* row = (const bf16*)a.xbc + (size_t)pl.t0 * ch;
    load_chunk<NP>(sB, row + inner + g_of * N, ch, pl.n, N);
    load_chunk<MP>(sx, row + h * P + p0, ch, pl.n, P - p0);
    cp_async_commit();
    chunk_decays(a, pl, h, sdt, scum, red);
    const float2 last = scum[MC - 1];
    if (threadIdx.x < MC) sdt[threadIdx.x] *= exp2_fast((last.x - scum[threadIdx.x].x) + (last.y - scum[threadIdx.x].y));
    if (blockIdx.x == 0 && threadIdx.x == 0) a.chunk_decay[(size_t)pl.slot * a.heads + h] = exp2_fast(last.x + last.y);
    cp_async_wait<0>();
    __syncthreads();
    float acc[NT][4];
    chunk_sum<NP>(sB, sx, sdt, pl.n, acc);
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * (NP / 2);
    float* E = a.chunk_state + (size_t)pl.slot * a.heads * P * N + (size_t)h * P * N;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int n = n0 + j * 8 + 2 * t, p = p0 + m0 + g;
        if (n >= N) continue;                         // (N is even)
        if (p < P) *(float2*)(E + (size_t)p * N + n) = make_float2(acc[j][0], acc[j][1]);
        if (p + 8 < P) *(float2*)(E + (size_t)(p + 8) * N + n) = make_float2(acc[j][2], acc[j][3]);
    }
}

// Every chunk's own sum becomes the state before the chunk; the sequence's state becomes the one after its last token.
__global__ void __launch_bounds__(256) mamba2_chunk_fold_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    const int b = blockIdx.y, per = a.P * a.N;
    const size_t hpn = (size_t)a.heads * per;
    const size_t e = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= hpn) return;
    const int h = (int)(e / per);
    pdl_wait();
    const int s0 = a.seq_start[b], len = a.seq_start[b + 1] - s0, n = (len + MC - 1) / MC, slot = s0 / MC + b;
    if (n <= 1) return;                               // (a sequence of one chunk: the outputs' launch)
    float* st = a.state + (size_t)a.slot_ids[b] * a.state_stride + e;
    float4 s = *(const float4*)st;
    float* E = a.chunk_state + (size_t)slot * hpn + e;
    const float* D = a.chunk_decay + (size_t)slot * a.heads + h;
    for (int c0 = 0; c0 < n; c0 += 8) {               // eight chunks' sums on their way together
        float4 x[8]; float d[8];
#pragma unroll
        for (int u = 0; u < 8; u++) if (c0 + u < n) { x[u] = *(const float4*)(E + (c0 + u) * hpn); d[u] = D[(size_t)(c0 + u) * a.heads]; }
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (c0 + u < n) {
                *(float4*)(E + (c0 + u) * hpn) = s;
                s.x = fmaf(d[u], s.x, x[u].x); s.y = fmaf(d[u], s.y, x[u].y); s.z = fmaf(d[u], s.z, x[u].z); s.w = fmaf(d[u], s.w, x[u].w);
            }
    }
    *(float4*)st = s;
}

// y of 128 tokens of one head, 64 values of P.  A warp: 16 tokens.  A sequence of one chunk starts from its slot and leaves its
// state there, in this launch alone: nobody else reads that part of the slot.
template <int NP>
__global__ void __launch_bounds__(MCT, 2) mamba2_chunk_out_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    constexpr int BPITCH = NP * 2 + 16, KS = NP / 16;
    constexpr int FIRST = MC * BPITCH > 3 * MP * BPITCH ? MC * BPITCH : 3 * MP * BPITCH;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* sS = smem;                               // [128][BPITCH] C, then [3][64][BPITCH] the state's three parts
    uint8_t* sB = sS + FIRST;                         // [128][BPITCH]
    uint8_t* sx = sB + MC * BPITCH;                   // [128][MXPITCH]
    float2* scum = (float2*)(sx + MC * MXPITCH);      // [128]
    float* sdt = (float*)(scum + MC);                 // [128]
    float* sw = sdt + MC;                             // [128] the tokens' weights in the state that a sequence of one chunk leaves
    __shared__ double red[4];
    const int h = blockIdx.y, p0 = blockIdx.x * MP, N = a.N, P = a.P;
    const int inner = a.heads * P, ch = inner + 2 * a.groups * N, g_of = h / (a.heads / a.groups);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // the 16 tokens of a warp: the later ones see more keys, and the two warps of an SM's quarter (w and w + 4) get nine
    // sixteens together whichever they are (in order the quarters had 6, 8, 10 and 12)
    const int wr = warp < 4 ? warp : 11 - warp;
    pdl_wait();
    const ChunkPlace pl = chunk_place(a, blockIdx.z);
    if (pl.n <= 0) return;
    const bf16* row = (const bf16*)a.xbc + (size_t)pl.t0 * ch;
    load_chunk<NP>(sS, row + inner + (a.groups + g_of) * N, ch, pl.n, N);
    cp_async_commit();
    load_chunk<NP>(sB, row + inner + g_of * N, ch, pl.n, N);
    load_chunk<MP>(sx, row + h * P + p0, ch, pl.n, P - p0);
    cp_async_commit();
    // the state, on its way through registers meanwhile: thread (p, part of n)
    float* S = (pl.alone ? a.state + (size_t)a.slot_ids[pl.b] * a.state_stride : a.chunk_state + (size_t)pl.slot * a.heads * P * N) + ((size_t)h * P + p0) * N;
    constexpr int Q = MP * NP / 4 / MCT;              // groups of four a thread
    float4 sv[Q];
#pragma unroll
    for (int u = 0; u < Q; u++) {
        const int i = tid + u * MCT, p = i / (NP / 4), n = (i % (NP / 4)) * 4;
        sv[u] = (p0 + p < P && n < N) ? *(const float4*)(S + (size_t)p * N + n) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    chunk_decays(a, pl, h, sdt, scum, red);
    const float2 last = scum[MC - 1];
    if (pl.alone && tid < MC) sw[tid] = sdt[tid] * exp2_fast((last.x - scum[tid].x) + (last.y - scum[tid].y));
    cp_async_wait<1>();
    __syncthreads();
    uint32_t q[KS][4];
#pragma unroll
    for (int ks = 0; ks < KS; ks++) ldsm_x4(smem_addr(sS + (wr * 16 + (lane & 15)) * BPITCH + (ks * 16 + (lane >> 4) * 8) * 2), q[ks]);
    __syncthreads();                                  // C is in registers: its place takes the state
#pragma unroll
    for (int u = 0; u < Q; u++) {
        const int i = tid + u * MCT, p = i / (NP / 4), n = (i % (NP / 4)) * 4;
        uint2 part[3];
        split3(sv[u].x, sv[u].y, part[0].x, part[1].x, part[2].x);
        split3(sv[u].z, sv[u].w, part[0].y, part[1].y, part[2].y);
#pragma unroll
        for (int k = 0; k < 3; k++) *(uint2*)(sS + (k * MP + p) * BPITCH + n * 2) = part[k];
    }
    cp_async_wait<0>();
    __syncthreads();
    // ---- what the state before the chunk gives
    float o[8][4];
#pragma unroll
    for (int j = 0; j < 8; j++) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f; }
    if (wr * 16 < pl.n) {                           // (rows past the end: nothing to write)
#pragma unroll
        for (int j = 0; j < 8; j += 2)
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                float u[2][4];
                set0(u);
#pragma unroll
                for (int k = 2; k >= 0; k--) {
                    uint32_t f[4];
                    ldsm_x4(smem_addr(sS + (k * MP + j * 8 + (lane >> 4) * 8 + (lane & 7)) * BPITCH + (ks * 16 + ((lane >> 3) & 1) * 8) * 2), f);
                    mma_bf16(u[0], q[ks], f[0], f[1]);
                    mma_bf16(u[1], q[ks], f[2], f[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; e++) { o[j][e] += u[0][e]; o[j + 1][e] += u[1][e]; }
            }
        const int ra = wr * 16 + g, rb = ra + 8;
        const float2 ca = scum[ra], cb = scum[rb];
        {
            const float fa = exp2_fast(ca.x + ca.y), fb = exp2_fast(cb.x + cb.y);
#pragma unroll
            for (int j = 0; j < 8; j++) { o[j][0] *= fa; o[j][1] *= fa; o[j][2] *= fb; o[j][3] *= fb; }
        }
        // ---- the chunk's own tokens, 16 keys at a time up to this warp's last row
        bool odd = false;                             // an x of this warp's own 16 tokens is not finite
        {
            uint32_t any = 0;
#pragma unroll
            for (int u = 0; u < MP * 2 / 32; u++) {
                const uint4 x = *(const uint4*)(sx + (wr * 16 + (lane >> 1)) * MXPITCH + (lane & 1) * MP + u * 16);
                any |= not_finite(x.x) | not_finite(x.y) | not_finite(x.z) | not_finite(x.w);
            }
            odd = __any_sync(0xffffffffu, (any & 0x80008000u) != 0);
        }
        uint32_t hi[4], mid[4], lo[4];
        for (int kk = 0; kk <= wr; kk++) {
            float s[2][4];
#pragma unroll
            for (int n = 0; n < 2; n++) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f; }
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                uint32_t f[4];
                float u[2][4];
                ldsm_x4(smem_addr(sB + (kk * 16 + (lane >> 4) * 8 + (lane & 7)) * BPITCH + (ks * 16 + ((lane >> 3) & 1) * 8) * 2), f);
                set0(u);
                mma_bf16(u[0], q[ks], f[0], f[1]);
                mma_bf16(u[1], q[ks], f[2], f[3]);
#pragma unroll
                for (int e = 0; e < 4; e++) { s[0][e] += u[0][e]; s[1][e] += u[1][e]; }
            }
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const int j = kk * 16 + n * 8 + 2 * t;
                const float4 cj = *(const float4*)(scum + j);          // tokens j and j + 1
                const float2 dj = *(const float2*)(sdt + j);
                const float x0 = j <= ra ? s[n][0] * (exp2_fast((ca.x - cj.x) + (ca.y - cj.y)) * dj.x) : 0.f;
                const float x1 = j + 1 <= ra ? s[n][1] * (exp2_fast((ca.x - cj.z) + (ca.y - cj.w)) * dj.y) : 0.f;
                const float x2 = j <= rb ? s[n][2] * (exp2_fast((cb.x - cj.x) + (cb.y - cj.y)) * dj.x) : 0.f;
                const float x3 = j + 1 <= rb ? s[n][3] * (exp2_fast((cb.x - cj.z) + (cb.y - cj.w)) * dj.y) : 0.f;
                split3(x0, x1, hi[n * 2], mid[n * 2], lo[n * 2]);
                split3(x2, x3, hi[n * 2 + 1], mid[n * 2 + 1], lo[n * 2 + 1]);
            }
            if (odd && kk == wr) break;
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                uint32_t f[4];
                ldsm_x4_t(smem_addr(sx + (kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * MXPITCH + (j * 8 + (lane >> 4) * 8) * 2), f);
                float u[2][4];
                set0(u);
                mma_bf16(u[0], lo, f[0], f[1]); mma_bf16(u[1], lo, f[2], f[3]);
                mma_bf16(u[0], mid, f[0], f[1]); mma_bf16(u[1], mid, f[2], f[3]);
                mma_bf16(u[0], hi, f[0], f[1]); mma_bf16(u[1], hi, f[2], f[3]);
#pragma unroll
                for (int e = 0; e < 4; e++) { o[j][e] += u[0][e]; o[j + 1][e] += u[1][e]; }
            }
        }
        if (odd) {                                    // (0 times a later token's x would be NaN: token by token, up to the row's own)
            for (int r = 0; r < 16; r++) {
                const int from = (lane & ~3) | ((r & 7) >> 1);
                uint32_t wa[3], wb[3];                // the weight of token r in rows ra and rb
#pragma unroll
                for (int e = 0; e < 3; e++) {
                    const uint32_t* part = e == 0 ? hi : e == 1 ? mid : lo;
                    wa[e] = __shfl_sync(0xffffffffu, r < 8 ? part[0] : part[2], from);
                    wb[e] = __shfl_sync(0xffffffffu, r < 8 ? part[1] : part[3], from);
                }
                const float fa = (r & 1) ? high3(wa) : low3(wa), fb = (r & 1) ? high3(wb) : low3(wb);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const uint32_t x = *(const uint32_t*)(sx + (wr * 16 + r) * MXPITCH + (j * 8 + 2 * t) * 2);
                    const float xa = __uint_as_float(x << 16), xb = __uint_as_float(x & 0xffff0000u);
                    if (r <= g) { o[j][0] = fmaf(fa, xa, o[j][0]); o[j][1] = fmaf(fa, xb, o[j][1]); }
                    if (r <= g + 8) { o[j][2] = fmaf(fb, xa, o[j][2]); o[j][3] = fmaf(fb, xb, o[j][3]); }
                }
            }
        }
        const float Dh = ((const float*)a.D)[h];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int r = e ? rb : ra;
            if (r >= pl.n) continue;
            float* y = a.y + (size_t)(pl.t0 + r) * inner + h * P + p0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int p = j * 8 + 2 * t;
                if (p0 + p >= P) continue;            // (P is even)
                const uint32_t xv = *(const uint32_t*)(sx + r * MXPITCH + p * 2);
                *(float2*)(y + p) = make_float2(o[j][2 * e] + Dh * __uint_as_float(xv << 16), o[j][2 * e + 1] + Dh * __uint_as_float(xv & 0xffff0000u));
            }
        }
    }
    if (!pl.alone) return;
    // ---- the state after the sequence (every thread has read its part of the one before, above the last barrier)
    float acc[NP / 16][4];
    chunk_sum<NP>(sB, sx, sw, pl.n, acc);
    const float all = exp2_fast(last.x + last.y);
    const int m0 = (warp & 3) * 16, n0 = (warp >> 2) * (NP / 2);
#pragma unroll
    for (int j = 0; j < NP / 16; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int n = n0 + j * 8 + 2 * t, p = m0 + g + e * 8;
            if (n >= N || p0 + p >= P) continue;
            float2* to = (float2*)(S + (size_t)p * N + n);
            const float2 s = *to;
            *to = make_float2(fmaf(all, s.x, acc[j][2 * e]), fmaf(all, s.y, acc[j][2 * e + 1]));
        }
}

// ---------------------------------------------------------------------------------------------------------
// out = groupnorm(y * silu(z)) * w: one CTA per (token, norm group).
template <typename T, typename TW>
__global__ void mamba2_gate_norm_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    const int inner = a.heads * a.P, gs = inner / a.norm_groups;
    const int t = blockIdx.x, c0 = blockIdx.y * gs;
    const float* y = a.y + (size_t)t * inner + c0;
    const T* z = (const T*)a.proj + (size_t)t * a.proj_stride + c0;
    float ss = 0.f;
    for (int i = threadIdx.x; i < gs; i += blockDim.x) {
        const float v = y[i] * silu_f(to_f<T>(z[i]));
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float r = 1.0f / sqrtf(ss / (float)gs + a.eps);
    const TW* w = (const TW*)a.norm_w + c0;
    T* out = (T*)a.out + (size_t)t * inner + c0;
    for (int i = threadIdx.x; i < gs; i += blockDim.x) {
        const float v = y[i] * silu_f(to_f<T>(z[i]));
        out[i] = from_f<T>(v * r * to_f<TW>(w[i]));
    }
}

// The same where a thread can keep its NV groups of four columns in registers, so that y and z are read once, 16 bytes of y
// and four values of z a load (group sizes that are multiples of 4).  FEW tokens (the launch's time is a chain of memory
// round trips): up to 1,024 threads a row and the weights fetched ahead of the wait; of a step of one token of 8,192 channels
// with cold caches, all launches, 13.9 us (256 threads, the weights after the sum: 18.2).  Many: 256 threads a row, 2,048 rows
// of 4,096 in 15 us (read twice: 37; 67 MB are 10).
__device__ __forceinline__ float4 four(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 four(const bf16* p) {
    const uint2 u = *(const uint2*)p;
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *(float4*)p = v; }
__device__ __forceinline__ void store4(bf16* p, float4 v) { *(uint2*)p = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }

template <typename T, int NV, bool FEW>
__global__ void __launch_bounds__(FEW ? 1024 : 256) mamba2_gate_norm_rows_kernel(Mamba2Args a) {
    pdl_launch_dependents();
    __shared__ float red[33];
    const int inner = a.heads * a.P, gs = inner / a.norm_groups;
    const int t = blockIdx.x, c0 = blockIdx.y * gs;
    float4 w[NV];
    if (FEW) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const int i = (threadIdx.x + k * blockDim.x) * 4;
            if (i < gs) w[k] = four((const float*)a.norm_w + c0 + i);
        }
    }
    pdl_wait();
    const float* y = a.y + (size_t)t * inner + c0;
    const T* z = (const T*)a.proj + (size_t)t * a.proj_stride + c0;
    float4 v[NV], u[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        v[k] = u[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < gs) { v[k] = four(y + i); u[k] = four(z + i); }
    }
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k].x *= silu_f(u[k].x); v[k].y *= silu_f(u[k].y); v[k].z *= silu_f(u[k].z); v[k].w *= silu_f(u[k].w);
        ss += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
    }
    ss = block_sum(ss, red);
    const float r = 1.0f / sqrtf(ss / (float)gs + a.eps);
    T* out = (T*)a.out + (size_t)t * inner + c0;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < gs) {
            if (!FEW) w[k] = four((const float*)a.norm_w + c0 + i);
            store4(out + i, make_float4(v[k].x * r * w[k].x, v[k].y * r * w[k].y, v[k].z * r * w[k].z, v[k].w * r * w[k].w));
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
static int check(const Mamba2Args& a) {
    if (a.heads <= 0 || a.P <= 0 || a.N <= 0 || a.groups <= 0 || a.taps <= 0 || a.norm_groups <= 0)
        return tb_refuse("mamba2: heads=%d P=%d N=%d groups=%d taps=%d norm_groups=%d", a.heads, a.P, a.N, a.groups, a.taps,
                         a.norm_groups);
    if (a.heads % a.groups) return tb_refuse("mamba2: %d heads cannot share %d groups", a.heads, a.groups);
    if ((a.heads * a.P) % a.norm_groups) return tb_refuse("mamba2: %d inner columns do not split into %d norm groups",
                                                          a.heads * a.P, a.norm_groups);
    if (a.N > 256) return tb_refuse("mamba2: state size %d (at most 256)", a.N);
    return 0;
}

// The small tensors (taps, biases, A_log, D, the norm's weight) enter 32-bit arithmetic and are taken in 32 bits.
#define DISPATCH2(ct, cw, ...)                                                             \
    do {                                                                                   \
        if ((cw) != TB_F32) return tb_refuse("mamba2: the small tensors must be float32 (code %d)", (cw)); \
        if ((ct) == TB_F32) { typedef float T; typedef float TW; __VA_ARGS__; }            \
        else if ((ct) == TB_BF16) { typedef bf16 T; typedef float TW; __VA_ARGS__; }       \
        else return tb_refuse("mamba2: unknown dtype code %d", (ct));                      \
    } while (0)

extern "C" int tb_mamba2_conv(const Mamba2Args* args, int dtype, int w_dtype, int one_token_each, cudaStream_t stream) {
    Mamba2Args a = *args;
    if (a.n_tokens <= 0) return 0;
    if (check(a)) return -1;
    const int ch = a.heads * a.P + 2 * a.groups * a.N;
    const unsigned gy = (ch + 127) / 128;
    if (one_token_each) {
        DISPATCH2(dtype, w_dtype, tb_launch(mamba2_conv_step_kernel<T, TW>, dim3(a.batch, gy), dim3(128), 0, stream, a));
        return tb_launch_status();
    }
    const bool wide = dtype == TB_BF16 && w_dtype == TB_F32 && a.taps == 4 && ch % 4 == 0 && (a.heads * a.P) % 4 == 0 && a.proj_stride % 4 == 0 &&
                      ((uintptr_t)a.proj & 7) == 0 && ((uintptr_t)a.xbc & 7) == 0 && ((uintptr_t)a.conv_w & 15) == 0;
    // eight tokens a thread where that leaves three CTAs an SM, else two (100 tokens of 2,176 channels: 65 CTAs of a long chain each)
    const long long wide_ctas = (long long)((a.n_tokens + 7) / 8) * ((ch / 4 + 127) / 128);
    if (wide && wide_ctas >= 3 * 148) tb_launch(mamba2_conv4_kernel<8>, dim3((a.n_tokens + 7) / 8, (ch / 4 + 127) / 128), dim3(128), 0, stream, a);
    else if (wide) tb_launch(mamba2_conv4_kernel<2>, dim3((a.n_tokens + 1) / 2, (ch / 4 + 127) / 128), dim3(128), 0, stream, a);
    else DISPATCH2(dtype, w_dtype, tb_launch(mamba2_conv_kernel<T, TW>, dim3(a.n_tokens, gy), dim3(128), 0, stream, a));
    int st = tb_launch_status();
    if (st) return st;
    if (a.taps > 1) {
        TB_DISPATCH_1(dtype, T, tb_launch(mamba2_conv_state_kernel<T>, dim3(a.batch, gy), dim3(128), 0, stream, a));
    }
    return tb_launch_status();
}

static int scan_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0; cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

// Into how many chunks (and of how many tokens) the longest prompt of a step is cut: 1 unless the (sequence, head,
// 32 values of P) tiles are fewer than four an SM and the prompt is long enough for chunks of 128 tokens and more.
extern "C" int tb_mamba2_plan(int heads, int P, int batch, int max_seq_len, int* chunk_len) {
    const long long tiles = (long long)((P + 31) / 32) * heads * batch;
    const int sms = scan_sms();
    int chunks = 1;
    if (tiles < 4LL * sms && max_seq_len >= 256) {
        chunks = (int)((6LL * sms + tiles - 1) / tiles);
        if (chunks > max_seq_len / 128) chunks = max_seq_len / 128;
        if (chunks > 64) chunks = 64;
    }
    int len = (max_seq_len + chunks - 1) / chunks;
    len = (len + SCAN_TT - 1) / SCAN_TT * SCAN_TT;
    if (len < SCAN_TT) len = SCAN_TT;
    chunks = (max_seq_len + len - 1) / len;
    if (chunks < 1) chunks = 1;
    if (chunk_len) *chunk_len = len;
    return chunks;
}

extern "C" int tb_mamba2_scan(const Mamba2Args* args, int dtype, int w_dtype, cudaStream_t stream) {
    Mamba2Args a = *args;
    if (a.n_tokens <= 0) return 0;
    if (check(a)) return -1;
    const int sms = scan_sms();
    const bool chunked = a.n_chunks > 1;
    if (chunked && (a.chunk_state == nullptr || a.chunk_decay == nullptr || a.chunk_len < SCAN_TT || a.chunk_len % SCAN_TT))
        return tb_refuse("mamba2: chunks need their scratch and a length that is a multiple of %d", SCAN_TT);
    const int zdim = a.batch * (chunked ? a.n_chunks : 1);
    // thirty-two values of P a CTA (128 threads), or sixteen where that would leave SMs without work
    const int pt = ((long long)((a.P + 31) / 32) * a.heads * zdim >= 2LL * sms) ? 32 : 16;
    const dim3 grid((a.P + pt - 1) / pt, a.heads, zdim);
    if (grid.y > 65535 || grid.z > 65535) return tb_refuse("mamba2: too many heads or sequences for one launch");
    const int nv = (a.N + 31) / 32;
    const int es = dtype == TB_BF16 ? 2 : 4;
    const int chn = a.heads * a.P + 2 * a.groups * a.N;
    const bool vec8 = a.N % 8 == 0 && ((size_t)chn * es) % 16 == 0 && ((size_t)a.heads * a.P * es) % 16 == 0 &&
                      ((uintptr_t)a.xbc & 15) == 0;
#define SCAN4(NV_, PT_, V8_, MODE_) \
        DISPATCH2(dtype, w_dtype, tb_launch(mamba2_scan_kernel<T, TW, NV_, PT_, V8_, MODE_>, dim3(grid), dim3(SCAN_NS * (PT_) / SCAN_PP), smem, stream, a))
#define SCAN3(NV_, PT_, MODE_) do { \
        const size_t smem = (size_t)(SCAN_TT * 2 * (NV_) * 32 + SCAN_TT * (PT_) + SCAN_TT * 2) * sizeof(float); \
        if (vec8) SCAN4(NV_, PT_, true, MODE_); else SCAN4(NV_, PT_, false, MODE_); \
    } while (0)
#define SCAN2(NV_, MODE_) do { if (pt == 32) SCAN3(NV_, 32, MODE_); else SCAN3(NV_, 16, MODE_); } while (0)
#define SCAN(MODE_) do { if (nv <= 1) SCAN2(1, MODE_); else if (nv <= 2) SCAN2(2, MODE_); else if (nv <= 4) SCAN2(4, MODE_); else SCAN2(8, MODE_); } while (0)
    if (!chunked) {
        SCAN(0);
        return tb_launch_status();
    }
    SCAN(1);
    const int st = tb_launch_status();
    if (st) return st;
    SCAN(2);
#undef SCAN
#undef SCAN2
#undef SCAN3
#undef SCAN4
    return tb_launch_status();
}

// Whether the product form takes these sizes: bfloat16, whole 16-byte pieces of x, B and C.
extern "C" int tb_mamba2_chunks_takes(int dtype, int heads, int P, int N, int groups) {
    return dtype == TB_BF16 && heads > 0 && groups > 0 && heads <= 65535 && P > 0 && P % 8 == 0 && N >= 8 && N <= 128 && N % 8 == 0;
}

// Scratch slots of a step: every sequence's chunks lie from slot floor(seq_start / 128) + its index on.
extern "C" int tb_mamba2_chunk_slots(int batch, int n_tokens) { return n_tokens / MC + batch; }

template <int NP>
static int run_chunks(const Mamba2Args& a, cudaStream_t stream) {
    constexpr int BPITCH = NP * 2 + 16, TAIL = MC * MXPITCH + MC * 16;
    constexpr int SUM = MC * BPITCH + TAIL, OUT = (MC * BPITCH > 3 * MP * BPITCH ? MC * BPITCH : 3 * MP * BPITCH) + MC * BPITCH + TAIL;
    cudaError_t e = cudaFuncSetAttribute(mamba2_chunk_sum_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SUM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(mamba2_chunk_out_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((a.P + MP - 1) / MP, a.heads, a.batch * a.n_chunks);
    if (a.n_chunks == 1) {
        tb_launch(mamba2_chunk_out_kernel<NP>, grid, dim3(MCT), OUT, stream, a);
        return tb_launch_status();
    }
    tb_launch(mamba2_chunk_sum_kernel<NP>, grid, dim3(MCT), SUM, stream, a);
    int st = tb_launch_status();
    if (st) return st;
    const long long quads = (long long)a.heads * a.P * a.N / 4;
    tb_launch(mamba2_chunk_fold_kernel, dim3((unsigned)((quads + 255) / 256), a.batch), dim3(256), 0, stream, a);
    st = tb_launch_status();
    if (st) return st;
    tb_launch(mamba2_chunk_out_kernel<NP>, grid, dim3(MCT), OUT, stream, a);
    return tb_launch_status();
}

// n_chunks: of the longest sequence; chunk_state [slots][heads * P * N] and chunk_decay [slots][heads] if more than one.
extern "C" int tb_mamba2_chunks(const Mamba2Args* args, int dtype, int w_dtype, cudaStream_t stream) {
    const Mamba2Args& a = *args;
    if (a.n_tokens <= 0 || a.batch <= 0) return 0;
    if (check(a)) return -1;
    const int ch = a.heads * a.P + 2 * a.groups * a.N;
    if (!tb_mamba2_chunks_takes(dtype, a.heads, a.P, a.N, a.groups) || w_dtype != TB_F32)
        return tb_refuse("mamba2: the product form takes bfloat16 with P and N in multiples of 8, N up to 128 (got P=%d N=%d)", a.P, a.N);
    if ((a.n_chunks > 1 && (a.chunk_state == nullptr || a.chunk_decay == nullptr)) || a.n_chunks < 1 || (long long)a.batch * a.n_chunks > 65535)
        return tb_refuse("mamba2: the product form needs its scratch, and at most 65535 chunks (%d sequences of %d)", a.batch, a.n_chunks);
    if (((uintptr_t)a.xbc & 15) || ch % 8 || ((uintptr_t)a.state & 15) || a.state_stride % 4 || ((uintptr_t)a.chunk_state & 15) || ((uintptr_t)a.y & 7))
        return tb_refuse("mamba2: the product form needs 16-byte aligned rows and states");
    return a.N <= 64 ? run_chunks<64>(a, stream) : run_chunks<128>(a, stream);
}

// Groups of four columns that a thread of the norm takes of rows of `gs` numbers (up to 16,384): for few tokens as few as 1,024
// threads allow, for many as 256 do.
constexpr int NORM_FEW = 64;
extern "C" int tb_mamba2_gate_norm_groups(int n_tokens, int gs) {
    int nv = 1;
    while (gs / 4 > nv * (n_tokens <= NORM_FEW ? 1024 : 256)) nv *= 2;
    return nv;
}

extern "C" int tb_mamba2_gate_norm(const Mamba2Args* args, int dtype, int w_dtype, cudaStream_t stream) {
    Mamba2Args a = *args;
    if (a.n_tokens <= 0) return 0;
    if (check(a)) return -1;
    const int gs = a.heads * a.P / a.norm_groups;
    int threads = (gs + 31) / 32 * 32;
    threads = threads < 64 ? 64 : (threads > 512 ? 512 : threads);
    if (a.norm_groups > 65535) return tb_refuse("mamba2: too many norm groups");
    const int es = dtype == TB_BF16 ? 2 : 4;
    if (w_dtype == TB_F32 && gs % 4 == 0 && gs <= 16384 && a.proj_stride % 4 == 0 && ((uintptr_t)a.y & 15) == 0 && ((uintptr_t)a.norm_w & 15) == 0 &&
        ((uintptr_t)a.proj & (4 * es - 1)) == 0 && ((uintptr_t)a.out & (4 * es - 1)) == 0) {
        const bool few = a.n_tokens <= NORM_FEW;
        const int nv = tb_mamba2_gate_norm_groups(a.n_tokens, gs);
        int th = ((gs / 4 + nv - 1) / nv + 31) / 32 * 32;
        if (th < 64) th = 64;
#define ROWS(NV_, FEW_) TB_DISPATCH_1(dtype, T, tb_launch(mamba2_gate_norm_rows_kernel<T, NV_, FEW_>, dim3(a.n_tokens, a.norm_groups), dim3(th), 0, stream, a))
        if (few) { if (nv == 1) ROWS(1, true); else if (nv == 2) ROWS(2, true); else ROWS(4, true); }
        else if (nv == 1) ROWS(1, false); else if (nv == 2) ROWS(2, false); else if (nv == 4) ROWS(4, false); else if (nv == 8) ROWS(8, false); else ROWS(16, false);
#undef ROWS
        return tb_launch_status();
    }
    DISPATCH2(dtype, w_dtype, tb_launch(mamba2_gate_norm_kernel<T, TW>, dim3(a.n_tokens, a.norm_groups), dim3(threads), 0, stream, a));
    return tb_launch_status();
}

// A step of whole prompts in the product form: convolution, chunks, gated norm in one call (a short prompt's step is bound by the
// host: 180 tokens of 32 heads 47.6 us with three).
extern "C" int tb_mamba2_prompts(const Mamba2Args* args, int dtype, int w_dtype, cudaStream_t stream) {
    int st = tb_mamba2_conv(args, dtype, w_dtype, 0, stream);
    if (st) return st;
    st = tb_mamba2_chunks(args, dtype, w_dtype, stream);
    return st ? st : tb_mamba2_gate_norm(args, dtype, w_dtype, stream);
}
