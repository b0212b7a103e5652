// Attention over cached latent rows: the kernels that are particular to it.
//
// A token leaves one row in the cache: [c (C numbers) | r (R numbers)], c a normed latent from which every
// head's keys and values are linear maps (k_h = Uk_h c, v_h = Uv_h c) and r a rotated key part that all
// heads share.  A head's score of query (a | b) against a token is  a . (Uk_h c) + b . r  =  (Uk_h^T a) . c + b . r,
// so with the query mapped once to q' = (Uk_h^T a | b) every head reads the same rows (keys of C + R numbers,
// values their first C numbers) and its output Uv_h (sum_j p_j c_j) is mapped back afterwards.
//
//   tb_latent_rows     from the 32-bit partial sums of the down projection: c = rms-normed first C columns
//                      times a weight, r = the last R columns rotated at the token's position (rotate-half
//                      pairing over the first rot_dims of them), times rot_scale; the row goes to the paged cache
//                      (a ring of ring_rows rows per sequence if that is set) and to a
//                      packed matrix; all arithmetic 32-bit, the row rounded once
//   tb_head_linear     y[t, h, :] = W[h] x[t, h, :] for per-head matrices W [heads][out][in]
//   tb_latent_decode   one query per sequence and head against the cached rows, the key range cut into
//                      splits; softmax with a sink: the denominator also holds exp(sink_h), which has no
//                      key and no value; partial (max, sum, o) per split are folded in split order
#include <cooperative_groups.h>
#include <cuda.h>
#include "common.cuh"
#include "async.cuh"

namespace cg = cooperative_groups;

TB_EXPORT_ERROR()

struct LatentRowsArgs {
    const float* dkv; int splits; long long split_stride;     // [splits][T][C + R]
    const float* norm_w; float eps;                            // [C]
    const float* inv_freq; int rot_dims;                       // [rot_dims / 2]
    int C, R, n_tokens;
    const int* positions; const int* token_seq;
    const int* page_table; int pt_stride; int page_rows;
    void* pool;                                                // [pages][page_rows][C + R]
    void* rows;                                                // [T][C + R]
    int ring_rows; const int* len_after;                       // ring_rows > 0: row = position mod ring_rows, and only the
                                                               // last ring_rows tokens of a sequence ([batch] lengths) are cached
    float rot_scale;                                           // the rotated part comes times this
    long long row_stride;                                      // numbers between two tokens' rows of dkv (0: C + R)
    // the same product may carry, behind the C + R columns, a latent of the queries (Q columns, RMS-normed times
    // q_norm_w with the same eps, written to cq_out [T][Q] in the output's dtype) and n_gate gate columns (their
    // sigmoid goes to gate_out [T][n_gate], 32-bit)
    int Q; const float* q_norm_w; void* cq_out;
    int n_gate; float* gate_out;
};

template <typename T>
__global__ void __launch_bounds__(1024) latent_rows_kernel(LatentRowsArgs a) {
    pdl_launch_dependents();
    extern __shared__ float row_s[];
    __shared__ float red[33];
    const int t = blockIdx.x, W = a.C + a.R, WA = W + a.Q + a.n_gate;
    const size_t rs = a.row_stride > 0 ? (size_t)a.row_stride : (size_t)W;
    pdl_wait();
    float sq = 0.f, sq_q = 0.f;
    for (int c = threadIdx.x; c < WA; c += blockDim.x) {
        const float* src = a.dkv + (size_t)t * rs + c;
        float v = 0.f;
        int s = 0;
        for (; s + 4 <= a.splits; s += 4) {            // four loads on their way at a time, added in split order
            const float v0 = src[(size_t)s * a.split_stride], v1 = src[(size_t)(s + 1) * a.split_stride];
            const float v2 = src[(size_t)(s + 2) * a.split_stride], v3 = src[(size_t)(s + 3) * a.split_stride];
            v = (((v + v0) + v1) + v2) + v3;
        }
        for (; s < a.splits; s++) v += src[(size_t)s * a.split_stride];
        row_s[c] = v;
        if (c < a.C) sq = fmaf(v, v, sq);
        else if (c >= W && c < W + a.Q) sq_q = fmaf(v, v, sq_q);
    }
    const float rinv = 1.f / sqrtf(block_sum(sq, red) / (float)a.C + a.eps);     // its barriers also publish row_s
    if (a.Q > 0) {
        const float qinv = 1.f / sqrtf(block_sum(sq_q, red) / (float)a.Q + a.eps);
        T* cq = (T*)a.cq_out + (size_t)t * a.Q;
        for (int c = threadIdx.x; c < a.Q; c += blockDim.x) cq[c] = from_f<T>(row_s[W + c] * qinv * a.q_norm_w[c]);
    }
    for (int c = threadIdx.x; c < a.n_gate; c += blockDim.x)
        a.gate_out[(size_t)t * a.n_gate + c] = 1.f / (1.f + expf(-row_s[W + a.Q + c]));
    const int pos = a.positions[t];
    const int b = a.token_seq[t];
    const int crow = a.ring_rows > 0 ? pos % a.ring_rows : pos;
    const bool keep = a.ring_rows <= 0 || pos >= a.len_after[b] - a.ring_rows;
    const int page = keep ? a.page_table[(size_t)b * a.pt_stride + crow / a.page_rows] : 0;
    T* cache = (T*)a.pool + ((size_t)page * a.page_rows + crow % a.page_rows) * W;
    T* out = (T*)a.rows + (size_t)t * W;
    const int half = a.rot_dims / 2;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        float v;
        if (c < a.C) {
            v = row_s[c] * rinv * a.norm_w[c];
        } else {
            const int i = c - a.C;
            if (i < half) {
                float sn, cs; sincosf((float)pos * a.inv_freq[i], &sn, &cs);
                v = (row_s[c] * cs - row_s[c + half] * sn) * a.rot_scale;
            } else if (i < 2 * half) {
                float sn, cs; sincosf((float)pos * a.inv_freq[i - half], &sn, &cs);
                v = (row_s[c] * cs + row_s[c - half] * sn) * a.rot_scale;
            } else {
                v = row_s[c];
            }
        }
        const T r = from_f<T>(v);
        if (keep) cache[c] = r;
        out[c] = r;
    }
}

// ---------------------------------------------------------------------------
constexpr int HL_TOK = 8, HL_ROWS = 4;

// y[t, h, o] = sum_i w[h, o, i] x[t, h, i]: eight tokens per CTA (their x in shared memory), a warp per group of four
// output rows whose weights are on their way together, 16 bytes per lane and load where the row allows it.
template <typename T>
__global__ void __launch_bounds__(128) head_linear_kernel(const T* __restrict__ x, long long x_stride, const T* __restrict__ w,
                                                          T* __restrict__ y, long long y_stride, int n_tokens, int in, int out) {
    pdl_launch_dependents();
    extern __shared__ float x_s[];                      // [HL_TOK][in]
    const int h = blockIdx.y, t0 = blockIdx.x * HL_TOK;
    const int nt = min(HL_TOK, n_tokens - t0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    pdl_wait();
    for (int i = threadIdx.x; i < HL_TOK * in; i += blockDim.x) {
        const int tt = i / in, c = i % in;
        x_s[i] = tt < nt ? to_f<T>(x[(size_t)(t0 + tt) * x_stride + (size_t)h * in + c]) : 0.f;
    }
    __syncthreads();
    const T* wh = w + (size_t)h * out * in;
    constexpr int VEC = 16 / sizeof(T);
    const bool vec = (in % VEC) == 0 && (((uintptr_t)wh) & 15) == 0;
    for (int o0 = (blockIdx.z * nwarp + warp) * HL_ROWS; o0 < out; o0 += gridDim.z * nwarp * HL_ROWS) {
        float acc[HL_ROWS][HL_TOK];
#pragma unroll
        for (int r = 0; r < HL_ROWS; r++)
#pragma unroll
            for (int tt = 0; tt < HL_TOK; tt++) acc[r][tt] = 0.f;
        if (vec) {
            for (int c = lane * VEC; c < in; c += 32 * VEC) {
                uint4 wv[HL_ROWS];
#pragma unroll
                for (int r = 0; r < HL_ROWS; r++)
                    wv[r] = (o0 + r < out) ? *(const uint4*)(wh + (size_t)(o0 + r) * in + c) : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int r = 0; r < HL_ROWS; r++) {
                    const T* e = (const T*)&wv[r];
#pragma unroll
                    for (int k = 0; k < VEC; k++) {
                        const float wf = to_f<T>(e[k]);
#pragma unroll
                        for (int tt = 0; tt < HL_TOK; tt++) acc[r][tt] = fmaf(wf, x_s[tt * in + c + k], acc[r][tt]);
                    }
                }
            }
        } else {
            for (int c = lane; c < in; c += 32) {
#pragma unroll
                for (int r = 0; r < HL_ROWS; r++) {
                    const float wf = (o0 + r < out) ? to_f<T>(wh[(size_t)(o0 + r) * in + c]) : 0.f;
#pragma unroll
                    for (int tt = 0; tt < HL_TOK; tt++) acc[r][tt] = fmaf(wf, x_s[tt * in + c], acc[r][tt]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < HL_ROWS; r++)
#pragma unroll
            for (int tt = 0; tt < HL_TOK; tt++) {
                const float sum = warp_sum(acc[r][tt]);
                if (lane == 0 && tt < nt && o0 + r < out) y[(size_t)(t0 + tt) * y_stride + (size_t)h * out + o0 + r] = from_f<T>(sum);
            }
    }
}

extern "C" int tb_head_linear(const void* x, long long x_stride, const void* w, void* y, long long y_stride, int dtype,
                              int n_tokens, int heads, int in, int out, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (heads <= 0 || heads > 65535 || in <= 0 || out <= 0 || in > 1536)
        return tb_refuse("head_linear: heads=%d in=%d out=%d (in at most 1536)", heads, in, out);
    int zs = (out + 4 * HL_ROWS - 1) / (4 * HL_ROWS);          // a CTA's four warps take 16 rows a round
    if (zs > 64) zs = 64;
    dim3 grid((n_tokens + HL_TOK - 1) / HL_TOK, heads, zs);
    TB_DISPATCH_1(dtype, T, tb_launch(head_linear_kernel<T>, dim3(grid), dim3(128), (size_t)HL_TOK * in * sizeof(float), stream,
                                      (const T*)x, x_stride, (const T*)w, (T*)y, y_stride, n_tokens, in, out));
    return tb_launch_status();
}

extern "C" int tb_latent_rows(const LatentRowsArgs* args, int dtype, cudaStream_t stream) {
    const LatentRowsArgs& a = *args;
    if (a.n_tokens <= 0) return 0;
    if (a.C <= 0 || a.R < 0 || a.rot_dims < 0 || a.rot_dims % 2 || a.rot_dims > a.R || a.page_rows <= 0)
        return tb_refuse("latent_rows: C=%d R=%d rot_dims=%d page_rows=%d", a.C, a.R, a.rot_dims, a.page_rows);
    if (a.Q < 0 || a.n_gate < 0 || (a.Q > 0 && (a.q_norm_w == nullptr || a.cq_out == nullptr)) || (a.n_gate > 0 && a.gate_out == nullptr))
        return tb_refuse("latent_rows: Q=%d gate=%d need their outputs", a.Q, a.n_gate);
    if (a.ring_rows > 0 && (a.ring_rows % a.page_rows || a.len_after == nullptr))
        return tb_refuse("latent_rows: a ring of %d rows needs whole pages and the sequences' lengths", a.ring_rows);
    // few tokens (a decode step) are a chain of memory waits per thread: eight times the threads a token shorten it
    const int threads = a.n_tokens <= 2 * 148 ? 1024 : 128;
    TB_DISPATCH_1(dtype, T, tb_launch(latent_rows_kernel<T>, dim3(a.n_tokens), dim3(threads),
                                      (size_t)(a.C + a.R + a.Q + a.n_gate) * sizeof(float), stream, a));
    return tb_launch_status();
}

// ---------------------------------------------------------------------------
struct LatentDecodeArgs {
    const void* q; long long q_stride;                 // [batch] rows of heads * (C + R): the mapped queries
    const void* pool;                                  // [pages][page_rows][C + R]
    const int* page_table; int pt_stride; int page_rows;
    const int* len_after;                              // [batch] rows in the cache, the new token's included
    const float* sink;                                 // [heads] or null
    void* out; long long out_stride;                   // [batch] rows of heads * out_dim; the first C of a head are written
    float* partial;                                    // [batch][heads][splits][C + 2] when splits > 1
    int heads, C, R, out_dim, n_splits;
    float scale;
    int window;                                        // 0: every earlier row; W: the last W rows, the query's own included
    int ring_rows;                                     // 0: row = position; else row = position mod ring_rows
};

__device__ __forceinline__ int latent_first_key(int window, int len) { return (window > 0 && len > window) ? len - window : 0; }

template <int NC>
struct LatAcc {
    float m, l, o[NC];
    __device__ void init() { m = -INFINITY; l = 0.f;
#pragma unroll
        for (int c = 0; c < NC; c++) o[c] = 0.f; }
};

template <typename T, int NC>
__global__ void __launch_bounds__(128) latent_decode_kernel(LatentDecodeArgs a) {
    pdl_launch_dependents();
    extern __shared__ float smem[];
    const int b = blockIdx.x, h = blockIdx.y, split = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int KD = a.C + a.R, C = a.C;
    float* q_s = smem;                                 // [KD]
    float* red = smem + KD;                            // [nwarp][C + 2]
    pdl_wait();
    const T* qrow = (const T*)a.q + (size_t)b * a.q_stride + (size_t)h * KD;
    for (int e = threadIdx.x; e < KD; e += blockDim.x) q_s[e] = to_f<T>(qrow[e]);
    __syncthreads();
    const int len = a.len_after[b];
    const int lo = latent_first_key(a.window, len), lo32 = lo & ~31;
    int per = (len - lo32 + a.n_splits - 1) / a.n_splits;
    per = (per + 31) & ~31;
    const int beg = lo32 + split * per, end = min(len, beg + per);
    const int* pt = a.page_table + (size_t)b * a.pt_stride;

    LatAcc<NC> acc; acc.init();
    for (int j0 = beg + warp * 32; j0 < end; j0 += nwarp * 32) {
        const int j = j0 + lane;
        const bool valid = j < end && j >= lo;
        const T* krow = nullptr;
        float s = -INFINITY;
        if (valid) {
            const int r = a.ring_rows > 0 ? j % a.ring_rows : j;
            krow = (const T*)a.pool + ((size_t)pt[r / a.page_rows] * a.page_rows + (r % a.page_rows)) * KD;
            float d = 0.f;
            for (int e = 0; e < KD; e++) d = fmaf(q_s[e], to_f<T>(krow[e]), d);
            s = d * a.scale;
        }
        const float cm = warp_max(s);
        if (cm == -INFINITY) continue;                 // 32 rows before the window's first
        const float m_new = fmaxf(acc.m, cm);
        const float corr = (acc.m == -INFINITY) ? 0.f : expf(acc.m - m_new);
        const float p = valid ? expf(s - m_new) : 0.f;
        acc.l = acc.l * corr + warp_sum(p);
        acc.m = m_new;
#pragma unroll
        for (int c = 0; c < NC; c++) acc.o[c] *= corr;
        for (int jj = 0; jj < 32; jj++) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const unsigned long long vp = __shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)krow, jj);
            if (pj == 0.f) continue;
            const T* v = (const T*)(uintptr_t)vp;
#pragma unroll
            for (int c = 0; c < NC; c++) { const int d = lane + 32 * c; if (d < C) acc.o[c] = fmaf(pj, to_f<T>(v[d]), acc.o[c]); }
        }
    }
    float* mine = red + (size_t)warp * (C + 2);
    if (lane == 0) { mine[C] = acc.m; mine[C + 1] = acc.l; }
#pragma unroll
    for (int c = 0; c < NC; c++) { const int d = lane + 32 * c; if (d < C) mine[d] = acc.o[c]; }
    __syncthreads();
    const float sink = (a.sink != nullptr) ? a.sink[h] : -INFINITY;
    float M = (a.n_splits == 1) ? sink : -INFINITY;
    for (int w = 0; w < nwarp; w++) M = fmaxf(M, red[(size_t)w * (C + 2) + C]);
    float L = 0.f;
    for (int w = 0; w < nwarp; w++) {
        const float mw = red[(size_t)w * (C + 2) + C];
        if (mw != -INFINITY) L += red[(size_t)w * (C + 2) + C + 1] * expf(mw - M);
    }
    if (a.n_splits == 1 && sink != -INFINITY) L += expf(sink - M);
    for (int d = threadIdx.x; d < C; d += blockDim.x) {
        float o = 0.f;
        for (int w = 0; w < nwarp; w++) {
            const float mw = red[(size_t)w * (C + 2) + C];
            if (mw != -INFINITY) o += red[(size_t)w * (C + 2) + d] * expf(mw - M);
        }
        if (a.n_splits == 1) ((T*)a.out)[(size_t)b * a.out_stride + (size_t)h * a.out_dim + d] = from_f<T>(o / L);
        else a.partial[(((size_t)b * a.heads + h) * a.n_splits + split) * (C + 2) + d] = o;
    }
    if (a.n_splits > 1 && threadIdx.x == 0) {
        float* p = a.partial + (((size_t)b * a.heads + h) * a.n_splits + split) * (C + 2);
        p[C] = M; p[C + 1] = L;
    }
}

template <typename T>
__global__ void __launch_bounds__(128) latent_combine_kernel(LatentDecodeArgs a) {
    pdl_launch_dependents();
    __shared__ float f_s[128];                           // e^(m_s - M) of up to 128 splits at a time
    __shared__ float M_s, L_s;
    pdl_wait();
    const int b = blockIdx.x, h = blockIdx.y, C = a.C, n = a.n_splits;
    const float* p = a.partial + ((size_t)b * a.heads + h) * n * (C + 2);
    const float sink = (a.sink != nullptr) ? a.sink[h] : -INFINITY;
    if (threadIdx.x < 32) {
        float m = sink;
        for (int s = threadIdx.x; s < n; s += 32) m = fmaxf(m, p[(size_t)s * (C + 2) + C]);
        m = warp_max(m);
        float l = 0.f;
        for (int s = threadIdx.x; s < n; s += 32) {
            const float ms = p[(size_t)s * (C + 2) + C];
            if (ms != -INFINITY) l += p[(size_t)s * (C + 2) + C + 1] * expf(ms - m);
        }
        l = warp_sum(l);
        if (threadIdx.x == 0) { M_s = m; L_s = l + ((sink != -INFINITY) ? expf(sink - m) : 0.f); }
    }
    __syncthreads();
    const float M = M_s, inv = 1.f / L_s;
    float o[4] = {0.f, 0.f, 0.f, 0.f};                   // columns threadIdx.x + 128 k (C <= 512)
    for (int s0 = 0; s0 < n; s0 += 128) {
        const int ns = min(128, n - s0);
        __syncthreads();
        if (threadIdx.x < ns) {
            const float ms = p[(size_t)(s0 + threadIdx.x) * (C + 2) + C];
            f_s[threadIdx.x] = (ms != -INFINITY) ? expf(ms - M) : 0.f;
        }
        __syncthreads();
        for (int s = 0; s < ns; s++) {
            const float f = f_s[s];
            const float* ps = p + (size_t)(s0 + s) * (C + 2);
#pragma unroll
            for (int k = 0; k < 4; k++) { const int d = threadIdx.x + 128 * k; if (d < C) o[k] = fmaf(ps[d], f, o[k]); }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int d = threadIdx.x + 128 * k;
        if (d < C) ((T*)a.out)[(size_t)b * a.out_stride + (size_t)h * a.out_dim + d] = from_f<T>(o[k] * inv);
    }
}

// ---------------------------------------------------------------------------
// The same decode on tensor cores (bfloat16): one CTA an SM takes up to 16 heads of a sequence and a range of its keys, so
// that a cached row is fetched once for all of them.  A warp of its own brings rows by tiled TMA copies (boxes of 32 rows x 64
// numbers with the 128-byte swizzle; a bulk copy a row came to 24 GB/s an SM), half a page at a time, into a ring that fills
// the shared memory (6 stages of 32 KB for rows of 512 numbers); KG groups of four warps take the tiles in turn, each with a
// softmax and sums of its own, so that one group's chain of instructions (scores, softmax, outputs; two barriers of the group)
// runs beside the others' and the copies never stop.  S = Q' K^T with 16 heads as the rows of mma.sync m16n8k16: a warp
// takes a quarter of the row's numbers for all 32 keys, so that its queries stay in registers and a row is read once (a
// quarter of the keys each read the queries from shared memory for every tile, most of its traffic); the four parts are
// added on the way into the softmax (eight threads a head).  O += P C with every warp taking a share of the latent's columns.
// The groups' sums meet in shared memory; the pieces of a sequence, as the CTAs of a cluster, in distributed shared memory
// (with the sink), or else as partial (max, sum, o) that latent_combine_kernel folds.
// 64 sequences of 1,536 to 2,048 rows of 448 + 64 numbers, 16 heads: 70 -> 42 us, at twice the rows 128 -> 68 (3.5 TB/s; the
// kernel before: a two-stage cp.async ring, all warps meeting at four barriers a tile); 32 heads take the rows twice (the
// second time from L2): 93 -> 68.  The copies alone would take 29 us, the groups' chains alone 35.
// ---------------------------------------------------------------------------
constexpr int LD_BN = 32, LD_SP = LD_BN + 4, LD_PP = LD_BN * 2 + 16;       // keys a tile; pitches of scores (floats) and weights (bytes)
constexpr int LD_H = 16, LD_GT = 128, LD_GW = 4;                           // heads of a CTA; threads and warps of a group

__device__ int g_latent_error = 0;

__device__ __forceinline__ uint32_t ld_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ld_ldsm4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ld_ldsm4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ld_mma(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ld_box(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1) : "memory");
}
// Byte offset of (row, 16-byte piece) in a tile: boxes of 64 numbers, [32 rows][128 bytes] each, pieces swizzled by the row.
constexpr int LD_BOX = LD_BN * 128;
__device__ __forceinline__ int ld_off(int row, int piece) { return (piece >> 3) * LD_BOX + row * 128 + (((piece & 7) ^ (row & 7)) << 4); }
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(LD_GT) : "memory"); }

// Bytes of a CTA's shared memory before the ring (1024: the ring's alignment), and of a tile of the ring.
template <int KG>
__host__ __device__ constexpr int ld_head_bytes() { return KG * LD_H * (4 * LD_SP * 4 + LD_PP + 4 + 8) + 256 + 1024; }
__host__ __device__ constexpr int ld_tile_bytes(int KD) { return (KD + 63) / 64 * LD_BOX; }

// NP: pairs of 8-column tiles of the latent per warp (C <= NP * 64).  KS: steps of 16 numbers of a row that a warp scores
// (C + R <= KS * 64).  CL: up to how many pieces meet in a cluster.  stages: tiles the ring holds (2 .. 16).
template <int NP, int KS, int KG, int CL>
__global__ void __launch_bounds__((LD_GW * KG + 1) * 32, 1)
latent_decode_mma_kernel(LatentDecodeArgs a, const __grid_constant__ CUtensorMap rows, int stages, int in_cluster) {
    pdl_launch_dependents();
    constexpr int HEADS = LD_H, MMA_WARPS = LD_GW * KG;
    extern __shared__ __align__(128) unsigned char sm[];
    const int KD = a.C + a.R, C = a.C, boxes = (KD + 63) / 64, tile = boxes * LD_BOX;
    uint64_t* full = (uint64_t*)sm;                                 // [16] the tile is there
    uint64_t* empty = full + 16;                                    // [16] its group has read it
    float* s_all = (float*)(sm + 256);                              // [KG][4][HEADS][LD_SP] parts of the scores
    float* corr_all = s_all + KG * 4 * HEADS * LD_SP;               // [KG][HEADS]
    float* ml_s = corr_all + KG * HEADS;                            // [KG][HEADS][2] maximum and sum
    unsigned char* p_all = (unsigned char*)(ml_s + KG * HEADS * 2); // [KG][HEADS][LD_PP] weights
    unsigned char* ring = (unsigned char*)(((uintptr_t)(p_all + KG * HEADS * LD_PP) + 1023) & ~(uintptr_t)1023);   // [stages] tiles, in the end [KG - 1][HEADS][C] sums
    const int b = blockIdx.x, h0 = blockIdx.y * HEADS, nh = min(HEADS, a.heads - h0), split = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; i++) { mbar_init(full + i, 1); mbar_init(empty + i, LD_GW); }
        mbar_init_fence();
    }
    pdl_wait();
    const int len = a.len_after[b];
    const int lo = latent_first_key(a.window, len), lo32 = lo / LD_BN * LD_BN;
    int per = (len - lo32 + a.n_splits - 1) / a.n_splits;
    per = (per + LD_BN - 1) / LD_BN * LD_BN;
    const int beg = lo32 + split * per, end = min(len, beg + per);
    const int n_tiles = beg < end ? (end - beg + LD_BN - 1) / LD_BN : 0;
    __syncthreads();
    bool bad = false;                                               // a wait ran out: no more waiting, the result is void
    auto wait = [&](uint64_t* bar, int use) {                       // the use-th completion of the barrier, counted from 0
        if (!bad && !mbar_wait(bar, use & 1)) { bad = true; g_latent_error = 1; }
    };
    float o[NP * 2][4];
#pragma unroll
    for (int n = 0; n < NP * 2; n++) { o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f; }
    const int kg = warp / LD_GW, w = warp % LD_GW, gt = threadIdx.x - kg * LD_GT;
    if (warp == MMA_WARPS) {
        // ---- the copies: a lane a box; the page numbers of 32 tiles at a time, asked for together
        const int* pt = a.page_table + (size_t)b * a.pt_stride;
        int row_of = 0;
        for (int it = 0; it < n_tiles; it++) {
            if (it % 32 == 0 && it + lane < n_tiles) {
                const int j = beg + (it + lane) * LD_BN, r = a.ring_rows > 0 ? j % a.ring_rows : j;    // 32 rows from a multiple of 32 on lie in one page
                row_of = pt[r / a.page_rows] * a.page_rows + r % a.page_rows;
            }
            const int st = it % stages, row = __shfl_sync(0xffffffffu, row_of, it % 32);
            if (it >= stages) wait(empty + st, it / stages - 1);
            if (lane == 0) mbar_expect_tx(full + st, (uint32_t)tile);
            __syncwarp();
            if (lane < boxes) ld_box(ring + (size_t)st * tile + lane * LD_BOX, &rows, full + st, lane * 64, row);
        }
        // every copy has landed before the ring becomes something else
        for (int it = max(0, n_tiles - stages); it < n_tiles; it++)
            if (!mbar_wait(full + it % stages, (it / stages) & 1)) g_latent_error = 1;
    } else {
        float* s_s = s_all + kg * 4 * HEADS * LD_SP;
        float* corr_s = corr_all + kg * HEADS;
        unsigned char* p_s = p_all + kg * HEADS * LD_PP;
        const int hr = gt >> 3, k4 = (gt & 7) * 4;                  // softmax: this thread's head and four keys
        float m_run = -INFINITY, l_run = 0.f;                       // (every one of a head's eight threads)
        const int first = w * KS, steps = min(KS, KD / 16 - first); // this warp's 16-number steps of a row
        uint32_t q[KS][4];                                          // its part of the queries (heads past the last one: zeros)
        {
            const int ra = lane >> 2, c = (lane & 3) * 2;
            const bf16* qa = (const bf16*)a.q + (size_t)b * a.q_stride + (size_t)(h0 + ra) * KD + first * 16 + c;
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                const bool in = ks < steps, ia = in && ra < nh, ib = in && ra + 8 < nh;
                q[ks][0] = ia ? *(const uint32_t*)(qa + ks * 16) : 0u;
                q[ks][1] = ib ? *(const uint32_t*)(qa + (size_t)8 * KD + ks * 16) : 0u;
                q[ks][2] = ia ? *(const uint32_t*)(qa + ks * 16 + 8) : 0u;
                q[ks][3] = ib ? *(const uint32_t*)(qa + (size_t)8 * KD + ks * 16 + 8) : 0u;
            }
        }
        for (int it = kg; it < n_tiles; it += KG) {
            const int st = it % stages, j0 = beg + it * LD_BN;
            unsigned char* kt = ring + (size_t)st * tile;
            wait(full + st, it / stages);
            if (j0 < lo || j0 + LD_BN > end) {                      // rows that are not the sequence's keys: whatever the page holds there stays out
                for (int r = 0; r < LD_BN; r++)
                    if (j0 + r < lo || j0 + r >= end)
                        for (int c = gt; c < boxes * 8; c += LD_GT) *(uint4*)(kt + ld_off(r, c)) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // (before a later copy into this place)
                group_sync(kg);
            }
            // ---- this warp's part of the scores: 16 heads x 32 keys
            const uint32_t kb = ld_smem(kt);
            float sc[4][4];
#pragma unroll
            for (int n = 0; n < 4; n++) { sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f; }
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
                if (ks >= steps) break;                             // (the same in every lane)
#pragma unroll
                for (int n = 0; n < 4; n += 2) {
                    uint32_t f[4];
                    ld_ldsm4(kb + ld_off(n * 8 + (lane >> 4) * 8 + (lane & 7), (first + ks) * 2 + ((lane >> 3) & 1)), f[0], f[1], f[2], f[3]);
                    ld_mma(sc[n], q[ks], f[0], f[1]);
                    ld_mma(sc[n + 1], q[ks], f[2], f[3]);
                }
            }
            {
                float* d = s_s + (w * HEADS + (lane >> 2)) * LD_SP + (lane & 3) * 2;
#pragma unroll
                for (int n = 0; n < 4; n++) {
                    *(float2*)(d + n * 8) = make_float2(sc[n][0], sc[n][1]);
                    *(float2*)(d + n * 8 + 8 * LD_SP) = make_float2(sc[n][2], sc[n][3]);
                }
            }
            group_sync(kg);
            // ---- softmax: eight threads a head, four keys each
            {
                float4 sv[4];
#pragma unroll
                for (int x = 0; x < 4; x++) sv[x] = *(const float4*)(s_s + (x * HEADS + hr) * LD_SP + k4);
                float v[4] = {((sv[0].x + sv[1].x) + (sv[2].x + sv[3].x)) * a.scale, ((sv[0].y + sv[1].y) + (sv[2].y + sv[3].y)) * a.scale,
                              ((sv[0].z + sv[1].z) + (sv[2].z + sv[3].z)) * a.scale, ((sv[0].w + sv[1].w) + (sv[2].w + sv[3].w)) * a.scale};
                float mx = -INFINITY;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int j = j0 + k4 + e;
                    if (j >= end || j < lo) v[e] = -INFINITY;
                    mx = fmaxf(mx, v[e]);
                }
#pragma unroll
                for (int x = 1; x < 8; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
                const float mn = fmaxf(m_run, mx);
                const float corr = (m_run == -INFINITY) ? 0.f : expf(m_run - mn);
                float sum = 0.f;
#pragma unroll
                for (int e = 0; e < 4; e++) { v[e] = (v[e] == -INFINITY) ? 0.f : expf(v[e] - mn); sum += v[e]; }
#pragma unroll
                for (int x = 1; x < 8; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
                l_run = l_run * corr + sum;
                m_run = mn;
                __nv_bfloat162 pa = __floats2bfloat162_rn(v[0], v[1]), pb = __floats2bfloat162_rn(v[2], v[3]);
                *(uint2*)(p_s + hr * LD_PP + k4 * 2) = make_uint2(*(uint32_t*)&pa, *(uint32_t*)&pb);
                if ((gt & 7) == 0) corr_s[hr] = corr;
            }
            group_sync(kg);
            // ---- O = O * corr + P C, this warp's share of the latent's columns
            const float ca = corr_s[lane >> 2], cb = corr_s[(lane >> 2) + 8];
            uint32_t pa[LD_BN / 16][4];
#pragma unroll
            for (int kk = 0; kk < LD_BN / 16; kk++)
                ld_ldsm4(ld_smem(p_s + (lane & 15) * LD_PP + (kk * 16 + (lane >> 4) * 8) * 2), pa[kk][0], pa[kk][1], pa[kk][2], pa[kk][3]);
#pragma unroll
            for (int j = 0; j < NP; j++) {
                const int col0 = (j * LD_GW + w) * 16;
                if (col0 >= C) continue;
                float* oa = o[2 * j]; float* ob = o[2 * j + 1];
                oa[0] *= ca; oa[1] *= ca; oa[2] *= cb; oa[3] *= cb; ob[0] *= ca; ob[1] *= ca; ob[2] *= cb; ob[3] *= cb;
#pragma unroll
                for (int kk = 0; kk < LD_BN / 16; kk++) {
                    uint32_t b0, b1, b2, b3;
                    ld_ldsm4_t(kb + ld_off(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), col0 / 8 + (lane >> 4)), b0, b1, b2, b3);
                    ld_mma(oa, pa[kk], b0, b1);
                    ld_mma(ob, pa[kk], b2, b3);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + st);
        }
        if ((gt & 7) == 0) { ml_s[(kg * HEADS + hr) * 2] = m_run; ml_s[(kg * HEADS + hr) * 2 + 1] = l_run; }
    }
    // ---- the groups' sums meet: the ring becomes [KG - 1][HEADS][C] floats, the first group adds them to its own
    __syncthreads();
    float* o_s = (float*)ring;
    auto each = [&](auto&& f) {                                     // f(second of its two heads, head of the CTA, column, two neighbouring sums)
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const int col0 = (j * LD_GW + w) * 16;
            if (col0 >= C) continue;
#pragma unroll
            for (int half = 0; half < 2; half++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    f(e, (lane >> 2) + e * 8, col0 + half * 8 + (lane & 3) * 2, o[2 * j + half][2 * e], o[2 * j + half][2 * e + 1]);
        }
    };
    if (warp < MMA_WARPS && kg > 0)
        each([&](int, int r, int c, float& x, float& y) { *(float2*)(o_s + ((size_t)(kg - 1) * HEADS + r) * C + c) = make_float2(x, y); });
    __syncthreads();
    if (warp < LD_GW) {
        float f[2][KG];                                             // the groups' factors for this thread's heads
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int r = (lane >> 2) + e * 8;
            float M = -INFINITY;
#pragma unroll
            for (int k = 0; k < KG; k++) M = fmaxf(M, ml_s[(k * HEADS + r) * 2]);
#pragma unroll
            for (int k = 0; k < KG; k++) { const float mk = ml_s[(k * HEADS + r) * 2]; f[e][k] = mk == -INFINITY ? 0.f : expf(mk - M); }
        }
        each([&](int e, int r, int c, float& x, float& y) {
            x *= f[e][0]; y *= f[e][0];
#pragma unroll
            for (int k = 1; k < KG; k++) {
                const float2 z = *(const float2*)(o_s + ((size_t)(k - 1) * HEADS + r) * C + c);
                x = fmaf(z.x, f[e][k], x); y = fmaf(z.y, f[e][k], y);
            }
        });
    }
    __syncthreads();                                                // (maxima and sums have been read)
    if (threadIdx.x < HEADS) {
        float M = -INFINITY, L = 0.f;
#pragma unroll
        for (int k = 0; k < KG; k++) M = fmaxf(M, ml_s[(k * HEADS + threadIdx.x) * 2]);
#pragma unroll
        for (int k = 0; k < KG; k++) { const float mk = ml_s[(k * HEADS + threadIdx.x) * 2]; if (mk != -INFINITY) L += ml_s[(k * HEADS + threadIdx.x) * 2 + 1] * expf(mk - M); }
        ml_s[threadIdx.x * 2] = M; ml_s[threadIdx.x * 2 + 1] = L;   // (group 0's place: each head's thread reads it before)
    }
    if (!in_cluster) {
        // ---- partial results: [b][h][split][C + 2]
        __syncthreads();
        float* p = a.partial + (((size_t)b * a.heads + h0) * a.n_splits + split) * (C + 2);
        const size_t step = (size_t)a.n_splits * (C + 2);
        if (warp < LD_GW) each([&](int, int r, int c, float& x, float& y) { if (r < nh) { p[r * step + c] = x; p[r * step + c + 1] = y; } });
        if (threadIdx.x < nh) { p[threadIdx.x * step + C] = ml_s[threadIdx.x * 2]; p[threadIdx.x * step + C + 1] = ml_s[threadIdx.x * 2 + 1]; }
        return;
    }
    // ---- the pieces of the sequence meet: every CTA of the cluster adds and writes a slice of the outputs
    if (warp < LD_GW) each([&](int, int r, int c, float& x, float& y) { *(float2*)(o_s + (size_t)r * C + c) = make_float2(x, y); });
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int S = a.n_splits, rank = (int)cluster.block_rank();
    float* f_s = s_all;                                             // [HEADS][CL]: every piece's share of the result (the scores are done with)
    if (threadIdx.x < nh) {
        const int r = threadIdx.x;
        const float sink = (a.sink != nullptr) ? a.sink[h0 + r] : -INFINITY;
        float m[CL], l[CL], M = sink;
#pragma unroll
        for (int k = 0; k < CL; k++) {
            m[k] = -INFINITY; l[k] = 0.f;
            if (k < S) { const float2 ml = *(const float2*)(cluster.map_shared_rank(ml_s, k) + r * 2); m[k] = ml.x; l[k] = ml.y; }
        }
#pragma unroll
        for (int k = 0; k < CL; k++) M = fmaxf(M, m[k]);
        float L = (sink != -INFINITY) ? expf(sink - M) : 0.f;
#pragma unroll
        for (int k = 0; k < CL; k++) { m[k] = m[k] == -INFINITY ? 0.f : expf(m[k] - M); L += l[k] * m[k]; }
#pragma unroll
        for (int k = 0; k < CL; k++) f_s[r * CL + k] = m[k] / L;
    }
    __syncthreads();
    const int quads = C / 4, per_cta = (nh * quads + S - 1) / S;    // four neighbouring columns a thread and turn
    for (int i = rank * per_cta + threadIdx.x; i < min(nh * quads, (rank + 1) * per_cta); i += blockDim.x) {
        const int r = i / quads, c = (i - r * quads) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < CL; k++)
            if (k < S) {
                const float4 x = *(const float4*)(cluster.map_shared_rank(o_s, k) + (size_t)r * C + c);
                const float f = f_s[r * CL + k];
                v.x = fmaf(x.x, f, v.x); v.y = fmaf(x.y, f, v.y); v.z = fmaf(x.z, f, v.z); v.w = fmaf(x.w, f, v.w);
            }
        bf16* out = (bf16*)a.out + (size_t)b * a.out_stride + (size_t)(h0 + r) * a.out_dim + c;
        out[0] = __float2bfloat16_rn(v.x); out[1] = __float2bfloat16_rn(v.y); out[2] = __float2bfloat16_rn(v.z); out[3] = __float2bfloat16_rn(v.w);
    }
    cluster.sync();                                                 // nobody leaves while its sums are being read
}

extern "C" int tb_latent_decode_mma_takes(int C, int R) {
    return C > 0 && C % 16 == 0 && (C + R) % 16 == 0 && C <= 512 && (C + R) <= 1024;
}

// Reads and clears the error word (1: a bounded wait on a copy of rows ran out; that launch's results are void).  Synchronises.
extern "C" int tb_latent_decode_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_latent_error, sizeof v) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_latent_error, &zero, sizeof zero);
    return v;
}

// Which pieces meet in a cluster: one, two or four (three leave SMs of a GPC empty), eight where that is up to 64 CTAs
// (128 sequences' pieces in clusters of eight take two rounds).
static int latent_units(int batch, int heads) { return batch * ((heads + LD_H - 1) / LD_H); }
static bool latent_in_cluster(int pieces, int units) { return pieces == 1 || pieces == 2 || pieces == 4 || (pieces == 8 && units <= 8); }
extern "C" int tb_latent_decode_folds(int pieces, int batch, int heads) { return !latent_in_cluster(pieces, latent_units(batch, heads)); }
// In how many pieces a launch of `batch` sequences of up to `rows` keys cuts each: the least of a cost in us that was fitted to
// 236 launches, each timed in up to 21 counts (1 to 64 units of 300 to 8,192 rows of 512 numbers): 6 and 2.4 a turn of the three
// groups for every round of CTAs (one an SM; contexts lie between their bucket's half and its end: 0.8 of it), and for the launch
// that folds 3.7, 0.18 a piece and, beyond four fifths of the SMs, up to 2 more (it starts on the free ones).  A piece's share of
// the start-up alone, as before, cut too finely: 5 sequences of 3,000 rows in 29 pieces 24 to 31 us, in 18: 22, in 12: 20.
// Clusters of four and eight do not fill more than one round (96 units of 3,000 rows in four: 95 us, in three: 79).
extern "C" int tb_latent_decode_pieces(int batch, int heads, int rows, int sms) {
    const int units = latent_units(batch, heads), tiles = (rows + LD_BN - 1) / LD_BN;
    int best = 1;
    double least = 0.0;
    for (int s = 1; s <= 64 && (s == 1 || s * 3 <= tiles + 2); s++) {
        const long long ctas = (long long)units * s, rounds = (ctas + sms - 1) / sms;
        const int usual = (int)((tiles * 4 + 5LL * s - 1) / (5LL * s));          // tiles of a piece
        double cost = (double)rounds * (6.0 + 2.4 * ((usual + 2) / 3));
        const double full = (double)ctas / ((double)rounds * sms) - 0.8;
        if (!latent_in_cluster(s, units)) cost += 3.7 + 0.18 * s + (full > 0.0 ? 10.0 * full : 0.0);
        else if (s >= 4 && rounds > 1) cost *= 2.0;
        if (s == 1 || cost < least - 1e-9) { best = s; least = cost; }
    }
    return best;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The pool as a matrix of rows of KD numbers (how many is not known here: the page table decides which are read); numbers
// past a row's end come as zeros.
static int rows_map(CUtensorMap* m, const void* pool, int KD) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
        if (!fn) return tb_refuse("latent_decode: the driver does not provide cuTensorMapEncodeTiled");
    }
    const cuuint64_t dims[2] = {(cuuint64_t)KD, (cuuint64_t)0x7fffff00}, strides[1] = {(cuuint64_t)KD * 2};
    const cuuint32_t box[2] = {64, LD_BN}, one[2] = {1, 1};
    const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)pool, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : tb_refuse("latent_decode: cuTensorMapEncodeTiled failed with %d", (int)r);
}

template <int NP, int KS, int KG, int CL>
static int run_latent_mma(const LatentDecodeArgs& a, int batch, cudaStream_t stream) {
    const int KD = a.C + a.R, head = ld_head_bytes<KG>(), tile = ld_tile_bytes(KD);
    int stages = (227 * 1024 - head) / tile;
    stages = stages > 16 ? 16 : stages;
    if (stages < 2) return tb_refuse("latent_decode_mma: rows of %d numbers leave no room for two tiles", KD);
    const int smem = head + stages * tile;
    const bool in_cluster = latent_in_cluster(a.n_splits, latent_units(batch, a.heads));
    const cudaError_t e = cudaFuncSetAttribute(latent_decode_mma_kernel<NP, KS, KG, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(batch, (a.heads + LD_H - 1) / LD_H, a.n_splits); cfg.blockDim = dim3((LD_GW * KG + 1) * 32);
    cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = in_cluster ? a.n_splits : 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    CUtensorMap rows;
    if (rows_map(&rows, a.pool, KD)) return -1;
    cudaLaunchKernelEx(&cfg, latent_decode_mma_kernel<NP, KS, KG, CL>, a, rows, stages, (int)in_cluster);
    int st = tb_launch_status();
    if (st || in_cluster) return st;
    tb_launch(latent_combine_kernel<bf16>, dim3(batch, a.heads), dim3(128), 0, stream, a);
    return tb_launch_status();
}

extern "C" int tb_latent_decode_mma(const LatentDecodeArgs* args, int batch, cudaStream_t stream) {
    if (batch <= 0) return 0;
    const LatentDecodeArgs& a = *args;
    if (!tb_latent_decode_mma_takes(a.C, a.R)) return tb_refuse("latent_decode_mma: C=%d R=%d (multiples of 16, C <= 512)", a.C, a.R);
    if (a.n_splits < 1 || a.n_splits > 65535 || (a.partial == nullptr && !latent_in_cluster(a.n_splits, latent_units(batch, a.heads))) || a.out_dim < a.C || a.page_rows % LD_BN)
        return tb_refuse("latent_decode_mma: n_splits=%d needs scratch; pages of %d rows", a.n_splits, a.page_rows);
    if (((uintptr_t)a.q & 15) || (a.q_stride % 8) || ((uintptr_t)a.pool & 15)) return tb_refuse("latent_decode_mma: rows must be 16-byte aligned");
    const int KD = a.C + a.R;
#define LD_RUN(N, K, G) (a.n_splits == 8 ? run_latent_mma<N, K, G, 8>(a, batch, stream) : run_latent_mma<N, K, G, 4>(a, batch, stream))
    return KD <= 256 ? LD_RUN(4, 4, 3) : KD <= 512 ? LD_RUN(8, 8, 3) : LD_RUN(8, 16, 2);
#undef LD_RUN
}

extern "C" int tb_latent_decode(const LatentDecodeArgs* args, int dtype, int batch, cudaStream_t stream) {
    if (batch <= 0) return 0;
    const LatentDecodeArgs& a = *args;
    if (a.heads <= 0 || a.heads > 65535 || a.C <= 0 || a.R < 0 || a.C > 512 || a.out_dim < a.C)
        return tb_refuse("latent_decode: heads=%d C=%d R=%d out_dim=%d (C at most 512)", a.heads, a.C, a.R, a.out_dim);
    if (a.n_splits < 1 || a.n_splits > 65535 || (a.n_splits > 1 && a.partial == nullptr))
        return tb_refuse("latent_decode: n_splits=%d needs scratch", a.n_splits);
    const int warps = 4;
    const size_t smem = ((size_t)(a.C + a.R) + (size_t)warps * (a.C + 2)) * sizeof(float);
    int nc = 1;
    while (nc * 32 < a.C) nc <<= 1;
    dim3 grid(batch, a.heads, a.n_splits);
#define LAT_DEC(N) TB_DISPATCH_1(dtype, T, tb_launch(latent_decode_kernel<T, N>, dim3(grid), dim3(warps * 32), smem, stream, a))
    switch (nc) {
    case 1: LAT_DEC(1); break;
    case 2: LAT_DEC(2); break;
    case 4: LAT_DEC(4); break;
    case 8: LAT_DEC(8); break;
    default: LAT_DEC(16); break;
    }
    int st = tb_launch_status();
    if (st || a.n_splits == 1) return st;
    TB_DISPATCH_1(dtype, T, tb_launch(latent_combine_kernel<T>, dim3(batch, a.heads), dim3(128), 0, stream, a));
    return tb_launch_status();
}
