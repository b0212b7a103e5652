// Choosing the next token from 32-bit logits, on the device.
//
//   tb_argmax  greedy: the largest logit, the smallest index on a tie.  Two stages
//              like the reference's argmax_stage1/2 (runtime/cuda/codebook_gemv.cu:544-591),
//              but for many rows at once; stage 1 writes (value, index) per chunk
//              to scratch, stage 2 folds the chunks in order.
//   tb_sample  what the reference's server does on the host (runtime/src/bin/serve.rs:41-72,
//              285-294), per row and in this order:
//                1. repetition penalty over the row's recent tokens, each distinct id
//                   once: logit > 0 ? logit / penalty : logit * penalty  (off if <= 1)
//                2. temperature <= 0: argmax.  Otherwise p_i ~ exp((l_i - max) / T)
//                3. nucleus: the smallest set of most probable tokens whose mass
//                   reaches top_p (all tokens if top_p >= 1)
//                4. a draw u in [0,1), given by the caller, picks the token at which
//                   the running sum of kept p_i, taken in index order, passes
//                   u * (kept mass)
//              The reference sorts and keeps the 256 largest logits before step 3
//              and walks them in sorted order; the kept set is the same whenever
//              the nucleus has at most 256 tokens, and the distribution of the
//              draw is the same.  Its draw comes from a xorshift seeded by the
//              wall clock; here the caller owns the generator, so a run repeats.
//
// All sums are 32-bit and taken in a fixed order.
#include <cooperative_groups.h>
#include "common.cuh"

namespace cg = cooperative_groups;

TB_EXPORT_ERROR()

#define ARGMAX_CHUNK 8192

struct ValIdx { float v; int i; };

__device__ __forceinline__ ValIdx better(ValIdx a, ValIdx b) {
    // NaN never wins; ties go to the smaller index
    if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
    return a;
}

__device__ __forceinline__ ValIdx block_best(ValIdx x, ValIdx* red /* 32 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ValIdx y; y.v = __shfl_xor_sync(0xffffffffu, x.v, o); y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
        x = better(x, y);
    }
    __syncthreads();
    if (lane == 0) red[warp] = x;
    __syncthreads();
    ValIdx t; t.v = -INFINITY; t.i = 0x7fffffff;
    if (lane < nwarp) t = red[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ValIdx y; y.v = __shfl_xor_sync(0xffffffffu, t.v, o); y.i = __shfl_xor_sync(0xffffffffu, t.i, o);
        t = better(t, y);
    }
    return t;
}

__global__ void argmax_stage1_kernel(const float* __restrict__ logits, long long row_stride, int vocab,
                                     float* __restrict__ pval, int* __restrict__ pidx, int n_chunks) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ ValIdx red[32];
    const int row = blockIdx.y, chunk = blockIdx.x;
    const float* x = logits + (size_t)row * row_stride;
    const int beg = chunk * ARGMAX_CHUNK, end = min(vocab, beg + ARGMAX_CHUNK);
    ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
    for (int i = beg + threadIdx.x; i < end; i += blockDim.x) { ValIdx c; c.v = x[i]; c.i = i; b = better(b, c); }
    b = block_best(b, red);
    if (threadIdx.x == 0) { pval[(size_t)row * n_chunks + chunk] = b.v; pidx[(size_t)row * n_chunks + chunk] = b.i; }
}

__global__ void argmax_stage2_kernel(const float* __restrict__ pval, const int* __restrict__ pidx,
                                     int n_chunks, int* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ ValIdx red[32];
    const int row = blockIdx.x;
    ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
    for (int i = threadIdx.x; i < n_chunks; i += blockDim.x) {
        ValIdx c; c.v = pval[(size_t)row * n_chunks + i]; c.i = pidx[(size_t)row * n_chunks + i];
        b = better(b, c);
    }
    b = block_best(b, red);
    if (threadIdx.x == 0) out[row] = (b.i == 0x7fffffff) ? 0 : b.i;
}

extern "C" long long tb_argmax_scratch_bytes(int rows, int vocab) {
    const long long chunks = (vocab + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
    return (long long)rows * chunks * 8;
}

extern "C" int tb_argmax(const float* logits, long long row_stride, int rows, int vocab, int* out,
                         void* scratch, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0) return tb_refuse("argmax: vocab=%d", vocab);
    if (rows > 65535) return tb_refuse("argmax: %d rows is more than one call takes", rows);
    const int n_chunks = (vocab + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
    float* pval = (float*)scratch;
    int* pidx = (int*)(pval + (size_t)rows * n_chunks);
    dim3 grid(n_chunks, rows);
    tb_launch(argmax_stage1_kernel, dim3(grid), dim3(256), 0, stream, logits, row_stride, vocab, pval, pidx, n_chunks);
    tb_launch(argmax_stage2_kernel, dim3(rows), dim3(128), 0, stream, pval, pidx, n_chunks, out);
    return tb_launch_status();
}

// ---------------------------------------------------------------------------
// Sampling: one CTA per row.
// ---------------------------------------------------------------------------

// Floats as unsigned keys whose order is the floats' order.
__device__ __forceinline__ unsigned f2key(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key2f(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct SampleArgs {
    float* logits; long long row_stride; int vocab;
    const float* temperature;      // [rows]
    const float* top_p;            // [rows]
    const float* penalty;          // [rows]
    const float* draw;             // [rows] u in [0,1)
    const int* recent; int n_recent;   // [rows, n_recent] recent token ids, -1 = none
    int* out;                      // [rows]
};

__global__ void __launch_bounds__(1024) sample_kernel(SampleArgs a) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[33];
    __shared__ ValIdx redvi[32];
    __shared__ float scan[1024];
    __shared__ int chosen;
    const int row = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    float* x = a.logits + (size_t)row * a.row_stride;
    const int V = a.vocab;

    // 1. repetition penalty, each distinct recent id once
    const float pen = a.penalty ? a.penalty[row] : 1.f;
    if (pen > 1.f && a.recent) {
        const int* rec = a.recent + (size_t)row * a.n_recent;
        for (int j = tid; j < a.n_recent; j += nt) {
            const int id = rec[j];
            if (id < 0 || id >= V) continue;
            bool first = true;
            for (int k = 0; k < j; k++) if (rec[k] == id) { first = false; break; }
            if (first) { const float l = x[id]; x[id] = l > 0.f ? l / pen : l * pen; }
        }
        __syncthreads();
    }

    // 2. greedy
    const float T = a.temperature ? a.temperature[row] : 0.f;
    if (!(T > 0.f)) {
        ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
        for (int i = tid; i < V; i += nt) { ValIdx c; c.v = x[i]; c.i = i; b = better(b, c); }
        b = block_best(b, redvi);
        if (tid == 0) a.out[row] = (b.i == 0x7fffffff) ? 0 : b.i;
        return;
    }

    float mx = -INFINITY;
    for (int i = tid; i < V; i += nt) mx = fmaxf(mx, x[i]);
    mx = block_max(mx, red);
    const float invT = 1.f / T;
    float z = 0.f;
    for (int i = tid; i < V; i += nt) z += expf((x[i] - mx) * invT);
    z = block_sum(z, red);

    // 3. nucleus: the largest threshold key whose mass still reaches top_p * z
    const float top_p = a.top_p ? a.top_p[row] : 1.f;
    unsigned thr = 0u;                               // keep everything
    float kept = z;
    if (top_p < 1.f) {
        const float want = top_p * z;
        unsigned lo = 0u;                            // mass(lo) >= want always holds
        for (int bit = 31; bit >= 0; bit--) {
            const unsigned cand = lo | (1u << bit);
            float s = 0.f;
            for (int i = tid; i < V; i += nt) { const float l = x[i]; if (f2key(l) >= cand) s += expf((l - mx) * invT); }
            s = block_sum(s, red);
            if (s >= want) { lo = cand; kept = s; }
        }
        thr = lo;
    }

    // 4. inverse CDF over the kept tokens in index order
    const float target = a.draw[row] * kept;
    const int per = (V + nt - 1) / nt;
    const int beg = min(V, tid * per), end = min(V, beg + per);
    float mine = 0.f;
    for (int i = beg; i < end; i++) { const float l = x[i]; if (f2key(l) >= thr) mine += expf((l - mx) * invT); }
    scan[tid] = mine;
    if (tid == 0) chosen = -1;
    __syncthreads();
    if (tid == 0) {                                   // serial prefix over 1024 partial sums: fixed order
        float run = 0.f;
        for (int t = 0; t < nt; t++) { const float v = scan[t]; scan[t] = run; run += v; }
    }
    __syncthreads();
    const float before = scan[tid];
    if (mine > 0.f && target >= before && target < before + mine) {
        float run = before; int pick = -1;
        for (int i = beg; i < end; i++) {
            const float l = x[i];
            if (f2key(l) >= thr) { run += expf((l - mx) * invT); pick = i; if (target < run) break; }
        }
        chosen = pick;
    }
    __syncthreads();
    if (chosen < 0) {
        // the draw fell past the last partial sum through rounding: take the last kept token
        ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
        for (int i = tid; i < V; i += nt) if (f2key(x[i]) >= thr) { ValIdx c; c.v = (float)i; c.i = -i; b = better(b, c); }
        b = block_best(b, redvi);
        if (tid == 0) chosen = (b.i == 0x7fffffff) ? 0 : -b.i;
        __syncthreads();
    }
    if (tid == 0) a.out[row] = chosen;
}

// ---------------------------------------------------------------------------
// Sampling over a large vocabulary: the same four steps, but a row's elements are spread over many CTAs and
// every pass over the row is one launch of (chunks x rows) CTAs, so that a row of 256,000 logits is read at the
// speed of the whole GPU and not of one SM (the one-CTA kernel above takes 1.7 ms for such rows with a nucleus,
// most of a decode step).
//
// Masses are fixed-point: m_i = round(2^32 e^((l_i - max) / T)), summed in 64-bit integers.  Integer sums do not
// depend on their order, so histograms can be built with atomics and the draw still repeats bit for bit.
// The nucleus threshold is the key (the order-preserving bits) of the logit at which the mass of that key and all above
// reaches top_p x total.  One histogram of mass over 2,048 equal steps of (max - l) / T, which the elements of a row spread
// over (they fall into few digits of the key, and same-address atomics of a warp wait for one another), finds the step; its
// elements, a thousandth of a row, are listed, and a CTA of the row finds the key among them by a radix search.
//
//   sample_chunk_max  per chunk: repetition penalty on the chunk's ids, then (max, index) and min  [also the greedy choice];
//                     clears the row's histogram
//   sample_hist       per chunk: mass per step; the row's last CTA finds the threshold's  [rows with a nucleus only]
//   sample_chunk_mass per chunk: mass of the elements above the threshold's step; lists those in it (without a nucleus:
//                     mass of all).  A step of too many to list (CROWDED: equal or coarse logits, or a bulk narrower than a
//                     thousandth of the row's range beside one far above it) is cut into 512 parts: mass per part and chunk
//   sample_pick       per row: the threshold from the listed elements, their kept masses added to their chunks', target = u x
//                     kept mass; the chunk and then the element at which the running sum of kept masses, in index order,
//                     passes the target.  A crowded row's cluster of CTAs reads it once more, for the elements of the
//                     threshold's part; if those are too many to list too, they are one number, or 0 and -0, or (a few
//                     neighbouring numbers, thousands of each) the CTAs search the row by the key's digits
// 256,000 logits, top_p 0.95, in a graph: 36 / 44 / 97 us for 1 / 8 / 64 rows; six launches that read the row five times (three
// histograms over the key's digits) took 41 / 73 / 154.  A bulk of 0.002 beside an outlier of 8: 60 / 78 / 211 (39 / 72 / 148).
// ---------------------------------------------------------------------------
#define S_CHUNK 8192
#define S_BINS 2048
#define S_PARTS 512               // parts of a crowded step
#define S_LIST 4096               // elements of the threshold's step, or part, that are listed
typedef unsigned long long u64;

struct SampleState {              // per row with a nucleus, left by sample_hist
    u64 want;                     // what the elements of the threshold's step have to reach
    int edge;                     // the threshold's step; S_BINS: there are no masses, everything is kept
    int crowded;                  // it may hold more elements (of a mass) than are listed
};

struct SampleWide {
    SampleArgs a;
    int n_chunks;                 // chunks of a row
    int vec;                      // rows start on 16-byte boundaries
    float* pmax; float* pmin; int* pidx;   // [rows][n_chunks]
    u64* hist;                    // [rows][S_BINS]
    u64* inner;                   // [rows][n_chunks][S_PARTS] of a crowded row: masses within the threshold's step
    u64* cmass;                   // [rows][n_chunks] mass above the threshold's step
    SampleState* state;           // [rows]
    int* done;                    // [rows] CTAs of sample_hist that have added their masses
    int* count;                   // [rows] listed elements (of a crowded row: those that would be, if they are too many)
    int* list;                    // [rows][S_LIST] their places
};

__device__ __forceinline__ u64 fixed_mass(float l, float mx, float invT) {
    return __float2ull_rn(expf((l - mx) * invT) * 4294967296.0f);
}
// f(logit, its place) over a chunk by 256 threads, 16 bytes a load and all of a thread's loads on their way together
// (true: thread t's u-th element is number (u / 4 * 256 + t) * 4 + u % 4 of the chunk; else u * 256 + t)
template <typename F>
__device__ __forceinline__ bool each_of_chunk(const SampleWide& w, const float* x, int chunk, F&& f) {
    const int beg = chunk * S_CHUNK, n = min(w.a.vocab - beg, S_CHUNK);
    if (w.vec && n == S_CHUNK) {
        float4 v[S_CHUNK / 1024];
#pragma unroll
        for (int u = 0; u < S_CHUNK / 1024; u++) v[u] = *(const float4*)(x + beg + (u * 256 + threadIdx.x) * 4);
#pragma unroll
        for (int u = 0; u < S_CHUNK / 1024; u++) {
            const int i = beg + (u * 256 + threadIdx.x) * 4;
            f(v[u].x, i); f(v[u].y, i + 1); f(v[u].z, i + 2); f(v[u].w, i + 3);
        }
        return true;
    }
    for (int i = threadIdx.x; i < n; i += 256) f(x[beg + i], beg + i);
    return false;
}
// the row's maximum and minimum from the chunks' (every thread of the CTA gets them)
__device__ __forceinline__ void row_range(const SampleWide& w, int row, float* red /* 33 */, float& mx, float& mn) {
    mx = -INFINITY; mn = INFINITY;
    for (int c = threadIdx.x; c < w.n_chunks; c += blockDim.x) {
        mx = fmaxf(mx, w.pmax[(size_t)row * w.n_chunks + c]);
        mn = fminf(mn, w.pmin[(size_t)row * w.n_chunks + c]);
    }
    mx = block_max(mx, red);
    mn = -block_max(-mn, red);
}
__device__ __forceinline__ bool row_has_nucleus(const SampleArgs& a, int row) {
    return (a.temperature ? a.temperature[row] : 0.f) > 0.f && (a.top_p ? a.top_p[row] : 1.f) < 1.f;
}
// Steps of (max - l) / T: from 0 to the row's range, or to 23, from where on a mass is 0 (2^32 e^-23 < 1/2).  Rounding is
// monotonic, so a larger logit is never in a later step.
struct Steps { float mx, invT, scale; };
__device__ __forceinline__ Steps row_steps(float mx, float mn, float T) {
    Steps s;
    s.mx = mx; s.invT = 1.f / T;
    const float reach = fminf((mx - mn) * s.invT, 23.f);            // (a range that is not a number: 23)
    s.scale = reach > 0.f ? (float)S_BINS / reach : 0.f;
    return s;
}
// the step of a logit; -1: its mass is 0; -2: not a number (a logit that is none, or an infinite one beside an infinite maximum)
__device__ __forceinline__ int step_of(const Steps& s, float l) {
    const float x = (s.mx - l) * s.invT;
    if (x < 23.f) return min((int)(x * s.scale), S_BINS - 1);
    return x >= 23.f ? -1 : -2;
}
// the place of a logit within its step, in parts: the remainder of step_of's product, rounded as there (a fused
// multiply-add would not be, and two kernels have to agree)
__device__ __forceinline__ int part_of(const Steps& s, float l, int step) {
    const float t = __fmul_rn((s.mx - l) * s.invT, s.scale);
    return min((int)(__fsub_rn(t, (float)step) * (float)S_PARTS), S_PARTS - 1);
}

__global__ void __launch_bounds__(256) sample_chunk_max_kernel(SampleWide w) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ ValIdx red[32];
    __shared__ float redf[33];
    __shared__ int rec_s[1024];
    const int row = blockIdx.y, tid = threadIdx.x;
    const SampleArgs& a = w.a;
    float* x = a.logits + (size_t)row * a.row_stride;
    // this CTA's share of the row's histogram starts at zero
    for (int i = blockIdx.x * 256 + tid; i < S_BINS; i += gridDim.x * 256) w.hist[(size_t)row * S_BINS + i] = 0ull;
    if (blockIdx.x == 0 && tid == 0) w.count[row] = w.done[row] = 0;
    const int chunk = blockIdx.x;
    const int beg = chunk * S_CHUNK, end = min(a.vocab, beg + S_CHUNK);
    // repetition penalty, each distinct recent id once; a CTA sees to the ids of its own chunks
    const float pen = a.penalty ? a.penalty[row] : 1.f;
    if (pen > 1.f && a.recent) {
        const int* rec = a.recent + (size_t)row * a.n_recent;
        for (int j0 = 0; j0 < a.n_recent; j0 += 1024) {        // (lists longer than 1024 in pieces; each id is
            const int n = min(1024, a.n_recent - j0);           //  compared with the whole list before it)
            __syncthreads();
            for (int j = tid; j < n; j += 256) rec_s[j] = rec[j0 + j];
            __syncthreads();
            for (int j = tid; j < n; j += 256) {
                const int id = rec_s[j];
                if (id < beg || id >= end) continue;
                bool first = true;
                for (int k = 0; k < j && first; k++) first = rec_s[k] != id;
                for (int k = 0; k < j0 && first; k++) first = rec[k] != id;
                if (first) { const float l = x[id]; x[id] = l > 0.f ? l / pen : l * pen; }
            }
        }
        __syncthreads();
    }
    ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
    float mn = INFINITY;
    each_of_chunk(w, x, chunk, [&](float l, int i) { ValIdx c; c.v = l; c.i = i; b = better(b, c); mn = fminf(mn, l); });
    b = block_best(b, red);
    mn = -block_max(-mn, redf);
    if (tid == 0) {
        w.pmax[(size_t)row * w.n_chunks + chunk] = b.v; w.pidx[(size_t)row * w.n_chunks + chunk] = b.i;
        w.pmin[(size_t)row * w.n_chunks + chunk] = mn;
    }
}

// Where the running sum of a histogram's masses reaches `want`: the entry, and the mass before it.  `down`: from the last
// entry to the first.  All zero: entry 0 (the last one).  `g`: S_BINS sums in shared memory; called by the whole CTA.
struct Reached { u64 before, total; int entry; };
__device__ void find_entry(const u64* g, u64* part /* 256 */, Reached* out, bool down, u64 want, float top_p) {
    const int tid = threadIdx.x, lane = tid & 31;
    auto at = [&](int i) { return g[down ? S_BINS - 1 - i : i]; };
    if (tid < 256) {
        u64 s = 0ull;
#pragma unroll
        for (int k = 0; k < 8; k++) s += at(tid * 8 + k);
        part[tid] = s;
    }
    __syncthreads();
    if (tid < 32) {
        u64 mine = 0ull;
#pragma unroll
        for (int k = 0; k < 8; k++) mine += part[lane * 8 + k];
        u64 incl = mine;
        for (int o = 1; o < 32; o <<= 1) { const u64 v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        const u64 tot = __shfl_sync(0xffffffffu, incl, 31);
        if (top_p > 0.f || want == 0ull) {                          // (the first search: what the nucleus has to reach)
            const double d = (double)top_p * (double)tot;
            want = d < 1.0 ? 1ull : (u64)d;
            if (want > tot) want = tot;
        }
        const u64 before = incl - mine;
        const bool here = before < want && incl >= want;
        u64 acc = before;
        int i = 0;
        if (here) {
            int t = lane * 8;
            for (; t < lane * 8 + 7; t++) { if (acc + part[t] >= want) break; acc += part[t]; }
            i = t * 8;
            for (; i < t * 8 + 7; i++) { if (acc + at(i) >= want) break; acc += at(i); }
        }
        const unsigned who = __ballot_sync(0xffffffffu, here);
        const int src = who ? __ffs(who) - 1 : 0;                   // (exactly one lane, unless the masses are all zero)
        acc = __shfl_sync(0xffffffffu, acc, src);
        i = __shfl_sync(0xffffffffu, i, src);
        if (lane == 0) { out->before = acc; out->total = want; out->entry = down ? S_BINS - 1 - i : i; }
    }
    __syncthreads();
}

// A mass is at most 2^32.  Its low 16 bits and the rest are summed in two 32-bit histograms, whose atomics the shared
// memory has natively (a 64-bit one is a compare-and-swap loop); the elements of seven chunks cannot overflow either.
constexpr int S_MOST_CHUNKS = 7;
__device__ __forceinline__ void add_mass(unsigned* lo, unsigned* hi, int entry, u64 m) {
    atomicAdd(&lo[entry], (unsigned)(m & 0xffffu));
    atomicAdd(&hi[entry], (unsigned)(m >> 16));
}

// The same by a whole warp, an entry a lane (-1: none): an entry that all of them share is added to once (equal logits, or
// digits that a step's elements have in common: their additions would wait for one another).
__device__ __forceinline__ void add_mass_of_warp(unsigned* lo, unsigned* hi, int entry, u64 m) {
    const unsigned in = __ballot_sync(0xffffffffu, entry >= 0);
    if (in == 0u) return;
    const int first = __shfl_sync(0xffffffffu, entry, __ffs(in) - 1);
    if (__all_sync(0xffffffffu, entry < 0 || entry == first)) {
        const unsigned a = __reduce_add_sync(0xffffffffu, entry >= 0 ? (unsigned)(m & 0xffffu) : 0u);
        const unsigned b = __reduce_add_sync(0xffffffffu, entry >= 0 ? (unsigned)(m >> 16) : 0u);
        if ((threadIdx.x & 31) == 0) { atomicAdd(&lo[first], a); atomicAdd(&hi[first], b); }
    } else if (entry >= 0) add_mass(lo, hi, entry, m);
}

__global__ void __launch_bounds__(256) sample_hist_kernel(SampleWide w) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(8) unsigned lo_hi[2 * S_BINS];
    __shared__ u64 part[256];
    __shared__ Reached s_at;
    __shared__ float red[33];
    __shared__ bool last;
    unsigned* lo = lo_hi;
    unsigned* hi = lo_hi + S_BINS;
    const int row = blockIdx.y;
    if (!row_has_nucleus(w.a, row)) return;
    for (int i = threadIdx.x; i < S_BINS; i += 256) lo[i] = hi[i] = 0u;
    const float* x = w.a.logits + (size_t)row * w.a.row_stride;
    float mx, mn;
    row_range(w, row, red, mx, mn);                                 // (has the barriers that the zeros need)
    const Steps st = row_steps(mx, mn, w.a.temperature[row]);
    each_of_chunk(w, x, blockIdx.x, [&](float l, int) {
        const int e = step_of(st, l);
        if (e >= 0) add_mass(lo, hi, e, fixed_mass(l, st.mx, st.invT));
    });
    __syncthreads();
    u64* out = w.hist + (size_t)row * S_BINS;
    for (int i = threadIdx.x; i < S_BINS; i += 256) {
        const u64 m = (u64)lo[i] + ((u64)hi[i] << 16);
        if (m) atomicAdd(&out[i], m);
    }
    // the CTA that comes last finds the threshold's step
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&w.done[row], 1) == w.n_chunks - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    u64* g = (u64*)lo_hi;
    for (int i = threadIdx.x; i < S_BINS; i += 256) g[i] = __ldcg(&out[i]);
    __syncthreads();
    find_entry(g, part, &s_at, false, 0ull, w.a.top_p[row]);
    if (threadIdx.x == 0) {
        w.state[row].want = s_at.total - s_at.before;
        w.state[row].edge = s_at.total > 0ull ? s_at.entry : S_BINS;
        // no element of the step that has a mass has less than one at the end of the step after it
        const u64 least = st.scale > 0.f ? __float2ull_rn(expf(-(float)(s_at.entry + 2) / st.scale) * 4294967296.0f) : 1ull;
        w.state[row].crowded = g[s_at.entry] / (least > 0ull ? least : 1ull) > (u64)S_LIST;
    }
}

// (five CTAs an SM: 64 rows of 256,000 take 97 us in all; with the registers that the crowded rows' branch would take, four, 100)
__global__ void __launch_bounds__(256, 5) sample_chunk_mass_kernel(SampleWide w, int nucleus) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ u64 red8[8];
    __shared__ float red[33];
    __shared__ unsigned lo[S_PARTS], hi[S_PARTS];
    const int row = blockIdx.y, chunk = blockIdx.x, lane = threadIdx.x & 31;
    const float T = w.a.temperature ? w.a.temperature[row] : 0.f;
    if (!(T > 0.f)) return;
    const int edge = nucleus && row_has_nucleus(w.a, row) ? w.state[row].edge : S_BINS;
    const bool crowded = edge < S_BINS && w.state[row].crowded;
    if (crowded)
        for (int i = threadIdx.x; i < S_PARTS; i += 256) lo[i] = hi[i] = 0u;
    float mx, mn;
    row_range(w, row, red, mx, mn);                                 // (has the barriers that the zeros need)
    const Steps st = row_steps(mx, mn, T);
    const float* x = w.a.logits + (size_t)row * w.a.row_stride;
    u64 m = 0ull;
    if (edge == S_BINS) {                                           // everything is kept
        each_of_chunk(w, x, chunk, [&](float l, int) { m += fixed_mass(l, st.mx, st.invT); });
    } else if (crowded) {
        const bool whole = w.vec && (chunk + 1) * S_CHUNK <= w.a.vocab;       // every lane has every element
        each_of_chunk(w, x, chunk, [&](float l, int) {
            const int e = step_of(st, l);
            const u64 f = e >= 0 && e <= edge ? fixed_mass(l, st.mx, st.invT) : 0ull;
            int p = -1;
            if (f > 0ull) { if (e < edge) m += f; else p = part_of(st, l, edge); }
            if (whole) add_mass_of_warp(lo, hi, p, f);
            else if (p >= 0) add_mass(lo, hi, p, f);
        });
        __syncthreads();
        for (int i = threadIdx.x; i < S_PARTS; i += 256) w.inner[((size_t)row * w.n_chunks + chunk) * S_PARTS + i] = (u64)lo[i] + ((u64)hi[i] << 16);
    } else {
        unsigned hits = 0u;                                         // which of this thread's elements lie in the threshold's step (and have a mass)
        int k = 0;
        const bool vec = each_of_chunk(w, x, chunk, [&](float l, int) {
            const int e = step_of(st, l);
            if (e >= 0 && e <= edge) {
                const u64 f = fixed_mass(l, st.mx, st.invT);
                if (e < edge) m += f; else hits |= (unsigned)(f > 0ull) << k;
            }
            k++;
        });
        // their places go to the row's list, one atomic a warp
        int before = __popc(hits);
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, before, o); if (lane >= o) before += v; }
        int base = 0;
        if (lane == 31 && before > 0) base = atomicAdd(&w.count[row], before);
        base = __shfl_sync(0xffffffffu, base, 31) + before - __popc(hits);
        for (; hits; hits &= hits - 1, base++) {
            const int u = __ffs(hits) - 1;
            if (base < S_LIST) w.list[(size_t)row * S_LIST + base] = chunk * S_CHUNK + (vec ? ((u >> 2) * 256 + threadIdx.x) * 4 + (u & 3) : u * 256 + threadIdx.x);
        }
    }
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    if (lane == 0) red8[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        u64 t = 0ull;
        for (int k = 0; k < 8; k++) t += red8[k];
        w.cmass[(size_t)row * w.n_chunks + chunk] = t;
    }
}

// the digit of pass R of a key, and whether the key matches the digits found before it
__device__ __forceinline__ bool digit_of(int R, unsigned key, unsigned prefix, int& bin) {
    if (R == 0) { bin = key >> 21; return true; }
    if (R == 1) { bin = (key >> 10) & 2047; return (key >> 21) == prefix; }
    bin = key & 1023; return (key >> 10) == prefix;
}

// f(logit, whether it is one) for the elements lo .. hi - 1, whole warps at a time, eight loads of a thread on their way.
template <int THREADS, typename F>
__device__ __forceinline__ void each_of_range(const float* x, int lo, int hi, F&& f) {
    for (int i = lo; i < hi; i += 8 * THREADS) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) { const int k = i + u * THREADS + (int)threadIdx.x; v[u] = k < hi ? x[k] : 0.f; }
#pragma unroll
        for (int u = 0; u < 8; u++) if (i + u * THREADS < hi) f(v[u], i + u * THREADS + (int)threadIdx.x < hi);
    }
}

__global__ void __launch_bounds__(512, 1) sample_pick_kernel(SampleWide w, int nucleus) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int THREADS = 512, PER = S_CHUNK / THREADS;            // consecutive elements per thread: index order
    __shared__ u64 g[S_BINS];
    __shared__ u64 part[THREADS];
    __shared__ u64 cm[256];                                          // the chunks' kept masses
    __shared__ Reached s_at;
    __shared__ float red[33];
    __shared__ int s_chunk;
    __shared__ u64 s_base, s_target;
    const int row = blockIdx.y, tid = threadIdx.x, rank = blockIdx.x, ctas = gridDim.x;
    const SampleArgs& a = w.a;
    const float T = a.temperature ? a.temperature[row] : 0.f;
    const bool has_edge = nucleus && row_has_nucleus(a, row) && w.state[row].edge < S_BINS;
    const bool crowded = has_edge && w.state[row].crowded;
    if (rank > 0 && !crowded) return;                               // (a cluster for the crowded rows)
    if (!(T > 0.f)) {
        // greedy: the best of the chunk maxima, the smallest index on a tie
        if (tid == 0) {
            ValIdx b; b.v = -INFINITY; b.i = 0x7fffffff;
            for (int c = 0; c < w.n_chunks; c++) {
                ValIdx v; v.v = w.pmax[(size_t)row * w.n_chunks + c]; v.i = w.pidx[(size_t)row * w.n_chunks + c];
                b = better(b, v);
            }
            a.out[row] = (b.i == 0x7fffffff) ? 0 : b.i;
        }
        return;
    }
    for (int c = tid; c < w.n_chunks; c += THREADS) cm[c] = w.cmass[(size_t)row * w.n_chunks + c];
    const float* x = a.logits + (size_t)row * a.row_stride;
    float mx, mn;
    row_range(w, row, red, mx, mn);                                 // (has the barriers that cm needs, too)
    const Steps st = row_steps(mx, mn, T);
    const float invT = st.invT;
    unsigned thr = 0u;
    if (has_edge) {
        const int edge = w.state[row].edge;
        u64 want = w.state[row].want;
        unsigned* lo = (unsigned*)g;
        unsigned* hi = lo + S_BINS;
        auto clear = [&]() {
            __syncthreads();
            for (int i = tid; i < 2 * S_BINS; i += THREADS) lo[i] = 0u;
            __syncthreads();
        };
        auto collect = [&](u64* m) {                                // the two halves of the sums
            __syncthreads();
#pragma unroll
            for (int u = 0; u < S_BINS / THREADS; u++) m[u] += (u64)lo[tid + u * THREADS] + ((u64)hi[tid + u * THREADS] << 16);
            __syncthreads();
        };
        auto advance = [&](int R) {
            want -= s_at.before;
            thr = (R == 0) ? (unsigned)s_at.entry : (R == 1) ? ((thr << 11) | (unsigned)s_at.entry) : ((thr << 10) | (unsigned)s_at.entry);
        };
        int n = 0;
        if (!crowded) n = w.count[row];
        else {
            __shared__ u64 total[S_BINS];
            __shared__ u64 from_all[256];                           // first CTA: a number per chunk, from the CTA that has it
            __shared__ unsigned s_least, s_most;                    // first CTA: the keys of the threshold's part
            __shared__ int s_many;
            cg::cluster_group cluster = cg::this_cluster();
            const int per = (w.n_chunks + ctas - 1) / ctas, c0 = min(w.n_chunks, rank * per), c1 = min(w.n_chunks, c0 + per), lane = tid & 31;
            const u64* inner = w.inner + (size_t)row * w.n_chunks * S_PARTS;
            for (int i = tid; i < S_BINS; i += THREADS) {
                u64 sum = 0ull;
                if (i < S_PARTS) for (int c = 0; c < w.n_chunks; c++) sum += inner[(size_t)c * S_PARTS + i];
                total[i] = sum;
            }
            if (tid == 0) { s_least = 0xffffffffu; s_most = 0u; s_many = 0; }
            if (tid < c1 - c0) g[tid] = 0ull;
            __syncthreads();
            find_entry(total, part, &s_at, false, want, 0.f);
            want -= s_at.before;
            const int level = s_at.entry;
            if (rank == 0)                                          // what lies above the part is kept
                for (int c = tid >> 5; c < w.n_chunks; c += THREADS / 32) {
                    u64 add = 0ull;
                    for (int i = lane; i < level; i += 32) add += inner[(size_t)c * S_PARTS + i];
                    for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
                    if (lane == 0) cm[c] += add;
                }
            // the part's elements of this CTA's chunks: to the list, until there are too many; the mass of those that are +0
            const float from = (float)edge + (float)level / S_PARTS;          // (exact)
            const float to = edge == S_BINS - 1 && level == S_PARTS - 1 ? INFINITY : (float)edge + (float)(level + 1) / S_PARTS;
            unsigned least = 0xffffffffu, most = 0u;
            float v[PER], next[PER];
            auto fetch = [&](int c) {
#pragma unroll
                for (int u = 0; u < PER; u++) {
                    const int i = c * S_CHUNK + u * THREADS + tid;
                    next[u] = c < c1 && i < a.vocab ? x[i] : 0.f;
                }
            };
            fetch(c0);
            for (int c = c0; c < c1; c++) {
#pragma unroll
                for (int u = 0; u < PER; u++) v[u] = next[u];
                fetch(c + 1);
                u64 zeros = 0ull;
#pragma unroll
                for (int u = 0; u < PER; u++) {
                    const float d = (mx - v[u]) * invT, t = __fmul_rn(d, st.scale);
                    const int i = c * S_CHUNK + u * THREADS + tid;
                    u64 f = 0ull;
                    if (i < a.vocab && d < 23.f && t >= from && t < to) {
                        f = fixed_mass(v[u], mx, invT);
                        if (f) {
                            const unsigned key = f2key(v[u]);
                            least = min(least, key); most = max(most, key);
                            if (key == 0x80000000u) zeros += f;
                        }
                    }
                    const unsigned hit = __ballot_sync(0xffffffffu, f > 0ull);
                    if (hit == 0u) continue;
                    int at = 0;
                    if (lane == 0) at = *(volatile int*)&s_many ? S_LIST : atomicAdd(&w.count[row], __popc(hit));
                    at = __shfl_sync(0xffffffffu, at, 0) + __popc(hit & ((1u << lane) - 1u));
                    if (f && at < S_LIST) w.list[(size_t)row * S_LIST + at] = i;
                    if (at >= S_LIST) *(volatile int*)&s_many = 1;
                }
                if (__any_sync(0xffffffffu, zeros > 0ull)) {
                    for (int o = 16; o > 0; o >>= 1) zeros += __shfl_xor_sync(0xffffffffu, zeros, o);
                    if (lane == 0) atomicAdd(&g[c - c0], zeros);
                }
            }
            cluster.sync();                                         // (the first CTA's numbers are set up; this one's zeros are added)
            least = __reduce_min_sync(0xffffffffu, least); most = __reduce_max_sync(0xffffffffu, most);
            if (lane == 0) { atomicMin(cluster.map_shared_rank(&s_least, 0), least); atomicMax(cluster.map_shared_rank(&s_most, 0), most); }
            if (tid < c1 - c0) cluster.map_shared_rank(from_all, 0)[c0 + tid] = g[tid];
            __threadfence();
            cluster.sync();                                         // all of it is there
            n = __ldcg(&w.count[row]);
            if (n > S_LIST) {
                least = *cluster.map_shared_rank(&s_least, 0); most = *cluster.map_shared_rank(&s_most, 0);
                cluster.sync();
                if (least == most || (least == 0x7fffffffu && most == 0x80000000u)) {
                    if (rank > 0) return;
                    u64 upper = 0ull;                               // one number; or -0 and +0, the next higher key
                    if (least != most) for (int c = 0; c < w.n_chunks; c++) upper += from_all[c];
                    thr = least == most || upper < want ? least : most;
                    for (int c = tid; c < w.n_chunks; c += THREADS) cm[c] += thr == least ? inner[(size_t)c * S_PARTS + level] : from_all[c];
                    __syncthreads();
                } else {
                    for (int R = 0; R < 3; R++) {
                        u64 m[S_BINS / THREADS] = {};
                        for (int c = c0; c < c1; c += S_MOST_CHUNKS) {
                            clear();
                            each_of_range<THREADS>(x, c * S_CHUNK, min(a.vocab, min(c1, c + S_MOST_CHUNKS) * S_CHUNK), [&](float l, bool in) {
                                int bin = -1;
                                if (!in || step_of(st, l) != edge || part_of(st, l, edge) != level || !digit_of(R, f2key(l), thr, bin)) bin = -1;
                                add_mass_of_warp(lo, hi, bin, bin >= 0 ? fixed_mass(l, mx, invT) : 0ull);
                            });
                            collect(m);
                        }
#pragma unroll
                        for (int u = 0; u < S_BINS / THREADS; u++) g[tid + u * THREADS] = m[u];
                        cluster.sync();
                        for (int i = tid; i < S_BINS / ctas; i += THREADS) {      // the sums of a share of the entries, for every CTA
                            const int e = rank * (S_BINS / ctas) + i;
                            u64 sum = 0ull;
                            for (int k = 0; k < ctas; k++) sum += cluster.map_shared_rank(g, k)[e];
                            for (int k = 0; k < ctas; k++) cluster.map_shared_rank(total, k)[e] = sum;
                        }
                        cluster.sync();
                        find_entry(total, part, &s_at, true, want, 0.f);
                        advance(R);
                    }
                    for (int c = c0; c < c1; c++) {
                        u64 add = 0ull;
                        each_of_range<THREADS>(x, c * S_CHUNK, min(a.vocab, (c + 1) * S_CHUNK), [&](float l, bool in) {
                            if (in && step_of(st, l) == edge && part_of(st, l, edge) == level && f2key(l) >= thr) add += fixed_mass(l, mx, invT);
                        });
                        __syncthreads();
                        if (tid == 0) g[0] = 0ull;
                        __syncthreads();
                        for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
                        if (lane == 0 && add) atomicAdd(&g[0], add);
                        __syncthreads();
                        if (tid == 0) cluster.map_shared_rank(from_all, 0)[c] = g[0];
                    }
                    cluster.sync();
                    if (rank == 0) for (int c = tid; c < w.n_chunks; c += THREADS) cm[c] += from_all[c];
                    __syncthreads();
                }
            }
            if (rank > 0) return;
        }
        if (n <= S_LIST) {
            const int* list = w.list + (size_t)row * S_LIST;
            for (int R = 0; R < 3; R++) {
                u64 m[S_BINS / THREADS] = {};
                clear();
                for (int k = tid; k < (n + 31) / 32 * 32; k += THREADS) {         // (whole warps)
                    const float l = k < n ? x[__ldcg(&list[k])] : 0.f;
                    int bin;
                    if (k >= n || !digit_of(R, f2key(l), thr, bin)) bin = -1;
                    add_mass_of_warp(lo, hi, bin, bin >= 0 ? fixed_mass(l, mx, invT) : 0ull);
                }
                collect(m);
#pragma unroll
                for (int u = 0; u < S_BINS / THREADS; u++) g[tid + u * THREADS] = m[u];
                __syncthreads();
                find_entry(g, part, &s_at, true, want, 0.f);
                advance(R);
            }
            clear();
            for (int k = tid; k < (n + 31) / 32 * 32; k += THREADS) {
                const int i = k < n ? __ldcg(&list[k]) : 0;
                const bool kept = k < n && f2key(x[i]) >= thr;
                add_mass_of_warp(lo, hi, kept ? i / S_CHUNK : -1, kept ? fixed_mass(x[i], mx, invT) : 0ull);
            }
            __syncthreads();
            for (int c = tid; c < w.n_chunks; c += THREADS) cm[c] += (u64)lo[c] + ((u64)hi[c] << 16);
            __syncthreads();
        }
    }
    if (tid == 0) {
        u64 kept = 0ull;
        for (int c = 0; c < w.n_chunks; c++) kept += cm[c];
        const double tg = (double)a.draw[row] * (double)kept;
        u64 target = (u64)tg;
        if (target >= kept) target = kept - 1;                      // (kept >= 2^32: the row's maximum has mass 2^32)
        u64 base = 0ull;
        int c = 0;
        for (; c < w.n_chunks - 1; c++) { if (base + cm[c] > target) break; base += cm[c]; }
        s_chunk = c; s_base = base; s_target = target;
    }
    __syncthreads();
    const int beg = s_chunk * S_CHUNK + tid * PER, end = min(a.vocab, beg + PER);
    __align__(16) float v[PER];
#pragma unroll
    for (int k = 0; k < PER; k += 4) {
        if (w.vec && beg + k + 4 <= end) *(float4*)(v + k) = *(const float4*)(x + beg + k);
        else
            for (int e = k; e < k + 4; e++) v[e] = beg + e < end ? x[beg + e] : 0.f;
    }
    u64 mine = 0ull;
#pragma unroll
    for (int k = 0; k < PER; k++) if (beg + k < end && f2key(v[k]) >= thr) mine += fixed_mass(v[k], mx, invT);
    part[tid] = mine;
    __syncthreads();
    if (tid < 32) {
        // exclusive prefix over the threads' sums: a lane sums its 16, the lanes scan, each lane writes its 16 prefixes
        constexpr int LS = THREADS / 32;
        u64 loc[LS], sum = 0ull;
#pragma unroll
        for (int k = 0; k < LS; k++) { loc[k] = part[tid * LS + k]; sum += loc[k]; }
        u64 incl = sum;
        for (int o = 1; o < 32; o <<= 1) { const u64 u = __shfl_up_sync(0xffffffffu, incl, o); if (tid >= o) incl += u; }
        u64 run = s_base + incl - sum;
#pragma unroll
        for (int k = 0; k < LS; k++) { part[tid * LS + k] = run; run += loc[k]; }
    }
    __syncthreads();
    const u64 before = part[tid], target = s_target;
    if (mine > 0ull && target >= before && target < before + mine) {
        u64 run = before; int pick = beg;
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (beg + k < end && target >= run && f2key(v[k]) >= thr) { run += fixed_mass(v[k], mx, invT); pick = beg + k; }
        a.out[row] = pick;
    }
}

extern "C" long long tb_sample_wide_scratch_bytes(int rows, int vocab) {
    const long long chunks = (vocab + S_CHUNK - 1) / S_CHUNK;
    return (long long)rows * (chunks * (4 + 4 + 4 + 8) + S_BINS * 8LL + chunks * S_PARTS * 8LL + (long long)sizeof(SampleState) + (2 + S_LIST) * 4LL) + 256;
}

// `nucleus`: 0 if the caller knows that every row has top_p >= 1 (the threshold's launch is then not made).
extern "C" int tb_sample_wide(const SampleArgs* args, int rows, void* scratch, int nucleus, cudaStream_t stream) {
    if (rows <= 0) return 0;
    SampleWide w;
    w.a = *args;
    if (w.a.vocab <= 0) return tb_refuse("sample: vocab=%d", w.a.vocab);
    if (w.a.draw == nullptr) return tb_refuse("sample: the draws are missing");
    if (rows > 65535) return tb_refuse("sample: %d rows is more than one call takes", rows);
    if ((w.a.vocab + S_CHUNK - 1) / S_CHUNK > 256) return tb_refuse("sample: a vocabulary of %d is more than this kernel takes", w.a.vocab);
    if (scratch == nullptr || ((uintptr_t)scratch & 15)) return tb_refuse("sample: needs 16-byte aligned scratch");
    w.n_chunks = (w.a.vocab + S_CHUNK - 1) / S_CHUNK;
    w.vec = ((uintptr_t)w.a.logits & 15) == 0 && w.a.row_stride % 4 == 0;
    char* p = (char*)scratch;
    w.hist = (u64*)p; p += (size_t)rows * S_BINS * 8;
    w.inner = (u64*)p; p += (size_t)rows * w.n_chunks * S_PARTS * 8;
    w.cmass = (u64*)p; p += (size_t)rows * w.n_chunks * 8;
    w.state = (SampleState*)p; p += (size_t)rows * sizeof(SampleState);
    w.pmax = (float*)p; p += (size_t)rows * w.n_chunks * 4;
    w.pmin = (float*)p; p += (size_t)rows * w.n_chunks * 4;
    w.pidx = (int*)p; p += (size_t)rows * w.n_chunks * 4;
    w.done = (int*)p; p += (size_t)rows * 4;
    w.count = (int*)p; p += (size_t)rows * 4;
    w.list = (int*)p;
    const dim3 per_chunk(w.n_chunks, rows);
    tb_launch(sample_chunk_max_kernel, dim3(per_chunk), dim3(256), 0, stream, w);
    if (nucleus) tb_launch(sample_hist_kernel, dim3(per_chunk), dim3(256), 0, stream, w);
    tb_launch(sample_chunk_mass_kernel, dim3(per_chunk), dim3(256), 0, stream, w, nucleus);
    cudaLaunchConfig_t cfg = {};
    // CTAs of a row's cluster, for crowded rows (the others' all leave but one): as many as leave no row waiting
    cfg.gridDim = dim3(!nucleus ? 1 : rows <= 18 ? 8 : rows <= 36 ? 4 : rows <= 72 ? 2 : 1, rows); cfg.blockDim = dim3(512); cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cfg.gridDim.x; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, sample_pick_kernel, w, nucleus);
    return tb_launch_status();
}

extern "C" int tb_sample(const SampleArgs* args, int rows, cudaStream_t stream) {
    if (rows <= 0) return 0;
    SampleArgs a = *args;
    if (a.vocab <= 0) return tb_refuse("sample: vocab=%d", a.vocab);
    if (a.draw == nullptr) return tb_refuse("sample: the draws are missing");
    tb_launch(sample_kernel, dim3(rows), dim3(1024), 0, stream, a);
    return tb_launch_status();
}
