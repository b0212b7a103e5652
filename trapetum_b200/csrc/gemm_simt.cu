// C[M,N] = A[M,K] * W[N,K]^T on the 32-bit FMA pipe.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no
// reduced-precision matrix mode) and the any-size fallback of the bfloat16 path
// (sizes the tensor-core kernel refuses: K not a multiple of 8 elements, or
// 32-bit weights).  Weights are [out, in] as the checkpoint stores them, so a
// row of W is one output column's dot-product vector, like the reference's
// dense GEMV (runtime/cuda/codebook_gemv.cu:482-517).  Products and sums are
// 32-bit; each C element adds its K terms in the same order whatever M and N are
// (k-tiles of 16 in ascending order, each tile summed on its own first; where the
// segments below apply, segment by segment), so a token's result does not depend
// on what else is in the batch.
// Optional epilogue: tanh soft cap (the final logit cap, runtime/src/lib.rs:4559-4560).
//
//   gemm_simt_rows_kernel   32-bit operands, few rows of A: the product is a read of W
//   gemm_simt_tile_kernel   32-bit operands, many rows: bound by the FMA pipe and the register file's ports
//   gemm_simt_kernel        any operand types, sizes and alignments: the generic form
// The first two cut a long K into as many segments as a cluster has CTAs (a number that depends on K alone), each segment
// summed like a product of its own and the segments' sums added in ascending order: the same bits from both kernels.
#include <cooperative_groups.h>
#include "common.cuh"

namespace cg = cooperative_groups;

TB_EXPORT_ERROR()

#define BM 64
#define BN 64
#define BK 16

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C,
                 int M, int N, int K, long long lda, long long ldw, long long ldc, float cap, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tr = tid / 16, tc = tid % 16;          // 16x16 threads, 4x4 outputs each
    const int lr = tid / 4, lk = (tid % 4) * 4;      // loader: row lr, k offset lk..lk+3
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + lk + j;
            const int m = m0 + lr, n = n0 + lr;
            As[lk + j][lr] = (m < M && k < K) ? to_f<TA>(A[(size_t)m * lda + k]) : 0.f;
            Ws[lk + j][lr] = (n < N && k < K) ? to_f<TW>(W[(size_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
        // blocked summation: the 16 products of a k-tile are added up on their own and the tile's sum is then
        // added to the running total, so that rounding errors grow with K/16 + 16 terms instead of K
        float part[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) part[i][j] = 0.f;
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[k][tr * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = Ws[k][tc * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) part[i][j] = fmaf(a[i], w[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] += part[i][j];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + tr * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tc * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (cap > 0.f) v = softcap_f(v, cap);
            C[(size_t)m * ldc + n] = from_f<TC>(v * scale);
        }
    }
}

// ---------------------------------------------------------------------------
// 32-bit operands whose rows are whole 16-byte pieces
// ---------------------------------------------------------------------------
__device__ __forceinline__ void copy16(float* dst, const float* src, bool valid) {
    const int n = valid ? 16 : 0;                    // 0 source bytes: the 16 destination bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float lane4(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// Pieces of about 1,024 to 2,048 k: a token's row sums in the same order whatever the number of rows, and a matrix of few
// columns (the 2B shape's down product: 2,304) still fills the GPU.
static int simt_segments(int K) { return K >= 8192 ? 8 : K >= 4096 ? 4 : K >= 2048 ? 2 : 1; }

struct SimtProduct {
    const float* A; const float* W; void* C;
    int M, N, K, seg;                                // seg: k of a segment, a multiple of the tiles kernel's stage
    long long lda, ldw, ldc;
    float cap, scale;
};

template <typename TC>
__device__ __forceinline__ void simt_store(const SimtProduct& p, int m, int n, float v) {
    if (m >= p.M || n >= p.N) return;
    if (p.cap > 0.f) v = softcap_f(v, p.cap);
    ((TC*)p.C)[(size_t)m * p.ldc + n] = from_f<TC>(v * p.scale);
}

// 64x64 outputs a CTA, 8x4 a thread (rows mi + 8 i, columns ni + 16 j), operands as they lie in memory in three stages of
// 32 k, a row padded to 36 words (eight neighbouring rows' 16-byte words touch all banks once).  The next four k's words are
// read while these four's products run.  8x8 a thread, transposed operands and packed pairs of products all ended at the
// same 42 to 44 TFLOP/s (2,048 rows; the one-stage kernel above: 25), 32x64 outputs 8 % lower.  In us, this kernel and the
// one above: 300 rows x 18,432 x 2,304: 664, 1,097; 300 x 2,304 x 9,216: 381, 1,273; 2,048 x 18,432 x 2,304: 4,097, 6,797.
constexpr int TK = 32, TPITCH = TK + 4, TSTAGES = 3, TTHREADS = 128, TM = 8, TN = 4, TBM = 8 * TM, TBN = 16 * TN;
constexpr int TSTAGE = (TBM + TBN) * TPITCH;

template <typename TC>
__global__ void __launch_bounds__(TTHREADS, 3) gemm_simt_tile_kernel(SimtProduct p) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sh[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int mi = (warp >> 1) * 4 + ((lane >> 4) << 1) + (lane & 1), ni = (warp & 1) * 8 + ((lane >> 1) & 7);
    const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
    const int k_lo = blockIdx.z * p.seg, k_hi = min(p.K, k_lo + p.seg);
    auto load = [&](int st, int k0) {
        float* dst = sh + st * TSTAGE;
#pragma unroll
        for (int c = 0; c < (TBM + TBN) * (TK / 4) / TTHREADS; c++) {
            const int i = tid + c * TTHREADS, r = i / (TK / 4), k = k0 + (i % (TK / 4)) * 4;
            const bool is_a = r < TBM;
            const int row = is_a ? m0 + r : n0 + r - TBM;
            const bool ok = k < k_hi && row < (is_a ? p.M : p.N);
            const float* src = is_a ? p.A + (ok ? (size_t)row * p.lda + k : 0) : p.W + (ok ? (size_t)row * p.ldw + k : 0);
            copy16(dst + r * TPITCH + (i % (TK / 4)) * 4, src, ok);
        }
        copies_commit();
    };
    float acc[TM][TN], part[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
    pdl_wait();
    const int rounds = k_hi > k_lo ? (k_hi - k_lo + TK - 1) / TK : 0;
#pragma unroll
    for (int s = 0; s < TSTAGES - 1; s++) { if (s < rounds) load(s, k_lo + s * TK); else copies_commit(); }
    for (int rd = 0; rd < rounds; rd++) {
        copies_wait<TSTAGES - 2>();
        __syncthreads();                             // this stage is there; the one that is refilled next has been read
        const int ahead = rd + TSTAGES - 1;
        if (ahead < rounds) load(ahead % TSTAGES, k_lo + ahead * TK); else copies_commit();
        const float* sA = sh + (rd % TSTAGES) * TSTAGE + mi * TPITCH;
        const float* sW = sh + (rd % TSTAGES) * TSTAGE + (TBM + ni) * TPITCH;
        float4 w[2][TN], a[2];
#pragma unroll
        for (int j = 0; j < TN; j++) w[0][j] = *(const float4*)(sW + j * 16 * TPITCH);
        a[0] = *(const float4*)sA;
#pragma unroll
        for (int q = 0; q < TK / 4; q++) {
            if (q % (BK / 4) == 0) {
#pragma unroll
                for (int i = 0; i < TM; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) part[i][j] = 0.f;
            }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                if (i + 1 < TM) a[(i + 1) & 1] = *(const float4*)(sA + (i + 1) * 8 * TPITCH + q * 4);
                else if (q + 1 < TK / 4) a[(i + 1) & 1] = *(const float4*)(sA + q * 4 + 4);
                if (q + 1 < TK / 4 && i < TN) w[(q + 1) & 1][i] = *(const float4*)(sW + i * 16 * TPITCH + q * 4 + 4);
                const float4 av = a[i & 1];
#pragma unroll
                for (int k = 0; k < 4; k++)
#pragma unroll
                    for (int j = 0; j < TN; j++) part[i][j] = fmaf(lane4(av, k), lane4(w[q & 1][j], k), part[i][j]);
            }
            if (q % (BK / 4) == BK / 4 - 1) {
#pragma unroll
                for (int i = 0; i < TM; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) acc[i][j] += part[i][j];
            }
        }
    }
    const int S = gridDim.z;
    if (S == 1) {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) simt_store<TC>(p, m0 + mi + 8 * i, n0 + ni + 16 * j, acc[i][j]);
        return;
    }
    // the segments meet: every CTA of the cluster leaves its sums in its own shared memory and adds a slice of the rows
    cg::cluster_group cluster = cg::this_cluster();
    copies_wait<0>();
    __syncthreads();                                 // the last stage has been read, no copy is on its way
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) sh[(mi + 8 * i) * TBN + ni + 16 * j] = acc[i][j];
    cluster.sync();
    const int per = TBM / S, r0 = (int)cluster.block_rank() * per;
    for (int i = tid; i < per * TBN; i += TTHREADS) {
        float v = 0.f;
        for (int s = 0; s < S; s++) v += cluster.map_shared_rank(sh, s)[r0 * TBN + i];
        simt_store<TC>(p, m0 + r0 + i / TBN, n0 + i % TBN, v);
    }
    cluster.sync();                                  // nobody leaves while its sums are being read
}

// Few rows: 16 rows of W and up to 8 of A a CTA.  Thread (g, kt, mh) sums k-tile kt of a stage's 256 k for rows g, g + 4,
// g + 8 and g + 12 of W (so that a word of A serves four) and every other row of A; the tiles' sums meet in shared memory,
// where a thread per output adds them in order.  A cluster's CTAs take a segment each, or one CTA all of them in turn.
// Of 18,432 x 2,304 numbers at 1 / 8 rows: 43.7 / 67.9 us (3.9 / 2.5 TB/s); the generic kernel 317 / 341.
constexpr int RBM = 8, RBN = 16, RK = 256, RPITCH = RK + 4, RSTAGES = 3, RTHREADS = RBM * RBN, RSTAGE = (RBM + RBN) * RPITCH;
constexpr int RTILES = RK / BK, RSP = RBM * RBN + 4;  // k-tiles a stage; pitch of a k-tile's sums
static_assert(RTHREADS == 2 * 4 * RTILES, "a thread per (g, kt, mh), and one per output");

template <typename TC>
__global__ void __launch_bounds__(RTHREADS) gemm_simt_rows_kernel(SimtProduct p, int m_blocks, int segments) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sh[];      // [RSTAGES][W: 16 | A: 8 rows][RPITCH], then [RTILES][RSP] sums
    float* sums = sh + RSTAGES * RSTAGE;
    const int tid = threadIdx.x, g = tid & 3, kt = (tid >> 2) % RTILES, mh = tid / (4 * RTILES);
    const int m0 = (int)(blockIdx.x % m_blocks) * RBM, n0 = (int)(blockIdx.x / m_blocks) * RBN;   // neighbours share rows of W
    const int rows = min(RBM, p.M - m0), per_seg = (p.seg + RK - 1) / RK;
    const int seg0 = blockIdx.z, n_seg = gridDim.z > 1 ? 1 : segments, rounds = n_seg * per_seg;
    auto load = [&](int rd) {                        // half of the threads a row's stage, a copy each
        const int seg = seg0 + rd / per_seg, k = seg * p.seg + rd % per_seg * RK + tid % (RK / 4) * 4;
        const bool in = k < min(p.K, (seg + 1) * p.seg);
        float* dst = sh + rd % RSTAGES * RSTAGE + tid % (RK / 4) * 4;
        const int r0 = tid / (RK / 4);
#pragma unroll
        for (int r = 0; r < RBN; r += 2) {
            const bool ok = in && n0 + r0 + r < p.N;
            copy16(dst + (r0 + r) * RPITCH, p.W + (ok ? (size_t)(n0 + r0 + r) * p.ldw + k : 0), ok);
        }
        for (int r = r0; r < rows; r += 2) copy16(dst + (RBN + r) * RPITCH, p.A + (in ? (size_t)(m0 + r) * p.lda + k : 0), in);
        copies_commit();
    };
    float acc = 0.f, total = 0.f;
    pdl_wait();
#pragma unroll
    for (int s = 0; s < RSTAGES - 1; s++) { if (s < rounds) load(s); else copies_commit(); }
    for (int rd = 0; rd < rounds; rd++) {
        copies_wait<RSTAGES - 2>();
        __syncthreads();                             // this stage is there; the one before and its sums have been read
        if (rd + RSTAGES - 1 < rounds) load(rd + RSTAGES - 1); else copies_commit();
        const float* sW = sh + rd % RSTAGES * RSTAGE + g * RPITCH + kt * BK;
        const float* sA = sh + rd % RSTAGES * RSTAGE + RBN * RPITCH + kt * BK;
        float4 w[RBN / 4][BK / 4];
#pragma unroll
        for (int j = 0; j < RBN / 4; j++)
#pragma unroll
            for (int q = 0; q < BK / 4; q++) w[j][q] = *(const float4*)(sW + j * 4 * RPITCH + q * 4);
#pragma unroll 2
        for (int m = mh; m < rows; m += 2) {
            float part[RBN / 4];
#pragma unroll
            for (int j = 0; j < RBN / 4; j++) part[j] = 0.f;
#pragma unroll
            for (int q = 0; q < BK / 4; q++) {
                const float4 a = *(const float4*)(sA + m * RPITCH + q * 4);
#pragma unroll
                for (int k = 0; k < 4; k++)
#pragma unroll
                    for (int j = 0; j < RBN / 4; j++) part[j] = fmaf(lane4(a, k), lane4(w[j][q], k), part[j]);
            }
#pragma unroll
            for (int j = 0; j < RBN / 4; j++) sums[kt * RSP + m * RBN + g + 4 * j] = part[j];
        }
        __syncthreads();
        const int k0 = (seg0 + rd / per_seg) * p.seg + rd % per_seg * RK;
        const int k_end = min(p.K, (seg0 + rd / per_seg + 1) * p.seg);
        const int tiles = max(0, min(RTILES, (k_end - k0 + BK - 1) / BK));
        if (tid / RBN < rows) {                      // output (m, n) = (tid / 16, tid % 16)
            if (tiles == RTILES) {
#pragma unroll
                for (int t = 0; t < RTILES; t++) acc += sums[t * RSP + tid];
            } else {
                for (int t = 0; t < tiles; t++) acc += sums[t * RSP + tid];
            }
        }
        if ((rd + 1) % per_seg == 0) { total += acc; acc = 0.f; }
    }
    const int S = gridDim.z;
    if (S > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        __syncthreads();                             // the last sums have been read
        sums[tid] = total;
        cluster.sync();
        if (cluster.block_rank() == 0) {
            total = 0.f;
            for (int s = 0; s < S; s++) total += cluster.map_shared_rank(sums, s)[tid];
        }
        cluster.sync();                              // nobody leaves while its sums are being read
        if (cluster.block_rank() != 0) return;
    }
    if (tid / RBN < rows) simt_store<TC>(p, m0 + tid / RBN, n0 + tid % RBN, total);
}

// The launch of a kernel above: clusters of the CTAs along z.
template <typename... KArgs, typename... Args>
static int launch_segments(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = grid.z;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
    return tb_launch_status();
}

// Up to this many rows the rows kernel is faster: 8 / 16 / 24 rows of 18,432 x 2,304: 68 / 135 / 199 us, the tiles kernel
// 141 us at each; of 2,304 x 9,216: 50 / 95 / 134 and 101.
constexpr int ROWS_UP_TO = 16;

template <typename TC>
static int launch_f32(SimtProduct p, cudaStream_t stream) {
    const int S = simt_segments(p.K);
    p.seg = ((p.K + S - 1) / S + TK - 1) / TK * TK;
    if (p.M <= ROWS_UP_TO) {
        const int mb = (p.M + RBM - 1) / RBM;
        const unsigned tiles = (unsigned)mb * (((unsigned)p.N + RBN - 1) / RBN);
        // two CTAs an SM: with four rounds of them and more, a CTA per segment would only pay its start-up more often
        // (18,432 x 2,304 at one row: 43.7 us, with a CTA per segment 50.5)
        return launch_segments(gemm_simt_rows_kernel<TC>, dim3(tiles, 1, tiles >= 1024 ? 1 : S), RTHREADS,
                               (size_t)(RSTAGES * RSTAGE + RTILES * RSP) * sizeof(float), stream, p, mb, S);
    }
    return launch_segments(gemm_simt_tile_kernel<TC>, dim3((p.N + TBN - 1) / TBN, (p.M + TBM - 1) / TBM, S), TTHREADS,
                           (size_t)TSTAGES * TSTAGE * sizeof(float), stream, p);
}

// out_scale: the output times this number (1: a plain product), applied after the cap.
extern "C" int tb_gemm_simt_ex(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                               int M, int N, int K, long long lda, long long ldw, long long ldc,
                               float softcap, float out_scale, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return tb_refuse("gemm: K=%d", K);
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return tb_refuse("gemm: M=%d is too many rows for one call", M);
    if (a_dtype == TB_F32 && w_dtype == TB_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 &&
        ((uintptr_t)W & 15) == 0 && (c_dtype == TB_F32 || c_dtype == TB_BF16)) {
        const SimtProduct p = {(const float*)A, (const float*)W, C, M, N, K, 0, lda, ldw, ldc, softcap, out_scale};
        return c_dtype == TB_F32 ? launch_f32<float>(p, stream) : launch_f32<bf16>(p, stream);
    }
    const int key = (a_dtype << 2) | (w_dtype << 1) | c_dtype;
#define LAUNCH(TA, TW, TC) tb_launch(gemm_simt_kernel<TA, TW, TC>, dim3(grid), dim3(256), 0, stream,  \
        (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc, softcap, out_scale)
    switch (key) {
    case 0: LAUNCH(float, float, float); break;
    case 1: LAUNCH(float, float, bf16); break;
    case 2: LAUNCH(float, bf16, float); break;
    case 3: LAUNCH(float, bf16, bf16); break;
    case 4: LAUNCH(bf16, float, float); break;
    case 5: LAUNCH(bf16, float, bf16); break;
    case 6: LAUNCH(bf16, bf16, float); break;
    case 7: LAUNCH(bf16, bf16, bf16); break;
    default: return tb_refuse("gemm: unknown dtype codes %d %d %d", a_dtype, w_dtype, c_dtype);
    }
#undef LAUNCH
    return tb_launch_status();
}

extern "C" int tb_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                            int M, int N, int K, long long lda, long long ldw, long long ldc,
                            float softcap, cudaStream_t stream) {
    return tb_gemm_simt_ex(A, a_dtype, W, w_dtype, C, c_dtype, M, N, K, lda, ldw, ldc, softcap, 1.0f, stream);
}
