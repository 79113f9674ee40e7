// Plain matrix product on CUDA cores: C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]),
// float32 accumulation with plain FFMA (no tensor-core mode of any precision).
//
// It is the matrix product of the 32-bit path, the LM head of the bfloat16 path
// when many rows are wanted at an odd shape, and the plain kernel beside the
// tensor-core products.  Every output element is the sum over k = 0..K-1 in that
// order, so a row of C does not depend on M, on N or on where the row sits in the
// batch.  Any M, N, K >= 1 and any leading dimensions are taken.
//
// Reference analogue: F.linear on [out, in] weights (servelab/parallel/
// tp_model.py:48-53,67-68,115-119).
#include "common.cuh"

#define GS_BM 64
#define GS_BN 64
#define GS_BK 16

// ACT 1: tanh on every element of A as it is loaded (the second product of a bottleneck).
template <typename TA, typename TW, typename TC, int ACT = 0>
__global__ void __launch_bounds__(256) gemm_tn_simt_kernel(
    const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, TC* __restrict__ C,
    int ldc, const float* __restrict__ bias, int M, int N, int K, long long batch_a,
    long long batch_w, long long batch_c) {
    __shared__ __align__(16) float As[GS_BK][GS_BM + 4];
    pdl_wait();
    A += (size_t)blockIdx.z * batch_a;          // a batch of products: one per grid z
    W += (size_t)blockIdx.z * batch_w;
    C += (size_t)blockIdx.z * batch_c;
    __shared__ __align__(16) float Ws[GS_BK][GS_BN + 4];
    const int tid = threadIdx.x;
    const int ty = tid >> 4, tx = tid & 15;
    const int m0 = blockIdx.y * GS_BM, n0 = blockIdx.x * GS_BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += GS_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int idx = tid + i * 256;
            const int row = idx >> 4, kk = idx & 15;
            const int gm = m0 + row, gn = n0 + row, gk = k0 + kk;
            float av = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
            if (ACT == 1) av = tanhf(av);
            As[kk][row] = av;
            Ws[kk][row] = (gn < N && gk < K) ? to_float(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GS_BK; ++kk) {
            const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            C[(size_t)gm * ldc + gn] = from_float<TC>(acc[i][j] + (bias ? bias[gn] : 0.f));
        }
    }
}

template <typename TA, typename TW, typename TC, int ACT = 0>
static int launch_gemm(const TA* A, int lda, const TW* W, int ldw, TC* C, int ldc,
                       const float* bias, int M, int N, int K, cudaStream_t st, int batch = 1,
                       long long batch_a = 0, long long batch_w = 0, long long batch_c = 0) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    if (K <= 0 || lda < K || ldw < K || ldc < N) return SLB_ERR_BAD_ARG;
    const int gy = (M + GS_BM - 1) / GS_BM;
    if (gy > 65535 || batch > 65535) return SLB_ERR_TOO_LARGE;
    return slb_launch(gemm_tn_simt_kernel<TA, TW, TC, ACT>, dim3((N + GS_BN - 1) / GS_BN, gy, batch), dim3(256),
                      0, st, A, lda, W, ldw, C, ldc, bias, M, N, K, batch_a, batch_w, batch_c);
}

// ---- float32 operands in whole 16-byte pieces --------------------------------------------------
// The same sums in the same order (one FFMA per product, k = 0..K-1: results are bit for bit those of
// the kernel above), with the operands brought in by cp.async through a ring of G_STAGES tiles.  What
// bounds it is the FFMA rate (74 TFLOP/s): the kernel above waits for scattered 4-byte loads twice a
// k-tile.  It reaches 46 TFLOP/s at 1,024 x 32,000 x 896, bound by shared-memory reads, and 32 and 20 at
// 257 x 9,728 x 896 and 257 x 896 x 4,864, whose last wave of tiles is ragged.  A tile row keeps its k
// elements side by side (as in memory, so a piece is copied as it is) with 4 floats of padding, which
// makes the 16-byte reads of 8 neighbouring rows free of bank conflicts; a thread owns rows ty + i TY and columns tx + j TX, so a warp's reads of W
// are neighbouring rows and its stores neighbouring columns.
#define G_STAGES 4
#define G_PAD 4

__device__ __forceinline__ void cp_async16_or_zero(float* dst, const float* src, bool valid) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = valid ? 16 : 0;                 // (0: the 16 bytes are filled with zeros)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <int BM, int BN, int TM, int TN, int BK>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_tn_f32_kernel(
    const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
    int ldc, const float* __restrict__ bias, int M, int N, int K, long long batch_a, long long batch_w,
    long long batch_c) {
    constexpr int TY = BM / TM, TX = BN / TN, NT = TY * TX, LD = BK + G_PAD, PIECES = BK / 4;
    extern __shared__ __align__(16) float g_smem[];
    constexpr int STAGE = (BM + BN) * LD;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    A += (size_t)blockIdx.z * batch_a;
    W += (size_t)blockIdx.z * batch_w;
    C += (size_t)blockIdx.z * batch_c;
    const int ktiles = (K + BK - 1) / BK;
    pdl_wait();
    auto fetch = [&](int kt) {
        float* st = g_smem + (size_t)(kt % G_STAGES) * STAGE;
        const int k0 = kt * BK;
#pragma unroll
        for (int p = tid; p < (BM + BN) * PIECES; p += NT) {
            const int row = p / PIECES, k = k0 + (p % PIECES) * 4;
            const bool is_a = row < BM;
            const int g = is_a ? m0 + row : n0 + row - BM;
            const bool valid = k < K && g < (is_a ? M : N);
            const float* src = is_a ? A + (valid ? (size_t)g * lda + k : 0) : W + (valid ? (size_t)g * ldw + k : 0);
            cp_async16_or_zero(st + row * LD + (p % PIECES) * 4, src, valid);
        }
    };
#pragma unroll
    for (int s = 0; s < G_STAGES - 1; ++s) {
        if (s < ktiles) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int kt = 0; kt < ktiles; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(G_STAGES - 2) : "memory");
        __syncthreads();                              // tile kt is there; tile kt - 1 has been read by all
        if (kt + G_STAGES - 1 < ktiles) fetch(kt + G_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = g_smem + (size_t)(kt % G_STAGES) * STAGE + ty * LD;
        const float* ws = g_smem + (size_t)(kt % G_STAGES) * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int q = 0; q < PIECES; ++q) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * TY * LD + q * 4);
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * TX * LD + q * 4);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + i * TY;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + j * TX;
            if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j] + (bias ? bias[gn] : 0.f);
        }
    }
}

struct F32Args {
    const float* A; int lda; const float* W; int ldw; float* C; int ldc; const float* bias;
    int M, N, K, batch; long long batch_a, batch_w, batch_c;
};

template <int BM, int BN, int TM, int TN, int BK>
static int launch_f32_tile(const F32Args& g, cudaStream_t st) {
    constexpr size_t smem = (size_t)G_STAGES * (BM + BN) * (BK + G_PAD) * sizeof(float);
    static unsigned long long configured = 0;
    auto kernel = gemm_tn_f32_kernel<BM, BN, TM, TN, BK>;
    const int err = slb_configure(&configured, kernel, smem);
    if (err) return err;
    return slb_launch_after(kernel, dim3((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, g.batch),
                            dim3((BM / TM) * (BN / TN)), smem, st, g.A, g.lda, g.W, g.ldw, g.C, g.ldc, g.bias, g.M, g.N,
                            g.K, g.batch_a, g.batch_w, g.batch_c);
}

// Which tile: the products are sums in order, so K is not split, and the tiles differ in how many
// blocks they make and how often a thread reads shared memory per FFMA.  Measured us at K = 896 of the
// first tile on an SM and of every further one (several are resident): 62 + 45 (64 x 128), 39.5 + 26
// (32 x 128), 23 + 13.5 (32 x 64), 19 + 10.5 (16 x 64); the tile that ends first is taken.  257 rows,
// the plain kernel against this one: [9728 x 896] 201 -> 142 us, [896 x 4864] 326 -> 112; one row: 79
// -> 28, 320 -> 87.  (128 x 128 with 256 threads: 103 + 104, never the first to end.)
static int launch_f32(const F32Args& g, cudaStream_t st) {
    struct Tile { int bm, bn; float first, next; };
    static const Tile tiles[] = {{64, 128, 62.f, 45.f}, {32, 128, 39.5f, 26.f}, {32, 64, 23.f, 13.5f}, {16, 64, 19.f, 10.5f}};
    const int sms = slb_num_sms();
    int best = 0;
    double least = 0.0;
    for (int i = 0; i < 4; ++i) {
        const long long n = (long long)((g.M + tiles[i].bm - 1) / tiles[i].bm) *
                            ((g.N + tiles[i].bn - 1) / tiles[i].bn) * g.batch;
        const double cost = tiles[i].first + (double)((n + sms - 1) / sms - 1) * tiles[i].next;
        if (i == 0 || cost < least) { least = cost; best = i; }
    }
    switch (best) {
        case 0: return launch_f32_tile<64, 128, 8, 8, 16>(g, st);
        case 1: return launch_f32_tile<32, 128, 4, 8, 16>(g, st);
        case 2: return launch_f32_tile<32, 64, 4, 4, 32>(g, st);
        default: return launch_f32_tile<16, 64, 2, 4, 32>(g, st);
    }
}

// The operands as cp.async wants them: rows, batches and addresses in whole 16-byte pieces.
static bool f32_pieces(const float* A, int lda, const float* W, int ldw, int M, int K, long long batch_a,
                       long long batch_w) {
    return ((lda | ldw | K) & 3) == 0 && ((batch_a | batch_w) & 3) == 0 &&
           (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && (M + 15) / 16 <= 65535;
}

extern "C" {
int slb_gemm_simt_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                      const float* bias, int M, int N, int K, cudaStream_t st) {
    if (M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N && f32_pieces(A, lda, W, ldw, M, K, 0, 0))
        return launch_f32(F32Args{A, lda, W, ldw, C, ldc, bias, M, N, K, 1, 0, 0, 0}, st);
    return launch_gemm<float, float, float>(A, lda, W, ldw, C, ldc, bias, M, N, K, st);
}
int slb_gemm_simt_bf16(const bf16* A, int lda, const bf16* W, int ldw, bf16* C, int ldc,
                       const float* bias, int M, int N, int K, cudaStream_t st) {
    return launch_gemm<bf16, bf16, bf16>(A, lda, W, ldw, C, ldc, bias, M, N, K, st);
}
// `batch` products in one launch: product b reads A + b * batch_a, W + b * batch_w and writes
// C + b * batch_c (element strides; the per-head products of a latent attention).
int slb_gemm_simt_batched_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M,
                              int N, int K, int batch, long long batch_a, long long batch_w,
                              long long batch_c, cudaStream_t st) {
    if (M > 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535 && lda >= K && ldw >= K && ldc >= N &&
        f32_pieces(A, lda, W, ldw, M, K, batch_a, batch_w))
        return launch_f32(F32Args{A, lda, W, ldw, C, ldc, nullptr, M, N, K, batch, batch_a, batch_w, batch_c}, st);
    return launch_gemm<float, float, float>(A, lda, W, ldw, C, ldc, nullptr, M, N, K, st, batch, batch_a,
                                            batch_w, batch_c);
}
int slb_gemm_simt_batched_bf16(const bf16* A, int lda, const bf16* W, int ldw, bf16* C, int ldc, int M,
                               int N, int K, int batch, long long batch_a, long long batch_w,
                               long long batch_c, cudaStream_t st) {
    return launch_gemm<bf16, bf16, bf16>(A, lda, W, ldw, C, ldc, nullptr, M, N, K, st, batch, batch_a,
                                         batch_w, batch_c);
}
int slb_gemm_simt_batched_bf16_f32out(const bf16* A, int lda, const bf16* W, int ldw, float* C, int ldc, int M,
                                      int N, int K, int batch, long long batch_a, long long batch_w,
                                      long long batch_c, cudaStream_t st) {
    return launch_gemm<bf16, bf16, float>(A, lda, W, ldw, C, ldc, nullptr, M, N, K, st, batch, batch_a, batch_w,
                                          batch_c);
}
// C = tanh(A) . W^T (+ bias), float32 results
int slb_gemm_simt_tanh_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                           const float* bias, int M, int N, int K, cudaStream_t st) {
    return launch_gemm<float, float, float, 1>(A, lda, W, ldw, C, ldc, bias, M, N, K, st);
}
int slb_gemm_simt_bf16_f32out(const bf16* A, int lda, const bf16* W, int ldw, float* C, int ldc,
                              const float* bias, int M, int N, int K, cudaStream_t st) {
    return launch_gemm<bf16, bf16, float>(A, lda, W, ldw, C, ldc, bias, M, N, K, st);
}
}
