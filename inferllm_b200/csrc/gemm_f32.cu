// True float32 matrix product C[M, N] = A[M, K] . W[N, K]^T with float32 FMA accumulation:
// the contraction of the float32 mode.  No tensor cores, no TF32, no split of K: every
// element of C is one thread's sum over k in ascending order, so a row of C is bit-identical
// whatever M is and wherever the row lies.  That makes the float32 mode show faults of the
// cache or the batching that rounding would otherwise excuse.
// The reference calls cublasSgemm here (src/kern/gpu/kernel_gpu.cu:420-435), formula
// src/kern/naive/naive.cpp:363-379 (weight row-major [out, in], no bias).
//
// Tile kernel: a BM x BN tile of C per block, TM x TN outputs a thread, slices of 16 values of k in two shared-memory
// buffers (k-major, so that the columns of a pair lie side by side), the next slice on its way to registers while
// this one is used, one barrier per slice.  What bounds it is the float32 FMA rate: two neighbouring columns share
// one packed fma.rn.f32x2 (each half rounded like a scalar fused multiply-add, so the chain per output and its bits
// stay what they were), and the large tile's 8 x 16 outputs a thread read 96 bytes of shared memory per 64 packed
// instructions, the lanes of a warp (4 along the rows by 8 along the columns) each 16-byte read in one pass.
#include "tc_common.cuh"

#define GF_BK 16

__device__ __forceinline__ unsigned long long gf_pair(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long gf_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// 16-byte pieces of a ROWS x 16 slice of a row-major matrix: a thread's share of them on their way through registers.
template <int ROWS, int THREADS>
struct GfSlice {
    static constexpr int N = ROWS * (GF_BK / 4) / THREADS;
    static_assert(N >= 1 && ROWS * (GF_BK / 4) % THREADS == 0, "a slice is whole pieces per thread");
    float4 v[N];
    // rows beyond the matrix and values beyond K arrive as zeros, which change no sum
    __device__ __forceinline__ void load(const float* __restrict__ src, int row0, int rows, int ld, int k0, int K, bool vec) {
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int piece = threadIdx.x + i * THREADS, row = row0 + (piece >> 2), k = k0 + (piece & 3) * 4;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < rows && k < K) {
                const float* p = src + (size_t)row * ld + k;
                if (vec) {                       // K % 4 == 0: a piece that begins inside ends inside
                    v[i] = *reinterpret_cast<const float4*>(p);
                } else {
                    v[i].x = p[0];
                    if (k + 1 < K) v[i].y = p[1];
                    if (k + 2 < K) v[i].z = p[2];
                    if (k + 3 < K) v[i].w = p[3];
                }
            }
        }
    }
    __device__ __forceinline__ void store(float (*dst)[ROWS + 4]) const {
#pragma unroll
        for (int i = 0; i < N; i++) {
            const int piece = threadIdx.x + i * THREADS, row = piece >> 2, k = (piece & 3) * 4;
            dst[k][row] = v[i].x;
            dst[k + 1][row] = v[i].y;
            dst[k + 2][row] = v[i].z;
            dst[k + 3][row] = v[i].w;
        }
    }
};

// A warp is 4 threads along the rows by 8 along the columns; a thread's rows and columns are pieces of four, 16 rows and 32
// columns apart.  TM: 4 or 8, TN: 4, 8 or 16.
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN >= 64 ? 2 : 4)
gemm_f32_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                   int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int THREADS = (BM / TM) * (BN / TN), WARPS_N = BN / (8 * TN);
    pdl_grid_sync();
    __shared__ __align__(16) float As[2][GF_BK][BM + 4];
    __shared__ __align__(16) float Ws[2][GF_BK][BN + 4];
    const int m_tiles = (M + BM - 1) / BM;          // the row tiles of a panel of W next to each other
    const int m0 = (int)(blockIdx.x % m_tiles) * BM, n0 = (int)(blockIdx.x / m_tiles) * BN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // first row and column of the thread's first piece; the second piece lies 16 rows / 32 columns further on
    const int tm = (warp / WARPS_N) * 4 * TM + (lane >> 3) * 4, tn = (warp % WARPS_N) * 8 * TN + (lane & 7) * 4;
    const bool vec = ((K & 3) == 0) && ((lda & 3) == 0) && ((ldw & 3) == 0) &&
                     ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) acc[i][j] = 0ull;

    GfSlice<BM, THREADS> a;
    GfSlice<BN, THREADS> w;
    a.load(A, m0, M, lda, 0, K, vec);
    w.load(W, n0, N, ldw, 0, K, vec);
    a.store(As[0]);
    w.store(Ws[0]);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += GF_BK, buf ^= 1) {
        const bool more = k0 + GF_BK < K;
        if (more) {
            a.load(A, m0, M, lda, k0 + GF_BK, K, vec);
            w.load(W, n0, N, ldw, k0 + GF_BK, K, vec);
        }
#pragma unroll
        for (int kk = 0; kk < GF_BK; kk++) {
            float av[TM];
            unsigned long long wv[TN / 2];
#pragma unroll
            for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(av + i) = *reinterpret_cast<const float4*>(&As[buf][kk][tm + 4 * i]);
#pragma unroll
            for (int j = 0; j < TN / 2; j += 2)
                *reinterpret_cast<ulonglong2*>(wv + j) = *reinterpret_cast<const ulonglong2*>(&Ws[buf][kk][tn + 16 * j]);
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const unsigned long long ai = gf_pair(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) acc[i][j] = gf_fma2(ai, wv[j], acc[i][j]);
            }
        }
        if (more) {
            // the other buffer was read in the round before, which every thread has left (the barrier below)
            a.store(As[buf ^ 1]);
            w.store(Ws[buf ^ 1]);
        }
        __syncthreads();
    }
    const bool vec_c = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + tm + (i >> 2) * 16 + (i & 3);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int n = n0 + tn + 8 * j;
            float r[4];
            asm("mov.b64 {%0, %1}, %2;" : "=f"(r[0]), "=f"(r[1]) : "l"(acc[i][j / 2]));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(r[2]), "=f"(r[3]) : "l"(acc[i][j / 2 + 1]));
            float* dst = C + (size_t)m * ldc + n;
            if (vec_c && n + 4 <= N) {
                *reinterpret_cast<float4*>(dst) = make_float4(r[0], r[1], r[2], r[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (n + c < N) dst[c] = r[c];
            }
        }
    }
}

// Blocks go where there is room first: launched while the kernel before still holds most SMs, a grid of fewer blocks than SMs comes
// to lie two and three to an SM beside idle ones (88 tiles of 64 x 64, K = 2,048: 190 us, spread out 80).  A grid that gives an SM at
// most three blocks therefore asks for so much shared memory that no more of them fit.
template <int BM, int BN, int TM, int TN>
static int launch_gemm_f32_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
    const long long tiles = ((long long)M + BM - 1) / BM * (((long long)N + BN - 1) / BN);
    if (tiles > 0x7fffffffLL) return ILLM_ERR_BAD_ARG;
    auto kern = gemm_f32_nt_kernel<BM, BN, TM, TN>;
    constexpr int SM_BYTES = 228 * 1024, OWN = 2 * GF_BK * (BM + BN + 8) * (int)sizeof(float), MOST = SM_BYTES / 2 - OWN;
    const int sms = illm_sm_count();
    const long long per = (tiles + sms - 1) / sms, share = SM_BYTES / (per + 1) - OWN;
    const int pad = per <= 3 && share > 0 ? (int)share : 0;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
    if (e != cudaSuccess) return (int)e;
    illm_launch(kern, dim3((unsigned)tiles), dim3((BM / TM) * (BN / TN)), pad, s, A, W, C, M, N, K, lda, ldw, ldc);
    return illm_launch_status();
}

// The same product for at most 8 rows (single tokens of a few sequences), where the tile kernel above
// leaves most of the GPU idle (N / 64 blocks that each wait for one 16-wide slice of K at a time).
// One warp per 32 outputs of a row: the warp streams its [32, K] slab of W through a ring of
// shared-memory stages of 128 values of k, each fetched as four TMA boxes of [32 rows x 32 floats]
// (128-byte rows, 128-byte swizzle) plus one box [MR x 128] of the activations, completion counted
// on the stage's mbarrier; rows past N and columns past K arrive as zeros.  (Earlier forms, with
// 16-byte cp.async or one 512-byte bulk copy per row, reached a quarter of the memory rate: the
// first is bounded by the load/store unit's miss queue, the second by the copy unit's rate of
// requests.)  Every lane owns one output column, whose sum it forms over k in ascending order with
// one fused multiply-add per k, starting from zero: the chain of the tile kernel, so the result is
// the same bits.  A lane reads its own row of a box, 16 bytes at a time, at the swizzled place
// (chunk c of row r lies at chunk c ^ (r & 7)): eight lanes then touch all 32 banks once.  The
// weights are requested before the wait for the kernels ahead (they are nobody's result), the
// activations after it.  The waits are bounded like those of the tensor-core kernels.
#define GS_STAGES(MR) ((MR) > 4 ? 5 : 6)             // two blocks per SM: at most 113 KB each
#define GS_KT 128                                   // values of k per stage
#define GS_W_BYTES (32 * GS_KT * 4)                 // 16 KB: four boxes of 4 KB
#define GS_SMEM(MR) (GS_STAGES(MR) * (GS_W_BYTES + (MR) * GS_KT * 4) + 1024)

template <int MR>
__global__ void __launch_bounds__(32)
gemm_f32_small_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                      float* __restrict__ C, int M, int N, int K, int ldc, int* __restrict__ err) {
    constexpr int S = GS_STAGES(MR);
    extern __shared__ unsigned char gs_raw[];
    __shared__ __align__(8) unsigned long long gs_full[S];
    constexpr unsigned X_BYTES = MR * GS_KT * 4, STAGE_TX = GS_W_BYTES + X_BYTES;
    const unsigned w_base = (tc_smem_u32(gs_raw) + 1023u) & ~1023u, x_base = w_base + S * GS_W_BYTES;
    const unsigned char* w_gen = gs_raw + (w_base - tc_smem_u32(gs_raw));
    const int lane = threadIdx.x, n0 = blockIdx.x * 32;
    const int n_tiles = (K + GS_KT - 1) / GS_KT;
    if (lane == 0) {
        for (int s = 0; s < S; s++) mbar_init(tc_smem_u32(&gs_full[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    auto issue_w = [&](int t) {
        const int s = t % S;
        const unsigned bar = tc_smem_u32(&gs_full[s]);
        mbar_expect_tx(bar, STAGE_TX);
#pragma unroll
        for (int q = 0; q < 4; q++) tma_load_2d(w_base + s * GS_W_BYTES + q * 4096, &map_w, t * GS_KT + q * 32, n0, bar);
    };
    auto issue_x = [&](int t) {
        const int s = t % S;
        tma_load_2d(x_base + s * X_BYTES, &map_a, t * GS_KT, 0, tc_smem_u32(&gs_full[s]));
    };
    const int n_pre = n_tiles < S - 1 ? n_tiles : S - 1;
    if (lane == 0)
        for (int t = 0; t < n_pre; t++) issue_w(t);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (lane == 0)
        for (int t = 0; t < n_pre; t++) issue_x(t);
    float acc[MR];
#pragma unroll
    for (int m = 0; m < MR; m++) acc[m] = 0.f;
    bool alive = true;
    int t = 0;
    for (; t < n_tiles; t++) {
        // the stage that was read in the round before is free (the __syncwarp below)
        if (lane == 0 && t + S - 1 < n_tiles) {
            issue_w(t + S - 1);
            issue_x(t + S - 1);
        }
        alive = __all_sync(0xffffffffu, mbar_wait(tc_smem_u32(&gs_full[t % S]), (t / S) & 1, err));
        if (!alive) break;
        const unsigned char* wst = w_gen + (size_t)(t % S) * GS_W_BYTES + lane * 128;
        const float* xs = reinterpret_cast<const float*>(w_gen + (size_t)S * GS_W_BYTES + (size_t)(t % S) * X_BYTES);
#pragma unroll
        for (int q = 0; q < 4; q++) {
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 w = *reinterpret_cast<const float4*>(wst + q * 4096 + ((c ^ (lane & 7)) << 4));
#pragma unroll
                for (int m = 0; m < MR; m++) {
                    const float4 x = *reinterpret_cast<const float4*>(xs + m * GS_KT + q * 32 + c * 4);
                    acc[m] = fmaf(x.x, w.x, acc[m]);
                    acc[m] = fmaf(x.y, w.y, acc[m]);
                    acc[m] = fmaf(x.z, w.z, acc[m]);
                    acc[m] = fmaf(x.w, w.w, acc[m]);
                }
            }
        }
        __syncwarp();      // the stage is refilled by the next round's requests
    }
    if (!alive) {
        // a wait ran out (the error word is set): no result; the copies still in flight are waited
        // for, each with a short limit, before the block gives its shared memory back
        for (int u = t + 1; u < n_tiles && u < t + S; u++)
            mbar_wait(tc_smem_u32(&gs_full[u % S]), (u / S) & 1, err, TC_ERR_TIMEOUT, 1LL << 24);
        return;
    }
    const int n = n0 + lane;
    if (n < N) {
#pragma unroll
        for (int m = 0; m < MR; m++)
            if (m < M) C[(size_t)m * ldc + n] = acc[m];
    }
}

typedef CUresult (*GsEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Tensor map of a row-major float32 matrix [rows, K] with row stride ld; boxes of [box_rows, box_k].
static int gs_make_map(CUtensorMap* map, const float* ptr, long long rows, long long K, long long ld, int box_rows, int box_k,
                       CUtensorMapSwizzle swizzle) {
    static GsEncodeTiledFn fn = nullptr;
    if (!fn) {
        void* q = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) != cudaSuccess ||
            r != cudaDriverEntryPointSuccess)
            return ILLM_ERR_BAD_ARG;
        fn = (GsEncodeTiledFn)q;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {(cuuint32_t)box_k, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : ILLM_ERR_BAD_ARG;
}

template <int MR>
static int launch_gemm_f32_small(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                 int* err, cudaStream_t s) {
    CUtensorMap mw, ma;
    int rc;
    if ((rc = gs_make_map(&mw, W, N, K, ldw, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B)) != 0) return rc;
    if ((rc = gs_make_map(&ma, A, M, K, lda, MR, GS_KT, CU_TENSOR_MAP_SWIZZLE_NONE)) != 0) return rc;
    auto kern = gemm_f32_small_kernel<MR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM(MR));
    if (e != cudaSuccess) return (int)e;
    illm_launch(kern, dim3((N + 31) / 32), dim3(32), (size_t)GS_SMEM(MR), s, mw, ma, C, M, N, K, ldc, err);
    return illm_launch_status();
}

// err: the device's error word for the bounded waits of the few-rows kernel (null: that kernel is
// not used and every size takes the tile kernel).
extern "C" int illm_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K,
                                int lda, int ldw, int ldc, int* err, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return ILLM_ERR_BAD_ARG;
    if (err != nullptr && M <= 8 && (K & 3) == 0 && (lda & 3) == 0 && (ldw & 3) == 0 &&
        ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0) {
        cudaStream_t s = (cudaStream_t)stream;
        if (M == 1) return launch_gemm_f32_small<1>(A, W, C, M, N, K, lda, ldw, ldc, err, s);
        if (M == 2) return launch_gemm_f32_small<2>(A, W, C, M, N, K, lda, ldw, ldc, err, s);
        if (M <= 4) return launch_gemm_f32_small<4>(A, W, C, M, N, K, lda, ldw, ldc, err, s);
        return launch_gemm_f32_small<8>(A, W, C, M, N, K, lda, ldw, ldc, err, s);
    }
    // A larger thread tile reads less shared memory per FMA, a smaller block leaves fewer SMs idle in the last round and fewer
    // rows beyond M: the tile with the least work on the busiest SM, per output 1 : 1.2 : 1.6.  (512 rows of 7B size: Q/K/V and
    // gate/up 47 TF/s, output and down products 41; over 294 shapes of 9 to 2,048 rows 0.55 of the time of one 64 x 64 tile of 4 x 4
    // outputs a thread, 0.83 where it gains least.)
    cudaStream_t s = (cudaStream_t)stream;
    const int sms = illm_sm_count();
    auto rounds = [&](long long bm, long long bn) { return (double)(((M + bm - 1) / bm * ((N + bn - 1) / bn) + sms - 1) / sms); };
    const double c0 = rounds(128, 128) * 128 * 128, c1 = rounds(64, 64) * 64 * 64 * 1.2, c2 = rounds(32, 64) * 32 * 64 * 1.6;
    if (c0 <= c1 && c0 <= c2) return launch_gemm_f32_tile<128, 128, 8, 16>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (c1 <= c2) return launch_gemm_f32_tile<64, 64, 8, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
    return launch_gemm_f32_tile<32, 64, 4, 4>(A, W, C, M, N, K, lda, ldw, ldc, s);
}
