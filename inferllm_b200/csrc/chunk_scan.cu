// Linear attention and the gated delta rule over a per-sequence float32 state, eight tokens at a time, for steps where that
// order of the sums is allowed (the bfloat16 mode's prompts).  With S [d, dv] the state before the eight tokens, G_j the product
// of the decays up to token j and D_ji the product of those behind i up to j (numbers, or one per key channel),
//     delta rule:         u_j = beta_j (v_j - S^T G_j k_j - sum_(i<j) (k_i . D_ji k_j) u_i)
//     linear attention:   u_j = v_j
//     o_j = S^T G_j q_j + sum_(i<=j) (k_i . D_ji q_j) u_i
//     S  <- G_7 S + sum_i (D_7i k_i) u_i^T
// so the sixteen (eight) products with S are independent of one another, and only short triangular sums follow in order.  The
// products k_i . D_ji k_j, which all columns share, are made by chunk_prep_kernel (chunk_prep_channel_kernel) and lie in a
// record per chunk and head.  Decays are multiplied, never divided by, so strong ones go to zero as they do token by
// token.  float32 throughout; tokens beyond a sequence's end count as k = q = 0, decay 1, beta 0.
//
// chunk_scan_kernel: a block owns 32 columns of one (sequence, head); a warp 8 of them, a thread 16 rows of 2 columns in
// registers (rows in pairs for fma.rn.f32x2).  What bounds it is the float32 FMA rate and the chain of a sequence's chunks.
// With one column of 8 rows per thread (what ran here before) the same products were bound by shared-memory reads
// (a 16-byte read per four FMAs) and by the shuffles that add a column's parts over its lanes; now a read serves two columns.
// (16 rows of 4 columns halve the reads again, but then 203 registers leave a scheduler two warps: 690 against 740 us in the
// first case below, and a single sequence's chain became slower.)  The lanes' parts are added by exchanging halves: of
// the eight lanes of a column group, lanes 0-3 end up with the eight sums S^T k of column l / 2 and lanes 4-7 with those of
// S^T q, in the order the triangular sums need them.
// Measured, a layer of 16 heads of 128 x 128: the delta rule with a decay per channel, eight sequences of 250 to 1,500 tokens,
// 1,318 -> 740 us; linear attention, one sequence of 2,048 tokens, 291 -> 167 us with its folds (eight segments before, 13 now),
// 8 heads and 32 sequences of 100 to 900 tokens 535 -> 426 us.
// Linear attention has no chain but the state's, which a.segments cuts: every segment of a sequence runs from a state of zero
// (the first from the sequence's), chunk_fold_kernel gives each the state at its start, S_in = a^len S_in + S of the
// segment before, and chunk_add_kernel adds what the tokens missed, a^(t - t0 + 1) S_in^T q_t.
#include "chunk_scan.h"

#include "common.cuh"
#include "kernels.h"

#define CS_T 8                                  // tokens per chunk
#define CS_TILE 16                              // tokens staged at a time
#define CS_D 128                                // rows of the state, with padding
#define CS_C 2                                  // columns per thread
#define CS_THREADS 128
#define CS_COLS (CS_THREADS / 8 * CS_C)         // columns per block
#define CS_REC (4 * CS_T + 2 * CS_T * CS_T)     // floats per (chunk, head): beta, beta G, G, D_7i, then M[j][i] and P[j][i]

// Chunk c of the step's sequence b has its record at slot cu_q[b] / CS_T + b + c (distinct for all chunks of a step).
__device__ __forceinline__ int cs_slot(int first, int b, int c) { return first / CS_T + b + c; }
long long chunk_scan_scratch(long long T, int B, int nh) { return (T / CS_T + B + 1) * nh * CS_REC; }

// One decay per head.  grid (chunks of the longest sequence, query/key heads, sequences), 128 threads: a thread per product of two
// rows (rows 4 floats further apart than they are long, so that the lanes' 16-byte reads meet different banks), then the
// records of the value heads that share the keys.
template <bool DELTA>
__global__ void __launch_bounds__(CS_THREADS) chunk_prep_kernel(const ChunkScanArgs p) {
    pdl_grid_sync();
    __shared__ __align__(16) float sk[CS_T][CS_D + 4], sq[CS_T][CS_D + 4];
    __shared__ float dots[2][CS_T][CS_T];        // k_i . k_j and k_i . q_j at [j][i]
    const int c = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    const int first = p.cu_q[b], n = p.cu_q[b + 1] - first, t0 = c * CS_T;
    if (t0 >= n) return;
    const int nt = min(CS_T, n - t0), d = p.d;
    for (int e = threadIdx.x; e < CS_T * CS_D; e += CS_THREADS) {
        const int j = e / CS_D, i = e % CS_D;
        const long long at = (first + t0 + j) * p.ld + (long long)hk * d + i;
        const bool in = j < nt && i < d;
        sk[j][i] = in ? p.k[at] : 0.f;
        sq[j][i] = in ? p.q[at] : 0.f;
    }
    __syncthreads();
    {
        const int e = threadIdx.x, which = e >> 6, j = (e >> 3) & 7, i = e & 7;
        if (DELTA || which) {
            const float4 *x = reinterpret_cast<const float4*>(sk[i]), *y = reinterpret_cast<const float4*>(which ? sq[j] : sk[j]);
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 8
            for (int r = 0; r < CS_D / 4; r++) {
                const float4 u = x[r], w = y[r];
                s0 = fmaf(u.x, w.x, s0), s1 = fmaf(u.y, w.y, s1), s2 = fmaf(u.z, w.z, s2), s3 = fmaf(u.w, w.w, s3);
            }
            dots[which][j][i] = (s0 + s1) + (s2 + s3);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < p.share * CS_T; e += CS_THREADS) {
        const int h = hk * p.share + e / CS_T, j = e % CS_T;
        float g[CS_T];
#pragma unroll
        for (int i = 0; i < CS_T; i++) g[i] = i < nt ? (DELTA ? p.g[(size_t)(first + t0 + i) * p.nh + h] : p.g[h]) : 1.f;
        const float beta = DELTA && j < nt ? p.beta[(size_t)(first + t0 + j) * p.nh + h] : 0.f;
        float G = 1.f, E = 1.f;
#pragma unroll
        for (int i = 0; i < CS_T; i++) {
            if (i <= j) G *= g[i];
            if (i > j) E *= g[i];
        }
        float* r = p.rec + ((size_t)cs_slot(first, b, c) * p.nh + h) * CS_REC;
        r[j] = beta;
        r[CS_T + j] = beta * G;
        r[2 * CS_T + j] = G;
        r[3 * CS_T + j] = E;
        float D = 1.f;                           // D_ji, from i = j down
#pragma unroll
        for (int i = CS_T - 1; i >= 0; i--) {
            if (i < j) D *= g[i + 1 < CS_T ? i + 1 : CS_T - 1];
            r[4 * CS_T + j * CS_T + i] = DELTA && i < j ? beta * D * dots[0][j][i] : 0.f;
            r[4 * CS_T + CS_T * CS_T + j * CS_T + i] = i <= j ? D * dots[1][j][i] : 0.f;
        }
    }
}

// A decay per head and key channel.  grid (chunks, value heads, sequences), 128 threads, a thread per channel: the running products of
// the decays give its part of all 64 sums (28 of M, 36 of P: k_i D_ji q_j at place [j][i], i <= j; k_i D_ji k_j at the mirrored
// place), which the lanes add by exchanging halves.
__global__ void __launch_bounds__(CS_THREADS) chunk_prep_channel_kernel(const ChunkScanArgs p) {
    pdl_grid_sync();
    __shared__ float part[CS_THREADS / 32][CS_T * CS_T];
    const int c = blockIdx.x, h = blockIdx.y, hk = h / p.share, b = blockIdx.z;
    const int first = p.cu_q[b], n = p.cu_q[b + 1] - first, t0 = c * CS_T;
    if (t0 >= n) return;
    const int nt = min(CS_T, n - t0), d = p.d, i0 = threadIdx.x, lane = threadIdx.x & 31;
    float k[CS_T], q[CS_T], g[CS_T], v[CS_T * CS_T];
#pragma unroll
    for (int j = 0; j < CS_T; j++) {
        const bool in = j < nt && i0 < d;
        const long long t = first + t0 + j;
        k[j] = in ? p.k[t * p.ld + (long long)hk * d + i0] : 0.f;
        q[j] = in ? p.q[t * p.ld + (long long)hk * d + i0] : 0.f;
        g[j] = in ? p.g[t * p.nh * d + (long long)h * d + i0] : 1.f;
    }
#pragma unroll
    for (int i = 0; i < CS_T; i++) {
        float x = k[i];
        v[i * CS_T + i] = x * q[i];
#pragma unroll
        for (int j = i + 1; j < CS_T; j++) {
            x *= g[j];
            v[j * CS_T + i] = x * q[j];
            v[i * CS_T + j] = x * k[j];
        }
    }
#pragma unroll
    for (int o = 16, m = CS_T * CS_T / 2; o >= 1; o >>= 1, m >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int x = 0; x < m; x++) {
            const float mine = up ? v[x + m] : v[x], theirs = up ? v[x] : v[x + m];
            v[x] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    }
    part[threadIdx.x >> 5][2 * lane] = v[0];
    part[threadIdx.x >> 5][2 * lane + 1] = v[1];
    __syncthreads();
    float* r = p.rec + ((size_t)cs_slot(first, b, c) * p.nh + h) * CS_REC;
    const int e = threadIdx.x;
    if (e < CS_T * CS_T) {
        const float s = (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
        const int row = e / CS_T, col = e % CS_T;
        if (col <= row) {
            r[4 * CS_T + CS_T * CS_T + e] = s;
        } else {
            const float beta = col < nt ? p.beta[(size_t)(first + t0 + col) * p.nh + h] : 0.f;
            r[4 * CS_T + col * CS_T + row] = beta * s;
        }
    } else if (e < CS_T * CS_T + CS_T) {
        const int j = e - CS_T * CS_T;
        r[j] = j < nt ? p.beta[(size_t)(first + t0 + j) * p.nh + h] : 0.f;
    }
}

__device__ __forceinline__ unsigned long long cs_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 cs_unpack(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long cs_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long cs_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void cs_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cs_cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// floats of one of the two buffers: q, k (and the channels' decays) of a tile, v, the two chunks' records
template <int KIND> struct CsBuf {
    static constexpr int ROWS = KIND == CHUNK_DELTA_CHANNEL ? 3 : 2;
    static constexpr int V_AT = ROWS * CS_TILE * CS_D, REC_AT = V_AT + CS_TILE * CS_COLS, SIZE = REC_AT + CS_TILE / CS_T * CS_REC;
    static constexpr int BYTES = (2 * SIZE + (KIND == CHUNK_DELTA_CHANNEL ? CS_TILE / CS_T * CS_D : 0)) * 4;
};

// A sequence's tokens of segment seg of P: whole tiles each, the last ones possibly empty.
__device__ __forceinline__ int cs_segment_len(int n, int P) { return P > 1 ? ((n + P - 1) / P + CS_TILE - 1) / CS_TILE * CS_TILE : n; }

// grid (columns / 32, heads, sequences x segments).  wide: 16-byte copies (d, dv, ld and the addresses allow them).
template <int KIND>
__global__ void __launch_bounds__(CS_THREADS, KIND == CHUNK_DELTA_HEAD ? 2 : 3) chunk_scan_kernel(const ChunkScanArgs p, const int wide) {
    pdl_grid_sync();
    extern __shared__ __align__(16) float sm[];
    using Buf = CsBuf<KIND>;
    constexpr bool DELTA = KIND != CHUNK_LINEAR, CHANNEL = KIND == CHUNK_DELTA_CHANNEL;
    const int P = KIND == CHUNK_LINEAR ? p.segments : 1, b = blockIdx.z / P, seg = blockIdx.z % P;
    const int h = blockIdx.y, hk = h / p.share, j0 = blockIdx.x * CS_COLS;
    const int d = p.d, dv = p.dv;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l = lane & 7;
    const int col0 = (warp * 4 + (lane >> 3)) * CS_C;       // the thread's columns within the block: col0, col0 + 1
    const int q0 = p.cu_q[b], seg_len = cs_segment_len(p.cu_q[b + 1] - q0, P);
    const int first = q0 + seg * seg_len, n = min(seg_len, p.cu_q[b + 1] - first);      // the segment's tokens
    const int chunk0 = seg * (seg_len / CS_T);              // its first chunk (whole tiles per segment)
    if (n <= 0) return;
    float* Sg = p.state + (size_t)p.slots[b] * p.state_stride + ((size_t)h * dv + j0 + col0) * d;
    float* Sout = P > 1 ? p.seg_state + (((size_t)b * P + seg) * p.nh + h) * dv * d + (size_t)(j0 + col0) * d : Sg;
    const bool fresh = seg > 0;
    // rows 4 (l + 8 r) .. + 3 of column c: pairs S[c][2 r], S[c][2 r + 1]
    unsigned long long S[CS_C][8];
#pragma unroll
    for (int c = 0; c < CS_C; c++)
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = 4 * (l + 8 * (r >> 1)) + 2 * (r & 1);
            const bool live = !fresh && j0 + col0 + c < dv;
            S[c][r] = cs_pack(live && i < d ? Sg[(size_t)c * d + i] : 0.f, live && i + 1 < d ? Sg[(size_t)c * d + i + 1] : 0.f);
        }
    if (d < CS_D) {                                         // rows beyond d: k = q = 0 in both buffers
        const int pad = CS_D - d;
        for (int e = threadIdx.x; e < 2 * Buf::ROWS * CS_TILE * pad; e += CS_THREADS) {
            const int row = e / pad;
            sm[(row / (Buf::ROWS * CS_TILE)) * Buf::SIZE + (row % (Buf::ROWS * CS_TILE)) * CS_D + d + e % pad] = 0.f;
        }
    }
    auto stage = [&](int buf, int t0) {
        float* sb = sm + buf * Buf::SIZE;
        const int nt = min(CS_TILE, n - t0), nc = (nt + CS_T - 1) / CS_T, np = nc * CS_T;      // np: with the last chunk's missing tokens
        const long long tok = first + t0;
        if (wide) {
            const int quads = d >> 2;
            for (int tt = warp; tt < np; tt += CS_THREADS / 32) {
                if (lane < quads) {
                    float* dst = sb + tt * CS_D + 4 * lane;
                    if (tt < nt) {
                        const long long at = (tok + tt) * p.ld + (long long)hk * d + 4 * lane;
                        cs_cp16(dst, p.q + at);
                        cs_cp16(dst + CS_TILE * CS_D, p.k + at);
                        if (CHANNEL) cs_cp16(dst + 2 * CS_TILE * CS_D, p.g + ((tok + tt) * p.nh + h) * d + 4 * lane);
                    } else {
                        *reinterpret_cast<float4*>(dst) = *reinterpret_cast<float4*>(dst + CS_TILE * CS_D) = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (CHANNEL) *reinterpret_cast<float4*>(dst + 2 * CS_TILE * CS_D) = make_float4(1.f, 1.f, 1.f, 1.f);
                    }
                }
            }
            for (int e = threadIdx.x; e < np * (CS_COLS / 4); e += CS_THREADS) {
                const int tt = e / (CS_COLS / 4), c = e % (CS_COLS / 4) * 4;
                float* dst = sb + Buf::V_AT + tt * CS_COLS + c;
                if (tt < nt && j0 + c < dv) cs_cp16(dst, p.v + (tok + tt) * p.ld + (long long)h * dv + j0 + c);
                else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else {
            for (int tt = warp; tt < np; tt += CS_THREADS / 32)
                for (int i = lane; i < d; i += 32) {
                    float* dst = sb + tt * CS_D + i;
                    if (tt < nt) {
                        const long long at = (tok + tt) * p.ld + (long long)hk * d + i;
                        cs_cp4(dst, p.q + at);
                        cs_cp4(dst + CS_TILE * CS_D, p.k + at);
                        if (CHANNEL) cs_cp4(dst + 2 * CS_TILE * CS_D, p.g + ((tok + tt) * p.nh + h) * d + i);
                    } else {
                        dst[0] = dst[CS_TILE * CS_D] = 0.f;
                        if (CHANNEL) dst[2 * CS_TILE * CS_D] = 1.f;
                    }
                }
            for (int e = threadIdx.x; e < np * CS_COLS; e += CS_THREADS) {
                const int tt = e / CS_COLS, c = e % CS_COLS;
                float* dst = sb + Buf::V_AT + e;
                if (tt < nt && j0 + c < dv) cs_cp4(dst, p.v + (tok + tt) * p.ld + (long long)h * dv + j0 + c);
                else *dst = 0.f;
            }
        }
        for (int e = threadIdx.x; e < nc * (CS_REC / 4); e += CS_THREADS) {
            const int cc = e / (CS_REC / 4), x = e % (CS_REC / 4) * 4;
            cs_cp16(sb + Buf::REC_AT + cc * CS_REC + x, p.rec + ((size_t)cs_slot(q0, b, chunk0 + t0 / CS_T + cc) * p.nh + h) * CS_REC + x);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    stage(0, 0);
    for (int t0 = 0, it = 0; t0 < n; t0 += CS_TILE, it ^= 1) {
        const int nt = min(CS_TILE, n - t0);
        if (t0 + CS_TILE < n) {
            stage(it ^ 1, t0 + CS_TILE);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        float* sb = sm + it * Buf::SIZE;
        float* s_end = sm + 2 * Buf::SIZE;                  // CHANNEL: the product of a chunk's decays per channel
        if (CHANNEL) {
            // in place: q_j <- G_j q_j, k_j <- G_j k_j, and where the decays lay D_7j k_j; a thread per channel
            for (int x = threadIdx.x; x < d; x += CS_THREADS) {
#pragma unroll 1
                for (int c0 = 0; c0 < nt; c0 += CS_T) {
                    float* col = sb + c0 * CS_D + x;
                    float g[CS_T], k[CS_T], G = 1.f;
#pragma unroll
                    for (int j = 0; j < CS_T; j++) {
                        g[j] = col[(2 * CS_TILE + j) * CS_D];
                        k[j] = col[(CS_TILE + j) * CS_D];
                        G *= g[j];
                        col[j * CS_D] *= G;
                        col[(CS_TILE + j) * CS_D] = k[j] * G;
                    }
                    s_end[c0 / CS_T * CS_D + x] = G;
                    G = 1.f;
#pragma unroll
                    for (int j = CS_T - 1; j >= 0; j--) {
                        col[(2 * CS_TILE + j) * CS_D] = k[j] * G;
                        G *= g[j];
                    }
                }
            }
            if (d < CS_D)
                for (int x = d + threadIdx.x; x < CS_D; x += CS_THREADS) s_end[x] = s_end[CS_D + x] = 0.f;
            __syncthreads();
        }
#pragma unroll 1
        for (int c0 = 0; c0 < nt; c0 += CS_T) {
            const float* rows = sb + c0 * CS_D + 4 * l;
            const float* rec = sb + Buf::REC_AT + c0 / CS_T * CS_REC;
            const float* vs = sb + Buf::V_AT + c0 * CS_COLS + col0;
            // the thread's parts of S^T x_j for the eight rows x_j of q (at 0) or k (at CS_TILE)
            auto dots = [&](const float* x, float (&r)[CS_T][CS_C]) {
                unsigned long long acc[CS_T][CS_C];
#pragma unroll
                for (int j = 0; j < CS_T; j++)
#pragma unroll
                    for (int c = 0; c < CS_C; c++) acc[j][c] = 0ull;
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int j = 0; j < CS_T; j++) {
                        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(x + j * CS_D + 32 * q);
#pragma unroll
                        for (int c = 0; c < CS_C; c++) acc[j][c] = cs_fma2(v.y, S[c][2 * q + 1], cs_fma2(v.x, S[c][2 * q], acc[j][c]));
                    }
#pragma unroll
                for (int j = 0; j < CS_T; j++)
#pragma unroll
                    for (int c = 0; c < CS_C; c++) {
                        const float2 f = cs_unpack(acc[j][c]);
                        r[j][c] = f.x + f.y;
                    }
            };
            // row j of a record's matrix; eight numbers of a record
            auto eight = [&](int at, float (&r)[CS_T]) {
                const float4 a = *reinterpret_cast<const float4*>(rec + at), c = *reinterpret_cast<const float4*>(rec + at + 4);
                r[0] = a.x, r[1] = a.y, r[2] = a.z, r[3] = a.w, r[4] = c.x, r[5] = c.y, r[6] = c.z, r[7] = c.w;
            };
            const bool up4 = (l & 4) != 0, up2 = (l & 2) != 0;
            const int cc = (l >> 1) & 1;                    // the column whose sums this lane ends up with
            unsigned long long w[CS_T][CS_C];               // D_7i u_i of the thread's columns, twice
            float O[CS_T][CS_C];
            dots(rows, O);
            if (DELTA) {
                float A[CS_T][CS_C], z[CS_T], u[CS_T], o[CS_T], beta[CS_T], x8[CS_T];
                dots(rows + CS_TILE * CS_D, A);
#pragma unroll
                for (int j = 0; j < CS_T; j++)
#pragma unroll
                    for (int c = 0; c < CS_C; c++) {
                        const float mine = up4 ? O[j][c] : A[j][c], theirs = up4 ? A[j][c] : O[j][c];
                        A[j][c] = mine + __shfl_xor_sync(0xffffffffu, theirs, 4);
                    }
                eight(0, beta);
                if (!CHANNEL) eight(CS_T, x8);
#pragma unroll
                for (int j = 0; j < CS_T; j++) {
                    const float mine = up2 ? A[j][1] : A[j][0], theirs = up2 ? A[j][0] : A[j][1];
                    z[j] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2);
                    u[j] = beta[j] * vs[j * CS_COLS + cc];
                }
#pragma unroll
                for (int j = 0; j < CS_T; j++) z[j] += __shfl_xor_sync(0xffffffffu, z[j], 1);
                // the triangular sums: u in the lanes that hold S^T k, then handed to those that hold S^T q
#pragma unroll
                for (int j = 0; j < CS_T; j++) {
                    float m[CS_T];
                    if (j > 0) eight(4 * CS_T + j * CS_T, m);
                    u[j] = fmaf(-(CHANNEL ? beta[j] : x8[j]), z[j], u[j]);
#pragma unroll
                    for (int i = 0; i < j; i++) u[j] = fmaf(-m[i], u[i], u[j]);
                }
                if (!CHANNEL) eight(2 * CS_T, x8);
#pragma unroll
                for (int j = 0; j < CS_T; j++) {
                    u[j] = __shfl_sync(0xffffffffu, u[j], lane & ~4);
                    o[j] = CHANNEL ? z[j] : x8[j] * z[j];
                }
                if (!CHANNEL) eight(3 * CS_T, x8);
#pragma unroll
                for (int i = 0; i < CS_T; i++) {
                    const float x = CHANNEL ? u[i] : x8[i] * u[i];
#pragma unroll
                    for (int c = 0; c < CS_C; c++) {
                        const float y = __shfl_sync(0xffffffffu, x, (lane & 24) | (2 * c));
                        w[i][c] = cs_pack(y, y);
                    }
                }
#pragma unroll
                for (int j = 0; j < CS_T; j++) {
                    float m[CS_T];
                    eight(4 * CS_T + CS_T * CS_T + j * CS_T, m);
#pragma unroll
                    for (int i = 0; i <= j; i++) o[j] = fmaf(m[i], u[i], o[j]);
                }
                // lanes 4 and 5 of a column group hold column 0, 6 and 7 column 1: the even one stores tokens 0-3, the odd one 4-7
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float r = (l & 1) ? o[j + 4] : o[j];
                    const int t = c0 + j + 4 * (l & 1);
                    if (up4 && t < nt && j0 + col0 + cc < dv) p.out[(size_t)(first + t0 + t) * p.nh * dv + (size_t)h * dv + j0 + col0 + cc] = r;
                }
            } else {
                // lane l: tokens 4 (l / 4) + 2 (l & 1) and the one behind of column (l / 2) & 1
                float v[CS_T], x8[CS_T];
#pragma unroll
                for (int i = 0; i < CS_T; i++) v[i] = vs[i * CS_COLS + cc];
#pragma unroll
                for (int j = 0; j < 4; j++)
#pragma unroll
                    for (int c = 0; c < CS_C; c++) {
                        const float mine = up4 ? O[j + 4][c] : O[j][c], theirs = up4 ? O[j][c] : O[j + 4][c];
                        O[j][c] = mine + __shfl_xor_sync(0xffffffffu, theirs, 4);
                    }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float mine = up2 ? O[j][1] : O[j][0], theirs = up2 ? O[j][0] : O[j][1];
                    O[j][0] = mine + __shfl_xor_sync(0xffffffffu, theirs, 2);
                }
#pragma unroll
                for (int jj = 0; jj < 2; jj++) {
                    const float mine = (l & 1) ? O[jj + 2][0] : O[jj][0], theirs = (l & 1) ? O[jj][0] : O[jj + 2][0];
                    const float z = mine + __shfl_xor_sync(0xffffffffu, theirs, 1);
                    const int j = (l & 4) + 2 * (l & 1) + jj;
                    float m[CS_T], o = rec[2 * CS_T + j] * z;
                    eight(4 * CS_T + CS_T * CS_T + j * CS_T, m);
#pragma unroll
                    for (int i = 0; i < CS_T; i++) o = i <= j ? fmaf(m[i], v[i], o) : o;     // (a later token's infinite value stays out)
                    if (c0 + j < nt && j0 + col0 + cc < dv)
                        p.out[(size_t)(first + t0 + c0 + j) * p.nh * dv + (size_t)h * dv + j0 + col0 + cc] = o;
                }
                eight(3 * CS_T, x8);
#pragma unroll
                for (int i = 0; i < CS_T; i++) {
                    const float2 x = *reinterpret_cast<const float2*>(vs + i * CS_COLS);
                    w[i][0] = cs_pack(x8[i] * x.x, x8[i] * x.x), w[i][1] = cs_pack(x8[i] * x.y, x8[i] * x.y);
                }
            }
            // the state behind the chunk
            const float* keys = rows + (CHANNEL ? 2 : 1) * CS_TILE * CS_D;
            const float G = CHANNEL ? 1.f : rec[2 * CS_T + CS_T - 1];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ulonglong2 g2 = make_ulonglong2(cs_pack(G, G), cs_pack(G, G));
                if (CHANNEL) g2 = *reinterpret_cast<const ulonglong2*>(s_end + c0 / CS_T * CS_D + 4 * l + 32 * q);
#pragma unroll
                for (int c = 0; c < CS_C; c++) S[c][2 * q] = cs_mul2(S[c][2 * q], g2.x), S[c][2 * q + 1] = cs_mul2(S[c][2 * q + 1], g2.y);
#pragma unroll
                for (int i = 0; i < CS_T; i++) {
                    const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(keys + i * CS_D + 32 * q);
#pragma unroll
                    for (int c = 0; c < CS_C; c++) {
                        S[c][2 * q] = cs_fma2(k.x, w[i][c], S[c][2 * q]);
                        S[c][2 * q + 1] = cs_fma2(k.y, w[i][c], S[c][2 * q + 1]);
                    }
                }
            }
        }
        __syncthreads();          // the tile after the next one goes into this buffer
    }
#pragma unroll
    for (int c = 0; c < CS_C; c++)
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = 4 * (l + 8 * (r >> 1)) + 2 * (r & 1);
            const float2 f = cs_unpack(S[c][r]);
            if (j0 + col0 + c < dv) {
                if (i < d) Sout[(size_t)c * d + i] = f.x;
                if (i + 1 < d) Sout[(size_t)c * d + i + 1] = f.y;
            }
        }
}


// The segments' states become the states at their starts (of the first: what the sequence brought is inside already), and the
// sequence gets its own.  grid (elements / 1024, heads, sequences), 256 threads, four elements a thread.
__global__ void __launch_bounds__(256) chunk_fold_kernel(const ChunkScanArgs p) {
    pdl_grid_sync();
    const int b = blockIdx.z, h = blockIdx.y, P = p.segments, n = p.cu_q[b + 1] - p.cu_q[b];
    if (n <= 0) return;
    const int elems = p.d * p.dv, len = cs_segment_len(n, P), used = (n + len - 1) / len;
    float whole = 1.f, last = 1.f;                          // a^len, and a^(tokens of the last segment)
    const float a = p.g[h];
    for (int i = 0; i < len; i++) whole *= a;
    for (int i = 0; i < n - (used - 1) * len; i++) last *= a;
    float* seg = p.seg_state + ((size_t)b * P * p.nh + h) * elems;
    const size_t stride = (size_t)p.nh * elems;
    float* Sg = p.state + (size_t)p.slots[b] * p.state_stride + (size_t)h * elems;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const int e = blockIdx.x * 1024 + x * 256 + threadIdx.x;
        if (e >= elems) break;
        float s = seg[e];
        for (int r = 1; r < used; r++) {
            const float own = seg[r * stride + e];
            seg[r * stride + e] = s;
            s = fmaf(s, r + 1 < used ? whole : last, own);
        }
        Sg[e] = s;
    }
}

// o_t += a^(t - t0 + 1) S_in^T q_t for the tokens of every segment but a sequence's first: a product of q [tokens, d] with the
// state at the segment's start.  grid (columns / 64 x pieces of 64 tokens, heads, sequences x (segments - 1)), 128
// threads, a thread 8 tokens x 4 columns, both operands channel by channel in shared memory (64 channels at a time).
__global__ void __launch_bounds__(128) chunk_add_kernel(const ChunkScanArgs p, const int col_blocks) {
    pdl_grid_sync();
    __shared__ __align__(16) float sq[64][64 + 4], ss[64][64 + 4];
    const int P = p.segments, b = blockIdx.z / (P - 1), seg = blockIdx.z % (P - 1) + 1, h = blockIdx.y, hk = h / p.share;
    const int j0 = blockIdx.x % col_blocks * 64, d = p.d, dv = p.dv;
    const int q0 = p.cu_q[b], n = p.cu_q[b + 1] - q0, len = cs_segment_len(n, P), piece = blockIdx.x / col_blocks * 64;
    const int t0 = q0 + seg * len + piece, nt = min(min(64, len - piece), q0 + n - t0);
    if (nt <= 0) return;
    const float* S = p.seg_state + (((size_t)b * P + seg) * p.nh + h) * dv * d;
    const int tt = threadIdx.x / 16 * 8, tc = threadIdx.x % 16 * 4;
    unsigned long long acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = 0ull;
    for (int i0 = 0; i0 < d; i0 += 64) {
        __syncthreads();
        for (int e = threadIdx.x; e < 64 * 64; e += 128) {
            const int r = e >> 6, i = e & 63;
            sq[i][r] = r < nt && i0 + i < d ? p.q[(long long)(t0 + r) * p.ld + (long long)hk * d + i0 + i] : 0.f;
            ss[i][r] = j0 + r < dv && i0 + i < d ? S[(size_t)(j0 + r) * d + i0 + i] : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int i = 0; i < 64; i++) {
            const float4 qa = *reinterpret_cast<const float4*>(&sq[i][tt]), qb = *reinterpret_cast<const float4*>(&sq[i][tt + 4]);
            const ulonglong2 sv = *reinterpret_cast<const ulonglong2*>(&ss[i][tc]);
            const float q[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const unsigned long long q2 = cs_pack(q[x], q[x]);
                acc[x][0] = cs_fma2(q2, sv.x, acc[x][0]);
                acc[x][1] = cs_fma2(q2, sv.y, acc[x][1]);
            }
        }
    }
    const float a = p.g[h];
    float f = 1.f;
    for (int i = 0; i < piece + tt; i++) f *= a;
#pragma unroll
    for (int x = 0; x < 8; x++) {
        f *= a;
        if (tt + x >= nt) break;
        const float2 lo = cs_unpack(acc[x][0]), hi = cs_unpack(acc[x][1]);
        float* o = p.out + (size_t)(t0 + tt + x) * p.nh * dv + (size_t)h * dv + j0 + tc;
        const float r[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (j0 + tc + c < dv) o[c] = fmaf(f, r[c], o[c]);
    }
}

template <int KIND>
static int cs_launch(const ChunkScanArgs& a, int B, int max_q, cudaStream_t s) {
    const int chunks = (max_q + CS_T - 1) / CS_T;
    if constexpr (KIND == CHUNK_DELTA_CHANNEL) illm_launch(chunk_prep_channel_kernel, dim3(chunks, a.nh, B), dim3(CS_THREADS), 0, s, a);
    else illm_launch(chunk_prep_kernel<KIND == CHUNK_DELTA_HEAD>, dim3(chunks, a.nh / a.share, B), dim3(CS_THREADS), 0, s, a);
    auto kern = chunk_scan_kernel<KIND>;
    const int P = KIND == CHUNK_LINEAR ? a.segments : 1;
    const dim3 grid((a.dv + CS_COLS - 1) / CS_COLS, a.nh, B * P);
    // A grid that fits the SMs once asks for more than half an SM's shared memory: launched behind kernels that still hold most SMs, its
    // blocks would otherwise be packed by threes onto those that are free first, and the slowest would decide.
    const size_t need = CsBuf<KIND>::BYTES, spread = (size_t)120 * 1024;
    const size_t smem = (long long)grid.x * grid.y * grid.z <= illm_sm_count() ? spread : need;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)spread);
    if (e != cudaSuccess) return (int)e;
    const int wide = !((a.d | a.dv) & 3) && !(a.ld & 3) && !(((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v) & 15) &&
                     (KIND != CHUNK_DELTA_CHANNEL || !((uintptr_t)a.g & 15));
    illm_launch(kern, grid, dim3(CS_THREADS), smem, s, a, wide);
    if (P > 1) {
        const int col_blocks = (a.dv + 63) / 64, longest = ((max_q + P - 1) / P + CS_TILE - 1) / CS_TILE * CS_TILE;
        illm_launch(chunk_fold_kernel, dim3((a.d * a.dv + 1023) / 1024, a.nh, B), dim3(256), 0, s, a);
        illm_launch(chunk_add_kernel, dim3(col_blocks * ((longest + 63) / 64), a.nh, B * (P - 1)), dim3(128), 0, s, a, col_blocks);
    }
    return illm_launch_status();
}

// As many segments of a sequence as leave the SMs about three blocks each, of at least 64 tokens: below that the states'
// way through memory (d x dv floats per segment, three times) costs more than the shorter chain gives.
int chunk_scan_segments(int kind, int B, int nh, int dv, int max_q) {
    if (kind != CHUNK_LINEAR) return 1;
    const long long blocks = (long long)B * nh * ((dv + CS_COLS - 1) / CS_COLS);
    long long P = (3LL * illm_sm_count() + blocks / 2) / blocks;
    if (P > max_q / 64) P = max_q / 64;
    return P > 32 ? 32 : (P < 2 ? 1 : (int)P);
}

int chunk_scan_launch(const ChunkScanArgs& a, int kind, int B, int max_q, cudaStream_t s) {
    if (!chunk_scan_takes(a.d) || a.dv <= 0 || a.nh <= 0 || a.nh > 65535 || a.segments < 1 || (long long)B * a.segments > 65535 || (a.segments > 1 && !a.seg_state) || a.share <= 0 || a.nh % a.share || max_q <= 0 || !a.rec ||
        ((uintptr_t)a.rec & 15))
        return ILLM_ERR_BAD_ARG;
    if (kind == CHUNK_LINEAR) return cs_launch<CHUNK_LINEAR>(a, B, max_q, s);
    if (kind == CHUNK_DELTA_HEAD) return cs_launch<CHUNK_DELTA_HEAD>(a, B, max_q, s);
    return cs_launch<CHUNK_DELTA_CHANNEL>(a, B, max_q, s);
}
