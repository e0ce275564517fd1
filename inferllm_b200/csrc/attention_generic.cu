// Causal attention of every token of a step over the paged cache: the generic kernel.
//
// It takes any head size up to 256 (16-byte loads where it is a multiple of 8, element by element
// otherwise), any number of heads and groups, any page size, float32 or bfloat16 storage, prompts
// and single tokens alike, and does all arithmetic in float32.  It is the whole attention of the float32 mode and the fall-back of
// the bfloat16 mode for head sizes that the tensor-core kernels do not take.
//
// The reference materialises the score matrix and runs four launches over it: a batched
// product Q K^T (src/kern/gpu/kernel_gpu.cu:576-591), scale + causal mask (:504-536), a
// three-pass row softmax (:78-125) and the batched product with V (:593-609); formulas
// src/kern/naive/naive.cpp:606-632, :531-553, :209-240, :664-691, grouped heads :576-604.
// Here the keys lo..p of a (token, head) are dealt to sixteen strands in blocks of 32 (a key per lane for the
// scores, a channel per lane for the values), each with a running maximum and sum, and the strands are merged in
// a fixed order.  The split of the keys depends only on the token's own position and window, so its result does
// not depend on the step it is part of.  Two kernels run these strands, with the same operations in the same order:
//   attention_generic_kernel       a (token, head) per cluster of 1 to 8 blocks, a strand per warp: single tokens,
//                                  and prompts behind a sliding window;
//   attention_generic_tile_kernel  eight tokens of a prompt and a head per block: a key or value row that a warp has
//                                  read serves all of them.
// In a step of both kinds of tokens each kernel takes its own tiles of eight neighbouring tokens (ag_dense).
//   score = (q . k) * scale;  keys lo..p with lo = first_visible(p, span): all, a window or a chunk
//
// Four options for mixers that are more than the plain softmax attention: values of another head
// size than the keys (dv); a sink, one learned number per head whose exponential joins the
// softmax denominator as one more term without a value (sinks[h], not scaled); an output gate,
// sigmoid(gate[t * gate_stride + h]) multiplied into the head's output (or, wide, one per value channel:
// sigmoid(gate[t * gate_stride + h * dv + c])); and a soft cap, score <- cap * tanh(score / cap).
#include <cooperative_groups.h>
#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

#define AG_WARPS 16
#define AG_MAX_D 256

// What both kernels do with a score, a strand's running sums and the strands of a (token, head): written with explicit
// roundings, so that the compiler has no choice of its own about fusing in either of them.
__device__ __forceinline__ float ag_score(float dot, float scale, float softcap) {
    const float s = __fmul_rn(dot, scale);
    return softcap > 0.f ? __fmul_rn(softcap, tanhf(__fdiv_rn(s, softcap))) : s;
}
// the strand's maximum and sum take in a block of scores (-inf: no key); returns the lane's weight, `corr` the factor on what was summed before
__device__ __forceinline__ float ag_take(float s, bool valid, float& m, float& l, float& corr) {
    const float m_new = fmaxf(m, warp_max(s));
    const float pe = valid ? expf(__fsub_rn(s, m_new)) : 0.f;
    corr = m == -INFINITY ? 0.f : expf(__fsub_rn(m, m_new));
    l = fmaf(l, corr, warp_sum(pe));
    m = m_new;
    return pe;
}
// the weights of the sixteen strands and 1 / (the denominator)
__device__ __forceinline__ float ag_merge(const float* m_s, const float* l_s, const float* sinks, int h, float* wgt) {
    float M = m_s[0], den = 0.f;
#pragma unroll
    for (int w = 1; w < AG_WARPS; w++) M = fmaxf(M, m_s[w]);
    if (sinks) {
        const float sk = sinks[h];
        M = fmaxf(M, sk);
        den = expf(__fsub_rn(sk, M));
    }
#pragma unroll
    for (int w = 0; w < AG_WARPS; w++) {
        wgt[w] = m_s[w] == -INFINITY ? 0.f : expf(__fsub_rn(m_s[w], M));
        den = fmaf(l_s[w], wgt[w], den);
    }
    return __fdiv_rn(1.0f, den);
}
__device__ __forceinline__ float ag_sigmoid(float g) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g))); }

struct AgArgs {
    const void *q, *kc, *vc;
    int q_stride;
    const int* block_table;
    int max_pages;
    const int *token_pos, *token_seq;
    void* out;
    int T, nh, nkv, d, page_size, span;
    float scale;
    int dv;
    const float *sinks, *gate;
    int gate_stride, gate_wide;
    float softcap;
    int mixed;          // the tile kernel takes the dense tiles of AG_TILE tokens alone, the other kernel the rest
};

#define AG_TILE 8
// Whether the tile of tokens t0 .. t0 + n - 1 is worth the tile kernel: it walks the keys once per sequence in the tile, for the
// price of about three tokens by themselves.  (512 prompt tokens beside 40 single tokens at 2,000 keys, 32 heads of 128 in
// float32: every token by itself 1,380 us, all by tiles 2,300, each kind its own way 850.)  ops::attention_generic_form counts with the same rule.
__device__ __forceinline__ bool ag_dense(const int* token_seq, int t0, int n) {
    int seqs = 1;
    for (int i = 1; i < n; i++) seqs += token_seq[t0 + i] != token_seq[t0 + i - 1];
    return 3 * seqs <= n;
}

// NV: value channels per lane (dv <= 32 NV).  G blocks of a cluster share a (token, head): each runs sixteen / G of its
// strands and leaves their sums in block 0's shared memory, which merges them.  A single token of a few heads is
// otherwise one block per head, and an SM takes in some 50 GB/s: 32 heads over 512 float32 keys took 40 us that way.
template <typename TA, int NV, int G>
__global__ void __launch_bounds__(AG_WARPS / G * 32) attention_generic_kernel(const AgArgs a) {
    pdl_grid_sync();
    extern __shared__ float smem[];
    float* qs = smem;                 // [d]
    float* acc_s = smem + a.d;        // [AG_WARPS][dv]
    __shared__ float m_s[AG_WARPS], l_s[AG_WARPS];

    const int d = a.d, dv = a.dv, page_size = a.page_size;
    const int t = blockIdx.x / G, h = blockIdx.y, part = blockIdx.x % G;
    if (G == 1 && a.mixed && ag_dense(a.token_seq, t / AG_TILE * AG_TILE, min(AG_TILE, a.T - t / AG_TILE * AG_TILE))) return;
    const int lane = threadIdx.x & 31, warp = part * (AG_WARPS / G) + (threadIdx.x >> 5);
    const int hk = h / (a.nh / a.nkv);
    const int p = a.token_pos[t];
    const int lo = first_visible(p, a.span);
    const int* bt = a.block_table + (size_t)a.token_seq[t] * a.max_pages;
    const TA *kc = (const TA*)a.kc, *vc = (const TA*)a.vc;

    const TA* qrow = (const TA*)a.q + (size_t)t * a.q_stride + (size_t)h * d;
    for (int c = threadIdx.x; c < d; c += blockDim.x) qs[c] = to_f32(qrow[c]);
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    float acc[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) acc[i] = 0.f;

    const bool vec = (d & 7) == 0;
    for (int kb = lo + warp * 32; kb <= p; kb += AG_WARPS * 32) {
        const int key = kb + lane;
        const bool valid = key <= p;
        float s = -INFINITY;
        long long off = 0;
        if (valid) {
            const int page = bt[key / page_size];
            off = ((long long)page * a.nkv + hk) * page_size + (key % page_size);      // in rows
            const TA* kr = kc + off * d;
            float dot = 0.f;
            if (vec) {
#pragma unroll 8
                for (int c = 0; c < d; c += 8) {
                    float f[8];
                    load8(kr + c, f);
#pragma unroll
                    for (int i = 0; i < 8; i++) dot = fmaf(qs[c + i], f[i], dot);
                }
            } else {
                for (int c = 0; c < d; c++) dot = fmaf(qs[c], to_f32(kr[c]), dot);
            }
            s = ag_score(dot, a.scale, a.softcap);
        }
        float corr;
        const float pe = ag_take(s, valid, m, l, corr);
#pragma unroll
        for (int i = 0; i < NV; i++) acc[i] = __fmul_rn(acc[i], corr);
        const int nk = (p - kb + 1 < 32) ? p - kb + 1 : 32;
#pragma unroll 8
        for (int j = 0; j < nk; j++) {
            const float pj = __shfl_sync(0xffffffffu, pe, j);
            const long long oj = __shfl_sync(0xffffffffu, off, j);
            const TA* vr = vc + oj * dv;
#pragma unroll
            for (int i = 0; i < NV; i++) {
                const int c = lane + 32 * i;
                if (c < dv) acc[i] = fmaf(pj, to_f32(vr[c]), acc[i]);
            }
        }
    }

    if (G > 1) {
        // the strands' sums go to block 0 (every block of the cluster has begun by then)
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        float *acc0 = cluster.map_shared_rank(acc_s, 0), *m0 = cluster.map_shared_rank(m_s, 0), *l0 = cluster.map_shared_rank(l_s, 0);
        if (lane == 0) {
            m0[warp] = m;
            l0[warp] = l;
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int c = lane + 32 * i;
            if (c < dv) acc0[warp * dv + c] = acc[i];
        }
        cluster.sync();
        if (part) return;
    } else {
        if (lane == 0) {
            m_s[warp] = m;
            l_s[warp] = l;
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int c = lane + 32 * i;
            if (c < dv) acc_s[warp * dv + c] = acc[i];
        }
        __syncthreads();
    }
    float wgt[AG_WARPS];
    float inv = ag_merge(m_s, l_s, a.sinks, h, wgt);
    if (a.gate && !a.gate_wide) inv = __fmul_rn(inv, ag_sigmoid(a.gate[(size_t)t * a.gate_stride + h]));
    TA* o = (TA*)a.out + ((size_t)t * a.nh + h) * dv;
    for (int c = threadIdx.x; c < dv; c += blockDim.x) {
        float num = 0.f;
#pragma unroll
        for (int w = 0; w < AG_WARPS; w++) num = fmaf(acc_s[w * dv + c], wgt[w], num);
        float r = __fmul_rn(num, inv);
        if (a.gate && a.gate_wide) r = __fmul_rn(r, ag_sigmoid(a.gate[(size_t)t * a.gate_stride + (size_t)h * dv + c]));
        o[c] = from_f32<TA>(r);
    }
}

// Eight tokens in turn and a head per block.  Tokens of one sequence that see from the same first key on (all of them without a
// window, those of a chunk with chunks) share the blocks of 32 keys, so a warp reads a key or value row once for
// all of them; a token's strand passes over blocks that lie behind it.  Eight warps run the sixteen strands.  Bound by the
// float32 multiply-adds (d + dv per key and token) and the shared-memory reads of q between them; a prompt of 512
// tokens and 32 heads of 128 in float32 took 1,140 us per layer with a block per (token, head), which read each key
// and value row from L2 once per token.
#define AG_TILE_WARPS 8
template <typename TA, int NV>
__global__ void __launch_bounds__(AG_TILE_WARPS * 32, 2) attention_generic_tile_kernel(const AgArgs a) {
    pdl_grid_sync();
    extern __shared__ __align__(16) float smem[];
    const int d = a.d, dv = a.dv, page_size = a.page_size;
    float* qs = smem;                                 // [AG_TILE][d]
    float* acc_s = qs + AG_TILE * d;                  // [AG_TILE][AG_WARPS][dv]
    __shared__ float m_s[AG_TILE][AG_WARPS], l_s[AG_TILE][AG_WARPS], w_s[AG_TILE][AG_WARPS], inv_s[AG_TILE];
    __shared__ int pos_s[AG_TILE], seq_s[AG_TILE];
    const int t0 = blockIdx.x * AG_TILE, h = blockIdx.y, n = a.T - t0 < AG_TILE ? a.T - t0 : AG_TILE;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int hk = h / (a.nh / a.nkv);
    const TA *kc = (const TA*)a.kc, *vc = (const TA*)a.vc;
    if (threadIdx.x < AG_TILE) {
        pos_s[threadIdx.x] = (int)threadIdx.x < n ? a.token_pos[t0 + threadIdx.x] : 0;
        seq_s[threadIdx.x] = (int)threadIdx.x < n ? a.token_seq[t0 + threadIdx.x] : -1;
    }
    if (a.mixed && !ag_dense(a.token_seq, t0, n)) return;
    __syncthreads();
    for (int f = 0, e; f < n; f = e) {                // tokens f .. e - 1 share their keys
        const int lo = first_visible(pos_s[f], a.span), seq = seq_s[f];
        for (e = f + 1; e < n && seq_s[e] == seq && pos_s[e] == pos_s[e - 1] + 1 && first_visible(pos_s[e], a.span) == lo; e++) {}
        const int p0 = pos_s[f], p_last = pos_s[e - 1], cnt = e - f;
        const int* bt = a.block_table + (size_t)seq * a.max_pages;
        for (int idx = threadIdx.x; idx < AG_TILE * d; idx += blockDim.x) {
            const int i = idx / d, c = idx - i * d;
            qs[idx] = i < cnt ? to_f32(((const TA*)a.q)[(size_t)(t0 + f + i) * a.q_stride + (size_t)h * d + c]) : 0.f;
        }
        __syncthreads();
        for (int strand = warp; strand < AG_WARPS; strand += AG_TILE_WARPS) {
            float m[AG_TILE], l[AG_TILE], acc[AG_TILE][NV];
#pragma unroll
            for (int i = 0; i < AG_TILE; i++) {
                m[i] = -INFINITY;
                l[i] = 0.f;
#pragma unroll
                for (int c = 0; c < NV; c++) acc[i][c] = 0.f;
            }
            for (int kb = lo + strand * 32; kb <= p_last; kb += AG_WARPS * 32) {
                const int key = kb + lane;
                long long off = 0;
                float s[AG_TILE];
#pragma unroll
                for (int i = 0; i < AG_TILE; i++) s[i] = 0.f;
                if (key <= p_last) {
                    off = ((long long)bt[key / page_size] * a.nkv + hk) * page_size + (key % page_size);
                    const TA* kr = kc + off * d;
#pragma unroll 2
                    for (int c = 0; c < d; c += 8) {
                        float k8[8];
                        load8(kr + c, k8);
#pragma unroll
                        for (int i = 0; i < AG_TILE; i++) {
                            const float4 qa = *reinterpret_cast<const float4*>(qs + i * d + c), qb = *reinterpret_cast<const float4*>(qs + i * d + c + 4);
                            s[i] = fmaf(qa.x, k8[0], s[i]), s[i] = fmaf(qa.y, k8[1], s[i]), s[i] = fmaf(qa.z, k8[2], s[i]), s[i] = fmaf(qa.w, k8[3], s[i]);
                            s[i] = fmaf(qb.x, k8[4], s[i]), s[i] = fmaf(qb.y, k8[5], s[i]), s[i] = fmaf(qb.z, k8[6], s[i]), s[i] = fmaf(qb.w, k8[7], s[i]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < AG_TILE; i++) {
                    if (i >= cnt || kb > p0 + i) {    // the block lies behind the token (uniform over the warp)
                        s[i] = 0.f;
                        continue;
                    }
                    const bool valid = key <= p0 + i;
                    float corr;
                    s[i] = ag_take(valid ? ag_score(s[i], a.scale, a.softcap) : -INFINITY, valid, m[i], l[i], corr);
#pragma unroll
                    for (int c = 0; c < NV; c++) acc[i][c] = __fmul_rn(acc[i][c], corr);
                }
                // value rows; a token takes in those up to its own place and leaves its sums alone behind it (a row that
                // is not the token's may hold anything)
                const int nk = p_last - kb + 1 < 32 ? p_last - kb + 1 : 32;
                const bool all = cnt == AG_TILE && kb + 31 <= p0;
                auto values = [&](int j, auto every) {
                    const TA* vr = vc + __shfl_sync(0xffffffffu, off, j) * dv;
                    float v[NV];
#pragma unroll
                    for (int c = 0; c < NV; c++) v[c] = lane + 32 * c < dv ? to_f32(vr[lane + 32 * c]) : 0.f;
#pragma unroll
                    for (int i = 0; i < AG_TILE; i++) {
                        const float pj = __shfl_sync(0xffffffffu, s[i], j);
                        if (decltype(every)::value || (i < cnt && kb + j <= p0 + i)) {
#pragma unroll
                            for (int c = 0; c < NV; c++) acc[i][c] = fmaf(pj, v[c], acc[i][c]);
                        }
                    }
                };
                if (all) {
#pragma unroll 4
                    for (int j = 0; j < 32; j++) values(j, std::true_type());
                } else {
                    for (int j = 0; j < nk; j++) values(j, std::false_type());
                }
            }
#pragma unroll
            for (int i = 0; i < AG_TILE; i++) {
                if (lane == 0) {
                    m_s[i][strand] = m[i];
                    l_s[i][strand] = l[i];
                }
#pragma unroll
                for (int c = 0; c < NV; c++)
                    if (lane + 32 * c < dv) acc_s[(i * AG_WARPS + strand) * dv + lane + 32 * c] = acc[i][c];
            }
        }
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int i = threadIdx.x;
            float wgt[AG_WARPS];
            float inv = ag_merge(m_s[i], l_s[i], a.sinks, h, wgt);
            if (a.gate && !a.gate_wide) inv = __fmul_rn(inv, ag_sigmoid(a.gate[(size_t)(t0 + f + i) * a.gate_stride + h]));
            inv_s[i] = inv;
#pragma unroll
            for (int w = 0; w < AG_WARPS; w++) w_s[i][w] = wgt[w];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < cnt * dv; idx += blockDim.x) {
            const int i = idx / dv, c = idx - i * dv;
            const size_t t = (size_t)t0 + f + i;
            float num = 0.f;
#pragma unroll
            for (int w = 0; w < AG_WARPS; w++) num = fmaf(acc_s[(i * AG_WARPS + w) * dv + c], w_s[i][w], num);
            float r = __fmul_rn(num, inv_s[i]);
            if (a.gate && a.gate_wide) r = __fmul_rn(r, ag_sigmoid(a.gate[t * a.gate_stride + (size_t)h * dv + c]));
            ((TA*)a.out)[(t * a.nh + h) * dv + c] = from_f32<TA>(r);
        }
        __syncthreads();
    }
}

template <typename TA, int NV, int G>
static int ag_launch(const AgArgs& a, cudaStream_t s) {
    const size_t smem = ((size_t)a.d + (size_t)AG_WARPS * a.dv) * sizeof(float);
    return illm_launch_cluster(attention_generic_kernel<TA, NV, G>, dim3((unsigned)a.T * G, a.nh), dim3(AG_WARPS / G * 32), G, smem, s, a);
}

template <typename TA, int NV>
static int ag_launch_for(AgArgs a, int prompts, cudaStream_t s) {
    // Tokens of prompts share key blocks unless every token's window begins somewhere else.
    a.mixed = 0;
    if (NV == 4 && prompts && a.span <= 0 && a.d <= 128 && a.d % 8 == 0) {
        a.mixed = prompts == 2;
        const size_t smem = (size_t)AG_TILE * ((size_t)a.d + (size_t)AG_WARPS * a.dv) * sizeof(float);
        auto kern = attention_generic_tile_kernel<TA, 4>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        illm_launch(kern, dim3((a.T + AG_TILE - 1) / AG_TILE, a.nh), dim3(AG_TILE_WARPS * 32), smem, s, a);
        return a.mixed ? ag_launch<TA, NV, 1>(a, s) : illm_launch_status();
    }
    // as many blocks per (token, head) as leave every SM at most about two
    const long long pairs = (long long)a.T * a.nh, sms = illm_sm_count();
    if (pairs <= sms / 4) return ag_launch<TA, NV, 8>(a, s);
    if (pairs <= sms / 2) return ag_launch<TA, NV, 4>(a, s);
    if (pairs <= sms) return ag_launch<TA, NV, 2>(a, s);
    return ag_launch<TA, NV, 1>(a, s);
}

// span: see first_visible; gate_wide: a gate per value channel; softcap 0: none; prompts: 0 every token by itself, 1 tokens by
// eights, 2 by eights where eight neighbours are worth it (which kernel runs follows from it; the results do not)
extern "C" int illm_attention_generic_ex(const void* q, int q_stride, const void* kc, const void* vc,
                                         const int* block_table, int max_pages, const int* token_pos,
                                         const int* token_seq, void* out, int act_dtype, int T, int nh,
                                         int nkv, int d, int page_size, int span, float scale,
                                         int dv, const float* sinks, const float* gate, int gate_stride,
                                         int gate_wide, float softcap, int prompts, void* stream) {
    if (T <= 0) return 0;
    if (dv <= 0) dv = d;
    if (d <= 0 || d > AG_MAX_D || dv > AG_MAX_D || nkv <= 0 || nh % nkv || nh > 65535) return ILLM_ERR_BAD_ARG;
    const AgArgs a{q, kc, vc, q_stride, block_table, max_pages, token_pos, token_seq, out, T, nh, nkv, d, page_size, span, scale, dv, sinks, gate,
                   gate_stride, gate_wide, softcap, 0};
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == ILLM_BF16) return dv <= 128 ? ag_launch_for<bf16, 4>(a, prompts, s) : ag_launch_for<bf16, 8>(a, prompts, s);
    if (act_dtype == ILLM_F32) return dv <= 128 ? ag_launch_for<float, 4>(a, prompts, s) : ag_launch_for<float, 8>(a, prompts, s);
    return ILLM_ERR_BAD_ARG;
}

extern "C" int illm_attention_generic(const void* q, int q_stride, const void* kc, const void* vc, const int* block_table, int max_pages,
                                      const int* token_pos, const int* token_seq, void* out, int act_dtype, int T, int nh, int nkv, int d,
                                      int page_size, int window, float scale, int dv, const float* sinks, const float* gate, int gate_stride,
                                      void* stream) {
    return illm_attention_generic_ex(q, q_stride, kc, vc, block_table, max_pages, token_pos, token_seq, out, act_dtype, T, nh, nkv, d, page_size,
                                     window, scale, dv, sinks, gate, gate_stride, 0, 0.f, 0, stream);
}
