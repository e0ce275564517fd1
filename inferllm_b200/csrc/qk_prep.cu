// What happens to the packed projection [T, ld] (float32, or the activation dtype) of an attention layer between the matrix
// product and the attention kernel, for mixers that do more there than rotate (rope_kv.cu):
//
//   q = x[q_off : q_off + nh d] + bq;   k = x[k_off : ...] + bk;   v = x[v_off : ...] + bv     (biases optional)
//   q = q / sqrt(mean(q^2) + eps) * wq,  the mean over the WHOLE projection of the token, all heads
//       together; likewise k with wk                                                            (optional)
//   or: every head of q is normed by itself, q_h / sqrt(mean(q_h^2) + eps) * wq with wq of one head's size; likewise k
//   the first `rot` channels of every q and k head are rotated by the token's position, either in the
//       interleaved layout (channel 2j with 2j + 1) or the rotate-half one (j with j + rot / 2), with
//       (cos, sin) from a float32 table [positions, rot / 2, 2] that may carry a magnitude factor
//   q goes to q_out [T, nh d] in the activation dtype; k and v go into the token's place in the pages
//       (k: [pages, nkv, page_size, d], v: [pages, nkv, page_size, dv]) if there are pages to write.
//
// Values may be mixed with another layer's values of the same tokens, v <- (1 - lambda) v + lambda v_first (v_first
// float32 rows, lambda one number on the device), and a layer's own, unmixed values may be kept for later layers (v_keep).
//
// A layer that attends to another layer's keys and values passes k_off < 0: only q is made.  A layer whose keys are
// also its values passes v_off < 0: k alone is stored.
// Everything is float32 until the stores.  One block per token; the sums have a fixed order.
#include "row_ops.cuh"

struct QkPrepArgs {
    const void* x;
    int ld, q_off, k_off, v_off;
    int nh, nkv, d, dv;
    const float *bq, *bk, *bv, *wq, *wk;
    float eps;
    const float* cos_sin;
    int rot, pairs, n_pos;
    const int *token_pos, *token_seq, *block_table;
    int max_pages, page_size;
    void *q_out, *kc, *vc;
    int* err;
    float qt_coef;      // query temperature: q *= 1 + qt_coef * ln((p + 1) / qt_every + 1), the division whole-numbered
    int qt_every;       // 0: none
    const float* v_first;       // [T, v_first_ld] or nullptr
    int v_first_ld;
    const float* v_lambda;
    float* v_keep;              // [T, nkv dv] or nullptr
    int head_norm;              // wq, wk: of one head's size, every head normed by itself
};

__device__ __forceinline__ float rotated(const float* buf, int e, int rot, int pairs, const float* cs) {
    // buf: one head; e < rot: the channel asked for
    int j, partner;
    bool first;
    if (pairs) {
        j = e >> 1;
        first = !(e & 1);
        partner = e ^ 1;
    } else {
        const int half = rot >> 1;
        first = e < half;
        j = first ? e : e - half;
        partner = first ? e + half : e - half;
    }
    const float c = cs[2 * j], s = cs[2 * j + 1];
    const float a = buf[e], b = buf[partner];
    return fmaf(a, c, first ? -__fmul_rn(b, s) : __fmul_rn(b, s));       // explicit: the same bits in every kernel of this file
}

__device__ __forceinline__ float mixed(float own, float first, float lambda) { return fmaf(1.0f - lambda, own, __fmul_rn(lambda, first)); }

template <typename TI, typename TA>
__global__ void __launch_bounds__(256) qk_prep_kernel(QkPrepArgs a) {
    pdl_grid_sync();
    extern __shared__ float buf[];      // [nh d] q, then [nkv d] k
    __shared__ float scratch[32];
    const int t = blockIdx.x;
    const int nq = a.nh * a.d, nk = a.k_off >= 0 ? a.nkv * a.d : 0;
    const TI* x = (const TI*)a.x + (size_t)t * a.ld;
    int p = a.token_pos[t];
    if (a.rot && (p < 0 || p >= a.n_pos)) {
        if (threadIdx.x == 0) atomicExch(a.err, 3);
        p = 0;
    }
    float ssq = 0.f, ssk = 0.f;
    const float q_temp = a.qt_every > 0 ? 1.0f + a.qt_coef * logf((float)((a.token_pos[t] + 1) / a.qt_every + 1)) : 1.0f;
    for (int c = threadIdx.x; c < nq; c += blockDim.x) {
        float v = to_f32(x[a.q_off + c]);
        if (a.bq) v += a.bq[c];
        if (a.qt_every > 0) v *= q_temp;
        buf[c] = v;
        ssq += v * v;
    }
    for (int c = threadIdx.x; c < nk; c += blockDim.x) {
        float v = to_f32(x[a.k_off + c]);
        if (a.bk) v += a.bk[c];
        buf[nq + c] = v;
        ssk += v * v;
    }
    if (a.head_norm) {
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, heads = a.nh + (nk ? a.nkv : 0);
        for (int hd = warp; hd < heads; hd += 8) {          // a warp per head, the sum in the order of the lanes' channels
            float* row = buf + (size_t)hd * a.d;
            const float* w = hd < a.nh ? a.wq : a.wk;
            float ss = 0.f;
            for (int c = lane; c < a.d; c += 32) ss = fmaf(row[c], row[c], ss);
            const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)a.d + a.eps);
            for (int c = lane; c < a.d; c += 32) row[c] = (row[c] * inv) * w[c];
        }
    }
    if (a.wq && !a.head_norm) {
        ssq = block_sum(ssq, scratch);
        const float inv = 1.0f / sqrtf(ssq / (float)nq + a.eps);
        for (int c = threadIdx.x; c < nq; c += blockDim.x) buf[c] = (buf[c] * inv) * a.wq[c];
    }
    if (a.wk && nk && !a.head_norm) {
        ssk = block_sum(ssk, scratch);
        const float inv = 1.0f / sqrtf(ssk / (float)nk + a.eps);
        for (int c = threadIdx.x; c < nk; c += blockDim.x) buf[nq + c] = (buf[nq + c] * inv) * a.wk[c];
    }
    __syncthreads();
    const float* cs = a.rot ? a.cos_sin + (size_t)p * a.rot : nullptr;      // rot / 2 pairs of (cos, sin)
    TA* qo = (TA*)a.q_out + (size_t)t * nq;
    for (int c = threadIdx.x; c < nq; c += blockDim.x) {
        const int e = c % a.d;
        qo[c] = from_f32<TA>(e < a.rot ? rotated(buf + (c - e), e, a.rot, a.pairs, cs) : buf[c]);
    }
    if (nk == 0 || a.kc == nullptr) return;
    const int pos = a.token_pos[t];
    const int page = a.block_table[(size_t)a.token_seq[t] * a.max_pages + pos / a.page_size];
    if (page < 0) {
        if (threadIdx.x == 0) atomicExch(a.err, 2);
        return;
    }
    const int slot = pos % a.page_size;
    for (int c = threadIdx.x; c < nk; c += blockDim.x) {
        const int hk = c / a.d, e = c - hk * a.d;
        const float v = e < a.rot ? rotated(buf + nq + (c - e), e, a.rot, a.pairs, cs) : buf[nq + c];
        ((TA*)a.kc)[(((size_t)page * a.nkv + hk) * a.page_size + slot) * a.d + e] = from_f32<TA>(v);
    }
    if (a.v_off < 0) return;        // the keys are also the values: nothing else to store
    const int nv = a.nkv * a.dv;
    const float lambda = a.v_first ? *a.v_lambda : 0.f;
    for (int c = threadIdx.x; c < nv; c += blockDim.x) {
        const int hk = c / a.dv, e = c - hk * a.dv;
        float v = to_f32(x[a.v_off + c]);
        if (a.bv) v += a.bv[c];
        if (a.v_keep) a.v_keep[(size_t)t * nv + c] = v;
        if (a.v_first) v = mixed(v, a.v_first[(size_t)t * a.v_first_ld + c], lambda);
        ((TA*)a.vc)[(((size_t)page * a.nkv + hk) * a.page_size + slot) * a.dv + e] = from_f32<TA>(v);
    }
}

// The same for rows of whole 16-byte pieces (sizes, offsets and strides of four channels): a thread holds IT pieces of four
// neighbouring channels of q, k and v in registers.  All its loads, the weights, biases, the value to mix in and the page's
// number among them, are on their way before the first sum, because a single token's block is bound by nothing but the
// latency of its dependent loads: the kernel above, which walks the channels one by one in five passes over shared memory,
// took 13 to 17 us for one token of 32 + 2 x 8 heads of 128.  A head's norm is added within the d / 4 lanes that hold the head (d / 4 a power
// of two up to 32).  Only the rotate-half layout, whose channels pair up across threads, goes through shared memory.
// The block size follows from the sizes alone, so that a row's sums have one order in every step.
// EARLY false: the same sums in the same order with the weights, biases and values to mix in read where they are used, so that two
// blocks lie on an SM, for steps of more tokens than SMs (2,000 tokens of 32 + 2 x 8 heads of 128, norms over all heads, rotate-half: 68 us,
// so 47).  Four pieces a thread leave no registers for early reads at any number of tokens.
template <typename TI, typename TA, int IT, bool EARLY>
__global__ void __launch_bounds__(1024, EARLY || IT > 2 ? 1 : 2) qk_prep_vec_kernel(const QkPrepArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(16) float buf[];      // the rotate-half layout: [nh d] q, then [nkv d] k
    __shared__ float scratch[32];
    const int t = blockIdx.x, threads = blockDim.x, d4 = a.d >> 2;
    const int nq4 = a.nh * d4, nk4 = a.k_off >= 0 ? a.nkv * d4 : 0, nv4 = nk4 && a.v_off >= 0 && a.kc ? a.nkv * (a.dv >> 2) : 0;
    const bool whole = a.wq && !a.head_norm, halves = a.rot && !a.pairs;
    // weights, biases and the indices of the step are no result of the kernel before
    const int pos = a.token_pos[t];
    auto weight = [&](int at) {
        const bool is_q = at < nq4, is_k = !is_q && at < nq4 + nk4;
        const float* wp = is_q ? a.wq : is_k ? a.wk : nullptr;
        const int c = is_q ? at : at - nq4;
        return wp ? row_load4(wp + 4 * (a.head_norm ? c % d4 : c)) : make_float4(1.f, 1.f, 1.f, 1.f);
    };
    auto bias_of = [&](int at) {
        const bool is_q = at < nq4, is_k = !is_q && at < nq4 + nk4;
        const float* bp = is_q ? a.bq : is_k ? a.bk : a.bv;
        return bp && at < nq4 + nk4 + nv4 ? row_load4(bp + 4 * (is_q ? at : is_k ? at - nq4 : at - nq4 - nk4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float4 w[IT], bias[IT];
    if (EARLY) {
#pragma unroll
        for (int i = 0; i < IT; i++) w[i] = weight(threadIdx.x + i * threads), bias[i] = bias_of(threadIdx.x + i * threads);
    }
    const int page = nk4 && a.kc ? a.block_table[(size_t)a.token_seq[t] * a.max_pages + pos / a.page_size] : -1;
    int p = pos;
    if (a.rot && (p < 0 || p >= a.n_pos)) {
        if (threadIdx.x == 0) atomicExch(a.err, 3);
        p = 0;
    }
    const float* cs = a.rot ? a.cos_sin + (size_t)p * a.rot : nullptr;      // rot / 2 pairs of (cos, sin)
    const float q_temp = a.qt_every > 0 ? 1.0f + a.qt_coef * logf((float)((pos + 1) / a.qt_every + 1)) : 1.0f;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const TI* x = (const TI*)a.x + (size_t)t * a.ld;
    const float lambda = a.v_first ? *a.v_lambda : 0.f;
    float4 v[IT], first[IT];
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int at = threadIdx.x + i * threads;
        const bool is_q = at < nq4, is_k = !is_q && at < nq4 + nk4, is_v = !is_q && !is_k && at < nq4 + nk4 + nv4;
        const int c = is_q ? at : is_k ? at - nq4 : at - nq4 - nk4, off = is_q ? a.q_off : is_k ? a.k_off : a.v_off;
        v[i] = is_q || is_k || is_v ? row_load4(x + off + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (EARLY) first[i] = is_v && a.v_first ? row_load4(a.v_first + (size_t)t * a.v_first_ld + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float ssq = 0.f, ssk = 0.f;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int at = threadIdx.x + i * threads;
        if (!EARLY) bias[i] = bias_of(at);
        v[i].x += bias[i].x, v[i].y += bias[i].y, v[i].z += bias[i].z, v[i].w += bias[i].w;
        if (at < nq4 && a.qt_every > 0) v[i].x *= q_temp, v[i].y *= q_temp, v[i].z *= q_temp, v[i].w *= q_temp;
        float s = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, v[i].w * v[i].w)));
        if (a.head_norm) {          // every head by itself; the lanes beyond k add among themselves what nobody uses
            for (int o = 1; o < d4; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (at < nq4 + nk4) {
                const float inv = 1.0f / sqrtf(s / (float)a.d + a.eps);
                if (!EARLY) w[i] = weight(at);
                v[i].x = (v[i].x * inv) * w[i].x, v[i].y = (v[i].y * inv) * w[i].y, v[i].z = (v[i].z * inv) * w[i].z, v[i].w = (v[i].w * inv) * w[i].w;
            }
        }
        if (at < nq4) ssq += s;
        else if (at < nq4 + nk4) ssk += s;
    }
    if (whole) {
        ssq = block_sum(ssq, scratch);
        if (nk4 && a.wk) ssk = block_sum(ssk, scratch);
        const float inv_q = 1.0f / sqrtf(ssq / (float)(4 * nq4) + a.eps), inv_k = nk4 ? 1.0f / sqrtf(ssk / (float)(4 * nk4) + a.eps) : 0.f;
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int at = threadIdx.x + i * threads;
            if (at >= nq4 && (at >= nq4 + nk4 || !a.wk)) continue;
            const float inv = at < nq4 ? inv_q : inv_k;
            if (!EARLY) w[i] = weight(at);
            v[i].x = (v[i].x * inv) * w[i].x, v[i].y = (v[i].y * inv) * w[i].y, v[i].z = (v[i].z * inv) * w[i].z, v[i].w = (v[i].w * inv) * w[i].w;
        }
    }
    if (halves) {
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int at = threadIdx.x + i * threads;
            if (at < nq4 + nk4) *reinterpret_cast<float4*>(buf + 4 * at) = v[i];
        }
        __syncthreads();
    }
    if (page < 0 && nk4 && a.kc && threadIdx.x == 0) atomicExch(a.err, 2);
    auto turn = [](float x, float c, float y, float s) { return fmaf(x, c, __fmul_rn(y, s)); };
    auto mix = [&](float x, float y) { return mixed(x, y, lambda); };
    const int slot = pos % a.page_size;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int at = threadIdx.x + i * threads;
        if (at >= nq4 + nk4 + nv4) continue;
        if (at < nq4 + nk4) {
            const int c = at < nq4 ? at : at - nq4, hd = c / d4, e = (c - hd * d4) * 4;
            if (e < a.rot) {
                if (a.pairs) {
                    const float4 f = *reinterpret_cast<const float4*>(cs + e);      // cos, sin of the two pairs
                    v[i] = make_float4(turn(v[i].x, f.x, -v[i].y, f.y), turn(v[i].y, f.x, v[i].x, f.y), turn(v[i].z, f.z, -v[i].w, f.w), turn(v[i].w, f.z, v[i].z, f.w));
                } else {
                    const float* head = buf + 4 * (at - (c - hd * d4));
                    v[i].x = rotated(head, e, a.rot, 0, cs);
                    if (e + 1 < a.rot) v[i].y = rotated(head, e + 1, a.rot, 0, cs);
                    if (e + 2 < a.rot) v[i].z = rotated(head, e + 2, a.rot, 0, cs);
                    if (e + 3 < a.rot) v[i].w = rotated(head, e + 3, a.rot, 0, cs);
                }
            }
            if (at < nq4) row_store4((TA*)a.q_out + (size_t)t * 4 * nq4 + 4 * c, v[i]);
            else if (a.kc && page >= 0) row_store4((TA*)a.kc + (((size_t)page * a.nkv + hd) * a.page_size + slot) * a.d + e, v[i]);
        } else if (page >= 0) {
            const int c = at - nq4 - nk4, hd = c / (a.dv >> 2), e = (c - hd * (a.dv >> 2)) * 4;
            if (a.v_keep) *reinterpret_cast<float4*>(a.v_keep + (size_t)t * 4 * nv4 + 4 * c) = v[i];
            if (!EARLY && a.v_first) first[i] = row_load4(a.v_first + (size_t)t * a.v_first_ld + 4 * c);
            if (a.v_first)
                v[i] = make_float4(mix(v[i].x, first[i].x), mix(v[i].y, first[i].y), mix(v[i].z, first[i].z), mix(v[i].w, first[i].w));
            row_store4((TA*)a.vc + (((size_t)page * a.nkv + hd) * a.page_size + slot) * a.dv + e, v[i]);
        }
    }
}

// Whether the rows are whole 16-byte pieces throughout, and the norm of a head lies within a warp.
static bool qk_prep_vec_takes(const QkPrepArgs& a) {
    if ((a.d | a.dv | a.ld | a.q_off) & 3) return false;
    if (a.k_off >= 0 && (a.k_off & 3)) return false;
    if (a.v_off >= 0 && (a.v_off & 3)) return false;
    if (a.pairs && (a.rot & 3)) return false;
    if (row_odd(a.x) || row_odd(a.q_out) || row_odd(a.kc) || row_odd(a.vc) || row_odd(a.bq) || row_odd(a.bk) || row_odd(a.bv) || row_odd(a.wq) || row_odd(a.wk) || row_odd(a.cos_sin) ||
        row_odd(a.v_keep) || row_odd(a.v_first) || (a.v_first && (a.v_first_ld & 3)))
        return false;
    if (a.wk && !a.wq) return false;
    if (a.head_norm && (a.d / 4 > 32 || (a.d / 4 & (a.d / 4 - 1)))) return false;
    return true;
}

template <typename TI, typename TA>
static int qk_prep_vec_launch(const QkPrepArgs& a, int T, cudaStream_t s) {
    const int pieces = (a.nh * a.d + (a.k_off >= 0 ? a.nkv * (a.d + (a.v_off >= 0 ? a.dv : 0)) : 0)) / 4;
    const int iters = pieces <= 1024 ? 1 : pieces <= 2048 ? 2 : pieces <= 4096 ? 4 : 0;
    if (!iters) return -1;
    const int threads = ((pieces + iters - 1) / iters + 31) / 32 * 32;
    const size_t smem = a.rot && !a.pairs ? (size_t)(a.nh + (a.k_off >= 0 ? a.nkv : 0)) * a.d * sizeof(float) : 0;
    if (smem > 200 * 1024) return -1;
#define ILLM_QKV(IT)                                                                                                                          \
    do {                                                                                                                                      \
        auto kern = T <= illm_sm_count() ? qk_prep_vec_kernel<TI, TA, IT, IT <= 2> : qk_prep_vec_kernel<TI, TA, IT, false>;                    \
        if (smem > 47 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                              \
        illm_launch(kern, dim3(T), dim3(threads), smem, s, a);                                                                                 \
    } while (0)
    if (iters == 1) ILLM_QKV(1);
    else if (iters == 2) ILLM_QKV(2);
    else ILLM_QKV(4);
#undef ILLM_QKV
    return illm_launch_status();
}

// the same with a temperature on the queries that grows with the position (qt_every 0: none), applied behind the bias
extern "C" int illm_qk_prep_ex(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                               const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                               int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                               int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                               void* stream);
// the same with mixed values (v_first nullptr: none) and the layer's own values kept (v_keep nullptr: not)
extern "C" int illm_qk_prep_mix(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                                const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                                int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                                int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                                const float* v_first, int v_first_ld, const float* v_lambda, float* v_keep, void* stream);
// the same with norms per head (head_norm != 0: wq and wk have one head's size)
extern "C" int illm_qk_prep_heads(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                                  const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                                  int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                                  int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                                  const float* v_first, int v_first_ld, const float* v_lambda, float* v_keep, int head_norm, void* stream);
extern "C" int illm_qk_prep(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                            const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                            int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                            int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, void* stream) {
    return illm_qk_prep_ex(x, x_dtype, ld, q_off, k_off, v_off, nh, nkv, d, dv, bq, bk, bv, wq, wk, eps, cos_sin, rot, pairs, n_pos, token_pos, token_seq,
                           block_table, max_pages, page_size, q_out, kc, vc, act_dtype, T, err, 0.f, 0, stream);
}
extern "C" int illm_qk_prep_ex(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                               const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                               int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                               int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                               void* stream) {
    return illm_qk_prep_mix(x, x_dtype, ld, q_off, k_off, v_off, nh, nkv, d, dv, bq, bk, bv, wq, wk, eps, cos_sin, rot, pairs, n_pos, token_pos, token_seq,
                            block_table, max_pages, page_size, q_out, kc, vc, act_dtype, T, err, qt_coef, qt_every, nullptr, 0, nullptr, nullptr, stream);
}
extern "C" int illm_qk_prep_mix(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                                const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                                int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                                int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                                const float* v_first, int v_first_ld, const float* v_lambda, float* v_keep, void* stream) {
    return illm_qk_prep_heads(x, x_dtype, ld, q_off, k_off, v_off, nh, nkv, d, dv, bq, bk, bv, wq, wk, eps, cos_sin, rot, pairs, n_pos, token_pos, token_seq,
                              block_table, max_pages, page_size, q_out, kc, vc, act_dtype, T, err, qt_coef, qt_every, v_first, v_first_ld, v_lambda, v_keep, 0,
                              stream);
}
extern "C" int illm_qk_prep_heads(const void* x, int x_dtype, int ld, int q_off, int k_off, int v_off, int nh, int nkv, int d, int dv, const float* bq,
                                  const float* bk, const float* bv, const float* wq, const float* wk, float eps, const float* cos_sin, int rot,
                                  int pairs, int n_pos, const int* token_pos, const int* token_seq, const int* block_table, int max_pages,
                                  int page_size, void* q_out, void* kc, void* vc, int act_dtype, int T, int* err, float qt_coef, int qt_every,
                                  const float* v_first, int v_first_ld, const float* v_lambda, float* v_keep, int head_norm, void* stream) {
    if (T <= 0) return 0;
    if (head_norm && (!wq || (k_off >= 0 && !wk))) return ILLM_ERR_BAD_ARG;
    if (qt_every < 0 || (v_first && (!v_lambda || v_first_ld < nkv * dv)) || ((v_first || v_keep) && (k_off < 0 || v_off < 0 || !vc))) return ILLM_ERR_BAD_ARG;
    if (nh <= 0 || d <= 0 || rot < 0 || rot > d || (rot & 1) || (rot && !cos_sin) || !x || !q_out) return ILLM_ERR_BAD_ARG;
    if (k_off >= 0 && (nkv <= 0 || dv <= 0)) return ILLM_ERR_BAD_ARG;      // v_off < 0 with k_off >= 0: keys alone are stored
    QkPrepArgs a{x, ld, q_off, k_off, v_off, nh, nkv, d, dv, bq, bk, bv, wq, wk, eps, cos_sin, rot, pairs, n_pos,
                 token_pos, token_seq, block_table, max_pages, page_size, q_out, kc, vc, err, qt_coef, qt_every,
                 v_first, v_first_ld, v_lambda, v_keep, head_norm};
    const size_t smem = (size_t)(nh * d + (k_off >= 0 ? nkv * d : 0)) * sizeof(float);
    if (smem > 200 * 1024) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (qk_prep_vec_takes(a)) {
        int rc = -1;
        if (x_dtype == ILLM_F32 && act_dtype == ILLM_BF16) rc = qk_prep_vec_launch<float, bf16>(a, T, s);
        else if (x_dtype == ILLM_F32 && act_dtype == ILLM_F32) rc = qk_prep_vec_launch<float, float>(a, T, s);
        else if (x_dtype == ILLM_BF16 && act_dtype == ILLM_BF16) rc = qk_prep_vec_launch<bf16, bf16>(a, T, s);
        if (rc >= 0) return rc;
    }
#define ILLM_QKP(TI, TA)                                                                                                    \
    do {                                                                                                                    \
        if (smem > 47 * 1024) cudaFuncSetAttribute(qk_prep_kernel<TI, TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        illm_launch(qk_prep_kernel<TI, TA>, dim3(T), dim3(256), smem, s, a);                                                \
    } while (0)
    if (x_dtype == ILLM_F32 && act_dtype == ILLM_BF16) ILLM_QKP(float, bf16);
    else if (x_dtype == ILLM_F32 && act_dtype == ILLM_F32) ILLM_QKP(float, float);
    else if (x_dtype == ILLM_BF16 && act_dtype == ILLM_BF16) ILLM_QKP(bf16, bf16);
    else return ILLM_ERR_BAD_ARG;
#undef ILLM_QKP
    return illm_launch_status();
}
