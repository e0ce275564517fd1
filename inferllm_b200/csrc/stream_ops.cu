// Small element-wise kernels between matrix products.
//
// gated_act:    out[t, i] = act(gu[t, 2i]) * gu[t, 2i + 1]  for the activations that the fused silu kernels do not
//               cover (act 1: silu, 2: relu, 3: tanh-form gelu, 4: clamped, g = min(gate, limit), u = clamp(up, -limit,
//               limit), g sigmoid(1.702 g) (u + 1)); the packed projection holds gate and up of an
//               output next to each other, as in swiglu.cu.
// take_columns: y[t, :] = x[t, off : off + n] of a float32 matrix with row stride ld, as a contiguous matrix of
//               the activation dtype (what a second, low-rank product reads).
// join_rows:    y[t, :] = [a[t, :], b[t, :]] of two float32 matrices of equal width, in the activation dtype.
// soft_cap:     x = cap * tanh(x / cap), in place, of a float32 array (a head's logits).
#include "row_ops.cuh"

__device__ __forceinline__ float gate_act_of(float v, int act) {
    if (act == 1) return v / (1.0f + expf(-v));
    if (act == 2) return fmaxf(v, 0.f);
    if (act == 3) return 0.5f * v * (1.0f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
    return v;
}

template <typename TA>
__global__ void gated_act_kernel(const TA* __restrict__ gu, TA* __restrict__ out, int I, long long n, int act, float limit) {
    pdl_grid_sync();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long t = i / I;
    const int c = (int)(i - t * I);
    const float g = to_f32(gu[t * 2 * I + 2 * c]), u = to_f32(gu[t * 2 * I + 2 * c + 1]);
    if (act == 4) {
        const float a = fminf(g, limit), b = fminf(fmaxf(u, -limit), limit);
        out[i] = from_f32<TA>(a / (1.0f + expf(-1.702f * a)) * (b + 1.0f));
        return;
    }
    out[i] = from_f32<TA>(gate_act_of(g, act) * u);
}

extern "C" int illm_gated_act_ex(const void* gu, void* out, int act_dtype, int T, int I, int act, float limit, void* stream) {
    if (T <= 0 || I <= 0) return 0;
    if (act < 1 || act > 4 || (act == 4 && !(limit > 0.f))) return ILLM_ERR_BAD_ARG;
    const long long n = (long long)T * I;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == ILLM_BF16) illm_launch(gated_act_kernel<bf16>, dim3(blocks), dim3(256), 0, s, (const bf16*)gu, (bf16*)out, I, n, act, limit);
    else if (act_dtype == ILLM_F32) illm_launch(gated_act_kernel<float>, dim3(blocks), dim3(256), 0, s, (const float*)gu, (float*)out, I, n, act, limit);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}
extern "C" int illm_gated_act(const void* gu, void* out, int act_dtype, int T, int I, int act, void* stream) {
    return illm_gated_act_ex(gu, out, act_dtype, T, I, act, 0.f, stream);
}

template <typename TA>
__global__ void take_columns_kernel(const float* __restrict__ x, int ld, int off, int n_cols, TA* __restrict__ y, long long n) {
    pdl_grid_sync();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long t = i / n_cols;
    y[i] = from_f32<TA>(x[t * ld + off + (i - t * n_cols)]);
}

extern "C" int illm_take_columns(const float* x, int ld, int off, int n_cols, void* y, int act_dtype, int T, void* stream) {
    if (T <= 0 || n_cols <= 0) return 0;
    const long long n = (long long)T * n_cols;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == ILLM_BF16) illm_launch(take_columns_kernel<bf16>, dim3(blocks), dim3(256), 0, s, x, ld, off, n_cols, (bf16*)y, n);
    else if (act_dtype == ILLM_F32) illm_launch(take_columns_kernel<float>, dim3(blocks), dim3(256), 0, s, x, ld, off, n_cols, (float*)y, n);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}

template <typename TA, bool VEC>          // VEC: eight neighbouring elements per thread
__global__ void join_rows_kernel(const float* __restrict__ a, const float* __restrict__ b, int H, TA* __restrict__ y, long long n) {
    pdl_grid_sync();
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * (VEC ? 8 : 1);
    if (i >= n) return;
    const long long t = i / (2 * H);
    const int c = (int)(i - t * 2 * H);
    const float* src = c < H ? a + t * H + c : b + t * H + c - H;
    if (VEC) {
        float v[8];
        load8(src, v);
        store8(y + i, v);
    } else {
        y[i] = from_f32<TA>(*src);
    }
}

extern "C" int illm_join_rows(const float* a, const float* b, int H, void* y, int act_dtype, int T, void* stream) {
    if (T <= 0 || H <= 0) return 0;
    const long long n = (long long)T * 2 * H;
    const bool vec = H % 8 == 0 && !(((uintptr_t)a | (uintptr_t)b | (uintptr_t)y) & 15);
    const unsigned blocks = (unsigned)(((vec ? n / 8 : n) + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (act_dtype == ILLM_BF16 && vec) illm_launch((join_rows_kernel<bf16, true>), dim3(blocks), dim3(256), 0, s, a, b, H, (bf16*)y, n);
    else if (act_dtype == ILLM_BF16) illm_launch((join_rows_kernel<bf16, false>), dim3(blocks), dim3(256), 0, s, a, b, H, (bf16*)y, n);
    else if (act_dtype == ILLM_F32 && vec) illm_launch((join_rows_kernel<float, true>), dim3(blocks), dim3(256), 0, s, a, b, H, (float*)y, n);
    else if (act_dtype == ILLM_F32) illm_launch((join_rows_kernel<float, false>), dim3(blocks), dim3(256), 0, s, a, b, H, (float*)y, n);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}

// add2_rmsnorm and scaled_add_rmsnorm (below) for rows of whole 16-byte pieces up to 16,384 wide: IT pieces per thread in
// registers, the weights on their way while the kernel before drains, every load of the row before its first sum.
// (Through shared memory, with the weight and the normed row element by element, a single row of 4,096 took 4.7 us and
// 1,777 rows 33 us for 102 MB.)  The block's size follows from the width alone.
// An addend may come as the unreduced K slices of its product (n slices, `stride` floats apart), which are added here.
struct RowSlices {
    const float* p;
    int n;
    long long stride;
};
template <typename TY, int IT, bool SCALED, bool SLICES>
__global__ void __launch_bounds__(1024)
row_add_rmsnorm_kernel(float* __restrict__ resid, const RowSlices d1, const RowSlices d2, const float* __restrict__ ls,
                       const float* __restrict__ w, TY* __restrict__ y, int H, float eps) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float scratch[32];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t base = (size_t)blockIdx.x * H;
    constexpr bool EARLY = IT <= 2;          // the registers hold no more than the row and its addends beyond
    float4 wv[IT], f[IT], v[IT], a[IT], b[IT];
    if (EARLY) {
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
            wv[i] = w && c < H ? *reinterpret_cast<const float4*>(w + c) : zero;
            f[i] = SCALED && c < H ? *reinterpret_cast<const float4*>(ls + c) : zero;
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        v[i] = c < H ? *reinterpret_cast<const float4*>(resid + base + c) : zero;
        a[i] = c >= H ? zero : SLICES ? row_sum_slices(d1.p + base + c, d1.n, d1.stride) : row_load4(d1.p + base + c);
        b[i] = SCALED || !d2.p || c >= H ? zero : SLICES ? row_sum_slices(d2.p + base + c, d2.n, d2.stride) : row_load4(d2.p + base + c);
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        if (SCALED) {
            if (!EARLY) f[i] = c < H ? *reinterpret_cast<const float4*>(ls + c) : zero;
            v[i] = make_float4(fmaf(a[i].x, f[i].x, v[i].x), fmaf(a[i].y, f[i].y, v[i].y), fmaf(a[i].z, f[i].z, v[i].z), fmaf(a[i].w, f[i].w, v[i].w));
        } else {
            v[i].x += a[i].x, v[i].y += a[i].y, v[i].z += a[i].z, v[i].w += a[i].w;
            if (d2.p) v[i].x += b[i].x, v[i].y += b[i].y, v[i].z += b[i].z, v[i].w += b[i].w;
        }
        if (c < H) *reinterpret_cast<float4*>(resid + base + c) = v[i];
        ss = fmaf(v[i].x, v[i].x, ss), ss = fmaf(v[i].y, v[i].y, ss), ss = fmaf(v[i].z, v[i].z, ss), ss = fmaf(v[i].w, v[i].w, ss);
    }
    if (!w) return;
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        if (c >= H) continue;
        if (!EARLY) wv[i] = *reinterpret_cast<const float4*>(w + c);
        const float4 r = make_float4((v[i].x * inv) * wv[i].x, (v[i].y * inv) * wv[i].y, (v[i].z * inv) * wv[i].z, (v[i].w * inv) * wv[i].w);
        row_store4(y + base + c, r);
    }
}

template <typename TY, bool SCALED>
static bool row_add_rmsnorm(float* resid, RowSlices d1, RowSlices d2, const float* ls, const float* w, void* y, int T, int H, float eps, cudaStream_t s) {
    // Beyond 8,192 channels a row fills the registers of an SM: finished addends go through shared memory
    // there (one row of 12,288 5.6 against 7.4 us, 2,048 rows of 16,384 132 against 152).
    if (H % 4 || !row_pieces(H) || (H > 8192 && d1.n <= 1 && d2.n <= 1) || (d1.stride & 3) || (d2.stride & 3) || row_odd(resid) || row_odd(d1.p) || row_odd(d2.p) || row_odd(ls) || row_odd(w) || row_odd(y))
        return false;
    const dim3 grid(T), block(row_threads(H));
    const bool slices = d1.n > 1 || d2.n > 1;
#define ILLM_RAN(IT, SLICES) illm_launch((row_add_rmsnorm_kernel<TY, IT, SCALED, SLICES>), grid, block, 0, s, resid, d1, d2, ls, w, (TY*)y, H, eps)
    if (row_pieces(H) == 1 && slices) ILLM_RAN(1, true);
    else if (row_pieces(H) == 1) ILLM_RAN(1, false);
    else if (row_pieces(H) == 2 && slices) ILLM_RAN(2, true);
    else if (row_pieces(H) == 2) ILLM_RAN(2, false);
    else ILLM_RAN(4, true);
#undef ILLM_RAN
    return true;
}

// add2_rmsnorm: resid[t, :] += d1[t, :] (+ d2[t, :]), all float32, and y[t, :] = resid[t, :] / sqrt(mean(resid^2) + eps) * w
// in the activation dtype: the two sublayer outputs of a parallel block folded into the next layer's norm.  A block
// per row, the row kept in shared memory between the two passes; the sum is (x + d1) + d2, as two separate additions give.
template <typename TY>
__global__ void __launch_bounds__(1024)
add2_rmsnorm_kernel(float* __restrict__ resid, const float* __restrict__ d1, const float* __restrict__ d2, const float* __restrict__ w,
                    TY* __restrict__ y, int H, float eps, int vec) {
    pdl_grid_sync();
    extern __shared__ __align__(16) float row_sm[];
    __shared__ float scratch[32];
    const size_t base = (size_t)blockIdx.x * H;
    float ss = 0.f;
    if (vec) {          // rows of whole 16-byte pieces: a thread's loads are all in flight before its first store
        const float4* r4 = reinterpret_cast<const float4*>(resid + base);
        const float4* a4 = reinterpret_cast<const float4*>(d1 + base);
        const float4* b4 = d2 ? reinterpret_cast<const float4*>(d2 + base) : nullptr;
        for (int c = threadIdx.x; c < H / 4; c += blockDim.x) {
            float4 v = r4[c];
            const float4 a = a4[c];
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            if (b4) {
                const float4 b = b4[c];
                v.x += b.x; v.y += b.y; v.z += b.z; v.w += b.w;
            }
            reinterpret_cast<float4*>(resid + base)[c] = v;
            reinterpret_cast<float4*>(row_sm)[c] = v;
            ss = fmaf(v.x, v.x, ss);
            ss = fmaf(v.y, v.y, ss);
            ss = fmaf(v.z, v.z, ss);
            ss = fmaf(v.w, v.w, ss);
        }
    } else {
        for (int c = threadIdx.x; c < H; c += blockDim.x) {
            float v = resid[base + c] + d1[base + c];
            if (d2) v += d2[base + c];
            resid[base + c] = v;
            row_sm[c] = v;
            ss = fmaf(v, v, ss);
        }
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    for (int c = threadIdx.x; c < H; c += blockDim.x) y[base + c] = from_f32<TY>((row_sm[c] * inv) * w[c]);
}

// n1, n2 > 1: d1, d2 are that many float32 slices, stride1 and stride2 floats apart, to be added up (rows of whole 16-byte pieces
// up to 16,384)
extern "C" int illm_add2_rmsnorm_slices(float* resid, const float* d1, int n1, long long stride1, const float* d2, int n2, long long stride2, const float* w,
                                        void* y, int act_dtype, int T, int H, float eps, void* stream) {
    if (T <= 0 || H <= 0) return 0;
    if (!d1 || (size_t)H * sizeof(float) > 200 * 1024) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t smem = (size_t)H * sizeof(float);
    static bool raised = false;
    if (!raised) {
        cudaFuncSetAttribute(add2_rmsnorm_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(add2_rmsnorm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        raised = true;
    }
    const RowSlices a{d1, n1, stride1}, b{d2, n2, stride2};
    if (act_dtype == ILLM_BF16 && w && row_add_rmsnorm<bf16, false>(resid, a, b, nullptr, w, y, T, H, eps, s)) return illm_launch_status();
    if (act_dtype == ILLM_F32 && w && row_add_rmsnorm<float, false>(resid, a, b, nullptr, w, y, T, H, eps, s)) return illm_launch_status();
    if (n1 > 1 || n2 > 1) return ILLM_ERR_BAD_ARG;
    const int vec = H % 4 == 0 && !row_odd(resid) && !row_odd(d1) && !row_odd(d2);
    int threads = ((vec ? H / 4 : H) + 31) / 32 * 32;       // the block size depends on the width alone
    threads = threads < 128 ? 128 : (threads > 1024 ? 1024 : threads);
    if (act_dtype == ILLM_BF16) illm_launch(add2_rmsnorm_kernel<bf16>, dim3(T), dim3(threads), smem, s, resid, d1, d2, w, (bf16*)y, H, eps, vec);
    else if (act_dtype == ILLM_F32) illm_launch(add2_rmsnorm_kernel<float>, dim3(T), dim3(threads), smem, s, resid, d1, d2, w, (float*)y, H, eps, vec);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}

extern "C" int illm_add2_rmsnorm(float* resid, const float* d1, const float* d2, const float* w, void* y, int act_dtype, int T, int H, float eps, void* stream) {
    return illm_add2_rmsnorm_slices(resid, d1, 1, 0, d2, 1, 0, w, y, act_dtype, T, H, eps, stream);
}

// scaled_add_rmsnorm: resid[t, :] += delta[t, :] * ls   (a sublayer's output through a per-channel layer scale,
// all float32), and, if w is given, y[t, :] = resid[t, :] / sqrt(mean(resid^2) + eps) * w in the activation dtype: the
// layer scale folded into the next norm.  A block per row, the row kept in shared memory between the two passes.
template <typename TY>
__global__ void __launch_bounds__(1024)
scaled_add_rmsnorm_kernel(float* __restrict__ resid, const float* __restrict__ delta, const float* __restrict__ ls,
                          const float* __restrict__ w, TY* __restrict__ y, int H, float eps, int vec) {
    pdl_grid_sync();
    extern __shared__ __align__(16) float row_sm[];
    __shared__ float scratch[32];
    const size_t base = (size_t)blockIdx.x * H;
    float ss = 0.f;
    if (vec) {          // rows of whole 16-byte pieces: a thread's loads are all in flight before its first store
        const float4* r4 = reinterpret_cast<const float4*>(resid + base);
        const float4* d4 = reinterpret_cast<const float4*>(delta + base);
        const float4* l4 = reinterpret_cast<const float4*>(ls);
        for (int c = threadIdx.x; c < H / 4; c += blockDim.x) {
            float4 v = r4[c];
            const float4 dl = d4[c], f = l4[c];
            v.x = fmaf(dl.x, f.x, v.x);
            v.y = fmaf(dl.y, f.y, v.y);
            v.z = fmaf(dl.z, f.z, v.z);
            v.w = fmaf(dl.w, f.w, v.w);
            reinterpret_cast<float4*>(resid + base)[c] = v;
            reinterpret_cast<float4*>(row_sm)[c] = v;
            ss = fmaf(v.x, v.x, ss);
            ss = fmaf(v.y, v.y, ss);
            ss = fmaf(v.z, v.z, ss);
            ss = fmaf(v.w, v.w, ss);
        }
    } else {
        for (int c = threadIdx.x; c < H; c += blockDim.x) {
            const float v = fmaf(delta[base + c], ls[c], resid[base + c]);
            resid[base + c] = v;
            row_sm[c] = v;
            ss = fmaf(v, v, ss);
        }
    }
    if (!w) return;
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    for (int c = threadIdx.x; c < H; c += blockDim.x) y[base + c] = from_f32<TY>((row_sm[c] * inv) * w[c]);
}

extern "C" int illm_scaled_add_rmsnorm_slices(float* resid, const float* delta, int splits, long long split_stride, const float* ls, const float* w, void* y,
                                              int act_dtype, int T, int H, float eps, void* stream) {
    if (T <= 0 || H <= 0) return 0;
    if (!delta || !ls || (w && !y) || (size_t)H * sizeof(float) > 200 * 1024) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t smem = (size_t)H * sizeof(float);
    static bool raised = false;
    if (!raised) {
        cudaFuncSetAttribute(scaled_add_rmsnorm_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(scaled_add_rmsnorm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        raised = true;
    }
    const RowSlices a{delta, splits, split_stride}, none{nullptr, 0, 0};
    if (act_dtype == ILLM_BF16 && row_add_rmsnorm<bf16, true>(resid, a, none, ls, w, y, T, H, eps, s)) return illm_launch_status();
    if (act_dtype == ILLM_F32 && row_add_rmsnorm<float, true>(resid, a, none, ls, w, y, T, H, eps, s)) return illm_launch_status();
    if (splits > 1) return ILLM_ERR_BAD_ARG;
    const int vec = H % 4 == 0 && !row_odd(resid) && !row_odd(delta) && !row_odd(ls);
    int threads = ((vec ? H / 4 : H) + 31) / 32 * 32;       // the block size depends on the width alone
    threads = threads < 128 ? 128 : (threads > 1024 ? 1024 : threads);
    if (act_dtype == ILLM_BF16) illm_launch(scaled_add_rmsnorm_kernel<bf16>, dim3(T), dim3(threads), smem, s, resid, delta, ls, w, (bf16*)y, H, eps, vec);
    else if (act_dtype == ILLM_F32) illm_launch(scaled_add_rmsnorm_kernel<float>, dim3(T), dim3(threads), smem, s, resid, delta, ls, w, (float*)y, H, eps, vec);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}

extern "C" int illm_scaled_add_rmsnorm(float* resid, const float* delta, const float* ls, const float* w, void* y, int act_dtype, int T, int H, float eps,
                                       void* stream) {
    return illm_scaled_add_rmsnorm_slices(resid, delta, 1, 0, ls, w, y, act_dtype, T, H, eps, stream);
}

// add_bias: y[t, c] += b[c] (b float32), in place, for a projection with a bias whose product kernel has no bias epilogue
// (VEC: four neighbouring columns per thread)
template <typename TA, bool VEC>
__global__ void add_bias_kernel(TA* __restrict__ y, const float* __restrict__ b, int H, long long n) {
    pdl_grid_sync();
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * (VEC ? 4 : 1);
    if (i >= n) return;
    if (VEC) {
        const float4 f = *reinterpret_cast<const float4*>(b + i % H);
        float4 v = *reinterpret_cast<const float4*>(y + i);
        v.x += f.x, v.y += f.y, v.z += f.z, v.w += f.w;
        *reinterpret_cast<float4*>(y + i) = v;
    } else {
        y[i] = from_f32<TA>(to_f32(y[i]) + b[i % H]);
    }
}
extern "C" int illm_add_bias(void* y, int dtype, const float* b, int T, int H, void* stream) {
    if (T <= 0 || H <= 0) return 0;
    if (!y || !b) return ILLM_ERR_BAD_ARG;
    const long long n = (long long)T * H;
    const bool vec = dtype == ILLM_F32 && H % 4 == 0 && !(((uintptr_t)y | (uintptr_t)b) & 15);
    const unsigned blocks = (unsigned)(((vec ? n / 4 : n) + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == ILLM_BF16) illm_launch((add_bias_kernel<bf16, false>), dim3(blocks), dim3(256), 0, s, (bf16*)y, b, H, n);
    else if (dtype == ILLM_F32 && vec) illm_launch((add_bias_kernel<float, true>), dim3(blocks), dim3(256), 0, s, (float*)y, b, H, n);
    else if (dtype == ILLM_F32) illm_launch((add_bias_kernel<float, false>), dim3(blocks), dim3(256), 0, s, (float*)y, b, H, n);
    else return ILLM_ERR_BAD_ARG;
    return illm_launch_status();
}

__global__ void soft_cap_kernel(float* __restrict__ x, long long n, float cap) {
    pdl_grid_sync();
    const float inv = 1.0f / cap;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) x[i] = cap * tanhf(x[i] * inv);
}

extern "C" int illm_soft_cap(float* x, long long n, float cap, void* stream) {
    if (n <= 0) return 0;
    if (!x || !(cap > 0.f)) return ILLM_ERR_BAD_ARG;
    const long long blocks = (n + 255) / 256;
    illm_launch(soft_cap_kernel, dim3((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0, (cudaStream_t)stream, x, n, cap);
    return illm_launch_status();
}
