// Layer norm or RMS norm with a weight and no bias, around the float32 residual stream of a block that norms a
// sublayer's input AND its output:
//
//   x[r] <- x[r] + a n(y[r]) * wb         (the sublayer's output y, normed, joins the stream; optional; a is a constant)
//   out[r] = n(x[r]) * w                  (what the next sublayer reads; optional)
//   n(v) = (v - mean(v)) / sqrt(mean((v - mean(v))^2) + eps)      CENTER (layer norm; a = 1)
//   n(v) = v / sqrt(mean(v^2) + eps)                              otherwise (RMS norm)
//
// in one kernel, because the second norm reads the row the first one has just made.  One block per row, every statistic of the layer norm in two passes (mean, then the mean squared deviation), the RMS norm's
// in one, with a fixed order of the sums, all float32.  `rows` (int32) gathers: only those rows are made, and x is then left as it is (the model's
// last norm, for the rows whose logits are wanted).
#include "row_ops.cuh"

// Any width, the row in shared memory.  V = 4: four neighbouring channels per thread at a time (rows of whole 16-byte pieces), V = 1: one.
template <typename TO, int V, bool CENTER>
__global__ void __launch_bounds__(1024, 2)
ln_sandwich_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ wb, const float* __restrict__ w,
                   TO* __restrict__ out, const int* __restrict__ rows, int H, float eps, float post_scale, int write_x) {
    pdl_grid_sync();
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[32];
    const int r = rows ? rows[blockIdx.x] : blockIdx.x;
    const float* src = (y ? y : x) + (size_t)r * H;
    float* xr = x + (size_t)r * H;
    const int first = threadIdx.x * V, step = blockDim.x * V;
    // the mean (CENTER) and 1 / sqrt(the mean square of the deviation + eps) of what lies in `row`, whose sum (CENTER) or sum of
    // squares the thread's own channels have given already
    auto statistics = [&](float own, float& mean) {
        mean = 0.f;
        if (CENTER) {
            mean = block_sum(own, scratch) / (float)H;
            own = 0.f;
            for (int c = first; c < H; c += step) {
#pragma unroll
                for (int i = 0; i < V; i++) {
                    const float dlt = row[c + i] - mean;
                    own = fmaf(dlt, dlt, own);
                }
            }
        }
        return 1.0f / sqrtf(block_sum(own, scratch) / (float)H + eps);
    };
    auto take = [&](float s, float v) { return CENTER ? s + v : fmaf(v, v, s); };
    float own = 0.f, mean;
    for (int c = first; c < H; c += step) {
        if (V == 4) {
            const float4 v = row_load4(src + c);
            row_store4(row + c, v);
            own = take(take(take(take(own, v.x), v.y), v.z), v.w);
        } else {
            row[c] = src[c];
            own = take(own, row[c]);
        }
    }
    if (y) {
        const float inv = statistics(own, mean);
        auto post = [&](float v, float weight, float onto) { return fmaf(post_scale, ((v - mean) * inv) * weight, onto); };
        own = 0.f;
        for (int c = first; c < H; c += step) {
            if (V == 4) {
                const float4 xv = row_load4(xr + c), wv = row_load4(wb + c), t = row_load4(row + c);
                const float4 v = make_float4(post(t.x, wv.x, xv.x), post(t.y, wv.y, xv.y), post(t.z, wv.z, xv.z), post(t.w, wv.w, xv.w));
                row_store4(row + c, v);
                if (write_x) row_store4(xr + c, v);
                own = take(take(take(take(own, v.x), v.y), v.z), v.w);
            } else {
                const float v = post(row[c], wb[c], xr[c]);
                row[c] = v;
                if (write_x) xr[c] = v;
                own = take(own, v);
            }
        }
    }
    if (!out) return;
    const float inv = statistics(own, mean);
    TO* o = out + (size_t)blockIdx.x * H;
    for (int c = first; c < H; c += step) {
        if (V == 4) {
            const float4 wv = row_load4(w + c), t = row_load4(row + c);
            row_store4(o + c, make_float4(((t.x - mean) * inv) * wv.x, ((t.y - mean) * inv) * wv.y, ((t.z - mean) * inv) * wv.z, ((t.w - mean) * inv) * wv.w));
        } else {
            o[c] = from_f32<TO>(((row[c] - mean) * inv) * w[c]);
        }
    }
}

// Rows of whole 16-byte pieces up to 16,384 wide: IT pieces per thread in registers.  Both rows and both weights are on
// their way before the first sum (the weights while the kernel before drains), so that a single token's block, which
// is bound by latency alone, waits for memory once (a row of 4,096 took 6.3 us with the row going through shared
// memory and the stream and the weights asked for behind the first sum).  y may come as the unreduced K slices of its
// product, which are added here.
// EARLY false: the same sums in the same order, the weights read where they are used, so that 32 registers do and two blocks of
// 1,024 threads lie on an SM, for steps of more rows than SMs (2,048 rows of 4,096 and 8,192, layer norms: 44 and 66 us, so 30 and
// 50).  SLICES: y comes as slices.
template <typename TO, int IT, bool CENTER, bool EARLY, bool SLICES>
__global__ void __launch_bounds__(1024, EARLY || IT > 2 ? 1 : 2)
ln_sandwich_vec_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ wb, const float* __restrict__ w,
                       TO* __restrict__ out, const int* __restrict__ rows, int H, float eps, float post_scale, int write_x, int splits,
                       long long split_stride) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float scratch[32];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v[IT], yv[IT], wv[IT], wbv[IT];
    if (EARLY) {
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
            wbv[i] = y && c < H ? *reinterpret_cast<const float4*>(wb + c) : zero;
            wv[i] = out && c < H ? *reinterpret_cast<const float4*>(w + c) : zero;
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int r = rows ? rows[blockIdx.x] : blockIdx.x;
    float* xr = x + (size_t)r * H;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        v[i] = c < H ? *reinterpret_cast<const float4*>(xr + c) : zero;
        yv[i] = !y || c >= H ? zero : SLICES ? row_sum_slices(y + (size_t)r * H + c, splits, split_stride) : row_load4(y + (size_t)r * H + c);
    }
    // the mean (CENTER) and 1 / sqrt(the mean square of the deviation + eps) of a row; pieces beyond it count for nothing
    auto statistics = [&](const float4 (&a)[IT], float& mean) {
        mean = 0.f;
        float s = 0.f;
        if (CENTER) {
#pragma unroll
            for (int i = 0; i < IT; i++) s += a[i].x, s += a[i].y, s += a[i].z, s += a[i].w;
            mean = block_sum(s, scratch) / (float)H;
            s = 0.f;
        }
#pragma unroll
        for (int i = 0; i < IT; i++) {
            if (CENTER && 4 * (threadIdx.x + i * (int)blockDim.x) >= (unsigned)H) continue;
            const float dx = a[i].x - mean, dy = a[i].y - mean, dz = a[i].z - mean, dw = a[i].w - mean;
            s = fmaf(dx, dx, s), s = fmaf(dy, dy, s), s = fmaf(dz, dz, s), s = fmaf(dw, dw, s);
        }
        return 1.0f / sqrtf(block_sum(s, scratch) / (float)H + eps);
    };
    float mean;
    if (y) {
        const float inv = statistics(yv, mean);
#pragma unroll
        for (int i = 0; i < IT; i++) {
            const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
            if (c >= H) continue;
            if (!EARLY) wbv[i] = *reinterpret_cast<const float4*>(wb + c);
            v[i].x = fmaf(post_scale, ((yv[i].x - mean) * inv) * wbv[i].x, v[i].x);
            v[i].y = fmaf(post_scale, ((yv[i].y - mean) * inv) * wbv[i].y, v[i].y);
            v[i].z = fmaf(post_scale, ((yv[i].z - mean) * inv) * wbv[i].z, v[i].z);
            v[i].w = fmaf(post_scale, ((yv[i].w - mean) * inv) * wbv[i].w, v[i].w);
            if (write_x) *reinterpret_cast<float4*>(xr + c) = v[i];
        }
    }
    if (!out) return;
    const float inv = statistics(v, mean);
    TO* o = out + (size_t)blockIdx.x * H;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        if (c >= H) continue;
        if (!EARLY) wv[i] = *reinterpret_cast<const float4*>(w + c);
        row_store4(o + c, make_float4(((v[i].x - mean) * inv) * wv[i].x, ((v[i].y - mean) * inv) * wv[i].y, ((v[i].z - mean) * inv) * wv[i].z,
                                      ((v[i].w - mean) * inv) * wv[i].w));
    }
}

template <typename TO, bool CENTER>
static int ln_launch(float* x, const float* y, const float* wb, const float* w, TO* out, const int* rows, int n_rows, int H, float eps,
                     float post_scale, int write_x, int splits, long long split_stride, cudaStream_t s) {
    // the threads and the order of a row's sums follow from the width and the layout alone, so a row has the same bits in every step
    const bool pieces = H % 4 == 0 && split_stride % 4 == 0 && !row_odd(x) && !row_odd(y) && !row_odd(wb) && !row_odd(w) && !row_odd(out);
    // Many rows beyond 8,192 channels go through shared memory: two rows fill the registers of an SM, whose one block's passes follow
    // one another (2,048 rows of 16,384: 121 us against 86; 64 rows 7.7 against 9.6).  The sums have the same order in both.
    const bool early = n_rows <= illm_sm_count();
    if (pieces && row_pieces(H) && (H <= 8192 || early || splits > 1)) {
        const dim3 grid(n_rows), block(row_threads(H));
#define ILLM_LNV(IT, EARLY, SLICES)                                                                                                            \
    illm_launch((ln_sandwich_vec_kernel<TO, IT, CENTER, EARLY, SLICES>), grid, block, 0, s, x, y, wb, w, out, rows, H, eps, post_scale, write_x, splits, split_stride)
#define ILLM_LNV_FOR(IT)                              \
    do {                                              \
        if (splits > 1) ILLM_LNV(IT, IT <= 2, true);  \
        else if (early) ILLM_LNV(IT, IT <= 2, false); \
        else ILLM_LNV(IT, false, false);              \
    } while (0)
        if (row_pieces(H) == 1) ILLM_LNV_FOR(1);
        else if (row_pieces(H) == 2) ILLM_LNV_FOR(2);
        else ILLM_LNV_FOR(4);
#undef ILLM_LNV_FOR
#undef ILLM_LNV
        return illm_launch_status();
    }
    if (splits > 1) return ILLM_ERR_BAD_ARG;
    const size_t smem = (size_t)H * sizeof(float);
    const bool raise = smem > 47 * 1024;        // beside the kernel's own few words
    if (pieces) {
        if (raise) cudaFuncSetAttribute(ln_sandwich_kernel<TO, 4, CENTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        illm_launch((ln_sandwich_kernel<TO, 4, CENTER>), dim3(n_rows), dim3(row_pieces(H) ? row_threads(H) : 512), smem, s, x, y, wb, w, out, rows, H, eps, post_scale, write_x);
    } else {
        if (raise) cudaFuncSetAttribute(ln_sandwich_kernel<TO, 1, CENTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        illm_launch((ln_sandwich_kernel<TO, 1, CENTER>), dim3(n_rows), dim3(256), smem, s, x, y, wb, w, out, rows, H, eps, post_scale, write_x);
    }
    return illm_launch_status();
}

// y, wb: nullptr for no addition; w, out: nullptr for the addition alone; rows: nullptr for rows 0 .. n_rows - 1;
// center: layer norm (post_scale is then 1), else RMS norm
// splits > 1: y is that many float32 slices, split_stride floats apart, to be added up (rows of whole 16-byte pieces up to 16,384)
extern "C" int illm_norm_sandwich_slices(float* x, const float* y, int splits, long long split_stride, const float* wb, const float* w, void* out,
                                         int out_dtype, const int* rows, int n_rows, int H, float eps, int write_x, int center, float post_scale,
                                         void* stream) {
    if (n_rows <= 0) return 0;
    if (H <= 0 || !x || (y && !wb) || ((out != nullptr) != (w != nullptr)) || splits < 1) return ILLM_ERR_BAD_ARG;
    if ((size_t)H * sizeof(float) > 200 * 1024 || (center && post_scale != 1.f)) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == ILLM_BF16 && center) return ln_launch<bf16, true>(x, y, wb, w, (bf16*)out, rows, n_rows, H, eps, 1.f, write_x, splits, split_stride, s);
    if (out_dtype == ILLM_BF16) return ln_launch<bf16, false>(x, y, wb, w, (bf16*)out, rows, n_rows, H, eps, post_scale, write_x, splits, split_stride, s);
    if (out_dtype == ILLM_F32 && center) return ln_launch<float, true>(x, y, wb, w, (float*)out, rows, n_rows, H, eps, 1.f, write_x, splits, split_stride, s);
    if (out_dtype == ILLM_F32) return ln_launch<float, false>(x, y, wb, w, (float*)out, rows, n_rows, H, eps, post_scale, write_x, splits, split_stride, s);
    return ILLM_ERR_BAD_ARG;
}
extern "C" int illm_norm_sandwich(float* x, const float* y, const float* wb, const float* w, void* out, int out_dtype, const int* rows,
                                  int n_rows, int H, float eps, int write_x, int center, float post_scale, void* stream) {
    return illm_norm_sandwich_slices(x, y, 1, 0, wb, w, out, out_dtype, rows, n_rows, H, eps, write_x, center, post_scale, stream);
}

extern "C" int illm_layernorm_sandwich(float* x, const float* y, const float* wb, const float* w, void* out, int out_dtype, const int* rows,
                                       int n_rows, int H, float eps, int write_x, void* stream) {
    return illm_norm_sandwich(x, y, wb, w, out, out_dtype, rows, n_rows, H, eps, write_x, 1, 1.f, stream);
}
