// Norm after the sum: the residual stream itself is replaced by the normed row.
//
//   v = alpha * x[r] + delta[r];   x[r] = v / sqrt(mean(v^2) + eps) * w;   y[r] = x[r] rounded to the compute dtype
//
// This is the arrangement "x <- norm(alpha * x + sublayer(x))": where add_rmsnorm (rmsnorm.cu) keeps the
// un-normed sum as the stream and hands the normed row to the next sublayer only, here the normed
// row is both.  The stream, the scaled sum, the mean of squares and the product with the weight are
// float32; w is float32 (a weight stored as an offset from one has the one added when it is loaded).
// The addend may also come as the unreduced K slices of a split matrix product (float32
// [splits, rows, H]); they are added in ascending order, as the stand-alone reduction would.
// One block per row and a fixed order of the sums, so a row's bits do not depend on the launch.
#include "row_ops.cuh"

template <typename TD, typename TY>
__global__ void __launch_bounds__(1024)
scale_add_rmsnorm_kernel(float* __restrict__ resid, const TD* __restrict__ delta, const float* __restrict__ w,
                         TY* __restrict__ y, int H, float alpha, float eps, const float* __restrict__ partials, int splits,
                         long long split_stride) {
    pdl_grid_sync();
    __shared__ float scratch[32];
    float* x = resid + (size_t)blockIdx.x * H;
    const TD* dl = delta ? delta + (size_t)blockIdx.x * H : nullptr;
    float ss = 0.f;
    for (int c = threadIdx.x; c < H; c += blockDim.x) {
        float v = alpha * x[c];
        if (dl) v += to_f32(dl[c]);
        if (partials) {
            // the loads of eight slices are in flight together; the additions keep the slices' order
            const float* ps = partials + (size_t)blockIdx.x * H + c;
            float sum = 0.f;
            int k = 0;
            for (; k + 8 <= splits; k += 8) {
                float t[8];
#pragma unroll
                for (int u = 0; u < 8; u++) t[u] = ps[(size_t)(k + u) * split_stride];
#pragma unroll
                for (int u = 0; u < 8; u++) sum += t[u];
            }
            for (; k < splits; k++) sum += ps[(size_t)k * split_stride];
            v += sum;
        }
        x[c] = v;            // read again below by the same thread
        ss += v * v;
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    TY* o = y ? y + (size_t)blockIdx.x * H : nullptr;
    for (int c = threadIdx.x; c < H; c += blockDim.x) {
        const float v = (x[c] * inv) * w[c];
        x[c] = v;
        if (o) o[c] = from_f32<TY>(v);
    }
}

// Rows of whole 16-byte pieces up to 16,384 wide: IT pieces per thread stay in registers, the weight is read while the kernel
// before drains, and the row's pieces of the stream, the addend and up to eight of its slices are on their way together: a
// single token's block is bound by the latency of its loads (one row of 2,048 with eight slices took 7 us channel by
// channel with the sum going out to the stream and back).
// SLICES: the addend comes as slices.
template <typename TD, typename TY, int IT, bool SLICES>
__global__ void __launch_bounds__(1024)
scale_add_rmsnorm_vec_kernel(float* __restrict__ resid, const TD* __restrict__ delta, const float* __restrict__ w, TY* __restrict__ y, int H,
                             float alpha, float eps, const float* __restrict__ partials, int splits, long long split_stride) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float scratch[32];
    float4 wv[IT], v[IT];
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        wv[i] = c < H ? row_load4(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const size_t base = (size_t)blockIdx.x * H;
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c >= H) continue;
        const float4 x = row_load4(resid + base + c);
        float4 add = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SLICES) add = row_sum_slices(partials + base + c, splits, split_stride);
        else if (delta) add = row_load4(delta + base + c);
        v[i] = make_float4(fmaf(alpha, x.x, add.x), fmaf(alpha, x.y, add.y), fmaf(alpha, x.z, add.z), fmaf(alpha, x.w, add.w));
        ss = fmaf(v[i].x, v[i].x, ss), ss = fmaf(v[i].y, v[i].y, ss), ss = fmaf(v[i].z, v[i].z, ss), ss = fmaf(v[i].w, v[i].w, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
#pragma unroll
    for (int i = 0; i < IT; i++) {
        const int c = 4 * (threadIdx.x + i * (int)blockDim.x);
        if (c >= H) continue;
        const float4 r = make_float4((v[i].x * inv) * wv[i].x, (v[i].y * inv) * wv[i].y, (v[i].z * inv) * wv[i].z, (v[i].w * inv) * wv[i].w);
        row_store4(resid + base + c, r);
        if (y) row_store4(y + base + c, r);
    }
}

extern "C" int illm_scale_add_rmsnorm(float* resid, const void* delta, int delta_dtype, const float* w, void* y, int y_dtype,
                                      int n_rows, int H, float alpha, float eps, const float* partials, int splits, long long split_stride,
                                      void* stream) {
    if (n_rows <= 0) return 0;
    if (H <= 0 || !resid || !w) return ILLM_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // which kernel runs and its threads follow from the width and the layout alone, so a row's sums have the same order in every launch
    if (H % 4 == 0 && row_pieces(H) && split_stride % 4 == 0 && !row_odd(resid) && !row_odd(delta) && !row_odd(w) && !row_odd(y) && !row_odd(partials)) {
        const int pieces = row_pieces(H), vthreads = row_threads(H);
        const bool slices = !delta && partials && splits > 0;
#define ILLM_PNV(TD, TY, IT)                                                                                                          \
    illm_launch(slices ? scale_add_rmsnorm_vec_kernel<TD, TY, IT, true> : scale_add_rmsnorm_vec_kernel<TD, TY, IT, false>, dim3(n_rows), dim3(vthreads), 0, s, resid, (const TD*)delta, w, (TY*)y, H, alpha, eps, \
                partials, splits, split_stride)
#define ILLM_PNV_FOR(TD, TY)                            \
    do {                                                \
        if (pieces == 1) ILLM_PNV(TD, TY, 1);           \
        else if (pieces == 2) ILLM_PNV(TD, TY, 2);      \
        else ILLM_PNV(TD, TY, 4);                       \
    } while (0)
        if (delta_dtype == ILLM_F32 && y_dtype == ILLM_F32) ILLM_PNV_FOR(float, float);
        else if (delta_dtype == ILLM_F32 && y_dtype == ILLM_BF16) ILLM_PNV_FOR(float, bf16);
        else if (delta_dtype == ILLM_BF16 && y_dtype == ILLM_BF16) ILLM_PNV_FOR(bf16, bf16);
        else if (delta_dtype == ILLM_BF16 && y_dtype == ILLM_F32) ILLM_PNV_FOR(bf16, float);
        else return ILLM_ERR_BAD_ARG;
#undef ILLM_PNV_FOR
#undef ILLM_PNV
        return illm_launch_status();
    }
    const int threads = H >= 4096 ? 1024 : H >= 1024 ? 512 : 256;
#define ILLM_PN(TD, TY) \
    illm_launch(scale_add_rmsnorm_kernel<TD, TY>, dim3(n_rows), dim3(threads), 0, s, resid, (const TD*)delta, w, (TY*)y, H, alpha, eps, partials, splits, \
                split_stride)
    if (delta_dtype == ILLM_F32 && y_dtype == ILLM_F32) ILLM_PN(float, float);
    else if (delta_dtype == ILLM_F32 && y_dtype == ILLM_BF16) ILLM_PN(float, bf16);
    else if (delta_dtype == ILLM_BF16 && y_dtype == ILLM_BF16) ILLM_PN(bf16, bf16);
    else if (delta_dtype == ILLM_BF16 && y_dtype == ILLM_F32) ILLM_PN(bf16, float);
    else return ILLM_ERR_BAD_ARG;
#undef ILLM_PN
    return illm_launch_status();
}
