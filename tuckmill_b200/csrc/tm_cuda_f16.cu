// F16-weight matrices: y[r] = dot(f32(w_row_r), x) with f32 accumulation -- the reference's
// tm_f16_gemv / tm_f16_gemm / tm_f16_row_f32 (native/metal/kernels.metal:296-315, 638-668,
// native/metal/tm_metal.h:142,156,179), which serve F16-weight artifacts: the reference's own
// model fixtures (crates/manifest/src/testing.rs:241-256) and F16 twins of quantized models.
// A matrix is rows * cols binary16 values, row-major, uploaded verbatim.
//
// One kernel serves the GEMV, the batched form (any batch: a (row, token) result does not depend
// on how many tokens share the launch, so batch 1 is bit-identical to the GEMV, the contract of
// tm_metal.h:160-164) and the fused forms the decode step uses (the elementwise prologue of the
// Q8_0 GEMV: RMS norm with the same canonical sum of squares, silu/gelu * up; store or accumulate).
// Lane l of a warp adds columns 8l .. 8l+7, 8l+256, ... of its rows in that order, the lanes are added with a xor
// butterfly.
#include "tm_cuda_internal.cuh"
#include "tm_cuda_device.cuh"

namespace {

constexpr int kThreads = tmdev::kThreads;
constexpr int kWarps = tmdev::kWarps;

struct f16_args {
    const __half *w;   // [rows][cols]
    const float *x;    // [M][cols]
    float *y;          // [M][rows]
    const float *pro;  // norm weight [cols] or the multiplicand [M][cols]
    uint32_t rows, cols;
    float eps;
    int prologue, epilogue;
};

// A warp takes R rows at a time, lane l the eight columns 8l..8l+7 of every 256: one 16-byte load per row and trip, the
// trip's activations read from shared memory once for all R rows and M tokens.  Which columns a lane adds, and in which
// order, depends on neither R nor M, so a (row, token) result is the same bits in every batch.
//   * one token: bound by bytes.  The first trip's weights are requested before the dependency wait and the next trip's
//     while one is multiplied (16 MB projection of a 0.6B decoder, 2-byte loads of 64 columns: 1.0 TB/s; now 3.4);
//   * several: bound by FMAs and the shared-memory reads that feed them, R x M products for M reads.
// Activations lie as two planes of half-octets, so that lanes read consecutive 16-byte words.
template <int M, int R>
__global__ void __launch_bounds__(kThreads) f16_gemv_kernel(const f16_args args) {
    f16_args a = args;
    if constexpr (M > 1) {  // a grid row per slice of M tokens
        const size_t t0 = (size_t)blockIdx.y * M;
        a.x += t0 * a.cols;
        a.y += t0 * a.rows;
        if (a.prologue == TM_CUDA_PRO_SILU_MUL || a.prologue == TM_CUDA_PRO_GELU_MUL) a.pro += t0 * a.cols;
    }
    extern __shared__ __align__(16) float xs[];  // [M][2][octets][4]
    __shared__ float red[kWarps];
    constexpr int U = M == 1 ? (R == 1 ? 4 : 2) : 1;  // 256-column trips requested together
    const uint32_t cols = a.cols, rows = a.rows, octets = (cols + 7u) / 8u;
    const uint32_t lane = threadIdx.x & 31, warp = tmdev::warp_index();
    const bool vec = (cols & 7u) == 0u && (((size_t)a.w) & 15u) == 0u;
    auto load = [&](uint32_t row, uint32_t o) -> int4 {
        if (o >= octets || row >= rows) return make_int4(0, 0, 0, 0);
        const __half *p = a.w + (size_t)row * cols + o * 8u;
        if (vec) return __ldg((const int4 *)p);
        __half h[8];
#pragma unroll
        for (uint32_t e = 0; e < 8u; ++e) h[e] = o * 8u + e < cols ? p[e] : __float2half_rn(0.0f);
        return *(const int4 *)h;
    };
    uint32_t row0 = (blockIdx.x * kWarps + warp) * R;
    int4 cur[U][R];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) cur[u][r] = load(row0 + r, lane + 32u * u);
    tmdev::pdl_trigger();
    tmdev::pdl_wait();
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
        const float *xm = a.x + (size_t)m * cols;
        float *xd = xs + (size_t)m * octets * 8u;
        float inv_rms = 0.0f;
        const bool one_pass = octets * 8u <= kThreads * 16u;  // the norm's sum from the registers that hold the row
        if (a.prologue == TM_CUDA_PRO_RMSNORM && !one_pass) {
            const float ss = tmdev::block_sumsq(xm, cols, red);
            inv_rms = 1.0f / sqrtf(ss / (float)cols + a.eps);
        }
        const float *pm = a.prologue == TM_CUDA_PRO_NONE ? nullptr : a.prologue == TM_CUDA_PRO_RMSNORM ? a.pro : a.pro + (size_t)m * cols;
        const bool quads = (cols & 3u) == 0u && (((size_t)xm | (size_t)pm) & 15u) == 0u;
        // A thread's 16 columns are loaded before any is computed: one column after the other, silu * up of 3072 columns
        // took half of a 12 us call.
        constexpr int B = 4;
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < octets * 8u; c0 += kThreads * 4u * B) {
            const uint32_t cb = c0 + threadIdx.x * 4u;
            float v[B][4], p[B][4];
#pragma unroll
            for (int i = 0; i < B; ++i) {
                const uint32_t c = cb + i * kThreads * 4u;
                if (quads && c < cols) {
                    *(float4 *)v[i] = *(const float4 *)(xm + c);
                    *(float4 *)p[i] = pm ? *(const float4 *)(pm + c) : make_float4(1.f, 1.f, 1.f, 1.f);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        v[i][j] = c + j < cols ? xm[c + j] : 0.0f;
                        p[i][j] = pm && c + j < cols ? pm[c + j] : 1.0f;
                    }
                }
            }
            if (a.prologue == TM_CUDA_PRO_RMSNORM && one_pass) {
                float ss = 0.0f;
#pragma unroll
                for (int i = 0; i < B; ++i) ss = tmdev::sumsq_quad(ss, make_float4(v[i][0], v[i][1], v[i][2], v[i][3]));
                inv_rms = 1.0f / sqrtf(tmdev::block_reduce_sumsq(ss, red) / (float)cols + a.eps);
            }
#pragma unroll
            for (int i = 0; i < B; ++i) {
                const uint32_t c = cb + i * kThreads * 4u;
                if (c >= octets * 8u) break;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (a.prologue == TM_CUDA_PRO_RMSNORM) v[i][j] = v[i][j] * inv_rms * p[i][j];
                    else if (a.prologue == TM_CUDA_PRO_SILU_MUL) v[i][j] = tmdev::silu_f(v[i][j]) * p[i][j];
                    else if (a.prologue == TM_CUDA_PRO_GELU_MUL) v[i][j] = tmdev::gelu_tanh_f(v[i][j]) * p[i][j];
                }
                *(float4 *)(xd + ((c & 4u) ? octets * 4u : 0u) + (c >> 3) * 4u) = *(const float4 *)v[i];
            }
        }
    }
    __syncthreads();
    const uint32_t stride = gridDim.x * kWarps * R;
    for (; row0 < rows; row0 += stride) {
        float acc[R][M];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < M; ++m) acc[r][m] = 0.0f;
#pragma unroll 1
        for (uint32_t o = lane; o - lane < octets; o += 32u * U) {
            int4 nxt[U][R];
            const bool more = o - lane + 32u * U < octets;  // else the next rows' first trip
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int r = 0; r < R; ++r)
                    nxt[u][r] = more ? load(row0 + r, o + 32u * (U + u)) : load(row0 + stride + r, lane + 32u * u);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t oc = o + 32u * u;
                if (oc < octets) {
                    float wf[R][8];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const __half2 *h = (const __half2 *)&cur[u][r];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float2 f = __half22float2(h[e]);
                            wf[r][2 * e] = f.x;
                            wf[r][2 * e + 1] = f.y;
                        }
                    }
#pragma unroll
                    for (int m = 0; m < M; ++m) {
                        const float *xd = xs + (size_t)m * octets * 8u + oc * 4u;
                        const float4 x0 = *(const float4 *)xd, x1 = *(const float4 *)(xd + octets * 4u);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            float t = acc[r][m];
                            t = fmaf(wf[r][0], x0.x, t);
                            t = fmaf(wf[r][1], x0.y, t);
                            t = fmaf(wf[r][2], x0.z, t);
                            t = fmaf(wf[r][3], x0.w, t);
                            t = fmaf(wf[r][4], x1.x, t);
                            t = fmaf(wf[r][5], x1.y, t);
                            t = fmaf(wf[r][6], x1.z, t);
                            acc[r][m] = fmaf(wf[r][7], x1.w, t);
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int r = 0; r < R; ++r) cur[u][r] = nxt[u][r];
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < M; ++m) {
                float v = acc[r][m];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0 && row0 + r < rows) {
                    float *yp = a.y + (size_t)m * rows + row0 + r;
                    *yp = a.epilogue == TM_CUDA_EPI_ADD ? *yp + v : v;
                }
            }
    }
}

template <int M, int R>
cudaError_t launch_f16_rows(tm_cuda_ctx *ctx, const f16_args &a, size_t smem, uint32_t slices) {
    static std::atomic<bool> attr_set[64] = {};
    const int dev = ctx->device;
    // (the kernel's own shared array counts towards the 48 KB that need no attribute)
    if (smem + 1024u > 48u * 1024u && (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire))) {
        cudaError_t e = cudaFuncSetAttribute(f16_gemv_kernel<M, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)ctx->smem_optin - 4096);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    // One resident wave: every CTA stages the activations once and walks its share of the rows.
    uint32_t per_sm = (uint32_t)(ctx->smem_optin / (smem + 2048u));
    per_sm = per_sm < 1u ? 1u : per_sm > (M == 1 ? 4u : 2u) ? (M == 1 ? 4u : 2u) : per_sm;
    uint32_t grid = (a.rows + kWarps * R - 1) / (kWarps * R);
    const uint32_t wave = (uint32_t)ctx->sm_count * per_sm / slices;
    if (grid > wave) grid = wave < 1u ? 1u : wave;
    return tm_launch_pdl(ctx, f16_gemv_kernel<M, R>, dim3(grid, slices), dim3(kThreads), smem, a);
}
// Rows per warp: as many as leave every SM a CTA (a 1024-row projection of one token keeps one row a warp).
template <int M>
cudaError_t launch_f16(tm_cuda_ctx *ctx, const f16_args &a, size_t smem, uint32_t slices) {
    const uint64_t warps = (uint64_t)ctx->sm_count * kWarps, rows = (uint64_t)a.rows * slices;
    if (rows >= 4u * warps || (M > 2 && rows >= 2u * warps)) return launch_f16_rows<M, 4>(ctx, a, smem, slices);
    if (rows >= 2u * warps || M > 2) return launch_f16_rows<M, 2>(ctx, a, smem, slices);
    return launch_f16_rows<M, 1>(ctx, a, smem, slices);
}

// out[c] = f32(w[row][c]) (* scale when non-zero); row < 0 writes zeros.
__device__ __forceinline__ void f16_row(const __half *w, uint32_t cols, long row, float scale, float *out) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (row >= 0) {
            v = __half2float(w[(size_t)row * cols + c]);
            if (scale != 0.0f) v *= scale;
        }
        out[c] = v;
    }
}
__global__ void f16_row_kernel(const __half *w, uint32_t cols, uint32_t row, float *out) {
    f16_row(w, cols, (long)row, 0.0f, out);
}
__global__ void f16_row_indirect_kernel(const __half *w, uint32_t rows, uint32_t cols, const uint32_t *ids, uint32_t slot,
                                        const uint32_t *pos, int bias, uint32_t ids_len, float scale, float *out) {
    tmdev::pdl_trigger();
    tmdev::pdl_wait();
    uint32_t s = slot;
    if (pos) s = slot + *pos + (uint32_t)bias;
    long row = -1;
    if (s < ids_len) {
        const uint32_t id = ids[s];
        if (id < rows) row = (long)id;
    }
    f16_row(w, cols, row, scale, out);
}
__global__ void f16_rows_gather_kernel(const __half *w, uint32_t rows, uint32_t cols, const uint32_t *ids,
                                       uint32_t first, float scale, float *out) {
    const uint32_t t = blockIdx.y, id = ids[first + t];
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (id < rows) {
            v = __half2float(w[(size_t)id * cols + c]);
            if (scale != 0.0f) v *= scale;
        }
        out[(size_t)t * cols + c] = v;
    }
}

int f16_common(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *x, tm_cuda_buffer *y, uint32_t rows, uint32_t cols,
               uint32_t batch, uint32_t x_off, uint32_t y_off, int prologue, tm_cuda_buffer *pro, float eps, int epilogue,
               const char *label, char *err, size_t err_cap) {
    if (rows == 0 || cols == 0)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "F16 geometry %u x %u", rows, cols);
    if (batch == 0 || batch > TM_CUDA_GEMM_MAX_BATCH)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "batch %u outside 1..%u", batch, TM_CUDA_GEMM_MAX_BATCH);
    TM_CHECK_AHEAD(w, (size_t)rows * cols * 2, "F16 weights");
    TM_CHECK_BUF(x, ((size_t)x_off + (size_t)batch * cols) * 4, "activation");
    TM_CHECK_BUF(y, ((size_t)y_off + (size_t)batch * rows) * 4, "output");
    if (prologue < TM_CUDA_PRO_NONE || prologue > TM_CUDA_PRO_GELU_MUL ||
        (epilogue != TM_CUDA_EPI_STORE && epilogue != TM_CUDA_EPI_ADD))
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "unknown prologue/epilogue");
    if (prologue == TM_CUDA_PRO_RMSNORM) TM_CHECK_IN(pro, (size_t)cols * 4, "norm weight");
    if (prologue == TM_CUDA_PRO_SILU_MUL || prologue == TM_CUDA_PRO_GELU_MUL)
        TM_CHECK_BUF(pro, (size_t)batch * cols * 4, "gate multiplicand");
    const size_t per_token = ((size_t)cols + 7u) / 8u * 32u, budget = ctx->smem_optin - 4096;
    if (per_token > budget)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "cols %u exceeds the activation stage of one CTA", cols);
    if (ctx->program)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "operator %s cannot be recorded into a persistent program", label);
    TM_OP_BEGIN(label);
    uint64_t kernels = 0;
    uint32_t done = 0;
    while (done < batch) {
        int m = 8;
        while (m > 1 && ((uint32_t)m > batch - done || (size_t)m * per_token > budget)) m >>= 1;
        f16_args a;
        a.w = (const __half *)w->dev;
        a.x = (const float *)x->dev + x_off + (size_t)done * cols;
        a.y = (float *)y->dev + y_off + (size_t)done * rows;
        a.pro = pro ? (const float *)pro->dev : nullptr;
        if (pro && (prologue == TM_CUDA_PRO_SILU_MUL || prologue == TM_CUDA_PRO_GELU_MUL)) a.pro += (size_t)done * cols;
        a.rows = rows;
        a.cols = cols;
        a.eps = eps;
        a.prologue = prologue;
        a.epilogue = epilogue;
        const size_t smem = (size_t)m * per_token;
        const uint32_t slices = m > 1 ? (batch - done) / (uint32_t)m : 1u;
        cudaError_t e = m == 8   ? launch_f16<8>(ctx, a, smem, slices)
                        : m == 4 ? launch_f16<4>(ctx, a, smem, slices)
                        : m == 2 ? launch_f16<2>(ctx, a, smem, slices)
                                 : launch_f16<1>(ctx, a, smem, 1u);
        if (e != cudaSuccess)
            return tm_fail(err, err_cap, TM_CUDA_ERR_INTERNAL, "F16 GEMV launch failed: %s", cudaGetErrorString(e));
        kernels += 1;
        done += (uint32_t)m * slices;
    }
    TM_OP_END(kernels);
}

}  // namespace

extern "C" {

int tm_cuda_f16_gemv(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *x, tm_cuda_buffer *y, uint32_t rows, uint32_t cols,
                     char *err, size_t err_cap) {
    TM_ENTER();
    return f16_common(ctx, w, x, y, rows, cols, 1, 0, 0, TM_CUDA_PRO_NONE, nullptr, 0.0f, TM_CUDA_EPI_STORE, "f16_gemv", err,
                      err_cap);
}

int tm_cuda_f16_gemm(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *x, tm_cuda_buffer *y, uint32_t rows, uint32_t cols,
                     uint32_t batch, uint32_t x_off, uint32_t y_off, char *err, size_t err_cap) {
    TM_ENTER();
    return f16_common(ctx, w, x, y, rows, cols, batch, x_off, y_off, TM_CUDA_PRO_NONE, nullptr, 0.0f, TM_CUDA_EPI_STORE,
                      "f16_gemm", err, err_cap);
}

int tm_cuda_f16_gemv_fused(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *x, tm_cuda_buffer *y, uint32_t rows,
                           uint32_t cols, int prologue, tm_cuda_buffer *pro, float eps, int epilogue, char *err,
                           size_t err_cap) {
    TM_ENTER();
    return f16_common(ctx, w, x, y, rows, cols, 1, 0, 0, prologue, pro, eps, epilogue, "f16_gemv_fused", err, err_cap);
}

int tm_cuda_f16_row_f32(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *out, uint32_t row, uint32_t cols,
                        uint32_t out_off, char *err, size_t err_cap) {
    TM_ENTER();
    if (cols == 0) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "F16 row of zero columns");
    TM_CHECK_IN(w, ((size_t)row + 1) * cols * 2, "F16 weights");
    TM_CHECK_BUF(out, ((size_t)out_off + cols) * 4, "row output");
    TM_OP_BEGIN("f16_row");
    f16_row_kernel<<<(cols + 255) / 256, 256, 0, ctx->stream>>>((const __half *)w->dev, cols, row,
                                                                 (float *)out->dev + out_off);
    TM_OP_END(1);
}

int tm_cuda_f16_row_indirect_f32_dev(tm_cuda_ctx *ctx, tm_cuda_buffer *w, uint32_t rows, uint32_t cols, tm_cuda_buffer *ids,
                                     uint32_t base, tm_cuda_buffer *pos_buf, uint32_t pos_index, int32_t bias, float scale,
                                     tm_cuda_buffer *out, char *err, size_t err_cap) {
    TM_ENTER();
    if (rows == 0 || cols == 0) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "F16 geometry %u x %u", rows, cols);
    TM_CHECK_IN(w, (size_t)rows * cols * 2, "F16 weights");
    TM_CHECK_BUF(ids, ((size_t)base + 1) * 4, "token ids");
    TM_CHECK_BUF(out, (size_t)cols * 4, "row output");
    const uint32_t *pos = nullptr;
    if (pos_buf) {
        TM_CHECK_BUF(pos_buf, ((size_t)pos_index + 1) * 4, "position");
        pos = (const uint32_t *)pos_buf->dev + pos_index;
    }
    TM_OP_BEGIN("f16_row_indirect");
    TM_CUDA_TRY(tm_launch_pdl(ctx, f16_row_indirect_kernel, dim3((cols + 255) / 256), dim3(256), 0, (const __half *)w->dev,
                              rows, cols, (const uint32_t *)ids->dev, base, pos, (int)bias, (uint32_t)(ids->len / 4), scale,
                              (float *)out->dev));
    TM_OP_END(1);
}

int tm_cuda_f16_rows_indirect_f32(tm_cuda_ctx *ctx, tm_cuda_buffer *w, uint32_t rows, uint32_t cols, tm_cuda_buffer *ids,
                                  uint32_t first, uint32_t n, float scale, tm_cuda_buffer *out, char *err, size_t err_cap) {
    TM_ENTER();
    if (rows == 0 || cols == 0) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "F16 geometry %u x %u", rows, cols);
    if (n == 0 || n > 65535u) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "row count %u outside 1..65535", n);
    TM_CHECK_IN(w, (size_t)rows * cols * 2, "F16 weights");
    TM_CHECK_BUF(ids, ((size_t)first + n) * 4, "token ids");
    TM_CHECK_BUF(out, (size_t)n * cols * 4, "rows output");
    TM_OP_BEGIN("f16_rows_indirect");
    f16_rows_gather_kernel<<<dim3((cols + 255) / 256, n), 256, 0, ctx->stream>>>(
        (const __half *)w->dev, rows, cols, (const uint32_t *)ids->dev, first, scale, (float *)out->dev);
    TM_OP_END(1);
}

}  // extern "C"
