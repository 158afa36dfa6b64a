// Decode attention, latency form: one token of each sequence against its cached keys and values, q / k RMS norm,
// RoPE and the f16 KV store folded in.  Tolerance-qualified (attention_decode_kernel in tm_cuda_ops.cu is the form
// that is bit-identical to the prefill kernel).
//
// What bounds it: a step's chain, not its bytes (a 0.6B decoder at position 700 reads 2.9 MB per layer).  A cluster
// of up to 16 CTAs serves the G query heads of one KV head; each CTA takes a contiguous run of the visible keys, 64
// at a time, and the CTAs' (max, sum, output) meet in distributed shared memory: every CTA pushes each peer the
// slice of value dims that peer finishes, and goes on when its own slice has arrived at a counted barrier.  The form this
// replaces met through a scratch buffer in HBM (store, fence, atomic, reload: three dependent memory trips) and
// launched a CTA per 64 positions of CAPACITY, each reading its rows before it knew whether they exist: 16.8 MB a
// layer at capacity 4096 and 8.9 us of the step at position 700, against 6.
// Code that runs once per launch comes from a cold instruction cache, so it is kept short and, where it can be, done
// before the dependency wait (rotation angles, later rows towards L2): 4 heads of 256 dims 11.5 -> 6.3 us after the
// wait, 4 of 128 at position 2060 11.4 -> 9, 2 of 128 4.9 -> 3.5.
#include "tm_cuda_attn_core.cuh"

namespace {

using namespace tmattn;

struct attn_args {
    const float *q, *k, *v, *q_norm, *k_norm, *inv_freq;
    __half *kc, *vc;
    float *out;
    const uint32_t *pos;
    uint32_t *status;
    uint32_t cap, window;
    float eps, scale;
    size_t sq, sk, sv, so, scache;  // elements between consecutive sequences
    tm_peer_waits waits;
};

template <int G, int HD>
__global__ void __launch_bounds__(kT, HD > 128 ? 1 : 2) attention_decode_cluster_kernel(const attn_args a) {
    constexpr int EPL = HD / 32;  // elements of a head vector per lane (strided by 32)
    constexpr uint32_t kQuads = G * HD / 4;
    static_assert(kQuads <= (uint32_t)kT, "a thread finishes one quad");
    __shared__ __align__(16) shared_state<G, HD> sh;
    __shared__ __align__(16) float recv[G * HD];                // [source CTA][this CTA's slice]
    __shared__ __align__(16) float recv_ml[kMaxCluster][G][2];  // every CTA's max and sum of the heads in the slice
    __shared__ __align__(8) uint64_t arrived;
    const uint32_t C = cluster_size(), rank = cluster_rank();
    const uint32_t kvh = blockIdx.x / C, seq_i = blockIdx.z, cap = a.cap;
    const int tid = threadIdx.x, lane = tid & 31, warp = tmdev::warp_index();
    // Quad i of the G HD values is finished by CTA i / E; C and E are powers of two.
    const uint32_t logc = 31u - (uint32_t)__clz((int)C), E = (uint32_t)(G * HD) >> logc;
    const uint32_t slice_heads = E > HD ? E / HD : 1u, bar = smem_addr(&arrived);
    if (tid == 0) tmdev::mbar_init(bar, C * (E * 4u + slice_heads * 8u) + a.waits.more(1u));
    cluster_arrive();  // before any peer's shared memory is written, every CTA must have started
    const float *q = a.q + seq_i * a.sq + (size_t)kvh * G * HD, *k = a.k + seq_i * a.sk + (size_t)kvh * HD;
    const float *v = a.v + seq_i * a.sv + (size_t)kvh * HD;
    __half *kp = a.kc + seq_i * a.scache + (size_t)kvh * cap * HD, *vp = a.vc + seq_i * a.scache + (size_t)kvh * cap * HD;
    const volatile uint32_t *pos_p = a.pos + seq_i;
    keys<G, HD> K;
    const uint32_t hint = tmdev::uniform(min(*pos_p, cap - 1u));
    K.early(kp, vp, hint, a.window, C, rank);
    rotation<HD> rot;  // as if the position stood already
    rot.set(a.inv_freq, hint);
    tmdev::pdl_wait();
    tmdev::pdl_trigger();
    // Warp g < G normalises and rotates query head g, warp G the new key; the loads go out with the position's.
    float x[EPL], w[EPL], vx[EPL];
    const bool is_k = warp == G;
    {
        const float *src = is_k ? k : q + (size_t)(warp < G ? warp : 0) * HD, *nw = is_k ? a.k_norm : a.q_norm;
#pragma unroll
        for (int r = 0; r < EPL; ++r) {
            x[r] = src[lane + 32 * r];
            w[r] = nw[lane + 32 * r];
            vx[r] = is_k ? v[lane + 32 * r] : 0.0f;
        }
    }
    const uint32_t pos = tmdev::uniform(*pos_p);
    if (pos >= cap) {  // uniform over the cluster
        if (tid == 0 && rank == 0) atomicOr(a.status, TM_CUDA_STATUS_PAST_CAPACITY);
        cluster_wait();
        return;
    }
    K.late(pos, a.window, C, rank);
    if (warp < G || (is_k && K.lo <= pos && pos < K.hi)) {
        if (pos != hint) rot.set(a.inv_freq, pos);
        norm_rope<HD>(x, w, rot, a.eps);
#pragma unroll
        for (int r = 0; r < EPL; ++r) {
            const uint32_t e = lane + 32 * r;
            if (is_k) {
                const __half hk = __float2half_rn(x[r]), hv = __float2half_rn(vx[r]);
                sh.kh[e] = hk;
                sh.vh[e] = hv;
                kp[(size_t)pos * HD + e] = hk;
                vp[(size_t)pos * HD + e] = hv;
            } else {
                sh.qs[warp][e] = x[r];
            }
        }
    }
    __syncthreads();
    K.attend(sh, pos, a.scale);
    cluster_wait();  // every CTA of the cluster has started
    __syncthreads();
    // ---- a quad of this CTA's values to the CTA that finishes it, the maximum and sum once a slice and head ----
    if ((uint32_t)warp * 32u < kQuads) {
        const uint32_t i = (uint32_t)tid * 4u, in = i & (E - 1u), to = i / E;
        float4 o;
        const float2 ml = keys<G, HD>::combined(sh, i / HD, i % HD, o);
        tmdev::send(smem_addr(&recv[rank * E + in]), bar, to, o);
        if ((in & (HD - 1u)) == 0u) tmdev::send(smem_addr(&recv_ml[rank][in / HD][0]), bar, to, ml);
    }
    if (__all_sync(0xffffffffu, tmdev::mbar_wait(bar, a.waits.limit(), a.status, TM_CUDA_STATUS_LATE))) {
        // ---- C lanes per quad: source s's share, added over the lanes ----
        if ((uint32_t)warp * 32u >= kQuads) return;
        const uint32_t src = tid & (C - 1u), in = ((uint32_t)tid >> logc) * 4u;
        const float M = recv_ml[src][in / HD][0];
        float L = recv_ml[src][in / HD][1];
        float4 O = *(const float4 *)&recv[src * E + in];
        float top = M;
#pragma unroll 1
        for (uint32_t off = C >> 1; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
        const float f = expf(M - top);  // a CTA without keys: exp(-inf) = 0
        L *= f, O.x *= f, O.y *= f, O.z *= f, O.w *= f;
#pragma unroll 1
        for (uint32_t off = C >> 1; off > 0; off >>= 1) {
            L += __shfl_xor_sync(0xffffffffu, L, off);
            O.x += __shfl_xor_sync(0xffffffffu, O.x, off);
            O.y += __shfl_xor_sync(0xffffffffu, O.y, off);
            O.z += __shfl_xor_sync(0xffffffffu, O.z, off);
            O.w += __shfl_xor_sync(0xffffffffu, O.w, off);
        }
        if (src == 0) {
            float *out = a.out + seq_i * a.so + (size_t)kvh * G * HD + rank * E + in;
            const float d[4] = {O.x / L, O.y / L, O.z / L, O.w / L};
#pragma unroll
            for (int r = 0; r < 4; ++r) out[r] = d[r];
        }
        return;
    }
    if (lane == 0) atomicOr(a.status, TM_CUDA_STATUS_LATE);  // (behind the code of every call)
    tmdev::linger(bar);
}

// The widest cluster this device can hold of the kernel (16 needs the non-portable size).
template <int G, int HD>
uint32_t max_cluster(int device) {
    static std::atomic<uint32_t> known[64] = {};
    if (device >= 0 && device < 64)
        if (const uint32_t c = known[device].load(std::memory_order_acquire)) return c;
    uint32_t c = 8;
    if (cudaFuncSetAttribute(attention_decode_cluster_kernel<G, HD>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMaxCluster);
        cfg.blockDim = dim3(kT);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kMaxCluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, attention_decode_cluster_kernel<G, HD>, &cfg) == cudaSuccess && n > 0)
            c = kMaxCluster;
    }
    cudaGetLastError();
    if (device >= 0 && device < 64) known[device].store(c, std::memory_order_release);
    return c;
}

template <int G, int HD>
cudaError_t launch(tm_cuda_ctx *ctx, const attn_args &a, uint32_t kv_heads, uint32_t n_seq) {
    // As many CTAs per KV head as keep the launch within two resident waves, a power of two.
    uint32_t c = max_cluster<G, HD>(ctx->device);
    while (c > 1u && (uint64_t)c * kv_heads * n_seq > 2ull * (uint32_t)ctx->sm_count) c >>= 1;
    return tm_launch_cluster_pdl(ctx, c, attention_decode_cluster_kernel<G, HD>, dim3(c * kv_heads, 1, n_seq), dim3(kT), 0, a);
}

}  // namespace

bool tm_attention_decode_fast_ok(uint32_t heads, uint32_t kv_heads, uint32_t hd, uint32_t n_rot) {
    const uint32_t g = heads / kv_heads;
    return (hd == 128 || hd == 256) && n_rot == hd && (g == 1 || g == 2 || g == 4);
}

cudaError_t tm_attention_decode_fast_launch(tm_cuda_ctx *ctx, const float *q, const float *k, const float *v,
                                            const float *qn, const float *kn, const float *inv_freq, void *kc, void *vc,
                                            float *out, const uint32_t *pos, uint32_t *status, uint32_t heads,
                                            uint32_t kv_heads, uint32_t hd, uint32_t cap, uint32_t window, float eps,
                                            float scale, uint32_t n_seq, size_t sq, size_t skv, size_t so, size_t scache) {
    attn_args a = {q, k, v, qn, kn, inv_freq, (__half *)kc, (__half *)vc, out, pos, status, cap, window, eps, scale,
                   sq, skv, skv, so, scache, ctx->waits};
    switch ((heads / kv_heads) * 1000 + hd) {
        case 1128: return launch<1, 128>(ctx, a, kv_heads, n_seq);
        case 2128: return launch<2, 128>(ctx, a, kv_heads, n_seq);
        case 4128: return launch<4, 128>(ctx, a, kv_heads, n_seq);
        case 1256: return launch<1, 256>(ctx, a, kv_heads, n_seq);
        case 2256: return launch<2, 256>(ctx, a, kv_heads, n_seq);
        default: return launch<4, 256>(ctx, a, kv_heads, n_seq);
    }
}
