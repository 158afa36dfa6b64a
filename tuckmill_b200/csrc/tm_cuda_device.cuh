// Device helpers shared by the kernel translation units.
#pragma once
#include <cuda_runtime.h>

namespace tmdev {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// A value that all lanes of the (whole, converged) warp hold, told to the compiler: it then knows that a branch on it
// keeps the warp together.  Behind a branch that may split the warp, every shuffle is compiled twice, the second time
// with the code that gathers the lanes first.
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ uint32_t warp_index() { return uniform(threadIdx.x >> 5); }

// Canonical sum of squares of a vector, shared by every kernel that computes an
// RMS norm so all of them produce the same bits:
//   * elements are taken in quads; quad Q belongs to thread Q % 256, which adds
//     its quads in increasing order, x*x folded in with one FMA per element;
//   * each warp adds its 32 partials with a xor butterfly (16, 8, 4, 2, 1);
//   * the 8 warp sums are added in order 0..7.
__device__ __forceinline__ float sumsq_quad(float s, const float4 v) {
    s = fmaf(v.x, v.x, s);
    s = fmaf(v.y, v.y, s);
    s = fmaf(v.z, v.z, s);
    s = fmaf(v.w, v.w, s);
    return s;
}

// Quad `quad` of x[0..n) (zeros past the end); vector load when `vec`.
__device__ __forceinline__ float4 load_quad(const float *x, uint32_t n, uint32_t quad, bool vec) {
    const uint32_t e = quad * 4u;
    if (vec) return *(const float4 *)(x + e);
    float4 v;
    v.x = e < n ? x[e] : 0.0f;
    v.y = e + 1 < n ? x[e + 1] : 0.0f;
    v.z = e + 2 < n ? x[e + 2] : 0.0f;
    v.w = e + 3 < n ? x[e + 3] : 0.0f;
    return v;
}

__device__ __forceinline__ bool quads_vectorizable(const float *x, uint32_t n) {
    return (((size_t)x) & 15u) == 0 && (n & 3u) == 0;
}

// Warp butterfly + ordered sum over the CTA's 8 warps of per-thread partials.
static __device__ float block_reduce_sumsq(float s, float *red /* [kWarps] */) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) t += red[w];
    return t;
}

static __device__ float block_sumsq(const float *x, uint32_t n, float *red /* [kWarps] */) {
    const bool vec = quads_vectorizable(x, n);
    const uint32_t quads = (n + 3u) / 4u;
    float s = 0.0f;
#pragma unroll 2
    for (uint32_t q0 = warp_index() * 32u; q0 < quads; q0 += kThreads) {
        const uint32_t q = q0 + (threadIdx.x & 31u);
        if (q < quads) s = sumsq_quad(s, load_quad(x, n, q, vec));
    }
    return block_reduce_sumsq(s, red);
}

// Programmatic dependent launch: a kernel launched with the stream-serialization
// attribute may start while its predecessor still runs.  `pdl_wait` blocks until
// the predecessor has completed and its writes are visible (a no-op for an
// ordinary launch); `pdl_trigger` lets the successor start launching.  Before the
// wait a kernel reads only operands that nothing in flight writes: its entry point
// says which (TM_CHECK_AHEAD in tm_cuda_internal.cuh).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

__device__ __forceinline__ float silu_f(float g) { return g / (1.0f + expf(-g)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
    const float inner = 0.7978845608028654f * x * (1.0f + 0.044715f * x * x);
    return 0.5f * x * (1.0f + tanhf(inner));
}

// D += A(16x32 s8, row) * B(32x8 s8, col), s32 accumulate.
__device__ __forceinline__ void mma_s8(int (&d)[4], int a0, int a1, int a2, int a3, int b0, int b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D += A(16x16 f16, row) * B(16x8 f16, col), f32 accumulate.
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Four consecutive values of a thread as digits (at `dst` of each plane, unless the thread is past the row); eight
// adjacent lanes own a 32-column block, whose four coefficients 2^(e - 7k) go to `coef`.  Whole warps call it.
// (`shift` > 0: 2^shift adjacent lanes hold the same four values.)
__device__ __forceinline__ void digitise_quad(const float (&v)[4], bool live, signed char *dst, uint32_t plane, float *coef, uint32_t lane,
                                              uint32_t shift = 0) {
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j)  // a non-finite value poisons its block (amax = inf -> NaN coefficient)
        amax = fmaxf(amax, fabsf(v[j]) <= 3.402823466e38f ? fabsf(v[j]) : INFINITY);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1u << shift));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2u << shift));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4u << shift));
    if (!live) return;
    const bool bad = !(amax <= 3.402823466e38f);
    int e = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 127 - 5;
    e = e < -100 ? -100 : e > 122 ? 122 : e;  // blocks below 2^-94 digitise to (near) zero
    const float inv = __uint_as_float((uint32_t)(127 - e) << 23);
    // t = v * 2^-e (|t| < 64, exact) is rounded once to a multiple of 2^-21
    // and split into balanced base-128 digits with integer arithmetic:
    // T = a0 2^21 + a1 2^14 + a2 2^7 + a3, a1..a3 in [-64, 63].
    const float inv21 = inv * 2097152.0f;
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int T = __float2int_rn(v[j] * inv21);
#pragma unroll
        for (int k = 3; k > 0; --k) {
            const int d = (int)((uint32_t)T << 25) >> 25;
            T = (T - d) >> 7;
            w[k] |= ((uint32_t)d & 0xffu) << (8 * j);
        }
        w[0] |= ((uint32_t)T & 0xffu) << (8 * j);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) *(uint32_t *)(dst + k * plane) = w[k];
    const uint32_t k = (lane >> shift) & 7u;
    if (k < 4u) {
        const int ex = 127 + e - 7 * (int)k;  // 2^(e - 7k); below the normal range -> 0
        float sc = ex > 0 ? __uint_as_float((uint32_t)ex << 23) : 0.0f;
        if (amax == 0.0f) sc = 0.0f;
        if (bad) sc = __uint_as_float(0x7fc00000u);
        coef[k] = sc;
    }
}

// ---- thread-block clusters: the CTA's place, barriers, a peer's shared memory ----
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t v;
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(v));
    return v;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t v;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ float ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote));
    return v;
}


// ---- values sent to a peer's shared memory that arrive at a barrier of the peer's, counted in bytes ----
// A cluster barrier takes a release of everything a CTA has stored and the last CTA's arrival; a CTA that waits for the
// bytes it needs goes on as soon as they are there.
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t bytes) {  // one use: `bytes` will arrive
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, uint32_t rank, float v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(map_rank(addr, rank)), "f"(v),
                 "r"(map_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, uint32_t rank, float2 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(map_rank(addr, rank)),
                 "f"(v.x), "f"(v.y), "r"(map_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, uint32_t rank, float4 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(map_rank(addr, rank)),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(map_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ bool arrived(uint32_t bar) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n selp.b32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(bar) : "memory");
    return done != 0u;
}
// Waits for a barrier's one use, at most `limit` polls (of 4.4 us each while nothing arrives); false when they run out, or
// after 256 where `flag` has a bit of `mask`: a wait has failed already, and nothing that depends on it is worth the full time.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t limit, const volatile uint32_t *flag, uint32_t mask) {
#pragma unroll 1
    for (uint32_t i = 0; i < limit; ++i) {
        if (arrived(bar)) return true;
        if ((i & 255u) == 255u && (*flag & mask) != 0u) return false;
    }
    return false;
}
// After the peers have sent all they will: what is on its way lands (as far as a millisecond shows; what was never sent does not).
__device__ __forceinline__ void landed(uint32_t bar) {
#pragma unroll 1
    for (uint32_t i = 0; i < 256u && !arrived(bar); ++i) {
    }
}
// The end of a warp that has not received everything: its CTA's shared memory stays until the other warps of the cluster have met it here
// or have ended (a cluster barrier counts the threads that have not), and until what they had sent has landed.
__device__ __forceinline__ void linger(uint32_t bar) {
    __syncwarp();
    cluster_sync();
    landed(bar);
}

}  // namespace tmdev
