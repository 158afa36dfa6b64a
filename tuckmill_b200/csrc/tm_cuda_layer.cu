// A decode token's layer in two launches: the attention block (residual add, norm, q|k|v, attention, o) and the
// feed-forward block (residual add, norm, gate|up, activation, down).
//
// What bounds a one-sequence step of a small decoder is the chain of its operators, not their bytes: a 0.6B decoder
// streams 633 MB per token (0.1 ms) but took 0.7 ms as five launches per layer, each 3-6 us of launch, activation
// load, norm + digit split, products, cross-warp sum and completion.  Here the operators that only exchange a few
// hundred values meet inside a cluster of 16 CTAs through distributed shared memory:
//   * cluster h of the attention block owns KV head h: its q, k and v rows, its keys, and the columns of o that its
//     heads feed; cluster c of the feed-forward block owns an eighth of the FFN width: its gate and up rows and its
//     columns of down.  Both end in one full-width partial product per cluster, a "slot";
//   * the slots are added (in order) to the residual stream by whoever reads it next, as the first thing its CTAs do
//     anyway; one cluster also stores the sum.  A layer's output norm is applied there too;
//   * weights never wait for activations: every warp copies its own 16-row x 64-column pieces of both projections to
//     shared memory before the dependency wait; both blocks' CTAs fit on an SM together, so a block's weights arrive
//     while the block before it computes.  (Only 7 of the 8 GPCs have the 16 SMs of a cluster: a block that fills more
//     than half an SM's shared memory runs its eighth cluster after the others, 20 us a layer instead of 11.)
// Products are the decode GEMV's (tm_cuda_q8.cu): int8 tensor-core MMAs on activations split into four 7-bit digits,
// exact sums per 32-column block.  How a row's columns are cut over warps, CTAs and clusters depends on the shape
// alone, and every sum has a fixed order.
#include "tm_cuda_attn_core.cuh"

namespace {

using namespace tmattn;

constexpr int kWarps = kT / 32;
constexpr uint32_t kSlotBytes = 1024u + 64u;  // 16 rows x 64 quants, 16 rows x 2 scales
constexpr uint32_t kC = 16;                   // CTAs per cluster
constexpr uint32_t kSlots = TM_CUDA_DECODE_SLOTS;
constexpr uint32_t kResident = 12;            // most pieces a warp keeps in shared memory

__host__ __device__ inline uint32_t plane_bytes(uint32_t cols) {  // 64 mod 128: the four digit planes hit distinct banks
    const uint32_t pad = (cols + 63u) & ~63u;
    return pad % 128u == 0u ? pad + 64u : pad;
}
__host__ __device__ inline uint32_t digit_bytes(uint32_t cols) { return (4u * plane_bytes(cols) + cols / 32u * 16u + 15u) & ~15u; }

__host__ __device__ inline uint32_t max_of(uint32_t a, uint32_t b) { return a > b ? a : b; }

struct residual_in {
    const float *x;       // [hidden]
    const float *slots;   // [n_slots][hidden] still to be added, or null
    const float *add_w;   // RMS norm weight of their sum (a layer's output norm), or null
    const float *norm_w;  // the block's own input norm
    float *x_out;         // the updated stream
    uint32_t n_slots, hidden;
    float eps;
};

using tmdev::mma_s8;

// Four consecutive columns of a vector into the digit planes (tmdev::digitise_quad; dead lanes with zeros).
__device__ __forceinline__ void digitise(const float (&v)[4], uint32_t c, bool live, unsigned char *dig, uint32_t plane) {
    tmdev::digitise_quad(v, live, (signed char *)dig + c, plane, (float *)(dig + 4u * plane) + (c >> 5) * 4u, threadIdx.x);
}

// Sum of every thread's value: one barrier (`red` is 8 floats no other sum between two barriers uses).
__device__ __forceinline__ float cta_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const float4 a = *(const float4 *)red, b = *(const float4 *)(red + 4);
    return ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
}

// x + [norm](sum of the slots), stored by cluster 0, then normed and split into digits: NB quads of columns per
// thread.  `red`: 16 floats.
template <int NB>
__device__ __forceinline__ void stage_residual(const residual_in &r, bool store, uint32_t rank, unsigned char *dig, float *red) {
    const uint32_t H = r.hidden, quads = H / 4u, plane = plane_bytes(H);
    const float inv_h = 1.0f / (float)H;
    float4 v[NB], nw[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        v[i] = nw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < quads) {
            v[i] = __ldcg((const float4 *)r.x + q);
            nw[i] = __ldg((const float4 *)r.norm_w + q);
        }
    }
    if (r.n_slots) {
        float4 p[NB], aw[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const uint32_t q = threadIdx.x + i * kT;
            p[i] = aw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q < quads) {
                if (r.add_w) aw[i] = __ldg((const float4 *)r.add_w + q);
                float4 s[kSlots];
#pragma unroll
                for (uint32_t k = 0; k < kSlots; ++k)
                    s[k] = k < r.n_slots ? __ldcg((const float4 *)(r.slots + (size_t)k * H) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (uint32_t k = 0; k < kSlots; ++k) {
                    p[i].x += s[k].x;
                    p[i].y += s[k].y;
                    p[i].z += s[k].z;
                    p[i].w += s[k].w;
                }
            }
        }
        if (r.add_w) {
            float sq = 0.0f;
#pragma unroll
            for (int i = 0; i < NB; ++i) sq = tmdev::sumsq_quad(sq, p[i]);
            const float inv = inv_sqrt(fmaf(cta_sum(sq, red + 8), inv_h, r.eps));
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                p[i].x = p[i].x * inv * aw[i].x;
                p[i].y = p[i].y * inv * aw[i].y;
                p[i].z = p[i].z * inv * aw[i].z;
                p[i].w = p[i].w * inv * aw[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            v[i].x += p[i].x;
            v[i].y += p[i].y;
            v[i].z += p[i].z;
            v[i].w += p[i].w;
        }
    }
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < NB; ++i) sq = tmdev::sumsq_quad(sq, v[i]);
    const float inv = inv_sqrt(fmaf(cta_sum(sq, red), inv_h, r.eps));
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        if ((q & ~31u) < quads) {
            const float y[4] = {v[i].x * inv * nw[i].x, v[i].y * inv * nw[i].y, v[i].z * inv * nw[i].z, v[i].w * inv * nw[i].w};
            digitise(y, q * 4u, q < quads, dig, plane);
        }
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        if (store && q < quads && q % kC == rank) ((float4 *)r.x_out)[q] = v[i];
    }
}

// One projection of a block as this CTA sees it: `tiles` 16-row tiles of `chunks` 64-column chunks, item i = tile
// i / chunks, chunk i % chunks; warp w multiplies items [w n / 8, (w + 1) n / 8) in order.
struct matrix_part {
    const signed char *q;
    const unsigned short *d;
    uint32_t cols, chunk0, tiles, chunks;
    __device__ __forceinline__ uint32_t first(uint32_t warp) const { return tiles * chunks * warp / kWarps; }
};

// A warp's weight pieces in shared memory: its items of the first projection, then those of the second, each one copy
// group with one wait.  Every lane copies, and later reads back, its own 16 bytes of rows g and g + 8 of a piece; the 32
// block scales ride along as 4-byte copies.  Every piece leaves its own partial sum: no bookkeeping between pieces (a
// commit, a wait and a running sum per piece cost more than 400 cycles each in a chain that multiplies six).
template <class RowOf1, class RowOf2>
struct weight_pieces {
    matrix_part m1, m2;
    RowOf1 row1;  // (tile, r): the weight row of row r of a tile
    RowOf2 row2;
    uint32_t base, slot;             // this warp's slots, the one consumed next
    const signed char *pa, *pb;      // next piece: this lane's bytes of rows g and g + 8
    const unsigned short *ps;        // and its scale pair
    uint32_t left_tile, left, tile;  // pieces left in the tile and in the projection, the tile's number
    bool second;

    __device__ __forceinline__ uint32_t lane() const { return threadIdx.x & 31u; }
    __device__ __forceinline__ uint32_t warp() const { return threadIdx.x >> 5; }

    __device__ __forceinline__ void point(const matrix_part &m, size_t ra, size_t rb, uint32_t chunk) {
        const uint32_t t4 = lane() & 3u, col = (m.chunk0 + chunk) * 64u;
        pa = m.q + ra * m.cols + col + t4 * 16u;
        pb = m.q + rb * m.cols + col + t4 * 16u;
        ps = m.d + ((t4 & 1u) ? rb : ra) * (m.cols / 32u) + col / 32u;
    }
    __device__ __forceinline__ void open_tile(uint32_t chunk) {
        const uint32_t g = lane() >> 2;
        if (second) point(m2, row2(tile, g), row2(tile, g + 8u), chunk);
        else point(m1, row1(tile, g), row1(tile, g + 8u), chunk);
        left_tile = (second ? m2.chunks : m1.chunks) - chunk;
    }
    __device__ __forceinline__ void open(bool sec) {
        second = sec;
        const uint32_t n = sec ? m2.chunks : m1.chunks;
        const uint32_t i0 = sec ? m2.first(warp()) : m1.first(warp());
        left = (sec ? m2.first(warp() + 1u) : m1.first(warp() + 1u)) - i0;
        tile = i0 / n;
        if (left) open_tile(i0 - tile * n);
    }
    // The next piece, if one is left, into slot `to`.
    __device__ __forceinline__ void issue(uint32_t to) {
        if (left) {
            const uint32_t dst = base + to * kSlotBytes, l = lane(), t4 = l & 3u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + l * 16u), "l"(pa) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512u + l * 16u), "l"(pb) : "memory");
            if (t4 < 2u)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 1024u + ((l >> 2) + 8u * t4) * 4u), "l"(ps) : "memory");
            pa += 64;
            pb += 64;
            ps += 2;
            if (--left != 0u && --left_tile == 0u) {
                ++tile;
                open_tile(0u);
            }
        }
    }
    static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    __device__ __forceinline__ void start(uint32_t ring) {
        base = ring;
        slot = 0;
        open(false);
#pragma unroll 1
        while (left) issue(slot++);
        commit();
        open(true);
#pragma unroll 1
        while (left) issue(slot++);
        commit();
        slot = 0;
    }
    // One piece: this lane's digits' share of rows g (x) and g + 8 (y).
    __device__ __forceinline__ float2 piece(uint32_t at, const unsigned char *dig, uint32_t plane, uint32_t ch) const {
        const uint32_t l = lane(), g = l >> 2, t4 = l & 3u, src = base + at * kSlotBytes, c0 = ch * 64u + t4 * 16u;
        int4 qa, qb;
        unsigned short sa, sb;
        asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(qa.x), "=r"(qa.y), "=r"(qa.z), "=r"(qa.w) : "r"(src + l * 16u));
        asm volatile("ld.shared.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(qb.x), "=r"(qb.y), "=r"(qb.z), "=r"(qb.w) : "r"(src + 512u + l * 16u));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sa) : "r"(src + 1024u + g * 4u + (t4 >> 1) * 2u));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sb) : "r"(src + 1056u + g * 4u + (t4 >> 1) * 2u));
        int4 bx = make_int4(0, 0, 0, 0);
        if ((t4 >> 1) == (g >> 2)) bx = *(const int4 *)(dig + (size_t)(g & 3u) * plane + c0);
        const float2 cx = *(const float2 *)(dig + 4u * plane + ((size_t)(c0 >> 5) * 4u + 2u * (t4 & 1u)) * 4u);
        int dd[4] = {0, 0, 0, 0};
        mma_s8(dd, qa.x, qb.x, qa.y, qb.y, bx.x, bx.y);
        mma_s8(dd, qa.z, qb.z, qa.w, qb.w, bx.z, bx.w);
        return make_float2(__half2float(__ushort_as_half(sa)) * fmaf((float)dd[1], cx.y, (float)dd[0] * cx.x),
                           __half2float(__ushort_as_half(sb)) * fmaf((float)dd[3], cx.y, (float)dd[2] * cx.x));
    }
    // This warp's pieces of one projection: piece i leaves its sums in part[i][16 rows].
    __device__ __forceinline__ void multiply(const matrix_part &m, bool sec, const unsigned char *dig, uint32_t plane, float *part) {
        const uint32_t l = lane(), g = l >> 2, t4 = l & 3u, i0 = m.first(warp()), end = m.first(warp() + 1u);
        uint32_t ch = i0 % m.chunks;
        if (sec) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();  // scales were copied by other lanes
#pragma unroll 1
        for (uint32_t i = i0; i < end; i += 3u) {
            float2 v[3];
#pragma unroll
            for (uint32_t k = 0; k < 3u; ++k) {
                v[k] = make_float2(0.0f, 0.0f);
                if (i + k < end) v[k] = piece(slot + k, dig, plane, ch);
                ch = ch + 1u == m.chunks ? 0u : ch + 1u;
            }
            slot += min(3u, end - i);
#pragma unroll
            for (uint32_t k = 0; k < 3u; ++k) {
                v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 1);
                v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 1);
                v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 2);
                v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 2);
                if (t4 == 0u && i + k < end) {
                    part[(i + k) * 16u + g] = v[k].x;
                    part[(i + k) * 16u + g + 8u] = v[k].y;
                }
            }
        }
    }
};

// Row r of tile t: the sum over the tile's pieces, by one thread (row_sum) or by the 16 lanes of half a warp, which all
// receive it (half_sum).
__device__ __forceinline__ float row_sum(const float *part, const matrix_part &m, uint32_t t, uint32_t r) {
    float v = 0.0f;
#pragma unroll 4
    for (uint32_t k = 0; k < m.chunks; ++k) v += part[(t * m.chunks + k) * 16u + r];
    return v;
}
__device__ __forceinline__ float half_sum(const float *part, const matrix_part &m, uint32_t t, uint32_t r) {
    float v = 0.0f;
    for (uint32_t k = threadIdx.x & 15u; k < m.chunks; k += 16u) v += part[(t * m.chunks + k) * 16u + r];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------- feed-forward block ----------------
struct ffn_args {
    residual_in in;
    const signed char *gu_q, *dn_q;          // [2 width][hidden], [hidden][width]
    const unsigned short *gu_d, *dn_d;
    float *slots_out;                        // [clusters][hidden]
    uint32_t width, gelu, tiles1, tiles2, acts;  // most tiles / activations a CTA / cluster has
};

// Shared memory: digits of x, digits of the activations, activations, partial sums, ring.
struct ffn_smem {
    uint32_t dig2, acts, part, red, ring, bytes;
};
__host__ __device__ inline ffn_smem ffn_layout(uint32_t hidden, uint32_t acts, uint32_t tiles1, uint32_t tiles2, uint32_t slots) {
    ffn_smem s;
    s.dig2 = digit_bytes(hidden);
    s.acts = s.dig2 + digit_bytes(acts);
    s.part = s.acts + acts * 4u;
    s.red = s.part + 64u * max_of(tiles1 * (hidden / 64u), tiles2 * (acts / 64u));
    s.ring = s.red + 64u;
    s.bytes = s.ring + kWarps * slots * kSlotBytes;
    return s;
}

template <int NB>
__global__ void __launch_bounds__(kT, 2) ffn_block_kernel(const ffn_args a, uint32_t ring_slots) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t rank = cluster_rank(), cluster = blockIdx.x / kC, n_clusters = gridDim.x / kC;
    const uint32_t H = a.in.hidden, F = a.width, chunks = F / 64u;
    const uint32_t fc0 = chunks * cluster / n_clusters, nfc = chunks * (cluster + 1u) / n_clusters - fc0;  // FFN chunks
    const uint32_t groups = nfc * 8u;                  // of 8 gate rows and the 8 up rows they gate: one tile
    const uint32_t g0 = groups * rank / kC, n1 = groups * (rank + 1u) / kC - g0;
    const uint32_t row_tiles = H / 16u, t0 = row_tiles * rank / kC, n2 = row_tiles * (rank + 1u) / kC - t0;
    const ffn_smem L = ffn_layout(H, a.acts, a.tiles1, a.tiles2, ring_slots);
    unsigned char *dig1 = smem, *dig2 = smem + L.dig2;
    float *acts = (float *)(smem + L.acts), *part = (float *)(smem + L.part), *red = (float *)(smem + L.red);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    cluster_arrive();
    auto row1 = [=](uint32_t tile, uint32_t r) -> size_t {
        return fc0 * 64u + (g0 + tile) * 8u + (r & 7u) + (r & 8u ? F : 0u);
    };
    auto row2 = [=](uint32_t tile, uint32_t r) -> size_t { return (t0 + tile) * 16u + r; };
    weight_pieces<decltype(row1), decltype(row2)> W = {
        {a.gu_q, a.gu_d, H, 0u, n1, H / 64u}, {a.dn_q, a.dn_d, F, fc0, n2, nfc}, row1, row2};
    W.start(smem_addr(smem + L.ring) + warp * ring_slots * kSlotBytes);
    tmdev::pdl_trigger();
    tmdev::pdl_wait();
    stage_residual<NB>(a.in, cluster == 0u, rank, dig1, red);
    __syncthreads();
    W.multiply(W.m1, false, dig1, plane_bytes(H), part);
    __syncthreads();
    cluster_wait();  // every CTA of the cluster has started
    // A warp finishes an activation: gate in its lower half, up in its upper; lane c of the lower half sends it to CTA c.
    for (uint32_t i = warp; i < n1 * 8u; i += kWarps) {
        const float sum = half_sum(part, W.m1, i >> 3, (i & 7u) + (lane & 16u) / 2u);
        const float up = __shfl_down_sync(0xffffffffu, sum, 16);
        const float v = (a.gelu ? tmdev::gelu_tanh_f(sum) : tmdev::silu_f(sum)) * up;
        if (lane < kC) st_cluster(smem_addr(acts + g0 * 8u + i), lane, v);
    }
    cluster_arrive();
    cluster_wait();
    for (uint32_t q = threadIdx.x; (q & ~31u) < nfc * 16u; q += kT) {
        const bool live = q < nfc * 16u;
        const float4 v = live ? *(const float4 *)(acts + q * 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float y[4] = {v.x, v.y, v.z, v.w};
        digitise(y, q * 4u, live, dig2, plane_bytes(a.acts));
    }
    __syncthreads();
    W.multiply(W.m2, true, dig2, plane_bytes(a.acts), part);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n2 * 16u; i += kT)
        a.slots_out[(size_t)cluster * H + t0 * 16u + i] = row_sum(part, W.m2, i >> 4, i & 15u);
}

// ---------------- attention block ----------------
struct attn_block_args {
    residual_in in;
    const signed char *qkv_q, *o_q;          // [(heads + 2 kv_heads) HD][hidden], [hidden][heads HD]
    const unsigned short *qkv_d, *o_d;
    const float *q_norm, *k_norm, *inv_freq;
    __half *kc, *vc;
    const uint32_t *pos;
    uint32_t *status;
    float *slots_out;                        // [kv_heads][hidden]
    uint32_t kv_heads, cap, window, tiles1, tiles2;
    float scale;
};

struct attn_smem {
    uint32_t dig2, state, qkv, recv, recv_ml, wgt, part, red, ring, bytes;
};
template <int G, int HD>
__host__ __device__ inline attn_smem attn_layout(uint32_t hidden, uint32_t tiles1, uint32_t tiles2, uint32_t slots) {
    attn_smem s;
    s.dig2 = digit_bytes(hidden);
    s.state = s.dig2 + digit_bytes(G * HD);
    s.qkv = s.state + (uint32_t)((sizeof(shared_state<G, HD>) + 15u) & ~15u);
    s.recv = s.qkv + (G + 2) * HD * 4u;
    s.recv_ml = s.recv + kC * G * HD * 4u;
    s.wgt = s.recv_ml + kC * G * 2u * 4u;
    s.part = s.wgt + kC * G * 4u;
    s.red = s.part + 64u * max_of(tiles1 * (hidden / 64u), tiles2 * (G * HD / 64u));
    s.ring = s.red + 64u;
    s.bytes = s.ring + kWarps * slots * kSlotBytes;
    return s;
}

template <int G, int HD, int NB>
__global__ void __launch_bounds__(kT, HD > 128 ? 1 : 2) attn_block_kernel(const attn_block_args a, uint32_t ring_slots) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int EPL = HD / 32;
    constexpr uint32_t kTiles = (G + 2) * HD / 16u;  // of this KV head's q, k and v rows
    const uint32_t rank = cluster_rank(), kvh = blockIdx.x / kC, H = a.in.hidden, cap = a.cap;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, tid = threadIdx.x;
    const uint32_t u0 = kTiles * rank / kC, n1 = kTiles * (rank + 1u) / kC - u0;
    const uint32_t row_tiles = H / 16u, t0 = row_tiles * rank / kC, n2 = row_tiles * (rank + 1u) / kC - t0;
    const attn_smem L = attn_layout<G, HD>(H, a.tiles1, a.tiles2, ring_slots);
    unsigned char *dig1 = smem, *dig2 = smem + L.dig2;
    shared_state<G, HD> &sh = *(shared_state<G, HD> *)(smem + L.state);
    float *qkv = (float *)(smem + L.qkv), *recv = (float *)(smem + L.recv), *recv_ml = (float *)(smem + L.recv_ml);
    float *wgt = (float *)(smem + L.wgt), *part = (float *)(smem + L.part), *red = (float *)(smem + L.red);
    cluster_arrive();
    // Row r of tile t, counted over this head's q rows, then its k rows, then its v rows.
    const uint32_t kvw = a.kv_heads * HD;
    auto row1 = [=](uint32_t tile, uint32_t r) -> size_t {
        const uint32_t i = (u0 + tile) * 16u + r;
        return i < G * HD         ? kvh * (G * HD) + i
               : i < (G + 1) * HD ? kvw * G + kvh * HD + (i - G * HD)
                                  : kvw * (G + 1) + kvh * HD + (i - (G + 1) * HD);
    };
    auto row2 = [=](uint32_t tile, uint32_t r) -> size_t { return (t0 + tile) * 16u + r; };
    weight_pieces<decltype(row1), decltype(row2)> W = {
        {a.qkv_q, a.qkv_d, H, 0u, n1, H / 64u}, {a.o_q, a.o_d, kvw * G, kvh * (G * HD / 64u), n2, G * HD / 64u}, row1, row2};
    W.start(smem_addr(smem + L.ring) + warp * ring_slots * kSlotBytes);
    __half *kp = a.kc + (size_t)kvh * cap * HD, *vp = a.vc + (size_t)kvh * cap * HD;
    const volatile uint32_t *pos_p = a.pos;
    keys<G, HD> K;
    K.early(kp, vp, min(*pos_p, cap - 1u), a.window, kC, rank);
    tmdev::pdl_wait();
    tmdev::pdl_trigger();  // only now: see tm_cuda_attn_core.cuh
    const uint32_t pos = *pos_p;
    stage_residual<NB>(a.in, kvh == 0u, rank, dig1, red);
    if (pos >= cap) {  // uniform over the cluster; the pieces's copies land before the CTA's memory goes away
        if (tid == 0 && rank == 0) atomicOr(a.status, 1u);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        cluster_wait();
        return;
    }
    K.late(pos, a.window, kC, rank);
    float nw[EPL];  // warp g < G: query head g; warp G: the new key
    rotation<HD> rot;
    if (warp <= G) {
        const float *src = warp == G ? a.k_norm : a.q_norm;
#pragma unroll
        for (int r = 0; r < EPL; ++r) nw[r] = __ldg(src + lane + 32 * r);
        rot.set(a.inv_freq, pos);
    }
    __syncthreads();
    W.multiply(W.m1, false, dig1, plane_bytes(H), part);
    __syncthreads();
    cluster_wait();  // every CTA of the cluster has started
    // Half a warp finishes a row; its lane c sends it to CTA c.
    for (uint32_t i = warp * 2u + (lane >> 4); i < n1 * 16u; i += 2u * kWarps)
        st_cluster(smem_addr(qkv + u0 * 16u + i), lane & 15u, half_sum(part, W.m1, i >> 4, i & 15u));
    cluster_arrive();
    cluster_wait();
    // ---- every CTA has the head's q, k and v ----
    if (warp < G || (warp == G && K.lo <= pos && pos < K.hi)) {
        float x[EPL];
#pragma unroll
        for (int r = 0; r < EPL; ++r) x[r] = qkv[warp * HD + lane + 32 * r];
        norm_rope<HD>(x, nw, rot, a.in.eps);
#pragma unroll
        for (int r = 0; r < EPL; ++r) {
            const uint32_t e = lane + 32 * r;
            if (warp == G) {
                const __half hk = __float2half_rn(x[r]), hv = __float2half_rn(qkv[(G + 1) * HD + e]);
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
    __syncthreads();
    keys<G, HD>::combine(sh);
    // ---- this CTA's (max, sum, output) to every CTA: each needs all of the head's output for its rows of o ----
    for (uint32_t i = tid; i < G * HD; i += kT) {
        const float o = keys<G, HD>::value(sh, i);
        const uint32_t at = smem_addr(recv + rank * G * HD + i);
#pragma unroll
        for (uint32_t to = 0; to < kC; ++to) st_cluster(at, (to + warp) % kC, o);
    }
    for (uint32_t i = tid; i < kC * G * 2u; i += kT) {
        const uint32_t e = i % (2u * G);
        st_cluster(smem_addr(recv_ml + rank * 2u * G + e), i / (2u * G), sh.l[e % G][e / G]);
    }
    cluster_arrive();
    cluster_wait();
    if (warp < G) {  // weight of source CTA `lane` in head `warp`
        const float m = lane < kC ? recv_ml[lane * 2u * G + warp] : -INFINITY;
        float M = m;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        const float f = lane < kC ? expf(m - M) : 0.0f;  // a CTA without keys: exp(-inf) = 0
        float l = lane < kC ? f * recv_ml[lane * 2u * G + G + warp] : 0.0f;
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
        if (lane < kC) wgt[warp * kC + lane] = f / l;
    }
    __syncthreads();
    for (uint32_t q = tid; (q & ~31u) < G * HD / 4u; q += kT) {
        const bool live = q < G * HD / 4u;
        float y[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (live) {
            const float *wg = wgt + (q * 4u / HD) * kC;
#pragma unroll
            for (uint32_t s = 0; s < kC; ++s) {
                const float4 o = *(const float4 *)(recv + s * G * HD + q * 4u);
                const float f = wg[s];
                y[0] = fmaf(f, o.x, y[0]);
                y[1] = fmaf(f, o.y, y[1]);
                y[2] = fmaf(f, o.z, y[2]);
                y[3] = fmaf(f, o.w, y[3]);
            }
        }
        digitise(y, q * 4u, live, dig2, plane_bytes(G * HD));
    }
    __syncthreads();
    W.multiply(W.m2, true, dig2, plane_bytes(G * HD), part);
    __syncthreads();
    for (uint32_t i = tid; i < n2 * 16u; i += kT)
        a.slots_out[(size_t)kvh * H + t0 * 16u + i] = row_sum(part, W.m2, i >> 4, i & 15u);
}

// ---------------- launches ----------------
uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1u) / b; }

template <class Kernel>
cudaError_t allow_clusters(Kernel kernel, int smem_optin) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
    return e == cudaSuccess ? cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : e;
}

// Whether the current device holds a cluster of the kernel with this much shared memory (16 CTAs are more than the
// portable size); where there is no device, the shape alone decides.
template <class Kernel>
bool cluster_fits(Kernel kernel, size_t smem) {
    int dev = 0, optin = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kC);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kC;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const bool ok = smem <= (size_t)optin && allow_clusters(kernel, optin) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
    cudaGetLastError();
    return ok;
}

template <class Kernel, class Args>
cudaError_t launch_clusters(tm_cuda_ctx *ctx, Kernel kernel, std::atomic<bool> *attr_set, uint32_t clusters, size_t smem,
                            const Args &a, uint32_t ring_slots) {
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = allow_clusters(kernel, (int)ctx->smem_optin);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    return tm_launch_cluster_pdl(ctx, kC, kernel, dim3(clusters * kC), dim3(kT), smem, a, ring_slots);
}

template <int NB>
cudaError_t launch_ffn(tm_cuda_ctx *ctx, const ffn_args &a, uint32_t slots) {
    static std::atomic<bool> attr_set[64] = {};  // per device; contexts of a process share it
    return launch_clusters(ctx, ffn_block_kernel<NB>, attr_set, kSlots,
                           ffn_layout(a.in.hidden, a.acts, a.tiles1, a.tiles2, slots).bytes, a, slots);
}
template <int G, int HD, int NB>
cudaError_t launch_attn(tm_cuda_ctx *ctx, const attn_block_args &a, uint32_t slots) {
    static std::atomic<bool> attr_set[64] = {};
    return launch_clusters(ctx, attn_block_kernel<G, HD, NB>, attr_set, a.kv_heads,
                           attn_layout<G, HD>(a.in.hidden, a.tiles1, a.tiles2, slots).bytes, a, slots);
}
// q|k|v and o pieces of a warp.
uint32_t attn_items(uint32_t hidden, uint32_t g, uint32_t hd) {
    return ceil_div(ceil_div((g + 2) * hd / 16u, kC) * (hidden / 64u), kWarps) +
           ceil_div(ceil_div(hidden / 16u, kC) * (g * hd / 64u), kWarps);
}
template <int G, int HD>
void attn_tiles(uint32_t hidden, uint32_t &tiles1, uint32_t &tiles2) {
    tiles1 = ceil_div((G + 2) * HD / 16u, kC);
    tiles2 = ceil_div(hidden / 16u, kC);
}
template <int G, int HD>
cudaError_t launch_attn_any(tm_cuda_ctx *ctx, attn_block_args a) {
    const uint32_t H = a.in.hidden;
    attn_tiles<G, HD>(H, a.tiles1, a.tiles2);
    const uint32_t items = attn_items(H, G, HD);
    return H <= 1024u ? launch_attn<G, HD, 1>(ctx, a, items) : launch_attn<G, HD, 2>(ctx, a, items);
}
template <int G, int HD>
bool attn_fits(uint32_t hidden) {
    uint32_t t1, t2;
    attn_tiles<G, HD>(hidden, t1, t2);
    const size_t smem = attn_layout<G, HD>(hidden, t1, t2, attn_items(hidden, G, HD)).bytes;
    return hidden <= 1024u ? cluster_fits(attn_block_kernel<G, HD, 1>, smem) : cluster_fits(attn_block_kernel<G, HD, 2>, smem);
}

// A block serves layers whose weights' pieces all stay in shared memory (0.6B shape: 6 and 9 a warp).  A layer that has
// to stream them is bound by bytes, and eight warps on 128 SMs do not pull them fast enough (8B shape: feed-forward
// block 79 us against 49 as two launches, attention block 34 against 30; 1B shape: 24 against 21), or has few KV heads
// and leaves most of the machine without work (1B shape, one KV head: 26 us against 18).
bool attn_shape(uint32_t hidden, uint32_t heads, uint32_t kv_heads, uint32_t hd) {
    const uint32_t g = kv_heads ? heads / kv_heads : 0u;
    return hidden >= 64u && hidden % 64u == 0u && hidden <= 2048u && (hd == 128u || hd == 256u) && kv_heads >= 1u &&
           kv_heads <= kSlots && heads == g * kv_heads && (g == 1u || g == 2u || g == 4u) && attn_items(hidden, g, hd) <= kResident;
}
ffn_args ffn_shape(uint32_t hidden, uint32_t width) {
    ffn_args a = {};
    a.in.hidden = hidden;
    a.width = width;
    const uint32_t nfc = ceil_div(width / 64u, kSlots);
    a.acts = nfc * 64u;
    a.tiles1 = ceil_div(nfc * 8u, kC);
    a.tiles2 = ceil_div(hidden / 16u, kC);
    return a;
}
uint32_t ffn_items(const ffn_args &a) {
    return ceil_div(a.tiles1 * (a.in.hidden / 64u), kWarps) + ceil_div(a.tiles2 * (a.acts / 64u), kWarps);
}
bool ffn_shape_ok(uint32_t hidden, uint32_t width) {
    return hidden >= 64u && hidden % 64u == 0u && hidden <= 2048u && width % 64u == 0u && width / 64u >= kSlots &&
           ffn_items(ffn_shape(hidden, width)) <= kResident;
}

int check_residual(tm_cuda_ctx *ctx, residual_in &r, tm_cuda_buffer *x, tm_cuda_buffer *slots, uint32_t n_slots,
                   tm_cuda_buffer *add_w, tm_cuda_buffer *norm_w, tm_cuda_buffer *x_out, tm_cuda_buffer *slots_out,
                   uint32_t n_slots_out, uint32_t hidden, float eps, char *err, size_t err_cap) {
    const size_t slots_out_bytes = (size_t)n_slots_out * hidden * 4;
    TM_CHECK_BUF(slots_out, slots_out_bytes, "slots output");
    TM_CHECK_BUF(x, (size_t)hidden * 4, "x");
    TM_CHECK_BUF(x_out, (size_t)hidden * 4, "x output");
    TM_CHECK_AHEAD(norm_w, (size_t)hidden * 4, "norm weight");
    if (n_slots > kSlots) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "%u slots, at most %u", n_slots, kSlots);
    if (n_slots) TM_CHECK_BUF(slots, (size_t)n_slots * hidden * 4, "slots");
    if (add_w) TM_CHECK_AHEAD(add_w, (size_t)hidden * 4, "output norm weight");
    // Every cluster reads the stream, the slots and the weights while others may have finished.
    const size_t row = (size_t)hidden * 4;
    const struct {
        const tm_cuda_buffer *buf;
        size_t bytes;
        const char *name;
    } in[4] = {{x, row, "x"}, {n_slots ? slots : nullptr, n_slots * row, "slots_in"}, {norm_w, row, "norm_w"}, {add_w, row, "add_w"}},
      out[2] = {{x_out, row, "x_out"}, {slots_out, slots_out_bytes, "slots_out"}};
    for (const auto &o : out)
        for (const auto &i : in)
            if (i.buf && o.buf->dev < i.buf->dev + i.bytes && i.buf->dev < o.buf->dev + o.bytes)
                return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "%s must be a buffer other than %s (every cluster reads it)",
                               o.name, i.name);
    if (((size_t)x->dev | (size_t)x_out->dev | (size_t)norm_w->dev | (n_slots ? (size_t)slots->dev : 0) | (add_w ? (size_t)add_w->dev : 0)) & 15u)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "residual operands are not 16-byte aligned");
    r.x = (const float *)x->dev;
    r.slots = n_slots ? (const float *)slots->dev : nullptr;
    r.add_w = n_slots && add_w ? (const float *)add_w->dev : nullptr;
    r.norm_w = (const float *)norm_w->dev;
    r.x_out = (float *)x_out->dev;
    r.n_slots = n_slots;
    r.hidden = hidden;
    r.eps = eps;
    return TM_CUDA_OK;
}

}  // namespace

extern "C" {

int tm_cuda_decode_attn_block_supported(uint32_t hidden, uint32_t heads, uint32_t kv_heads, uint32_t head_dim, uint32_t n_rot) {
    if (n_rot != head_dim || !attn_shape(hidden, heads, kv_heads, head_dim)) return 0;
    switch ((heads / kv_heads) * 1000 + head_dim) {
        case 1128: return attn_fits<1, 128>(hidden);
        case 2128: return attn_fits<2, 128>(hidden);
        case 4128: return attn_fits<4, 128>(hidden);
        case 1256: return attn_fits<1, 256>(hidden);
        case 2256: return attn_fits<2, 256>(hidden);
        default: return attn_fits<4, 256>(hidden);
    }
}
int tm_cuda_decode_ffn_block_supported(uint32_t hidden, uint32_t width) {
    if (!ffn_shape_ok(hidden, width)) return 0;
    const ffn_args a = ffn_shape(hidden, width);
    const size_t smem = ffn_layout(hidden, a.acts, a.tiles1, a.tiles2, ffn_items(a)).bytes;
    return hidden <= 1024u ? cluster_fits(ffn_block_kernel<1>, smem) : cluster_fits(ffn_block_kernel<2>, smem);
}

int tm_cuda_decode_attn_block(tm_cuda_ctx *ctx, tm_cuda_buffer *x, tm_cuda_buffer *slots_in, uint32_t n_slots,
                              tm_cuda_buffer *add_w, tm_cuda_buffer *norm_w, tm_cuda_buffer *x_out, tm_cuda_buffer *qkv,
                              tm_cuda_buffer *o, tm_cuda_buffer *q_norm, tm_cuda_buffer *k_norm, tm_cuda_buffer *inv_freq,
                              tm_cuda_buffer *k_cache, tm_cuda_buffer *v_cache, tm_cuda_buffer *pos_buf, uint32_t pos_index,
                              tm_cuda_buffer *status, tm_cuda_buffer *slots_out, uint32_t hidden, uint32_t heads,
                              uint32_t kv_heads, uint32_t head_dim, uint32_t cap, uint32_t window, float eps, float scale,
                              char *err, size_t err_cap) {
    TM_ENTER();
    if (!attn_shape(hidden, heads, kv_heads, head_dim) || cap == 0)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "attention block of hidden %u, heads %u/%u of %u", hidden, heads,
                       kv_heads, head_dim);
    int rc = tm_check_packed(ctx, qkv, (heads + 2 * kv_heads) * head_dim, hidden, err, err_cap);
    if (rc == TM_CUDA_OK) rc = tm_check_packed(ctx, o, hidden, heads * head_dim, err, err_cap);
    attn_block_args a = {};
    if (rc == TM_CUDA_OK) rc = check_residual(ctx, a.in, x, slots_in, n_slots, add_w, norm_w, x_out, slots_out, kv_heads, hidden, eps, err, err_cap);
    if (rc != TM_CUDA_OK) return rc;
    const size_t plane = (size_t)kv_heads * cap * head_dim * 2;
    TM_CHECK_AHEAD(q_norm, (size_t)head_dim * 4, "q norm");
    TM_CHECK_AHEAD(k_norm, (size_t)head_dim * 4, "k norm");
    TM_CHECK_AHEAD(inv_freq, (size_t)(head_dim / 2) * 4, "inv_freq");
    TM_CHECK_IN(k_cache, plane, "k cache");
    TM_CHECK_IN(v_cache, plane, "v cache");
    TM_CHECK_BUF(pos_buf, ((size_t)pos_index + 1) * 4, "position");
    TM_CHECK_BUF(status, 4, "status");
    tm_read_cache_ahead(ctx, k_cache, (const uint32_t *)pos_buf->dev + pos_index);
    tm_read_cache_ahead(ctx, v_cache, (const uint32_t *)pos_buf->dev + pos_index);
    a.qkv_q = (const signed char *)qkv->qp;
    a.qkv_d = (const unsigned short *)qkv->dp;
    a.o_q = (const signed char *)o->qp;
    a.o_d = (const unsigned short *)o->dp;
    a.q_norm = (const float *)q_norm->dev;
    a.k_norm = (const float *)k_norm->dev;
    a.inv_freq = (const float *)inv_freq->dev;
    a.kc = (__half *)k_cache->dev;
    a.vc = (__half *)v_cache->dev;
    a.pos = (const uint32_t *)pos_buf->dev + pos_index;
    a.status = (uint32_t *)status->dev;
    a.slots_out = (float *)slots_out->dev;
    a.kv_heads = kv_heads;
    a.cap = cap;
    a.window = window;
    a.scale = scale;
    TM_OP_BEGIN("decode_attn_block");
    cudaError_t e = cudaErrorInvalidConfiguration;
    switch ((heads / kv_heads) * 1000 + head_dim) {
        case 1128: e = launch_attn_any<1, 128>(ctx, a); break;
        case 2128: e = launch_attn_any<2, 128>(ctx, a); break;
        case 4128: e = launch_attn_any<4, 128>(ctx, a); break;
        case 1256: e = launch_attn_any<1, 256>(ctx, a); break;
        case 2256: e = launch_attn_any<2, 256>(ctx, a); break;
        default: e = launch_attn_any<4, 256>(ctx, a); break;
    }
    TM_CUDA_TRY(e);
    TM_OP_END(1);
}

int tm_cuda_decode_ffn_block(tm_cuda_ctx *ctx, tm_cuda_buffer *x, tm_cuda_buffer *slots_in, uint32_t n_slots,
                             tm_cuda_buffer *add_w, tm_cuda_buffer *norm_w, tm_cuda_buffer *x_out, tm_cuda_buffer *gate_up,
                             tm_cuda_buffer *down, tm_cuda_buffer *slots_out, uint32_t hidden, uint32_t width, int gelu,
                             float eps, char *err, size_t err_cap) {
    TM_ENTER();
    if (!ffn_shape_ok(hidden, width))
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "feed-forward block of hidden %u, width %u", hidden, width);
    int rc = tm_check_packed(ctx, gate_up, 2 * width, hidden, err, err_cap);
    if (rc == TM_CUDA_OK) rc = tm_check_packed(ctx, down, hidden, width, err, err_cap);
    ffn_args a = ffn_shape(hidden, width);
    if (rc == TM_CUDA_OK) rc = check_residual(ctx, a.in, x, slots_in, n_slots, add_w, norm_w, x_out, slots_out, kSlots, hidden, eps, err, err_cap);
    if (rc != TM_CUDA_OK) return rc;
    a.gu_q = (const signed char *)gate_up->qp;
    a.gu_d = (const unsigned short *)gate_up->dp;
    a.dn_q = (const signed char *)down->qp;
    a.dn_d = (const unsigned short *)down->dp;
    a.slots_out = (float *)slots_out->dev;
    a.gelu = gelu ? 1u : 0u;
    const uint32_t items = ffn_items(a);
    TM_OP_BEGIN("decode_ffn_block");
    TM_CUDA_TRY(hidden <= 1024u ? launch_ffn<1>(ctx, a, items) : launch_ffn<2>(ctx, a, items));
    TM_OP_END(1);
}

}  // extern "C"
