// A decode token's layer in two launches: the attention block (residual add, norm, q|k|v, attention, o) and the
// feed-forward block (residual add, norm, gate|up, activation, down).
//
// What bounds a one-sequence step of a small decoder is the chain of its operators, not their bytes: a 0.6B decoder
// streams 633 MB per token (0.1 ms) but took 0.7 ms as five launches per layer, each 3-6 us of launch, activation
// load, norm + digit split, products, cross-warp sum and completion.  Here the operators that only exchange a few
// hundred values meet inside a cluster of 16 CTAs through distributed shared memory:
//   * cluster h of the attention block owns KV head h: its q, k and v rows, its keys, and the columns of o that its
//     heads feed; cluster c of the feed-forward block owns a sixth (or an eighth, see ffn_shape) of the FFN width: its gate
//     and up rows and its columns of down.  Both end in one full-width partial product per cluster, a "slot";
//   * the slots are added (in order) to the residual stream by whoever reads it next, as the first thing its CTAs do
//     anyway; one cluster also stores the sum.  A layer's output norm is applied there too;
//   * weights never wait for activations: every warp copies its own 16-row x 64-column pieces of both projections to
//     shared memory before the dependency wait; both blocks' CTAs fit on an SM together, so a block's weights arrive
//     while the block before it computes.  Only 7 of the 8 GPCs have the 16 SMs of a cluster, so 14 clusters are in
//     flight at two CTAs an SM: eight of attention (a KV head each) and six of feed-forward.  With eight of each the last
//     two of a block started when the block before it had gone, and loaded their weights after that (0.6B shape, 512 +
//     256 tokens: 138.3 -> 134.7 ms, although a warp multiplies 12 pieces instead of 9).
//   * the code is short, because every launch runs it once: a chain of two kernels of 66 and 33 KB never finds it in
//     an SM's 32 KB instruction cache.  Both projections go through the same digit split and products (one loop of two
//     turns), and branches are on values that the compiler knows to be the same in a warp (tmdev::uniform): behind
//     others it repeats every shuffle in a form that gathers the lanes first, 200 cycles each instead of 30.  From the
//     dependency wait on, attention 23.0 -> 17.7 thousand cycles, feed-forward 13.1 -> 10.4 (143.8 -> 138.3 ms).
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
constexpr uint32_t kFfnClusters = 6;          // where a warp can keep its pieces, else kSlots
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
    uint32_t *late;       // set when an exchange inside a cluster did not arrive
    uint32_t n_slots, hidden;
    float eps;
    tm_peer_waits waits;
};

using tmdev::mma_s8;

// Sum of every thread's value: one barrier (`red` is 8 floats no other sum between two barriers uses).
__device__ __forceinline__ float cta_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const float4 a = *(const float4 *)red, b = *(const float4 *)(red + 4);
    return ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
}

// The weights of the input norm, asked for before the dependency wait.  (What is left of the residual, 3 thousand cycles,
// is 128 CTAs that ask for the same 36 KB.)
template <int NB>
__device__ __forceinline__ void norm_weights(const residual_in &r, float4 (&nw)[NB]) {
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        nw[i] = q < r.hidden / 4u ? __ldg((const float4 *)r.norm_w + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
// v = rmsnorm(x + [norm](sum of the slots)): NB quads of columns per thread, the sum stored by cluster 0.  `red`: 16
// floats.  `meanwhile` runs while the loads are on their way.
template <int NB, class F>
__device__ __forceinline__ void residual_norm(const residual_in &r, bool store, uint32_t rank, const float4 (&nw)[NB], float4 (&v)[NB],
                                              float *red, F meanwhile) {
    const uint32_t H = r.hidden, quads = H / 4u;
    const float inv_h = 1.0f / (float)H;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        v[i] = q < quads ? __ldcg((const float4 *)r.x + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float4 p[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        float4 s[kSlots];
#pragma unroll
        for (uint32_t k = 0; k < kSlots; ++k)
            s[k] = q < quads && k < r.n_slots ? __ldcg((const float4 *)(r.slots + (size_t)k * H) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (i == 0) meanwhile();
        p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (uint32_t k = 0; k < kSlots; ++k) {
            p[i].x += s[k].x;
            p[i].y += s[k].y;
            p[i].z += s[k].z;
            p[i].w += s[k].w;
        }
    }
    if (r.n_slots) {
        if (r.add_w) {
            float sq = 0.0f;
#pragma unroll
            for (int i = 0; i < NB; ++i) sq = tmdev::sumsq_quad(sq, p[i]);
            const float inv = inv_sqrt(fmaf(cta_sum(sq, red + 8), inv_h, r.eps));
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const uint32_t q = threadIdx.x + i * kT;
                const float4 aw = q < quads ? __ldg((const float4 *)r.add_w + q) : make_float4(0.f, 0.f, 0.f, 0.f);
                p[i].x = p[i].x * inv * aw.x;
                p[i].y = p[i].y * inv * aw.y;
                p[i].z = p[i].z * inv * aw.z;
                p[i].w = p[i].w * inv * aw.w;
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
    for (int i = 0; i < NB; ++i) {
        const uint32_t q = threadIdx.x + i * kT;
        sq = tmdev::sumsq_quad(sq, v[i]);
        if (store && q < quads && q % kC == rank) ((float4 *)r.x_out)[q] = v[i];
    }
    const float inv = inv_sqrt(fmaf(cta_sum(sq, red), inv_h, r.eps));
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        v[i].x = v[i].x * inv * nw[i].x;
        v[i].y = v[i].y * inv * nw[i].y;
        v[i].z = v[i].z * inv * nw[i].z;
        v[i].w = v[i].w * inv * nw[i].w;
    }
}

// The sum alone, with residual_norm's bits, where the position leaves a block nothing else to do: short code, because it
// lies beside code that runs every time.
__device__ __forceinline__ void store_sum(const residual_in &r, uint32_t rank, float *red) {
    float inv = 1.0f;
#pragma unroll 1
    for (uint32_t pass = r.n_slots && r.add_w ? 0u : 1u; pass < 2u; ++pass) {
        float sq = 0.0f;
#pragma unroll 1
        for (uint32_t q = threadIdx.x; q < r.hidden / 4u; q += kT) {
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
            for (uint32_t k = 0; k < r.n_slots; ++k) {
                const float4 s = __ldcg((const float4 *)(r.slots + (size_t)k * r.hidden) + q);
                p.x += s.x, p.y += s.y, p.z += s.z, p.w += s.w;
            }
            sq = tmdev::sumsq_quad(sq, p);
            if (pass == 0u || q % kC != rank) continue;
            float4 v = __ldcg((const float4 *)r.x + q);
            if (r.n_slots) {
                if (r.add_w) {
                    const float4 w = __ldg((const float4 *)r.add_w + q);
                    p.x = p.x * inv * w.x, p.y = p.y * inv * w.y, p.z = p.z * inv * w.z, p.w = p.w * inv * w.w;
                }
                v.x += p.x, v.y += p.y, v.z += p.z, v.w += p.w;
            }
            ((float4 *)r.x_out)[q] = v;
        }
        if (pass == 0u) inv = inv_sqrt(fmaf(cta_sum(sq, red + 8), 1.0f / (float)r.hidden, r.eps));
    }
}

// Waits for an exchange; false (and the word set) when it did not arrive.  The next barrier tells the whole CTA, which then
// leaves by give_up().
__device__ __forceinline__ bool await(const residual_in &r, uint32_t bar) {
    const bool ok = tmdev::mbar_wait(bar, r.waits.limit(), r.late, ~0u);
    if (!ok) *(volatile uint32_t *)r.late = 1u;
    return ok;
}
// Leaves once no peer writes to this CTA any more (`bars` counted barriers from `bar` on) and its own copies have landed.
__device__ __forceinline__ void give_up(uint32_t bar, uint32_t bars) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    tmdev::linger(bar);
    if (bars > 1u) tmdev::landed(bar + 8u);
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
// `row_of(second, tile)` is the weight row of row 0 of a tile, and where row 8 lies from it.
template <class RowOf>
__device__ __forceinline__ void load_pieces(const matrix_part &m1, const matrix_part &m2, uint32_t ring, RowOf row_of) {
    const uint32_t lane = threadIdx.x & 31u, warp = tmdev::warp_index(), g = lane >> 2, t4 = lane & 3u;
    uint32_t dst = ring + lane * 16u, dst_s = ring + 1024u + (g + 8u * t4) * 4u;
#pragma unroll 1
    for (uint32_t sec = 0; sec < 2u; ++sec) {
        const signed char *q = sec ? m2.q : m1.q;
        const unsigned short *d = sec ? m2.d : m1.d;
        const uint32_t cols = sec ? m2.cols : m1.cols, chunk0 = sec ? m2.chunk0 : m1.chunk0, chunks = sec ? m2.chunks : m1.chunks;
        const uint32_t all = chunks * (sec ? m2.tiles : m1.tiles), end = all * (warp + 1u) / kWarps;
        uint32_t i = all * warp / kWarps, tile = i / chunks, ch = i - tile * chunks;
#pragma unroll 1
        for (; i < end; ++i) {
            const uint2 row = row_of(sec, tile);
            const size_t ra = row.x + g, rb = ra + row.y, col = (chunk0 + ch) * 64u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(q + ra * cols + col + t4 * 16u) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512u), "l"(q + rb * cols + col + t4 * 16u) : "memory");
            if (t4 < 2u)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst_s), "l"(d + ((t4 ? rb : ra) * cols + col) / 32u) : "memory");
            dst += kSlotBytes;
            dst_s += kSlotBytes;
            if (++ch == chunks) {
                ch = 0u;
                ++tile;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
}

// One piece (in shared memory at `src`): this lane's digits' share of rows g (x) and g + 8 (y).
__device__ __forceinline__ float2 piece(uint32_t src, const unsigned char *dig, uint32_t plane, uint32_t ch) {
    const uint32_t l = threadIdx.x & 31u, g = l >> 2, t4 = l & 3u, c0 = ch * 64u + t4 * 16u;
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
// This warp's items [first, end) of a projection, the first one's chunk, and where its pieces lie.
struct span {
    uint32_t first, end, chunk, src;
    __device__ __forceinline__ span(const matrix_part &m, uint32_t at) {
        const uint32_t warp = tmdev::warp_index();
        first = m.first(warp);
        end = m.first(warp + 1u);
        chunk = first % m.chunks;
        src = at;
    }
};
// Item i leaves its sums in part[i][16 rows].
__device__ __forceinline__ void multiply(const span &w, uint32_t chunks, bool sec, const unsigned char *dig, uint32_t plane, float *part) {
    const uint32_t l = threadIdx.x & 31u, g = l >> 2, t4 = l & 3u;
    uint32_t ch = w.chunk, src = w.src;
    if (sec) asm volatile("cp.async.wait_group 0;" ::: "memory");
    else asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();  // scales were copied by other lanes
#pragma unroll 1
    for (uint32_t i = w.first; i < w.end; i += 4u) {
        float2 v[4];
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {  // (past the end: the last piece again)
            v[k] = piece(src, dig, plane, ch);
            if (i + k + 1u < w.end) {
                src += kSlotBytes;
                ch = ch + 1u == chunks ? 0u : ch + 1u;
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 4u; ++k) {
            v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 1);
            v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 1);
            v[k].x += __shfl_xor_sync(0xffffffffu, v[k].x, 2);
            v[k].y += __shfl_xor_sync(0xffffffffu, v[k].y, 2);
            if (t4 == 0u && i + k < w.end) {
                part[(i + k) * 16u + g] = v[k].x;
                part[(i + k) * 16u + g + 8u] = v[k].y;
            }
        }
    }
}

// Row `row` (16 tile + r) of a projection: the sum over its tile's pieces, by four adjacent lanes, which all receive it.
__device__ __forceinline__ float quad_sum(const float *part, uint32_t chunks, uint32_t row) {
    const uint32_t sub = threadIdx.x & 3u;
    const float *p = part + ((row >> 4) * chunks + sub) * 16u + (row & 15u);
    float v = 0.0f;
#pragma unroll 2
    for (uint32_t k = 0; k < chunks; k += 4u)
        if (k + sub < chunks) v += p[k * 16u];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
// This CTA's rows of the second projection, into the cluster's slot.
__device__ __forceinline__ void store_slot(const float *part, const matrix_part &m, float *out) {
#pragma unroll 1
    for (uint32_t i0 = tmdev::warp_index() * 8u; i0 < m.tiles * 16u; i0 += kT / 4u) {
        const uint32_t i = i0 + (threadIdx.x & 31u) / 4u;
        const float v = quad_sum(part, m.chunks, i);
        if ((threadIdx.x & 3u) == 0u) out[i] = v;
    }
}

// ---------------- feed-forward block ----------------
struct ffn_args {
    residual_in in;
    const signed char *gu_q, *dn_q;          // [2 width][hidden], [hidden][width]
    const unsigned short *gu_d, *dn_d;
    float *slots_out;                        // [clusters][hidden]
    uint32_t width, gelu, clusters, tiles1, tiles2, acts;  // most tiles / activations a CTA / cluster has
};

// Shared memory: digits (of x, then of the activations), activations, partial sums, ring.
struct ffn_smem {
    uint32_t acts, part, red, bar, ring, bytes;
};
__host__ __device__ inline ffn_smem ffn_layout(uint32_t hidden, uint32_t acts, uint32_t tiles1, uint32_t tiles2, uint32_t slots) {
    ffn_smem s;
    s.acts = digit_bytes(max_of(hidden, acts));
    s.part = s.acts + acts * 4u;
    s.red = s.part + 64u * max_of(tiles1 * (hidden / 64u), tiles2 * (acts / 64u));
    s.bar = s.red + 64u;
    s.ring = s.bar + 16u;
    s.bytes = s.ring + kWarps * slots * kSlotBytes;
    return s;
}

template <int NB>
__global__ void __launch_bounds__(kT, 2) ffn_block_kernel(const ffn_args a, uint32_t ring_slots) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t rank = cluster_rank(), cluster = blockIdx.x / kC;
    const uint32_t H = a.in.hidden, F = a.width, chunks = F / 64u;
    const uint32_t fc0 = chunks * cluster / a.clusters, nfc = chunks * (cluster + 1u) / a.clusters - fc0;  // FFN chunks
    const uint32_t groups = nfc * 8u;                  // of 8 gate rows and the 8 up rows they gate: one tile
    const uint32_t g0 = groups * rank / kC, n1 = groups * (rank + 1u) / kC - g0;
    const uint32_t row_tiles = H / 16u, t0 = row_tiles * rank / kC, n2 = row_tiles * (rank + 1u) / kC - t0;
    const ffn_smem L = ffn_layout(H, a.acts, a.tiles1, a.tiles2, ring_slots);
    float *acts = (float *)(smem + L.acts), *part = (float *)(smem + L.part), *red = (float *)(smem + L.red);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tmdev::warp_index();
    const uint32_t bar = smem_addr(smem + L.bar);
    if (tid == 0) tmdev::mbar_init(bar, nfc * 256u + a.in.waits.more(1u));  // all activations of the cluster
    cluster_arrive();
    const matrix_part m1 = {a.gu_q, a.gu_d, H, 0u, n1, H / 64u}, m2 = {a.dn_q, a.dn_d, F, fc0, n2, nfc};
    const uint32_t ring = smem_addr(smem + L.ring) + warp * ring_slots * kSlotBytes;
    load_pieces(m1, m2, ring, [=](uint32_t sec, uint32_t tile) {
        return sec ? make_uint2((t0 + tile) * 16u, 8u) : make_uint2(fc0 * 64u + (g0 + tile) * 8u, F);
    });
    float4 nw[NB];
    norm_weights<NB>(a.in, nw);
    const span w1(m1, ring), w2(m2, ring + (w1.end - w1.first) * kSlotBytes);
    tmdev::pdl_trigger();
    tmdev::pdl_wait();
#pragma unroll 1
    for (uint32_t sec = 0; sec < 2u; ++sec) {
        const uint32_t quads = sec ? nfc * 16u : H / 4u, plane = plane_bytes(sec ? a.acts : H);
        float4 v[NB];
        bool ok = true;
        if (sec == 0u) {
            residual_norm<NB>(a.in, cluster == 0u, rank, nw, v, red, [] {});
        } else {
            cluster_wait();  // every CTA of the cluster has started
            // A warp finishes four activations: the gate rows in its lower half, the up rows in its upper; the four lanes
            // of an activation send it to four CTAs each.
#pragma unroll 1
            for (uint32_t i = warp; i < n1 * 2u; i += kWarps) {
                const uint32_t act = i * 4u + ((lane >> 2) & 3u);
                const float sum = quad_sum(part, m1.chunks, (act >> 3) * 16u + (act & 7u) + (lane & 16u) / 2u);
                const float up = __shfl_down_sync(0xffffffffu, sum, 16);
                const float z = (a.gelu ? tmdev::gelu_tanh_f(sum) : tmdev::silu_f(sum)) * up;
                if (lane < 16u)
#pragma unroll
                    for (uint32_t k = 0; k < kC / 4u; ++k) tmdev::send(smem_addr(acts + g0 * 8u + act), bar, (lane & 3u) * (kC / 4u) + k, z);
            }
            ok = await(a.in, bar);
        }
#pragma unroll 1
        for (uint32_t q0 = warp * 32u; q0 < quads; q0 += NB * kT)
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const uint32_t q = q0 + i * kT + lane;
                if (q0 + i * kT >= quads) break;
                if (sec) v[i] = q < quads ? *(const float4 *)(acts + q * 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float y[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
                tmdev::digitise_quad(y, q < quads, (signed char *)smem + q * 4u, plane, (float *)(smem + 4u * plane) + (q >> 3) * 4u, lane);
            }
        if (__syncthreads_or(!ok)) return give_up(bar, 1u);
        multiply(sec ? w2 : w1, sec ? m2.chunks : m1.chunks, sec, smem, plane, part);
        __syncthreads();
    }
    store_slot(part, m2, a.slots_out + (size_t)cluster * H + t0 * 16u);
    for (uint32_t s = cluster + a.clusters; s < kSlots; s += a.clusters)  // slots without a cluster
        for (uint32_t i = tid; i < n2 * 16u; i += kT) a.slots_out[(size_t)s * H + t0 * 16u + i] = 0.0f;
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
    uint32_t state, qkv, recv, recv_ml, part, red, bar, ring, bytes;
};
template <int G, int HD>
__host__ __device__ inline attn_smem attn_layout(uint32_t hidden, uint32_t tiles1, uint32_t tiles2, uint32_t slots) {
    attn_smem s;
    s.state = digit_bytes(max_of(hidden, G * HD));
    s.qkv = s.state + (uint32_t)((sizeof(shared_state<G, HD>) + 15u) & ~15u);
    s.recv = s.qkv + (G + 2) * HD * 4u;
    s.recv_ml = s.recv + kC * G * HD * 4u;
    s.part = s.recv_ml + kC * G * 2u * 4u;
    s.red = s.part + 64u * max_of(tiles1 * (hidden / 64u), tiles2 * (G * HD / 64u));
    s.bar = s.red + 64u;
    s.ring = s.bar + 16u;
    s.bytes = s.ring + kWarps * slots * kSlotBytes;
    return s;
}

template <int G, int HD, int NB>
__global__ void __launch_bounds__(kT, HD > 128 ? 1 : 2) attn_block_kernel(const attn_block_args a, uint32_t ring_slots) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int EPL = HD / 32;
    constexpr uint32_t kTiles = (G + 2) * HD / 16u;  // of this KV head's q, k and v rows
    const uint32_t rank = cluster_rank(), kvh = blockIdx.x / kC, H = a.in.hidden, cap = a.cap;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tmdev::warp_index();
    const uint32_t u0 = kTiles * rank / kC, n1 = kTiles * (rank + 1u) / kC - u0;
    const uint32_t row_tiles = H / 16u, t0 = row_tiles * rank / kC, n2 = row_tiles * (rank + 1u) / kC - t0;
    const attn_smem L = attn_layout<G, HD>(H, a.tiles1, a.tiles2, ring_slots);
    shared_state<G, HD> &sh = *(shared_state<G, HD> *)(smem + L.state);
    float *qkv = (float *)(smem + L.qkv), *recv = (float *)(smem + L.recv), *recv_ml = (float *)(smem + L.recv_ml);
    float *part = (float *)(smem + L.part), *red = (float *)(smem + L.red);
    const uint32_t bar = smem_addr(smem + L.bar);
    if (tid == 0) {
        tmdev::mbar_init(bar, (G + 2) * HD * 4u + a.in.waits.more(1u));               // this head's q, k and v
        tmdev::mbar_init(bar + 8u, kC * (G * HD + 2 * G) * 4u + a.in.waits.more(2u));  // every CTA's (max, sum, output)
    }
    cluster_arrive();
    const uint32_t kvw = a.kv_heads * HD;
    const matrix_part m1 = {a.qkv_q, a.qkv_d, H, 0u, n1, H / 64u}, m2 = {a.o_q, a.o_d, kvw * G, kvh * (G * HD / 64u), n2, G * HD / 64u};
    const uint32_t ring = smem_addr(smem + L.ring) + warp * ring_slots * kSlotBytes;
    // Tiles are counted over this head's q rows, then its k rows, then its v rows.
    load_pieces(m1, m2, ring, [=](uint32_t sec, uint32_t tile) {
        const uint32_t i = (u0 + tile) * 16u;
        return make_uint2(sec             ? (t0 + tile) * 16u
                          : i < G * HD    ? kvh * (G * HD) + i
                          : i < (G + 1) * HD ? kvw * G + kvh * HD + (i - G * HD)
                                          : kvw * (G + 1) + kvh * HD + (i - (G + 1) * HD),
                          8u);
    });
    float4 nw[NB];
    norm_weights<NB>(a.in, nw);
    const span w1(m1, ring), w2(m2, ring + (w1.end - w1.first) * kSlotBytes);
    __half *kp = a.kc + (size_t)kvh * cap * HD, *vp = a.vc + (size_t)kvh * cap * HD;
    const volatile uint32_t *pos_p = a.pos;
    keys<G, HD> K;
    float hw[EPL];  // warp g < G: query head g; warp G: the new key
    rotation<HD> rot;
    uint32_t pos = tmdev::uniform(min(*pos_p, cap - 1u));
    K.ask(kp, vp, pos, a.window, kC, rank);
#pragma unroll
    for (int r = 0; r < EPL; ++r) hw[r] = __ldg((warp == G ? a.k_norm : a.q_norm) + lane + 32 * r);
#pragma unroll 1
    for (uint32_t hint = pos;;) {  // the angles of the position as it reads before the wait, again where it was another
        if (warp <= G) rot.set(a.inv_freq, min(pos, cap - 1u));
        if (hint == ~0u) break;
        tmdev::pdl_wait();
        tmdev::pdl_trigger();  // only now: see tm_cuda_attn_core.cuh
        pos = tmdev::uniform(*pos_p);
        if (pos == hint) break;
        hint = ~0u;
    }
    if (pos >= cap) goto past;  // uniform over the cluster
#pragma unroll 1
    for (uint32_t sec = 0; sec < 2u; ++sec) {
        const uint32_t quads = (sec ? G * HD : H) / 4u, plane = plane_bytes(sec ? G * HD : H);
        float4 v[NB];
        bool ok = true;
        if (sec == 0u) {
            residual_norm<NB>(a.in, kvh == 0u, rank, nw, v, red, [&] { K.first_tile(pos, a.window, kC, rank); });
        } else {
            cluster_wait();  // every CTA of the cluster has started
            // Four lanes finish a row and send it to four CTAs each.
#pragma unroll 1
            for (uint32_t i0 = warp * 8u; i0 < n1 * 16u; i0 += kT / 4u) {
                const uint32_t i = i0 + lane / 4u;
                const float z = quad_sum(part, m1.chunks, i);
#pragma unroll
                for (uint32_t k = 0; k < kC / 4u; ++k) tmdev::send(smem_addr(qkv + u0 * 16u + i), bar, (lane & 3u) * (kC / 4u) + k, z);
            }
            ok = await(a.in, bar);
            // ---- every CTA has the head's q, k and v ----
            if (warp < G || (warp == G && K.lo <= pos && pos < K.hi)) {
                float x[EPL];
#pragma unroll
                for (int r = 0; r < EPL; ++r) x[r] = qkv[warp * HD + lane + 32 * r];
                norm_rope<HD>(x, hw, rot, a.in.eps);
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
            if (__syncthreads_or(!ok)) return give_up(bar, 2u);
            K.attend(sh, pos, a.scale);
            __syncthreads();
            // ---- this CTA's (max, sum, output) to every CTA: each needs all of the head's output for its rows of o ----
            {
                constexpr uint32_t kQuads = G * HD / 4, kDest = kC * kQuads / kT;  // a thread's quad goes to kDest CTAs
                const uint32_t quad = tid % kQuads, to = tid / kQuads * kDest, head = quad * 4u / HD;
                float4 o;
                const float2 ml = keys<G, HD>::combined(sh, head, quad * 4u % HD, o);
#pragma unroll 1
                for (uint32_t k = 0; k < kDest; ++k) {
                    tmdev::send(smem_addr(recv + (rank * kQuads + quad) * 4u), bar + 8u, to + k, o);
                    if (quad % (HD / 4u) == 0u) tmdev::send(smem_addr(recv_ml + (rank * G + head) * 2u), bar + 8u, to + k, ml);
                }
            }
            ok = await(a.in, bar + 8u);
        }
        // Four lanes to a quad of the attention's output, each with a quarter of the source CTAs.
        const uint32_t shift = sec ? 2u : 0u;
#pragma unroll 1
        for (uint32_t q0 = (warp * 32u) >> shift; q0 < quads; q0 += NB * (kT >> shift))
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const uint32_t q = q0 + i * (kT >> shift) + (lane >> shift);
                if (q0 + i * (kT >> shift) >= quads) break;
                if (sec) {
                    const uint32_t head = q * 4u / HD, c0 = (lane & 3u) * (kC / 4u);
                    float m[kC / 4u], M = -INFINITY, l = 0.0f;
#pragma unroll
                    for (uint32_t k = 0; k < kC / 4u; ++k) {
                        m[k] = recv_ml[((c0 + k) * G + head) * 2u];
                        M = fmaxf(M, m[k]);
                    }
                    M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 1));
                    M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, 2));
                    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (uint32_t k = 0; k < kC / 4u; ++k) {
                        const float4 o = *(const float4 *)(recv + (c0 + k) * G * HD + q * 4u);
                        const float f = expf(m[k] - M);  // a CTA without keys: exp(-inf) = 0
                        l = fmaf(f, recv_ml[((c0 + k) * G + head) * 2u + 1u], l);
                        v[i].x = fmaf(f, o.x, v[i].x);
                        v[i].y = fmaf(f, o.y, v[i].y);
                        v[i].z = fmaf(f, o.z, v[i].z);
                        v[i].w = fmaf(f, o.w, v[i].w);
                    }
#pragma unroll
                    for (int off = 1; off < 4; off <<= 1) {
                        l += __shfl_xor_sync(0xffffffffu, l, off);
                        v[i].x += __shfl_xor_sync(0xffffffffu, v[i].x, off);
                        v[i].y += __shfl_xor_sync(0xffffffffu, v[i].y, off);
                        v[i].z += __shfl_xor_sync(0xffffffffu, v[i].z, off);
                        v[i].w += __shfl_xor_sync(0xffffffffu, v[i].w, off);
                    }
                    const float inv = 1.0f / l;
                    v[i] = make_float4(v[i].x * inv, v[i].y * inv, v[i].z * inv, v[i].w * inv);
                }
                const float y[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
                tmdev::digitise_quad(y, q < quads, (signed char *)smem + q * 4u, plane, (float *)(smem + 4u * plane) + (q >> 3) * 4u, lane, shift);
            }
        if (__syncthreads_or(!ok)) return give_up(bar, 2u);
        multiply(sec ? w2 : w1, sec ? m2.chunks : m1.chunks, sec, smem, plane, part);
        __syncthreads();
    }
    store_slot(part, m2, a.slots_out + (size_t)kvh * H + t0 * 16u);
    return;
past:  // The pieces' copies land before the CTA's memory goes away.  (As a way out of the loop, or before it, 16 bytes of a
       // thread's registers spill: 0.3 us a block, 127.9 against 125.5 ms for a request of 512 + 256 tokens.)
    if (kvh == 0u) store_sum(a.in, rank, red);
    if (tid == 0 && rank == 0) atomicOr(a.status, TM_CUDA_STATUS_PAST_CAPACITY);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    cluster_wait();
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
    return launch_clusters(ctx, ffn_block_kernel<NB>, attr_set, a.clusters,
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
uint32_t ffn_items(const ffn_args &a) {
    return ceil_div(a.tiles1 * (a.in.hidden / 64u), kWarps) + ceil_div(a.tiles2 * (a.acts / 64u), kWarps);
}
// Six clusters find a place beside attention's eight (above); eight where a sixth's pieces do not stay in shared memory.
ffn_args ffn_shape(uint32_t hidden, uint32_t width) {
    ffn_args a = {};
    a.in.hidden = hidden;
    a.width = width;
    for (uint32_t clusters : {kFfnClusters, kSlots}) {
        const uint32_t nfc = ceil_div(width / 64u, clusters);
        a.clusters = clusters;
        a.acts = nfc * 64u;
        a.tiles1 = ceil_div(nfc * 8u, kC);
        a.tiles2 = ceil_div(hidden / 16u, kC);
        if (ffn_items(a) <= kResident) break;
    }
    return a;
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
    TM_CUDA_TRY(tm_ensure_abort_flag(ctx));
    r.late = (uint32_t *)ctx->mma_abort;
    r.waits = ctx->waits;
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
