// One CTA's share of a decode token's attention: the G query heads of a KV head against a contiguous run of its
// cached keys, 256 threads, 64 keys at a time.  Shared by the stand-alone decode attention and by the fused
// attention block.
//
// A warp takes 8 keys of every tile and carries its own running (max, sum, output): scores, softmax weights and the
// value sum never leave its registers, so the tiles need no barrier; the warps' states meet once at the end.  (With
// the softmax of a tile as a CTA-wide step, three barriers around it were most of the time at short contexts.)
//
// (Stand-alone form; the fused block has its projections between the wait and the scores and reads no row before it.)
// Cached rows are read before the predecessor kernel finishes.  The position read at that moment only says which
// rows to ask for; it is read again afterwards, and a changed one reloads them.  Row pos - 1 is always read after the
// wait: the attention call of the previous token may still be storing it.  Calls further back have finished, because
// a kernel that stores KV rows lets its successor start only after its own predecessor is complete.  Where another
// operator has written the cache or the table of frequencies, or the call before took its position from another word,
// the launch does not overlap what is before it (tm_read_cache_ahead).
#pragma once
#include "tm_cuda_internal.cuh"
#include "tm_cuda_device.cuh"

namespace tmattn {

constexpr int kT = 256;     // threads per CTA
constexpr int kTile = 64;   // keys at a time
constexpr uint32_t kMaxCluster = 16;

using tmdev::cluster_arrive;
using tmdev::cluster_rank;
using tmdev::cluster_size;
using tmdev::cluster_wait;
using tmdev::smem_addr;

// CTA `rank` of C owns keys [lo, hi) of a step at position p: equal contiguous runs of whole eights.
__device__ __forceinline__ void key_range(uint32_t p, uint32_t window, uint32_t C, uint32_t rank, uint32_t &lo, uint32_t &hi) {
    const uint32_t seq = p + 1u, start = window != 0u && seq > window ? seq - window : 0u;
    const uint32_t per = ((seq - start + C - 1u) / C + 7u) & ~7u;
    lo = start + rank * per;
    hi = min(lo + per, seq);
}

// 1 / sqrt(v): the hardware's approximation y and one Newton step from the residual 1 - v y^2, which fused multiply-adds
// give without its rounding errors.  Within 0.5000 ulp of the true value at every float from 1e-38 up (1.0f / sqrtf(v): 1.4903)
// and without the division, a tenth of a microsecond of the chains that use it.  0 and infinity give infinity and 0.
__device__ __forceinline__ float inv_sqrt(float v) {
    const float y = rsqrtf(v), h = v * y, l = fmaf(v, y, -h);  // v y = h + l
    const float r = fmaf(-l, y, fmaf(-h, y, 1.0f));
    return y > 0.0f && y < INFINITY ? fmaf(0.5f * y, r, y) : y;
}

// sin and cos of the rotation of a lane's pairs (i, i + HD/2), i = lane + 32 r; needs the position only.
template <int HD>
struct rotation {
    float sn[HD / 64], cs[HD / 64];
    __device__ __forceinline__ void set(const float *inv_freq, uint32_t pos) {
#pragma unroll
        for (int r = 0; r < HD / 64; ++r) sincosf((float)pos * __ldg(inv_freq + (threadIdx.x & 31u) + 32 * r), &sn[r], &cs[r]);
    }
};
// RMS norm times w, then the full rotation, of a head vector held as x[r] = element lane + 32 r.
template <int HD>
__device__ __forceinline__ void norm_rope(float (&x)[HD / 32], const float (&w)[HD / 32], const rotation<HD> &rot, float eps) {
    constexpr int EPL = HD / 32;
    float ss = 0.0f;
#pragma unroll
    for (int r = 0; r < EPL; ++r) ss = fmaf(x[r], x[r], ss);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float inv = inv_sqrt(ss * (1.0f / (float)HD) + eps);
#pragma unroll
    for (int r = 0; r < EPL; ++r) x[r] = x[r] * inv * w[r];
#pragma unroll
    for (int r = 0; r < EPL / 2; ++r) {
        const float a0 = x[r], b0 = x[r + EPL / 2];
        x[r] = a0 * rot.cs[r] - b0 * rot.sn[r];
        x[r + EPL / 2] = a0 * rot.sn[r] + b0 * rot.cs[r];
    }
}

template <int G, int HD>
struct shared_state {
    __align__(16) float qs[G][HD];
    __align__(16) __half kh[HD];   // this step's own key and value
    __align__(16) __half vh[HD];
    // Every warp's maximum, sum and output.
    float m[G][kT / 32], l[G][kT / 32];
    __align__(16) float opart[kT / 32][G][HD];
};

template <int G, int HD>
struct keys {
    using S = shared_state<G, HD>;
    static constexpr int NL = HD / 32;             // 16-byte loads of a thread's quarter of a key row
    static constexpr int TV = HD / 8;              // lanes per value row
    static constexpr int RV = 32 / TV;             // value rows of a warp's pass
    static constexpr int VP = 8 / RV;              // passes over the warp's 8 rows
    const __half *kp, *vp;                         // this KV head's planes
    uint32_t lo, hi, hint;
    uint32_t kk, kq, vr, vd;                       // key of the tile, quarter of its dims; first value row, first dim
    int4 kraw[NL], vraw[VP];

    __device__ __forceinline__ void load_k(uint32_t j) {
#pragma unroll
        for (int i = 0; i < NL; ++i) kraw[i] = __ldcg((const int4 *)(kp + (size_t)j * HD + i * 32 + kq * 8u));
    }
    __device__ __forceinline__ void load_v(int p, uint32_t j) { vraw[p] = __ldcg((const int4 *)(vp + (size_t)j * HD + vd)); }

    __device__ __forceinline__ void place(const __half *k_plane, const __half *v_plane) {
        const uint32_t lane = threadIdx.x & 31u, warp = tmdev::warp_index();
        kp = k_plane;
        vp = v_plane;
        kk = warp * 8u + (lane >> 2);
        kq = lane & 3u;
        vr = warp * 8u + lane / TV;
        vd = (lane % TV) * 8u;
    }
    // Rows from `from` on: towards L2.
    __device__ __forceinline__ void prefetch(uint32_t from) const {
#pragma unroll 1
        for (uint32_t t = from; t < hi; t += kTile) {
            const uint32_t j = min(t + threadIdx.x / (kT / kTile), hi - 1u);
#pragma unroll 1
            for (uint32_t b = (threadIdx.x & 1u) * 128u; b < HD * 2u; b += 256u)
                asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)((threadIdx.x & 2u ? vp : kp) + (size_t)j * HD) + b));
        }
    }
    // Before the dependency wait, where there is work between it and the scores: all rows towards L2 (no value is read) ...
    __device__ __forceinline__ void ask(const __half *k_plane, const __half *v_plane, uint32_t pos_hint, uint32_t window,
                                        uint32_t C, uint32_t rank) {
        place(k_plane, v_plane);
        key_range(pos_hint, window, C, rank, lo, hi);
        prefetch(lo);
    }
    // ... and after it the first tile.
    __device__ __forceinline__ void first_tile(uint32_t pos, uint32_t window, uint32_t C, uint32_t rank) {
        key_range(pos, window, C, rank, lo, hi);
        load_tile(lo);
    }
    // Rows past the range are read as its last one (whose weight there is 0).
    __device__ __forceinline__ void load_tile(uint32_t t0) {
        load_k(min(t0 + kk, hi - 1u));
#pragma unroll
        for (int p = 0; p < VP; ++p) load_v(p, min(t0 + vr + p * RV, hi - 1u));
    }

    // Before the dependency wait: rows up to hint - 2 of the first tile.
    __device__ __forceinline__ void early(const __half *k_plane, const __half *v_plane, uint32_t pos_hint, uint32_t window,
                                          uint32_t C, uint32_t rank) {
        place(k_plane, v_plane);
        hint = pos_hint;
        key_range(hint, window, C, rank, lo, hi);
#pragma unroll
        for (int i = 0; i < NL; ++i) kraw[i] = make_int4(0, 0, 0, 0);
        if (lo + kk < hi && lo + kk + 1u < hint) load_k(lo + kk);
#pragma unroll
        for (int p = 0; p < VP; ++p) {
            const uint32_t j = lo + vr + p * RV;
            vraw[p] = make_int4(0, 0, 0, 0);
            if (j < hi && j + 1u < hint) load_v(p, j);
        }
        prefetch(lo + kTile);  // the rows after those
    }
    // After it: the rows of the first tile that were not to be read early.
    __device__ __forceinline__ void late(uint32_t pos, uint32_t window, uint32_t C, uint32_t rank) {
        if (pos != hint) key_range(pos, window, C, rank, lo, hi);
        const uint32_t j = lo + kk;
        if (j < hi && j != pos && (pos != hint || j + 1u == pos)) load_k(j);
#pragma unroll
        for (int p = 0; p < VP; ++p) {
            const uint32_t jv = lo + vr + p * RV;
            if (jv < hi && jv != pos && (pos != hint || jv + 1u == pos)) load_v(p, jv);
        }
    }
    // All tiles; s.qs, s.kh and s.vh are set (one barrier ago).  Leaves every warp's (max, sum, output) in s.
    __device__ __forceinline__ void attend(S &s, uint32_t pos, float scale) {
        const uint32_t lane = threadIdx.x & 31u, warp = tmdev::warp_index();
        float acc[G][8], m[G], l[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[g][e] = 0.0f;
        }
#pragma unroll 1
        for (uint32_t t0 = lo; t0 + warp * 8u < hi; t0 += kTile) {  // uniform over the warp
            // ---- scores: four lanes per key, interleaved 8-dim pieces ----
            const uint32_t j = t0 + kk, last = hi - 1u;
            if (min(j, last) == pos)
#pragma unroll
                for (int i = 0; i < NL; ++i) kraw[i] = *(const int4 *)(s.kh + i * 32 + kq * 8u);
            float p[G];
#pragma unroll
            for (int g = 0; g < G; ++g) p[g] = 0.0f;
#pragma unroll
            for (int i = 0; i < NL; ++i) {
                const __half2 *h2 = (const __half2 *)&kraw[i];
                float kf[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __half22float2(h2[e]);
                    kf[2 * e] = f.x;
                    kf[2 * e + 1] = f.y;
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float4 q0 = *(const float4 *)&s.qs[g][i * 32 + kq * 8u];
                    const float4 q1 = *(const float4 *)&s.qs[g][i * 32 + kq * 8u + 4];
                    float t = p[g];
                    t = fmaf(q0.x, kf[0], t); t = fmaf(q0.y, kf[1], t); t = fmaf(q0.z, kf[2], t); t = fmaf(q0.w, kf[3], t);
                    t = fmaf(q1.x, kf[4], t); t = fmaf(q1.y, kf[5], t); t = fmaf(q1.z, kf[6], t); t = fmaf(q1.w, kf[7], t);
                    p[g] = t;
                }
            }
            load_k(min(j + kTile, last));  // the next tile's
            // ---- softmax weights against the warp's running maximum ----
            float al[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                p[g] += __shfl_xor_sync(0xffffffffu, p[g], 1);
                p[g] += __shfl_xor_sync(0xffffffffu, p[g], 2);
                p[g] = j < hi ? p[g] * scale : -INFINITY;
                float mx = p[g];
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                mx = fmaxf(mx, m[g]);  // finite: the warp's 8 rows hold at least one key
                p[g] = expf(p[g] - mx);
                al[g] = expf(m[g] - mx);
                m[g] = mx;
                l[g] = fmaf(l[g], al[g], p[g]);  // this lane's key only (four lanes count it)
            }
            // ---- values: a lane owns 8 dims of the rows of its half (or of all) ----
            if (t0 != lo)
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[g][e] *= al[g];
#pragma unroll
            for (int v = 0; v < VP; ++v) {
                const uint32_t row = lane / TV + v * RV, jv = t0 + vr + v * RV;
                int4 raw = vraw[v];
                if (jv == pos) raw = *(const int4 *)(s.vh + vd);
                if (jv > last) raw = make_int4(0, 0, 0, 0);  // weight 0 there, and 0 times an infinity is NaN
                const __half2 *h2 = (const __half2 *)&raw;
                float f[8];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 u = __half22float2(h2[e]);
                    f[2 * e] = u.x;
                    f[2 * e + 1] = u.y;
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float pj = __shfl_sync(0xffffffffu, p[g], row * 4u);
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[g][e] = fmaf(pj, f[e], acc[g][e]);
                }
                load_v(v, min(jv + kTile, last));
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            l[g] += __shfl_xor_sync(0xffffffffu, l[g], 4);
            l[g] += __shfl_xor_sync(0xffffffffu, l[g], 8);
            l[g] += __shfl_xor_sync(0xffffffffu, l[g], 16);
            if (RV > 1)
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[g][e] += __shfl_xor_sync(0xffffffffu, acc[g][e], 16);
            if (lane < TV) {
                *(float4 *)&s.opart[warp][g][vd] = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
                *(float4 *)&s.opart[warp][g][vd + 4] = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
            }
            if (lane == 0) {
                s.m[g][warp] = m[g];
                s.l[g][warp] = l[g];
            }
        }
    }
    // After a barrier: dims d .. d + 3 of head g (not yet divided by the sum) by one thread, with the CTA's maximum and sum:
    // every factor once, and no barrier.  A CTA without keys has maximum -inf, sum 0 and values 0.
    static __device__ __forceinline__ float2 combined(const S &s, uint32_t g, uint32_t d, float4 &o) {
        float m[kT / 32], M = -INFINITY, L = 0.0f;
        o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kT / 32; ++w) M = fmaxf(M, m[w] = s.m[g][w]);
#pragma unroll
        for (int w = 0; w < kT / 32; ++w) {
            const float f = M == -INFINITY ? 0.0f : expf(m[w] - M);
            const float4 v = *(const float4 *)&s.opart[w][g][d];
            L = fmaf(f, s.l[g][w], L);
            o.x = fmaf(f, v.x, o.x);
            o.y = fmaf(f, v.y, o.y);
            o.z = fmaf(f, v.z, o.z);
            o.w = fmaf(f, v.w, o.w);
        }
        return make_float2(M, L);
    }
};

}  // namespace tmattn
