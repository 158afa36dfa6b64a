// Prefill attention on the tensor cores, tolerance-qualified.
//
// Same contract as the chunk attention operator (native/metal/tm_metal.h:367,
// native/metal/kernels.metal: query row t of a chunk at pos0 attends keys
// [start, pos0 + t], start = seq > window ? seq - window : 0, softmax over
// q.k * scale, f16 K/V cache) but not its arithmetic order: Q and the softmax
// weights are rounded to binary16 and multiplied with mma.sync (m16n8k16, f32
// accumulate), keys are visited in tiles of 64 with a running maximum.  The
// engine uses it unless `exact` is asked; the blockwise kernel stays the
// bit-identical form.  Attention is not the Q8_0 hot path: this kernel exists
// because a 512-token prefill otherwise spends half its time here.
//
// A CTA of 8 warps serves 64 or 128 queries of one head: a warp takes 32 of them and every second or fourth block of
// 32 keys, and the warps that share queries add their results at the end.  When the head dim exceeds 128 a CTA makes
// one 128-wide half of the value dims (grid.y).
#include "tm_cuda_internal.cuh"
#include "tm_cuda_device.cuh"

namespace {

constexpr int kBKV = 64, kThreads = 128;  // of the decode kernel

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Byte offset of 16-byte chunk `chunk` of row `row` in a tile of PITCH-byte rows, XOR-swizzled so
// that the eight rows an ldmatrix touches fall into distinct bank groups.
template <int PITCH>
__device__ __forceinline__ uint32_t sw(uint32_t row, uint32_t chunk) {
    if (PITCH >= 128) return row * PITCH + ((chunk ^ (row & 7u)) << 4);
    return row * PITCH + ((chunk ^ ((row >> 1) & 3u)) << 4);  // 64-byte rows: two rows per 128 bytes
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
using tmdev::mma_f16;
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *(const uint32_t *)&h;
}

// The rows of one launch: up to 64 runs of consecutive positions, each of one sequence (of one prompt's chunk there is
// one run).  Runs lie one after the other in the row-major operands.
struct attn_segs {
    uint32_t n;
    uint32_t row0[TM_CUDA_PREFILL_SEGMENTS + 1];  // first row; [n]: all rows
    uint32_t pos0[TM_CUDA_PREFILL_SEGMENTS], seq[TM_CUDA_PREFILL_SEGMENTS];
};

struct attn_args {
    const float *q;  // [rows][heads][HD]
    const float *q_norm, *inv_freq;  // q_norm null: q is normed and rotated already
    const __half *kc;  // [sequences][kv_heads][cap][HD]
    const __half *vc;
    void *out;  // [rows][heads][HD], f32 or binary16
    size_t seq_stride;
    uint32_t heads, group, cap, window, n_rot, out_f16;
    float scale_log2e, eps;  // the scale's magnitude: its sign multiplies the queries (attn_scale)
    float q_sign;
    attn_segs segs;
};

// RMS norm and split-half RoPE of one HD-vector by one warp; element lane + 32 r in x[r].
template <int R>
__device__ __forceinline__ void norm_rope_row(float (&x)[R], const float *nw, const float *inv_freq, uint32_t n_rot,
                                              uint32_t pos, float eps, uint32_t lane) {
    float ss = 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) ss = fmaf(x[r], x[r], ss);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float inv = 1.0f / sqrtf(ss / (float)(32 * R) + eps);
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = x[r] * inv * nw[lane + 32u * r];
    const uint32_t half = n_rot / 2u;
    if (R > 1 && n_rot == 32u * R) {  // partners are R/2 registers apart in the same lane
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
            float sn, cs;
            sincosf((float)pos * inv_freq[lane + 32u * r], &sn, &cs);
            const float a = x[r], b = x[r + R / 2];
            x[r] = a * cs - b * sn;
            x[r + R / 2] = a * sn + b * cs;
        }
        return;
    }
    float y[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = lane + 32u * r;
        const bool first = e < half, second = e >= half && e < n_rot;
        const uint32_t pe = first ? e + half : e - half;
        float partner = 0.0f;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) {
            const float cand = __shfl_sync(0xffffffffu, x[rr], (int)(pe & 31u));
            if ((first || second) && (uint32_t)rr == (pe >> 5)) partner = cand;
        }
        y[r] = x[r];
        if (first || second) {
            float sn, cs;
            sincosf((float)pos * inv_freq[first ? e : e - half], &sn, &cs);
            y[r] = first ? x[r] * cs - partner * sn : partner * sn + x[r] * cs;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = y[r];
}

// RW warps of 32 queries, 8 / RW of them to a set of queries: warp (rw, sp) takes the 32-key block sp of every round.
//   * 32 queries a warp: an ldmatrix of keys or values serves two MMAs.  With 16 the shared-memory reads took as long
//     as the MMAs (256 of 270 cycles for 16 queries x 64 keys on an SM);
//   * keys split between warps: a 512-token chunk of 16 heads is 128 CTAs of 64 queries.  Four warps of 16 queries and
//     all keys were one warp per scheduler, each alone with its chain of product, maximum, exponential, product.
template <int HD, int RW>
struct attn_cfg {
    static constexpr int kSP = 8 / RW, kBQ = 32 * RW, kRound = 32 * kSP;
    static constexpr int kDV = HD > 128 ? 128 : HD;  // value dims per CTA
    static constexpr int kQPitch = HD * 2, kVPitch = kDV * 2, kOPitch = kDV + 8;
    static constexpr uint32_t kQBytes = kBQ * kQPitch, kKBytes = kRound * kQPitch, kVBytes = kRound * kVPitch;
    static constexpr uint32_t kStage = kKBytes + kVBytes;
    static constexpr uint32_t kMerge = kBQ * kOPitch * 4 + 2 * kSP * kBQ * 4;  // after the loop, over the stages
    static constexpr uint32_t kLoop = 2 * kStage > kMerge ? 2 * kStage : kMerge;
    static constexpr uint32_t kBytes = kQBytes + kLoop;
};
constexpr int kChunkThreads = 256;

template <int HD, int RW>
__global__ void __launch_bounds__(kChunkThreads, 1) attention_chunk_mma_kernel(const __grid_constant__ attn_args a) {
    using C = attn_cfg<HD, RW>;
    constexpr int DV = C::kDV, SP = C::kSP, BQ = C::kBQ, KR = C::kRound;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *sQ = smem, *sKV = smem + C::kQBytes;
    // (With a warp index that the compiler knows to be uniform the rounds of keys take 3 % longer; nor does it pay to leave out
    // the rescale of an empty sum: both together 512 rows at position 1000 32.8 -> 34.9 us.)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int rw = warp % RW, sp = warp / RW;
    // Tiles of queries from the last one down (the last of a chunk sees the most keys), heads next to one another.
    const uint32_t head = blockIdx.x % a.heads, kvh = head / a.group;
    const uint32_t dv0 = blockIdx.y * DV;
    uint32_t seg = 0, q0 = (gridDim.x - 1u - blockIdx.x) / a.heads;
    for (; seg + 1u < a.segs.n; ++seg) {
        const uint32_t tiles = (a.segs.row0[seg + 1] - a.segs.row0[seg] + BQ - 1) / BQ;
        if (q0 < tiles) break;
        q0 -= tiles;
    }
    q0 *= BQ;  // first query of this CTA, of the run's n at pos0
    const uint32_t row0 = a.segs.row0[seg], n = a.segs.row0[seg + 1] - row0, pos0 = a.segs.pos0[seg];
    const uint32_t q_last = min(q0 + BQ, n) - 1u;
    // Keys any query of the block may see: from the first query's window start to the last query's position.
    const uint32_t seq_first = pos0 + q0 + 1u;
    const uint32_t kv_lo = (a.window != 0u && seq_first > a.window) ? seq_first - a.window : 0u;
    const uint32_t kv_hi = pos0 + q_last;  // inclusive
    const uint32_t round_lo = kv_lo / KR, round_hi = kv_hi / KR;
    const size_t plane = (size_t)a.segs.seq[seg] * a.seq_stride + (size_t)kvh * a.cap * HD;
    const __half *kp = a.kc + plane, *vp = a.vc + plane;
    tmdev::pdl_wait();
    tmdev::pdl_trigger();

    auto load_round = [&](uint32_t round) {
        unsigned char *sK = sKV + (round & 1u) * C::kStage, *sV = sK + C::kKBytes;
        const uint32_t j0 = round * KR;
        constexpr int KCH = HD / 8, VCH = DV / 8;  // 16-byte chunks per row
        for (int i = tid; i < KR * KCH; i += kChunkThreads) {
            const uint32_t r = i / KCH, c = i % KCH;
            const uint32_t j = min(j0 + r, kv_hi);  // rows past the last visible key repeat it (they are masked)
            cp_async16(smem_u32(sK) + sw<C::kQPitch>(r, c), kp + (size_t)j * HD + c * 8);
        }
        for (int i = tid; i < KR * VCH; i += kChunkThreads) {
            const uint32_t r = i / VCH, c = i % VCH;
            const uint32_t j = min(j0 + r, kv_hi);
            cp_async16(smem_u32(sV) + sw<C::kVPitch>(r, c), vp + (size_t)j * HD + dv0 + c * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_round(round_lo);

    // Q: f32 -> f16 into the swizzled tile (rows past the run are zero).
    if (a.q_norm) {
        constexpr int R = HD / 32;
        const uint32_t rows = min((uint32_t)BQ, n - q0);
        float nx[R];  // the next row, on its way
        auto fetch = [&](uint32_t r) {
            const float *src = a.q + ((size_t)(row0 + q0 + min(r, rows - 1u)) * a.heads + head) * HD;
#pragma unroll
            for (int i = 0; i < R; ++i) nx[i] = src[lane + 32 * i];
        };
        fetch(warp);
#pragma unroll 2
        for (uint32_t r = warp; r < BQ; r += 8) {
            float x[R];
#pragma unroll
            for (int i = 0; i < R; ++i) x[i] = nx[i];
            if (r < rows) {
                fetch(r + 8u);
                norm_rope_row<R>(x, a.q_norm, a.inv_freq, a.n_rot, pos0 + q0 + r, a.eps, lane);
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const uint32_t e = lane + 32u * i;
                *(__half *)(sQ + sw<C::kQPitch>(r, e >> 3) + (e & 7u) * 2u) = r < rows ? __float2half_rn(x[i] * a.q_sign) : __half(0);
            }
        }
    } else {
        for (int i = tid; i < BQ * (HD / 8); i += kChunkThreads) {
            const uint32_t r = i / (HD / 8), c = i % (HD / 8);
            uint4 w = make_uint4(0, 0, 0, 0);
            if (q0 + r < n) {
                const float *src = a.q + ((size_t)(row0 + q0 + r) * a.heads + head) * HD + c * 8;
                float4 f0 = *(const float4 *)src, f1 = *(const float4 *)(src + 4);
                f0.x *= a.q_sign, f0.y *= a.q_sign, f0.z *= a.q_sign, f0.w *= a.q_sign;
                f1.x *= a.q_sign, f1.y *= a.q_sign, f1.z *= a.q_sign, f1.w *= a.q_sign;
                w = make_uint4(pack_h2(f0.x, f0.y), pack_h2(f0.z, f0.w), pack_h2(f1.x, f1.y), pack_h2(f1.z, f1.w));
            }
            *(uint4 *)(sQ + sw<C::kQPitch>(r, c)) = w;
        }
    }

    float o[2][DV / 8][4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int i = 0; i < DV / 8; ++i) o[mt][i][0] = o[mt][i][1] = o[mt][i][2] = o[mt][i][3] = 0.0f;
    float m_run[2][2], l_run[2][2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) m_run[mt][h] = -INFINITY, l_run[mt][h] = 0.0f;
    // Query rows of this thread: rw*32 + 16 mt + 8 h + g.
    const uint32_t w_first = pos0 + q0 + rw * 32, w_last = w_first + 31u;
    const bool idle = q0 + rw * 32 >= n;  // every query of this warp is past the run

    for (uint32_t round = round_lo; round <= round_hi; ++round) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this round has landed, and every warp is done with the stage the next one goes to
        if (round < round_hi) load_round(round + 1);
        const uint32_t j0 = round * KR + sp * 32;
        if (idle || j0 > w_last || (a.window != 0u && j0 + 31u + a.window <= w_first)) continue;  // nothing visible
        const uint32_t sK = smem_u32(sKV + (round & 1u) * C::kStage), sV = sK + C::kKBytes;

        // ---- S = Q K^T for 32 queries x 32 keys ----
        float s[2][4][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[mt][i][0] = s[mt][i][1] = s[mt][i][2] = s[mt][i][3] = 0.0f;
        const uint32_t m = lane >> 3;
#pragma unroll
        for (int kt = 0; kt < HD / 16; ++kt) {
            uint32_t q[2][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const uint32_t row = rw * 32 + mt * 16 + (m & 1u) * 8 + (lane & 7), chunk = kt * 2 + (m >> 1);
                ldsm_x4(smem_u32(sQ) + sw<C::kQPitch>(row, chunk), q[mt][0], q[mt][1], q[mt][2], q[mt][3]);
            }
#pragma unroll
            for (int np = 0; np < 2; ++np) {  // two key n-tiles per ldmatrix
                uint32_t b0, b1, b2, b3;
                const uint32_t row = sp * 32 + np * 16 + (m >> 1) * 8 + (lane & 7), chunk = kt * 2 + (m & 1u);
                ldsm_x4(sK + sw<C::kQPitch>(row, chunk), b0, b1, b2, b3);
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    mma_f16(s[mt][2 * np], q[mt][0], q[mt][1], q[mt][2], q[mt][3], b0, b1);
                    mma_f16(s[mt][2 * np + 1], q[mt][0], q[mt][1], q[mt][2], q[mt][3], b2, b3);
                }
            }
        }
        // ---- mask (only blocks that the diagonal or the window's edge cuts), running maximum, exponentials ----
        if (j0 + 31u > w_first || (a.window != 0u && j0 + a.window <= w_last)) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t qpos = w_first + mt * 16 + (e >> 1) * 8 + g;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t j = j0 + i * 8 + 2 * t + (e & 1);
                        if (j > qpos || (a.window != 0u && j + a.window <= qpos)) s[mt][i][e] = -INFINITY;
                    }
                }
        }
        uint32_t pa[2][2][4];  // the weights as A fragments of the second product
        bool moved = false;
        float alpha[2][2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float mx = s[mt][0][2 * h];
#pragma unroll
                for (int i = 0; i < 4; ++i) mx = fmaxf(mx, fmaxf(s[mt][i][2 * h], s[mt][i][2 * h + 1]));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                const float m_new = fmaxf(m_run[mt][h], mx * a.scale_log2e);
                const float m_use = m_new == -INFINITY ? 0.0f : m_new;  // nothing visible yet: every weight is 0
                alpha[mt][h] = exp2f(m_run[mt][h] - m_use);             // m_run = -inf gives 0
                moved = moved || m_new != m_run[mt][h];
                m_run[mt][h] = m_new;
                float rs = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float p0 = exp2f(fmaf(s[mt][i][2 * h], a.scale_log2e, -m_use));
                    const float p1 = exp2f(fmaf(s[mt][i][2 * h + 1], a.scale_log2e, -m_use));
                    rs += p0 + p1;
                    pa[mt][i >> 1][(i & 1) * 2 + h] = pack_h2(p0, p1);
                }
                l_run[mt][h] = l_run[mt][h] * alpha[mt][h] + rs;  // (this thread's keys; the quad is added at the end)
            }
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int i = 0; i < DV / 8; ++i) {
                    o[mt][i][0] *= alpha[mt][0];
                    o[mt][i][1] *= alpha[mt][0];
                    o[mt][i][2] *= alpha[mt][1];
                    o[mt][i][3] *= alpha[mt][1];
                }
        }
        // ---- O += P V ----
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
#pragma unroll
            for (int dp = 0; dp < DV / 16; ++dp) {  // two dim n-tiles per ldmatrix
                uint32_t b0, b1, b2, b3;
                const uint32_t row = sp * 32 + kk * 16 + (m & 1u) * 8 + (lane & 7), chunk = dp * 2 + (m >> 1);
                ldsm_x4_t(sV + sw<C::kVPitch>(row, chunk), b0, b1, b2, b3);
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    mma_f16(o[mt][2 * dp], pa[mt][kk][0], pa[mt][kk][1], pa[mt][kk][2], pa[mt][kk][3], b0, b1);
                    mma_f16(o[mt][2 * dp + 1], pa[mt][kk][0], pa[mt][kk][1], pa[mt][kk][2], pa[mt][kk][3], b2, b3);
                }
            }
        }
    }
    // ---- the splits' results, brought to one maximum and added in order; normalise and store ----
    __syncthreads();
    float *sO = (float *)sKV, *sM = sO + BQ * C::kOPitch, *sL = sM + SP * BQ;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float l = l_run[mt][h];
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            const int row = rw * 32 + mt * 16 + h * 8 + g;
            if (t == 0) {
                sM[sp * BQ + row] = m_run[mt][h];
                sL[sp * BQ + row] = l;
            }
        }
    __syncthreads();
    float inv[2][2];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = rw * 32 + mt * 16 + h * 8 + g;
            float mx = -INFINITY, l = 0.0f;
#pragma unroll
            for (int p = 0; p < SP; ++p) mx = fmaxf(mx, sM[p * BQ + row]);
            if (mx == -INFINITY) mx = 0.0f;  // (a row past the run)
#pragma unroll
            for (int p = 0; p < SP; ++p) l += sL[p * BQ + row] * exp2f(sM[p * BQ + row] - mx);
            inv[mt][h] = exp2f(m_run[mt][h] - mx) / l;
        }
#pragma unroll 1
    for (int p = 0; p < SP; ++p) {
        if (sp == p) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float *dst = sO + (rw * 32 + mt * 16 + h * 8 + g) * C::kOPitch + 2 * t;
#pragma unroll
                    for (int i = 0; i < DV / 8; ++i) {
                        float2 v = make_float2(o[mt][i][2 * h] * inv[mt][h], o[mt][i][2 * h + 1] * inv[mt][h]);
                        if (p > 0) {
                            const float2 w = *(const float2 *)(dst + i * 8);
                            v.x += w.x;
                            v.y += w.y;
                        }
                        *(float2 *)(dst + i * 8) = v;
                    }
                }
        }
        __syncthreads();
    }
    for (int i = tid; i < BQ * (DV / 4); i += kChunkThreads) {
        const uint32_t r = i / (DV / 4), c = i % (DV / 4);
        if (q0 + r >= n) break;
        const float4 v = *(const float4 *)(sO + r * C::kOPitch + c * 4);
        const size_t at = ((size_t)(row0 + q0 + r) * a.heads + head) * HD + dv0 + c * 4;
        if (a.out_f16) *(uint2 *)((__half *)a.out + at) = make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
        else *(float4 *)((float *)a.out + at) = v;
    }
}

// The cache rows of a launch's runs: k normed, rotated and rounded, v rounded.  One warp per (row, KV head).
template <int HD>
__global__ void __launch_bounds__(256) kv_store_rows_kernel(const float *k, const float *v, const float *k_norm,
                                                            const float *inv_freq, __half *kc, __half *vc, size_t seq_stride,
                                                            uint32_t kvh, uint32_t n_rot, uint32_t cap, float eps,
                                                            const __grid_constant__ attn_segs segs) {
    constexpr int R = HD / 32;
    const uint32_t lane = threadIdx.x & 31u, vec = blockIdx.x * 8u + (threadIdx.x >> 5);
    tmdev::pdl_wait();
    tmdev::pdl_trigger();
    if (vec >= segs.row0[segs.n] * kvh) return;
    const uint32_t row = vec / kvh, kh = vec % kvh;
    uint32_t seg = 0;
    while (seg + 1u < segs.n && row >= segs.row0[seg + 1]) ++seg;
    const uint32_t pos = segs.pos0[seg] + row - segs.row0[seg];
    float x[R], y[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        x[r] = k[(size_t)vec * HD + lane + 32 * r];
        y[r] = v[(size_t)vec * HD + lane + 32 * r];
    }
    norm_rope_row<R>(x, k_norm, inv_freq, n_rot, pos, eps, lane);
    const size_t dst = (size_t)segs.seq[seg] * seq_stride + ((size_t)kh * cap + pos) * HD + lane;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        kc[dst + 32 * r] = __float2half_rn(x[r]);
        vc[dst + 32 * r] = __float2half_rn(y[r]);
    }
}

// Per-head RMS norm of q and k, split-half RoPE at pos0 + t, f16 K/V store: the four launches that
// precede chunk attention (rmsnorm x2, rope, kv_store) as one.  One warp per (token, vector),
// vectors = query heads, then KV heads; q is normed and rotated in place, k is normed, rotated and
// written to the cache together with v (k itself is left as it was).  Warp-shuffle sum of squares,
// so the low bits differ from the one-CTA-per-row norm: part of the tolerance-qualified prefill.
__global__ void __launch_bounds__(256) qk_prep_chunk_kernel(float *q, const float *k, const float *v,
                                                             const float *q_norm, const float *k_norm,
                                                             const float *inv_freq, __half *kc, __half *vc,
                                                             uint32_t heads, uint32_t kvh, uint32_t hd, uint32_t n_rot,
                                                             uint32_t pos0, uint32_t cap, uint32_t n, float eps) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t vec = blockIdx.x * 8u + (threadIdx.x >> 5), per_tok = heads + kvh;
    if (vec >= n * per_tok) return;
    const uint32_t t = vec / per_tok, h = vec % per_tok;
    const bool is_k = h >= heads;
    const uint32_t kh = h - heads;
    float *qrow = q + ((size_t)t * heads + h) * hd;
    const float *src = is_k ? k + ((size_t)t * kvh + kh) * hd : qrow;
    const float *nw = is_k ? k_norm : q_norm;
    constexpr int kMax = 8;  // head dims up to 256
    float x[kMax];
    float ss = 0.0f;
#pragma unroll
    for (int r = 0; r < kMax; ++r) {
        const uint32_t e = lane + 32u * r;
        x[r] = e < hd ? src[e] : 0.0f;
        ss = fmaf(x[r], x[r], ss);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float inv = 1.0f / sqrtf(ss / (float)hd + eps);
#pragma unroll
    for (int r = 0; r < kMax; ++r) {
        const uint32_t e = lane + 32u * r;
        if (e < hd) x[r] = x[r] * inv * nw[e];
    }
    // Pairs (i, i + n_rot/2): with lane-strided elements the partner sits r_half registers away in the
    // same lane when n_rot/2 is a multiple of 32, otherwise it is fetched from another lane.
    const uint32_t half = n_rot / 2u, pos = pos0 + t;
    float y[kMax];
#pragma unroll
    for (int r = 0; r < kMax; ++r) y[r] = x[r];
#pragma unroll
    for (int r = 0; r < kMax; ++r) {
        const uint32_t e = lane + 32u * r;
        // partner element index and whether e is the first or the second member of its pair
        const bool first = e < half, second = e >= half && e < n_rot;
        const uint32_t pe = first ? e + half : e - half;
        float partner = 0.0f;
        // the partner lives at register (pe / 32) of lane (pe % 32); when half the rotated width is a
        // multiple of 32 (head sizes 64 and up, fully rotated) that is this lane: no shuffles
        if ((half & 31u) == 0u) {
#pragma unroll
            for (int rr = 0; rr < kMax; ++rr)
                if ((first || second) && (uint32_t)rr == (pe >> 5)) partner = x[rr];
        } else {
#pragma unroll
            for (int rr = 0; rr < kMax; ++rr) {
                const float cand = __shfl_sync(0xffffffffu, x[rr], (int)(pe & 31u));
                if ((first || second) && (uint32_t)rr == (pe >> 5)) partner = cand;
            }
        }
        if (first || second) {
            const uint32_t i = first ? e : e - half;
            float sn, cs;
            sincosf((float)pos * inv_freq[i], &sn, &cs);
            y[r] = first ? x[r] * cs - partner * sn : partner * sn + x[r] * cs;
        }
    }
    if (!is_k) {
#pragma unroll
        for (int r = 0; r < kMax; ++r) {
            const uint32_t e = lane + 32u * r;
            if (e < hd) qrow[e] = y[r];
        }
    } else {
        const float *vsrc = v + ((size_t)t * kvh + kh) * hd;
        const size_t dst = ((size_t)kh * cap + pos) * hd;
#pragma unroll
        for (int r = 0; r < kMax; ++r) {
            const uint32_t e = lane + 32u * r;
            if (e < hd) {
                kc[dst + e] = __float2half_rn(y[r]);
                vc[dst + e] = __float2half_rn(vsrc[e]);
            }
        }
    }
}

// ---- decode attention for many sequences on the tensor cores ---------------------------------
// The per-token core (per-head q/k RMS norm, RoPE, f16 KV store, windowed causal attention) for one
// row per sequence, throughput form: when tens of sequences decode together the step reads every
// sequence's K and V rows and is bandwidth-bound, which the latency-optimised kernel (scalar dot
// products, two threads per key) cannot feed.  Here one CTA of 4 warps serves ONE (sequence, KV head,
// equal run of 64-key tiles): the G query heads of the group are the rows of a 16-row MMA tile,
// K/V tiles arrive by cp.async (a ring of two or three), warp w owns keys 16w..16w+15 of every tile with its
// own running (max, sum, output), the four are merged through shared memory, and the splits of a
// (sequence, KV head) by last arrival through `scratch` (no waiting).  Same mathematics as the other
// decode kernels, f16 Q and softmax weights, base-2 exponentials: tolerance-qualified.
//   scratch (per sequence): float part[kv_heads][nsplit][G][HD + 2] = (m, l, o[HD]); then, at the offset
//   the other decode kernels use, u32 count[kv_heads] (left at zero).
struct decode_mma_args {
    const float *q, *k, *v, *q_norm, *k_norm, *inv_freq;
    __half *kc, *vc;
    float *out, *scratch;
    const uint32_t *pos;
    uint32_t *status;
    uint32_t kv_heads, cap, window, splits, count_off;  // count_off: floats from a sequence's scratch to its counters
    float eps, scale_log2e;
    size_t sq, sk, sv, so, scache, sscratch;  // element strides between sequences
};

template <int G, int HD, uint32_t kDecodeStages>
__global__ void __launch_bounds__(kThreads) attention_decode_mma_kernel(const decode_mma_args a) {
    constexpr int PITCH = HD * 2, EPL = HD / 32;
    constexpr uint32_t kQBytes = 16 * PITCH, kTile = kBKV * PITCH, kStage = 2 * kTile;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *sQ = smem, *sKV = smem + kQBytes;
    __shared__ __align__(16) __half kh[HD];
    __shared__ __align__(16) __half vh[HD];
    __shared__ float wm[4][G], wl[4][G];
    __shared__ uint32_t s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t kvh = blockIdx.x, split = blockIdx.y;
    const size_t sidx = blockIdx.z;
    const float *q = a.q + sidx * a.sq, *k = a.k + sidx * a.sk, *v = a.v + sidx * a.sv;
    __half *kc = a.kc + sidx * a.scache + (size_t)kvh * a.cap * HD, *vc = a.vc + sidx * a.scache + (size_t)kvh * a.cap * HD;
    float *out = a.out + sidx * a.so, *scratch = a.scratch + sidx * a.sscratch;
    // The tiles of a sequence at position p that this split takes: equal runs.
    uint32_t start, last_tile, tile_lo, tile_hi, nact;
    auto take = [&](uint32_t p) {
        const uint32_t n = p + 1u;
        start = (a.window != 0u && n > a.window) ? n - a.window : 0u;
        last_tile = p / kBKV;
        const uint32_t first_tile = start / kBKV, used = last_tile - first_tile + 1u;
        const uint32_t per = (used + gridDim.y - 1u) / gridDim.y;
        nact = (used + per - 1u) / per;  // splits of this (sequence, KV head) with work
        tile_lo = first_tile + split * per;
        tile_hi = min(tile_lo + per - 1u, last_tile);
    };
    // Before the wait, as if the position stood already: cached rows towards L2 (never closer: an earlier step's call
    // may still be storing one), the rotation's angles, the padding rows of Q.
    const uint32_t hint = min(*(const volatile uint32_t *)(a.pos + sidx), a.cap - 1u);
    take(hint);
    if (tile_lo <= last_tile)
        for (uint32_t j = tile_lo * kBKV + tid / 2; j < min((tile_hi + 1u) * kBKV, hint); j += kThreads / 2)
#pragma unroll
            for (uint32_t c = 0; c < PITCH; c += 128u)
                asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)((tid & 1 ? vc : kc) + (size_t)j * HD) + c));
    float sn[EPL / 2], cs[EPL / 2];
    auto angles = [&](uint32_t p) {
#pragma unroll
        for (int r = 0; r < EPL / 2; ++r) sincosf((float)p * a.inv_freq[lane + 32 * r], &sn[r], &cs[r]);
    };
    angles(hint);
    for (int i = tid; i < 16 * (HD / 8); i += kThreads) *(uint4 *)(sQ + i * 16) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    float x[EPL], nw[EPL];  // warp w < G: head w; warp G: the new key
    auto fetch = [&](int vec) {
        const float *src = vec == G ? k + (size_t)kvh * HD : q + ((size_t)kvh * G + vec) * HD;
        const float *wsrc = vec == G ? a.k_norm : a.q_norm;
#pragma unroll
        for (int r = 0; r < EPL; ++r) {
            x[r] = src[lane + 32 * r];
            nw[r] = wsrc[lane + 32 * r];
        }
    };
    if (warp <= G) fetch(warp);  // (with the position's own trip)
    const uint32_t pos = a.pos[sidx];
    if (pos >= a.cap) {
        if (tid == 0 && split == 0 && kvh == 0) atomicOr(a.status, TM_CUDA_STATUS_PAST_CAPACITY);
        return;
    }
    if (pos != hint) {
        take(pos);
        angles(pos);
    }
    if (tile_lo > last_tile) return;
    const bool owns_new = tile_hi == last_tile;

    auto load_tile = [&](uint32_t tile, int stage) {
        unsigned char *sK = sKV + stage * kStage, *sV = sK + kTile;
        const uint32_t j0 = tile * kBKV;
        constexpr int CH = HD / 8;  // 16-byte chunks per row
        for (int i = tid; i < kBKV * CH; i += kThreads) {
            const uint32_t r = i / CH, c = i % CH;
            const uint32_t j = min(j0 + r, pos);  // rows past the position repeat its row (masked below)
            cp_async16(smem_u32(sK) + sw<PITCH>(r, c), kc + (size_t)j * HD + c * 8);
            cp_async16(smem_u32(sV) + sw<PITCH>(r, c), vc + (size_t)j * HD + c * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (uint32_t i = 0; i < kDecodeStages - 1; ++i)
        if (tile_lo + i <= tile_hi) load_tile(tile_lo + i, (int)i);
        else asm volatile("cp.async.commit_group;" ::: "memory");

    // ---- q_0..q_{G-1} (and k, v for the split that holds the position): RMS norm + RoPE, a warp each ----
    for (int vec = warp; vec < G + (owns_new ? 1 : 0); vec += kThreads / 32) {
        const bool is_k = vec == G;
        if (vec != warp) fetch(vec);
        float ss = 0.0f;
#pragma unroll
        for (int r = 0; r < EPL; ++r) ss = fmaf(x[r], x[r], ss);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
        const float inv = 1.0f / sqrtf(ss / (float)HD + a.eps);
#pragma unroll
        for (int r = 0; r < EPL; ++r) x[r] = x[r] * inv * nw[r];
        // full rotation: pair (i, i + HD/2), i = lane + 32 r, has both members in this lane
#pragma unroll
        for (int r = 0; r < EPL / 2; ++r) {
            const float a0 = x[r], b0 = x[r + EPL / 2];
            x[r] = a0 * cs[r] - b0 * sn[r];
            x[r + EPL / 2] = a0 * sn[r] + b0 * cs[r];
        }
        if (is_k) {
            const float *vsrc = v + (size_t)kvh * HD;
#pragma unroll
            for (int r = 0; r < EPL; ++r) {
                const uint32_t e = lane + 32 * r;
                const __half hk = __float2half_rn(x[r]), hv = __float2half_rn(vsrc[e]);
                kh[e] = hk;
                vh[e] = hv;
                kc[(size_t)pos * HD + e] = hk;
                vc[(size_t)pos * HD + e] = hv;
            }
        } else {
#pragma unroll
            for (int r = 0; r < EPL; ++r) {
                const uint32_t e = lane + 32 * r;
                *(__half *)(sQ + sw<PITCH>((uint32_t)vec, e >> 3) + (e & 7u) * 2u) = __float2half_rn(x[r]);
            }
        }
    }

    // This warp's running state over its 16 keys of every tile; rows g < G are the group's heads.
    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
    float m_run = -INFINITY, l_run = 0.0f;
    const bool row_live = g < G;

    for (uint32_t tile = tile_lo; tile <= tile_hi; ++tile) {
        const int stage = (int)((tile - tile_lo) % kDecodeStages);
        asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeStages - 2) : "memory");
        __syncthreads();  // the tile has landed, the one before it is done (first time round: Q and the new row are written)
        if (tile + kDecodeStages - 1 <= tile_hi) load_tile(tile + kDecodeStages - 1, (int)((tile - tile_lo + kDecodeStages - 1) % kDecodeStages));
        else asm volatile("cp.async.commit_group;" ::: "memory");
        const uint32_t j0 = tile * kBKV;
        if (tile == last_tile) {  // the position's own row comes from this step, not from the cache
            const uint32_t r = pos - j0;
            unsigned char *sK = sKV + stage * kStage, *sV = sK + kTile;
            if (tid < HD / 8) *(uint4 *)(sK + sw<PITCH>(r, tid)) = *(const uint4 *)(kh + tid * 8);
            else if (tid < HD / 4) *(uint4 *)(sV + sw<PITCH>(r, tid - HD / 8)) = *(const uint4 *)(vh + (tid - HD / 8) * 8);
            __syncthreads();
        }
        const uint32_t sK = smem_u32(sKV + stage * kStage), sV = sK + kTile;
        // ---- S = Q K^T: 16 rows x this warp's 16 keys ----
        float s[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.0f;
#pragma unroll
        for (int kt = 0; kt < HD / 16; ++kt) {
            uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
            const uint32_t m = lane >> 3;
            ldsm_x4(smem_u32(sQ) + sw<PITCH>((m & 1u) * 8 + (lane & 7), kt * 2 + (m >> 1)), a0, a1, a2, a3);
            ldsm_x4(sK + sw<PITCH>(warp * 16 + (m >> 1) * 8 + (lane & 7), kt * 2 + (m & 1u)), b0, b1, b2, b3);
            mma_f16(s[0], a0, a1, a2, a3, b0, b1);
            mma_f16(s[1], a0, a1, a2, a3, b2, b3);
        }
        // ---- mask, running maximum, weights (rows g only: rows g + 8 are padding) ----
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint32_t j = j0 + warp * 16 + i * 8 + 2 * t + e;
                const bool vis = row_live && j >= start && j <= pos;
                s[i][e] = vis ? s[i][e] * a.scale_log2e : -INFINITY;
                mx = fmaxf(mx, s[i][e]);
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m_run, mx);
        const float m_use = m_new == -INFINITY ? 0.0f : m_new;
        const float alpha = exp2f(m_run - m_use);
        m_run = m_new;
        const float p00 = exp2f(s[0][0] - m_use), p01 = exp2f(s[0][1] - m_use);
        const float p10 = exp2f(s[1][0] - m_use), p11 = exp2f(s[1][1] - m_use);
        float rs = p00 + p01 + p10 + p11;
        rs += __shfl_xor_sync(0xffffffffu, rs, 1);
        rs += __shfl_xor_sync(0xffffffffu, rs, 2);
        l_run = l_run * alpha + rs;
        const uint32_t pa0 = pack_h2(p00, p01), pa2 = pack_h2(p10, p11);  // rows g: keys 0-7 / 8-15; rows g + 8: zero
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) {
            o[i][0] *= alpha;
            o[i][1] *= alpha;
        }
        // ---- O += P V over this warp's 16 keys.  A row that weighs 0 is read as zeros (from Q's last row), because 0 times an
        // infinity is NaN; zero-filled copies of such rows took 3 to 8 % longer with one head a KV head. ----
        const uint32_t vm = lane >> 3, vr = warp * 16 + (vm & 1u) * 8 + (lane & 7), zeros = smem_u32(sQ) + sw<PITCH>(15u, 0u);
        const bool seen = j0 + vr - start <= pos - start;
#pragma unroll
        for (int dp = 0; dp < HD / 16; ++dp) {
            uint32_t b0, b1, b2, b3;
            ldsm_x4_t(seen ? sV + sw<PITCH>(vr, dp * 2 + (vm >> 1)) : zeros, b0, b1, b2, b3);
            mma_f16(o[2 * dp], pa0, 0u, pa2, 0u, b0, b1);
            mma_f16(o[2 * dp + 1], pa0, 0u, pa2, 0u, b2, b3);
        }
    }
    __syncthreads();

    // ---- the four warps' (m, l, o) -> this split's; the K/V stages are free now ----
    float *wo = (float *)sKV;  // [4][G][HD]
    if (row_live) {
        if (t == 0) {
            wm[warp][g] = m_run;
            wl[warp][g] = l_run;
        }
#pragma unroll
        for (int i = 0; i < HD / 8; ++i)
            *(float2 *)(wo + ((size_t)warp * G + g) * HD + i * 8 + 2 * t) = make_float2(o[i][0], o[i][1]);
    }
    __syncthreads();
    constexpr uint32_t stride = HD + 2;
    const uint32_t nsplit = gridDim.y;
    float *part = scratch + ((size_t)kvh * nsplit + split) * G * stride;
    const bool single = nact == 1u;
    for (uint32_t i = tid; i < G * HD; i += kThreads) {
        const uint32_t gg = i / HD, d = i % HD;
        float M = fmaxf(fmaxf(wm[0][gg], wm[1][gg]), fmaxf(wm[2][gg], wm[3][gg]));
        float L = 0.0f, O = 0.0f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float f = exp2f(wm[w][gg] - M);  // a warp that saw no key: exp2(-inf) = 0
            L = fmaf(f, wl[w][gg], L);
            O = fmaf(f, wo[((size_t)w * G + gg) * HD + d], O);
        }
        if (single) {
            out[((size_t)kvh * G + gg) * HD + d] = O / L;
        } else {
            part[gg * stride + 2 + d] = O;
            if (d == 0) {
                part[gg * stride] = M;
                part[gg * stride + 1] = L;
            }
        }
    }
    if (single) return;
    __threadfence();
    __syncthreads();
    uint32_t *count = (uint32_t *)(scratch + a.count_off) + kvh;
    if (tid == 0) s_last = atomicAdd(count, 1u) == nact - 1u ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t i = tid; i < G * HD; i += kThreads) {
        const uint32_t gg = i / HD, d = i % HD;
        const float *base = scratch + (size_t)kvh * nsplit * G * stride + gg * stride;
        float M = -INFINITY, L = 0.0f, O = 0.0f;
        for (uint32_t s0 = 0; s0 < nact; s0 += 8) {
            float mb[8], lb[8], ob[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float *pb = base + (size_t)(s0 + c < nact ? s0 + c : nact - 1) * G * stride;
                mb[c] = __ldcg(pb);
                lb[c] = __ldcg(pb + 1);
                ob[c] = __ldcg(pb + 2 + d);
            }
            float mx = M;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (s0 + c < nact) mx = fmaxf(mx, mb[c]);
            const float al = exp2f(M - mx);
            L *= al;
            O *= al;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (s0 + c < nact) {
                    const float wgt = exp2f(mb[c] - mx);
                    L = fmaf(wgt, lb[c], L);
                    O = fmaf(wgt, ob[c], O);
                }
            M = mx;
        }
        out[((size_t)kvh * G + gg) * HD + d] = O / L;
    }
    if (tid == 0) *count = 0u;  // ready for the next launch on this stream
}

template <int G, int HD, uint32_t kDecodeStages>
cudaError_t launch_decode_mma(tm_cuda_ctx *ctx, const decode_mma_args &a, uint32_t n_seq) {
    constexpr uint32_t kBytes = 16 * HD * 2 + kDecodeStages * 2 * kBKV * HD * 2;
    static std::atomic<bool> attr_done[64] = {};
    const int device = ctx->device;
    if (device < 0 || device >= 64 || !attr_done[device].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(attention_decode_mma_kernel<G, HD, kDecodeStages>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBytes);
        if (e != cudaSuccess) return e;
        if (device >= 0 && device < 64) attr_done[device].store(true, std::memory_order_release);
    }
    const dim3 grid(a.kv_heads, a.splits, n_seq);
    return tm_launch_pdl(ctx, attention_decode_mma_kernel<G, HD, kDecodeStages>, grid, dim3(kThreads), kBytes, a);
}

// The kernel masks scores with -inf and takes their maximum before it scales them, which needs a positive factor: a
// negative scale becomes its magnitude times negated queries, zero becomes any factor times zero queries.
void attn_scale(attn_args &a, float scale) {
    a.q_sign = scale < 0.0f ? -1.0f : scale == 0.0f ? 0.0f : 1.0f;
    a.scale_log2e = (scale == 0.0f ? 1.0f : scale * a.q_sign) * 1.4426950408889634f;
}

attn_segs attn_segments(uint32_t pos0, uint32_t n) {
    attn_segs s;
    s.n = 1;
    s.row0[0] = 0;
    s.row0[1] = n;
    s.pos0[0] = pos0;
    s.seq[0] = 0;
    return s;
}

template <int HD, int RW>
cudaError_t launch_attn_rows(tm_cuda_ctx *ctx, const attn_args &a, uint32_t tiles) {
    using C = attn_cfg<HD, RW>;
    const int device = ctx->device;
    static std::atomic<bool> attr_done[64] = {};  // per device; contexts of a process share it
    if (device < 0 || device >= 64 || !attr_done[device].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(attention_chunk_mma_kernel<HD, RW>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kBytes);
        if (e != cudaSuccess) return e;
        if (device >= 0 && device < 64) attr_done[device].store(true, std::memory_order_release);
    }
    return tm_launch_pdl(ctx, attention_chunk_mma_kernel<HD, RW>, dim3(tiles * a.heads, HD / C::kDV), dim3(kChunkThreads),
                         C::kBytes, a);
}
// 128 queries a CTA (half the key and value traffic from L2) where that leaves every SM two CTAs, else 64.
template <int HD>
cudaError_t launch_attn(tm_cuda_ctx *ctx, const attn_args &a) {
    uint32_t t64 = 0, t128 = 0;
    for (uint32_t i = 0; i < a.segs.n; ++i) {
        const uint32_t n = a.segs.row0[i + 1] - a.segs.row0[i];
        t64 += (n + 63u) / 64u;
        t128 += (n + 127u) / 128u;
    }
    if ((uint64_t)t128 * a.heads * (HD / attn_cfg<HD, 4>::kDV) >= 2u * (uint64_t)ctx->sm_count)
        return launch_attn_rows<HD, 4>(ctx, a, t128);
    return launch_attn_rows<HD, 2>(ctx, a, t64);
}

}  // namespace

// Whether the tensor-core decode form serves this geometry.
bool tm_attention_decode_mma_ok(uint32_t heads, uint32_t kv_heads, uint32_t hd, uint32_t n_rot) {
    const uint32_t g = kv_heads ? heads / kv_heads : 0;
    return hd == 128 && n_rot == hd && (g == 1 || g == 2 || g == 4);
}

// One launch for n_seq sequences (pointers are sequence 0's; strides in elements between sequences).
cudaError_t tm_attention_decode_mma_launch(tm_cuda_ctx *ctx, const float *q, const float *k, const float *v,
                                           const float *qn, const float *kn, const float *inv_freq, void *kc, void *vc,
                                           float *out, float *scratch, const uint32_t *pos, uint32_t *status,
                                           uint32_t heads, uint32_t kv_heads, uint32_t hd, uint32_t cap, uint32_t window,
                                           float eps, float scale, uint32_t n_seq, size_t sq, size_t skv, size_t so,
                                           size_t scache, size_t sscratch, uint32_t count_off) {
    decode_mma_args a;
    a.q = q; a.k = k; a.v = v; a.q_norm = qn; a.k_norm = kn; a.inv_freq = inv_freq;
    a.kc = (__half *)kc; a.vc = (__half *)vc;
    a.out = out; a.scratch = scratch; a.pos = pos; a.status = status;
    a.kv_heads = kv_heads; a.cap = cap; a.window = window;
    a.count_off = count_off;
    a.eps = eps;
    a.scale_log2e = scale * 1.4426950408889634f;
    a.sq = sq; a.sk = a.sv = skv; a.so = so; a.scache = scache; a.sscratch = sscratch;
    // As many splits as find a place at once (two CTAs of three tiles in shared memory to an SM): the splits of a head
    // meet through memory (store, fence, atomic, reload: 5 us), so many sequences are better off without any.  Three
    // CTAs of two tiles where one CTA a head is more than that.  (By the capacity, 1024 CTAs of which half had nothing
    // to do: 32 sequences at 100 to 460 of 1024 positions 13.9 us, now 12.1; 32 of 50 to 250, groups of four heads,
    // 11.5, now 8.4; 4 at 200 to 620 16.2, now 12.8.)
    const uint32_t n_tiles = (cap + kBKV - 1) / kBKV, heads_all = n_seq * kv_heads, places = 2u * (uint32_t)ctx->sm_count;
    const uint32_t splits = places / heads_all;
    a.splits = splits < 1u ? 1u : splits > n_tiles ? n_tiles : splits;
    (void)hd;
    const bool deep = heads_all <= places;
    switch (heads / kv_heads) {
        case 1: return deep ? launch_decode_mma<1, 128, 3>(ctx, a, n_seq) : launch_decode_mma<1, 128, 2>(ctx, a, n_seq);
        case 2: return deep ? launch_decode_mma<2, 128, 3>(ctx, a, n_seq) : launch_decode_mma<2, 128, 2>(ctx, a, n_seq);
        default: return deep ? launch_decode_mma<4, 128, 3>(ctx, a, n_seq) : launch_decode_mma<4, 128, 2>(ctx, a, n_seq);
    }
}

extern "C" {

int tm_cuda_attention_chunk_mma_supported(uint32_t head_dim) {
    return head_dim == 32 || head_dim == 64 || head_dim == 128 || head_dim == 256;
}

int tm_cuda_qk_prep_chunk(tm_cuda_ctx *ctx, tm_cuda_buffer *q, tm_cuda_buffer *k, tm_cuda_buffer *v,
                          tm_cuda_buffer *q_norm, tm_cuda_buffer *k_norm, tm_cuda_buffer *inv_freq,
                          tm_cuda_buffer *k_cache, tm_cuda_buffer *v_cache, uint32_t heads, uint32_t kv_heads,
                          uint32_t head_dim, uint32_t n_rot, uint32_t pos0, uint32_t cap, uint32_t n, float eps,
                          char *err, size_t err_cap) {
    TM_ENTER();
    if (heads == 0 || kv_heads == 0 || head_dim == 0 || head_dim > 256 || n_rot == 0 || n_rot > head_dim ||
        n_rot % 2 != 0 || n == 0 || (size_t)pos0 + n > cap)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS,
                       "q/k preparation: heads %u/%u, head_dim %u (<= 256), n_rot %u, rows %u..%u of capacity %u", heads,
                       kv_heads, head_dim, n_rot, pos0, pos0 + n, cap);
    const size_t plane = (size_t)kv_heads * cap * head_dim * 2;
    TM_CHECK_BUF(q, (size_t)n * heads * head_dim * 4, "q");
    TM_CHECK_BUF(k, (size_t)n * kv_heads * head_dim * 4, "k");
    TM_CHECK_BUF(v, (size_t)n * kv_heads * head_dim * 4, "v");
    TM_CHECK_IN(q_norm, (size_t)head_dim * 4, "q norm");
    TM_CHECK_IN(k_norm, (size_t)head_dim * 4, "k norm");
    TM_CHECK_IN(inv_freq, (size_t)(n_rot / 2) * 4, "inv_freq");
    TM_CHECK_BUF(k_cache, plane, "K cache");
    TM_CHECK_BUF(v_cache, plane, "V cache");
    TM_OP_BEGIN("qk_prep_chunk");
    const uint32_t vecs = n * (heads + kv_heads);
    qk_prep_chunk_kernel<<<(vecs + 7) / 8, 256, 0, ctx->stream>>>(
        (float *)q->dev, (const float *)k->dev, (const float *)v->dev, (const float *)q_norm->dev,
        (const float *)k_norm->dev, (const float *)inv_freq->dev, (__half *)k_cache->dev, (__half *)v_cache->dev, heads,
        kv_heads, head_dim, n_rot, pos0, cap, n, eps);
    TM_OP_END(1);
}

int tm_cuda_attention_chunk_mma(tm_cuda_ctx *ctx, tm_cuda_buffer *q, tm_cuda_buffer *k_cache, tm_cuda_buffer *v_cache,
                                tm_cuda_buffer *out, uint32_t heads, uint32_t pos0, uint32_t cap, uint32_t head_dim,
                                uint32_t group, float scale, uint32_t n, uint32_t window, char *err, size_t err_cap) {
    TM_ENTER();
    if (!tm_cuda_attention_chunk_mma_supported(head_dim) || heads == 0 || group == 0 || heads % group != 0 || n == 0 ||
        cap == 0 || (size_t)pos0 + n > cap)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS,
                       "tensor-core chunk attention: heads %u, group %u, head_dim %u (32, 64, 128 or 256), rows "
                       "%u..%u of capacity %u", heads, group, head_dim, pos0, pos0 + n, cap);
    const uint32_t kv_heads = heads / group;
    const size_t plane = (size_t)kv_heads * cap * head_dim * 2;
    TM_CHECK_IN(q, (size_t)n * heads * head_dim * 4, "q");
    TM_CHECK_BUF(out, (size_t)n * heads * head_dim * 4, "attention output");
    TM_CHECK_IN(k_cache, plane, "K cache");
    TM_CHECK_IN(v_cache, plane, "V cache");
    if (((size_t)q->dev | (size_t)out->dev | (size_t)k_cache->dev | (size_t)v_cache->dev) & 15u)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "tensor-core chunk attention needs 16-byte aligned buffers");
    attn_args a;
    a.q = (const float *)q->dev;
    a.q_norm = nullptr;  // the queries are normed and rotated already
    a.kc = (const __half *)k_cache->dev;
    a.vc = (const __half *)v_cache->dev;
    a.out = out->dev;
    a.out_f16 = 0;
    a.heads = heads;
    a.group = group;
    a.cap = cap;
    a.window = window;
    a.seq_stride = 0;
    attn_scale(a, scale);
    a.segs = attn_segments(pos0, n);
    TM_OP_BEGIN("attention_chunk_mma");
    cudaError_t e = head_dim == 32    ? launch_attn<32>(ctx, a)
                    : head_dim == 64  ? launch_attn<64>(ctx, a)
                    : head_dim == 128 ? launch_attn<128>(ctx, a)
                                      : launch_attn<256>(ctx, a);
    TM_CUDA_TRY(e);
    TM_OP_END(1);
}

int tm_cuda_attention_prefill(tm_cuda_ctx *ctx, tm_cuda_buffer *q, tm_cuda_buffer *k, tm_cuda_buffer *v,
                              tm_cuda_buffer *q_norm, tm_cuda_buffer *k_norm, tm_cuda_buffer *inv_freq,
                              tm_cuda_buffer *k_cache, tm_cuda_buffer *v_cache, tm_cuda_buffer *out, uint32_t heads,
                              uint32_t kv_heads, uint32_t head_dim, uint32_t n_rot, uint32_t cap, uint32_t window,
                              float eps, float scale, int out_f16, uint32_t n_segments, const uint32_t *segments,
                              char *err, size_t err_cap) {
    TM_ENTER();
    if (!tm_cuda_attention_chunk_mma_supported(head_dim) || heads == 0 || kv_heads == 0 || heads % kv_heads != 0 ||
        n_rot == 0 || n_rot > head_dim || n_rot % 2 != 0 || cap == 0 || n_segments == 0 ||
        n_segments > TM_CUDA_PREFILL_SEGMENTS || !segments)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS,
                       "prefill attention: heads %u/%u, head_dim %u (32, 64, 128 or 256), n_rot %u, capacity %u, %u runs "
                       "(1 .. %u)", heads, kv_heads, head_dim, n_rot, cap, n_segments, (unsigned)TM_CUDA_PREFILL_SEGMENTS);
    attn_args a;
    a.segs.n = n_segments;
    uint32_t seqs = 0;
    size_t rows = 0;
    for (uint32_t i = 0; i < n_segments; ++i) {
        const uint32_t *s = segments + 3 * (size_t)i;
        if (s[2] == 0 || (size_t)s[1] + s[2] > cap || s[0] > 0xfffffffeu)
            return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "run %u: rows %u..%zu of capacity %u", i, s[1],
                           (size_t)s[1] + s[2], cap);
        a.segs.row0[i] = (uint32_t)rows;
        a.segs.seq[i] = s[0];
        a.segs.pos0[i] = s[1];
        rows += s[2];
        if (s[0] >= seqs) seqs = s[0] + 1u;
    }
    if (rows * (heads + kv_heads) > 0x7fffffffu)
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "prefill attention: %zu rows", rows);
    a.segs.row0[n_segments] = (uint32_t)rows;
    a.seq_stride = (size_t)kv_heads * cap * head_dim;
    TM_CHECK_BUF(q, rows * heads * head_dim * 4, "q");
    TM_CHECK_BUF(k, rows * kv_heads * head_dim * 4, "k");
    TM_CHECK_BUF(v, rows * kv_heads * head_dim * 4, "v");
    TM_CHECK_IN(q_norm, (size_t)head_dim * 4, "q norm");
    TM_CHECK_IN(k_norm, (size_t)head_dim * 4, "k norm");
    TM_CHECK_IN(inv_freq, (size_t)(n_rot / 2) * 4, "inv_freq");
    TM_CHECK_BUF(out, rows * heads * head_dim * (out_f16 ? 2 : 4), "attention output");
    TM_CHECK_BUF(k_cache, (size_t)seqs * a.seq_stride * 2, "K cache");
    TM_CHECK_BUF(v_cache, (size_t)seqs * a.seq_stride * 2, "V cache");
    if (((size_t)out->dev | (size_t)k_cache->dev | (size_t)v_cache->dev) & 15u)
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "prefill attention needs 16-byte aligned buffers");
    a.q = (const float *)q->dev;
    a.q_norm = (const float *)q_norm->dev;
    a.inv_freq = (const float *)inv_freq->dev;
    a.kc = (const __half *)k_cache->dev;
    a.vc = (const __half *)v_cache->dev;
    a.out = out->dev;
    a.out_f16 = out_f16 ? 1u : 0u;
    a.heads = heads;
    a.group = heads / kv_heads;
    a.cap = cap;
    a.window = window;
    a.n_rot = n_rot;
    a.eps = eps;
    attn_scale(a, scale);
    TM_OP_BEGIN("attention_prefill");
    const dim3 grid(((uint32_t)rows * kv_heads + 7u) / 8u);
    auto store = [&](auto kernel) {
        return tm_launch_pdl(ctx, kernel, grid, dim3(256), 0, (const float *)k->dev, (const float *)v->dev,
                             (const float *)k_norm->dev, a.inv_freq, (__half *)k_cache->dev, (__half *)v_cache->dev,
                             a.seq_stride, kv_heads, n_rot, cap, eps, a.segs);
    };
    TM_CUDA_TRY(head_dim == 32    ? store(kv_store_rows_kernel<32>)
                : head_dim == 64  ? store(kv_store_rows_kernel<64>)
                : head_dim == 128 ? store(kv_store_rows_kernel<128>)
                                  : store(kv_store_rows_kernel<256>));
    TM_CUDA_TRY(head_dim == 32    ? launch_attn<32>(ctx, a)
                : head_dim == 64  ? launch_attn<64>(ctx, a)
                : head_dim == 128 ? launch_attn<128>(ctx, a)
                                  : launch_attn<256>(ctx, a));
    TM_OP_END(2);
}

}  // extern "C"
