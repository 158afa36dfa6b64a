// The f16-operand multiply for a few rows of activations (a decode step of several sequences, a short prompt):
// Y[b, :] = W X[b, :] for b < batch <= 32, the numerical profile of the tcgen05 GEMM in tm_cuda_mma.cu (x and
// d * q rounded to binary16 once each, products summed in f32) on a kernel shaped like the decode GEMV.
//
// What bounds it: the weights' bytes, and below ~8 MB the chain launch -> activations -> products -> sum.  The
// tcgen05 kernel is bound by neither at these batches: its weight tile goes TMA -> shared memory -> registers ->
// tensor memory -> MMA as one serial chain of 0.7 us per 64 columns, 12-15 us for a 4096 x 1024 projection of 32
// rows that is 0.7 us of HBM traffic.  Here a warp reads int8 quants the way the GEMV does (16 bytes per lane
// and row through a cp.async ring), turns them into the A operand in registers -- 7 instructions per 4 weights,
// once for all rows of X -- and multiplies with m16n8k16 at most four token tiles.  At 32 rows that is 0.4 of the
// issue slots the weight stream leaves, so mma.sync suffices; from 33 rows on the tcgen05 kernel serves.
//
// Split.  A unit is 32 weight rows (two 16-row tiles, so that one read of the token fragments feeds two tiles).
// A cluster of P CTAs serves a unit, each CTA a P-th of K, each of its 8 warps every 8th 64-column chunk of that.
// Sums meet in a fixed order: the 8 warps through shared memory, the P CTAs through distributed shared memory -- no
// workspace, no counters.  P is the part count of least cost (see plan_rows).
//
// X.  A unit's columns of X are read by one warp each, so nothing is gained by keeping them in shared memory for one
// unit: a lane loads the 32 bytes of its 16 columns of a token straight into the B operand, while the weights that the
// warp asked for before the dependency wait are on their way.  That takes the round trip through shared memory and its
// barrier out of a chain that is all latency, and 40 KB of shared memory in place of 100-220 let two CTAs share an SM,
// so the next launch's weights are in flight while this one ends.  32 tokens by 6144 x 1024 6.9 -> 4.9 us, 1024 x 3072
// 5.7 -> 4.6, 4096 x 4096 13.2 -> 9.8, 1152 x 6912 15.6 -> 7.0; 19 tokens by 4096 x 1024 5.6 -> 4.0.
// Only up to 8 tokens, or 16 in a narrow matrix, by many units keep X staged, in CTAs that stay (STAGED): at 8 tokens 12288 x
// 4096 15.4 us against 17.4, 24576 x 4096 27.7 / 29.7, 151936 x 4096 128 / 143.  (At 16 tokens 18.5 / 19.1, 33.8 / 33.9, 152 /
// 163: two tiles of tokens are not worth it there, and from 24 tokens on it is the slower one, 26 / 20.)
#include "tm_cuda_internal.cuh"
#include "tm_cuda_device.cuh"

namespace {

constexpr int kWarps = 8, kThreads = 256;
constexpr uint32_t kSlot = 2048u + 128u;  // 32 rows x 64 quants, 32 rows x 2 scales
constexpr uint32_t kRowPad = 36;          // floats per token of a partial sum: lanes (g, t) land in 32 banks

enum : uint32_t { kPlain = 0, kSilu = 1, kGelu = 2 };

struct rows_args {
    const signed char *q;
    const unsigned short *d;
    const __half *x;       // [batch][cols]
    float *y[3];           // up to three consecutive row ranges with dense outputs of their own
    uint32_t part_end[3];  // exclusive row bound of each (multiples of 32 but the last)
    __half *act;           // gated forms: act(gate) * up, [batch][rows / 2]
    uint32_t rows, cols, batch, units, accumulate, mode, ring;
    uint32_t x32;          // X is 32-byte aligned: one load takes a lane's 16 columns
};

using tmdev::cluster_rank;
using tmdev::cluster_size;
using tmdev::cluster_sync;
using tmdev::ld_cluster;
using tmdev::mma_f16;

// Four quants -> two half2 of RN(d * q): bytes become f16 1024 + (q + 128) by permutes, minus 1152, times d.
__device__ __forceinline__ void dequant4(uint32_t w, __half2 d2, uint32_t &lo, uint32_t &hi) {
    const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0x6480));
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t p = __byte_perm(u, 0x64646464u, 0x4140), s = __byte_perm(u, 0x64646464u, 0x4342);
    const __half2 a = __hmul2(__hsub2(*(const __half2 *)&p, bias), d2);
    const __half2 b = __hmul2(__hsub2(*(const __half2 *)&s, bias), d2);
    lo = *(const uint32_t *)&a;
    hi = *(const uint32_t *)&b;
}

// Shared memory of a CTA that stages no activations: its ring, then its sums.
__host__ __device__ constexpr uint32_t ring_or_sums(uint32_t tok, uint32_t ring) {
    return kWarps * (ring * kSlot > tok * kRowPad * 4u ? ring * kSlot : tok * kRowPad * 4u);
}

template <int NT, bool STAGED>
__global__ void __launch_bounds__(kThreads, STAGED ? 1 : 2) q8_gemm_rows_kernel(const rows_args a) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr uint32_t kTok = NT * 8;
    const uint32_t P = cluster_size(), rank = P > 1 ? cluster_rank() : 0u;
    const uint32_t n_clusters = gridDim.x / P, cluster = blockIdx.x / P;
    const uint32_t warp = tmdev::warp_index(), lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const uint32_t n_chunks = a.cols / 64u, nb = a.cols / 32u;
    const uint32_t c0 = n_chunks * rank / P, c1 = n_chunks * (rank + 1) / P;
    const uint32_t kc_max = (n_chunks + P - 1) / P;
    const uint32_t xstride = kc_max * 128u + 16u;  // 16 mod 128: the 16-byte reads of 8 lanes hit distinct banks
    unsigned char *xs = smem;
    // [warp][token][kRowPad]; not STAGED, a CTA has one unit and the sums take the ring's place once it has been read
    float *red = (float *)(smem + (STAGED ? kTok * xstride : 0u));
    float *part = STAGED ? red + kWarps * kTok * kRowPad : (float *)(smem + ring_or_sums(kTok, a.ring));  // [2][token][32]
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(STAGED ? (unsigned char *)(part + (P > 1 ? 2 * kTok * 32 : 0)) : smem) +
                          warp * a.ring * kSlot;
    const uint32_t half_rows = a.rows / 2u;

    // Row r (0..31) of a unit: consecutive rows, or 16 gate rows and the 16 up rows they gate.
    auto row_of = [&](uint32_t unit, uint32_t r) -> uint32_t {
        if (a.mode == kPlain) return min(unit * 32u + r, a.rows - 1u);
        return unit * 16u + (r & 15u) + (r >= 16u ? half_rows : 0u);
    };
    uint32_t ld_unit = cluster, ld_c = c0 + warp;
    if (ld_c >= c1) ld_unit = a.units;  // fewer chunks than warps: this one only adds zeros
    auto issue = [&](uint32_t slot) {
        if (ld_unit < a.units) {
            const uint32_t dst = ring + slot * kSlot;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const signed char *p = a.q + (size_t)row_of(ld_unit, g + 8u * i) * a.cols + ld_c * 64u + t4 * 16u;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 512u + lane * 16u), "l"(p) : "memory");
            }
            const unsigned short *s = a.d + (size_t)row_of(ld_unit, lane) * nb + ld_c * 2u;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 2048u + lane * 4u), "l"(s) : "memory");
            ld_c += kWarps;
            if (ld_c >= c1) {
                ld_c = c0 + warp;
                ld_unit += n_clusters;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const uint32_t depth = a.ring;
    for (uint32_t i = 0; i < depth; ++i) issue(i);

    tmdev::pdl_trigger();
    tmdev::pdl_wait();
    uint32_t xb[STAGED ? 1 : NT][8];  // this lane's 16 columns of the chunk at hand, of token 8 n + g
    auto load_x = [&](int n, uint32_t c) {
        uint32_t(&v)[8] = xb[STAGED ? 0 : n];
        const uint32_t tok = (uint32_t)n * 8u + g;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0u;
        if (c >= c1 || tok >= a.batch) return;
        const __half *p = a.x + (size_t)tok * a.cols + c * 64u + t4 * 16u;
        if (a.x32) {
            asm volatile("ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                         : "l"(p)
                         : "memory");
        } else {
            const uint4 lo = __ldcg((const uint4 *)p), hi = __ldcg((const uint4 *)p + 1);
            v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
        }
    };
    if (!STAGED) {
#pragma unroll
        for (int n = 0; n < NT; ++n) load_x(n, c0 + warp);
    } else {  // this CTA's columns of X; rows past the batch are zero
        const uint32_t q16 = (c1 - c0) * 8u, total = kTok * q16;  // 16-byte pieces
        constexpr uint32_t kBatch = 8;
        for (uint32_t b = threadIdx.x; b < total; b += kThreads * kBatch) {
            int4 v[kBatch];
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                const uint32_t at = b + i * kThreads, t = at / q16, c = at % q16;
                v[i] = make_int4(0, 0, 0, 0);
                if (at < total && t < a.batch) v[i] = __ldcg((const int4 *)(a.x + (size_t)t * a.cols + c0 * 64u) + c);
            }
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                const uint32_t at = b + i * kThreads, t = at / q16, c = at % q16;
                if (at < total) *(int4 *)(xs + t * xstride + c * 16u) = v[i];
            }
        }
        __syncthreads();
    }

    uint32_t slot = 0, it = 0;
    for (uint32_t unit = cluster; unit < a.units; unit += n_clusters, ++it) {
        float acc[2][NT][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.0f;
#pragma unroll 1
        for (uint32_t c = c0 + warp; c < c1; c += kWarps) {
            // The oldest group has landed when at most depth - 1 are outstanding (depth is 2, 3, 4 or 6).
            if (depth == 6) asm volatile("cp.async.wait_group 5;" ::: "memory");
            else if (depth == 4) asm volatile("cp.async.wait_group 3;" ::: "memory");
            else if (depth == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
            else asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            const uint32_t src = ring + slot * kSlot;
            uint32_t w[4][4];
            __half2 d2[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[i][0]), "=r"(w[i][1]), "=r"(w[i][2]), "=r"(w[i][3]) : "r"(src + i * 512u + lane * 16u));
                unsigned short h;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h) : "r"(src + 2048u + (g + 8u * i) * 4u + (t4 >> 1) * 2u));
                d2[i] = __half2half2(__ushort_as_half(h));
            }
            __syncwarp();
            issue(slot);
            slot = slot + 1u == depth ? 0u : slot + 1u;
            const unsigned char *xp = xs + g * xstride + (c - c0) * 128u + t4 * 32u;
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // two 16-byte pieces of x, two MMAs of K = 16 each
                uint32_t af[2][2][4];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        dequant4(w[2 * m][2 * h + j], d2[2 * m], af[j][m][0], af[j][m][2]);
                        dequant4(w[2 * m + 1][2 * h + j], d2[2 * m + 1], af[j][m][1], af[j][m][3]);
                    }
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const uint32_t(&v)[8] = xb[STAGED ? 0 : n];
                    const uint4 b = STAGED ? *(const uint4 *)(xp + n * 8u * xstride + h * 16u)
                                           : make_uint4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        mma_f16(acc[m][n], af[0][m][0], af[0][m][1], af[0][m][2], af[0][m][3], b.x, b.y);
                        mma_f16(acc[m][n], af[1][m][0], af[1][m][1], af[1][m][2], af[1][m][3], b.z, b.w);
                    }
                    if (!STAGED && h == 1) load_x(n, c + kWarps);
                }
            }
        }
        // ---- the 8 warps' sums, then the CTAs' ----
        if (!STAGED) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float *r = red + (warp * kTok + n * 8u + 2u * t4) * kRowPad + m * 16u + g;
                r[0] = acc[m][n][0];
                r[kRowPad] = acc[m][n][1];
                r[8] = acc[m][n][2];
                r[kRowPad + 8] = acc[m][n][3];
            }
        __syncthreads();
        float *mine = part + (it & 1u) * kTok * 32u;
        float sum[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const uint32_t tok = warp + 8u * i;
            float v = 0.0f;
#pragma unroll
            for (int k = 0; k < kWarps; ++k) v += red[(k * kTok + tok) * kRowPad + lane];
            sum[i] = v;
            if (P > 1) mine[tok * 32u + lane] = v;
        }
        if (P > 1) cluster_sync();  // also: every warp has read `red`
        else __syncthreads();
        // Token tok of the unit is finished by CTA tok % P (all of them when P is 1).
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const uint32_t tok = P > 1 ? rank + P * (warp + 8u * i) : warp + 8u * i;
            if (tok >= a.batch) break;
            float v = sum[i];
            if (P > 1) {
                const uint32_t at = (uint32_t)__cvta_generic_to_shared(mine + tok * 32u + lane);
                float pv[8];
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) pv[k] = k < P ? ld_cluster(at, k) : 0.0f;
                v = pv[0];
#pragma unroll
                for (uint32_t k = 1; k < 8; ++k)
                    if (k < P) v += pv[k];
            }
            if (a.mode == kPlain) {
                const uint32_t row0 = unit * 32u, row = row0 + lane;
                const bool p0 = row0 < a.part_end[0], p1 = row0 < a.part_end[1];
                const uint32_t lo = p0 ? 0u : p1 ? a.part_end[0] : a.part_end[1];
                const uint32_t hi = p0 ? a.part_end[0] : p1 ? a.part_end[1] : a.part_end[2];
                if (row < a.rows) {
                    float *yp = (p0 ? a.y[0] : p1 ? a.y[1] : a.y[2]) + (size_t)tok * (hi - lo) + (row - lo);
                    *yp = a.accumulate ? *yp + v : v;
                }
            } else {
                const float up = __shfl_down_sync(0xffffffffu, v, 16);
                if (lane < 16u) {
                    const float r = (a.mode == kSilu ? tmdev::silu_f(v) : tmdev::gelu_tanh_f(v)) * up;
                    a.act[(size_t)tok * half_rows + unit * 16u + lane] = __float2half_rn(r);
                }
            }
        }
    }
    if (P > 1) cluster_sync();  // nobody leaves while its sums are being read
}

size_t rows_smem(uint32_t cols, uint32_t nt, uint32_t p, uint32_t ring, bool staged) {
    const uint32_t tok = nt * 8u, kc = (cols / 64u + p - 1u) / p;
    if (!staged) return ring_or_sums(tok, ring) + (p > 1 ? 2u * tok * 32u * 4u : 0u);
    return (size_t)tok * (kc * 128u + 16u) + (size_t)kWarps * tok * kRowPad * 4u + (p > 1 ? 2u * tok * 32u * 4u : 0u) +
           (size_t)kWarps * ring * kSlot;
}

// Clusters of p CTAs, one CTA to an SM, that find a place at once.  (Where more were launched than that, 12288 x 12288 at 8
// tokens took 75 us in three parts; 47 without staging.)
uint32_t cluster_places(uint32_t sms, uint32_t p) { return (p <= 2u ? sms : p <= 4u ? sms - sms / 8u : sms - sms / 4u) / p; }

struct rows_plan {
    uint32_t p = 0, ring = 0;
    bool staged = false;
};

// K parts.  Not staged: a CTA's time in hundredths of a microsecond, fitted to measurements at 8, 19 and 32 tokens and
// P = 1..8: per chunk of a warp 0.35 us of latency and, times the CTAs that share an SM, 0.35 + 0.1 per 8 tokens for the
// weights, the products and X from L2; 0.5 us for the CTAs' sums.  The parts of a unit have to be resident together, and
// clusters of three and more find a place each only well below two CTAs an SM (1152 x 6912 by 32 tokens: 6 parts, 216
// CTAs, 6.7 us; 8 parts, 288 CTAs, 10.4), so P stops there; units alone may take turns.  The ring is as deep as a warp's
// stream is long, at most 6.
// Staged: a CTA's time in cycles, its rounds of units, each the chunks one warp streams plus the ordered sum, and once
// its share of X; P is the part count with the least of that whose share of X leaves room for a ring.
rows_plan plan_rows(uint32_t sms, size_t smem_optin, uint32_t units, uint32_t cols, uint32_t nt) {
    const uint32_t chunks = cols / 64u;
    rows_plan best;
    uint32_t cost = 0;
    // Staged: units for more than two rounds of every SM, and either at most 8 chunks, one a warp, so that the CTAs that come
    // and go cost more than they stream, or (up to 8 tokens) a stream that is longer than X is wide; where the third round
    // is hardly begun, a still longer one.  us staged / not: 8 tokens by 10464 x 320 4.7 / 5.3, 12288 x 512 5.4 / 5.9, 24576 x
    // 512 9.0 / 8.4, 24576 x 1024 12.3 / 11.8, 32768 x 1024 14.0 / 14.7, 16384 x 1536 11.7 / 11.2, 24576 x 1536 15.1 / 15.4,
    // 12288 x 2048 12.0 / 11.8, 20480 x 2048 16.7 / 17.2, 12288 x 4096 18.5 / 18.9, 98304 x 3072 70 / 85, and with 297 to 364
    // units 9504 x 6144 24.3 / 23.8, 9504 x 8192 29.2 / 30.1, 10240 x 11264 37 / 45; 16 tokens by 20480 x 128 6.0 / 7.1, 20480 x
    // 512 8.1 / 8.9, 16384 x 640 9.4 / 8.2.  (24 tokens by 16384 x 128 5.9 / 6.4, x 512 9.3 / 7.8: no third form for that.)
    const bool long_stream = units * chunks >= (2u * units > 5u * sms ? 13000u : 35000u);
    if (nt <= 2u && units > 2u * sms && (chunks <= 8u || (nt == 1u && long_stream))) {
        best.staged = true;
        for (uint32_t p = 1; p <= 8u && p <= chunks; ++p) {
            const uint32_t kc = (chunks + p - 1u) / p, at_once = cluster_places(sms, p), rounds = (units + at_once - 1u) / at_once;
            const uint32_t per_warp = (kc + kWarps - 1u) / kWarps;
            const uint32_t c = rounds * (per_warp * (500u + 200u * nt) + 900u + 200u * nt + (p > 1u ? 300u : 0u)) + kc * 20u * nt;
            if (best.p && c >= cost) continue;
            uint32_t ring = 0;
            for (uint32_t r : {6u, 4u, 3u, 2u})
                if ((r <= rounds * per_warp || r == 2u) && rows_smem(cols, nt, p, r, true) <= smem_optin) {
                    ring = r;
                    break;
                }
            if (!ring) continue;
            best.p = p;
            best.ring = ring;
            cost = c;
        }
        if (best.p) return best;
        best = rows_plan();
    }
    for (uint32_t p = 1; p <= 8u && p <= chunks; ++p) {
        const uint32_t ctas = units * p, per_warp = ((chunks + p - 1u) / p + kWarps - 1u) / kWarps;
        if (p > 1u && ctas > (p == 2u ? 2u * sms : sms + sms / 2u)) break;
        const uint32_t c = (uint32_t)((uint64_t)per_warp * (35ull * sms + (35ull + 10ull * nt) * ctas) / sms) + (p > 1u ? 50u : 0u);
        if (best.p && c >= cost) continue;
        best.p = p;
        best.ring = per_warp >= 6u ? 6u : per_warp >= 4u ? 4u : per_warp == 3u ? 3u : 2u;
        cost = c;
    }
    return best;
}

bool rows_ok(uint32_t rows, uint32_t cols, uint32_t batch, bool gated) {
    return batch >= 1u && batch <= TM_CUDA_GEMM_ROWS_MAX_BATCH && rows > 0u && cols > 0u && cols % 64u == 0u &&
           cols <= 16384u && (!gated || rows % 32u == 0u);
}

template <int NT, bool STAGED>
cudaError_t launch_rows_as(tm_cuda_ctx *ctx, const rows_args &args, const rows_plan &pl) {
    rows_args a = args;
    a.ring = pl.ring;
    const size_t smem = rows_smem(a.cols, NT, pl.p, pl.ring, STAGED);
    static std::atomic<bool> attr_set[64] = {};  // per device; contexts of a process share it
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(q8_gemm_rows_kernel<NT, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)ctx->smem_optin);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    // Resident clusters: by shared memory (1 KB per CTA is the system's) and registers at most two CTAs per SM.
    const uint32_t per_sm = 2u * (smem + 1024u) <= 228u * 1024u ? 2u : 1u;
    uint32_t clusters = cluster_places((uint32_t)ctx->sm_count, pl.p) * per_sm;
    if (!STAGED || clusters > a.units) clusters = a.units;
    return tm_launch_cluster_pdl(ctx, pl.p, q8_gemm_rows_kernel<NT, STAGED>, dim3(clusters * pl.p), dim3(kThreads), smem, a);
}

template <int NT>
cudaError_t launch_rows(tm_cuda_ctx *ctx, const rows_args &a, const rows_plan &pl) {
    if constexpr (NT <= 2)
        if (pl.staged) return launch_rows_as<NT, true>(ctx, a, pl);
    return launch_rows_as<NT, false>(ctx, a, pl);
}

}  // namespace

extern "C" {

// Where the multiply for a few rows beats the tcgen05 GEMM, both with the f16 copy of X.  Up to 8 tokens: everywhere but in
// narrow matrices of many bytes (us, this form / tcgen05: 65536 x 1536 30 / 34, 98304 x 3072 70 / 87, 98304 x 4096 96 / 118,
// but 262144 x 1152 86 / 79).  From 9 tokens on the two cross wherever the one's units or the other's 128-row tiles have
// just begun another round of the SMs, so both times are estimated, in hundredths of a microsecond, fitted to 279 shapes of
// 64 to 16384 columns and 3 to 130 M weights at 9 to 32 tokens: one of nine takes the slower form, by 4 % (11 at most).
// At 16 tokens 20480 x 2048 19.4 / 23.7, 16384 x 4096 26.7 / 24.2, 131072 x 512 38 / 26; at 24 8192 x 3072 13.4 / 15.0,
// 6144 x 4096 15.5 / 16.4, 16384 x 2048 17.7 / 15.9; at 32 8704 x 2048 11.5 / 13.2, 4096 x 4096 12.5 / 13.3, 12288 x 2048
// 16.1 / 14.9.  (Lines at a number of weights, 64, 32 and 17 M, cost 5, 5 and 2 % in the mean and up to 97.)
static bool rows_are_faster(uint32_t rows, uint32_t cols, uint32_t batch) {
    constexpr uint32_t kSms = 148;  // of the part that the times were taken on
    if (batch <= 8u) return cols >= 1536u || (uint64_t)rows * cols <= 128u << 20;
    const uint32_t nt = (batch + 7u) / 8u, units = rows / 32u + (rows % 32u != 0u);
    const rows_plan pl = plan_rows(kSms, 0, units, cols, nt);  // (no shared memory: X not staged)
    // Rounds of two CTAs an SM, and the chunks that the warps of the fullest SM stream (some of it behind the launch).
    const int64_t ctas = (int64_t)units * pl.p, turns = (ctas + 2 * kSms - 1) / (2 * kSms), per_sm = (ctas + kSms - 1) / kSms;
    const int64_t cost = 191 + turns * 227 + per_sm * ((int64_t)cols * (35 + 14 * nt) / (512 * pl.p) - 36) + (pl.p > 1u ? 109 : 0);
    return cost < (int64_t)tm_mma_few_tokens_cost(kSms, rows, cols);
}
int tm_cuda_q8_0_gemm_rows_pays(uint32_t rows, uint32_t cols, uint32_t batch, int gated) {
    return rows_ok(rows, cols, batch, gated != 0) && rows_are_faster(rows, cols, batch);
}

int tm_cuda_gemm_rows_last_form(tm_cuda_ctx *ctx) {
    if (!ctx) return 0;
    std::lock_guard<std::mutex> lock(ctx->mu);
    return ctx->rows_last_form;
}

int tm_cuda_q8_0_gemm_rows(tm_cuda_ctx *ctx, tm_cuda_buffer *w, tm_cuda_buffer *x, uint32_t rows, uint32_t cols,
                           uint32_t batch, uint32_t n_parts, tm_cuda_buffer *const *y_parts, const uint32_t *part_rows,
                           int prologue, tm_cuda_buffer *pro, float eps, int epilogue, char *err, size_t err_cap) {
    if (prologue != TM_CUDA_PRO_F16) {
        const int rc = tm_mma_ensure_workspace(ctx, cols, batch, err, err_cap);
        if (rc != TM_CUDA_OK) return rc;
    }
    TM_ENTER();
    int rc = tm_check_packed(ctx, w, rows, cols, err, err_cap);
    if (rc != TM_CUDA_OK) return rc;
    const bool gated = epilogue == TM_CUDA_EPI_SILU_MUL_F16 || epilogue == TM_CUDA_EPI_GELU_MUL_F16;
    if (!rows_ok(rows, cols, batch, gated))
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "%u x %u for %u rows: 1..%d rows, whole 64-column chunks%s", rows,
                       cols, batch, TM_CUDA_GEMM_ROWS_MAX_BATCH, gated ? ", gate and up of whole 16-row tiles" : "");
    if (prologue < TM_CUDA_PRO_NONE || prologue > TM_CUDA_PRO_F16 ||
        (!gated && epilogue != TM_CUDA_EPI_STORE && epilogue != TM_CUDA_EPI_ADD))
        return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "unknown prologue %d / epilogue %d", prologue, epilogue);
    if (n_parts < 1 || n_parts > 3 || !y_parts || !part_rows || (gated && n_parts != 1))
        return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "1 to 3 output parts (1 for a gated output), got %u", n_parts);
    rows_args a = {};
    if (gated) {
        if (part_rows[0] != rows / 2u) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "a gated output has %u rows", rows / 2u);
        TM_CHECK_BUF(y_parts[0], (size_t)batch * (rows / 2u) * 2, "gated output");
        a.act = (__half *)y_parts[0]->dev;
        a.units = rows / 32u;
        a.mode = epilogue == TM_CUDA_EPI_SILU_MUL_F16 ? kSilu : kGelu;
    } else {
        uint32_t sum = 0;
        for (uint32_t p = 0; p < 3; ++p) a.part_end[p] = rows;
        for (uint32_t p = 0; p < n_parts; ++p) {
            if (part_rows[p] == 0 || (p + 1 < n_parts && part_rows[p] % 32u != 0))
                return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED,
                               "part %u has %u rows: every part but the last must be a multiple of 32", p, part_rows[p]);
            TM_CHECK_BUF(y_parts[p], (size_t)batch * part_rows[p] * 4, "output part");
            a.y[p] = (float *)y_parts[p]->dev;
            sum += part_rows[p];
            a.part_end[p] = sum;
        }
        if (sum != rows) return tm_fail(err, err_cap, TM_CUDA_ERR_BOUNDS, "parts cover %u of %u rows", sum, rows);
        a.units = (rows + 31u) / 32u;
        a.mode = kPlain;
    }
    a.q = (const signed char *)w->qp;
    a.d = (const unsigned short *)w->dp;
    a.rows = rows;
    a.cols = cols;
    a.batch = batch;
    a.accumulate = epilogue == TM_CUDA_EPI_ADD;
    const uint32_t nt = (batch + 7u) / 8u;
    const rows_plan pl = plan_rows((uint32_t)ctx->sm_count, ctx->smem_optin, a.units, cols, nt);
    if (!pl.p) return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "cols %u exceeds the activation stage of a cluster", cols);
    if (prologue == TM_CUDA_PRO_F16) {
        TM_CHECK_BUF(x, (size_t)batch * cols * 2, "activation");
        if (((size_t)x->dev & 15u) != 0) return tm_fail(err, err_cap, TM_CUDA_ERR_UNSUPPORTED, "f16 activations are not 16-byte aligned");
        a.x = (const __half *)x->dev;
    } else {
        TM_CHECK_BUF(x, (size_t)batch * cols * 4, "activation");
        if (prologue == TM_CUDA_PRO_RMSNORM) TM_CHECK_IN(pro, (size_t)cols * 4, "norm weight");
        else if (prologue != TM_CUDA_PRO_NONE) TM_CHECK_BUF(pro, (size_t)batch * cols * 4, "gate operand");
        a.x = (const __half *)ctx->mma_scratch;
    }
    a.x32 = ((size_t)a.x & 31u) == 0;
    ctx->rows_last_form = pl.staged ? -(int)pl.p : (int)pl.p;
    TM_OP_BEGIN("q8_0_gemm_rows");
    if (prologue != TM_CUDA_PRO_F16)
        TM_CUDA_TRY(tm_x_prep_launch(ctx, prologue, (const float *)x->dev, pro ? (const float *)pro->dev : nullptr, cols,
                                     batch, eps));
    TM_CUDA_TRY(nt == 1   ? launch_rows<1>(ctx, a, pl)
                : nt == 2 ? launch_rows<2>(ctx, a, pl)
                : nt == 3 ? launch_rows<3>(ctx, a, pl)
                          : launch_rows<4>(ctx, a, pl));
    TM_OP_END(prologue == TM_CUDA_PRO_F16 ? 1 : 2);
}

}  // extern "C"
