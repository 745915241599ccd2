// Prefill attention over the quantised caches (q8 rows, q8 blocks of 32, TurboQuant) on the tensor cores, in 32-bit
// precision.
//
// The cached operands are small whole numbers: int8 codes, the residual signs of the TurboQuant rows, and its four
// centroids, which are alpha * {-6128, -1837, 1837, 6128} to 2e-8 (the f32 constants themselves are only given to
// 3e-8). All of them are exact in f16. The other operand of each product (q, or the softmax weight times the value
// scale) is an f32 number x, scaled by a power of two into f16's range and split as x = hi + lo with two f16 of 11
// significant bits each: what is left out is at most 2^-23 |x|, one bit more than f32's rounding, or 2^-38 of the largest
// element that shares the power of two (lo of an element 2^-15 below that is subnormal). So
//   q . code = hi . code + lo . code     and     P V = P_hi V + P_lo V
// are two f16 MMAs with f32 accumulation; the scales are applied in f32, and the sums over the keys of one tile are
// added to the running output by f32 additions, so no accumulation in the tensor core is longer than 64 keys.
//
// A CTA owns 64 rows, each one (token, query head) pair of one KV head: row r of a KV head is token r / G, head r % G,
// so any group size packs densely and a tile spans 64 / G tokens of the causal diagonal. Tiles of 64 keys come in raw
// through a two-stage cp.async ring and are expanded to f16 once for all 64 rows.
//   q8:    four warps of 16 rows, two CTAs per SM (one expands while the other multiplies).
//   Turbo: eight warps; warps w and w + 4 share 16 rows, one takes the centroid part of scores and values and the other
//          the residual-sign part (score = sigma (Q_r C^T) + rho (Q_p S^T), src/engine/runtime/inference.rs:1246-1269):
//          the partial scores change hands through shared memory, and each keeps one of the two output accumulators.
// Where the row tiles do not fill the GPU, the keys are split over CTAs and the last one of a tile merges.
//
// The other places that are not f32 FMAs: the centroids' common factor (2e-8) and the sums of 16 products, which the tensor
// core rounds in its own way. Outputs against 64-bit attention over the same cache: q8 1000 rows, 3.2e-5 (the angles of RoPE),
// as the f32 CUDA-core kernel; the two kernels differ by 2.3e-7 there and by 5.6e-7 for 512 TurboQuant rows.
//
// Bound: latency of a chain per warp (expand, barrier, Q K^T, softmax, split, P V) at eight warps per SM, 255 registers each.
// Measured on a B200, per layer, against the f32 CUDA-core kernels (attn_simt_kernel, attn_turbo_kernel), rope and append
// included: 32/8 heads of 128, 1000 rows, q8: 1464 -> 106 us; 16/8 heads, 512 rows behind 700, TurboQuant: 1200 -> 130 us.
#pragma once

#include <cuda_fp16.h>

#include "attn_turbo.cuh"
#include "attn_turbo_mma.cuh"

namespace ggr {

constexpr int kPsRows = 64;  // (token, head) rows of a CTA
constexpr int kPsKeys = 64;  // keys of a tile
constexpr int kPsMaxSplits = 32;

// shared memory: two raw stages, the expanded tiles, and for TurboQuant the partial scores
template <int FMT, int D>
struct PsLayout {
    static constexpr bool turbo = FMT == KV_TURBO;
    static constexpr int threads = turbo ? 256 : 128, ctas_per_sm = turbo ? 1 : 2;
    static constexpr int nsc = FMT == KV_Q8_BLOCK32 ? D / 32 : 1;  // scales of a key and head (TurboQuant: sigma, and a norm)
    static constexpr int code_bytes = kPsKeys * (turbo ? D / 4 : D), sign_bytes = turbo ? kPsKeys * D / 8 : 0;
    static constexpr int scale_bytes = kPsKeys * nsc * 4 * (turbo ? 2 : 1);
    static constexpr int raw = 2 * (code_bytes + sign_bytes + scale_bytes);  // K and V
    static constexpr int tile = kPsKeys * D * 2;
    static constexpr int n_tiles = turbo ? 4 : 2;
    static constexpr int tiles_at = 2 * raw;
    static constexpr int xchg_at = tiles_at + n_tiles * tile;
    static constexpr int bytes = xchg_at + (turbo ? 8 * 16 * kPsKeys * 4 : 0);
};

__device__ __forceinline__ void mma_f16_16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// (x, y) -> f16 pairs hi and lo with hi + lo = (x, y) to 2^-23, for x and y in f16's normal range
__device__ __forceinline__ void split_f16x2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(__fsub_rn(x, f.x), __fsub_rn(y, f.y));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ float exp2i(int e) { return __int_as_float((e + 127) << 23); }  // -126 <= e <= 127

// exponent of the power of two that brings `top` into [2^13, 2^14)
__device__ __forceinline__ int f16_exponent(float top) {
    return max(-126, min(126, 13 - ((int)((__float_as_uint(top) >> 23) & 0xffu) - 127)));
}

// four int8 -> four f16: |0x64|byte + 128| is 1024 + 128 + code as an f16
__device__ __forceinline__ uint2 codes_to_f16(uint32_t w) {
    w ^= 0x80808080u;
    const __half2 bias = __half2half2(__ushort_as_half(0x6480));
    const uint32_t a = prmt(w, 0x64646464u, 0x4140u), b = prmt(w, 0x64646464u, 0x4342u);
    const __half2 ha = __hsub2(*reinterpret_cast<const __half2*>(&a), bias), hb = __hsub2(*reinterpret_cast<const __half2*>(&b), bias);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&ha), *reinterpret_cast<const uint32_t*>(&hb));
}

// Eight 2-bit codes -> eight f16 of {-6128, -1837, 1837, 6128} (0xEDFC 0xE72D 0x672D 0x6DFC), as turbo_centroids8
__device__ __forceinline__ uint4 turbo_levels8(uint32_t x) {
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    const uint32_t hi_tab = 0x6D67E7EDu, lo_tab = 0xFC2D2DFCu;
    const uint32_t s0 = x & 0xFFFFu, s1 = x >> 16;
    const uint32_t hi0 = prmt(hi_tab, lo_tab, s0), lo0 = prmt(hi_tab, lo_tab, s0 | 0x4444u);
    const uint32_t hi1 = prmt(hi_tab, lo_tab, s1), lo1 = prmt(hi_tab, lo_tab, s1 | 0x4444u);
    return make_uint4(prmt(lo0, hi0, 0x5140u), prmt(lo0, hi0, 0x7362u), prmt(lo1, hi1, 0x5140u), prmt(lo1, hi1, 0x7362u));
}
// alpha: the mean of the two ratios centroid / whole number, which differ by 4e-8
constexpr float kTurboAlpha = (float)(0.5 * ((double)0.45278f / 1837.0 + (double)1.510417f / 6128.0));

// Eight sign bits (1 = positive) -> eight f16 +1 / -1
__device__ __forceinline__ uint4 turbo_signs8_f16(uint32_t x) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = 0xBC00BC00u ^ (((x >> (2 * i)) & 1u) << 15) ^ (((x >> (2 * i + 1)) & 1u) << 31);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

inline bool prefill_split_supported(int fmt, int D) {
    return ((fmt == KV_Q8_ROW || fmt == KV_Q8_BLOCK32) && (D == 64 || D == 128)) || (fmt == KV_TURBO && D == 128);
}

template <int FMT, int D>
__global__ void __launch_bounds__(PsLayout<FMT, D>::threads, PsLayout<FMT, D>::ctas_per_sm)
    prefill_split_kernel(AttnArgs a) {
    using L = PsLayout<FMT, D>;
    constexpr bool turbo = FMT == KV_TURBO;
    constexpr int NTHR = L::threads, NWARP = NTHR / 32, KS = D / 16, NT = D / 8, TK = kPsKeys, NS = TK / 8;
    extern __shared__ __align__(128) unsigned char psm[];
    __shared__ int s_lo, s_hi, s_lo_in, s_hi_in, s_last;
    __shared__ float s_m[kPsRows], s_l[kPsRows];

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int gq = lane >> 2, tq = lane & 3;
    const int part = turbo ? warp >> 2 : 0, rw = warp & 3;
    const int G = a.kv.G, Hq = a.kv.Hq, Hkv = a.kv.Hkv, kv_dim = a.kv.kv_dim;
    const int kvh = blockIdx.x, row_tile = gridDim.y - 1 - blockIdx.y, split = blockIdx.z;  // longest rows first
    const int n_rows = a.items.n * G, r_first = row_tile * kPsRows;
    const int seq = a.items.seq0;
    const int64_t row0 = a.kv.row(seq, a.layer, a.kv.pos_begin);
    grid_wait();
    grid_allow_dependents();

    if (tid == 0) {
        s_lo = INT_MAX;
        s_hi = 0;
        s_lo_in = 0;
        s_hi_in = INT_MAX;
    }
    __syncthreads();
    if (tid < kPsRows && r_first + tid < n_rows) {
        int vs, ve;
        a.vis.range(a.items.base_pos + (r_first + tid) / G, vs, ve);
        atomicMin(&s_lo, vs);
        atomicMax(&s_hi, ve);
        atomicMax(&s_lo_in, vs);
        atomicMin(&s_hi_in, ve);
    }
    // this thread's two rows of the MMA tile
    int vis_s[2], vis_e[2];
    int64_t qrow[2];
    bool used[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = r_first + rw * 16 + gq + 8 * i;
        used[i] = r < n_rows;
        vis_s[i] = vis_e[i] = 0;
        const int item = used[i] ? r / G : 0, g = used[i] ? r - item * G : 0;
        if (used[i]) a.vis.range(a.items.base_pos + item, vis_s[i], vis_e[i]);
        qrow[i] = ((int64_t)item * Hq + (int64_t)kvh * G + g) * D;
    }
    __syncthreads();
    const int all_lo = s_lo & ~(TK - 1), all_hi = s_hi;
    const int chunk = ((all_hi - all_lo + a.n_split - 1) / a.n_split + TK - 1) / TK * TK;
    const int k_lo = all_lo + split * chunk, k_hi = min(all_hi, k_lo + chunk);
    const int n_kt = k_hi > k_lo ? (k_hi - k_lo + TK - 1) / TK : 0;
    const int in_lo = s_lo_in, in_hi = s_hi_in;

    // raw K and V of key tile `it` into its stage: codes, sign bits, scales; keys past the range come in as zeros
    auto issue = [&](int it) {
        if (it < n_kt) {
            unsigned char* st = psm + (it & 1) * L::raw;
            constexpr int gpk = L::code_bytes / TK / 16;  // 16-byte pieces of a key's codes
            for (int i = tid; i < 2 * TK * gpk; i += NTHR) {
                const int kv = i / (TK * gpk), rem = i - kv * (TK * gpk), key = rem / gpk, c = rem - key * gpk;
                const int t = k_lo + it * TK + key, valid = t < k_hi;
                const int64_t e = ((row0 + (valid ? t : k_lo)) * kv_dim + (int64_t)kvh * D) / (turbo ? 4 : 1);
                cp_async_16(smem_u32(st + kv * L::code_bytes + key * (gpk * 16) + c * 16),
                            reinterpret_cast<const unsigned char*>(kv ? a.kv.v : a.kv.k) + e + c * 16, valid ? 16 : 0);
            }
            unsigned char* sg = st + 2 * L::code_bytes;
            if (turbo) {
                for (int i = tid; i < 2 * TK; i += NTHR) {
                    const int kv = i / TK, key = i - kv * TK, t = k_lo + it * TK + key, valid = t < k_hi;
                    const int64_t e = ((row0 + (valid ? t : k_lo)) * kv_dim + (int64_t)kvh * D) / 8;
                    cp_async_16(smem_u32(sg + kv * L::sign_bytes + key * 16), (kv ? a.kv.v_sign : a.kv.k_sign) + e, valid ? 16 : 0);
                }
            }
            // scales: K [key][nsc], V [key][nsc]; TurboQuant: sigma_k, gamma_k, sigma_v, gamma_v [key]
            float* sc = reinterpret_cast<float*>(sg + 2 * L::sign_bytes);
            for (int i = tid; i < L::scale_bytes / 2; i += NTHR) {
                const int sect = i / (TK * L::nsc), rem = i - sect * (TK * L::nsc), key = rem / L::nsc, b = rem - key * L::nsc;
                const int t = k_lo + it * TK + key, valid = t < k_hi;
                const float* src = turbo ? (sect == 0 ? a.kv.ks : sect == 1 ? a.kv.k_rn : sect == 2 ? a.kv.vs : a.kv.v_rn)
                                         : (sect ? a.kv.vs : a.kv.ks);
                const int64_t at = (row0 + (valid ? t : k_lo)) * a.kv.n_scales + (FMT == KV_Q8_ROW ? 0 : (int64_t)kvh * L::nsc + b);
                cp_async_4(smem_u32(sc + i), src + at, valid ? 4 : 0);
            }
        }
        cp_async_commit();
    };
    issue(0);

    // A fragments of the queries, hi and lo; rf[i] takes a row's sums back to log2-unit scores
    uint32_t qh[KS][4], ql[KS][4];
    float rf[2];
    {
        const float* src = a.q;
        int64_t at[2] = {qrow[0], qrow[1]};
        float* prep = reinterpret_cast<float*>(psm + L::tiles_at);  // [2][64][D]: q_r, q_p (:954-968)
        if (turbo) {
            const unsigned char* sl[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) sl[s] = turbo_sign_slot(a.kv, s, a.layer, kvh);
            for (int r = warp; r < kPsRows; r += NWARP) {
                const int rr = r_first + r, item = rr / G, g = rr - item * G;
                float x[4] = {0.f, 0.f, 0.f, 0.f};
                if (rr < n_rows) {
                    const float4 v = *reinterpret_cast<const float4*>(a.q + ((int64_t)item * Hq + (int64_t)kvh * G + g) * D + lane * 4);
                    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
                }
                turbo_transform_regs(x, sl[0], sl[1], lane);
                *reinterpret_cast<float4*>(prep + r * D + lane * 4) = make_float4(x[0], x[1], x[2], x[3]);
                turbo_transform_regs(x, sl[2], sl[3], lane);
                *reinterpret_cast<float4*>(prep + (kPsRows + r) * D + lane * 4) = make_float4(x[0], x[1], x[2], x[3]);
            }
            __syncthreads();
            src = prep + part * kPsRows * D;
            at[0] = (int64_t)(rw * 16 + gq) * D;
            at[1] = at[0] + 8 * D;
        }
        float x[2][KS][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float top = 0.f;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                float2 u = make_float2(0.f, 0.f), v = u;
                if (used[i]) {
                    u = *reinterpret_cast<const float2*>(src + at[i] + ks * 16 + tq * 2);
                    v = *reinterpret_cast<const float2*>(src + at[i] + ks * 16 + tq * 2 + 8);
                }
                x[i][ks][0] = u.x, x[i][ks][1] = u.y, x[i][ks][2] = v.x, x[i][ks][3] = v.y;
                top = fmaxf(fmaxf(top, fmaxf(fabsf(u.x), fabsf(u.y))), fmaxf(fabsf(v.x), fabsf(v.y)));
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const int e = f16_exponent(top);
            const float up = exp2i(e);
            rf[i] = a.score_scale * exp2i(-e);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                split_f16x2(x[i][ks][0] * up, x[i][ks][1] * up, qh[ks][i], ql[ks][i]);
                split_f16x2(x[i][ks][2] * up, x[i][ks][3] * up, qh[ks][2 + i], ql[ks][2 + i]);
            }
        }
    }

    float o[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    float wtop[2] = {0.f, 0.f};  // largest weight in the row's accumulator, and the exponent it is scaled by
    int we[2] = {0, 0};
    const float rho_unit = __fsqrt_rn(__fdiv_rn(1.57079632679489661923f, (float)D));  // :975-982
    const uint32_t t_k = smem_u32(psm + L::tiles_at) + part * L::tile, t_v = t_k + (turbo ? 2 : 1) * L::tile;

    for (int it = 0; it < n_kt; ++it) {
        const unsigned char* st = psm + (it & 1) * L::raw;
        const float* sc = reinterpret_cast<const float*>(st + 2 * L::code_bytes + 2 * L::sign_bytes);
        cp_async_wait<0>();
        __syncthreads();  // the raw tile is complete, and every warp is done with the expanded one before it
        issue(it + 1);
        // expand: rows of D f16, 16-byte chunk c of row r at c ^ (r & 7)
        if (turbo) {
            const int key = tid & 63, half = (tid >> 6) & 1, kv = tid >> 7;  // 64 codes and 64 signs each
            const uint4 cw = *reinterpret_cast<const uint4*>(st + kv * L::code_bytes + key * 32 + half * 16);
            const uint2 sw = *reinterpret_cast<const uint2*>(st + 2 * L::code_bytes + kv * L::sign_bytes + key * 16 + half * 8);
            const uint32_t cws[4] = {cw.x, cw.y, cw.z, cw.w}, sws[2] = {sw.x, sw.y};
            unsigned char* dst = psm + L::tiles_at + kv * 2 * L::tile + key * (D * 2);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int off = ((half * 8 + j) ^ (key & 7)) << 4;
                *reinterpret_cast<uint4*>(dst + off) = turbo_levels8((cws[j >> 1] >> ((j & 1) * 16)) & 0xffffu);
                *reinterpret_cast<uint4*>(dst + L::tile + off) = turbo_signs8_f16((sws[j >> 2] >> ((j & 3) * 8)) & 0xffu);
            }
        } else {
            constexpr int cpk = D / 8;  // 16-byte chunks of an expanded row
#pragma unroll 8
            for (int i = tid; i < 2 * TK * cpk; i += NTHR) {
                const int row = i / cpk, c = i - row * cpk;  // rows 0 .. 63 of K, then of V
                const uint2 w = *reinterpret_cast<const uint2*>(st + row * D + c * 8);
                const uint2 lo = codes_to_f16(w.x), hi = codes_to_f16(w.y);
                *reinterpret_cast<uint4*>(psm + L::tiles_at + row * (D * 2) + ((c ^ (row & 7)) << 4)) = make_uint4(lo.x, lo.y, hi.x, hi.y);
            }
        }
        __syncthreads();

        // scores of 16 rows x 64 keys, in log2 units
        float s[NS][4];
        const int key0 = k_lo + it * TK;
#pragma unroll
        for (int np = 0; np < NS / 2; ++np) {
            constexpr int nblk = L::nsc, kpb = KS / nblk;  // k-steps that share a scale
            float acc[2][4] = {};
#pragma unroll
            for (int b = 0; b < nblk; ++b) {
                float th[2][4] = {}, tl[2][4] = {};
#pragma unroll
                for (int kk = 0; kk < kpb; ++kk) {
                    const int ks = b * kpb + kk;
                    const int row = np * 16 + (lane & 7) + ((lane >> 4) & 1) * 8, c = 2 * ks + ((lane >> 3) & 1);
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4(t_k + row * (D * 2) + ((c ^ (row & 7)) << 4), b0, b1, b2, b3);
                    mma_f16_16816(tl[0], ql[ks], b0, b1);
                    mma_f16_16816(tl[1], ql[ks], b2, b3);
                    mma_f16_16816(th[0], qh[ks], b0, b1);
                    mma_f16_16816(th[1], qh[ks], b2, b3);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int key = (2 * np + j) * 8 + tq * 2 + i;
                        const float ksc = turbo ? (part ? sc[TK + key] * rho_unit : sc[key] * kTurboAlpha) : sc[key * nblk + b];
                        acc[j][i] = fmaf(th[j][i] + tl[j][i], ksc, acc[j][i]);
                        acc[j][2 + i] = fmaf(th[j][2 + i] + tl[j][2 + i], ksc, acc[j][2 + i]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[2 * np + j][i] = acc[j][i] * rf[i >> 1];
        }
        if (turbo) {
            // the partner warp holds the other half of each score at the same lane
            float* mine = reinterpret_cast<float*>(psm + L::xchg_at) + warp * (16 * TK);
            const float* other = reinterpret_cast<const float*>(psm + L::xchg_at) + (warp ^ 4) * (16 * TK);
#pragma unroll
            for (int n = 0; n < NS; ++n) *reinterpret_cast<float4*>(mine + (n * 32 + lane) * 4) = make_float4(s[n][0], s[n][1], s[n][2], s[n][3]);
            asm volatile("bar.sync %0, 64;" ::"r"(1 + rw) : "memory");
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                const float4 x = *reinterpret_cast<const float4*>(other + (n * 32 + lane) * 4);
                s[n][0] += x.x, s[n][1] += x.y, s[n][2] += x.z, s[n][3] += x.w;
            }
        }
        // a tile that every row of the CTA sees whole needs no mask
        const bool masked = key0 < in_lo || key0 + TK > in_hi || key0 + TK > k_hi;
        if (masked) {
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int key = key0 + n * 8 + tq * 2 + (i & 1);
                    if (key < vis_s[i >> 1] || key >= min(vis_e[i >> 1], k_hi)) s[n][i] = -INFINITY;
                }
        }
        // online softmax; s becomes the softmax weight p
        float factor[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float mx = m[r];
#pragma unroll
            for (int n = 0; n < NS; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * r], s[n][2 * r + 1]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float ref = mx == -INFINITY ? 0.f : mx;
            factor[r] = exp2f(m[r] - ref);
            m[r] = mx;
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < NS; ++n) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float p = exp2f(s[n][2 * r + i] - ref);
                    s[n][2 * r + i] = p;
                    sum += p;
                }
            }
            l[r] = fmaf(l[r], factor[r], sum);
        }
        // Weights w = p * value scale, scaled by a power of two per row so that the largest one seen sits at the top
        // of f16's range: a weight 2^-39 of the largest still contributes (p alone or the scale alone may be far
        // from it). TurboQuant: sigma * alpha or rho; q8 blocks: one set of weights per block of 32 columns.
        const float* vsc = sc + (turbo ? (2 + part) * TK : TK * L::nsc);
        const float vunit = turbo ? (part ? rho_unit : kTurboAlpha) : 1.0f;
        auto weight = [&](int n, int i, int b) {
            const float w = s[n][i] * (turbo ? vsc[n * 8 + tq * 2 + (i & 1)] * vunit : vsc[(n * 8 + tq * 2 + (i & 1)) * L::nsc + b]);
            return masked && s[n][i] == 0.f ? 0.f : w;  // the scale of a key that is not visible may be anything
        };
        if constexpr (L::nsc == 1) {
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[n][i] = weight(n, i, 0);
        }
        auto scaled = [&](int n, int i, int b) { return L::nsc == 1 ? s[n][i] : weight(n, i, b); };
        float up[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float top = 0.f;
#pragma unroll
            for (int b = 0; b < L::nsc; ++b)
#pragma unroll
                for (int n = 0; n < NS; ++n) top = fmaxf(top, fmaxf(fabsf(scaled(n, 2 * r, b)), fabsf(scaled(n, 2 * r + 1, b))));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            wtop[r] = fmaxf(wtop[r] * factor[r], top);
            const int e = wtop[r] > 0.f ? f16_exponent(wtop[r]) : we[r];
            factor[r] *= exp2i(max(-126, min(126, e - we[r])));
            we[r] = e;
            up[r] = exp2i(e);
        }
        constexpr int npb = NT / 2 / L::nsc;  // pairs of 8-column tiles that share their weights
#pragma unroll
        for (int b = 0; b < L::nsc; ++b) {
            uint32_t ph[TK / 16][4], pl[TK / 16][4];
#pragma unroll
            for (int ks = 0; ks < TK / 16; ++ks)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        split_f16x2(scaled(2 * ks + h, 2 * r, b) * up[r], scaled(2 * ks + h, 2 * r + 1, b) * up[r], ph[ks][2 * h + r],
                                    pl[ks][2 * h + r]);
#pragma unroll
            for (int q = 0; q < npb; ++q) {
                const int np = b * npb + q;
                float th[2][4] = {}, tl[2][4] = {};
#pragma unroll
                for (int ks = 0; ks < TK / 16; ++ks) {
                    const int row = ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, c = 2 * np + ((lane >> 4) & 1);
                    uint32_t b0, b1, b2, b3;
                    ldmatrix_x4_trans(t_v + row * (D * 2) + ((c ^ (row & 7)) << 4), b0, b1, b2, b3);
                    mma_f16_16816(tl[0], pl[ks], b0, b1);
                    mma_f16_16816(tl[1], pl[ks], b2, b3);
                    mma_f16_16816(th[0], ph[ks], b0, b1);
                    mma_f16_16816(th[1], ph[ks], b2, b3);
                }
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[2 * np + j][i] = fmaf(o[2 * np + j][i], factor[i >> 1], th[j][i] + tl[j][i]);
            }
        }
    }
    cp_async_wait<0>();

#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        const float down = exp2i(-we[r]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            o[nt][2 * r] *= down;
            o[nt][2 * r + 1] *= down;
        }
        if (tq == 0 && part == 0) {
            s_m[rw * 16 + gq + 8 * r] = m[r];
            s_l[rw * 16 + gq + 8 * r] = l[r];
        }
    }
    // the rows go out through shared memory: whole rows per warp (and the inverse transforms of TurboQuant need them)
    constexpr int LD = (turbo ? 2 * D : D) + 4;
    static_assert(kPsRows * LD * 4 <= L::bytes, "output staging");
    float* stage = reinterpret_cast<float*>(psm);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
            *reinterpret_cast<float2*>(stage + (rw * 16 + gq + 8 * r) * LD + part * D + nt * 8 + tq * 2) =
                make_float2(o[nt][2 * r], o[nt][2 * r + 1]);
    __syncthreads();
    constexpr int EPL = D / 32;
    for (int r = warp; r < kPsRows && r_first + r < n_rows; r += NWARP) {
        const int rr = r_first + r, item = rr / G, h = kvh * G + rr - item * G;
        float x[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) x[e] = stage[r * LD + lane * EPL + e];
        if constexpr (turbo) {
            // res <- T(res; res_post, res_pre); base += res; out = T(base; rot_post, rot_pre) (:1323-1334)
            float y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = stage[r * LD + D + lane * 4 + e];
            turbo_transform_regs(y, turbo_sign_slot(a.kv, 3, a.layer, kvh), turbo_sign_slot(a.kv, 2, a.layer, kvh), lane);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] += y[e];
            turbo_transform_regs(x, turbo_sign_slot(a.kv, 1, a.layer, kvh), turbo_sign_slot(a.kv, 0, a.layer, kvh), lane);
        }
        if (a.n_split == 1) {
#pragma unroll
            for (int e = 0; e < EPL; ++e) store_final(a, item, h, lane * EPL + e, x[e], s_m[r], s_l[r]);
        } else {
            float* pp = a.part + (((int64_t)item * Hq + h) * a.n_split + split) * (D + 2);
#pragma unroll
            for (int e = 0; e < EPL; e += 2) *reinterpret_cast<float2*>(pp + lane * EPL + e) = make_float2(x[e], x[e + 1]);
            if (lane == 0) *reinterpret_cast<float2*>(pp + D) = make_float2(s_m[r], s_l[r]);
        }
    }
    if (a.n_split == 1) return;
    // the last CTA of the row tile merges (see split_merge_store for the fences)
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(&a.counters[row_tile * Hkv + kvh], 1u) == (unsigned)a.n_split - 1u;
        if (s_last) __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) a.counters[row_tile * Hkv + kvh] = 0u;
    for (int r = warp; r < kPsRows && r_first + r < n_rows; r += NWARP) {
        const int rr = r_first + r, item = rr / G, h = kvh * G + rr - item * G;
        const float* pp = a.part + ((int64_t)item * Hq + h) * a.n_split * (D + 2);
        float2 ml = make_float2(-INFINITY, 0.f);
        if (lane < a.n_split) ml = __ldcg(reinterpret_cast<const float2*>(pp + (int64_t)lane * (D + 2) + D));
        const float ms = warp_max(ml.x);
        const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - ms);
        const float ls = warp_sum(f * ml.y);
        float x[EPL] = {};
        for (int sp = 0; sp < a.n_split; ++sp) {
            const float fs = __shfl_sync(0xffffffffu, f, sp);
#pragma unroll
            for (int e = 0; e < EPL; e += 2) {
                const float2 v = __ldcg(reinterpret_cast<const float2*>(pp + (int64_t)sp * (D + 2) + lane * EPL + e));
                x[e] = fmaf(fs, v.x, x[e]);
                x[e + 1] = fmaf(fs, v.y, x[e + 1]);
            }
        }
#pragma unroll
        for (int e = 0; e < EPL; ++e) store_final(a, item, h, lane * EPL + e, x[e], ms, ls);
    }
}

template <int FMT, int D>
inline cudaError_t launch_prefill_split_inst(const AttnArgs& a, dim3 grid, int smem_optin, int device, cudaStream_t stream) {
    static KernelSmemSetup setup;
    const cudaError_t e = setup.ensure(prefill_split_kernel<FMT, D>, device, smem_optin, PsLayout<FMT, D>::bytes);
    if (e != cudaSuccess) return e;
    return launch_chained(a.chained, prefill_split_kernel<FMT, D>, grid, PsLayout<FMT, D>::threads, PsLayout<FMT, D>::bytes, stream, a);
}

inline cudaError_t launch_prefill_split(const AttnArgs& a, dim3 grid, int smem_optin, int device, cudaStream_t stream) {
    switch (a.kv.fmt) {
        case KV_Q8_ROW:
            return a.kv.D == 64 ? launch_prefill_split_inst<KV_Q8_ROW, 64>(a, grid, smem_optin, device, stream)
                                : launch_prefill_split_inst<KV_Q8_ROW, 128>(a, grid, smem_optin, device, stream);
        case KV_Q8_BLOCK32:
            return a.kv.D == 64 ? launch_prefill_split_inst<KV_Q8_BLOCK32, 64>(a, grid, smem_optin, device, stream)
                                : launch_prefill_split_inst<KV_Q8_BLOCK32, 128>(a, grid, smem_optin, device, stream);
        case KV_TURBO: return launch_prefill_split_inst<KV_TURBO, 128>(a, grid, smem_optin, device, stream);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace ggr
