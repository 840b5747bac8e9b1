// The true 32-bit matrix product on the tensor cores:  Y[M,N] = X[M,K] * W[N,K]^T, float32 in and out.
//
// A float32 is the sum of three bfloat16: x = x1 + x2 + x3 with x1 the upper 16 bits, x2 the next 8 significant bits (rounded)
// and x3 what is left (8 bits, exact).  The product needs six of the nine products of such parts: x1w1, x1w2, x2w1, x1w3, x2w2, x3w1;
// the other three are below 2^-23 of it and of changing sign.  tcgen05.mma forms each product of parts exactly and adds in 32 bits,
// but without rounding to nearest, so a tile's sum must not stay in the tensor cores for long: every 32 k start a new accumulator
// (the small products first, the large ones last), and the epilogue warps add those into registers with ordinary additions.
// Error against 64 bits (norm of the error over norm of the result, normal numbers), here and on the CUDA cores: K = 896 1.2e-7 and
// 5.4e-7, K = 4,864 2.3e-7 and 1.25e-6; with K in splits 8e-8 to 1.0e-7 and 1.5e-7 to 3.1e-7.
// (K = 8 5.54e-8 and 5.35e-8: the caller leaves sums of fewer than 20 numbers to the CUDA cores.)  A part ends at 2^-133, the smallest
// bfloat16, so numbers below 2^-110 lose their last bits here.
//
// Measured (us, the CUDA-core kernel's in brackets): 1,999 tokens x 9,728 x 896 194 [802], x 896 x 4,864 106 [871], 4,096^3 704
// [2,966]; 64 tokens x 9,728 x 896 18.5 [54.5], x 896 x 4,864 10.2 [25.9], x 151,936 x 896 145 [459]; 1 token x 9,728 x 896 13.6 [62],
// x 151,936 x 896 95 [380], x 64 x 64 3.2 [4.5].  A prompt's product is held by the traffic of shared memory (136 KB per 32 k: raw
// tiles in and out, token parts in, MMA operands out; without the splits 133 us), one of few tokens by the weights' conversion.
//
//   * 128 weight rows are the accumulator's lanes, BN = 16 .. 128 tokens its columns, for prompts and decode steps alike.
//   * TMA brings float32 tiles of 32 k (128-byte rows).  Converter warps split them: weights go to tensor memory as the MMA's A
//     operand (a thread holds a row, so the layout needs no exchange, and the MMAs read nothing but the tokens from shared memory:
//     with both operands there, 128 x 128 products alone would take all of its bandwidth), tokens to shared memory (64-byte rows,
//     64-byte swizzle).  Nothing is converted in memory: the weights stay as they are, and a decode step reads 4 bytes of each.
//   * The bound is the 12 MMAs of 128 x BN x 16 per 32 k (768 cycles at BN = 128) beside 5.5 instructions for each of 32 * (128 + BN)
//     numbers that are split; for few tokens it is the weight stream.
//   * CTAs are persistent: every role walks the same list of tiles, so the loads and splits of the next tile run while this one's
//     sums are finished and written.
//
// A sum that is not a finite number (an infinity meets a part that is zero or not a number, or a stage's sum overflows) is formed again
// with FMAs by the warp that holds it, 128 numbers of the two rows at a time; a token with a NaN among its numbers needs only the
// look at them.  (One thread a sum, over the whole of K: 1,999 tokens x 896 x 4,864 with an infinity or a NaN in every token 42 ms, now
// 3.6 and 0.7; with none 0.10, on the CUDA cores 0.63.)
#pragma once
#include "f32_parts.cuh"

enum { FS_STORE = 0, FS_ADD = 2, FS_PARTIAL = 3, FS_SWIGLU = 4 };

struct FsParams {
    const float* X;          // for results that have to be formed again
    const float* W;
    void* out;
    const void* bias;
    int bias_is_f32;
    int M, N, K, ldx, ldo, mode;
    int tiles_m, tiles_n, splits, kb_split;        // kb_split: stages of 32 k per split
    int* status;
};

template <int BN> struct FsLayout {
    // One CTA per SM.  (Two with four converter warps each, at 64 tokens: 9,728 x 896 29 instead of 18.5 us, 896 x 4,864 in 8
    // splits 21 instead of 13.4 us: each CTA's stages follow one another with nothing beside them.)
    static constexpr int epi_warps = BN >= 64 ? 8 : 4;
    static constexpr int conv_warps = 8;
    static constexpr int threads = (epi_warps + conv_warps + 2) * 32;
    static constexpr int ctas = 1;
    static constexpr uint32_t w_bytes = 128 * 128, x_bytes = BN * 128;
    static constexpr uint32_t stage_bytes = w_bytes + x_bytes;
    static constexpr uint32_t plane_bytes = BN * 64;               // bf16 [BN][32]
    static constexpr int stages = BN == 128 ? 4 : 6;
    static constexpr uint32_t tmem_cols = BN >= 64 ? 512 : 256;          // 2 BN + 48 bufs
    static constexpr int bufs = BN >= 64 ? 4 : 2;                  // split stages on their way to the MMAs (1,999 x 9,728 x 896 with 2: 194 us, with 4: 186)
    static constexpr int n_bars = 2 * stages + 2 * bufs + 4;
    static constexpr size_t smem = (size_t)stages * stage_bytes + bufs * 3 * plane_bytes + n_bars * 8 + 16 + 1024;
};

// K-major tile of 64-byte rows with the 64-byte swizzle: 8-row groups are 512 bytes apart.
__device__ __forceinline__ uint64_t fs_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}
// A token's results of this warp's 32 weight rows from the numbers in memory, where `mine` asks for them (whole warps).
__device__ __forceinline__ void fs_again_token(const FsParams& p, bool mine, int m, int n, int k0, int k1, int split, float bias) {
    const int lane = threadIdx.x & 31, n0 = n - lane;
    const float* x = p.X + (size_t)m * p.ldx;
    bool nan = false;
#pragma unroll 1
    for (int k = k0 + 4 * lane; k < k1; k += 128) {
        const float4 v = *reinterpret_cast<const float4*>(x + k);
        nan = nan || isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w);
    }
    float d = __int_as_float(0x7fffffff);
    const uint32_t asked = __ballot_sync(0xffffffffu, mine);
    if (!__any_sync(0xffffffffu, nan))
#pragma unroll 1
        for (int g = 0; g < 32; g += 8) {                 // eight weight rows at a time
            if (!(asked >> g & 0xffu)) continue;
            float v[8] = {};
#pragma unroll 1
            for (int k = k0 + 4 * lane; k < k1; k += 128) {
                const float4 a = *reinterpret_cast<const float4*>(x + k);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 b = *reinterpret_cast<const float4*>(p.W + (size_t)min(n0 + g + q, p.N - 1) * p.K + k);
                    v[q] = fmaf(a.x, b.x, v[q]); v[q] = fmaf(a.y, b.y, v[q]); v[q] = fmaf(a.z, b.z, v[q]); v[q] = fmaf(a.w, b.w, v[q]);
                }
            }
            // the lanes share out the eight sums: row 4 i + 2 j + k ends in the lanes with bits 16 i, 8 j and 4 k
            int off = 16;
#pragma unroll
            for (int h = 4; h >= 1; h >>= 1, off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int q = 0; q < h; ++q) {
                    const float got = __shfl_xor_sync(0xffffffffu, up ? v[q] : v[q + h], off);
                    v[q] = (up ? v[q + h] : v[q]) + got;
                }
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            const float sum = __shfl_sync(0xffffffffu, v[0], (lane & 7) << 2);
            if ((lane & ~7) == g) d = sum;
        }
    float* o = reinterpret_cast<float*>(p.out) + (size_t)m * p.ldo;
    if (p.mode == FS_SWIGLU) {                            // (both of a pair's lanes ask)
        const float u = __shfl_xor_sync(0xffffffffu, d, 1);
        if (mine && !(lane & 1)) o[n >> 1] = d / (1.f + expf(-d)) * u;
    } else if (mine) {
        if (p.mode == FS_ADD) o[n] += d + bias;
        else if (p.mode == FS_PARTIAL) o[(size_t)split * p.M * p.ldo + n] = d;
        else o[n] = d + bias;
    }
}

// The results of tile t that this epilogue warp's lanes mark in odd0 and odd1.  (Inline, finding all it needs from t again, and with its
// loops rolled up: as a call it cost the kernel's main loops registers, 194 instead of 180 us for 1,999 x 9,728 x 896.)
template <int BN>
__device__ __forceinline__ void fs_again(const FsParams& p, uint32_t odd0, uint32_t odd1, int t) {
    constexpr int EC = BN / (FsLayout<BN>::epi_warps / 4);
    const int warp = threadIdx.x >> 5, split = t / (p.tiles_m * p.tiles_n), mc = (t % p.tiles_m) * BN + (warp >> 2) * EC;
    const int n = ((t / p.tiles_m) % p.tiles_n) * 128 + (warp & 3) * 32 + (threadIdx.x & 31);
    const int k0 = split * p.kb_split * FS_BK, k1 = min(p.K, k0 + p.kb_split * FS_BK);
    const float bias = (p.bias != nullptr && p.mode != FS_PARTIAL && n < p.N) ? load_vec(p.bias, p.bias_is_f32, n) : 0.f;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {
        uint32_t asked = n < p.N ? (i ? odd1 : odd0) : 0u;
        const uint32_t beside = __shfl_xor_sync(0xffffffffu, asked, 1);
        if (p.mode == FS_SWIGLU) asked |= beside;
#pragma unroll 1
        for (uint32_t left = __reduce_or_sync(0xffffffffu, asked); left; left &= left - 1) {
            const int j = __ffs(left) - 1, m = mc + i * 32 + j;
            if (m < p.M) fs_again_token(p, (asked >> j) & 1, m, n, k0, k1, split, bias);
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(FsLayout<BN>::threads, FsLayout<BN>::ctas)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const FsParams p) {
    using L = FsLayout<BN>;
    constexpr int S = L::stages, EW = L::epi_warps, CW = L::conv_warps, NB = L::bufs;
    constexpr int EC = BN / (EW / 4);                     // columns of an epilogue warp
    constexpr uint32_t TM_A = 2 * BN;                     // tensor memory: two accumulators, then split weights (3 x 16 columns a stage)

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* planes = smem + S * L::stage_bytes;          // [NB buffers][3 parts][BN rows][64 bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(planes + NB * 3 * L::plane_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::n_bars);
    __shared__ int abort_flag;
    const uint32_t b_raw_full = smem_u32(bars), b_raw_empty = b_raw_full + 8 * S;
    const uint32_t b_cv_full = b_raw_empty + 8 * S, b_cv_empty = b_cv_full + 8 * NB;
    const uint32_t b_acc_full = b_cv_empty + 8 * NB, b_acc_empty = b_acc_full + 16;

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < S; ++s) {
            mbar_init(b_raw_full + 8 * s, 1);
            mbar_init(b_raw_empty + 8 * s, 4);
        }
        for (int b = 0; b < NB; ++b) {
            mbar_init(b_cv_full + 8 * b, 4);
            mbar_init(b_cv_empty + 8 * b, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(b_acc_full + 8 * b, 1);
            mbar_init(b_acc_empty + 8 * b, EW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    }
    if (warp == EW + CW) {
        tcgen05_alloc(smem_u32(tmem_slot), L::tmem_cols);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;

    const int n_tiles = p.tiles_m * p.tiles_n * p.splits;
    const int kb_all = (p.K + FS_BK - 1) / FS_BK;
    // tile t: token tile t % tiles_m (neighbours share a weight tile in L2), weight tile, split of K
    auto tile_of = [&](int t, int& m0, int& n0, int& kb0, int& kb1) {
        m0 = (t % p.tiles_m) * BN;
        n0 = ((t / p.tiles_m) % p.tiles_n) * 128;
        kb0 = (t / (p.tiles_m * p.tiles_n)) * p.kb_split;
        kb1 = min(kb_all, kb0 + p.kb_split);
    };

    if (warp == EW + CW) {
        // ---------------- producer
        if (lane == 0) {
            int pre = 0, it = 0;
            if ((int)blockIdx.x < n_tiles) {              // the weights do not depend on the kernel before this one
                int m0, n0, kb0, kb1;
                tile_of(blockIdx.x, m0, n0, kb0, kb1);
                pre = min(S, kb1 - kb0);
                for (int i = 0; i < pre; ++i) {
                    mbar_expect_tx(b_raw_full + 8 * i, L::stage_bytes);
                    tma_load_2d(smem_u32(smem + i * L::stage_bytes), &map_w, (kb0 + i) * FS_BK, n0, b_raw_full + 8 * i);
                }
            }
            pdl_wait();
            for (int t = blockIdx.x; t < n_tiles && !abort_flag; t += gridDim.x) {
                int m0, n0, kb0, kb1;
                tile_of(t, m0, n0, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % S;
                    const uint32_t full = b_raw_full + 8 * s, dst = smem_u32(smem + s * L::stage_bytes);
                    if (it >= pre) {
                        if (!mbar_wait(b_raw_empty + 8 * s, ((it / S) & 1) ^ 1, &abort_flag)) break;
                        mbar_expect_tx(full, L::stage_bytes);
                        tma_load_2d(dst, &map_w, kb * FS_BK, n0, full);
                    }
                    tma_load_2d(dst + L::w_bytes, &map_x, kb * FS_BK, m0, full);
                }
            }
        }
    } else if (warp == EW + CW + 1) {
        // ---------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc(BN);
            int it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
                int m0, n0, kb0, kb1;
                tile_of(t, m0, n0, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const int b = it & 1, c = it % NB;
                    ok = mbar_wait(b_acc_empty + 8 * b, ((it >> 1) & 1) ^ 1, &abort_flag) &&
                         mbar_wait(b_cv_full + 8 * c, (it / NB) & 1, &abort_flag);
                    if (!ok) break;
                    tcgen05_fence_after();
                    const uint32_t d = tmem + b * BN, a = tmem + TM_A + c * 48;
                    const uint32_t x = smem_u32(planes) + c * 3 * L::plane_bytes;
                    // parts (weight, token) of a product, the smallest first
                    constexpr int pw[6] = {2, 1, 0, 1, 0, 0}, px[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
                    for (int q = 0; q < 6; ++q)
#pragma unroll
                        for (int h = 0; h < 2; ++h)       // 16 k each
                            tcgen05_mma_bf16_ts(d, a + pw[q] * 16 + h * 8, fs_desc(x + px[q] * L::plane_bytes + h * 32), idesc,
                                                (q | h) ? 1u : 0u);
                    tcgen05_commit(b_cv_empty + 8 * c);
                    tcgen05_commit(b_acc_full + 8 * b);
                }
            }
        }
    } else if (warp >= EW) {
        // ---------------- converters.  Four warps split a whole stage, a thread one weight row and some of the tokens'; with
        // eight warps the two fours take turns, so that one's waits and loads lie beside the other's arithmetic (all eight on
        // the same stage: 198 us for 1,999 x 9,728 x 896)
        constexpr int GROUPS = CW / 4, XU = (BN * 4 + 127) / 128;     // token pieces of 8 numbers per thread
        const int quarter = warp & 3, row = quarter * 32 + lane, group = (warp - EW) >> 2;
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            int m0, n0, kb0, kb1;
            tile_of(t, m0, n0, kb0, kb1);
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                if (GROUPS == 2 && (it & 1) != group) continue;
                const int s = it % S, b = it % NB;
                ok = mbar_wait(b_raw_full + 8 * s, (it / S) & 1, &abort_flag);
                if (!ok) break;
                const uint32_t w = smem_u32(smem + s * L::stage_bytes) + row * 128, x = smem_u32(smem + s * L::stage_bytes) + L::w_bytes;
                float4 wv[8], xv[2 * XU];
#pragma unroll
                for (int c = 0; c < 8; ++c) wv[c] = fs_lds(w + ((c ^ (row & 7)) << 4));
#pragma unroll
                for (int i = 0; i < XU; ++i) {
                    const int u = row + 128 * i, r = u % BN, c = u / BN;
                    if (BN * 4 >= 128 || u < BN * 4) {
                        xv[2 * i] = fs_lds(x + r * 128 + (((2 * c) ^ (r & 7)) << 4));
                        xv[2 * i + 1] = fs_lds(x + r * 128 + (((2 * c + 1) ^ (r & 7)) << 4));
                    }
                }
                ok = mbar_wait(b_cv_empty + 8 * b, ((it / NB) & 1) ^ 1, &abort_flag);
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t ta = tmem + TM_A + b * 48 + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t p1[8], p2[8], p3[8];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 v = wv[h * 4 + c];
                        fs_split2(v.x, v.y, p1[2 * c], p2[2 * c], p3[2 * c]);
                        fs_split2(v.z, v.w, p1[2 * c + 1], p2[2 * c + 1], p3[2 * c + 1]);
                    }
                    fs_st8(ta + h * 8, p1);
                    fs_st8(ta + 16 + h * 8, p2);
                    fs_st8(ta + 32 + h * 8, p3);
                }
                const uint32_t pl = smem_u32(planes) + b * 3 * L::plane_bytes;
#pragma unroll
                for (int i = 0; i < XU; ++i) {
                    const int u = row + 128 * i, r = u % BN, c = u / BN;
                    if (BN * 4 >= 128 || u < BN * 4) {
                        const float4 v0 = xv[2 * i], v1 = xv[2 * i + 1];
                        uint32_t q1[4], q2[4], q3[4];
                        fs_split2(v0.x, v0.y, q1[0], q2[0], q3[0]);
                        fs_split2(v0.z, v0.w, q1[1], q2[1], q3[1]);
                        fs_split2(v1.x, v1.y, q1[2], q2[2], q3[2]);
                        fs_split2(v1.z, v1.w, q1[3], q2[3], q3[3]);
                        const uint32_t o = pl + r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o), "r"(q1[0]), "r"(q1[1]), "r"(q1[2]), "r"(q1[3]) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + L::plane_bytes), "r"(q2[0]), "r"(q2[1]), "r"(q2[2]), "r"(q2[3]) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + 2 * L::plane_bytes), "r"(q3[0]), "r"(q3[1]), "r"(q3[2]), "r"(q3[3]) : "memory");
                    }
                }
                tcgen05_wait_st();
                tcgen05_fence_before();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    at_arrive(b_raw_empty + 8 * s);
                    at_arrive(b_cv_full + 8 * b);
                }
            }
        }
    } else {
        // ---------------- epilogue: the stages' sums into registers, then out
        const int quarter = warp & 3, c_first = (warp >> 2) * EC;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        pdl_wait();                                       // the output may still be read by the kernel before us
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            int m0, n0, kb0, kb1;
            tile_of(t, m0, n0, kb0, kb1);
            float acc[EC];
#pragma unroll
            for (int j = 0; j < EC; ++j) acc[j] = 0.f;
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const int b = it & 1;
                ok = mbar_wait(b_acc_full + 8 * b, (it >> 1) & 1, &abort_flag);
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t ta = tmem + b * BN + lane_base + c_first;
#pragma unroll
                for (int c0 = 0; c0 < EC; c0 += 16) {
                    uint32_t r[16];
                    tcgen05_ld16(ta + c0, r);
                    tcgen05_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(r[j]);
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) at_arrive(b_acc_empty + 8 * b);
            }
            if (!ok) break;
            const int n = n0 + quarter * 32 + lane;
            const int mc = m0 + c_first;                  // the first token of this warp's columns
            const int split = t / (p.tiles_m * p.tiles_n);
            const float bias = (p.bias != nullptr && p.mode != FS_PARTIAL && n < p.N) ? load_vec(p.bias, p.bias_is_f32, n) : 0.f;
            if (p.mode == FS_SWIGLU) {
                // gate in even lanes, up in the odd lane beside it; two tokens at a time, so that every lane evaluates and stores
                const bool odd = lane & 1;
                float* o = reinterpret_cast<float*>(p.out) + (n >> 1);
#pragma unroll
                for (int j = 0; j < EC; j += 2) {
                    const float got = __shfl_xor_sync(0xffffffffu, odd ? acc[j] : acc[j + 1], 1);
                    const float g = odd ? got : acc[j], u = odd ? acc[j + 1] : got;
                    const int m = mc + j + (odd ? 1 : 0);
                    if (m < p.M && (n | 1) < p.N) o[(size_t)m * p.ldo] = g / (1.f + expf(-g)) * u;
                }
            } else if (n < p.N) {
                float* o = reinterpret_cast<float*>(p.out) + (p.mode == FS_PARTIAL ? (size_t)split * p.M * p.ldo : (size_t)0) + n;
                if (p.mode == FS_ADD) {
#pragma unroll
                    for (int j = 0; j < EC; ++j)
                        if (mc + j < p.M && fabsf(acc[j]) <= 3.402823466e38f) o[(size_t)(mc + j) * p.ldo] += acc[j] + bias;
                } else {
#pragma unroll
                    for (int j = 0; j < EC; ++j)
                        if (mc + j < p.M) o[(size_t)(mc + j) * p.ldo] = acc[j] + bias;
                }
            }
            // the ones that are not finite, formed again and written over what was written above
            static_assert(EC <= 64, "two words of marks");
            uint32_t odd0 = 0u, odd1 = 0u;
#pragma unroll
            for (int j = 0; j < EC; ++j)
                if (!(fabsf(acc[j]) <= 3.402823466e38f)) { if (j < 32) odd0 |= 1u << (j & 31); else odd1 |= 1u << (j & 31); }
            if (__any_sync(0xffffffffu, (odd0 | odd1) != 0)) {
                __syncwarp();                             // what is written over comes after what was written
                fs_again<BN>(p, odd0, odd1, t);
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == EW + CW) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem, L::tmem_cols);
    }
    if (threadIdx.x == 0 && abort_flag && p.status) atomicExch(p.status, 11);
}

// ---------------------------------------------------------------- host side
template <int BN>
static int fs_launch(FsParams p, int sms, cudaStream_t st) {
    using L = FsLayout<BN>;
    static PerDevice<bool> devices;
    bool& configured = devices.here();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    CUtensorMap mw, mx;
    int e;
    if ((e = fs_map(&mw, p.W, p.N, p.K, p.K, 128)) || (e = fs_map(&mx, p.X, p.M, p.K, p.ldx, BN))) return e;
    p.tiles_m = (p.M + BN - 1) / BN;
    p.tiles_n = (p.N + 127) / 128;
    const long long tiles = (long long)p.tiles_m * p.tiles_n * p.splits;
    if (tiles > 0x3fffffff) return RF_ERR_UNSUPPORTED;
    const int grid = (int)(tiles < (long long)sms * L::ctas ? tiles : (long long)sms * L::ctas);
    cudaError_t le = rf_launch(gemm_f32_tc_kernel<BN>, dim3(grid), dim3(L::threads), L::smem, st, mw, mx, p);
    if (le != cudaSuccess) return (int)le;
    RF_LAUNCH_CHECK();
    return 0;
}

extern "C" {

// Whether the tensor cores take this product: 16-byte rows (K, ldx multiples of 4 and aligned bases are the caller's to check).
int rf_gemm_f32_tc_supported(int M, int N, int K) { return M > 0 && N > 0 && K > 0 && K % 4 == 0 && encode_fn() != nullptr; }

// mode 0: out [M, N] = X W^T (+ bias);  2: out += X W^T (+ bias);  3: out [splits, M, N] = partial sums of K ranges;
// 4: out [M, N/2] = silu(gate) * up of row-interleaved gate/up weights (no bias).  ldo: row stride of out.  bn: tokens of a
// tile (16, 32, 64 or 128).
int rf_gemm_f32_tc(const void* X, int ldx, const void* W, const void* bias, int bias_is_f32, void* out, int ldo, int M, int N, int K,
                   int mode, int splits, int bn, int sms, int* status, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (!rf_gemm_f32_tc_supported(M, N, K)) return RF_ERR_UNSUPPORTED;
    if ((mode != FS_STORE && mode != FS_ADD && mode != FS_PARTIAL && mode != FS_SWIGLU) || splits < 1 || sms < 1) return RF_ERR_BAD_ARG;
    if (splits > 1 && mode != FS_PARTIAL) return RF_ERR_BAD_ARG;
    if (mode == FS_PARTIAL && ldo != N) return RF_ERR_BAD_ARG;
    if (mode == FS_SWIGLU && (N % 2 || bias)) return RF_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(W) & 15) || ldx % 4 || ldx < K) return RF_ERR_BAD_ARG;
    const int kb = (K + FS_BK - 1) / FS_BK, per = (kb + splits - 1) / splits;
    if ((splits - 1) * per >= kb) return RF_ERR_BAD_ARG;          // an empty split would leave its partial sums unwritten
    FsParams p{reinterpret_cast<const float*>(X), reinterpret_cast<const float*>(W), out, bias, bias_is_f32, M, N, K, ldx, ldo, mode,
               0, 0, splits, per, status};
    if (bn == 16) return fs_launch<16>(p, sms, st);
    if (bn == 32) return fs_launch<32>(p, sms, st);
    if (bn == 64) return fs_launch<64>(p, sms, st);
    if (bn == 128) return fs_launch<128>(p, sms, st);
    return RF_ERR_BAD_ARG;
}

}
