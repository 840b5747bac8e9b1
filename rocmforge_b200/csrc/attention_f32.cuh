// Attention of the true 32-bit path for heads of 64 or 128 (prompts) and of 32, 64 or 128 numbers (single tokens), over the paged
// cache.  Plain softmax with a window or chunks; the generic kernel beside it serves every other size and option.
//
// Prompts: both products on the tensor cores, every number split into three bfloat16 parts and six of the nine products of parts
// formed, as in gemm_f32_tc.cuh (whose file says why that is a 32-bit product).  A CTA owns 128 consecutive new tokens of a
// sequence and a query head.  The queries' parts stay in tensor memory as the A operand; keys and values arrive as float32 tiles by
// TMA, converter warps split them into swizzled tiles in shared memory; a thread per query row takes its scores from tensor memory,
// forms the softmax in 32 bits, splits the weights and writes their parts back as the A operand of the second product.  The sums
// of a tile's values are added to the row's sums in registers (the tensor cores do not round to nearest when they add, so no sum
// stays there for longer than a tile).
//
// Single tokens: a cluster of CTAs per (token, kv head), a warp takes 4 * 32 / LPK keys at a time straight from memory (a lane holds
// four dimensions of a key, LPK = head size / 4 lanes a key), for all query heads of the group at once.
//
// What the kernel before wrote (queries, keys, values) is read through pointers without __restrict__: the compiler takes loads
// through const __restrict__ pointers for loads of what nobody writes, and may move them up across the wait for that kernel (it did
// so with the queries of the token kernel).
//
// Measured (us, the generic kernel's in brackets; 14 heads of 64 on 2 kv heads): a prompt of 1,999 tokens 68 [1,775], 8 of 16..1,024
// 63 [1,205]; 28 heads of 128, 1,024 tokens 66 [1,886]; single tokens of 64 sequences of 16..1,024 keys 22.5 [142], of one with 20,000
// 56 [2,240].  Error against 64 bits 1.7e-7 [2.6e-7], 1.4e-7 [2.6e-7] for single tokens.  A prompt's tile of 64 keys takes 2.7 us
// where its MMAs need 0.8: one softmax warp a scheduler forms, splits and writes 64 weights a row with nothing beside it.
#pragma once
#include "f32_parts.cuh"

__device__ __forceinline__ void fs_lds8(uint32_t a0, uint32_t a1, float4& u, float4& v) { u = fs_lds(a0); v = fs_lds(a1); }

#define FA_WARPS 10                                  // 4 softmax, 4 converters, producer, MMA issuer

template <int HD> struct FaLayout {
    static constexpr int KT = 4096 / HD;                        // keys of a tile
    static constexpr uint32_t raw_bytes = KT * HD * 4;          // 16 KB
    static constexpr uint32_t plane_bytes = KT * HD * 2;        // 8 KB: HD / 64 blocks of [KT rows][128 bytes]
    static constexpr uint32_t block_bytes = KT * 128;
    static constexpr int raws = 4;
    static constexpr size_t smem = raws * raw_bytes + 2 * 2 * 3 * plane_bytes + 32 * 8 + 16 + 1024;
    static constexpr uint32_t tm_s = 0, tm_p = 2 * KT, tm_o = tm_p + 3 * KT / 2, tm_q = tm_o + HD;     // 512 columns at most
};

// Rows of a warp's 32 again (a bit each in `rows`), key after key in ascending order, by the whole warp: what rows that are not finite
// get.  A lane holds HD / 32 dimensions.  A row's sum of weights that is no number stays so and gives zeros, as in the generic kernel,
// so the walk ends there.  (One thread a row with its sums in memory: 1,999 tokens of 14 heads with an infinite value
// 250 ms, now 7.3, and 0.09 with a key that is not a number; without either 0.067, the generic kernel 1.8.)
template <int HD>
__device__ __noinline__ void fa_again(uint32_t rows, const float* q, int q_stride, float* out, int out_stride, const float* k_pages,
                                      const float* v_pages, const int* bt, int kvh, int nkv, int window, int pos_first, float scale) {
    constexpr int E = HD / 32, U = 4, R = 4;             // four rows and four keys at a time
    struct alignas(4 * E) Piece { float v[E]; };
    const int lane = threadIdx.x & 31;
    while (rows) {
        int row[R];
        Piece qv[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {                    // (the last row again where fewer are left: the same numbers, written twice)
            row[r] = rows ? __ffs(rows) - 1 : row[r > 0 ? r - 1 : 0];
            rows &= rows - 1;
            qv[r] = *reinterpret_cast<const Piece*>(q + (size_t)row[r] * q_stride + lane * E);
        }
        const int first = rf_first_key(pos_first + row[0], window), last = pos_first + row[R - 1];       // (rows ascend)
        float m[R], l[R], o[R][E] = {};
        int lo[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { m[r] = -INFINITY; l[r] = 0.f; lo[r] = rf_first_key(pos_first + row[r], window); }
#pragma unroll 1
        for (int j0 = first; j0 <= last; j0 += U) {
            float s[R][U];
            Piece vv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = min(j0 + u, last);
                const size_t at = (((size_t)bt[j / RF_PAGE] * nkv + kvh) * RF_PAGE + (j % RF_PAGE)) * HD + lane * E;
                const Piece kk = *reinterpret_cast<const Piece*>(k_pages + at);
                vv[u] = *reinterpret_cast<const Piece*>(v_pages + at);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    s[r][u] = 0.f;
#pragma unroll
                    for (int d = 0; d < E; ++d) s[r][u] = fmaf(qv[r].v[d], kk.v[d], s[r][u]);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int u = 0; u < U; ++u) s[r][u] = warp_sum(s[r][u]) * scale;
            bool more = false;
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (j0 + u < lo[r] || j0 + u > pos_first + row[r]) continue;
                    const float mn = fmaxf(m[r], s[r][u]), c = m[r] == -INFINITY ? 0.f : expf(m[r] - mn), p = s[r][u] == -INFINITY ? 0.f : expf(s[r][u] - mn);
                    l[r] = l[r] * c + p;
#pragma unroll
                    for (int d = 0; d < E; ++d) o[r][d] = o[r][d] * c + p * vv[u].v[d];
                    m[r] = mn;
                }
                more = more || !isnan(l[r]);
            }
            if (!more) break;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            Piece y;
#pragma unroll
            for (int d = 0; d < E; ++d) y.v[d] = l[r] > 0.f ? o[r][d] / l[r] : 0.f;
            *reinterpret_cast<Piece*>(out + (size_t)row[r] * out_stride + lane * E) = y;
        }
    }
}

template <int HD>
__global__ void __launch_bounds__(FA_WARPS * 32, 1)
attention_f32_prompt_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                            const float* q, int q_stride, float* out, int out_stride,
                            const float* k_pages, const float* v_pages, const int* __restrict__ tiles,
                            const int* __restrict__ seq_slot, const int* __restrict__ seq_start, const int* __restrict__ seq_nnew,
                            const int* __restrict__ cu_q, const int* __restrict__ block_table, int max_pages, int nh, int nkv,
                            float scale, int window, int* __restrict__ status) {
    using L = FaLayout<HD>;
    constexpr int KT = L::KT, R = L::raws;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* planes = smem + R * L::raw_bytes;                  // [K | V][2 buffers][3 parts][HD / 64 blocks][KT rows][128 bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(planes + 2 * 2 * 3 * L::plane_bytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
    __shared__ int abort_flag;
    const uint32_t b0 = smem_u32(bars);
    const uint32_t b_raw_full = b0, b_raw_empty = b0 + 32, b_cv_full = b0 + 64, b_cv_free = b0 + 96;      // cv: [K0, K1, V0, V1]
    const uint32_t b_q = b0 + 128, b_s = b0 + 136, b_p = b0 + 152, b_pv = b0 + 168;                       // s, p, pv: two each

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile_idx = gridDim.y - 1 - blockIdx.y;            // the tiles with the most keys first
    const int seq = tiles[2 * tile_idx], q0 = tiles[2 * tile_idx + 1];
    const int head = blockIdx.x, kvh = head / (nh / nkv);
    const int start = seq_start[seq], n_new = seq_nnew[seq];
    const int* bt = block_table + (size_t)seq_slot[seq] * max_pages;
    const int row_base = cu_q[seq] + q0, rows_here = min(n_new - q0, 128);
    const int pos_first = start + q0, pos_last = pos_first + rows_here - 1, seq_last = start + n_new - 1;
    const int t_lo = rf_first_key(pos_first, window) / KT, n_t = pos_last / KT - t_lo + 1;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < 4; ++i) {
            mbar_init(b_raw_full + 8 * i, 1); mbar_init(b_raw_empty + 8 * i, 4);
            mbar_init(b_cv_full + 8 * i, 4); mbar_init(b_cv_free + 8 * i, 1);
        }
        mbar_init(b_q, 128);
        for (int i = 0; i < 2; ++i) { mbar_init(b_s + 8 * i, 1); mbar_init(b_p + 8 * i, 128); mbar_init(b_pv + 8 * i, 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    }
    if (warp == 9) {
        tcgen05_alloc(smem_u32(tmem_slot), 512);
        tcgen05_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();                                                 // queries, keys and values come from the kernel before us

    if (warp == 8) {
        // ---------------- producer: item 2t is tile t's keys, 2t + 1 its values
        if (lane == 0) {
            for (int i = 0; i < 2 * n_t; ++i) {
                const int s = i % R, key0 = (t_lo + (i >> 1)) * KT;
                if (!mbar_wait(b_raw_empty + 8 * s, ((i / R) & 1) ^ 1, &abort_flag)) break;
                mbar_expect_tx(b_raw_full + 8 * s, L::raw_bytes);
                const int row = (bt[key0 / RF_PAGE] * nkv + kvh) * RF_PAGE + key0 % RF_PAGE;
                for (int c = 0; c < HD / 32; ++c)
                    tma_load_2d(smem_u32(smem + s * L::raw_bytes + c * L::block_bytes), (i & 1) ? &map_v : &map_k, c * 32, row, b_raw_full + 8 * s);
            }
        }
    } else if (warp == 9) {
        // ---------------- MMA issuer
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc(KT), idesc_o = make_idesc(HD) | (1u << 16);           // values: MN-major
            constexpr int pa[6] = {2, 1, 0, 1, 0, 0}, pb[6] = {0, 1, 2, 0, 1, 0};                          // parts, the smallest products first
            auto issue_s = [&](int t) -> bool {
                const int b = t & 1;
                if (!mbar_wait(b_cv_full + 8 * b, (t >> 1) & 1, &abort_flag)) return false;
                tcgen05_fence_after();
                const uint32_t k = smem_u32(planes) + b * 3 * L::plane_bytes;
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks)
                        tcgen05_mma_bf16_ts(tmem + L::tm_s + b * KT, tmem + L::tm_q + pa[i] * (HD / 2) + ks * 8,
                                            make_smem_desc(k + pb[i] * L::plane_bytes + (ks >> 2) * L::block_bytes + (ks & 3) * 32), idesc_s,
                                            (i | ks) ? 1u : 0u);
                tcgen05_commit(b_s + 8 * b);
                tcgen05_commit(b_cv_free + 8 * b);
                return true;
            };
            bool ok = mbar_wait(b_q, 0, &abort_flag) && issue_s(0);
            for (int t = 0; t < n_t && ok; ++t) {
                const int b = t & 1;
                if (t + 1 < n_t && !(ok = issue_s(t + 1))) break;         // its buffer of scores was read before P(t - 1) was handed over
                ok = mbar_wait(b_p + 8 * b, (t >> 1) & 1, &abort_flag) && mbar_wait(b_cv_full + 16 + 8 * b, (t >> 1) & 1, &abort_flag);
                if (!ok) break;
                tcgen05_fence_after();
                const uint32_t v = smem_u32(planes) + (2 + b) * 3 * L::plane_bytes;
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int ks = 0; ks < KT / 16; ++ks)
                        tcgen05_mma_bf16_ts(tmem + L::tm_o, tmem + L::tm_p + pa[i] * (KT / 2) + ks * 8,
                                            make_smem_desc_mn(v + pb[i] * L::plane_bytes + ks * 16 * 128, L::block_bytes), idesc_o, (i | ks) ? 1u : 0u);
                tcgen05_commit(b_pv + 8 * b);
                tcgen05_commit(b_cv_free + 16 + 8 * b);
            }
        }
    } else if (warp >= 4) {
        // ---------------- converters: raw tiles into parts
        const int ct = threadIdx.x - 128;
        for (int i = 0; i < 2 * n_t; ++i) {
            const int s = i % R, t = i >> 1, cv = (i & 1) * 2 + (t & 1);
            const int valid = seq_last - (t_lo + t) * KT;                 // rows beyond this were never written
            if (!mbar_wait(b_raw_full + 8 * s, (i / R) & 1, &abort_flag)) break;
            const uint32_t raw = smem_u32(smem + s * L::raw_bytes), pl = smem_u32(planes) + cv * 3 * L::plane_bytes;
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {                                 // 8 numbers of a row: piece c of HD / 8
                const int id = ct + 128 * u, r = id % KT, c = id / KT;
                const uint32_t a = raw + (c >> 2) * L::block_bytes + r * 128;
                fs_lds8(a + (((2 * (c & 3)) ^ (r & 7)) << 4), a + (((2 * (c & 3) + 1) ^ (r & 7)) << 4), v[2 * u], v[2 * u + 1]);
                if (r > valid) v[2 * u] = v[2 * u + 1] = make_float4(0.f, 0.f, 0.f, 0.f);      // weights of zero must meet numbers
            }
            if (!mbar_wait(b_cv_free + 8 * cv, ((t >> 1) & 1) ^ 1, &abort_flag)) break;
            tcgen05_fence_after();
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int id = ct + 128 * u, r = id % KT, c = id / KT;
                uint32_t q1[4], q2[4], q3[4];
                fs_split2(v[2 * u].x, v[2 * u].y, q1[0], q2[0], q3[0]);
                fs_split2(v[2 * u].z, v[2 * u].w, q1[1], q2[1], q3[1]);
                fs_split2(v[2 * u + 1].x, v[2 * u + 1].y, q1[2], q2[2], q3[2]);
                fs_split2(v[2 * u + 1].z, v[2 * u + 1].w, q1[3], q2[3], q3[3]);
                const uint32_t o = pl + (c >> 3) * L::block_bytes + r * 128 + (((c & 7) ^ (r & 7)) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o), "r"(q1[0]), "r"(q1[1]), "r"(q1[2]), "r"(q1[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + L::plane_bytes), "r"(q2[0]), "r"(q2[1]), "r"(q2[2]), "r"(q2[3]) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + 2 * L::plane_bytes), "r"(q3[0]), "r"(q3[1]), "r"(q3[2]), "r"(q3[3]) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                at_arrive(b_raw_empty + 8 * s);
                at_arrive(b_cv_full + 8 * cv);
            }
        }
    } else {
        // ---------------- softmax, one thread per query row
        const int row = threadIdx.x;
        const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
        const bool row_ok = row < rows_here;
        const int pos_i = pos_first + row, lo_i = rf_first_key(pos_i, window);
        const float* qr = q + (size_t)(row_base + row) * q_stride + (size_t)head * HD;
#pragma unroll 1
        for (int d = 0; d < HD; d += 16) {                      // the row's parts: 8 columns of tensor memory per 16 numbers and part
            uint32_t p1[8], p2[8], p3[8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float4 x = row_ok ? *reinterpret_cast<const float4*>(qr + d + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
                fs_split2(x.x, x.y, p1[2 * c], p2[2 * c], p3[2 * c]);
                fs_split2(x.z, x.w, p1[2 * c + 1], p2[2 * c + 1], p3[2 * c + 1]);
            }
            fs_st8(tl + L::tm_q + d / 2, p1);
            fs_st8(tl + L::tm_q + HD / 2 + d / 2, p2);
            fs_st8(tl + L::tm_q + HD + d / 2, p3);
        }
        tcgen05_wait_st();
        tcgen05_fence_before();
        at_arrive(b_q);
        const float sl2 = scale * 1.4426950408889634f;
        float m_ref = -INFINITY, l = 0.f, acc[HD];
#pragma unroll
        for (int d = 0; d < HD; ++d) acc[d] = 0.f;
        auto take = [&]() {                                     // the tile's sums of values into the row's
#pragma unroll
            for (int c0 = 0; c0 < HD; c0 += 16) {
                uint32_t r[16];
                tcgen05_ld16(tl + L::tm_o + c0, r);
                tcgen05_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c0 + j] += __uint_as_float(r[j]);
            }
        };
        bool ok = true;
        for (int t = 0; t < n_t; ++t) {
            const int b = t & 1, key0 = (t_lo + t) * KT;
            if (!(ok = mbar_wait(b_s + 8 * b, (t >> 1) & 1, &abort_flag))) break;
            tcgen05_fence_after();
            float s[KT];
#pragma unroll
            for (int c0 = 0; c0 < KT; c0 += 32) {
                uint32_t r[32];
                tcgen05_ld32(tl + L::tm_s + b * KT + c0, r);
                tcgen05_wait_ld();
#pragma unroll
                for (int j = 0; j < 32; ++j) s[c0 + j] = __uint_as_float(r[j]);
            }
            if (!(key0 + KT - 1 <= pos_first && rows_here == 128 && key0 >= rf_first_key(pos_last, window))) {
                const int last = row_ok ? pos_i - key0 : -1, low = lo_i - key0;
#pragma unroll
                for (int j = 0; j < KT; ++j)
                    if (j > last || j < low) s[j] = -INFINITY;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < KT; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], s[j]);
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
            float corr = 1.f;
            if (mx > m_ref + 8.f) {                             // the reference moves only when the maximum has grown by more than 2^8
                corr = m_ref == -INFINITY ? 0.f : at_exp2(m_ref - mx);
                m_ref = mx;
            }
            const float nref = m_ref == -INFINITY ? 0.f : -m_ref;
            float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < KT; ++j) {
                s[j] = at_exp2(fmaf(s[j], sl2, nref));
                sum4[j & 3] += s[j];
            }
            if (t > 0) {
                if (!(ok = mbar_wait(b_pv + 8 * (b ^ 1), ((t - 1) >> 1) & 1, &abort_flag))) break;      // P's place is free, the sums are there
                tcgen05_fence_after();
                take();
            }
            l = l * corr + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
            if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
                for (int d = 0; d < HD; ++d) acc[d] *= corr;
            }
#pragma unroll
            for (int j0 = 0; j0 < KT; j0 += 16) {
                uint32_t p1[8], p2[8], p3[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) fs_split2(s[j0 + 2 * c], s[j0 + 2 * c + 1], p1[c], p2[c], p3[c]);
                fs_st8(tl + L::tm_p + j0 / 2, p1);
                fs_st8(tl + L::tm_p + KT / 2 + j0 / 2, p2);
                fs_st8(tl + L::tm_p + KT + j0 / 2, p3);
            }
            tcgen05_wait_st();
            tcgen05_fence_before();
            at_arrive(b_p + 8 * b);
        }
        if (ok && (ok = mbar_wait(b_pv + 8 * ((n_t - 1) & 1), ((n_t - 1) >> 1) & 1, &abort_flag))) {
            tcgen05_fence_after();
            take();
            float* o = out + (size_t)(row_base + row) * out_stride + (size_t)head * HD;
            const float inv = l > 0.f ? 1.f / l : 0.f;
            bool fine = l <= 3.402823466e38f;
#pragma unroll
            for (int d = 0; d < HD; d += 4) {
                const float4 y = make_float4(acc[d] * inv, acc[d + 1] * inv, acc[d + 2] * inv, acc[d + 3] * inv);
                fine = fine && fabsf(y.x) <= 3.402823466e38f && fabsf(y.y) <= 3.402823466e38f && fabsf(y.z) <= 3.402823466e38f && fabsf(y.w) <= 3.402823466e38f;
                if (row_ok) *reinterpret_cast<float4*>(o + d) = y;
            }
            const uint32_t again = __ballot_sync(0xffffffffu, row_ok && !fine);
            if (again) {
                __syncwarp();                                   // what is written over comes after what was written
                const int row0 = warp * 32;
                fa_again<HD>(again, q + (size_t)(row_base + row0) * q_stride + (size_t)head * HD, q_stride,
                             out + (size_t)(row_base + row0) * out_stride + (size_t)head * HD, out_stride, k_pages, v_pages, bt, kvh, nkv, window,
                             pos_first + row0, scale);
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 9) {
        tcgen05_fence_after();
        tcgen05_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && abort_flag && status) atomicExch(status, 12);
}

// ---------------------------------------------------------------- single tokens

#define FD_WARPS 8
#define FD_U 4                                       // loads of a batch: 4 * 32 / LPK keys
#define FD_SHARES 8

__device__ __forceinline__ float eight_max(float v) {        // over eight neighbouring lanes (whole warps)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float eight_sum(float v) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// (rows of the output need no alignment)
__device__ __forceinline__ void fd_store(float* out, float4 O, float L) {
    out[0] = L > 0.f ? O.x / L : 0.f; out[1] = L > 0.f ? O.y / L : 0.f; out[2] = L > 0.f ? O.z / L : 0.f; out[3] = L > 0.f ? O.w / L : 0.f;
}

// LPK: lanes per key (head size / 4); GP: query heads of a pass.  gridDim.x = tokens * splits (a cluster of `splits`), y = kv heads,
// z = passes over the group's heads.  rows: the step's tokens that are taken (null: all).
//
// The keys a token sees are dealt to 1 .. 8 shares by their number alone (a share is at least a batch a warp), so its sums do not
// depend on what else is in the step; the CTAs, whose number follows the step's size, take the shares in turn and their results
// meet in the shares' order.  us, 14 heads of 64 on 2 kv heads, and with one share a CTA, whose sums followed the step's size: 1
// sequence of 1,023 keys 6.9 and 7.1, 8 of 16..1,024 7.9 and 8.0, 64 of them 22.5 and 19.4 (two CTAs take four shares each there).
// Tried: two batches a warp (64 sequences 22.6, 8 8.6); a number of CTAs that follows the keys alone, 256 a CTA (23.1 and 9.8:
// a cluster waits for the room of its idle CTAs too).
template <int LPK, int GP>
__global__ void __launch_bounds__(FD_WARPS * 32, 2)
attention_f32_token_kernel(const float* q, int q_stride, float* out, int out_stride,
                           const float* k_pages, const float* v_pages, const int* __restrict__ tok_seq,
                           const int* __restrict__ tok_pos, const int* __restrict__ seq_slot, const int* __restrict__ block_table,
                           int max_pages, int nh, int nkv, float scale, int window, int splits, int slots, const int* __restrict__ rows) {
    constexpr int HD = LPK * 4, KPL = 32 / LPK, BATCH = FD_U * KPL;
    extern __shared__ __align__(16) float wo[];      // [slots][warps][GP][HD]: a warp's sums of a share; then the shares' own
    float* co = wo + slots * FD_WARPS * GP * HD;     // [8 / splits, rounded up][GP][HD]
    __shared__ __align__(16) float pbuf[FD_WARPS][BATCH][GP];
    __shared__ __align__(16) float wc[FD_WARPS][GP], wm[FD_SHARES][FD_WARPS][GP], wl[FD_SHARES][FD_WARPS][GP];
    __shared__ float cm[FD_SHARES][GP], cl[FD_SHARES][GP], factor[FD_SHARES][8][GP], all_l[GP];
    constexpr int FOLD = GP * 8;                     // threads that fold the factors of a share: eight lanes a head
    static_assert(FD_WARPS == 8 && FD_SHARES == 8, "eight lanes fold the warps' and the shares' factors");
    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LPK, part = lane % LPK;
    const int rank = blockIdx.x % splits, t = rows != nullptr ? rows[blockIdx.x / splits] : blockIdx.x / splits, kvh = blockIdx.y;
    const int G = nh / nkv, g0 = blockIdx.z * GP, gb = min(GP, G - g0);
    const int pos = tok_pos[t], lo = rf_first_key(pos, window);
    const int* bt = block_table + (size_t)seq_slot[tok_seq[t]] * max_pages;
    const int shares = min(FD_SHARES, (pos - lo + FD_WARPS * BATCH) / (FD_WARPS * BATCH)), ctas = min(splits, shares);
    if (rank >= shares) return;                      // (rank 0 waits for the kernel before; a cluster's barriers do not wait for who has left)
    pdl_wait();
    float4 qv[GP];
#pragma unroll
    for (int g = 0; g < GP; ++g)
        qv[g] = g < gb ? *reinterpret_cast<const float4*>(q + (size_t)t * q_stride + (size_t)(kvh * G + g0 + g) * HD + part * 4)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
    // which head's score a lane ends up with, and whether it is the one that writes it
    int my_head = 0, off_left = LPK / 2;
#pragma unroll
    for (int h = GP / 2; h >= 1; h >>= 1, off_left >>= 1) if (lane & off_left) my_head += h;
    bool writes = true;
#pragma unroll
    for (int o = LPK / GP / 2; o >= 1; o >>= 1) if (lane & o) writes = false;
    for (int share0 = rank; share0 < shares; share0 += splits * slots) {
    if (share0 > rank) __syncthreads();              // the shares before have been summed up
    // the warps go through up to `slots` shares without waiting for each other
    int n_slots = 0;
    for (int share = share0; share < shares && n_slots < slots; share += splits, ++n_slots) {
    float m = -INFINITY, l = 0.f;                    // of my_head, over this lane's keys (m over the warp's)
    float4 o[GP];
#pragma unroll
    for (int g = 0; g < GP; ++g) o[g] = make_float4(0.f, 0.f, 0.f, 0.f);

    const int u_last = pos / BATCH, stride = shares * FD_WARPS;
    for (int u = lo / BATCH + share * FD_WARPS + warp; u <= u_last; u += stride) {
        const int key0 = u * BATCH;                  // a batch lies in one page
        const size_t base = (((size_t)bt[key0 / RF_PAGE] * nkv + kvh) * RF_PAGE + key0 % RF_PAGE) * HD + part * 4;
        float4 kv[FD_U], vv[FD_U];
#pragma unroll
        for (int j = 0; j < FD_U; ++j) {
            const int r = j * KPL + sub, key = key0 + r;
            const bool in = key >= lo && key <= pos;
            kv[j] = in ? *reinterpret_cast<const float4*>(k_pages + base + (size_t)r * HD) : make_float4(0.f, 0.f, 0.f, 0.f);
            vv[j] = in ? *reinterpret_cast<const float4*>(v_pages + base + (size_t)r * HD) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float s[FD_U], mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < FD_U; ++j) {
            float d[GP];
#pragma unroll
            for (int g = 0; g < GP; ++g)
                d[g] = fmaf(qv[g].w, kv[j].w, fmaf(qv[g].z, kv[j].z, fmaf(qv[g].y, kv[j].y, qv[g].x * kv[j].x)));
            // the lanes of a key trade halves of their heads until each has one head's sum
            int off = LPK / 2;
#pragma unroll
            for (int h = GP / 2; h >= 1; h >>= 1, off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int g = 0; g < h; ++g) {
                    const float got = __shfl_xor_sync(0xffffffffu, up ? d[g] : d[g + h], off);
                    d[g] = (up ? d[g + h] : d[g]) + got;
                }
            }
#pragma unroll
            for (; off >= 1; off >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], off);
            const int key = key0 + j * KPL + sub;
            s[j] = (key >= lo && key <= pos) ? d[0] * scale : -INFINITY;
            mx = fmaxf(mx, s[j]);
        }
#pragma unroll
        for (int off = LPK; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float mn = fmaxf(m, mx);
        const float corr = m == -INFINITY ? 0.f : expf(m - mn);
        m = mn;
        __syncwarp();                                // the batch before this one is used up
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < FD_U; ++j) {
            const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - mn);
            sum += p;
            if (writes) pbuf[warp][j * KPL + sub][my_head] = p;
        }
        l = l * corr + sum;
        if (__any_sync(0xffffffffu, corr != 1.f)) {
            if (writes && sub == 0) wc[warp][my_head] = corr;
            __syncwarp();
#pragma unroll
            for (int g = 0; g < GP; ++g) {
                const float c = wc[warp][g];
                o[g].x *= c; o[g].y *= c; o[g].z *= c; o[g].w *= c;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < FD_U; ++j) {
            float p[GP];
#pragma unroll
            for (int g = 0; g < GP; ++g) p[g] = pbuf[warp][j * KPL + sub][g];
#pragma unroll
            for (int g = 0; g < GP; ++g) {
                o[g].x = fmaf(p[g], vv[j].x, o[g].x); o[g].y = fmaf(p[g], vv[j].y, o[g].y);
                o[g].z = fmaf(p[g], vv[j].z, o[g].z); o[g].w = fmaf(p[g], vv[j].w, o[g].w);
            }
        }
    }
    // ---- the warp's state: sums over the lanes that held different keys
#pragma unroll
    for (int off = LPK; off < 32; off <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
        for (int g = 0; g < GP; ++g) {
            o[g].x += __shfl_xor_sync(0xffffffffu, o[g].x, off); o[g].y += __shfl_xor_sync(0xffffffffu, o[g].y, off);
            o[g].z += __shfl_xor_sync(0xffffffffu, o[g].z, off); o[g].w += __shfl_xor_sync(0xffffffffu, o[g].w, off);
        }
    }
    __syncwarp();
    if (sub == 0) {
        if (writes) { wm[n_slots][warp][my_head] = m; wl[n_slots][warp][my_head] = l; }
#pragma unroll
        for (int g = 0; g < GP; ++g) *reinterpret_cast<float4*>(wo + ((n_slots * FD_WARPS + warp) * GP + g) * HD + part * 4) = o[g];
    }
    }
    __syncthreads();
    // ---- each share's, warps in index order: their factors first, then the sums, four dimensions a thread
    const int at0 = share0 / splits;
    for (int i = threadIdx.x; i < (n_slots * FOLD + 31) / 32 * 32; i += FD_WARPS * 32) {      // (whole warps)
        const int k = min(i / FOLD, n_slots - 1), g = i / FD_WARPS % GP, w = i % FD_WARPS;
        const float mw = wm[k][w][g], M = eight_max(mw), f = mw == -INFINITY ? 0.f : expf(mw - M), L = eight_sum(f * wl[k][w][g]);
        if (i < n_slots * FOLD) {
            factor[k][w][g] = f;
            if (w == 0) { cm[at0 + k][g] = M; cl[at0 + k][g] = L; }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x * 4; i < n_slots * GP * HD; i += FD_WARPS * 128) {
        const int k = i / (GP * HD), e = i % (GP * HD), g = e / HD;
        float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < FD_WARPS; ++w) {
            const float f = factor[k][w][g];
            const float4 x = *reinterpret_cast<const float4*>(wo + (k * FD_WARPS + w) * GP * HD + e);
            O.x = fmaf(f, x.x, O.x); O.y = fmaf(f, x.y, O.y); O.z = fmaf(f, x.z, O.z); O.w = fmaf(f, x.w, O.w);
        }
        if (shares == 1) {
            if (g < gb) fd_store(out + (size_t)t * out_stride + (size_t)(kvh * G + g0) * HD + e, O, cl[0][g]);
        } else *reinterpret_cast<float4*>(co + at0 * GP * HD + i) = O;
    }
    }
    if (shares == 1) return;
    // ---- all shares, in their order, the same way; each CTA writes some of the dimensions
    if (ctas > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else __syncthreads();
    auto place = [&](const float* p, int r) {
        uint32_t a;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(r % splits));
        return a;
    };
    for (int i = threadIdx.x; i < (FOLD + 31) / 32 * 32; i += FD_WARPS * 32) {
        const int g = i / FD_SHARES % GP, r = i % FD_SHARES;
        float mr = -INFINITY, lr = 0.f;
        if (r < shares) {
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(mr) : "r"(place(&cm[r / splits][g], r)) : "memory");
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(lr) : "r"(place(&cl[r / splits][g], r)) : "memory");
        }
        const float M = eight_max(mr), f = mr == -INFINITY ? 0.f : expf(mr - M), L = eight_sum(f * lr);
        if (i < FOLD) {
            factor[0][r][g] = f;
            if (r == 0) all_l[g] = L;
        }
    }
    __syncthreads();
    for (int i = (rank * FD_WARPS * 32 + threadIdx.x) * 4; i < gb * HD; i += ctas * FD_WARPS * 128) {
        const int g = i / HD;
        float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < shares; ++r) {
            const float f = factor[0][r][g];
            float4 x;
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                         : "r"(place(co + (r / splits) * GP * HD + i, r)) : "memory");
            O.x = fmaf(f, x.x, O.x); O.y = fmaf(f, x.y, O.y); O.z = fmaf(f, x.z, O.z); O.w = fmaf(f, x.w, O.w);
        }
        fd_store(out + (size_t)t * out_stride + (size_t)(kvh * G + g0) * HD + i, O, all_l[g]);
    }
    if (ctas > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");    // nobody's memory goes while a peer reads it
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// ---------------------------------------------------------------- host side
template <int HD>
static int fa_launch(const float* q, int q_stride, float* out, int out_stride, const float* k_pages, const float* v_pages, long long n_pages,
                     const int* tiles, int n_tiles, const int* seq_slot, const int* seq_start, const int* seq_nnew, const int* cu_q,
                     const int* block_table, int max_pages, int nh, int nkv, float scale, int window, int* status, cudaStream_t st) {
    using L = FaLayout<HD>;
    static PerDevice<bool> devices;
    bool& configured = devices.here();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_f32_prompt_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    CUtensorMap mk, mv;
    int e;
    const long long rows = n_pages * nkv * RF_PAGE;
    if ((e = fs_map(&mk, k_pages, rows, HD, HD, L::KT)) || (e = fs_map(&mv, v_pages, rows, HD, HD, L::KT))) return e;
    cudaError_t le = rf_launch(attention_f32_prompt_kernel<HD>, dim3(nh, n_tiles), dim3(FA_WARPS * 32), L::smem, st, mk, mv, q, q_stride,
                               out, out_stride, k_pages, v_pages, tiles, seq_slot, seq_start, seq_nnew, cu_q, block_table, max_pages, nh, nkv,
                               scale, window, status);
    if (le != cudaSuccess) return (int)le;
    RF_LAUNCH_CHECK();
    return 0;
}

template <int LPK, int GP>
static int fd_launch(const float* q, int q_stride, float* out, int out_stride, const float* k_pages, const float* v_pages, const int* tok_seq,
                     const int* tok_pos, const int* seq_slot, const int* block_table, int max_pages, int nh, int nkv, float scale, int window,
                     int T, int splits, const int* rows, cudaStream_t st) {
    const int G = nh / nkv;
    dim3 grid(T * splits, nkv, (G + GP - 1) / GP);
    // the shares of a CTA, and how many of them its warps may go through before their sums meet: as many as 64 KB hold
    const size_t share = (size_t)GP * LPK * 4 * sizeof(float);
    const int most = (FD_SHARES + splits - 1) / splits, fit = (int)((64 << 10) / (FD_WARPS * share)), slots = most < fit ? most : fit;
    const size_t smem = (slots * FD_WARPS + most) * share;
    static PerDevice<size_t> devices;
    size_t& configured = devices.here();
    if (smem > configured) {
        cudaError_t e = cudaFuncSetAttribute(attention_f32_token_kernel<LPK, GP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = smem;
    }
    cudaError_t le = splits > 1
        ? rf_launch_cluster(attention_f32_token_kernel<LPK, GP>, grid, dim3(FD_WARPS * 32), smem, st, splits, q, q_stride, out, out_stride, k_pages,
                            v_pages, tok_seq, tok_pos, seq_slot, block_table, max_pages, nh, nkv, scale, window, splits, slots, rows)
        : rf_launch(attention_f32_token_kernel<LPK, GP>, grid, dim3(FD_WARPS * 32), smem, st, q, q_stride, out, out_stride, k_pages, v_pages,
                    tok_seq, tok_pos, seq_slot, block_table, max_pages, nh, nkv, scale, window, splits, slots, rows);
    if (le != cudaSuccess) return (int)le;
    RF_LAUNCH_CHECK();
    return 0;
}

extern "C" {

int rf_attention_f32_prompt_supported(int nh, int nkv, int hd) {
    return nkv > 0 && nh % nkv == 0 && nh <= 65535 && (hd == 64 || hd == 128) && encode_fn() != nullptr;
}

// tiles: n_tiles pairs (sequence index, first new-token row of the tile within the sequence), 128 rows a tile, by the keys they see.
int rf_attention_f32_prompt(const float* q, int q_stride, float* out, int out_stride, const float* k_pages, const float* v_pages,
                            long long n_pages, const int* tiles, int n_tiles, const int* seq_slot, const int* seq_start, const int* seq_nnew,
                            const int* cu_q, const int* block_table, int max_pages, int nh, int nkv, int hd, float scale, int window,
                            int* status, cudaStream_t st) {
    if (n_tiles <= 0) return 0;
    if (!rf_attention_f32_prompt_supported(nh, nkv, hd) || n_tiles > 65535) return RF_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(k_pages) |
         reinterpret_cast<uintptr_t>(v_pages)) & 15 || q_stride % 4 || out_stride % 4 || !(scale > 0.f))
        return RF_ERR_BAD_ARG;
    return hd == 64 ? fa_launch<64>(q, q_stride, out, out_stride, k_pages, v_pages, n_pages, tiles, n_tiles, seq_slot, seq_start, seq_nnew,
                                    cu_q, block_table, max_pages, nh, nkv, scale, window, status, st)
                    : fa_launch<128>(q, q_stride, out, out_stride, k_pages, v_pages, n_pages, tiles, n_tiles, seq_slot, seq_start, seq_nnew,
                                     cu_q, block_table, max_pages, nh, nkv, scale, window, status, st);
}

int rf_attention_f32_token_supported(int nh, int nkv, int hd) {
    return nkv > 0 && nkv <= 65535 && nh % nkv == 0 && (hd == 32 || hd == 64 || hd == 128);
}

// splits: CTAs that share one (token, kv head), 1, 2, 4 or 8.  rows: T indices of the step's tokens, or null for the first T.
int rf_attention_f32_token(const float* q, int q_stride, float* out, int out_stride, const float* k_pages, const float* v_pages,
                           const int* tok_seq, const int* tok_pos, const int* seq_slot, const int* block_table, int max_pages, int nh, int nkv,
                           int hd, float scale, int window, int T, int splits, const int* rows, cudaStream_t st) {
    if (T <= 0) return 0;
    if (!rf_attention_f32_token_supported(nh, nkv, hd)) return RF_ERR_UNSUPPORTED;
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return RF_ERR_BAD_ARG;
    if ((long long)T * splits > 0x7fffffff || nh / nkv > 65535 * 2) return RF_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages)) & 15 || q_stride % 4)
        return RF_ERR_BAD_ARG;
    const int G = nh / nkv;
#define FD_GO(LPK, GP) fd_launch<LPK, GP>(q, q_stride, out, out_stride, k_pages, v_pages, tok_seq, tok_pos, seq_slot, block_table, max_pages, \
                                          nh, nkv, scale, window, T, splits, rows, st)
    if (hd == 32) return G <= 2 ? FD_GO(8, 2) : (G <= 4 ? FD_GO(8, 4) : FD_GO(8, 8));
    if (hd == 64) return G <= 2 ? FD_GO(16, 2) : (G <= 4 ? FD_GO(16, 4) : FD_GO(16, 8));
    return G <= 2 ? FD_GO(32, 2) : (G <= 4 ? FD_GO(32, 4) : FD_GO(32, 8));
#undef FD_GO
}

}
