// Softmax attention of a prompt pass (many queries of one sequence) on the tensor cores: attention_weights!, the division by
// sqrt(head_size), softmax! and combine_values! (src/inference.jl:263-278, 169-220) for every token of the pass at once.
//
// Block = 128 query rows (128 / GQ tokens x the GQ heads that share a key / value head), walking the cached positions 64 at a
// time.  Queries, keys, values and softmax weights are f32 and enter the tensor cores as two fp16 terms each, scaled by a power
// of two of their own (each query, key and value; weights, times the scales of their values, per query and tile), so that a
// product is high*high + high*low + low*high: what is left out is 2^-24 of it, and a query's result hangs on no position behind
// it.  The tensor core rounds its sums toward zero, so they are kept short (32 dims, 32 positions) and continued in f32
// registers; maxima, exponentials and their sums are f32.  Error against 64 bits, of the split kernel's in attention.cuh: 1.0 - 1.2 at 128 and
// 300 positions, 0.9 - 1.05 at 512, 0.6 at 1700; one value or key a million times its neighbours: 1.2 - 2.3 of it per row.
//
//   6 conversion warps  keys (thread = position, 8 dims) and values (thread = dim, 8 positions) from the caches to operand layout
//                       (core matrices of 8 rows x 16 bytes); the next tile's values are fetched while this one is waited for
//   MMA warp            S(j) = Q K^T, O(j) = P V
//   8 softmax warps     thread = query row, half of the positions, half of the output
//
// A tile of 64 positions takes 2.5 us (32 dims) to 6.8 us (128 dims): the conversion warps' own instructions.  With one scale per tile of keys and
// of values it was 4.6 us, but a value 2^-16 below its tile's largest lost bits, and an infinity or NaN reached the queries before it.
// What it replaces here read every position once per query: 128 times the cache traffic, on the CUDA cores.
#pragma once
#include <cuda_fp16.h>

#include "attention.cuh"
#include "kq_gemm.cuh"

namespace l2b {

constexpr int PA_ROWS = 128, PA_KEYS = 64;
constexpr int PA_CONV_WARPS = 6;  // 15 warps: four to a scheduler, so that 128 registers a thread are left (the softmax threads hold 64 outputs)
constexpr int PA_THREADS = (9 + PA_CONV_WARPS) * 32;  // warps 0-7 softmax, 8 MMA, 9 .. conversion
constexpr int PA_MAX_HS = 128;

struct PromptAttnParams {
    const float* q;      // [n][q_stride], after RoPE
    const float *kc, *vc;  // [kv_head][seq_len][hs]
    float* out;          // [n][q_stride]
    int n, pos0, q_stride, n_heads, n_kv, hs, seq_len;
    int* status;
};

// Of the positions of a tile: 1 / scale of the key; 1 / scale of the value and its exponent.
struct PaScales {
    float key[PA_KEYS], value[PA_KEYS], value_exp[PA_KEYS];
};
// Of the conversion warps: largest parts of the keys (three threads each) and values (bits of magnitudes; cleared two tiles ahead), the tile's scales.
struct PaConv {
    float key_max[3][PA_KEYS];
    unsigned value_max[3][PA_KEYS];
    float key_scale[PA_KEYS], value_scale[PA_KEYS];
};
struct PaSmem {
    int off_bar, off_max, off_sum, off_scale, off_conv, off_q, off_k, off_v, off_p, total;
};
__host__ __device__ inline PaSmem pa_smem_layout(int hs) {
    PaSmem s;
    s.off_bar = 0;       // k_ready p_ready s_full[2] v_ready[2] pv_full[2]; tensor memory address and the flag of non-finite values behind them
    s.off_max = 128;     // [2][2][128] {largest score, largest score + exponent of the value's scale} of the two halves, by tile parity
    s.off_sum = s.off_max + 4096;    // [2][128]
    s.off_scale = s.off_sum + 1024;  // [4] by tile: PaScales
    s.off_conv = s.off_scale + 4 * (int)sizeof(PaScales);  // PaConv
    s.off_q = (s.off_conv + (int)sizeof(PaConv) + 1023) & ~1023;
    s.off_k = s.off_q + 2 * PA_ROWS * hs * 2;  // [term][hs / 8][rows][16 bytes]
    s.off_v = s.off_k + 2 * PA_KEYS * hs * 2;
    s.off_p = s.off_v + 2 * 2 * PA_KEYS * hs * 2;  // two slots of values
    s.total = s.off_p + 2 * PA_ROWS * PA_KEYS * 2;
    return s;
}

__device__ __forceinline__ void pa_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Power of two that brings a largest magnitude of mx into [2^13, 2^14), and its inverse.
__device__ __forceinline__ float pa_scale(float mx, float& inv) {
    const int ex = (int)(__float_as_uint(mx) >> 23) & 255;
    const int up = mx == 0.f || ex == 255 ? 127 : min(267 - ex, 252);
    inv = __uint_as_float((uint32_t)(254 - up) << 23);
    return __uint_as_float((uint32_t)up << 23);
}
// Eight values times their scales as two fp16 terms: 16 bytes each.
__device__ __forceinline__ void pa_terms(const float (&v)[8], const float (&s)[8], uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = v[2 * i] * s[2 * i], b = v[2 * i + 1] * s[2 * i + 1];
        const __half2 x = __floats2half2_rn(a, b);
        const float2 y = __half22float2(x);
        h[i] = h2_raw(x);
        l[i] = h2_raw(__floats2half2_rn(a - y.x, b - y.y));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ void pa_terms(const float (&v)[8], float s, uint4& hi, uint4& lo) {
    const float all[8] = {s, s, s, s, s, s, s, s};
    pa_terms(v, all, hi, lo);
}

template <int GQ>
__global__ void __launch_bounds__(PA_THREADS, 1) prompt_attention_kernel(const __grid_constant__ PromptAttnParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int hs = p.hs, ns = hs >> 4;
    const PaSmem L = pa_smem_layout(hs);
    uint64_t* k_ready = reinterpret_cast<uint64_t*>(smem + L.off_bar);
    uint64_t *p_ready = k_ready + 1, *s_full = k_ready + 2, *v_ready = k_ready + 4, *pv_full = k_ready + 6;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(k_ready + 8);
    int* odd_values = reinterpret_cast<int*>(tmem_slot + 1);  // a value of this block is not finite
    float2* s_max = reinterpret_cast<float2*>(smem + L.off_max);
    float* s_sum = reinterpret_cast<float*>(smem + L.off_sum);
    PaScales* s_scale = reinterpret_cast<PaScales*>(smem + L.off_scale);
    PaConv& conv = *reinterpret_cast<PaConv*>(smem + L.off_conv);
    constexpr int TQ = PA_ROWS / GQ;  // tokens per block
    const int tok0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TQ;  // blocks with the most positions first
    const int hg = blockIdx.y, kvh = hg * GQ / (p.n_heads / p.n_kv);
    const int last = p.pos0 + min(p.n, tok0 + TQ) - 1;  // last position that a row of this block attends to
    const int tiles = last / PA_KEYS + 1;
    const int q_term = PA_ROWS * hs * 2, kv_term = PA_KEYS * hs * 2, p_term = PA_ROWS * PA_KEYS * 2;

    if (threadIdx.x < 3 * PA_KEYS) conv.value_max[threadIdx.x / PA_KEYS][threadIdx.x % PA_KEYS] = 0u;
    if (threadIdx.x == 0) {
        *odd_values = 0;
        mbar_init(k_ready, PA_CONV_WARPS);
        mbar_init(p_ready, 8);
        for (int i = 0; i < 2; ++i) {
            mbar_init(s_full + i, 1);
            mbar_init(v_ready + i, PA_CONV_WARPS);
            mbar_init(pv_full + i, 1);
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 8) tmem_alloc(tmem_slot, 512);
    pdl_wait();
    float q_inv = 1.f;
    if (warp < 8) {  // two threads per query row: its two terms (all loads in flight at once: one after the other they had taken 10 us)
        const int r = threadIdx.x & 127, half = threadIdx.x >> 7, t = min(tok0 + r % TQ, p.n - 1), h = hg * GQ + r / TQ, oct = hs >> 4;
        const float4* src = reinterpret_cast<const float4*>(p.q + (size_t)t * p.q_stride + (size_t)h * hs + half * (hs >> 1));
        float v[PA_MAX_HS / 16][8];
        float mx = 0.f;
#pragma unroll
        for (int i = 0; i < PA_MAX_HS / 16; ++i) {
            const float4 a = i < oct ? __ldcg(src + 2 * i) : make_float4(0.f, 0.f, 0.f, 0.f), b = i < oct ? __ldcg(src + 2 * i + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w; v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
        }
#pragma unroll
        for (int i = 0; i < PA_MAX_HS / 16; ++i)
#pragma unroll
            for (int k = 0; k < 8; ++k) mx = fmaxf(mx, fabsf(v[i][k]));
        s_max[half * 128 + r].x = mx;
        pa_bar_sync(1, 256);
        const float s = pa_scale(fmaxf(mx, s_max[(half ^ 1) * 128 + r].x), q_inv);
#pragma unroll
        for (int i = 0; i < PA_MAX_HS / 16; ++i)
            if (i < oct) {
                uint4 hi, lo;
                pa_terms(v[i], s, hi, lo);
                uint8_t* dst = smem + L.off_q + (half * oct + i) * (PA_ROWS * 16) + r * 16;
                *reinterpret_cast<uint4*>(dst) = hi;
                *reinterpret_cast<uint4*>(dst + q_term) = lo;
            }
        fence_proxy_async();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // tensor memory: S as up to four sums of 64 positions over `per` steps of 16 dims each; O behind it as two sums (32 positions each) of 128 columns
    const int per = (ns + 3) >> 2;
    bool ok = true;

    if (warp == 8) {
        // ================= MMA issue =================
        const uint32_t idesc_s = umma_idesc_f16(PA_ROWS, PA_KEYS), idesc_o = umma_idesc_f16(PA_ROWS, hs);
        const uint64_t dq = umma_desc(smem + L.off_q, PA_ROWS * 16, 128), dk = umma_desc(smem + L.off_k, PA_KEYS * 16, 128);
        const uint64_t dv = umma_desc(smem + L.off_v, hs * 16, 128), dp = umma_desc(smem + L.off_p, PA_ROWS * 16, 128);
        const uint32_t q_lo = q_term >> 4, kv_lo = kv_term >> 4, p_lo = p_term >> 4;
        auto scores = [&](int j) {
            if (!mbar_wait_warp(k_ready, (uint32_t)(j & 1))) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll 1
                for (int i0 = 0; i0 < ns; i0 += per) {
                    const int i1 = min(ns, i0 + per);
                    const uint32_t d = tmem + (uint32_t)(i0 / per * 64);
                    uint32_t acc = 0;
#pragma unroll 1
                    for (int t = 0; t < 3; ++t) {  // low terms first
                        const uint64_t a = dq + (t == 0 ? q_lo : 0u), b = dk + (t == 1 ? kv_lo : 0u);
#pragma unroll 1
                        for (int i = i0; i < i1; ++i) {
                            umma_f16(d, a + (uint64_t)(i * (2 * PA_ROWS)), b + (uint64_t)(i * (2 * PA_KEYS)), idesc_s, acc);
                            acc = 1;
                        }
                    }
                }
                umma_commit(s_full + (j & 1));
            }
            __syncwarp();
            return true;
        };
        ok = scores(0);
        for (int j = 0; j < tiles && ok; ++j) {
            if (!mbar_wait_warp(p_ready, (uint32_t)(j & 1)) || !mbar_wait_warp(v_ready + (j & 1), (uint32_t)((j >> 1) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint64_t v = dv + (uint64_t)((j & 1) * (2 * kv_term >> 4));
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {  // 32 positions each
                    uint32_t acc = 0;
#pragma unroll 1
                    for (int t = 0; t < 3; ++t) {
                        const uint64_t a = dp + (t == 0 ? p_lo : 0u), b = v + (t == 1 ? kv_lo : 0u);
#pragma unroll
                        for (int i = 0; i < PA_KEYS / 32; ++i) {
                            const int step = half * (PA_KEYS / 32) + i;
                            umma_f16(tmem + 256u + (uint32_t)(half * 128), a + (uint64_t)(step * (2 * PA_ROWS)), b + (uint64_t)(step * 2 * hs), idesc_o, acc);
                            acc = 1;
                        }
                    }
                }
                umma_commit(pv_full + (j & 1));
            }
            __syncwarp();
            if (j + 1 < tiles && !scores(j + 1)) ok = false;  // (all softmax threads have read S(j))
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    } else if (warp > 8) {
        // ================= conversion =================
        const int id = threadIdx.x - 9 * 32;
        const float* kbase = p.kc + (size_t)kvh * p.seq_len * hs;
        const float* vbase = p.vc + (size_t)kvh * p.seq_len * hs;
        constexpr int CT = PA_CONV_WARPS * 32, ITEMS = (PA_MAX_HS * PA_KEYS / 8 + CT - 1) / CT;
        const int items = hs * PA_KEYS / 8;
        float kv[ITEMS][8], vv[ITEMS][8];
        const int key = id & 63, chunk0 = id >> 6;
        const bool two_sets = (hs & 31) != 0;
        int v_pos[ITEMS];  // of this thread's values: first of eight positions
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) v_pos[u] = (id + CT * u) / hs * 8;
        auto fetch_k = [&](int j) {
            const int pos = j * PA_KEYS + key;
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const int c = chunk0 + CT / 64 * u;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                if (c < hs / 8 && pos <= last) {
                    const float4* src = reinterpret_cast<const float4*>(kbase + (size_t)pos * hs + 8 * c);
                    a = __ldcg(src);
                    b = __ldcg(src + 1);
                }
                kv[u][0] = a.x; kv[u][1] = a.y; kv[u][2] = a.z; kv[u][3] = a.w;
                kv[u][4] = b.x; kv[u][5] = b.y; kv[u][6] = b.z; kv[u][7] = b.w;
            }
        };
        auto fetch_v = [&](int j) {
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
                const int left = id + CT * u < items ? last - (j * PA_KEYS + v_pos[u]) : -1;
                const float* src = vbase + (size_t)j * PA_KEYS * hs + (id + CT * u + (v_pos[u] >> 3) * 7 * hs);  // dim (id + CT * u) % hs
#pragma unroll
                for (int k = 0; k < 8; ++k) vv[u][k] = k <= left ? __ldcg(src + k * hs) : 0.f;
            }
        };
        fetch_k(0);
        fetch_v(0);
        for (int j = 0; j < tiles; ++j) {
            float mk = 0.f;
            unsigned* const value_max = conv.value_max[j % 3];
#pragma unroll
            for (int u = 0; u < ITEMS; ++u) {
#pragma unroll
                for (int k = 0; k < 8; ++k) mk = fmaxf(mk, fabsf(kv[u][k]));
                if (id - lane + CT * u >= items) continue;  // (the same for a warp's threads: items are a multiple of 128)
                unsigned of_mine, all;  // lane k holds the maximum of the position k places on
                for (;;) {  // maxima over 32 dims of eight positions, over 16 where a warp's dims belong to two sets of positions
                    all = of_mine = 0u;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const unsigned bits = __float_as_uint(vv[u][k]) & 0x7FFFFFFFu;
                        unsigned m = __reduce_max_sync(0xffffffffu, two_sets && lane >= 16 ? 0u : bits);
                        if (two_sets) {
                            const unsigned upper = __reduce_max_sync(0xffffffffu, lane >= 16 ? bits : 0u);
                            if (lane >= 16) m = upper;
                        }
                        all = max(all, m);
                        if ((lane & 7) == k) of_mine = m;
                    }
                    if (!__any_sync(0xffffffffu, all >= 0x7F800000u)) break;
                    *odd_values = 1;  // infinities and NaN stay out of the product; the output adds them for the rows that see them
#pragma unroll
                    for (int k = 0; k < 8; ++k) vv[u][k] = fabsf(vv[u][k]) < INFINITY ? vv[u][k] : 0.f;
                }
                if ((lane & (two_sets ? 15 : 31)) < 8) atomicMax(value_max + v_pos[u] + (lane & 7), of_mine);
            }
            conv.key_max[chunk0][key] = mk;
            pa_bar_sync(2, CT);
            PaScales& scales = s_scale[j & 3];
            if (id < PA_KEYS) {
                const float vm = __uint_as_float(value_max[id]);
                conv.key_scale[id] = pa_scale(fmaxf(fmaxf(conv.key_max[0][id], conv.key_max[1][id]), conv.key_max[2][id]), scales.key[id]);
                float inv;
                conv.value_scale[id] = pa_scale(vm, inv);
                scales.value[id] = vm == 0.f ? 0.f : inv;
                scales.value_exp[id] = vm == 0.f ? -INFINITY : (float)((int)(__float_as_uint(inv) >> 23) - 127);
            } else if (id < 2 * PA_KEYS) {
                conv.value_max[(j + 2) % 3][id - PA_KEYS] = 0u;
            }
            pa_bar_sync(2, CT);
            const float ks = conv.key_scale[key];
            if (ok && j > 0 && !mbar_wait_warp(s_full + ((j - 1) & 1), (uint32_t)(((j - 1) >> 1) & 1))) ok = false;  // the last scores have read the keys
            if (ok) {
#pragma unroll
                for (int u = 0; u < ITEMS; ++u) {
                    const int c = chunk0 + CT / 64 * u;
                    if (c < hs / 8) {
                        uint4 hi, lo;
                        pa_terms(kv[u], ks, hi, lo);
                        uint8_t* dst = smem + L.off_k + c * (PA_KEYS * 16) + key * 16;
                        *reinterpret_cast<uint4*>(dst) = hi;
                        *reinterpret_cast<uint4*>(dst + kv_term) = lo;
                    }
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(k_ready);
            if (j + 1 < tiles) fetch_k(j + 1);
            if (ok && j > 1 && !mbar_wait_warp(pv_full + (j & 1), (uint32_t)(((j - 2) >> 1) & 1))) ok = false;
            if (ok) {
#pragma unroll
                for (int u = 0; u < ITEMS; ++u) {
                    const int idx = id + CT * u;
                    if (idx < items) {
                        const float4 s0 = *reinterpret_cast<const float4*>(conv.value_scale + v_pos[u]), s1 = *reinterpret_cast<const float4*>(conv.value_scale + v_pos[u] + 4);
                        const float vs[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
                        uint4 hi, lo;
                        pa_terms(vv[u], vs, hi, lo);
                        uint8_t* dst = smem + L.off_v + (j & 1) * 2 * kv_term + idx * 16;
                        *reinterpret_cast<uint4*>(dst) = hi;
                        *reinterpret_cast<uint4*>(dst + kv_term) = lo;
                    }
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(v_ready + (j & 1));
            if (j + 1 < tiles) fetch_v(j + 1);
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    } else {
        // ================= softmax and output: thread = query row; warps w and w + 4 share rows =================
        const int quad = warp & 3, half = warp >> 2, r = 32 * quad + lane;
        const int tok = tok0 + r % TQ, head = hg * GQ + r / TQ;
        const int pos = min(p.pos0 + tok, last);
        const uint32_t lanes = tmem + ((uint32_t)(32 * quad) << 16);
        const float fac = q_inv * (1.4426950408889634f * __frsqrt_rn((float)hs));
        const int dims = hs >> 1;
        float o[PA_MAX_HS / 2];
#pragma unroll
        for (int i = 0; i < PA_MAX_HS / 2; ++i) o[i] = 0.f;
        float m = -INFINITY, l = 0.f, alpha_prev = 0.f, vfac_prev = 0.f;
        auto add_output = [&]() {  // o = o * alpha + the tile's product
#pragma unroll
            for (int c0 = 0; c0 < PA_MAX_HS / 2; c0 += 16) {
                if (c0 >= dims) break;
                float v[16];
                tmem_ld16f(lanes + 256u + (uint32_t)(dims * half + c0), v);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c0 + i] = fmaf(o[c0 + i], alpha_prev, v[i] * vfac_prev);
                tmem_ld16f(lanes + 384u + (uint32_t)(dims * half + c0), v);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c0 + i] = fmaf(v[i], vfac_prev, o[c0 + i]);
            }
        };
        for (int j = 0; j < tiles; ++j) {
            // (both halves' warps meet at the barrier below, so a wait that runs out is carried along and not left by)
            if (ok && !mbar_wait_warp(s_full + (j & 1), (uint32_t)((j >> 1) & 1))) ok = false;
            float s[32];
            if (ok) {
                tc_fence_after();
                tmem_ld32f(lanes + (uint32_t)(32 * half), s);
#pragma unroll 1
                for (int i0 = per; i0 < ns; i0 += per) {
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        float s2[16];
                        tmem_ld16f(lanes + (uint32_t)(i0 / per * 64 + 32 * half + c), s2);
#pragma unroll
                        for (int i = 0; i < 16; ++i) s[c + i] += s2[i];
                    }
                }
                tc_fence_before();
            }
            const PaScales& scales = s_scale[j & 3];
            const float4* const key_inv = reinterpret_cast<const float4*>(scales.key + 32 * half);
            const float4* const value_exp = reinterpret_cast<const float4*>(scales.value_exp + 32 * half);
            const int left = pos - (j * PA_KEYS + 32 * half);  // positions 0 .. left of this half are seen
            float mx = -INFINITY, tx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 f = key_inv[i / 4], e = value_exp[i / 4];
                const float f4[4] = {f.x, f.y, f.z, f.w}, e4[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[i + k] = i + k <= left ? s[i + k] * (fac * f4[k]) : -INFINITY;
                    mx = fmaxf(mx, s[i + k]);
                    tx = fmaxf(tx, s[i + k] + e4[k]);
                }
            }
            float2* mrow = s_max + (j & 1) * 256;
            mrow[half * 128 + r] = make_float2(mx, tx);
            pa_bar_sync(1, 256);
            const float2 other = mrow[(half ^ 1) * 128 + r];
            const float mn = fmaxf(m, fmaxf(mx, other.x));
            const float alpha = exp2f(m - mn);
            m = mn;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                s[i] = exp2f(s[i] - mn);
                sum += s[i];
            }
            l = fmaf(l, alpha, sum);
            // weights take the scales of their values along; a power of two per row brings the largest of them to 2^12 .. 2^13
            const int ie = (int)fminf(fmaxf(ceilf(fmaxf(tx, other.y) - mn), -100.f), 126.f);
            const float w_scale = __uint_as_float((uint32_t)(140 - ie) << 23);
            if (ok && j > 0 && !mbar_wait_warp(pv_full + ((j - 1) & 1), (uint32_t)(((j - 1) >> 1) & 1))) ok = false;
            if (ok) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4* const value_inv = reinterpret_cast<const float4*>(scales.value + 32 * half + 8 * c);
                    const float4 f0 = value_inv[0], f1 = value_inv[1];
                    const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
                    float w[8], fs[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = s[8 * c + i], fs[i] = fminf(f[i] * w_scale, 1.329228e36f);  // (2^120: times a weight of 0)
                    uint4 hi, lo;
                    pa_terms(w, fs, hi, lo);
                    uint8_t* dst = smem + L.off_p + (4 * half + c) * (PA_ROWS * 16) + r * 16;
                    *reinterpret_cast<uint4*>(dst) = hi;
                    *reinterpret_cast<uint4*>(dst + p_term) = lo;
                }
                fence_proxy_async();
            }
            if (ok && j > 0) {
                tc_fence_after();
                add_output();
                tc_fence_before();
            }
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(p_ready);
            alpha_prev = alpha;
            vfac_prev = __uint_as_float((uint32_t)(114 + ie) << 23);
        }
        if (ok && !mbar_wait_warp(pv_full + ((tiles - 1) & 1), (uint32_t)(((tiles - 1) >> 1) & 1))) ok = false;
        if (ok) {
            tc_fence_after();
            add_output();
        }
        if (*odd_values) {  // (weights are positive: an infinity or NaN comes out as it would with its weight)
            const float* v = p.vc + (size_t)kvh * p.seq_len * hs + dims * half;
#pragma unroll 1
            for (int i = 0; i <= pos; ++i, v += hs)
#pragma unroll
                for (int d = 0; d < PA_MAX_HS / 2; ++d)
                    if (d < dims) {
                        const float x = __ldcg(v + d);
                        if (!(fabsf(x) < INFINITY)) o[d] += x;
                    }
        }
        s_sum[half * 128 + r] = l;
        pa_bar_sync(1, 256);
        if (ok && tok < p.n) {
            const float inv = __frcp_rn(s_sum[r] + s_sum[128 + r]);
            float4* dst = reinterpret_cast<float4*>(p.out + (size_t)tok * p.q_stride + (size_t)head * hs + dims * half);
#pragma unroll
            for (int i = 0; i < PA_MAX_HS / 8; ++i)
                if (4 * i < dims) dst[i] = make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    }
    pdl_launch_dependents();
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 512);
}

}  // namespace l2b
