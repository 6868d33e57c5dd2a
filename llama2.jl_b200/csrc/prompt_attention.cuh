// Softmax attention of a prompt pass (many queries of one sequence) on the tensor cores: attention_weights!, the division by
// sqrt(head_size), softmax! and combine_values! (src/inference.jl:263-278, 169-220) for every token of the pass at once.
//
// Block = 128 query rows (128 / GQ tokens x the GQ heads that share a key / value head), walking the cached positions 64 at a
// time.  Queries, keys, values and softmax weights are f32 and enter the tensor cores as two fp16 terms each, scaled by a power
// of two (a query row; a tile of keys or values; weights by 2^13), so that a product is high*high + high*low + low*high: what is
// left out is 2^-24 of it.  The tensor core rounds its sums toward zero, so they are kept short (half a head size, or 64 positions)
// and continued in f32 registers; maxima, exponentials and their sums are f32.
//
//   6 conversion warps  keys (thread = position, 8 dims) and values (thread = dim, 8 positions) from the caches to operand layout
//                       (core matrices of 8 rows x 16 bytes); the next tile's values are fetched while this one is waited for
//   MMA warp            S(j) = Q K^T, O(j) = P V; S(j + 1) is issued before O(j)
//   8 softmax warps     thread = query row, half of the positions, half of the output
//
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

struct PaSmem {
    int off_bar, off_max, off_sum, off_scale, off_conv, off_q, off_k, off_v, off_p, total;
};
__host__ __device__ inline PaSmem pa_smem_layout(int hs) {
    PaSmem s;
    s.off_bar = 0;       // k_ready p_ready s_full[2] v_ready[2] pv_full[2]; tensor memory address behind them
    s.off_max = 128;     // [2][2][128] row maxima of the two halves, by tile parity
    s.off_sum = s.off_max + 2048;    // [2][128]
    s.off_scale = s.off_sum + 1024;  // [4] {keys, values}
    s.off_conv = s.off_scale + 64;   // [2][8] {keys, values} maxima of the conversion warps
    s.off_q = (s.off_conv + 128 + 1023) & ~1023;
    s.off_k = s.off_q + 2 * PA_ROWS * hs * 2;  // [term][hs / 8][rows][16 bytes]
    s.off_v = s.off_k + 2 * PA_KEYS * hs * 2;
    s.off_p = s.off_v + 2 * 2 * PA_KEYS * hs * 2;  // two slots of values
    s.total = s.off_p + 2 * PA_ROWS * PA_KEYS * 2;
    return s;
}

__device__ __forceinline__ void pa_bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Power of two that brings a largest value of mx into [2^13, 2^14), and its inverse.
__device__ __forceinline__ float pa_scale(float mx, float& inv) {
    const int ex = (int)(__float_as_uint(mx) >> 23) & 255;
    const int up = ex == 0 || ex == 255 ? 127 : min(267 - ex, 252);
    inv = __uint_as_float((uint32_t)(254 - up) << 23);
    return __uint_as_float((uint32_t)up << 23);
}
// Eight values as two fp16 terms: 16 bytes each.
__device__ __forceinline__ void pa_terms(const float (&v)[8], float s, uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = v[2 * i] * s, b = v[2 * i + 1] * s;
        const __half2 x = __floats2half2_rn(a, b);
        const float2 y = __half22float2(x);
        h[i] = h2_raw(x);
        l[i] = h2_raw(__floats2half2_rn(a - y.x, b - y.y));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
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
    float* s_max = reinterpret_cast<float*>(smem + L.off_max);
    float* s_sum = reinterpret_cast<float*>(smem + L.off_sum);
    float2* s_scale = reinterpret_cast<float2*>(smem + L.off_scale);
    float2* s_conv = reinterpret_cast<float2*>(smem + L.off_conv);
    constexpr int TQ = PA_ROWS / GQ;  // tokens per block
    const int tok0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TQ;  // blocks with the most positions first
    const int hg = blockIdx.y, kvh = hg * GQ / (p.n_heads / p.n_kv);
    const int last = p.pos0 + min(p.n, tok0 + TQ) - 1;  // last position that a row of this block attends to
    const int tiles = last / PA_KEYS + 1;
    const int q_term = PA_ROWS * hs * 2, kv_term = PA_KEYS * hs * 2, p_term = PA_ROWS * PA_KEYS * 2;

    if (threadIdx.x == 0) {
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
        s_max[half * 128 + r] = mx;
        pa_bar_sync(1, 256);
        const float s = pa_scale(fmaxf(mx, s_max[(half ^ 1) * 128 + r]), q_inv);
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
    // tensor memory: S in slots of 128 columns (two sums of 64 positions), O in slots of 128 columns behind them
    bool ok = true;

    if (warp == 8) {
        // ================= MMA issue =================
        const uint32_t idesc_s = umma_idesc_f16(PA_ROWS, PA_KEYS), idesc_o = umma_idesc_f16(PA_ROWS, hs);
        const uint64_t dq = umma_desc(smem + L.off_q, PA_ROWS * 16, 128), dk = umma_desc(smem + L.off_k, PA_KEYS * 16, 128);
        const uint64_t dv = umma_desc(smem + L.off_v, hs * 16, 128), dp = umma_desc(smem + L.off_p, PA_ROWS * 16, 128);
        const uint32_t q_lo = q_term >> 4, kv_lo = kv_term >> 4, p_lo = p_term >> 4;
        const int split = (ns + 1) >> 1;  // steps of the first sum
        auto scores = [&](int j) {
            if (!mbar_wait_parked(k_ready, (uint32_t)(j & 1))) return false;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int i0 = half ? split : 0, i1 = half ? ns : split;
                    const uint32_t d = tmem + (uint32_t)((j & 1) * 128 + half * 64);
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
            if (j + 1 < tiles && !scores(j + 1)) {
                ok = false;
                break;
            }
            if (!mbar_wait_parked(p_ready, (uint32_t)(j & 1)) || !mbar_wait_parked(v_ready + (j & 1), (uint32_t)((j >> 1) & 1))) {
                ok = false;
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t d = tmem + 256u + (uint32_t)((j & 1) * 128);
                const uint64_t v = dv + (uint64_t)((j & 1) * (2 * kv_term >> 4));
                uint32_t acc = 0;
#pragma unroll 1
                for (int t = 0; t < 3; ++t) {
                    const uint64_t a = dp + (t == 0 ? p_lo : 0u), b = v + (t == 1 ? kv_lo : 0u);
#pragma unroll
                    for (int i = 0; i < PA_KEYS / 16; ++i) {
                        umma_f16(d, a + (uint64_t)(i * (2 * PA_ROWS)), b + (uint64_t)(i * 2 * hs), idesc_o, acc);
                        acc = 1;
                    }
                }
                umma_commit(pv_full + (j & 1));
            }
            __syncwarp();
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
        int v_off[ITEMS], v_pos[ITEMS];  // of this thread's values: dim, first of eight positions
#pragma unroll
        for (int u = 0; u < ITEMS; ++u) {
            const int idx = id + CT * u;
            v_pos[u] = idx / hs * 8;
            v_off[u] = idx % hs + v_pos[u] * hs;
        }
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
                const float* src = vbase + (size_t)j * PA_KEYS * hs + v_off[u];
#pragma unroll
                for (int k = 0; k < 8; ++k) vv[u][k] = k <= left ? __ldcg(src + k * hs) : 0.f;
            }
        };
        fetch_k(0);
        fetch_v(0);
        for (int j = 0; j < tiles; ++j) {
            float mk = 0.f, mv = 0.f;
#pragma unroll
            for (int u = 0; u < ITEMS; ++u)
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    mk = fmaxf(mk, fabsf(kv[u][k]));
                    mv = fmaxf(mv, fabsf(vv[u][k]));
                }
            mk = warp_max(mk);
            mv = warp_max(mv);
            if (lane == 0) s_conv[(j & 1) * 8 + warp - 9] = make_float2(mk, mv);
            pa_bar_sync(2, CT);
#pragma unroll
            for (int i = 0; i < PA_CONV_WARPS; ++i) {
                const float2 m = s_conv[(j & 1) * 8 + i];
                mk = fmaxf(mk, m.x);
                mv = fmaxf(mv, m.y);
            }
            float k_inv, v_inv;
            const float ks = pa_scale(mk, k_inv), vs = pa_scale(mv, v_inv);
            if (ok && j > 0 && !mbar_wait_parked(s_full + ((j - 1) & 1), (uint32_t)(((j - 1) >> 1) & 1))) ok = false;  // the last scores have read the keys
            if (ok) {
                if (id == 0) s_scale[j & 3] = make_float2(k_inv, v_inv);
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
            if (ok && j > 1 && !mbar_wait_parked(pv_full + (j & 1), (uint32_t)(((j - 2) >> 1) & 1))) ok = false;
            if (ok) {
#pragma unroll
                for (int u = 0; u < ITEMS; ++u) {
                    const int idx = id + CT * u;
                    if (idx < items) {
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
        auto add_output = [&](int j) {  // o = o * alpha + the tile's product
#pragma unroll
            for (int c0 = 0; c0 < PA_MAX_HS / 2; c0 += 16) {
                if (c0 >= dims) break;
                float v[16];
                tmem_ld16f(lanes + 256u + (uint32_t)((j & 1) * 128 + dims * half + c0), v);
#pragma unroll
                for (int i = 0; i < 16; ++i) o[c0 + i] = fmaf(o[c0 + i], alpha_prev, v[i] * vfac_prev);
            }
        };
        for (int j = 0; j < tiles; ++j) {
            // (both halves' warps meet at the barrier below, so a wait that runs out is carried along and not left by)
            if (ok && !mbar_wait_parked(s_full + (j & 1), (uint32_t)((j >> 1) & 1))) ok = false;
            float s[32];
            if (ok) {
                tc_fence_after();
                tmem_ld32f(lanes + (uint32_t)((j & 1) * 128 + 32 * half), s);
                if (ns > 1) {
                    float s2[16];
#pragma unroll
                    for (int c = 0; c < 32; c += 16) {
                        tmem_ld16f(lanes + (uint32_t)((j & 1) * 128 + 64 + 32 * half + c), s2);
#pragma unroll
                        for (int i = 0; i < 16; ++i) s[c + i] += s2[i];
                    }
                }
                tc_fence_before();
            }
            const float2 sc = s_scale[j & 3];
            const float f = fac * sc.x;
            const int left = pos - (j * PA_KEYS + 32 * half);  // positions 0 .. left of this half are seen
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                s[i] = i <= left ? s[i] * f : -INFINITY;
                mx = fmaxf(mx, s[i]);
            }
            float* mrow = s_max + (j & 1) * 256;
            mrow[half * 128 + r] = mx;
            pa_bar_sync(1, 256);
            const float mn = fmaxf(m, fmaxf(mx, mrow[(half ^ 1) * 128 + r]));
            const float alpha = exp2f(m - mn);
            m = mn;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                s[i] = exp2f(s[i] - mn);
                sum += s[i];
            }
            l = fmaf(l, alpha, sum);
            if (ok && j > 0 && !mbar_wait_parked(pv_full + ((j - 1) & 1), (uint32_t)(((j - 1) >> 1) & 1))) ok = false;
            if (ok) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[i] = s[8 * c + i];
                    uint4 hi, lo;
                    pa_terms(w, 8192.f, hi, lo);
                    uint8_t* dst = smem + L.off_p + (4 * half + c) * (PA_ROWS * 16) + r * 16;
                    *reinterpret_cast<uint4*>(dst) = hi;
                    *reinterpret_cast<uint4*>(dst + p_term) = lo;
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(p_ready);
            if (ok && j > 0) {
                tc_fence_after();
                add_output(j - 1);
                tc_fence_before();
            }
            alpha_prev = alpha;
            vfac_prev = sc.y * 1.220703125e-4f;  // 2^-13
        }
        if (ok && !mbar_wait_parked(pv_full + ((tiles - 1) & 1), (uint32_t)(((tiles - 1) >> 1) & 1))) ok = false;
        if (ok) {
            tc_fence_after();
            add_output(tiles - 1);
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
    tc_fence_before();
    __syncthreads();
    if (warp == 8) tmem_dealloc(tmem, 512);
}

}  // namespace l2b
