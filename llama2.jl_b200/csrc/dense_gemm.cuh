// Matrix products of many-token passes of layer-stack models: bf16 weights x n activation vectors.
//   bf16_gemm_kernel  bf16 activations on the 5th-generation tensor cores (tcgen05 + TMA + tensor memory);
//   f32_gemm_kernel   f32 activations on the CUDA cores in f32 (the 32-bit mode: bf16 weights are exact in f32).
//
// bf16_gemm_kernel: a pair of blocks (a cluster) works on 256 weight rows x N tokens with tcgen05.mma of cta_group::2; each block brings its
// own 128 rows and half of the tokens, and holds the results of its rows.  Weight rows are the M dimension: a thread of the epilogue owns
// one row, and consecutive lanes store consecutive results of a token.  What bounds a large product is the way from L2 to the SMs (about 48
// bytes per cycle and SM): alone, an SM would read 384 rows of operands for 128 x 256 results, in a pair it reads 256.
//   1000 tokens x 28672 rows (gate and up) x 4096: 240 -> 169 us (1390 TFLOP/s), 4096 x 14336: 143 -> 91 us, against a kernel of single SMs
//   with tiles of 256 x 128; prompts of 3 .. 1500 tokens 1.04 - 1.29 times as fast.
// Persistent: a pair walks tiles (token tiles innermost, so that a weight tile is read from L2 after its first use), with two sets of N
// accumulator columns in tensor memory, so that a tile's epilogue runs beside the next tile's products.
// Two weight matrices (gate and up): a block's 128 rows are 64 of each, and the threads of a pair of rows exchange half of their tokens
// through shared memory.
//   warp 0     producer (each block for itself): TMA tiled copies, 128 values of K per stage as two tiles of 64 (128-byte swizzle)
//   warp 1     MMA issue (of the pair's first block): eight K = 16 steps per stage
//   warps 2-9  epilogue: every other 32 tokens, tcgen05.ld, then what follows the product
// Every mbarrier wait is bounded; a wait that runs out sets the status word, and both blocks still free their tensor memory.
#pragma once
#include "dense_ops.cuh"
#include "tcgen05.cuh"

namespace l2b {

constexpr int BG_KB = 128, BG_MAX_STAGES = 6, BG_EPI_WARPS = 8, BG_THREADS = (2 + BG_EPI_WARPS) * 32;
constexpr int BG_SWAP_BYTES = 2 * 2 * 16 * 64 * 4;  // [group of epilogue warps][direction][16 tokens][64 rows]

struct GemmDenseParams {
    int rows;   // results per token
    int n_tok, k;
    int N;      // tokens per tile, a multiple of 32
    int mtiles, ntiles, stages;
    DenseEpilogue epi;
    int* status;
};
__host__ __device__ constexpr int bg_stage_bytes(int N) { return (128 + N / 2) * BG_KB * 2; }

// ---- pairs of blocks ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrives on the barrier at this place in both blocks of the pair when the products issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// A tiled copy into this block's shared memory, counted by a barrier of either block of the pair (its cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(bar_addr)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_addr) : "memory");
}

// 32 consecutive tokens (n of them exist) of one result row (products of one matrix).  What has to be read is read for all of them first.
template <int KIND>
__device__ __forceinline__ void epilogue_tokens(const DenseEpilogue& e, int t0, int n, int f, const float (&v)[32]) {
    bf16* const act = static_cast<bf16*>(e.act);
    if (KIND == DE_RESIDUAL) {
        float r[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) r[k] = e.y[(size_t)(t0 + min(k, n - 1)) * e.ld + f];
#pragma unroll
        for (int k = 0; k < 32; ++k)
            if (k < n) e.y[(size_t)(t0 + k) * e.ld + f] = r[k] + v[k];
    } else if (KIND == DE_SIDE) {
        float r[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) r[k] = side_value(e, t0 + min(k, n - 1), f);
#pragma unroll
        for (int k = 0; k < 32; ++k)
            if (k < n) put(act + (size_t)(t0 + k) * e.ld + f, gelu_tanh(v[k]) * r[k]);
    } else if (KIND == DE_STORE_T && n == 32 && (e.ld & 7) == 0) {  // a thread's 32 tokens are contiguous
        uint4* dst = reinterpret_cast<uint4*>(act + (size_t)f * e.ld + t0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 pk = __floats2bfloat162_rn(v[8 * k + 2 * i], v[8 * k + 2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&pk);
            }
            dst[k] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
        const float bias = KIND == DE_AFFINE && e.bias ? __ldg(e.bias + f) : 0.f;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            if (k >= n) continue;
            if (KIND == DE_STORE) e.y[(size_t)(t0 + k) * e.ld + f] = v[k];
            if (KIND == DE_AFFINE) e.y[(size_t)(t0 + k) * e.ld + f] = fmaf(v[k], e.mul, bias);
            if (KIND == DE_STORE_ACT) put(act + (size_t)(t0 + k) * e.ld + f, v[k]);
            if (KIND == DE_STORE_T) put(act + (size_t)f * e.ld + t0 + k, v[k]);
        }
    }
}
__device__ __forceinline__ void epilogue_tokens(const DenseEpilogue& e, int t0, int n, int f, const float (&v)[32]) {
    switch (e.kind) {
        case DE_RESIDUAL: epilogue_tokens<DE_RESIDUAL>(e, t0, n, f, v); break;
        case DE_AFFINE: epilogue_tokens<DE_AFFINE>(e, t0, n, f, v); break;
        case DE_SIDE: epilogue_tokens<DE_SIDE>(e, t0, n, f, v); break;
        case DE_STORE_ACT: epilogue_tokens<DE_STORE_ACT>(e, t0, n, f, v); break;
        case DE_STORE_T: epilogue_tokens<DE_STORE_T>(e, t0, n, f, v); break;
        default: epilogue_tokens<DE_STORE>(e, t0, n, f, v); break;
    }
}

template <bool DUAL>
__global__ void __launch_bounds__(BG_THREADS, 1) bf16_gemm_kernel(const __grid_constant__ GemmDenseParams p, const __grid_constant__ CUtensorMap map_a,
                                                                       const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_b) {
    extern __shared__ __align__(1024) uint8_t bg_raw[];
    __shared__ __align__(8) uint64_t s_full[BG_MAX_STAGES], s_free[BG_MAX_STAGES], s_acc[2], s_acc_free[2];
    __shared__ uint32_t s_tmem;
    uint8_t* smem = bg_raw + ((1024u - (smem_u32(bg_raw) & 1023u)) & 1023u);
    const int stage = bg_stage_bytes(p.N), off_b = 128 * BG_KB * 2, sub_b = p.N / 2 * 128;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_rank();
    const int tile_rows = DUAL ? 128 : 256;
    const int nk = (p.k + BG_KB - 1) / BG_KB, tiles = p.mtiles * p.ntiles, pairs = (int)gridDim.x >> 1, first = (int)blockIdx.x >> 1;
    if (threadIdx.x == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(s_full + i, 1);  // of the first block: operands of both blocks
            mbar_init(s_free + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(s_acc + i, 1);
            mbar_init(s_acc_free + i, 2 * BG_EPI_WARPS);  // of the first block: both blocks' epilogues
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc_pair(&s_tmem, 512);
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int s = 0;
            uint32_t parity = 1;
            bool again = false;
            for (int tile = first; tile < tiles && ok; tile += pairs) {
                const int row0 = tile / p.ntiles * tile_rows + rank * (tile_rows / 2), tok0 = tile % p.ntiles * p.N + rank * (p.N / 2);
                for (int j = 0; j < nk; ++j) {
                    if (again && !mbar_wait_bounded(s_free + s, parity)) {
                        ok = false;
                        break;
                    }
                    uint8_t* st = smem + (size_t)s * stage;
                    if (rank == 0) mbar_arrive_expect_tx(s_full + s, (uint32_t)(2 * stage));
                    const uint32_t bar = cluster_map(s_full + s, 0);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int x = j * BG_KB + 64 * h;
                        if (DUAL) {
                            tma_load_2d_pair(st + h * 16384, &map_a, x, row0, bar);
                            tma_load_2d_pair(st + h * 16384 + 8192, &map_a2, x, row0, bar);
                        } else {
                            tma_load_2d_pair(st + h * 16384, &map_a, x, row0, bar);
                        }
                        tma_load_2d_pair(st + off_b + h * sub_b, &map_b, x, tok0, bar);
                    }
                    if (++s == p.stages) {
                        s = 0;
                        again = true;
                        parity ^= 1u;
                    }
                }
            }
            if (!ok) {
                atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
                for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // copies in flight land within microseconds
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(256, p.N);
            // descriptors of stage 0; the others lie a multiple of 16 bytes further
            const uint64_t da0 = umma_desc_sw128(smem, 0), db0 = umma_desc_sw128(smem + off_b, 0);
            bool ok = true;
            int s = 0, n = 0;
            uint32_t par = 0;
            for (int tile = first; tile < tiles && ok; tile += pairs, ++n) {
                const int buf = n & 1;
                if (n >= 2 && !mbar_wait_bounded(s_acc_free + buf, (uint32_t)(((n - 2) >> 1) & 1))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(buf * 256);
                uint32_t acc = 0;
                for (int j = 0; j < nk; ++j) {
                    if (!mbar_wait_bounded(s_full + s, par)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = da0 + (uint64_t)((s * stage) >> 4), db = db0 + (uint64_t)((s * stage) >> 4);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            umma_bf16_pair(d, da + (uint64_t)((h * 16384 + kk * 32) >> 4), db + (uint64_t)((h * sub_b + kk * 32) >> 4), idesc, acc);
                            acc = 1;
                        }
                    umma_commit_pair(s_free + s);
                    if (++s == p.stages) s = 0, par ^= 1u;
                }
                if (ok) umma_commit_pair(s_acc + buf);
            }
            if (!ok) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
        }
    } else {
        const int qd = warp & 3, group = (warp - 2) >> 2;
        const int r = 32 * qd + lane;
        float* swap = reinterpret_cast<float*>(smem + (size_t)p.stages * stage) + group * (2 * 16 * 64);
        bf16* const act = static_cast<bf16*>(p.epi.act);
        int n = 0;
        bool ok = true;
        for (int tile = first; tile < tiles; tile += pairs, ++n) {
            const int buf = n & 1, tok0 = tile % p.ntiles * p.N;
            const int f = DUAL ? tile / p.ntiles * 128 + rank * 64 + (r & 63) : tile / p.ntiles * 256 + rank * 128 + r;
            // (the warps of a group meet at the barriers below, so a wait that runs out is carried along and not left by; nothing is stored then)
            if (ok && !__all_sync(0xffffffffu, mbar_wait_bounded(s_acc + buf, (uint32_t)((n >> 1) & 1)))) ok = false;
            tc_fence_after();
            const uint32_t ta = tmem + ((uint32_t)(32 * qd) << 16) + (uint32_t)(buf * 256);
#pragma unroll 1
            for (int c = 32 * group; c < p.N; c += 64) {
                const int left = min(32, p.n_tok - tok0 - c);
                if (left <= 0) break;
                __syncwarp();
                float v[32];
                tmem_ld32f(ta + (uint32_t)c, v);
                if (DUAL) {
                    const bool is_up = r >= 64;
                    const int row = r & 63;
                    // gate threads finish tokens 0-15 of the 32, up threads the others
                    float* const to = swap + (is_up ? 0 : 16 * 64) + row;
                    const float* const from = swap + (is_up ? 16 * 64 : 0) + row;
#pragma unroll
                    for (int k = 0; k < 16; ++k) to[64 * k] = is_up ? v[k] : v[16 + k];
                    asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory");
                    const int t0 = tok0 + c + (is_up ? 16 : 0), mine = left - (is_up ? 16 : 0);
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const float other = from[64 * k], own = is_up ? v[16 + k] : v[k];
                        const float g = is_up ? other : own, u = is_up ? own : other;
                        if (ok && k < mine && f < p.rows) put(act + (size_t)(t0 + k) * p.epi.ld + f, (p.epi.kind == DE_SWIGLU ? silu(g) : gelu_tanh(g)) * u);
                    }
                    asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory");
                } else if (ok && f < p.rows) {
                    epilogue_tokens(p.epi, tok0 + c, left, f, v);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mbar_arrive_cluster(cluster_map(s_acc_free + buf, 0));
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    }
    // every path ends here, in both blocks: no products, arrivals or copies of the other one are under way when this one leaves
    __syncwarp();
    pdl_launch_dependents();  // (a block's first warp here releases the next kernel: the second block's warp 1 at once, the first one's producer behind its last copy)
    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

// ---- f32 --------------------------------------------------------------------------------------------
// One block = 64 weight rows x 64 tokens, thread = 4 x 4 results; DUAL: two weight rows per result (rows f and f of the second
// matrix).  x [n_tok][ldx] f32, w rows wstride elements apart.
struct GemmF32Params {
    const bf16* w;
    const bf16* w2;
    size_t wstride;
    const float* x;
    int ldx;
    int rows, n_tok, k;
    DenseEpilogue epi;
};
template <bool DUAL>
__global__ void __launch_bounds__(256) f32_gemm_kernel(const __grid_constant__ GemmF32Params p) {
    constexpr int T = 64, KB = 16;
    __shared__ float sw[DUAL ? 2 : 1][KB][T + 4], sx[KB][T + 4];
    const int tid = threadIdx.x, fr = tid & 15, tr = tid >> 4;
    const int f0 = (int)blockIdx.x * T, n0 = (int)blockIdx.y * T;
    float acc[4][4], acc2[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = acc2[i][j] = 0.f;
    for (int k0 = 0; k0 < p.k; k0 += KB) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = tid + u * 256, k = i & 15, r = i >> 4;
            const bool kin = k0 + k < p.k;
            sw[0][k][r] = kin && f0 + r < p.rows ? __bfloat162float(p.w[(size_t)(f0 + r) * p.wstride + k0 + k]) : 0.f;
            if (DUAL) sw[DUAL ? 1 : 0][k][r] = kin && f0 + r < p.rows ? __bfloat162float(p.w2[(size_t)(f0 + r) * p.wstride + k0 + k]) : 0.f;
            sx[k][r] = kin && n0 + r < p.n_tok ? p.x[(size_t)(n0 + r) * p.ldx + k0 + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            float w[4], w2[4], x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                w[i] = sw[0][k][fr + 16 * i];
                w2[i] = DUAL ? sw[DUAL ? 1 : 0][k][fr + 16 * i] : 0.f;
                x[i] = sx[k][tr + 16 * i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] = fmaf(w[i], x[j], acc[i][j]);
                    if (DUAL) acc2[i][j] = fmaf(w2[i], x[j], acc2[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int f = f0 + fr + 16 * i, t = n0 + tr + 16 * j;
            if (f < p.rows && t < p.n_tok) dense_epilogue<float>(p.epi, t, f, acc[i][j], acc2[i][j]);
        }
}

}  // namespace l2b
