// k-quant weights x many activation vectors on the 5th-generation tensor cores (tcgen05): the dense GEMM that prompt
// prefill, batched decode and matmul! over several columns need.  The reference feeds a prompt one token at a time through
// matmul! (src/matmul.jl:13-23, src/inference.jl:349-356); here up to 128 tokens share one pass over the weights.
//
//   Y[t][o] = sum_b ( d_ob * sum_k A_obk * X_tbk  +  sum_j C_obj * xs_tbj )
//
// b: 256-value super-blocks of a row, j: sub-blocks of 32, xs_tbj: sum of the sub-block's activations.
//   A = sub-block scale times (quant - centre), centre 8 (q4_K), 16 (q5_K), 32 (q6_K): an integer of at most 11 bits, exact in
//       fp16 (q6_K: 12 bits, so its scale is cut into an even part and the last bit, two passes).
//   X = the activations, scaled per token by a power of two, as two fp16 terms (high, low): 24 significant bits, as many as
//       f32 has.  Products are exact in f32; sums run over 64 values inside the tensor core, which rounds toward zero, and from
//       there in f32 registers: with sums over 256 values the rounding of the tensor core is what the error consists of.
//   C = centre * d * scale - dmin * min, the part of the weight that a sub-block's values share, as two fp16 terms.
//
// Work is counted in super-blocks of 128 weight rows: chunk c holds units c*U .. c*U + U - 1 of the list (row tile, super-block),
// whatever tile they belong to, so that every SM has the same share; a block takes a chunk for up to 128 tokens at a time.  A row tile
// that lies in several chunks leaves one partial result per chunk in a buffer of its own (no atomics: the sum's order is fixed); the
// kernel that reads the product anyway (norm, SwiGLU, RoPE) adds them.  The cuts come from the matrices alone, never from the number of
// tokens: buffers grow with the tokens and nothing else.
//
//   packed-copy warp  one TMA tiled copy (cp.async.bulk.tensor) per super-block: a 128-row box of the stored blocks
//   2 operand warps   one bulk copy per 64 values: the tokens' two terms, already in operand layout (split_rows_kernel); a thread takes 750
//                     cycles to see a slot free and issue a copy, so two take turns
//   unpack warps      groups of four; thread = row: nibbles -> fp16 times scale, into tensor memory (lane = row) or, for tiles of 33 - 64
//                     tokens, into core matrices (8 rows x 16 bytes)
//   MMA warp          tcgen05.mma.kind::f16 (M 128, K 16), four or eight per 64 values
//   8 epilogue warps  thread = weight row, half of the tokens: tensor memory -> times d -> f32 accumulators, and those of four
//                     super-blocks -> f32 sums in tensor memory (one chain over 14336 values would be 280 roundings long)
//
// Every mbarrier wait is bounded; a wait that runs out sets the status word, after which the block drains and still frees
// its tensor memory.
#pragma once
#include <cuda_fp16.h>

#include "fused_matvec.cuh"
#include "tcgen05.cuh"

namespace l2b {

constexpr int GM_ROWS = 128;          // weight rows per tile = MMA M
constexpr int GM_MAX_TOK = 128;       // tokens per tile
constexpr int GM_GROUP_BYTES = 2048;  // operand of 8 tokens x 64 values: [term][k / 16][half][8 rows][16 bytes]
constexpr int GM_XS_BYTES = 256;      // sub-block sums of 8 tokens x one super-block: [term][8 rows][8 sub-blocks] fp16
constexpr int GM_A_BYTES = GM_ROWS * 64 * 2;
constexpr int GM_MAX_SEG = 3;         // matrices of one launch
constexpr int GM_HDRS = 4;
constexpr int GM_EPI_WARPS = 8;

// How a product's tiles are shared out; the kernels that read the partial results derive their number from it.
struct GemmSplit {
    int U;        // units (super-blocks of a row tile) per chunk
    int nb;       // units per row tile
    int ntile;    // token tiles
    int tok;      // tokens per tile (a multiple of 16)
};
// Parts that the results of this row are in.
__host__ __device__ inline int gm_parts(const GemmSplit& s, int row) {
    const unsigned lo = (unsigned)(row / GM_ROWS) * s.nb;
    return (int)((lo + s.nb - 1) / s.U - lo / s.U) + 1;
}

struct GemmSeg {
    int type, rows, row_tiles;
    int kb;               // super-blocks per stored column panel (nb when the matrix is not stored as panels)
    const __half* d6;     // q6_K: block scales [row][nb]
};
struct GemmParams {
    GemmSeg seg[GM_MAX_SEG];
    int nseg;
    GemmSplit sp;
    int total, chunks;    // units; chunks of sp.U of them
    int n_tok, groups;    // tokens; groups of 8 in the operand buffers
    int np;               // slots for packed super-blocks
    const uint8_t* act;   // [nb][4][groups] x GM_GROUP_BYTES
    const uint8_t* xs;    // [nb][groups] x GM_XS_BYTES
    const float* scale;   // [groups * 8] factor of a token's results
    float* y;             // [part][n_tok][ldy]; the segments' rows follow one another, each starting at a multiple of 128
    size_t part_stride;
    int ldy;
    int* status;
};
struct GemmMaps {
    CUtensorMap main[GM_MAX_SEG], tail[GM_MAX_SEG];  // [panels][rows][kb * block bytes]; tail: the last, narrower panel
};

// ---- shared memory -----------------------------------------------------------------------------
// NT tokens at most per tile.
// CH chunks of 64 values per step.  What a step costs beyond its MMAs is hand-overs: the MMA warp, the operand warps and the epilogue each spend
// about 600 cycles per step whatever it holds.  With 128 tokens a chunk's MMAs take 512 cycles and tensor memory holds the sums of no
// more, so a step is one chunk (and the shared part C a step of its own); with fewer a step is two chunks, each with a sum of its own, and
// the second step of a super-block takes the shared part along.
// NS slots for operands, ND for accumulators; as many slots for packed super-blocks as fit (2 .. 5).
// UG groups of four unpack warps, GS of them on a step (with 64 tokens, two: a chunk each), UG / GS steps in turn.  A group waits for the slot's
// last use by parity, so it must have seen the use before that: its own last step lies at most NS steps back, UG / GS <= NS.  (More groups
// are no help: all read the scales of every super-block they take part in, 200 instructions a row, which with four groups on the steps
// of one super-block made the kernel issue-bound.)
// AT: with 128 tokens the products read 64 KB of shared memory per 64 values when the weights come from there too (each of the two terms
// reads them again), as much as an SM delivers while they run, and copies and unpacking want another 57 KB.  From tensor memory the weights cost
// nothing of it, and there is room for four slots of activations: 1240 -> 930 cycles per step (q4_K 28672 x 4096 times 128).  That leaves two
// sets of accumulators instead of three.  (Blocks in pairs that share the activations, cta_group::2: 1270 - 1350 cycles; 16 epilogue warps: no
// faster.)  With 32 tokens an MMA takes 46 cycles instead of 16 for the weights' sake, and the unpack warps, whose instructions bound the kernel
// there, wait behind it: 24 sequences of the 8B shape 10.6 -> 10.1 ms, 29 tokens 2.46 -> 2.31 ms.  With 64 there is no room beside two slots of
// accumulators; a chunk per step, which leaves some, costs more in hand-overs (56 against 53 us, q5_K 14336 x 4096 times 37, weights not in L2).
// The same matrix by columns, launches back to back / with L2 flushed before: 16: 33 / 49 us, 30: 35 / 46, 37: 41 / 53, 64: 42 / 55, 65: 46 / 58, 128: 50 / 63.
// Whatever the tile holds, a column's sums are the same ones in the same order: low terms, then high terms of 64 values in one accumulator,
// added to the f32 sum chunk by chunk, the shared part behind them.  So a column's result does not hang on how many columns came with it.
template <int NT>
struct GmCfg {
    static constexpr int CH = NT == 128 ? 1 : 2;
    static constexpr bool AT = NT != 64;  // weights go through tensor memory
    static constexpr int NS = NT == 64 ? 2 : NT == 32 ? 3 : 4, ND = 2;
    static constexpr int GS = NT == 64 ? 2 : 1, UG = NT == 128 ? 2 : NT == 64 ? 4 : 3;
    static_assert(UG / GS <= NS, "a group would miss a phase");
    static constexpr int DCOLS = CH == 1 ? NT : 3 * NT;  // accumulator columns per slot: 128, 192, 96
    static constexpr int SUMS = ND * DCOLS, A_COLS = SUMS + NT;  // columns where the sums and the weights stand
    static_assert(ND <= NS, "a step's accumulators are waited for at its own slot");
    static constexpr int A_SLOT = CH == 2 ? 80 : 32;  // 32 a chunk, 16 for the shared part
    static_assert(A_COLS + (AT ? A_SLOT * NS : 0) <= 512, "accumulators, sums, weights");
    static constexpr int THREADS = (GM_EPI_WARPS + 4 + 4 * UG) * 32;  // warps 0-7 epilogue, 8 packed copies, 9 MMA, 10 and 11 operand copies, 12 .. unpack
};
constexpr int GM_MAX_PACKED = 5;
constexpr int GM_SMEM = 227 * 1024;
struct GmSmem {
    int off_bar, off_tmem, off_hdr, off_a, off_b, off_packed, slot_a, slot_b, slot_packed, total;
};
// shared: some matrix of the launch has the part C (all but q6_K)
template <int NT>
__host__ __device__ inline GmSmem gm_smem_layout(int max_block_bytes, int np, bool shared) {
    constexpr int CH = GmCfg<NT>::CH;
    GmSmem s;
    s.off_bar = 0;  // done[4] ready[4] p_full[5] p_free[5]
    s.off_tmem = 18 * 8;
    s.off_hdr = 256;  // [GM_HDRS][128] {d, factor of the shared part}
    s.off_a = (s.off_hdr + GM_HDRS * GM_ROWS * 8 + 1023) & ~1023;
    s.slot_a = GmCfg<NT>::AT ? 0 : CH * GM_A_BYTES + (CH == 2 && shared ? GM_A_BYTES / 2 : 0);
    s.slot_b = CH * NT * 256 + (CH == 2 && shared ? NT * 32 : 0);
    s.off_b = s.off_a + GmCfg<NT>::NS * s.slot_a;
    s.off_packed = s.off_b + GmCfg<NT>::NS * s.slot_b;
    s.slot_packed = (GM_ROWS * max_block_bytes + 1023) & ~1023;
    s.total = s.off_packed + np * s.slot_packed;
    return s;
}

// ---- activations: f32 rows -> two fp16 terms in operand layout --------------------------------------------
// A token is one cluster of blocks (split_rows_shape), a warp one super-block.  Where the values come from:
//   SR_PLAIN    x[t][i]
//   SR_RESIDUAL x[t][i] + the product's partial results, stored back to x: the residual update of src/inference.jl:285, :305
//   SR_SWIGLU   silu(gate) * up of the product's partial results (src/inference.jl:295-299), the last token's stored to x as well
// then, where `gain` is given, rmsnorm (src/inference.jl:102-110): terms of gain .* x, 1/rms in the token's factor.
// Value k of a super-block: chunk k / 64, MMA step 2 * (k / 16 % 2) + (k / 32 % 2), half k / 8 % 2, and inside four values the order 0 2 1 3:
// the order in which the unpack warps meet the nibbles.  Bound by latency: a read from L2, the row's maximum and sum across the cluster, a write.
// SwiGLU rows of 14336 values: 24 tokens 15.3 -> 7.5 us, 128 tokens 15.9 -> 14.3 us against one block of 16 warps per token and two passes over the row.
enum : int { SR_PLAIN = 0, SR_RESIDUAL = 1, SR_SWIGLU = 2 };
struct SplitRowsParams {
    float* x;            // [n_tok][n]
    const float* gain;
    const float* y;      // partial results [part][n_tok][ldy] of the product before
    size_t part_stride;
    int ldy, up_row;     // SR_SWIGLU: rows of the up projection begin here
    GemmSplit sp;
    int n, n_tok, groups;
    uint8_t *act, *xs;   // null: only the values are wanted (x; not with SR_SWIGLU)
    float* scale;
};
constexpr int SR_MAX_CLUSTER = 8, SR_MAX_WARPS = 16, SR_KEEP = 2;  // SR_KEEP: super-blocks that a warp keeps in registers
// Blocks per token (a cluster) and warps per block.  The sum of squares is added up super-block by super-block, whatever the shape is.  As many
// blocks as give every SM two: beyond that clusters cost more than they bring (512 tokens of 8192 values, SwiGLU: 45 us with eight blocks each, 21 with one).
struct SplitRowsShape {
    int cluster, warps;
};
inline SplitRowsShape split_rows_shape(int n, int n_tok, int sms) {
    const int nb = n / QK_K;
    int cl = SR_MAX_CLUSTER;
    while (cl > 1 && (cl * n_tok > 2 * sms || nb < 2 * cl)) cl /= 2;
    const int per = (nb + cl - 1) / cl;
    return {cl, per < SR_MAX_WARPS ? per : SR_MAX_WARPS};
}

__device__ __forceinline__ void gm_sum_parts8(const float* y, size_t part_stride, const GemmSplit& sp, int tok, int ldy, int row, float (&v)[8]) {
    const int parts = gm_parts(sp, row);
    const float* src = y + (size_t)tok * ldy + row;
    float4 a = __ldcg(reinterpret_cast<const float4*>(src)), b = __ldcg(reinterpret_cast<const float4*>(src) + 1);
    for (int p = 1; p < parts; p += 2) {  // two parts' reads in flight together
        const bool two = p + 1 < parts;
        const float4* s = reinterpret_cast<const float4*>(src + p * part_stride);
        const float4* s2 = reinterpret_cast<const float4*>(src + (two ? p + 1 : p) * part_stride);
        const float4 c = __ldcg(s), d = __ldcg(s + 1), e = __ldcg(s2), f = __ldcg(s2 + 1);
        a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
        b.x += d.x; b.y += d.y; b.z += d.z; b.w += d.w;
        if (two) {
            a.x += e.x; a.y += e.y; a.z += e.z; a.w += e.w;
            b.x += f.x; b.y += f.y; b.z += f.z; b.w += f.w;
        }
    }
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <int MODE>
__global__ void __launch_bounds__(SR_MAX_WARPS * 32) split_rows_kernel(const __grid_constant__ SplitRowsParams p) {
    extern __shared__ float s_sum[];  // [nb] sums of squares of the token's super-blocks
    __shared__ float s_max[SR_MAX_WARPS], s_all[SR_MAX_CLUSTER];  // largest magnitudes of this block's warps, of the cluster's blocks
    const int tok = blockIdx.y, rank = blockIdx.x, cl = gridDim.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    const int nb = p.n / QK_K, per = (nb + cl - 1) / cl, b0 = rank * per, b1 = min(nb, b0 + per);
    const bool operands = p.act != nullptr, kept = per <= SR_KEEP * W;
    float* x = p.x + (size_t)tok * p.n;
    pdl_launch_dependents();
    cluster_arrive();  // (the cluster's blocks have to have started before one writes to another)
    float mx = 0.f, v[SR_KEEP][8];
    auto load8 = [](const float* src, float (&d)[8]) {
        const float4* s = reinterpret_cast<const float4*>(src);
        const float4 a = __ldcg(s), b = __ldcg(s + 1);
        d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w; d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
    };
    auto times_gain = [&](int e, const float (&a)[8], float (&d)[8]) {
        if (p.gain) {
            const float4* s = reinterpret_cast<const float4*>(p.gain + e);
            const float4 g = __ldg(s), h = __ldg(s + 1);
            d[0] = a[0] * g.x; d[1] = a[1] * g.y; d[2] = a[2] * g.z; d[3] = a[3] * g.w;
            d[4] = a[4] * h.x; d[5] = a[5] * h.y; d[6] = a[6] * h.z; d[7] = a[7] * h.w;
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) d[k] = a[k];
        }
    };
    cluster_wait();
    pdl_wait();
    // (the loop over the kept ones is unrolled, so that they are registers; what is not kept is stored and read again)
    for (int c0 = b0 + warp; c0 < b1; c0 += SR_KEEP * W) {
#pragma unroll
        for (int c = 0; c < SR_KEEP; ++c) {
            const int b = c0 + c * W, e = 256 * b + 8 * lane;
            if (b >= b1) break;
            if (MODE == SR_SWIGLU) {
                float u[8];
                gm_sum_parts8(p.y, p.part_stride, p.sp, tok, p.ldy, e, v[c]);
                gm_sum_parts8(p.y, p.part_stride, p.sp, tok, p.ldy, p.up_row + e, u);
#pragma unroll
                for (int k = 0; k < 8; ++k) v[c][k] = (v[c][k] * (1.0f / (1.0f + expf(-v[c][k])))) * u[k];
            } else {
                load8(x + e, v[c]);
                if (MODE == SR_RESIDUAL) {
                    float u[8];
                    gm_sum_parts8(p.y, p.part_stride, p.sp, tok, p.ldy, e, u);
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[c][k] += u[k];
                }
            }
            if (MODE == SR_RESIDUAL || (MODE == SR_SWIGLU && (!kept || tok == p.n_tok - 1))) {
                __stcg(reinterpret_cast<float4*>(x + e), make_float4(v[c][0], v[c][1], v[c][2], v[c][3]));
                __stcg(reinterpret_cast<float4*>(x + e) + 1, make_float4(v[c][4], v[c][5], v[c][6], v[c][7]));
            }
            if (!operands) continue;
            float ss = 0.f, d[8];
            times_gain(e, v[c], d);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                ss = fmaf(v[c][k], v[c][k], ss);
                mx = fmaxf(mx, fabsf(d[k]));
            }
            if (p.gain) {
                ss = warp_sum(ss);
                if (lane < cl) st_cluster_f32(cluster_map(s_sum + b, lane), ss);
            }
        }
    }
    if (!operands) return;
    mx = warp_max(mx);
    if (lane == 0) s_max[warp] = mx;
    __syncthreads();
    if (threadIdx.x < cl) {  // this block's maximum to every block of the cluster
        mx = 0.f;
        for (int i = 0; i < W; ++i) mx = fmaxf(mx, s_max[i]);
        st_cluster_f32(cluster_map(s_all + rank, threadIdx.x), mx);
    }
    cluster_sync_all();
    float ss = 0.f;
    mx = 0.f;
    for (int i = 0; i < cl; ++i) mx = fmaxf(mx, s_all[i]);
    if (p.gain) {
#pragma unroll 4
        for (int b = 0; b < nb; ++b) ss += s_sum[b];
    }
    // power of two that brings the largest value into [2^13, 2^14): a value 2^-16 of the largest still has 24 significant bits in its
    // two terms, and sums of 32 values, over 32, stay below 2^14 too
    const int ex = (int)(__float_as_uint(mx) >> 23);
    const int up = ex == 0 || ex == 255 ? 127 : min(267 - ex, 252);  // 127 + 13 - (ex - 127)
    const float s = __uint_as_float((uint32_t)up << 23), inv = __uint_as_float((uint32_t)(254 - up) << 23);
    const float rms = p.gain ? 1.0f / sqrtf(ss / (float)p.n + 1e-5f) : 1.f;
    if (rank == 0 && threadIdx.x == 0) p.scale[tok] = inv * rms;
    const int group = tok >> 3, row = tok & 7;
    for (int c0 = b0 + warp; c0 < b1; c0 += SR_KEEP * W) {
#pragma unroll
        for (int cc = 0; cc < SR_KEEP; ++cc) {
            const int b = c0 + cc * W;
            if (b >= b1) break;
            if (!kept) load8(x + 256 * b + 8 * lane, v[cc]);
            float sum = 0.f, d[8];
            times_gain(256 * b + 8 * lane, v[cc], d);
            __half h[8], l[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                d[k] *= s;
                h[k] = __float2half_rn(d[k]);
                l[k] = __float2half_rn(d[k] - __half2float(h[k]));
                sum += d[k];
            }
            auto pack = [](__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); };
            const int q = lane;  // which eight values of the super-block
            const int c = q >> 3, step = 2 * ((q >> 1) & 1) + ((q >> 2) & 1), half = q & 1;
            uint8_t* dst = p.act + ((size_t)(b * 4 + c) * p.groups + group) * GM_GROUP_BYTES + step * 256 + half * 128 + row * 16;
            *reinterpret_cast<uint4*>(dst) = make_uint4(pack(h[0], h[2]), pack(h[1], h[3]), pack(h[4], h[6]), pack(h[5], h[7]));
            *reinterpret_cast<uint4*>(dst + 1024) = make_uint4(pack(l[0], l[2]), pack(l[1], l[3]), pack(l[4], l[6]), pack(l[5], l[7]));
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if ((q & 3) == 0) {
                sum *= 0.03125f;
                const __half sh = __float2half_rn(sum), sl = __float2half_rn(sum - __half2float(sh));
                uint8_t* xd = p.xs + ((size_t)b * p.groups + group) * GM_XS_BYTES + row * 16 + (q >> 2) * 2;
                *reinterpret_cast<__half*>(xd) = sh;
                *reinterpret_cast<__half*>(xd + 128) = sl;
            }
        }
    }
}

// A product that is wanted as such: dst[t][i] = the sum of its partial results.  Grid (blocks per row, n_tok): at most 65535 tokens.
__global__ void sum_parts_kernel(const float* y, size_t part_stride, const __grid_constant__ GemmSplit sp, int ldy, int rows, float* __restrict__ dst) {
    const int tok = blockIdx.y;
    pdl_launch_dependents();
    pdl_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
        const int parts = gm_parts(sp, i);
        float v = __ldcg(y + (size_t)tok * ldy + i);
        for (int p = 1; p < parts; ++p) v += __ldcg(y + p * part_stride + (size_t)tok * ldy + i);
        dst[(size_t)tok * rows + i] = v;
    }
}

// Two f32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)), "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&r);
}

// ---- unpacking -------------------------------------------------------------------------------------------
__device__ __forceinline__ __half2 h2_bits(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t h2_raw(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 h2_small_int(uint32_t u8) { return __hsub2(h2_bits(u8 * 0x00010001u | 0x64006400u), h2_bits(0x64006400u)); }
__device__ __forceinline__ float f_small_int(uint32_t u8) { return __uint_as_float(0x4B000000u | u8) - 8388608.f; }

// Quant bits become fp16 numbers where they stand: a field at bits i .. of a 16-bit lane (i + its width <= 10) is the subnormal
// field * 2^(i - 24), and one fused multiply-add with a power of two times the scale puts it where it belongs: no shifts, no
// conversions.  Everything is (quant - centre) * scale * 2^-GM_A_EXP, at most 11 significant bits and a multiple of 2^-20: exact.
// (Shifting the fields into the mantissa of a number in [64, 128) takes 19 instructions per 8 q5_K values, 13 of them on the
// half-rate integer pipe; this takes 17, 9 of them integer.)
constexpr int GM_A_EXP = 20;
struct GmScale {
    __half2 low, high, off;  // scale * 2^4 (bits 0-3), scale (bits 4-7), -centre * scale * 2^-20
};
__device__ __forceinline__ GmScale gm_scale(__half2 S, float centre) {
    GmScale g;
    g.low = __hmul2(S, __float2half2_rn(16.f));
    g.high = S;
    g.off = __hmul2(S, __float2half2_rn(-centre * 9.5367431640625e-07f));
    return g;
}
// 16 values of one MMA step from the nibbles of q (HIGH: the upper ones); f: words whose bits `top_mask` of every byte stand above the
// nibble, with the factor `top`.  Pairs are bytes (0, 2) and (1, 3) of a word.
template <bool HIGH, bool TOP>
__device__ __forceinline__ void gm_values16(const uint4& q, const uint4& f, uint32_t top_mask, __half2 top, const GmScale& g, uint32_t (&o)[8]) {
    const uint32_t qw[4] = {q.x, q.y, q.z, q.w}, fw[4] = {f.x, f.y, f.z, f.w};
    const uint32_t m = HIGH ? 0x00F000F0u : 0x000F000Fu;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t w = e ? qw[i] >> 8 : qw[i];
            __half2 v = __hfma2(h2_bits(w & m), HIGH ? g.high : g.low, g.off);
            if (TOP) v = __hfma2(h2_bits((e ? fw[i] >> 8 : fw[i]) & top_mask), top, v);
            o[2 * i + e] = h2_raw(v);
        }
    }
}
// Where a row's operand values go: the 16 of MMA step kk of a slot, into core matrices in shared memory or eight columns of tensor memory.
template <bool AT>
struct GmDest {
    uint8_t* smem;
    uint32_t tmem;
    __device__ __forceinline__ void put(int kk, const uint32_t (&o)[8]) const {
        if (AT) {
            tmem_st8(tmem + (uint32_t)(8 * kk), o);
        } else {
            *reinterpret_cast<uint4*>(smem + kk * 4096) = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4*>(smem + kk * 4096 + 2048) = make_uint4(o[4], o[5], o[6], o[7]);
        }
    }
};

// ---- the GEMM ----------------------------------------------------------------------------------------
// Steps per super-block: q6_K has eight chunks (its two passes) and no shared part.
template <int CH>
__device__ __forceinline__ int gm_steps(int type) { return CH == 2 ? (type == T_Q6_K ? 4 : 2) : (type == T_Q6_K ? 8 : 5); }

template <int NT>
__global__ void __launch_bounds__(GmCfg<NT>::THREADS, 1) kq_gemm_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ GemmMaps maps) {
    constexpr bool AT = GmCfg<NT>::AT;
    constexpr int NS = GmCfg<NT>::NS, ND = GmCfg<NT>::ND, UG = GmCfg<NT>::UG, GS = GmCfg<NT>::GS, DCOLS = GmCfg<NT>::DCOLS, CH = GmCfg<NT>::CH;
    const int NP = p.np;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the copies and operands want their alignment
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (the same for a warp's threads, and known to be)
    int max_bb = 0;
    bool shared = false;
    for (int i = 0; i < p.nseg; ++i) {
        max_bb = max(max_bb, dev_block_bytes(p.seg[i].type));
        shared = shared || p.seg[i].type != T_Q6_K;
    }
    const GmSmem L = gm_smem_layout<NT>(max_bb, p.np, shared);
    uint64_t* done = reinterpret_cast<uint64_t*>(smem + L.off_bar);
    // ready: weights unpacked, activations landed and the accumulators of the slot's last use read.  One barrier for all three, because the
    // MMA thread's own instructions bound this kernel: with a barrier each it took 1450 cycles per step of 64 values, whatever the tile.
    uint64_t *ready = done + 4, *p_full = done + 8, *p_free = done + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L.off_tmem);
    float2* hdr = reinterpret_cast<float2*>(smem + L.off_hdr);

    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(done + i, 1);
            mbar_init(ready + i, 4 * GS + 1 + GM_EPI_WARPS);
        }
        for (int i = 0; i < NP; ++i) {
            mbar_init(p_full + i, 1);
            mbar_init(p_free + i, 4 * UG);
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 9) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // the walk over this block's units, the same for every role: chunks of token tile 0, of token tile 1, ..., every gridDim.x-th of them
    const int nb = p.sp.nb, items = p.chunks * p.sp.ntile;
    struct Where {
        int u, end;                  // unit, first one behind the chunk
        int seg, row_tile, ntile, b; // matrix, its row tile, token tile, super-block
        int type, steps;             // of the matrix (an indexed read of a parameter is slow)
    };
    auto enter = [&](Where& w) {
        w.type = p.seg[w.seg].type;
        w.steps = gm_steps<CH>(w.type);
    };
    auto first_unit = [&](int item) {
        Where w;
        w.ntile = item / p.chunks;
        w.u = (item - w.ntile * p.chunks) * p.sp.U;
        w.end = min(w.u + p.sp.U, p.total);
        w.row_tile = w.u / nb;
        w.b = w.u - w.row_tile * nb;
        w.seg = 0;
        while (w.seg + 1 < p.nseg && w.row_tile >= p.seg[w.seg].row_tiles) w.row_tile -= p.seg[w.seg++].row_tiles;
        enter(w);
        return w;
    };
    auto advance = [&](Where& w) {  // (divisions here, once per super-block and role, had cost 2000 cycles of every 5700)
        ++w.u;
        if (++w.b < nb) return;
        w.b = 0;
        if (++w.row_tile < p.seg[w.seg].row_tiles || w.seg + 1 == p.nseg) return;
        w.row_tile = 0;
        ++w.seg;
        enter(w);
    };
    const int chunk_b = p.sp.tok * 256;  // bytes of a chunk of X in its slot
    bool ok = true;

    if (warp == 8) {
        // ================= packed weights: one tiled copy per super-block =================
        if (lane == 0) {
            int s = 0;
            bool first = true;
            uint32_t parity = 1;  // of the use before
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
            for (Where w = first_unit(item); w.u < w.end; advance(w)) {
                if (!first && !mbar_wait_parked(p_free + s, parity)) {
                    ok = false;
                    break;
                }
                const GemmSeg& sg = p.seg[w.seg];
                const int bb = dev_block_bytes(w.type), panel = w.b / sg.kb;
                mbar_arrive_expect_tx(p_full + s, (uint32_t)(GM_ROWS * bb));
                const bool tail = (panel + 1) * sg.kb > nb;
                tma_load_3d(smem + L.off_packed + s * L.slot_packed, tail ? &maps.tail[w.seg] : &maps.main[w.seg], (w.b - panel * sg.kb) * bb,
                            w.row_tile * GM_ROWS, tail ? 0 : panel, p_full + s);
                if (++s == NP) {
                    s = 0;
                    first = false;
                    parity ^= 1u;
                }
            }
            if (!ok) {
                atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
                for (int i = 0; i < 2000; ++i) __nanosleep(1000);  // copies in flight land within microseconds
            }
        }
    } else if (warp == 10 || warp == 11) {
        // ================= activation operands: one bulk copy per 64 values =================
        pdl_wait();  // (weights are constant: the copies and the unpacking of the first ones do not wait)
        if (lane == 0) {
            int s = 0, turn = warp - 10;
            bool first = true;
            uint32_t parity = 1;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
            for (Where w = first_unit(item); w.u < w.end && ok; advance(w)) {
                const int steps = w.steps, g0 = (w.ntile * p.sp.tok) >> 3, ng = min(p.sp.tok >> 3, p.groups - g0);
                const uint8_t* act = p.act + ((size_t)w.b * 4 * p.groups + g0) * GM_GROUP_BYTES;
                for (int k = 0; k < steps; ++k, turn ^= 1) {
                    if (turn == 0) {
                        if (!first && !mbar_wait_parked(done + s, parity)) {
                            ok = false;
                            break;
                        }
                        uint8_t* dst = smem + L.off_b + s * L.slot_b;
                        const uint32_t xs_bytes = (uint32_t)(ng * GM_XS_BYTES), bytes = (uint32_t)(ng * GM_GROUP_BYTES);
                        const uint8_t* xs = p.xs + ((size_t)w.b * p.groups + g0) * GM_XS_BYTES;
                        if (CH == 1) {
                            const bool shared_part = steps == 5 && k == 4;
                            mbar_arrive_expect_tx(ready + s, shared_part ? xs_bytes : bytes);
                            if (shared_part) bulk_g2s_plain(dst, xs, xs_bytes, ready + s);
                            else bulk_g2s_plain(dst, act + (size_t)(k & 3) * p.groups * GM_GROUP_BYTES, bytes, ready + s);
                        } else {
                            const bool shared_part = steps == 2 && k == 1;
                            const uint8_t* src = act + (size_t)(2 * (k & 1)) * p.groups * GM_GROUP_BYTES;
                            mbar_arrive_expect_tx(ready + s, 2 * bytes + (shared_part ? xs_bytes : 0u));
                            if (ng == p.groups) {  // the two chunks lie behind one another, here and there
                                bulk_g2s_plain(dst, src, 2 * bytes, ready + s);
                            } else {
                                bulk_g2s_plain(dst, src, bytes, ready + s);
                                bulk_g2s_plain(dst + chunk_b, src + (size_t)p.groups * GM_GROUP_BYTES, bytes, ready + s);
                            }
                            if (shared_part) bulk_g2s_plain(dst + 2 * chunk_b, xs, xs_bytes, ready + s);
                        }
                    }
                    if (++s == NS) {
                        s = 0;
                        first = false;
                        parity ^= 1u;
                    }
                }
            }
            if (!ok) {
                atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
                for (int i = 0; i < 2000; ++i) __nanosleep(1000);
            }
        }
    } else if (warp == 9) {
        // ================= MMA issue: the whole warp walks along, one thread issues =================
        const uint32_t idesc = umma_idesc_f16(GM_ROWS, p.sp.tok);
        // operand descriptors of slot 0; the others lie a multiple of 16 bytes further
        const uint64_t desc_a = umma_desc(smem + L.off_a, 2048, 128), desc_b = umma_desc(smem + L.off_b, 128, GM_GROUP_BYTES);
        const uint64_t desc_xs = umma_desc(smem + L.off_b, 128, GM_XS_BYTES);
        // a: slot of the weights; ka, kb: bytes further in it and in the operand of the activations
        auto mma = [&](uint32_t d, int a, int ka, uint64_t b, uint32_t accumulate) {
            if (AT) umma_f16_at(d, tmem_base + (uint32_t)(GmCfg<NT>::A_COLS + GmCfg<NT>::A_SLOT * a + (ka >> 9)), b, idesc, accumulate);  // (4096 bytes: 8 columns)
            else umma_f16(d, desc_a + (uint64_t)((a * L.slot_a + ka) >> 4), b, idesc, accumulate);
        };
        int s = 0, ds = 0;
        uint32_t parity = 0;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
        for (Where w = first_unit(item); w.u < w.end && ok; advance(w)) {
            const int steps = w.steps;
            for (int k = 0; k < steps; ++k) {
                if (!mbar_wait_warp(ready + s, parity)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(ds * DCOLS);
                const uint64_t db = desc_b + (uint64_t)(s * (L.slot_b >> 4));
                const bool shared_part = k == (CH == 2 ? 1 : 4) && (CH == 2 ? steps == 2 : steps == 5);
                if (elect_one()) {
                    if (CH == 2 || !shared_part) {
#pragma unroll
                        for (int c = 0; c < CH; ++c)
#pragma unroll
                            for (int t = 1; t >= 0; --t)  // low terms of X first
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    mma(d + (uint32_t)(c * NT), s, c * GM_A_BYTES + kk * 4096, db + (uint64_t)((c * chunk_b + t * 1024 + kk * 256) >> 4),
                                        t == 1 && kk == 0 ? 0u : 1u);
                    }
                    if (shared_part) {  // low terms of C first
                        constexpr int ax = CH == 2 ? 2 * GM_A_BYTES : 0;
                        const uint64_t dx = desc_xs + (uint64_t)((s * L.slot_b + (CH == 2 ? 2 * chunk_b : 0)) >> 4);
                        const uint32_t dd = d + (uint32_t)(CH == 2 ? 2 * NT : 0);
                        mma(dd, s, ax + 4096, dx, 0u);
                        mma(dd, s, ax, dx, 1u);
                    }
                    umma_commit(done + s);
                }
                __syncwarp();
                if (++ds == ND) ds = 0;
                if (++s == NS) {
                    s = 0;
                    parity ^= 1u;
                }
            }
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    } else if (warp > 11) {
        // ================= unpack: thread = row =================
        const int id = threadIdx.x - 12 * 32, r = id & 127, group = (warp - 12) >> 2;
        const int row_off = (r >> 3) * 128 + (r & 7) * 16;
        auto q6_scale = [&](const Where& w) -> float {
            if (w.type != T_Q6_K) return 0.f;
            const GemmSeg& sg = p.seg[w.seg];
            const int row = w.row_tile * GM_ROWS + r;
            return row < sg.rows ? __half2float(__ldg(sg.d6 + (size_t)row * nb + w.b)) : 0.f;
        };
        constexpr int TURNS = UG / GS;
        const int my_turn = group / GS, sub = group % GS;
        int s = 0, turn = 0, ps = 0, hs = GM_HDRS - 1;  // slot, whose turn it is, packed slot, set of factors
        bool first = true, fresh = true;  // fresh: the first super-block of a chunk
        float d6_next = 0.f;
        uint32_t parity = 1, p_parity = 0;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
        for (Where w = first_unit(item); w.u < w.end && ok;) {
            const int type = w.type, bb = dev_block_bytes(type), steps = w.steps;
            hs = (hs + 1) % GM_HDRS;
            const float d6 = fresh ? q6_scale(w) : d6_next;
            advance(w);
            fresh = w.u == w.end;
            if (!fresh) d6_next = q6_scale(w);  // a super-block ahead: the latency of a global read
            if (!mbar_wait_warp(p_full + ps, p_parity)) {  // (every group follows every packed slot, with or without a step in it)
                ok = false;
                break;
            }
            const uint8_t* blk = smem + L.off_packed + ps * L.slot_packed + r * bb;
            int ahead = my_turn - turn;  // steps until this group's next one
            if (ahead < 0) ahead += TURNS;
            const bool mine_here = ahead < steps;
            uint64_t sc8 = 0, m8 = 0;
            uint4 top0 = make_uint4(0u, 0u, 0u, 0u), top1 = top0;  // q5_K: fifth bits; q6_K: scales
            float d = d6, dmin = 0.f, s_up = 1.f, s_dn = 1.f;
            if (!mine_here) {
            } else if (type != T_Q6_K) {
                const uint4 h = *reinterpret_cast<const uint4*>(blk);
                decode_scales_k4(h, sc8, m8);
                d = half_bits_to_float(h.x & 0xFFFFu);
                dmin = half_bits_to_float(h.x >> 16);
                if (type == T_Q5_K) {
                    top0 = *reinterpret_cast<const uint4*>(blk + 16);
                    top1 = *reinterpret_cast<const uint4*>(blk + 32);
                }
                // power of two that keeps the shared part C and its second term inside the range of fp16
                const int ex = (int)(__float_as_uint(fmaxf(fabsf(d) * 1024.f, fabsf(dmin) * 64.f)) >> 23);
                if (ex != 0 && ex < 254) {
                    s_up = __uint_as_float((uint32_t)(254 - ex) << 23);
                    s_dn = __uint_as_float((uint32_t)ex << 23);
                }
            } else {
                top0 = *reinterpret_cast<const uint4*>(blk + 192);
            }
            const float cen = type == T_Q5_K ? 16.f : 8.f;
            for (int k = 0; k < steps; ++k) {
                const int slot = s;
                const bool mine = turn == my_turn, reused = !first;
                const uint32_t use_parity = parity;
                if (++turn == TURNS) turn = 0;
                if (++s == NS) {
                    s = 0;
                    first = false;
                    parity ^= 1u;
                }
                if (!mine) continue;
                if (reused && !mbar_wait_warp(done + slot, use_parity)) {
                    ok = false;
                    break;
                }
                if (AT) tc_fence_after();
                // (the epilogue may still be at the super-block before the last one: four sets of factors are enough)
                if (k == 0 && sub == 0) hdr[hs * GM_ROWS + r] = make_float2(d * (float)(1 << GM_A_EXP), 32.f * s_dn);
                uint8_t* const a_slot = smem + L.off_a + slot * L.slot_a + row_off;
                const uint32_t a_cols = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(GmCfg<NT>::A_COLS + GmCfg<NT>::A_SLOT * slot);
                if (CH == 2 || type == T_Q6_K || k < 4) {
#pragma unroll 1
                    for (int e = sub; e < CH; e += GS) {
                        const int kc = CH * k + e;
                        const GmDest<AT> dst = {a_slot + e * GM_A_BYTES, a_cols + (uint32_t)(32 * e)};
                        uint32_t o[8];
                        if (type == T_Q6_K) {
                            const int c = kc & 3, hh = c >> 1, odd = c & 1;
                            const uint32_t scw = c == 0 ? top0.x : c == 1 ? top0.y : c == 2 ? top0.z : top0.w;
#pragma unroll
                            for (int part = 0; part < 2; ++part) {
                                const uint4 f = *reinterpret_cast<const uint4*>(blk + 128 + 32 * hh + 16 * part);
#pragma unroll
                                for (int hi = 0; hi < 2; ++hi) {
                                    const int sc = (int)(int8_t)(scw >> (8 * (2 * hi + part)));
                                    const __half2 S = __half2half2(__int2half_rn(kc < 4 ? sc - (sc & 1) : (sc & 1)));
                                    const GmScale g = gm_scale(S, 32.f);
                                    const uint4 q = *reinterpret_cast<const uint4*>(blk + 64 * hh + 32 * hi + 16 * part);
                                    const int idx = 2 * odd + hi;  // which two bits of the byte: value 16 at bit 2 * idx
                                    const __half2 up = __hmul2(S, h2_bits(((uint32_t)(23 - 2 * idx) << 10) * 0x00010001u));  // 2^(8 - 2 idx)
                                    if (odd) gm_values16<true, true>(q, f, 0x00030003u << (2 * idx), up, g, o);
                                    else gm_values16<false, true>(q, f, 0x00030003u << (2 * idx), up, g, o);
                                    dst.put(2 * part + hi, o);
                                }
                            }
                        } else {
                            const uint32_t two = (uint32_t)(sc8 >> (16 * kc));
                            const GmScale g0 = gm_scale(h2_small_int(two & 0xFFu), cen), g1 = gm_scale(h2_small_int((two >> 8) & 0xFFu), cen);
                            if (type == T_Q5_K) {  // the fifth bit of sub-block j is bit j: value 16 from 2^(j - 24) takes 2^(8 - j)
                                const uint32_t p0 = (uint32_t)(23 - 2 * kc) << 10;
                                const __half2 up0 = __hmul2(g0.high, h2_bits(p0 * 0x00010001u)), up1 = __hmul2(g1.high, h2_bits((p0 - 1024u) * 0x00010001u));
                                const uint32_t bit = 0x00010001u << (2 * kc);
#pragma unroll
                                for (int part = 0; part < 2; ++part) {
                                    const uint4 q = *reinterpret_cast<const uint4*>(blk + 48 + 32 * kc + 16 * part);
                                    gm_values16<false, true>(q, part ? top1 : top0, bit, up0, g0, o);
                                    dst.put(2 * part, o);
                                    gm_values16<true, true>(q, part ? top1 : top0, bit << 1, up1, g1, o);
                                    dst.put(2 * part + 1, o);
                                }
                            } else {
#pragma unroll
                                for (int part = 0; part < 2; ++part) {
                                    const uint4 q = *reinterpret_cast<const uint4*>(blk + 16 + 32 * kc + 16 * part);
                                    gm_values16<false, false>(q, q, 0u, g0.high, g0, o);
                                    dst.put(2 * part, o);
                                    gm_values16<true, false>(q, q, 0u, g1.high, g1, o);
                                    dst.put(2 * part + 1, o);
                                }
                            }
                        }
                    }
                }
                if (type != T_Q6_K && k == (CH == 2 ? 1 : 4) && sub == GS - 1) {
                    const GmDest<AT> dst = {a_slot + (CH == 2 ? 2 * GM_A_BYTES : 0), a_cols + (CH == 2 ? 64u : 0u)};
                    uint32_t o[8], o2[8];
#pragma unroll
                    for (int j2 = 0; j2 < 4; ++j2) {
                        float f2[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int j = 2 * j2 + e;
                            const float sc = f_small_int((uint32_t)byte64(sc8, j)), m = f_small_int((uint32_t)byte64(m8, j));
                            f2[e] = fmaf(-dmin, m, d * cen * sc) * s_up;
                        }
                        const __half2 hi = __floats2half2_rn(f2[0], f2[1]);
                        const float2 back = __half22float2(hi);
                        o[j2] = o[j2 + 4] = h2_raw(hi);
                        o2[j2] = o2[j2 + 4] = h2_raw(__floats2half2_rn(f2[0] - back.x, f2[1] - back.y));
                    }
                    dst.put(0, o);  // each term times the high and the low terms of the sums
                    dst.put(1, o2);
                }
                if (AT) {
                    tmem_wait_st();
                    tc_fence_before();
                } else {
                    fence_proxy_async();  // the tensor core reads shared memory through the asynchronous proxy
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(ready + slot);
            }
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(p_free + ps);
            if (++ps == NP) {
                ps = 0;
                p_parity ^= 1u;
            }
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    } else {
        // ================= epilogue: thread = weight row; warps e and e + 4 split the tokens =================
        pdl_wait();
        constexpr int NH = NT / 2;
        const int q = warp & 3, half = warp >> 2;
        const int r = 32 * q + lane;
        const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16);
        const int mine = max(0, min(NH, p.sp.tok - NH * half));  // of the tile's tokens
        float2 acc[NH / 2];
#pragma unroll
        for (int t = 0; t < NH / 2; ++t) acc[t] = make_float2(0.f, 0.f);
        if (lane < ND) mbar_arrive(ready + lane);  // no accumulators to wait for at first
        bool held = false;  // sums of this part are in tensor memory
        int s = 0, hs = 0, ds = 0, next = ND % NS;  // next: the step that will use these accumulators again
        uint32_t parity = 0;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x)
        for (Where w = first_unit(item); w.u < w.end && ok; advance(w)) {
            const int steps = w.steps;
            float2 f = make_float2(0.f, 0.f);
            for (int k = 0; k < steps; ++k) {
                if (!mbar_wait_warp(done + s, parity)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                if (k == 0) f = hdr[hs * GM_ROWS + r];
                const bool shared_part = k == (CH == 2 ? 1 : 4) && (CH == 2 ? steps == 2 : steps == 5);
                const float2 md = make_float2(f.x, f.x), mc = make_float2(f.y, f.y);
                const uint32_t td = taddr + (uint32_t)(ds * DCOLS);
                if (CH == 2) {
#pragma unroll
                    for (int c0 = 0; c0 < NH; c0 += 16) {
                        if (c0 >= mine) break;
                        float v[16], w2[16];
                        tmem_ld16f(td + (uint32_t)(NH * half + c0), v);
                        tmem_ld16f(td + (uint32_t)(NT + NH * half + c0), w2);
#pragma unroll
                        for (int t = 0; t < 16; t += 2)
                            acc[(c0 + t) / 2] = fma2(md, make_float2(w2[t], w2[t + 1]), fma2(md, make_float2(v[t], v[t + 1]), acc[(c0 + t) / 2]));
                    }
                }
                if (CH == 1 || shared_part) {
                    const float2 mm = shared_part ? mc : md;
#pragma unroll
                    for (int c0 = 0; c0 < NH; c0 += 16) {
                        if (c0 >= mine) break;
                        float v[16];
                        tmem_ld16f(td + (uint32_t)((CH == 2 ? 2 * NT : 0) + NH * half + c0), v);
#pragma unroll
                        for (int t = 0; t < 16; t += 2) acc[(c0 + t) / 2] = fma2(mm, make_float2(v[t], v[t + 1]), acc[(c0 + t) / 2]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(ready + next);
                if (++next == NS) next = 0;
                if (++ds == ND) ds = 0;
                if (++s == NS) {
                    s = 0;
                    parity ^= 1u;
                }
            }
            hs = (hs + 1) % GM_HDRS;
            const bool last = w.b == nb - 1 || w.u == w.end - 1;  // this chunk's part of the tile is complete
            if (ok && (last || ((w.b + 1) & (w.type == T_Q6_K ? 1 : 3)) == 0)) {  // 20 (q6_K: 16) values have been added up
                const uint32_t sums = taddr + (uint32_t)(GmCfg<NT>::SUMS + NH * half);
#pragma unroll
                for (int c0 = 0; c0 < NH; c0 += 16) {
                    if (!held || c0 >= mine) break;
                    float v[16];
                    tmem_ld16f(sums + (uint32_t)c0, v);
#pragma unroll
                    for (int t = 0; t < 16; t += 2) acc[(c0 + t) / 2] = make_float2(v[t] + acc[(c0 + t) / 2].x, v[t + 1] + acc[(c0 + t) / 2].y);
                }
                if (!last) {
#pragma unroll
                    for (int c0 = 0; c0 < NH; c0 += 16)
                        if (c0 < mine) tmem_st16f(sums + (uint32_t)c0, reinterpret_cast<const float(&)[16]>(acc[c0 / 2]));
#pragma unroll
                    for (int t = 0; t < NH / 2; ++t) acc[t] = make_float2(0.f, 0.f);
                }
                held = !last;
            }
            if (ok && last) {
                const int part = (w.u / p.sp.U) - (w.u - w.b) / p.sp.U;
                int row = w.row_tile * GM_ROWS + r;
                const bool valid = row < p.seg[w.seg].rows;
                for (int e = 0; e < w.seg; ++e) row += p.seg[e].row_tiles * GM_ROWS;
                float* dst = p.y + (size_t)part * p.part_stride + row;
                float scale[(NH + 31) / 32];  // the tokens' factors, a lane each: read from L2 in front of every store, they would be NH reads in a row
#pragma unroll
                for (int i = 0; i < (NH + 31) / 32; ++i) {
                    const int t = 32 * i + lane, tok = w.ntile * p.sp.tok + NH * half + t;
                    scale[i] = t < mine && tok < p.n_tok ? __ldcg(p.scale + tok) : 0.f;
                }
#pragma unroll
                for (int t = 0; t < NH; ++t) {
                    const int tok = w.ntile * p.sp.tok + NH * half + t;
                    const float of_tok = __shfl_sync(0xffffffffu, scale[t / 32], t & 31);
                    if (valid && t < mine && tok < p.n_tok) dst[(size_t)tok * p.ldy] = (t & 1 ? acc[t / 2].y : acc[t / 2].x) * of_tok;
                }
#pragma unroll
                for (int t = 0; t < NH / 2; ++t) acc[t] = make_float2(0.f, 0.f);
            }
        }
        if (!ok && lane == 0) atomicExch(p.status, DEV_ERR_TMA_TIMEOUT);
    }
    // every path ends here; the tensor memory is freed by the warp that allocated it
    // A block has released the next kernel when its first warp comes here: the one of the packed copies, with the last of them under way.  (At the start it
    // would let the next kernel's blocks crowd onto the few SMs that this grid leaves free.)
    pdl_launch_dependents();
    tc_fence_before();
    __syncthreads();
    if (warp == 9) tmem_dealloc(tmem_base, 512);
}

}  // namespace l2b
