// y[M, N] = x[M, K] w[N, K]^T (+ bias[N]) for float32 operands, at the precision of float32 products, on the tensor cores of pairs of SMs
// (the CUDA-core product of csrc/gemm_simt.cu runs where this one does not pay).
//
// A float32 number is the sum of three bfloat16 numbers exactly: the nearest one, the nearest to what is left, and the rest (`split`); the second is at most
// 2^-8 of the number, the third 2^-17.  Of the nine products of parts six are formed, in float32: the three left out are at most 2^-24 of the product
// together, as much as one rounding of a float32 product may lose, and of either sign.  (Parts cut off towards zero would leave out up to 2^-21, always of the
// product's sign, so that a sum of products of one sign never lost it again.)  The tensor core's own float32 sums are cut off rather than rounded, so
// a sum stays there for 64 products only (small parts first); every 64-wide chunk of K is taken out of tensor memory and added to a
// float32 register, rounded to nearest.  Against 64 bits the error is 1.04e-7 to 1.31e-7 at K 2,048 (with and without shares of K) and 1.25e-7 at K 5,632
// (2-norm; parts cut off towards zero 1.42e-7 to 1.63e-7) where one chain of K fused multiply-adds leaves 8.1e-7 and 1.35e-6.
// A number that is not finite, one too small for its parts, or a sum that overflows on the way makes the sum of the parts infinite or NaN: an output that is not finite is
// worked out again as one chain of fused multiply-adds from the operands themselves, so it is what the CUDA-core product gives: by the whole block, once its
// tiles are done and nothing waits for it, 64 x 64 outputs at a time (`sp_again`).
//
//   split    [rows, K] float32 -> three bfloat16 planes: bound by memory, 10 bytes a number (11,264 x 2,048: 45 us, 5.1 TB/s).
//   product  a pair of blocks owns 256 rows of w and BN (64, 128 or 256) tokens; per 64-wide chunk of K each block's stage
//            holds its half of both operands' three planes (TMA, 128-byte swizzle), 24 cta_group::2 MMAs of K 16 go into one of
//            two to four accumulators, and eight warps move a finished one into their registers (a thread a row of w, half of the tokens).
//            Rows of w on the 128-lane side: what a warp stores for a token is 128 contiguous bytes, and a few tokens waste nothing.
//            The pair runs persistently over items: tiles with all of K first, then the shares of K of the remaining tiles, which meet in `partial` and
//            which a last small kernel adds up in order.  Tiles that are one wave of pairs and a few more would take two waves: as shares the few are spread over
//            all pairs (509 x 11,264 x 2,048, 88 tiles on 74 pairs: 161 -> 140 - 143 us; 1,000 x 2,560 x 2,048, 80 tiles of 128 tokens, 73 -> 66 us).
//
// Bound: the tensor pipe (6 bfloat16 products for one float32 one: a sixth of its rate) for many tokens, memory (4 bytes of w read, 6
// written and read again) for few.  2,048 x 11,264 x 2,048: 2,707 us on the CUDA cores -> 403 us (235 TFLOP/s);
// 509 x 11,264 x 2,048 1,008 -> 140 - 143 us; 509 x 2,048 x 5,632 1,195 -> 78 us; 17 x 2,048 x 2,048, w from memory, 209 -> 24 us.  Chunks of 32 in a deeper ring were slower
// (550 us at 2,048 tokens): the way from a full accumulator to an empty one costs about 2 us, so what counts is the work per accumulator and their number.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "tcgen05_common.cuh"

typedef __nv_bfloat16 bf16;

#define SP_THREADS 320            // a producer warp, an MMA warp, eight warps that add up
#define SP_BK 64
#define SP_MAX_STAGES 3
#define SP_MAX_ACCS 4
#define SP_A_PLANE 16384u         // 128 rows of w x 64 x 2 bytes

struct SpParams {
    float* out; int64_t out_stride;              // [M][out_stride], the first column that of w's first row here
    const void* bias; int bias_tag;
    float* partial;                              // [splits][M][cols] when splits > 1, less n_shared: indexed by the output's column
    const float* x; const float* w;              // the operands themselves (an output that is not finite)
    int M, N, K, k_tiles, splits, k_per_split;   // splits: shares of K of the tiles behind the first `whole` ones, whose rows of w start at n_shared
    int whole, shared, n_shared, cols;           // (shared: how many tiles those are; cols: how many rows)
    int tiles_m, num_items, stages, blocks_w, blocks_x;      // tiles_m: tiles of tokens; blocks: of 128 rows of w, of BN / 2 tokens
    int* error;
};

__device__ __forceinline__ void sp_tma_load(uint32_t dst, const CUtensorMap* map, uint32_t leader_bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sp_mma(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void sp_commit(uint64_t* bar) {       // arrives on this barrier in both blocks of the pair
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void sp_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void sp_ld32(uint32_t addr, float* v) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
                   "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                   "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ bool is_finite_f32(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// The outputs of tokens m0 .. m0 + mc and rows n0 .. n0 + nc of w that are not finite, worked out again from the operands themselves by the whole block (256 threads or
// more), one chain of fused multiply-adds each: 64 x 64 outputs a step, 32 of K at a time through `sm` (2 x 64 x 33 floats), four by four a thread; what is
// finite stays as it is, and a thread whose outputs all are only helps with the loads.
#define SP_AGAIN_FLOATS (2 * 64 * 33)
__device__ __noinline__ void sp_again(const SpParams& p, float* sm, int m0, int mc, int n0, int nc) {
    float* xs = sm;
    float* ws = sm + 64 * 33;
    const int tid = threadIdx.x, ty = (tid >> 4) * 4, tx = tid & 15;
    const int m_end = min(m0 + mc, p.M), n_end = min(n0 + nc, p.N);
    for (int mt = m0; mt < m_end; mt += 64)
        for (int nt = n0; nt < n_end; nt += 64) {
            uint32_t again = 0;
            float* o = p.out + (int64_t)(mt + ty) * p.out_stride + nt + tx;
            if (tid < 256) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (mt + ty + i < m_end && nt + tx + 16 * j < n_end && !is_finite_f32(o[i * p.out_stride + 16 * j])) again |= 1u << (4 * i + j);
            }
            if (!__syncthreads_or(again != 0)) continue;
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
            for (int k0 = 0; k0 < p.K; k0 += 32) {
                for (int i = tid; i < 64 * 32; i += blockDim.x) {
                    const int r = i >> 5, k = i & 31;
                    xs[r * 33 + k] = mt + r < m_end && k0 + k < p.K ? p.x[(int64_t)(mt + r) * p.K + k0 + k] : 0.f;
                    ws[r * 33 + k] = nt + r < n_end && k0 + k < p.K ? p.w[(int64_t)(nt + r) * p.K + k0 + k] : 0.f;
                }
                __syncthreads();
                if (again) {
                    const int n = min(32, p.K - k0);
                    for (int k = 0; k < n; ++k) {
                        float a[4], b[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) { a[i] = xs[(ty + i) * 33 + k]; b[i] = ws[(tx + 16 * i) * 33 + k]; }
#pragma unroll
                        for (int i = 0; i < 4; ++i)
#pragma unroll
                            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
                    }
                }
                __syncthreads();
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if ((again >> (4 * i + j)) & 1) o[i * p.out_stride + 16 * j] = acc[i][j] + (p.bias ? load_tagged(p.bias, nt + tx + 16 * j, p.bias_tag) : 0.f);
        }
}

// --------------------------------------------------------------------------- split

// A number as its nearest bfloat16 number, the nearest to what is left, and the rest, which is one too: pairs of numbers, the first in the lower halves.
__device__ __forceinline__ uint32_t nearest2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void cut3(float v0, float v1, uint32_t& a, uint32_t& b, uint32_t& c) {
    a = nearest2(v0, v1);
    const float r0 = v0 - __uint_as_float(a << 16), r1 = v1 - __uint_as_float(a & 0xffff0000u);                // differences are exact
    b = nearest2(r0, r1);
    c = nearest2(r0 - __uint_as_float(b << 16), r1 - __uint_as_float(b & 0xffff0000u));                        // (at most 7 bits: nothing is rounded)
}
// Zero, or a number whose parts are normal numbers: from 2^-102 on, and below what rounds to infinity.
__device__ __forceinline__ bool ordinary(float v) {
    const uint32_t t = __float_as_uint(v) & 0x7fffffffu;
    return t - 0x0c800000u < 0x7f7f8000u - 0x0c800000u || t == 0u;
}
// The others: no rest behind a number that is not finite; the first part towards zero where rounding leaves the range; a number so small that a part leaves
// the normal numbers (bfloat16's last bit is 2^-133, float32's 2^-149) goes on as NaN, and its outputs with it: they are then worked out from the operands.
__device__ __noinline__ void cut3_other(float v, uint32_t& a, uint32_t& b, uint32_t& c) {
    const uint32_t u = __float_as_uint(v);
    b = c = 0u;
    a = u >> 16;
    if ((u & 0x7f800000u) == 0x7f800000u) { if (u & 0x007fffffu) a = 0x7fc0u; return; }
    if ((u & 0x7fffffffu) >= 0x7f7f8000u) {
        const float r = v - __uint_as_float(u & 0xffff0000u);
        b = nearest2(r, 0.f);
        c = nearest2(r - __uint_as_float(b << 16), 0.f);
        return;
    }
    cut3(v, 0.f, a, b, c);
    auto too_small = [](uint32_t p) { return (p & 0x7f80u) == 0u && (p & 0x007fu) != 0u; };
    const float rest = (v - __uint_as_float(a << 16)) - __uint_as_float(b << 16);
    if (too_small(a) || too_small(b) || too_small(c) || rest != __uint_as_float(c << 16)) { a = 0x7fc0u; b = c = 0u; }
}

// src [rows, K] -> dst [Kp / 64][row blocks][3 planes][block rows][64]: what one stage of the product reads of one block of rows is one stretch
// of memory.  A warp takes 4 rows x 64 numbers of K (a thread eight numbers): it reads 256 bytes of a row and writes 512 in a row three times.
__global__ void __launch_bounds__(256) split_kernel(const float* __restrict__ src, bf16* __restrict__ dst, int rows, int K, int chunks, int block,
                                                    int row_blocks, bool vec_ok) {
    pdl_enter();
    const int lane = threadIdx.x & 31, r_in = lane >> 3, piece = lane & 7;
    const int64_t items = (int64_t)((rows + 3) >> 2) * chunks, step = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t it = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += step) {
        const int g = (int)(it / chunks), kc = (int)(it - (int64_t)g * chunks), row = g * 4 + r_in, k = kc * SP_BK + piece * 8;
        if (row >= rows) continue;                            // (rows that pad a block hold whatever was there: they feed outputs that are not stored)
        const float* p = src + (int64_t)row * K + k;
        float v[8];
        if (vec_ok && k + 8 <= K) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + 4);
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = k + i < K ? p[i] : 0.f;
        }
        uint32_t o[3][4];
        bool plain = true;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            cut3(v[2 * i], v[2 * i + 1], o[0][i], o[1][i], o[2][i]);
            plain = plain && ordinary(v[2 * i]) && ordinary(v[2 * i + 1]);
        }
        if (!plain) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t lo[3], hi[3];
                cut3_other(v[2 * i], lo[0], lo[1], lo[2]);
                cut3_other(v[2 * i + 1], hi[0], hi[1], hi[2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) o[j][i] = lo[j] | hi[j] << 16;
            }
        }
        const int rb = row / block;
        bf16* d = dst + ((((int64_t)kc * row_blocks + rb) * 3) * block + (row - rb * block)) * SP_BK + piece * 8;
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint4*>(d + (int64_t)j * block * SP_BK) = make_uint4(o[j][0], o[j][1], o[j][2], o[j][3]);
    }
}

// --------------------------------------------------------------------------- product

// item -> (tile of w, tile of tokens, chunks of K, share); tokens fastest, so that the pairs of a wave share panels of w
struct SpItem { int tile_w, tile_x, split, k_lo, k_hi; };             // split: -1 for all of K
__device__ __forceinline__ SpItem sp_item(const SpParams& p, int item) {
    SpItem t{0, 0, -1, 0, p.k_tiles};
    if (item >= p.whole) {
        t.split = (item - p.whole) / p.shared;
        item -= t.split * p.shared;
        t.k_lo = t.split * p.k_per_split;
        t.k_hi = min(p.k_tiles, t.k_lo + p.k_per_split);
    }
    t.tile_w = item / p.tiles_m;
    t.tile_x = item - t.tile_w * p.tiles_m;
    return t;
}

template <int BN>
__global__ void __launch_bounds__(SP_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ SpParams p) {
    constexpr int BNH = BN / 2;                                   // tokens a block loads; tokens a thread adds up
    constexpr uint32_t B_PLANE = BNH * 128u, STAGE = 3 * SP_A_PLANE + 3 * B_PLANE;
    constexpr int ACCS = 512 / BN < SP_MAX_ACCS ? 512 / BN : SP_MAX_ACCS, TMEM_COLS = ACCS * BN;
    extern __shared__ unsigned char smem_dyn[];
    __shared__ __align__(8) uint64_t full[SP_MAX_STAGES], empty[SP_MAX_STAGES], acc_full[SP_MAX_ACCS], acc_empty[SP_MAX_ACCS];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag, again;                             // again: an output of this block is not finite

    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int S = p.stages;
    volatile int* abort_p = &abort_flag;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        abort_flag = again = 0;
        for (int s = 0; s < SP_MAX_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < SP_MAX_ACCS; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }     // eight warps of two blocks
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    pdl_wait();

    if (warp == 0) {
        int s = 0;
        uint32_t round = 0;
        const uint32_t bar0 = cluster_addr(smem_u32(&full[0]), 0);
        bool ok = true;
        for (int item = pair; item < p.num_items && ok; item += pairs) {
            const SpItem t = sp_item(p, item);
            const int block_w = t.tile_w * 2 + (int)rank, block_x = t.tile_x * 2 + (int)rank;
            for (int kt = t.k_lo; kt < t.k_hi; ++kt) {
                if (round > 0 && !__all_sync(0xffffffffu, mbar_wait(&empty[s], (round - 1) & 1, abort_p))) { ok = false; break; }
                if (elect_one()) {
                    if (rank == 0) mbar_expect_tx(&full[s], 2 * STAGE);
                    const uint32_t bar = bar0 + (uint32_t)s * 8u, dst = base + (uint32_t)s * STAGE;
                    const int at_w = (kt * p.blocks_w + block_w) * 384, at_x = (kt * p.blocks_x + block_x) * 3 * BNH;
                    sp_tma_load(dst, &map_w, bar, 0, at_w);
                    sp_tma_load(dst + 192 * 128, &map_w, bar, 0, at_w + 192);
                    sp_tma_load(dst + 3 * SP_A_PLANE, &map_x, bar, 0, at_x);
                    if constexpr (BN == 256) sp_tma_load(dst + 3 * SP_A_PLANE + 192 * 128, &map_x, bar, 0, at_x + 192);
                }
                __syncwarp();
                if (++s == S) { s = 0; ++round; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = umma_idesc_bf16(256, BN);
            int s = 0;
            uint32_t round = 0, chunk = 0;
            bool ok = true;
            for (int item = pair; item < p.num_items && ok; item += pairs) {
                const SpItem it = sp_item(p, item);
                for (int kt = it.k_lo; kt < it.k_hi; ++kt, ++chunk) {
                    const uint32_t buf = chunk % ACCS, use = chunk / ACCS;
                    if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], (use - 1) & 1, abort_p))) { ok = false; break; }
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[s], round & 1, abort_p))) { ok = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t at = base + (uint32_t)s * STAGE;
                        const uint64_t da = umma_desc_sw128(at), db = umma_desc_sw128(at + 3 * SP_A_PLANE);
                        const uint32_t d_at = tmem_base + buf * (uint32_t)BN;
                        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};       // the parts' products, small ones first
#pragma unroll
                        for (int t = 0; t < 6; ++t)
#pragma unroll
                            for (int ks = 0; ks < SP_BK / 16; ++ks)
                                sp_mma(d_at, da + (uint64_t)(PA[t] * (SP_A_PLANE >> 4) + ks * 2), db + (uint64_t)(PB[t] * (B_PLANE >> 4) + ks * 2),
                                       idesc, t > 0 || ks > 0);
                        sp_commit(&empty[s]);
                        sp_commit(&acc_full[buf]);
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ++round; }
                }
            }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * BNH);
        const uint32_t acc_empty_leader = cluster_addr(smem_u32(&acc_empty[0]), 0);
        uint32_t chunk = 0;
        bool ok = true;
        for (int item = pair; item < p.num_items && ok; item += pairs) {
            const SpItem ks = sp_item(p, item);
            const uint32_t end = chunk + (uint32_t)(ks.k_hi - ks.k_lo);
            float acc[BNH];
#pragma unroll
            for (int i = 0; i < BNH; ++i) acc[i] = 0.f;
            for (; chunk < end; ++chunk) {
                const uint32_t buf = chunk % ACCS, use = chunk / ACCS;
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[buf], use & 1, abort_p))) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < BNH; c += 32) {
                    float v[32];
                    sp_ld32(lane_addr + buf * (uint32_t)BN + (uint32_t)c, v);
#pragma unroll
                    for (int i = 0; i < 32; ++i) acc[c + i] += v[i];
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) sp_arrive_cluster(acc_empty_leader + buf * 8u);
            }
            if (!ok) break;
            asm volatile("" : "+r"(item));                        // (worked out again: the loop above has no registers for it)
            const SpItem t = sp_item(p, item);
            const int n = t.tile_w * 256 + (int)rank * 128 + q * 32 + lane, m0 = t.tile_x * BN + half * BNH;
            if (n < p.N) {
                if (t.split >= 0) {
                    float* o = p.partial + ((int64_t)t.split * p.M + m0) * p.cols + n;
#pragma unroll
                    for (int i = 0; i < BNH; ++i) if (m0 + i < p.M) o[(int64_t)i * p.cols] = acc[i];
                } else {
                    const float b = p.bias ? load_tagged(p.bias, n, p.bias_tag) : 0.f;
                    float* o = p.out + (int64_t)m0 * p.out_stride + n;
                    bool fine = true;
#pragma unroll
                    for (int i = 0; i < BNH; ++i) {
                        fine = fine && (m0 + i >= p.M || is_finite_f32(acc[i]));
                        if (m0 + i < p.M) o[(int64_t)i * p.out_stride] = acc[i] + b;
                    }
                    if (!fine) again = 1;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.error, 1);
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    } else if (again) {                                            // (every copy has arrived and every MMA has read it: the stages' memory is free)
        float* sm = reinterpret_cast<float*>(smem_dyn + (base - smem_u32(smem_dyn)));
        for (int item = pair; item < p.whole; item += pairs)
            sp_again(p, sm, (item % p.tiles_m) * BN, BN, (item / p.tiles_m) * 256 + (int)rank * 128, 128);
    }
    cluster_sync_all();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// The shares of K added up in order: a block 128 columns of 2 V tokens, a thread V columns next to one another.
template <int V>
__global__ void __launch_bounds__(256, 7) split_sum_kernel(const __grid_constant__ SpParams p) {
    __shared__ float sm[SP_AGAIN_FLOATS];
    pdl_enter();
    constexpr int TOKENS = 2 * V;
    const int tiles_n = (p.cols + 127) / 128, m0 = (int)(blockIdx.x / tiles_n) * TOKENS, n0 = p.n_shared + (int)(blockIdx.x % tiles_n) * 128;
    const int m = m0 + threadIdx.x / (128 / V), n = n0 + threadIdx.x % (128 / V) * V;
    bool fine = true;
    if (m < p.M && n < p.N) {
        const int64_t per = (int64_t)p.M * p.cols;
        const float* src = p.partial + (int64_t)m * p.cols + n;
        float v[V];
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = 0.f;
        for (int s = 0; s < p.splits; ++s) {
            float u[V];
            if constexpr (V == 4) *reinterpret_cast<float4*>(u) = __ldcg(reinterpret_cast<const float4*>(src + s * per));
            else u[0] = __ldcg(src + s * per);
#pragma unroll
            for (int i = 0; i < V; ++i) v[i] += u[i];
        }
#pragma unroll
        for (int i = 0; i < V; ++i) {
            fine = fine && is_finite_f32(v[i]);
            if (p.bias) v[i] += load_tagged(p.bias, n + i, p.bias_tag);
            p.out[(int64_t)m * p.out_stride + n + i] = v[i];
        }
    }
    if (__syncthreads_or(!fine)) sp_again(p, sm, m0, TOKENS, n0, 128);
}

// --------------------------------------------------------------------------- host side

static int sp_map(CUtensorMap* map, const void* ptr, int64_t rows, int box_rows) {
    cuuint64_t gdim[2] = {SP_BK, (cuuint64_t)rows};
    cuuint64_t gstride[1] = {SP_BK * 2};
    cuuint32_t box[2] = {SP_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 1000 + (int)r;
}

// src [rows, K] float32 -> dst: see split_kernel.  `block` rows a block (a multiple of 8); dst holds ceil(K / 64) * `row_blocks` * 3 * block * 64 numbers, 16-byte
// aligned, and row_blocks * block >= rows.
extern "C" int mie_split3(const float* src, void* dst, int rows, int K, int block, int row_blocks, cudaStream_t stream) {
    if (rows <= 0 || K <= 0) return 0;
    if (block < 8 || block % 8 || (int64_t)row_blocks * block < rows || (reinterpret_cast<uintptr_t>(dst) & 15)) return MIE_ERR_BAD_ARG;
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && K % 4 == 0;
    const int chunks = (K + SP_BK - 1) / SP_BK;
    const int64_t blocks = ((int64_t)((rows + 3) / 4) * chunks + 7) / 8, most = (int64_t)device_sm_count() * 16;
    return launch_kernel(split_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, stream, src, (bf16*)dst, rows, K, chunks, block, row_blocks, vec);
}

template <int BN>
static int sp_launch(const CUtensorMap& mw, const CUtensorMap& mx, SpParams& p, cudaStream_t stream) {
    constexpr int STAGE = 3 * (int)SP_A_PLANE + 3 * (BN / 2) * 128;
    p.stages = 226 * 1024 / STAGE < SP_MAX_STAGES ? 226 * 1024 / STAGE : SP_MAX_STAGES;
    const int smem = p.stages * STAGE + 1024;
    const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    int pairs = device_sm_count() / 2;
    if (pairs > p.num_items) pairs = p.num_items;
    return launch_kernel_cluster(gemm_split_kernel<BN>, dim3(2 * pairs), dim3(SP_THREADS), smem, stream, dim3(2, 1, 1), mw, mx, p);
}

// y (columns of a matrix with `y_stride` columns) from the planes xs (blocks of bn / 2 rows) and ws (blocks of 128 rows), both an even number of blocks, of
// x [M, K], w [N, K] float32 row-major.  bn 64, 128 or 256 tokens a tile; the first `whole` tiles of 256 rows of w take all of K at once, those behind them
// `splits` shares of K (1: no partial, and `whole` does not count); partial [splits][M][N - 256 whole] float32.
extern "C" int mie_gemm_split(const void* xs, const void* ws, const float* x, const float* w, const void* bias, int bias_tag, float* y,
                              long long y_stride, float* partial, int M, int N, int K, int bn, int splits, int whole,
                              cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    const int chunks = (K + SP_BK - 1) / SP_BK, blocks_w = (N + 255) / 256 * 2, blocks_x = bn > 0 ? (M + bn - 1) / bn * 2 : 0;
    if (K <= 0 || (bn != 64 && bn != 128 && bn != 256) || splits < 1 || splits > chunks || (splits > 1 && (!partial || whole < 0 || whole >= (N + 255) / 256))) return MIE_ERR_BAD_ARG;
    if (((reinterpret_cast<uintptr_t>(xs) | reinterpret_cast<uintptr_t>(ws)) & 127) || (reinterpret_cast<uintptr_t>(partial) & 15)) return MIE_ERR_BAD_ARG;
    const int64_t rows_w = (int64_t)chunks * blocks_w * 384, rows_x = (int64_t)chunks * blocks_x * 3 * (bn / 2);
    if (rows_w > 0x7fffffff || rows_x > 0x7fffffff) return MIE_ERR_TOO_LARGE;
    int rc = tc_setup();
    if (rc) return rc;
    CUtensorMap mw, mx;
    if ((rc = sp_map(&mw, ws, rows_w, 192))) return rc;
    if ((rc = sp_map(&mx, xs, rows_x, bn == 64 ? 96 : 192))) return rc;
    SpParams p{};
    p.out = y; p.out_stride = y_stride; p.bias = bias; p.bias_tag = bias_tag; p.partial = partial; p.x = x; p.w = w;
    p.M = M; p.N = N; p.K = K; p.k_tiles = chunks; p.blocks_w = blocks_w; p.blocks_x = blocks_x; p.error = g_error_dev;
    p.k_per_split = (p.k_tiles + splits - 1) / splits;
    p.splits = (p.k_tiles + p.k_per_split - 1) / p.k_per_split;       // no empty share
    p.tiles_m = (M + bn - 1) / bn;
    const int tiles = p.tiles_m * ((N + 255) / 256);
    p.whole = p.splits > 1 ? whole * p.tiles_m : tiles;
    p.shared = tiles - p.whole;
    p.n_shared = p.splits > 1 ? whole * 256 : 0;
    p.cols = N - p.n_shared;
    if (partial) p.partial = partial - p.n_shared;
    p.num_items = p.whole + p.shared * p.splits;
    rc = bn == 64 ? sp_launch<64>(mw, mx, p, stream) : bn == 128 ? sp_launch<128>(mw, mx, p, stream) : sp_launch<256>(mw, mx, p, stream);
    if (rc || p.splits == 1) return rc;
    const unsigned tiles_n = (unsigned)((p.cols + 127) / 128);
    if (N % 4 == 0) return launch_kernel(split_sum_kernel<4>, dim3(tiles_n * (unsigned)((M + 7) / 8)), dim3(256), 0, stream, p);
    return launch_kernel(split_sum_kernel<1>, dim3(tiles_n * (unsigned)((M + 1) / 2)), dim3(256), 0, stream, p);
}

extern "C" int mie_gemm_split_error(void) { return g_error_host ? *g_error_host : 0; }
extern "C" void mie_gemm_split_clear_error(void) { if (g_error_host) *g_error_host = 0; }
