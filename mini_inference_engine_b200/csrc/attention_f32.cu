// Paged causal attention of prompt portions in float32 (the true 32-bit path): rows with many new tokens; csrc/attention_simt.cu serves the
// others, and every row in bfloat16.  The same rules: masks, kept first keys, score modifiers, sink, range checks; float32 fused multiply-adds throughout.
//
// A block owns 64 (token, query head) pairs that share a key head -- tokens of one row, the group's heads side by side -- so a tile of
// 64 keys and values in shared memory serves all heads of the group.  A thread holds 8 (or 4) pairs x 4 keys of the scores and
// the same pairs x 4 (or 8) entries of the output, where a warp that owns one pair reads its keys and values once per pair.  The next tile's keys arrive
// (cp.async) under the product with the values, the next values under the scores.  Tiles of a row go longest first.  Bound: latencies at three warps a
// scheduler -- 640 tokens of 32 heads of 64 (156 us under the profiler): a scheduler has an instruction to issue in 45 % of the cycles, the multiply-add pipe is at 32 %
// of its peak, L1 and shared memory at 30 %.  A layer of TinyLlama's sizes over 1,000 tokens of two requests, products included: 958 us with the other kernel -> 318 us.
#include "common.cuh"
#include "range_check.cuh"

#define MIE_K_ATTENTION_F32 14     // this kernel's number in the range report (csrc/range_check.cuh)
#define F32_PAIRS 64
#define F32_KEYS 64
#define F32_PS 80                 // stride of a row of probabilities: neighbouring rows 16 banks apart

struct F32Params {
    const float* q; int64_t q_stride; const float* k_cache; const float* v_cache;
    const int* block_tables; int table_stride;
    const int* row_q_start; const int* row_q_len; const int* row_ctx_len; int num_rows;
    float* out; int num_heads, num_kv_heads, head_dim, page_size, page_shift; float scale; int window, keep, min_q_len;
    int64_t num_pages; int* report; ScoreMods mods;
};

__device__ __forceinline__ void f32_copy16(float* dst, const float* src, bool on) {       // zeros where `on` is false (nothing is read then)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}

template <bool B> struct Bool { static constexpr bool value = B; };

// DT: entries of a head as the block holds them (head_dim padded with zeros); THREADS 128 or 256; the probabilities take the keys' memory
// where SHARE (two blocks on an SM at DT 128).
template <int DT, int THREADS, bool SHARE>
__global__ void __launch_bounds__(THREADS, DT == 64 ? 3 : 2) f32_attention_kernel(const F32Params p) {
    constexpr int TY = THREADS / 16, RI = F32_PAIRS / TY, QS = DT + 4, KS = DT + 4, CG = DT / 64;
    extern __shared__ __align__(16) float sm[];
    float* Q = sm;                                    // [64][QS]
    float* K = Q + F32_PAIRS * QS;                    // [64][KS]
    float* V = K + F32_KEYS * KS;                     // [64][DT]
    float* P = SHARE ? K : V + F32_KEYS * DT;         // [64][F32_PS]
    __shared__ int s_row, s_tile;
    const int D = p.head_dim, G = p.num_heads / p.num_kv_heads, kvh = blockIdx.y;
    pdl_launch_dependents();
    if (threadIdx.x < 32) {
        int within, items;
        const int found = warp_find_row(p.row_q_len, p.num_rows, (int)blockIdx.x,
                                        [&](int n) { return n >= p.min_q_len ? (n * G + F32_PAIRS - 1) / F32_PAIRS : 0; }, within, items);
        if (threadIdx.x == 0) { s_row = found; s_tile = items - 1 - within; }
    }
    __syncthreads();
    const int r = s_row;
    pdl_wait();                                       // (a block without work waits too: see common.cuh)
    if (r < 0) return;
    const int q_len = p.row_q_len[r], ctx_len = p.row_ctx_len[r], q_start = p.row_q_start[r], pair0 = s_tile * F32_PAIRS;
    if (ctx_len > p.table_stride * p.page_size) {
        if (threadIdx.x == 0) range_report(p.report, MIE_RANGE_POSITION, MIE_K_ATTENTION_F32, r, ctx_len);
        return;
    }
    const int lane = threadIdx.x & 31, tx = lane & 15, ty = (threadIdx.x >> 5) * 2 + (lane >> 4);
    const int pairs = q_len * G, last = min(pair0 + F32_PAIRS, pairs) - 1, base_pos = ctx_len - q_len;
    const int first_pos = base_pos + pair0 / G, last_pos = base_pos + last / G;
    const int k_hi = last_pos + 1, k_lo = mask_first_key(first_pos, p.window);

    for (int i = threadIdx.x; i < F32_PAIRS * (DT / 4); i += THREADS) {
        const int pr = i / (DT / 4), d = (i - pr * (DT / 4)) * 4, at = pair0 + pr;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (at < pairs && d < D) {
            const int token = q_start + at / G, head = kvh * G + at % G;
            const float* src = p.q + (int64_t)token * p.q_stride + (int64_t)head * D + d;
            v = make_float4(src[0] * p.scale, src[1] * p.scale, src[2] * p.scale, src[3] * p.scale);
        }
        *reinterpret_cast<float4*>(Q + pr * QS + d) = v;
    }
    int pos[RI], head[RI];
    float m[RI], l[RI], o[RI][4 * CG];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int at = pair0 + ty + TY * i;
        pos[i] = at < pairs ? base_pos + at / G : -1;              // (a pair that does not exist reads no key)
        head[i] = kvh * G + at % G;
        m[i] = -INFINITY;
        l[i] = 0.f;
        if (p.mods.sink && at < pairs) { m[i] = p.mods.sink[head[i]]; l[i] = tx == 0 ? 1.f : 0.f; }
#pragma unroll
        for (int c = 0; c < 4 * CG; ++c) o[i][c] = 0.f;
    }
    const int* table = p.block_tables + (int64_t)r * p.table_stride;
    const int kbeg = k_lo & ~(F32_KEYS - 1), kept = mask_kept_tiles(p.keep, kbeg, F32_KEYS);
    const int tiles = kept + (k_hi - kbeg + F32_KEYS - 1) / F32_KEYS;
    auto tile_key = [&](int t) { return t < kept ? t * F32_KEYS : kbeg + (t - kept) * F32_KEYS; };
    auto issue = [&](const float* cache, float* dst, int stride, int t) {
        if (t < tiles) {
            const int k0 = tile_key(t);
#pragma unroll 4
            for (int i = threadIdx.x; i < F32_KEYS * (DT / 4); i += THREADS) {
                const int jj = i / (DT / 4), d = (i - jj * (DT / 4)) * 4, key = k0 + jj;
                const bool on = (key >= k_lo || key < p.keep) && key < k_hi && d < D;
                const float* src = cache;
                if (on) {
                    const int page = checked_page(table[key >> p.page_shift], p.num_pages, p.report, MIE_K_ATTENTION_F32, key >> p.page_shift);
                    src = cache + (((int64_t)page * p.num_kv_heads + kvh) * p.page_size + (key & (p.page_size - 1))) * D + d;
                }
                f32_copy16(dst + jj * stride + d, src, on);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");       // every thread one group, also an empty one
    };
    const bool plain = !(p.mods.softcap > 0.f) && !p.mods.dist_bias && !p.mods.slope;
    issue(p.k_cache, K, KS, 0);
    issue(p.v_cache, V, DT, 0);
    for (int t = 0; t < tiles; ++t) {
        const int k0 = tile_key(t);
        asm volatile("cp.async.wait_group 1;" ::: "memory");       // this tile's keys (its values may still be on the way)
        __syncthreads();
        float s[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
        for (int d = 0; d < DT; d += 4) {
            float4 kk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const float4*>(K + (tx + 16 * j) * KS + d);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                const float4 qq = *reinterpret_cast<const float4*>(Q + (ty + TY * i) * QS + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(qq.x, kk[j].x, s[i][j]);
                    s[i][j] = fmaf(qq.y, kk[j].y, s[i][j]);
                    s[i][j] = fmaf(qq.z, kk[j].z, s[i][j]);
                    s[i][j] = fmaf(qq.w, kk[j].w, s[i][j]);
                }
            }
        }
        if constexpr (SHARE) __syncthreads();                      // the keys are done with: their memory takes the probabilities
        // a tile that every pair sees whole needs no mask: all keys at or before the first pair's position, none before the last one's first key
        const bool whole = k0 + F32_KEYS - 1 <= first_pos && k0 >= mask_first_key(last_pos, p.window) && last - pair0 == F32_PAIRS - 1;
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            float top = -INFINITY;
            int unseen = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + tx + 16 * j;
                if (!plain) s[i][j] = mod_score(s[i][j], p.mods, head[i], p.num_heads, pos[i] - key);
                if (!whole && !mask_reads(pos[i], key, p.window, p.keep)) { s[i][j] = -INFINITY; unseen |= 1 << j; }
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
            const float m_new = fmaxf(m[i], top);
            const bool any = m_new > -INFINITY;                    // else every key so far is masked for this pair
            const float alpha = any ? expf(m[i] - m_new) : 1.f;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = any ? expf(s[i][j] - m_new) : 0.f;
                sum += e;
                P[(ty + TY * i) * F32_PS + tx + 16 * j] = (unseen >> j) & 1 ? -1.f : e;
            }
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * CG; ++c) o[i][c] *= alpha;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");       // the values
        __syncthreads();
        if constexpr (!SHARE) issue(p.k_cache, K, KS, t + 1);
        auto add_values = [&](auto masked) {
#pragma unroll 2
        for (int kk = 0; kk < F32_KEYS; kk += 4) {
            float4 pp[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) pp[i] = *reinterpret_cast<const float4*>(P + (ty + TY * i) * F32_PS + kk);
#pragma unroll
            for (int c = 0; c < CG; ++c) {
                float4 v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float4*>(V + (kk + e) * DT + 64 * c + 4 * tx);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    float* oo = o[i] + 4 * c;
                    const float pe[4] = {pp[i].x, pp[i].y, pp[i].z, pp[i].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (decltype(masked)::value && pe[e] < 0.f) continue;         // a key out of sight: its value may be anything
                        oo[0] = fmaf(pe[e], v[e].x, oo[0]);
                        oo[1] = fmaf(pe[e], v[e].y, oo[1]);
                        oo[2] = fmaf(pe[e], v[e].z, oo[2]);
                        oo[3] = fmaf(pe[e], v[e].w, oo[3]);
                    }
                }
            }
        }
        };
        if (whole) add_values(Bool<false>{});
        else add_values(Bool<true>{});
        __syncthreads();
        if constexpr (SHARE) issue(p.k_cache, K, KS, t + 1);
        issue(p.v_cache, V, DT, t + 1);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        float sum = l[i];
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
        if (pos[i] < 0) continue;
        float* op = p.out + ((int64_t)(q_start + pos[i] - base_pos) * p.num_heads + head[i]) * D;
#pragma unroll
        for (int c = 0; c < CG; ++c) {
            const int d = 64 * c + 4 * tx;
            if (d < D) *reinterpret_cast<float4*>(op + d) = make_float4(o[i][4 * c] * inv, o[i][4 * c + 1] * inv, o[i][4 * c + 2] * inv, o[i][4 * c + 3] * inv);
        }
    }
}

template <int DT, int THREADS, bool SHARE>
static int f32_launch(const F32Params& p, dim3 grid, cudaStream_t stream) {
    const int smem = (F32_PAIRS * (DT + 4) + F32_KEYS * (DT + 4) + F32_KEYS * DT + (SHARE ? 0 : F32_PAIRS * F32_PS)) * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(f32_attention_kernel<DT, THREADS, SHARE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    return launch_kernel(f32_attention_kernel<DT, THREADS, SHARE>, grid, dim3(THREADS), smem, stream, p);
}

// Rows with fewer than `min_q_len` new tokens are left alone; `tiles`: an upper bound of the 64-pair tiles of the others.  Heads of 16 .. 128 in steps
// of 16, caches and out 16-byte aligned; the rest as mie_paged_attention.
extern "C" int mie_attention_f32(const float* q, int64_t q_stride, const float* k_cache, const float* v_cache, const int* block_tables, int table_stride,
                                 const int* row_q_start, const int* row_q_len, const int* row_ctx_len, int num_rows, int tiles, float* out,
                                 int num_heads, int num_kv_heads, int head_dim, int page_size, float scale, int window, int keep, int min_q_len,
                                 long long num_pages, float softcap, const float* sink, const float* dist_bias, int dist_len, const float* slope,
                                 cudaStream_t stream) {
    if (num_rows <= 0 || tiles <= 0) return 0;
    if (head_dim < 16 || head_dim > 128 || head_dim % 16 || min_q_len < 1 || (dist_bias && dist_len <= 0)) return MIE_ERR_BAD_ARG;
    if (num_kv_heads <= 0 || num_heads % num_kv_heads || page_size < 1 || (page_size & (page_size - 1))) return MIE_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(out)) & 15) return MIE_ERR_BAD_ARG;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    const F32Params p{q, q_stride, k_cache, v_cache, block_tables, table_stride, row_q_start, row_q_len, row_ctx_len, num_rows, out, num_heads,
                      num_kv_heads, head_dim, page_size, page_shift, scale, window, keep, min_q_len, (int64_t)num_pages, g_range_report,
                      ScoreMods{softcap, sink, dist_bias, dist_len, slope}};
    const dim3 grid(tiles, num_kv_heads);
    return head_dim <= 64 ? f32_launch<64, 128, false>(p, grid, stream) : f32_launch<128, 256, true>(p, grid, stream);
}
