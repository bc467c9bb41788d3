// Paged causal attention in float32 (the true 32-bit path) by tiles of (token, head) pairs: rows with many new tokens, and on long contexts rows of a few and of one (the line is
// drawn in kernels/attention.py); csrc/attention_simt.cu, a warp a pair, serves the others, and every row in bfloat16.  The same rules: masks, kept first keys, score modifiers, sink, range checks.  Scores and outputs are products on the tensor cores
// with every operand as three bfloat16 parts (triple_mma.cuh); weights, sums and everything else are float32.
//
// A block owns 16 (token, query head) pairs a warp that share a key head -- tokens of one row, the group's heads side by side -- so a tile of
// 64 keys and values in shared memory serves all heads of the group.  Queries, keys and values lie there as parts, split by the threads that fetched them; the scores of a
// warp's pairs become the left operand of the product with the values where they are.  A walk of keys may be shared out over the blocks of a cluster, every n-th tile a block;
// their sums meet in shared memory.  A tile whose scores in sight are all NaN counts as out of sight for a pair that has met no number yet and makes its output NaN behind the
// first number; so that the shares decide as one walk does, each keeps the first tile where a pair met a number and the last one that it passed over.  The next tile's keys arrive (cp.async) under the product with the
// values, the values under the scores.  Tiles of a row go longest first, over all heads.
//
// A tile with keys or values that have no three parts (not finite, or beyond 2^127) is multiplied number by number, and a weight that does not exist then meets no value.
//
// Bound: the tensor pipe while a tile's products run (8.2 cycles an instruction with four warps a scheduler, 8 its rate), about 60 % of the time; the rest are the softmax, the
// splitting and the blocks' ends.  Kernel, us: 333 tokens on 300 positions beside 667, 32 heads of 64: 177 (register tiles on the CUDA cores) -> 94; 1,024 tokens 128; a layer of
// TinyLlama's sizes over both rows, products included, 314 -> 230; 200 tokens on 800 positions 320 -> 120.  Against 64 bits the layer is 2.7e-7 off (2-norm), 3.6e-7 before.
#include <algorithm>
#include <cmath>

#include "range_check.cuh"
#include "triple_mma.cuh"

#define MIE_K_ATTENTION_F32 14     // this kernel's number in the range report (csrc/range_check.cuh)
#define F32_KEYS 64

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

__device__ __noinline__ float f32_dot(const float* q, const float* k, int D, float scale) {
    float sum = 0.f;
    for (int d = 0; d < D; ++d) sum = fmaf(q[d] * scale, k[d], sum);
    return sum;
}

// DT: entries of a head as the block holds them (head_dim padded with zeros); WARPS of 16 pairs each.
// Blocks of 4 warps over heads of 65 to 128 have no memory for keys on their way if two are to fit on an SM: they fetch a tile when they split it, from L2 (asked for ahead), under
// the other block's products.
template <int DT, int WARPS> constexpr bool f32_direct = DT == 128 && WARPS == 4;
template <int DT, int WARPS> constexpr int f32_bytes() { return 3 * 16 * WARPS * DT * 2 + 3 * F32_KEYS * DT * 2 + (f32_direct<DT, WARPS> ? 0 : F32_KEYS * DT * 4); }
template <int DT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, DT == 128 ? 8 / WARPS : WARPS == 4 ? 3 : 2) f32_attention_kernel(const F32Params p, int splits) {
    constexpr int GROUP = WARPS == 4 && DT == 64 ? 4 : 2;         // column tiles at a time: as many as the registers have room for
    constexpr int THREADS = 32 * WARPS, PAIRS = 16 * WARPS, Q_PLANE = PAIRS * DT * 2, K_PLANE = F32_KEYS * DT * 2, KS = DT / 16, NT = DT / 8;
    constexpr int QUADS = F32_KEYS * DT / 4 / THREADS, STEP = THREADS / (DT / 4);
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* Q = smem;                                // [PAIRS][DT] as parts
    uint8_t* KV = Q + 3 * Q_PLANE;                    // keys, then values [64][DT]; then weights [16][32] a warp where a tile is multiplied number by number
    float* raw = reinterpret_cast<float*>(KV + 3 * K_PLANE);       // keys or values on their way [64][DT]: a thread splits what it fetched
    __shared__ int s_row, s_tile, s_page[2][F32_KEYS];             // the pages of a tile's keys (-1: a key that nobody reads), the next tile's besides
    __shared__ int s_number[PAIRS], s_none[PAIRS];                 // a pair's first tile with a number; the last one of NaN that it passed over
    const int share = blockIdx.x % splits, item = blockIdx.x / splits;
    const int D = p.head_dim, G = p.num_heads / p.num_kv_heads, kvh = item % p.num_kv_heads;
    pdl_launch_dependents();
    if (threadIdx.x < 32) {
        int within, items;
        const int found = warp_find_row(p.row_q_len, p.num_rows, item / p.num_kv_heads,
                                        [&](int n) { return n >= p.min_q_len ? (n * G + PAIRS - 1) / PAIRS : 0; }, within, items);
        if (threadIdx.x == 0) { s_row = found; s_tile = items - 1 - within; }
    }
    __syncthreads();
    const int r = s_row;
    pdl_wait();                                       // (a block without work waits too: see common.cuh)
    if (r < 0) return;
    const int q_len = p.row_q_len[r], ctx_len = p.row_ctx_len[r], q_start = p.row_q_start[r], pair0 = s_tile * PAIRS;
    if (ctx_len > p.table_stride * p.page_size) {
        if (threadIdx.x == 0) range_report(p.report, MIE_RANGE_POSITION, MIE_K_ATTENTION_F32, r, ctx_len);
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = lane >> 2, c0 = (lane & 3) * 2;
    const int pairs = q_len * G, last = min(pair0 + PAIRS, pairs) - 1, base_pos = ctx_len - q_len;
    const int first_pos = base_pos + pair0 / G, last_pos = base_pos + last / G;
    const int k_hi = last_pos + 1, k_lo = mask_first_key(first_pos, p.window);
    const int* table = p.block_tables + (int64_t)r * p.table_stride;
    const int kbeg = k_lo & ~(F32_KEYS - 1), kept = mask_kept_tiles(p.keep, kbeg, F32_KEYS);
    const int tiles = kept + (k_hi - kbeg + F32_KEYS - 1) / F32_KEYS;
    auto tile_key = [&](int t) { return t < kept ? t * F32_KEYS : kbeg + (t - kept) * F32_KEYS; };
    auto in_reach = [&](int key) { return (key >= k_lo || key < p.keep) && key < k_hi; };
    auto row_in = [&](const float* cache, int page, int key) { return cache + (((int64_t)page * p.num_kv_heads + kvh) * p.page_size + (key & (p.page_size - 1))) * D; };
    auto page_of = [&](int t) {                       // of this thread's key of a tile
        const int key = tile_key(t) + (int)threadIdx.x;
        return t < tiles && threadIdx.x < F32_KEYS && in_reach(key) ? checked_page(table[key >> p.page_shift], p.num_pages, p.report, MIE_K_ATTENTION_F32, key >> p.page_shift) : -1;
    };
    const int my_d = (threadIdx.x % (DT / 4)) * 4, my_row = threadIdx.x / (DT / 4);
    auto issue = [&](const float* cache, int t) {
        if (t < tiles) {
            const int k0 = tile_key(t);
#pragma unroll
            for (int i = 0; i < QUADS; ++i) {
                const int jj = my_row + i * STEP, page = s_page[(t / splits) & 1][jj];
                const bool on = page >= 0 && my_d < D;
                if constexpr (f32_direct<DT, WARPS>) {
                    if (on && (my_d & 31) == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(row_in(cache, page, k0 + jj) + my_d));
                } else f32_copy16(raw + jj * DT + my_d, on ? row_in(cache, page, k0 + jj) + my_d : cache, on);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto put = [&](uint8_t* tile, int plane, int row, int d, float4 v) {
        uint2 part[3];
        split3(v.x, v.y, part[0].x, part[1].x, part[2].x);
        split3(v.z, v.w, part[0].y, part[1].y, part[2].y);
        uint8_t* at = tile + tile_at<DT>(row, d >> 3) + (d & 4) * 2;
#pragma unroll
        for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(at + j * plane) = part[j];
        return magnitude(v);
    };
    auto split = [&](const float* cache, int t) {     // what this thread fetched, once every warp is done with what lay there; whether a number of the block's has no parts
        uint32_t most = 0;
        if constexpr (f32_direct<DT, WARPS>) {
            constexpr int AHEAD = 8;                  // quads asked for before the first is split
            __syncthreads();
            const int k0 = tile_key(t);
#pragma unroll
            for (int first = 0; first < QUADS; first += AHEAD) {
                float4 v[AHEAD];
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) {
                    const int jj = my_row + (first + i) * STEP, page = s_page[(t / splits) & 1][jj];
                    v[i] = page >= 0 && my_d < D ? *reinterpret_cast<const float4*>(row_in(cache, page, k0 + jj) + my_d) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < AHEAD; ++i) most = max(most, put(KV, K_PLANE, my_row + (first + i) * STEP, my_d, v[i]));
            }
            return __syncthreads_or(has_no_parts(most)) != 0;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int jj = my_row + i * STEP;
            most = max(most, put(KV, K_PLANE, jj, my_d, *reinterpret_cast<const float4*>(raw + jj * DT + my_d)));
        }
        return __syncthreads_or(has_no_parts(most)) != 0;
    };
    if (threadIdx.x < F32_KEYS) s_page[0][threadIdx.x] = page_of(share);
    __syncthreads();
    issue(p.k_cache, share);
    uint32_t q_most = 0;
    {
        constexpr int TURNS = PAIRS * (DT / 4) / THREADS;
        float4 v[TURNS];                              // (all asked for before the first is split)
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            const int at = pair0 + my_row + i * STEP, token = at / G, head = kvh * G + at - token * G;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (at < pairs && my_d < D) {
                const float* src = p.q + (int64_t)(q_start + token) * p.q_stride + (int64_t)head * D + my_d;
                v[i] = make_float4(src[0], src[1], src[2], src[3]);
            }
        }
#pragma unroll
        for (int i = 0; i < TURNS; ++i)
            q_most = max(q_most, put(Q, Q_PLANE, my_row + i * STEP, my_d, make_float4(v[i].x * p.scale, v[i].y * p.scale, v[i].z * p.scale, v[i].w * p.scale)));
    }
    // this lane's pairs: r0 and r0 + 8 of the warp's sixteen
    int pos[2], head[2], from[2];                     // (and the first position that each reads beside the kept ones)
    float m[2], l[2], o[NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int at = pair0 + warp * 16 + r0 + 8 * i;
        pos[i] = at < pairs ? base_pos + at / G : -1;              // (a pair that does not exist reads no key)
        head[i] = kvh * G + at % G;
        from[i] = mask_first_key(max(pos[i], 0), p.window);
        m[i] = -INFINITY;
        l[i] = 0.f;
        if (p.mods.sink && at < pairs && share == 0) { m[i] = p.mods.sink[head[i]]; l[i] = c0 == 0 ? 1.f : 0.f; }
        if (c0 == 0) { s_number[at - pair0] = m[i] > -INFINITY ? -1 : 0x7fffffff; s_none[at - pair0] = -1; }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
    const bool plain = !(p.mods.softcap > 0.f) && !p.mods.dist_bias && !p.mods.slope, q_bad = has_no_parts(q_most);
    const bool block_q_bad = __syncthreads_or(q_bad) != 0;
    const uint32_t q_at = (uint32_t)__cvta_generic_to_shared(Q), kv_at = (uint32_t)__cvta_generic_to_shared(KV);
    for (int t = share; t < tiles; t += splits) {
        const int k0 = tile_key(t);
        const int next_page = page_of(t + splits);
        const int* pages = s_page[(t / splits) & 1];
        const bool k_bad = split(p.k_cache, t) || block_q_bad;
        issue(p.v_cache, t);
        float s[8][4];
        // a tile that every pair sees whole needs no mask: all keys at or before the first pair's position, none before the last one's first key
        const bool whole = k0 + F32_KEYS - 1 <= first_pos && k0 >= mask_first_key(last_pos, p.window) && last - pair0 == PAIRS - 1;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
        if (!k_bad) {
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                uint32_t a[3][4];
                left_rows<DT>(a, q_at, Q_PLANE, warp, k, lane);
#pragma unroll
                for (int n = 0; n < 8; n += GROUP) {
                    uint32_t b[3][GROUP][2];
#pragma unroll
                    for (int j = 0; j < GROUP; j += 2) right_columns<DT>(b, j, kv_at, K_PLANE, k, n + j, lane);
                    triple_step<GROUP>(s + n, a, b);
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float* q = p.q + (int64_t)(q_start + max(pos[i] - base_pos, 0)) * p.q_stride + (int64_t)head[i] * D;
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int key = k0 + n * 8 + c0 + e;
                        s[n][2 * i + e] = pos[i] >= 0 && pages[key - k0] >= 0 ? f32_dot(q, row_in(p.k_cache, pages[key - k0], key), D, p.scale) : 0.f;
                    }
            }
        }
        uint32_t unseen = 0;                                       // a bit a score, of keys out of sight
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (!plain)
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) s[n][2 * i + e] = mod_score(s[n][2 * i + e], p.mods, head[i], p.num_heads, pos[i] - (k0 + n * 8 + c0 + e));
            if (!whole)
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int key = k0 + n * 8 + c0 + e;
                        if (key > pos[i] || (key < from[i] && key >= p.keep)) { s[n][2 * i + e] = -INFINITY; unseen |= 1u << (4 * n + 2 * i + e); }
                    }
            float top = fmaxf(s[0][2 * i], s[0][2 * i + 1]);
#pragma unroll
            for (int n = 1; n < 8; ++n) top = fmaxf(top, fmaxf(s[n][2 * i], s[n][2 * i + 1]));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float m_new = fmaxf(m[i], top), base = m_new > -INFINITY ? m_new : 0.f;
            if (!(m_new > -INFINITY)) {                            // every key so far is masked for this pair, or its score no number: no weights
                bool none = false;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    none |= isnan(s[n][2 * i]) || isnan(s[n][2 * i + 1]);
                    s[n][2 * i] = s[n][2 * i + 1] = -INFINITY;
                }
                if (none) s_none[warp * 16 + r0 + 8 * i] = t;
            } else if (!(m[i] > -INFINITY)) s_number[warp * 16 + r0 + 8 * i] = t;
            const float alpha = expf(m[i] - base);
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float x = expf(s[n][2 * i + e] - base);
                    sum += x;
                    s[n][2 * i + e] = x;
                }
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int n = 0; n < NT; ++n) { o[n][2 * i] *= alpha; o[n][2 * i + 1] *= alpha; }
        }
        if (threadIdx.x < F32_KEYS) s_page[(t / splits + 1) & 1][threadIdx.x] = next_page;
        const bool v_bad = split(p.v_cache, t);
        issue(p.k_cache, t + splits);
        if (!v_bad) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t a[3][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) split3(s[2 * k + (i >> 1)][2 * (i & 1)], s[2 * k + (i >> 1)][2 * (i & 1) + 1], a[0][i], a[1][i], a[2][i]);
#pragma unroll
                for (int n = 0; n < NT; n += GROUP) {
                    uint32_t b[3][GROUP][2];
#pragma unroll
                    for (int j = 0; j < GROUP; j += 2) right_rows<DT>(b, j, kv_at, K_PLANE, k, n + j, lane);
                    triple_step<GROUP>(o + n, a, b);
                }
            }
        } else {
            // half of the keys at a time: all warps' weights fit the values' parts, which nobody reads now, and stay clear of the next keys that arrive behind them
            constexpr int HALF = F32_KEYS / 2;
            static_assert(WARPS * 16 * HALF * (int)sizeof(float) <= 3 * K_PLANE, "weights written over the next keys");
            float* P = reinterpret_cast<float*>(KV) + warp * 16 * HALF;
#pragma unroll 1
            for (int j0 = 0; j0 < F32_KEYS; j0 += HALF) {
                __syncwarp();
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    if (n / 4 != j0 / HALF) continue;
#pragma unroll
                    for (int i = 0; i < 4; ++i) P[(r0 + 8 * (i >> 1)) * HALF + n % 4 * 8 + c0 + (i & 1)] = (unseen >> (4 * n + i)) & 1 ? -1.f : s[n][i];
                }
                __syncwarp();
#pragma unroll 1
                for (int j = 0; j < HALF; ++j) {
                    const int key = k0 + j0 + j, page = pages[j0 + j];
                    if (page < 0) continue;
                    const float* v = row_in(p.v_cache, page, key);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float w = P[(r0 + 8 * i) * HALF + j];
                        if (w < 0.f) continue;                     // a key out of sight: its value may be anything
#pragma unroll
                        for (int n = 0; n < NT; ++n)
#pragma unroll
                            for (int e = 0; e < 2; ++e)
                                if (n * 8 + c0 + e < D) o[n][2 * i + e] = fmaf(w, v[n * 8 + c0 + e], o[n][2 * i + e]);
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    }
    if (splits == 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (pos[i] < 0) continue;
            const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
            float* op = p.out + ((int64_t)(q_start + pos[i] - base_pos) * p.num_heads + head[i]) * D;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int d = n * 8 + c0;
                if (d < D) *reinterpret_cast<float2*>(op + d) = make_float2(o[n][2 * i] * inv, o[n][2 * i + 1] * inv);
            }
        }
        return;
    }
    // the shares of the keys meet: every block of the cluster adds up its part of the pairs
    constexpr int OS = DT + 4;
    float* sums = reinterpret_cast<float*>(smem);     // [PAIRS][OS], then a pair's largest score, sum of weights, first tile with a number, last one of NaN passed over
    float4* ends = reinterpret_cast<float4*>(sums + PAIRS * OS);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = warp * 16 + r0 + 8 * i;
        if (c0 == 0) ends[row] = make_float4(m[i], l[i], __int_as_float(s_number[row]), __int_as_float(s_none[row]));
#pragma unroll
        for (int n = 0; n < NT; ++n) *reinterpret_cast<float2*>(sums + row * OS + n * 8 + c0) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
    }
    cluster_sync_all();
    const uint32_t at0 = (uint32_t)__cvta_generic_to_shared(sums), end0 = (uint32_t)__cvta_generic_to_shared(ends);
    const int mine = PAIRS / splits;
    for (int i = threadIdx.x; i < mine * (DT / 4); i += THREADS) {
        const int row = share * mine + i / (DT / 4), d = (i % (DT / 4)) * 4, at = pair0 + row;
        if (at >= pairs || d >= D) continue;
        float top = -INFINITY;
        int number = 0x7fffffff, none = -1;
        for (int j = 0; j < splits; ++j) {
            const float4 end = ld_cluster_f32x4(cluster_addr(end0 + row * 16, j));
            top = fmaxf(top, end.x);
            number = min(number, __float_as_int(end.z));
            none = max(none, __float_as_int(end.w));
        }
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        float weight = 0.f;
        for (int j = 0; j < splits; ++j) {
            const float4 end = ld_cluster_f32x4(cluster_addr(end0 + row * 16, j)), x = ld_cluster_f32x4(cluster_addr(at0 + (row * OS + d) * 4, j));
            const float f = end.x > -INFINITY ? expf(end.x - top) : 0.f;
            weight = fmaf(f, end.y, weight);
            sum.x = fmaf(f, x.x, sum.x); sum.y = fmaf(f, x.y, sum.y); sum.z = fmaf(f, x.z, sum.z); sum.w = fmaf(f, x.w, sum.w);
        }
        if (none > number) sum = make_float4(NAN, NAN, NAN, NAN);
        const float inv = weight > 0.f ? 1.0f / weight : 0.f;
        const int token = at / G;
        *reinterpret_cast<float4*>(p.out + ((int64_t)(q_start + token) * p.num_heads + kvh * G + at - token * G) * D + d) = make_float4(sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv);
    }
    cluster_sync_all();                               // (the others may still read this block's memory)
}

// The launch: blocks of 8 or 4 warps, shares of a walk, and (tile of pairs, key head) items.
// Heads of 64: blocks of 8 warps, two on an SM, where they are as many as the SMs and their walks long (each in two
// shares, so that the longest walks do not end alone: 1,024 tokens of 32 heads 147 -> 128 us, 333 on 300 beside 667 109 -> 94; shares of blocks of 4 warps 136 and 115; five rows of 120
// on 100 positions 47 us, by blocks of 4 warps 39).  Else blocks of 4 warps, three on an SM, in as many shares as fit beside one another (64 tokens on 900 positions: 1, 2, 4, 8 shares
// 109, 61, 35, 25 us; 200 on 800: 110, 71, 52, 73; 100 alone: 17.6, 15.0, 16.0, 27).  A walk of one tile has no shares: the second would have nothing and
// the meeting costs 4 to 6 us (64 tokens alone 14.1 -> 10.7).
// Heads of 65 to 128: blocks of 8 warps have an SM to themselves, those of 4 share it in twos (f32_direct), so that a block too many costs a whole round: the width and the number of shares that take
// the least estimated time.  Measured, us: a block of 8 warps 6.7 and 12.5 for every tile of its walk, of 4 warps 8.4 and 13.1 (16.9 where two share an SM), the meeting of two, four and eight shares
// 6.7, 4.1 and 4.4 (6.3, 3.5 and 4.0); clusters of four and eight fill the SMs but for a ninth and a quarter (1/36 and an eighth), since one lies within a part of the chip.  Rows' tiles have
// walks of different lengths, longest first: beyond one round the places fill up, and the last and shortest end three quarters of a block later; where all are alike it is whole rounds.  Over 468 steps
// of 1 to 32 rows, 32 heads on 8, 16 on 2, 16 on 16 and 8 on 8, within 0.5 % of the best plan on average.  Us, as many shares of blocks of 8 warps as fit : as here -- 32 heads on 8: 8 rows of 40 tokens
// 50 : 20, 4 of 100 51 : 32, 4 of 100 on 300 121 : 95, 2 of 64 on 1,000 126 : 75, 16 rows of one token on 400 116 : 73; 16 heads of 96 on 16, 32 rows of 64 tokens 73 : 53, of 64 on 130 224 : 152.
struct F32Plan { int warps, shares; int64_t items; };
static F32Plan f32_plan(int64_t pairs, int rows, int num_heads, int num_kv_heads, int head_dim, int window, int keep, int max_ctx, int sms) {
    using std::max; using std::min;
    const int reach = window > 0 ? min(max_ctx, window + keep + F32_KEYS) : window < 0 ? min(max_ctx, keep - window) : max_ctx;
    const int walk = (reach + F32_KEYS - 1) / F32_KEYS, most = walk > 1 ? max(2 * walk / 3, min(walk + 1, 4)) : 1;      // (walk: the longest one, in tiles of keys)
    // tiles of `per` pairs: a row's pairs are a multiple of the group's heads, so its last tile lacks at most per - gcd(per, heads)
    const int group = num_heads / num_kv_heads, fits = group & -group;
    auto items = [&](int per) { return (pairs + (int64_t)rows * (per - min(per, fits))) / per * num_kv_heads; };
    auto shares = [&](int64_t blocks, int two, int four, int eight) {         // places for blocks in so many shares
        int n = 1;
        while (n < 8 && 2 * n <= most && 2 * n * blocks <= (n == 1 ? two : n == 2 ? four : eight)) n *= 2;
        return n;
    };
    if (head_dim > 64) {
        const double tokens = (double)pairs / group / rows;        // of a row, as if they were alike
        F32Plan best{8, 1, 0};
        double least = 0;
        for (int warps = 8; warps >= 4; warps -= 4) {
            const int per = 16 * warps;
            const double first = max(1.0, min((double)walk, std::ceil((max_ctx - tokens + (double)per / group) / F32_KEYS)));
            const double shortest = window ? walk : first, mean = (walk + shortest) / 2;           // walks of a row's tiles
            const int64_t tiles = (int64_t)rows * (int64_t)std::ceil((double)pairs / rows / per) * num_kv_heads;
            const int wide[] = {sms, sms, sms * 8 / 9, sms * 3 / 4}, narrow[] = {2 * sms, 2 * sms, sms * 35 / 18, sms * 7 / 4};
            const double meet_wide[] = {0, 6.7, 4.1, 4.4}, meet_narrow[] = {0, 6.3, 3.5, 4.0};
            for (int n = 1, i = 0; n <= 8 && (n == 1 || walk > 1); n *= 2, ++i) {
                const double blocks = (double)(tiles * n), rounds = blocks / max(1, warps == 8 ? wide[i] : narrow[i]);
                const double start = warps == 8 ? 6.7 + meet_wide[i] : 8.4 + meet_narrow[i], step = warps == 8 ? 12.5 : 13.1 + 3.8 * (max(1.0, min(2.0, blocks / sms)) - 1);
                const double longest = start + step * ((walk + n - 1) / n), usual = start + step * max(1.0, mean / n), last = start + step * max(1.0, shortest / n);
                const double us = rounds <= 1 ? longest : max(longest, min(std::ceil(rounds) * longest, rounds * usual + 0.75 * last));
                if (least == 0 || us < least) { best = {warps, n, 0}; least = us; }
            }
        }
        best.items = items(16 * best.warps);
        return best;
    }
    if (pairs / 128 * num_kv_heads >= sms && walk >= 6) return {8, 2, items(128)};
    return {4, shares(items(64), 3 * sms, 3 * sms * 15 / 16, 3 * sms * 13 / 16), items(64)};
}
// The plan, for tests on the host: 256 x items + 16 x shares + warps.
extern "C" long long mie_attention_f32_plan(long long pairs, int rows, int num_heads, int num_kv_heads, int head_dim, int window, int keep, int max_ctx, int sms) {
    const F32Plan plan = f32_plan(pairs, rows, num_heads, num_kv_heads, head_dim, window, keep, max_ctx, sms);
    return 256 * plan.items + 16 * plan.shares + plan.warps;
}

template <int DT, int WARPS>
static int f32_launch(const F32Params& p, const F32Plan& plan, cudaStream_t stream) {
    const int splits = plan.shares;
    if (plan.items * splits > 0x7fffffff) return MIE_ERR_TOO_LARGE;
    const cudaError_t e = cudaFuncSetAttribute(f32_attention_kernel<DT, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, f32_bytes<DT, WARPS>());
    if (e != cudaSuccess) return (int)e;
    return launch_kernel_cluster(f32_attention_kernel<DT, WARPS>, dim3((unsigned)(plan.items * splits)), dim3(32 * WARPS), f32_bytes<DT, WARPS>(), stream, dim3(splits, 1, 1), p, splits);
}

// Rows with fewer than `min_q_len` new tokens are left alone; `max_ctx`: no row has more positions (it only shapes the launch); `rows`, `pairs`: upper bounds of the others' number and of their (token, head of a group) pairs.  Heads of
// 16 .. 128 in steps of 16, caches and out 16-byte aligned; the rest as mie_paged_attention.
extern "C" int mie_attention_f32(const float* q, int64_t q_stride, const float* k_cache, const float* v_cache, const int* block_tables, int table_stride,
                                 const int* row_q_start, const int* row_q_len, const int* row_ctx_len, int num_rows, int rows, long long pairs, float* out,
                                 int num_heads, int num_kv_heads, int head_dim, int page_size, float scale, int window, int keep, int min_q_len, int max_ctx,
                                 long long num_pages, float softcap, const float* sink, const float* dist_bias, int dist_len, const float* slope,
                                 cudaStream_t stream) {
    if (num_rows <= 0 || rows <= 0 || pairs <= 0) return 0;
    if (head_dim < 16 || head_dim > 128 || head_dim % 16 || min_q_len < 1 || (dist_bias && dist_len <= 0)) return MIE_ERR_BAD_ARG;
    if (num_kv_heads <= 0 || num_heads % num_kv_heads || page_size < 1 || (page_size & (page_size - 1))) return MIE_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(out)) & 15) return MIE_ERR_BAD_ARG;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    const F32Params p{q, q_stride, k_cache, v_cache, block_tables, table_stride, row_q_start, row_q_len, row_ctx_len, num_rows, out, num_heads,
                      num_kv_heads, head_dim, page_size, page_shift, scale, window, keep, min_q_len, (int64_t)num_pages, g_range_report,
                      ScoreMods{softcap, sink, dist_bias, dist_len, slope}};
    const F32Plan plan = f32_plan(pairs, rows, num_heads, num_kv_heads, head_dim, window, keep, max_ctx, device_sm_count());
    if (head_dim > 64) return plan.warps == 8 ? f32_launch<128, 8>(p, plan, stream) : f32_launch<128, 4>(p, plan, stream);
    return plan.warps == 8 ? f32_launch<64, 8>(p, plan, stream) : f32_launch<64, 4>(p, plan, stream);
}
