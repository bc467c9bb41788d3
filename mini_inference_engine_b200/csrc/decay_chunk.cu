// Linear attention with decays over long portions, in chunks of 64 tokens as matrix products (csrc/retention.cu walks token by token):
//
//   S_t = a_t S_{t-1} + k_t v_t^T,   o_t = S_t^T q_t                                        (a_t: one decay per head, or one per token and head)
//
// With G_i the product of a chunk's decays up to token i, M_ij the product of those behind token j up to token i and S the state in front of the chunk,
//   O = diag(G) Q S + (Q K^T * M) V,       what the chunk adds to the state = sum over t of M_{last, t} k_t v_t^T,       S <- G_last S + that,
// so a token costs 2 D Dv multiply-adds and half a chunk's of Q K^T and P V, out of shared memory in tiles of registers, where token by token it costs
// 5 D Dv in two passes, with a shared-memory read for every one or two.  Products of decays are products (no logarithms: a decay may be 0).  Float32 on the CUDA cores throughout.
//
//   local    a block per (chunk, head, half of the value columns): P = Q K^T * M (lower triangle) and G into scratch memory, and what the chunk adds to the state -> states[chunk].
//   combine  per row in order: states[chunk] becomes the state in front of the chunk; the state after the last goes to the request's slot.
//   output   a block per (chunk, head, 64 value columns).
//
// Rows of one chunk are left to retention.cu.  q and k come prepared (rotated or activated, scaled) as float32 from its first kernel.  Bound: the
// CUDA cores' multiply-adds.
#include "common.cuh"

#define DC_L 64                // tokens a chunk
#define DC_P 68                // stride of rows of 64: neighbouring rows four banks apart

__device__ __forceinline__ int dc_chunks(int n) { return n > DC_L ? (n + DC_L - 1) / DC_L : 0; }

struct DcParams {
    const float* q; const float* k;            // [T, H, D]
    const void* v; int64_t v_stride;           // [T][v_stride], a head's Dv_in columns side by side
    const int* row_q_start; const int* row_q_len; const int* state_slots; int num_rows;
    const float* decay; const float* tok_decay;
    float* state; float* states; float* scratch;        // scratch per (chunk, head): P [64, 64], G [64]
    float* out; int H, D, Dv_in, Dv, v_act;
    int h0, heads;                             // the heads of this pass: states and scratch hold these only
};
__device__ __forceinline__ float* dc_scratch(const DcParams& p, int64_t chunk, int h) { return p.scratch + (chunk * p.heads + h - p.h0) * (DC_L * DC_L + DC_L); }

__device__ __forceinline__ void dc_copy16(float* dst, const float* src, bool on) {       // zeros where `on` is false (nothing is read then)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void dc_wait_all() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }

// 64 rows of up to DT entries (the rest zero) into rows of DT + 4
template <int DT>
__device__ __forceinline__ void dc_rows(float* dst, const float* src, int64_t stride, int D, int count) {
    for (int c = threadIdx.x; c < DC_L * (DT / 4); c += blockDim.x) {
        const int r = c / (DT / 4), d = (c - r * (DT / 4)) * 4;
        const bool on = r < count && d < D;
        dc_copy16(dst + r * (DT + 4) + d, on ? src + r * stride + d : src, on);
    }
}

template <typename T>
__device__ __forceinline__ float dc_value(const DcParams& p, int64_t token, int h, int col) {
    const float v = to_f32<T>(reinterpret_cast<const T*>(p.v)[token * p.v_stride + (int64_t)h * p.Dv_in + col]);
    return p.v_act ? v / (1.0f + expf(-v)) : v;
}

// Which chunk this block has: its row, its number in the row; the blocks count chunks of rows of two or more.
__device__ __forceinline__ bool dc_find(const DcParams& p, int* s_row, int* s_chunk) {
    if (threadIdx.x < 32) {
        int within, items;
        const int r = warp_find_row(p.row_q_len, p.num_rows, (int)blockIdx.x, dc_chunks, within, items);
        if (threadIdx.x == 0) { *s_row = r; *s_chunk = within; }
    }
    __syncthreads();
    return *s_row >= 0;
}

template <typename T, int DT>
__global__ void __launch_bounds__(256, 2) decay_local_kernel(const DcParams p, int halves) {
    constexpr int DP = DT + 4;
    extern __shared__ __align__(16) float sm[];
    float* Q = sm;                                     // [64][DP]
    float* K = Q + DC_L * DP;                          // [64][DP]
    float* M = K + DC_L * DP;                          // [64][DC_P]: products of decays; then a tile of values [64 tokens][DC_P]
    __shared__ float a[DC_L], G[DC_L];
    __shared__ int s_row, s_chunk;
    pdl_launch_dependents();
    const bool mine = dc_find(p, &s_row, &s_chunk);
    pdl_wait();                                        // (a block without work waits too: see common.cuh)
    if (!mine) return;
    const int h = p.h0 + blockIdx.y, H = p.H, D = p.D, half = blockIdx.z;
    const int t0 = p.row_q_start[s_row] + s_chunk * DC_L, count = min(DC_L, p.row_q_len[s_row] - s_chunk * DC_L);
    dc_rows<DT>(K, p.k + ((int64_t)t0 * H + h) * D, (int64_t)H * D, D, count);
    if (half == 0) dc_rows<DT>(Q, p.q + ((int64_t)t0 * H + h) * D, (int64_t)H * D, D, count);
    if (threadIdx.x < DC_L)
        a[threadIdx.x] = threadIdx.x >= count ? 1.f : p.tok_decay ? p.tok_decay[(int64_t)(t0 + threadIdx.x) * H + h] : p.decay[h];
    __syncthreads();
    if (threadIdx.x < DC_L) {                          // a column of M a thread
        const int j = threadIdx.x;
        float run = 1.f;
#pragma unroll 8
        for (int i = 0; i < DC_L; ++i) {
            if (i > j) run *= a[i];
            M[i * DC_P + j] = i >= j ? run : 0.f;
        }
    } else if (threadIdx.x == DC_L) {
        float run = 1.f;
#pragma unroll 8
        for (int i = 0; i < DC_L; ++i) { run *= a[i]; G[i] = run; }
    }
    dc_wait_all();
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    if (half == 0) {
        float* out = dc_scratch(p, blockIdx.x, h);
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d = 0; d < DT; d += 4) {
            float4 kk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const float4*>(K + (tx + 16 * j) * DP + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 qq = *reinterpret_cast<const float4*>(Q + (ty + 16 * i) * DP + d);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j > i) continue;               // wholly above the diagonal
                    s[i][j] = fmaf(qq.x, kk[j].x, s[i][j]);
                    s[i][j] = fmaf(qq.y, kk[j].y, s[i][j]);
                    s[i][j] = fmaf(qq.z, kk[j].z, s[i][j]);
                    s[i][j] = fmaf(qq.w, kk[j].w, s[i][j]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = ty + 16 * i, c = tx + 16 * j;
                out[r * DC_L + c] = c <= r ? s[i][j] * M[r * DC_P + c] : 0.f;
            }
        if (threadIdx.x < DC_L) out[DC_L * DC_L + threadIdx.x] = G[threadIdx.x];
    }
    // keys with what is left of them at the chunk's end (in place: the scores are done with them once every thread is here)
    const float w_mine = M[(count - 1) * DC_P + (threadIdx.x & 63)];
    __syncthreads();
    if (threadIdx.x < DC_L) a[threadIdx.x] = threadIdx.x < count ? w_mine : 0.f;
    __syncthreads();
    for (int i = threadIdx.x; i < DC_L * (DT / 4); i += 256) {
        const int r = i / (DT / 4);
        float4* at = reinterpret_cast<float4*>(K + r * DP + (i - r * (DT / 4)) * 4);
        float4 v = *at;
        const float w = a[r];
        v.x *= w; v.y *= w; v.z *= w; v.w *= w;
        *at = v;
    }
    // the state's columns, 64 at a time: column 4 ty + c, entries 4 tx + 64 e .. + 3
    float* to = p.states + ((int64_t)blockIdx.x * p.heads + blockIdx.y) * (int64_t)p.Dv * D;
    constexpr int E = DT / 64;
    const int tiles = (p.Dv_in + 63) / 64, per = (tiles + halves - 1) / halves;
    for (int tile = half * per; tile < min(tiles, (half + 1) * per); ++tile) {
        __syncthreads();
        for (int i = threadIdx.x; i < DC_L * 64; i += 256) {
            const int t = i >> 6, c = i & 63, col = tile * 64 + c;
            M[t * DC_P + c] = t < count && col < p.Dv_in ? dc_value<T>(p, t0 + t, h, col) : 0.f;
        }
        __syncthreads();
        float s[4][4 * E];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 4 * E; ++e) s[c][e] = 0.f;
#pragma unroll 4
        for (int t = 0; t < DC_L; ++t) {
            const float4 vv = *reinterpret_cast<const float4*>(M + t * DC_P + 4 * ty);
            const float vc[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const float4 kk = *reinterpret_cast<const float4*>(K + t * DP + 64 * e + 4 * tx);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[c][4 * e] = fmaf(vc[c], kk.x, s[c][4 * e]);
                    s[c][4 * e + 1] = fmaf(vc[c], kk.y, s[c][4 * e + 1]);
                    s[c][4 * e + 2] = fmaf(vc[c], kk.z, s[c][4 * e + 2]);
                    s[c][4 * e + 3] = fmaf(vc[c], kk.w, s[c][4 * e + 3]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int col = tile * 64 + 4 * ty + c;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int d = 64 * e + 4 * tx;
                if (col < p.Dv_in && d < D)
                    *reinterpret_cast<float4*>(to + (int64_t)col * D + d) = make_float4(s[c][4 * e], s[c][4 * e + 1], s[c][4 * e + 2], s[c][4 * e + 3]);
            }
        }
    }
    if (half == 0 && p.Dv > p.Dv_in && threadIdx.x < D) {      // the column fed with ones: the sum of the keys
        float sum = 0.f;
        for (int t = 0; t < DC_L; ++t) sum += K[t * DP + threadIdx.x];
        to[(int64_t)p.Dv_in * D + threadIdx.x] = sum;
    }
}

// A thread four entries of a state; eight chunks' additions are read ahead of the chain.  blockIdx.y counts the rows of two chunks or more only: beside 64
// single tokens the blocks of rows that have no chunks had cost more than the chunks (a portion of 100 tokens, 16 heads of 128 x 256).
__global__ void __launch_bounds__(128) decay_combine_kernel(const DcParams p) {
    pdl_enter();
    const int64_t per_state = (int64_t)p.heads * p.Dv * p.D, e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    int within, one;
    const int row = warp_find_row(p.row_q_len, p.num_rows, (int)blockIdx.y, [](int n) { return dc_chunks(n) > 0 ? 1 : 0; }, within, one);
    if (row < 0) return;
    int first = 0;                                     // where the row's chunks begin
    for (int r = threadIdx.x & 31; r < row; r += 32) first += dc_chunks(p.row_q_len[r]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
    const int items = dc_chunks(p.row_q_len[row]);
    if (e >= per_state) return;
    const int h = p.h0 + (int)(e / ((int64_t)p.Dv * p.D));
    float* end = p.state + ((int64_t)p.state_slots[row] * p.H + p.h0) * p.Dv * p.D + e;
    float4 cur = *reinterpret_cast<const float4*>(end);
    float* slot = p.states + (int64_t)first * per_state + e;
    const int last = p.row_q_len[row] - (items - 1) * DC_L - 1;
    for (int j0 = 0; j0 < items; j0 += 8) {
        float4 add[8];
        float g[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (j0 + k < items) {
                add[k] = *reinterpret_cast<const float4*>(slot + (int64_t)(j0 + k) * per_state);
                g[k] = dc_scratch(p, first + j0 + k, h)[DC_L * DC_L + (j0 + k == items - 1 ? last : DC_L - 1)];
            }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (j0 + k < items) {
                *reinterpret_cast<float4*>(slot + (int64_t)(j0 + k) * per_state) = cur;
                cur.x = fmaf(g[k], cur.x, add[k].x); cur.y = fmaf(g[k], cur.y, add[k].y);
                cur.z = fmaf(g[k], cur.z, add[k].z); cur.w = fmaf(g[k], cur.w, add[k].w);
            }
    }
    *reinterpret_cast<float4*>(end) = cur;
}

template <typename T, int DT>
__global__ void __launch_bounds__(256, 2) decay_output_kernel(const DcParams p) {
    constexpr int DP = DT + 4;
    extern __shared__ __align__(16) float sm[];
    float* Q = sm;                                     // [64][DP]
    float* S = Q + DC_L * DP;                          // the state's columns [64][DP]
    float* P = S + 64 * DP;                            // [64][DC_P]
    float* VT = P + DC_L * DC_P;                       // values, a column a row [64][DC_P]
    __shared__ float G[DC_L];
    __shared__ __align__(16) float n[DT];
    __shared__ int s_row, s_chunk;
    pdl_launch_dependents();
    const bool mine = dc_find(p, &s_row, &s_chunk);
    pdl_wait();                                        // (a block without work waits too: see common.cuh)
    if (!mine) return;
    const int h = p.h0 + blockIdx.y, H = p.H, D = p.D, c0 = blockIdx.z * 64;
    const int t0 = p.row_q_start[s_row] + s_chunk * DC_L, count = min(DC_L, p.row_q_len[s_row] - s_chunk * DC_L);
    const float* from = p.states + ((int64_t)blockIdx.x * p.heads + blockIdx.y) * (int64_t)p.Dv * D;
    const float* pg = dc_scratch(p, blockIdx.x, h);
    const bool ones = blockIdx.z == 0 && p.Dv > p.Dv_in;
    dc_rows<DT>(Q, p.q + ((int64_t)t0 * H + h) * D, (int64_t)H * D, D, count);
    dc_rows<DT>(S, from + (int64_t)c0 * D, D, D, min(64, p.Dv_in - c0));
    for (int i = threadIdx.x; i < DC_L * (DC_L / 4); i += 256) dc_copy16(P + (i >> 4) * DC_P + (i & 15) * 4, pg + i * 4, true);
    if (threadIdx.x < DC_L) G[threadIdx.x] = pg[DC_L * DC_L + threadIdx.x];
    if (ones && threadIdx.x < DT) n[threadIdx.x] = threadIdx.x < D ? from[(int64_t)p.Dv_in * D + threadIdx.x] : 0.f;
    for (int i = threadIdx.x; i < DC_L * 64; i += 256) {
        const int t = i >> 6, c = i & 63;
        VT[c * DC_P + t] = t < count && c0 + c < p.Dv_in ? dc_value<T>(p, t0 + t, h, c0 + c) : 0.f;
    }
    dc_wait_all();
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < DT; d += 4) {
        float4 ss[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) ss[j] = *reinterpret_cast<const float4*>(S + (tx + 16 * j) * DP + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 qq = *reinterpret_cast<const float4*>(Q + (ty + 16 * i) * DP + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[i][j] = fmaf(qq.x, ss[j].x, o[i][j]);
                o[i][j] = fmaf(qq.y, ss[j].y, o[i][j]);
                o[i][j] = fmaf(qq.z, ss[j].z, o[i][j]);
                o[i][j] = fmaf(qq.w, ss[j].w, o[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float g = G[ty + 16 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] *= g;
    }
    for (int t = 0; t < DC_L; t += 4) {
        float4 vv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) vv[j] = *reinterpret_cast<const float4*>(VT + (tx + 16 * j) * DC_P + t);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty + 16 * i;
            if (t > r) continue;                       // (later tokens: their values, whatever they are, do not enter)
            const float4 pp = *reinterpret_cast<const float4*>(P + r * DC_P + t);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[i][j] = fmaf(pp.x, vv[j].x, o[i][j]);
                if (t + 1 <= r) o[i][j] = fmaf(pp.y, vv[j].y, o[i][j]);
                if (t + 2 <= r) o[i][j] = fmaf(pp.z, vv[j].z, o[i][j]);
                if (t + 3 <= r) o[i][j] = fmaf(pp.w, vv[j].w, o[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i;
        if (r >= count) continue;
        float* to = p.out + ((int64_t)(t0 + r) * H + h) * p.Dv;
#pragma unroll
        for (int j = 0; j < 4; ++j) if (c0 + tx + 16 * j < p.Dv_in) to[c0 + tx + 16 * j] = o[i][j];
    }
    if (ones) {                                        // n . q: four lanes a token
        const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
        float dot = 0.f, sum = 0.f;
        for (int d = part; d < DT; d += 4) dot = fmaf(Q[r * DP + d], n[d], dot);
        for (int t = part; t <= r; t += 4) sum += P[r * DC_P + t];
        float v = fmaf(G[r], dot, sum);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (part == 0 && r < count) p.out[((int64_t)(t0 + r) * H + h) * p.Dv + p.Dv_in] = v;
    }
}

// Floats of `scratch` a (chunk, head) needs.
extern "C" int mie_decay_chunk_floats() { return DC_L * DC_L + DC_L; }

// Rows of more than 64 new tokens.  q, k [T, H, D] float32, v [T][v_stride] of `v_tag`'s type; decay [H] or tok_decay [T, H]; state [slots, H, Dv, D],
// `per_pass` heads at a time, on the same scratch memory: states [chunks, per_pass, Dv, D], scratch [chunks, per_pass, mie_decay_chunk_floats()], `chunks` at least the chunks of those rows; out [T, H, Dv] with Dv = Dv_in or
// Dv_in + 1 (the last column fed with ones).  D a multiple of 4 up to 128; q, k, state, states 16-byte aligned.
extern "C" int mie_decay_chunks(const float* q, const float* k, const void* v, int v_tag, long long v_stride, const int* row_q_start, const int* row_q_len,
                                const int* state_slots, int num_rows, const float* decay, const float* tok_decay, float* state, float* states,
                                float* scratch, int chunks, float* out, int H, int D, int Dv_in, int Dv, int v_act, int per_pass, cudaStream_t stream) {
    if (num_rows <= 0 || chunks <= 0) return 0;
    if (H <= 0 || D < 4 || D > 128 || D % 4 || Dv_in <= 0 || Dv < Dv_in || Dv > Dv_in + 1 || (!decay && !tok_decay) || per_pass < 1) return MIE_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(states) |
         reinterpret_cast<uintptr_t>(scratch)) & 15) return MIE_ERR_BAD_ARG;
    DcParams p{q, k, v, v_stride, row_q_start, row_q_len, state_slots, num_rows, decay, tok_decay, state, states, scratch, out, H, D, Dv_in, Dv, v_act, 0, 0};
    const int halves = Dv_in > 64 ? 2 : 1;
    const int long_rows = num_rows < chunks / 2 ? num_rows : chunks / 2 > 0 ? chunks / 2 : 1;      // (each has two chunks at least)
    int rc;
#define DC_LAUNCH(T, DT)                                                                                                                  \
    {                                                                                                                                     \
        const int smem_l = (2 * DC_L * (DT + 4) + DC_L * DC_P) * 4, smem_o = ((DC_L + 64) * (DT + 4) + 2 * DC_L * DC_P) * 4;              \
        cudaError_t e = cudaFuncSetAttribute(decay_local_kernel<T, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_l);             \
        if (e == cudaSuccess) e = cudaFuncSetAttribute(decay_output_kernel<T, DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_o);  \
        if (e != cudaSuccess) return (int)e;                                                                                              \
        for (p.h0 = 0; p.h0 < H; p.h0 += per_pass) {                                                                                      \
            p.heads = H - p.h0 < per_pass ? H - p.h0 : per_pass;                                                                          \
            rc = launch_kernel(decay_local_kernel<T, DT>, dim3(chunks, p.heads, halves), dim3(256), smem_l, stream, p, halves);           \
            if (rc) return rc;                                                                                                            \
            const int64_t quads = (int64_t)p.heads * Dv * D / 4;                                                                          \
            rc = launch_kernel(decay_combine_kernel, dim3((unsigned)((quads + 127) / 128), long_rows), dim3(128), 0, stream, p);          \
            if (rc) return rc;                                                                                                            \
            rc = launch_kernel(decay_output_kernel<T, DT>, dim3(chunks, p.heads, (Dv_in + 63) / 64), dim3(256), smem_o, stream, p);       \
            if (rc) return rc;                                                                                                            \
        }                                                                                                                                 \
        return 0;                                                                                                                         \
    }
    if (v_tag == MIE_F32) { if (D <= 64) DC_LAUNCH(float, 64) else DC_LAUNCH(float, 128) }
    if (v_tag == MIE_BF16) { if (D <= 64) DC_LAUNCH(bf16, 64) else DC_LAUNCH(bf16, 128) }
#undef DC_LAUNCH
    return MIE_ERR_BAD_ARG;
}
