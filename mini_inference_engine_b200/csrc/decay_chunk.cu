// Linear attention with decays over long portions, in chunks of 64 tokens as matrix products (csrc/retention.cu walks token by token):
//
//   S_t = a_t S_{t-1} + k_t v_t^T,   o_t = S_t^T q_t                                        (a_t: one decay per head, or one per token and head)
//
// With G_i the product of a chunk's decays up to token i, M_ij the product of those behind token j up to token i and S the state in front of the chunk,
//   O = diag(G) Q S + (Q K^T * M) V,       what the chunk adds to the state = sum over t of M_{last, t} k_t v_t^T,       S <- G_last S + that,
// so a token costs 2 D Dv multiply-adds and half a chunk's of Q K^T and P V, where token by token it costs
// 5 D Dv in two passes, with a shared-memory read for every one or two.  Products of decays are products (no logarithms: a decay may be 0).  The products run on the tensor
// cores with every float32 operand as three bfloat16 parts (triple_mma.cuh); values that are bfloat16 as they come are one part, so that half of the part products fall away.
//
//   local    a block per (chunk, head): P = Q K^T * M (lower triangle) and G into scratch memory, and what the chunk adds to the state -> states[chunk].
//   combine  per row in order: states[chunk] becomes the state in front of the chunk; the state after the last goes to the request's slot.
//   output   a block per (chunk, head, 128 or 64 value columns).
//
// Numbers without three parts (not finite, or beyond 2^127) make their block do its products one multiply-add after the other, without the zeros of the triangle.
//
// Rows of one chunk are left to retention.cu.  q and k come prepared (rotated or activated, scaled) as float32 from its first kernel.
// Bound: the tensor pipe at 8 cycles an instruction on each quarter of an SM, kept busy for 24 - 30 % of the time (operands' way from memory and the blocks' ends are the
// rest).  2,048 tokens of 8 heads of 128 x 256 from bfloat16 values, us: local 51.7 -> 30, output 78.7 -> 40 (register tiles on the CUDA cores before); the layer
// with a decay per head 209 -> 146, of 100 tokens 58 -> 46.  float32 values, or bfloat16 ones behind an activation, in heads above 64 (three
// parts, 117 KB, so one block of `local` on an SM where two of bfloat16 values fit): the whole scan of those sizes 159 -> 107 and 172 -> 122 us, 512 tokens 58 -> 46 and 64 -> 50, 100 tokens 43 -> 31 and 50 -> 37.  Against 64 bits the outputs are 1.0e-7 to 2.7e-7 off (2-norm; the CUDA cores' 2.1e-7 to 3.5e-7), the states
// 4.7e-8 to 3.0e-7 (4.8e-8 to 3.1e-7).
#include "triple_mma.cuh"

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

#define DC_THREADS 256
#define DC_COLS 64             // value columns of the local kernel at a time

// Eight neighbouring values of a token as they lie in memory, those from `left` on zero; and as numbers (nothing is computed from them where they are asked for, so that
// nothing waits there).
template <typename T> struct alignas(16) Eight { T x[8]; };
template <typename T>
__device__ __forceinline__ Eight<T> dc_values8(const DcParams& p, int64_t token, int h, int col, int left) {
    Eight<T> r;
    const T* at = reinterpret_cast<const T*>(p.v) + token * p.v_stride + (int64_t)h * p.Dv_in + col;
    uint4* to = reinterpret_cast<uint4*>(r.x);
    if (left >= 8 && (reinterpret_cast<uintptr_t>(at) & 15) == 0) {
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; ++i) to[i] = reinterpret_cast<const uint4*>(at)[i];
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) r.x[i] = i < left ? at[i] : from_f32<T>(0.f);
    }
    return r;
}
template <typename T>
__device__ __forceinline__ void dc_numbers(float (&x)[8], const Eight<T>& r, const DcParams& p) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        x[i] = to_f32<T>(r.x[i]);
        if (p.v_act) x[i] = x[i] / (1.0f + expf(-x[i]));
    }
}

// Left operand (16 columns x 16 rows of the tile) from tiles [64][COLS] whose rows run along the contraction.
template <int COLS, int PARTS>
__device__ __forceinline__ void dc_left(uint32_t (&a)[PARTS][4], uint32_t tile, int plane, int m, int k, int lane) {
    const uint32_t at = tile + tile_at<COLS>(k * 16 + (lane & 7) + ((lane >> 4) << 3), m * 2 + ((lane >> 3) & 1));
#pragma unroll
    for (int p = 0; p < PARTS; ++p) ldm4t(a[p][0], a[p][1], a[p][2], a[p][3], at + p * plane);
}
// sum[n] += A B_n over 16 of the contraction, one of the two operands a single part.
template <int N>
__device__ __forceinline__ void one_left_step(float (*sum)[4], const uint32_t (&a)[1][4], const uint32_t (&b)[3][N][2]) {
    float t[N][4], h[N][4];
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(t[n], a[0], b[2][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(h[n], a[0], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[0], b[1][n]);
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[n][i] = h[n][i] + (sum[n][i] + t[n][i]);
}
template <int N>
__device__ __forceinline__ void one_right_step(float (*sum)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[1][N][2]) {
    float t[N][4], h[N][4];
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(t[n], a[2], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_zero(h[n], a[0], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n) mma_more(t[n], a[1], b[0][n]);
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[n][i] = h[n][i] + (sum[n][i] + t[n][i]);
}

// A lane's eight numbers of the left operand with rows r0, r0 + 8 and columns d, d + 1, d + 8, d + 9 of float32 rows; those beyond the rows or the columns are zero.
struct DcLeft { float4 v, w; };
__device__ __forceinline__ DcLeft dc_left_rows(const float* rows, int64_t stride, int r0, int d, int count, int D) {
    auto two = [&](int r, int c) { return r < count && c < D ? *reinterpret_cast<const float2*>(rows + r * stride + c) : make_float2(0.f, 0.f); };
    const float2 a = two(r0, d), b = two(r0 + 8, d), e = two(r0, d + 8), f = two(r0 + 8, d + 8);
    return DcLeft{make_float4(a.x, a.y, b.x, b.y), make_float4(e.x, e.y, f.x, f.y)};
}

// What a chunk adds to the state, a multiply-add after the other; ww: what is left of each token at the chunk's end.
template <typename T>
__device__ __noinline__ void dc_walk_state(const DcParams& p, const float* kp, const float* ww, float* to, int t0, int h, int count, int first, int end) {
    for (int i = first * p.D + threadIdx.x; i < end * p.D; i += DC_THREADS) {
        const int col = i / p.D, d = i - col * p.D;
        float sum = 0.f;
        for (int t = 0; t < count; ++t) sum = fmaf(col < p.Dv_in ? dc_value<T>(p, t0 + t, h, col) : 1.f, ww[t] * kp[(int64_t)t * p.H * p.D + d], sum);
        to[i] = sum;
    }
}
__device__ __noinline__ void dc_walk_scores(const DcParams& p, const float* qp, const float* kp, const float* M, float* out, int count) {
    for (int i = threadIdx.x; i < DC_L * DC_L; i += DC_THREADS) {
        const int r = i >> 6, c = i & 63;
        float sum = 0.f;
        if (c <= r && r < count)
            for (int d = 0; d < p.D; ++d) sum = fmaf(qp[(int64_t)r * p.H * p.D + d], kp[(int64_t)c * p.H * p.D + d], sum);
        out[i] = c <= r ? sum * M[r * DC_P + c] : 0.f;
    }
}

// ONE: the values are bfloat16 as they come.  blockIdx.z: a share of the value columns -- with fewer (chunk, head) pairs than SMs a pair's columns go to as many blocks as there is
// room for (the first share makes P too): 100 tokens of 8 heads of 128 x 256, 4 shares, the kernel and the output kernel's narrow blocks, layer 58.6 -> 46.1 us; shares
// for two blocks an SM instead of one: 1,024 tokens 19.4 -> 18.6 us, 512 tokens 14.6 -> 14.9.
template <typename T, int DT, bool ONE>
__global__ void __launch_bounds__(DC_THREADS, 2) decay_local_kernel(const DcParams p, int splits) {
    constexpr int AHEAD = 3;                           // steps of the contraction that the queries are asked for ahead
    constexpr int PLANE = DC_L * DT * 2, V_PLANE = DC_L * DC_COLS * 2, PARTS = ONE ? 1 : 3, KS = DT / 16, QUADS = DC_L * DT / 4 / DC_THREADS, STEP = DC_THREADS / (DT / 4);
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* keys = smem;                              // [64][DT] as parts; then with what is left of them at the chunk's end
    uint8_t* values = smem + 3 * PLANE;                // two buffers of [64][64]
    float* M = reinterpret_cast<float*>(values + 2 * PARTS * V_PLANE);     // [64][DC_P]: products of decays
    __shared__ float a[DC_L], G[DC_L];
    __shared__ int s_row, s_chunk;
    pdl_launch_dependents();
    const bool mine = dc_find(p, &s_row, &s_chunk);
    pdl_wait();                                        // (a block without work waits too: see common.cuh)
    if (!mine) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = p.h0 + blockIdx.y, H = p.H, D = p.D;
    const int t0 = p.row_q_start[s_row] + s_chunk * DC_L, count = min(DC_L, p.row_q_len[s_row] - s_chunk * DC_L);
    const int tiles = (p.Dv_in + DC_COLS - 1) / DC_COLS, per = (tiles + splits - 1) / splits, part_no = blockIdx.z;       // this block's share of the value columns
    const int first_col = part_no * per * DC_COLS, end_col = min((part_no + 1) * per * DC_COLS, p.Dv_in);
    const float* kp = p.k + ((int64_t)t0 * H + h) * D;
    const float* qp = p.q + ((int64_t)t0 * H + h) * D;
    const int64_t stride = (int64_t)H * D;
    const int kr = threadIdx.x / (DT / 4), kd = (threadIdx.x % (DT / 4)) * 4;
    uint32_t most = 0;                                 // the largest magnitude of keys, queries and values this thread met
    float4 key[QUADS];
#pragma unroll
    for (int i = 0; i < QUADS; ++i)
        key[i] = kr + i * STEP < count && kd < D ? *reinterpret_cast<const float4*>(kp + (kr + i * STEP) * stride + kd) : make_float4(0.f, 0.f, 0.f, 0.f);
    auto put_keys = [&](auto factor) {
        uint32_t f_most = 0;
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int r = kr + i * STEP;
            const float f = factor(r);
            most = max(most, magnitude(key[i]));
            f_most = max(f_most, magnitude(f));
            uint8_t* at = keys + tile_at<DT>(r, kd >> 3) + (kd & 4) * 2;
            uint2 part[3];
            split3(key[i].x * f, key[i].y * f, part[0].x, part[1].x, part[2].x);
            split3(key[i].z * f, key[i].w * f, part[0].y, part[1].y, part[2].y);
#pragma unroll
            for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(at + j * PLANE) = part[j];
        }
        most = max(most, magnitude(__uint_as_float(most) * __uint_as_float(f_most)));      // (a decay may be infinite, or beyond 1)
    };
    if (threadIdx.x < DC_L)
        a[threadIdx.x] = threadIdx.x >= count ? 1.f : p.tok_decay ? p.tok_decay[(int64_t)(t0 + threadIdx.x) * H + h] : p.decay[h];
    put_keys([](int) { return 1.f; });
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
    // values of 64 columns, two runs of eight a thread; those of the next columns are asked for while these are multiplied
    Eight<T> raw[2];
    auto ask = [&](int j0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = (threadIdx.x >> 3) + 32 * i, c = j0 + (threadIdx.x & 7) * 8;
            raw[i] = dc_values8<T>(p, t0 + min(t, count - 1), h, c, t < count ? end_col - c : 0);
        }
    };
    ask(first_col);
    float* out = dc_scratch(p, blockIdx.x, h);
    if (part_no == 0) {
        // Q K^T: 16 rows a warp, every other pair of column tiles up to the diagonal; the queries go straight from memory into operands
        const int m = warp < 4 ? warp : 7 - warp, odd = warp >> 2, r = m * 16 + (lane >> 2), c0 = (lane & 3) * 2;
        const uint32_t right = (uint32_t)__cvta_generic_to_shared(keys);
        float sum[4][4] = {};
        DcLeft q[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) q[k] = dc_left_rows(qp, stride, r, k * 16 + c0, count, D);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            uint32_t left[3][4];
            const DcLeft x = q[k % AHEAD];
            most = max(most, max(magnitude(x.v), magnitude(x.w)));
            split_left(left, x.v, x.w);
            if (k + AHEAD < KS) q[k % AHEAD] = dc_left_rows(qp, stride, r, (k + AHEAD) * 16 + c0, count, D);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (odd + 2 * j > m) break;
                uint32_t b[3][2][2];
                right_columns<DT>(b, 0, right, PLANE, k, 2 * (odd + 2 * j), lane);
                triple_step<2>(sum + 2 * j, left, b);
            }
        }
        __syncthreads();                               // M
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = (odd + 2 * (j >> 1)) * 16 + (j & 1) * 8 + c0;
            if (odd + 2 * (j >> 1) > m) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int rr = r + 8 * i;
                const float2 f = *reinterpret_cast<const float2*>(M + rr * DC_P + c);
                *reinterpret_cast<float2*>(out + rr * DC_L + c) = make_float2(c <= rr ? sum[j][2 * i] * f.x : 0.f, c + 1 <= rr ? sum[j][2 * i + 1] * f.y : 0.f);
            }
        }
        if (threadIdx.x < DC_L) out[DC_L * DC_L + threadIdx.x] = G[threadIdx.x];
    } else __syncthreads();
    if (threadIdx.x < DC_L) a[threadIdx.x] = threadIdx.x < count ? M[(count - 1) * DC_P + threadIdx.x] : 0.f;      // what is left of each token at the chunk's end
    __syncthreads();                                   // (the keys are done with)
    put_keys([&](int r) { return a[r]; });
    float* to = p.states + ((int64_t)blockIdx.x * p.heads + blockIdx.y) * (int64_t)p.Dv * D;
    for (int j0 = first_col, buf = 0; j0 < end_col; j0 += DC_COLS, buf ^= 1) {
        uint8_t* tile = values + buf * PARTS * V_PLANE;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint8_t* at = tile + tile_at<DC_COLS>((threadIdx.x >> 3) + 32 * i, threadIdx.x & 7);
            uint32_t part[3][4];
            float x[8];
            dc_numbers(x, raw[i], p);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (ONE) part[0][e] = nearest2(x[2 * e], x[2 * e + 1]);
                else split3(x[2 * e], x[2 * e + 1], part[0][e], part[1][e], part[2][e]);
                most = max(most, max(magnitude(x[2 * e]), magnitude(x[2 * e + 1])));       // (one part too: an infinite value must not meet parts of a key that are zero)
            }
#pragma unroll
            for (int j = 0; j < PARTS; ++j) *reinterpret_cast<uint4*>(at + j * V_PLANE) = make_uint4(part[j][0], part[j][1], part[j][2], part[j][3]);
        }
        ask(j0 + DC_COLS);
        __syncthreads();
        // 32 of the columns (rows of the product) and a quarter of the channels a warp
        const int cg = warp & 1, d0 = (warp >> 1) * (DT / 4), c = j0 + cg * 32;
        const uint32_t left = (uint32_t)__cvta_generic_to_shared(tile), right = (uint32_t)__cvta_generic_to_shared(keys);
        if (c < end_col) {
            constexpr int NT = DT / 32;                // column tiles of a warp: 4 or 2
            float sum[2][NT][4] = {};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t v[2][PARTS][4];
#pragma unroll
                for (int m = 0; m < 2; ++m) dc_left<DC_COLS, PARTS>(v[m], left, V_PLANE, cg * 2 + m, k, lane);
#pragma unroll
                for (int n = 0; n < NT; n += 2) {
                    uint32_t b[3][2][2];
                    right_rows<DT>(b, 0, right, PLANE, k, d0 / 8 + n, lane);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        if constexpr (ONE) one_left_step<2>(sum[m] + n, v[m], b);
                        else triple_step<2>(sum[m] + n, v[m], b);
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int col = c + m * 16 + (lane >> 2) + 8 * i;
                    if (col >= end_col) continue;
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const int d = d0 + n * 8 + (lane & 3) * 2;
                        if (d < D) *reinterpret_cast<float2*>(to + (int64_t)col * D + d) = make_float2(sum[m][n][2 * i], sum[m][n][2 * i + 1]);
                    }
                }
        }
    }
    if (part_no == 0 && p.Dv > p.Dv_in) {              // the column fed with ones: the sum of the keys, from their parts
        const int d = threadIdx.x % DT, first = threadIdx.x / DT * (DT / 4);
        float sum = 0.f;
#pragma unroll 8
        for (int t = first; t < first + DT / 4; ++t) {
            const uint8_t* at = keys + tile_at<DT>(t, d >> 3) + (d & 7) * 2;
            const float h = __bfloat162float(*reinterpret_cast<const bf16*>(at)), m = __bfloat162float(*reinterpret_cast<const bf16*>(at + PLANE)),
                        l = __bfloat162float(*reinterpret_cast<const bf16*>(at + 2 * PLANE));
            sum += h + (m + l);
        }
        float* part = reinterpret_cast<float*>(values);
        __syncthreads();                               // (the values are done with)
        part[threadIdx.x] = sum;
        __syncthreads();
        if (threadIdx.x < D) {
#pragma unroll
            for (int i = 1; i < DC_THREADS / DT; ++i) sum += part[i * DT + threadIdx.x];
            to[(int64_t)p.Dv_in * D + threadIdx.x] = sum;
        }
    }
    if (__syncthreads_or(has_no_parts(most))) {
        dc_walk_state<T>(p, kp, a, to, t0, h, count, first_col, end_col);
        if (part_no == 0) {                            // (the column of ones is the first share's, like P)
            dc_walk_state<T>(p, kp, a, to, t0, h, count, p.Dv_in, p.Dv);
            dc_walk_scores(p, qp, kp, M, out, count);
        }
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

// A block per (chunk, head, 128 or 64 value columns): 16 of them a warp, all of the chunk's tokens.  Q, P and the values as parts in shared memory, the state from memory
// straight into operands.  ONE: the values are bfloat16 as they come.  WARPS 8; 4 where blocks of 8 would leave half of the SMs without one
// (512 tokens of 8 heads: 15.4 us by blocks of 8 warps, 16.8 by blocks of 4).  Three blocks an SM in 80 registers each: 44 -> 51 us at 2,048 tokens.
template <int DT, bool ONE, int WARPS> constexpr int output_bytes() { return (4 * (DT / 16) + 10) * 1536 + (ONE ? 1 : 3) * DC_L * 16 * WARPS * 2; }
template <typename T, int DT, bool ONE, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 2) decay_output_kernel(const DcParams p) {
    constexpr int KS = DT / 16, PARTS = ONE ? 1 : 3, AHEAD = 4;
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t* left = reinterpret_cast<uint32_t*>(smem); // Q [4 * KS][part][lane][4], then P's tiles up to the diagonal, row by row
    uint8_t* values = smem + (4 * KS + 10) * 1536;     // [64][16 * WARPS] as parts
    constexpr int THREADS = 32 * WARPS, WIDE = 16 * WARPS, V_PLANE = DC_L * WIDE * 2;
    __shared__ float G[DC_L];
    __shared__ int s_row, s_chunk;
    pdl_launch_dependents();
    const bool mine = dc_find(p, &s_row, &s_chunk);
    pdl_wait();                                        // (a block without work waits too: see common.cuh)
    if (!mine) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, h = p.h0 + blockIdx.y, H = p.H, D = p.D, r0 = lane >> 2, c0 = (lane & 3) * 2;
    const int t0 = p.row_q_start[s_row] + s_chunk * DC_L, count = min(DC_L, p.row_q_len[s_row] - s_chunk * DC_L);
    const float* from = p.states + ((int64_t)blockIdx.x * p.heads + blockIdx.y) * (int64_t)p.Dv * D;
    const float* pg = dc_scratch(p, blockIdx.x, h);
    const float* qp = p.q + ((int64_t)t0 * H + h) * D;
    const int64_t stride = (int64_t)H * D;
    const int j0 = (blockIdx.z * WARPS + warp) * 16;
    // the state's 16 channels of two tiles of 8 columns, asked for ahead: they come from L2 at best
    auto ask = [&](float2 (&x)[4], int k) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int col = j0 + (i >> 1) * 8 + r0, d = k * 16 + (i & 1) * 8 + c0;
            x[i] = col < p.Dv_in && d < D ? *reinterpret_cast<const float2*>(from + (int64_t)col * D + d) : make_float2(0.f, 0.f);
        }
    };
    float2 raw[AHEAD][4];
#pragma unroll
    for (int k = 0; k < AHEAD; ++k) ask(raw[k], k);
    auto diagonal = [](int m) { return m * (m + 1) / 2; };
    uint32_t most = 0;                                 // the largest magnitude among the queries, the state and the values that this thread met
    constexpr int RUNS = DC_L * WIDE / 8 / THREADS;         // of eight values a thread
    Eight<T> run[RUNS];
#pragma unroll
    for (int o = 0; o < RUNS; ++o) {
        const int i = threadIdx.x + o * THREADS, t = i / (WIDE / 8), col = blockIdx.z * WIDE + i % (WIDE / 8) * 8;
        run[o] = dc_values8<T>(p, t0 + min(t, count - 1), h, col, t < count ? p.Dv_in - col : 0);
    }
    if (threadIdx.x < DC_L) G[threadIdx.x] = pg[DC_L * DC_L + threadIdx.x];
    constexpr int TURNS = (4 * KS + 10 + WARPS - 1) / WARPS, HALF = (TURNS + 1) / 2;
#pragma unroll
    for (int first = 0; first < TURNS; first += HALF) {        // (half of the operands asked for at a time)
        DcLeft x[HALF];
#pragma unroll
        for (int o = 0; o < HALF; ++o) {
            const int i = warp + (first + o) * WARPS, j = i - 4 * KS, m = j < 0 ? i / KS : j < 1 ? 0 : j < 3 ? 1 : j < 6 ? 2 : 3;
            if (j < 0) x[o] = dc_left_rows(qp, stride, m * 16 + r0, (i % KS) * 16 + c0, count, D);
            else if (j < 10) x[o] = dc_left_rows(pg, DC_L, m * 16 + r0, (j - diagonal(m)) * 16 + c0, DC_L, DC_L);
        }
#pragma unroll
        for (int o = 0; o < HALF; ++o) {
            const int i = warp + (first + o) * WARPS;
            if (i >= 4 * KS + 10) break;
            uint32_t a[3][4];
            most = max(most, max(magnitude(x[o].v), magnitude(x[o].w)));
            split_left(a, x[o].v, x[o].w);
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(left + i * 384 + q * 128 + lane * 4) = make_uint4(a[q][0], a[q][1], a[q][2], a[q][3]);
        }
    }
#pragma unroll
    for (int o = 0; o < RUNS; ++o) {
        const int i = threadIdx.x + o * THREADS;
        float x[8];
        dc_numbers(x, run[o], p);
        uint8_t* at = values + tile_at<WIDE>(i / (WIDE / 8), i % (WIDE / 8));
        uint32_t part[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            most = max(most, max(magnitude(x[2 * e]), magnitude(x[2 * e + 1])));
            if (ONE) part[0][e] = nearest2(x[2 * e], x[2 * e + 1]);
            else split3(x[2 * e], x[2 * e + 1], part[0][e], part[1][e], part[2][e]);
        }
#pragma unroll
        for (int j = 0; j < PARTS; ++j) *reinterpret_cast<uint4*>(at + j * V_PLANE) = make_uint4(part[j][0], part[j][1], part[j][2], part[j][3]);
    }
    bool bad = __syncthreads_or(has_no_parts(most));
    auto operand = [&](uint32_t (&a)[3][4], int i) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const uint4 v = *reinterpret_cast<const uint4*>(left + i * 384 + q * 128 + lane * 4);
            a[q][0] = v.x; a[q][1] = v.y; a[q][2] = v.z; a[q][3] = v.w;
        }
    };
    if (j0 < p.Dv_in) {
        float sum[4][2][4] = {};
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            uint32_t b[3][2][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 x = raw[k % AHEAD][i];
                most = max(most, max(magnitude(x.x), magnitude(x.y)));
                split3(x.x, x.y, b[0][i >> 1][i & 1], b[1][i >> 1][i & 1], b[2][i >> 1][i & 1]);
            }
            if (k + AHEAD < KS) ask(raw[k % AHEAD], k + AHEAD);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                uint32_t a[3][4];
                operand(a, m * KS + k);
                triple_step<2>(sum[m], a, b);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float f = G[m * 16 + r0 + 8 * i];
#pragma unroll
                for (int n = 0; n < 2; ++n) { sum[m][n][2 * i] *= f; sum[m][n][2 * i + 1] *= f; }
            }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t b[PARTS][2][2];
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(values) + tile_at<WIDE>(k * 16 + (lane & 15), warp * 2 + (lane >> 4));
#pragma unroll
            for (int q = 0; q < PARTS; ++q) ldm4t(b[q][0][0], b[q][0][1], b[q][1][0], b[q][1][1], at + q * V_PLANE);
#pragma unroll
            for (int m = k; m < 4; ++m) {
                uint32_t a[3][4];
                operand(a, 4 * KS + diagonal(m) + k);
                if constexpr (ONE) one_right_step<2>(sum[m], a, b);
                else triple_step<2>(sum[m], a, b);
            }
        }
        bad |= __any_sync(0xffffffffu, has_no_parts(most));
        // (later tokens: their values, whatever they are, do not enter)
        auto again = [&](int r, int col) {
            float dot = 0.f;
            for (int d = 0; d < D; ++d) dot = fmaf(qp[r * stride + d], from[(int64_t)col * D + d], dot);
            dot *= pg[DC_L * DC_L + r];
            for (int t = 0; t <= r; ++t) dot = fmaf(pg[r * DC_L + t], dc_value<T>(p, t0 + t, h, col), dot);
            return dot;
        };
        if (!bad) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = m * 16 + r0 + 8 * i;
                    if (r >= count) continue;
                    float* to = p.out + ((int64_t)(t0 + r) * H + h) * p.Dv;
#pragma unroll
                    for (int n = 0; n < 2; ++n)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int col = j0 + n * 8 + c0 + e;
                            if (col < p.Dv_in) to[col] = sum[m][n][2 * i + e];
                        }
                }
        } else {
#pragma unroll 1
            for (int o = lane; o < count * 16; o += 32) {
                const int r = o >> 4, col = j0 + (o & 15);
                if (col < p.Dv_in) p.out[((int64_t)(t0 + r) * H + h) * p.Dv + col] = again(r, col);
            }
        }
    }
    if (blockIdx.z == 0 && p.Dv > p.Dv_in) {           // the column fed with ones, n . q: four lanes a token
        const float* n = from + (int64_t)p.Dv_in * D;
        for (int first = 0; first < DC_L; first += THREADS / 4) {
            const int r = first + (threadIdx.x >> 2), part = threadIdx.x & 3;
            float dot = 0.f, sum = 0.f;
            if (r < count) {
                for (int d = part * 4; d < D; d += 16) {
                    const float4 x = *reinterpret_cast<const float4*>(qp + r * stride + d), y = *reinterpret_cast<const float4*>(n + d);
                    dot = fmaf(x.x, y.x, dot); dot = fmaf(x.y, y.y, dot); dot = fmaf(x.z, y.z, dot); dot = fmaf(x.w, y.w, dot);
                }
                for (int t = part; t <= r; t += 4) sum += pg[r * DC_L + t];
            }
            float v = r < count ? fmaf(pg[DC_L * DC_L + r], dot, sum) : 0.f;
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (part == 0 && r < count) p.out[((int64_t)(t0 + r) * H + h) * p.Dv + p.Dv_in] = v;
        }
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
    const int sms = device_sm_count();
    const int long_rows = num_rows < chunks / 2 ? num_rows : chunks / 2 > 0 ? chunks / 2 : 1;      // (each has two chunks at least)
    int rc;
#define DC_OUTPUT(T, DT, ONE, WARPS)                                                                                                                      \
    {                                                                                                                                                     \
        auto kernel = decay_output_kernel<T, DT, ONE, WARPS>;                                                                                             \
        constexpr int bytes = output_bytes<DT, ONE, WARPS>();                                                                                             \
        const cudaError_t f = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);                                            \
        rc = f != cudaSuccess ? (int)f                                                                                                                    \
                              : launch_kernel(kernel, dim3(chunks, p.heads, (Dv_in + 16 * WARPS - 1) / (16 * WARPS)), dim3(32 * WARPS), bytes, stream, p); \
    }
#define DC_LAUNCH(T, DT, ONE)                                                                                                                             \
    {                                                                                                                                                     \
        const int smem_l = 3 * DC_L * DT * 2 + 2 * (ONE ? 1 : 3) * DC_L * DC_COLS * 2 + DC_L * DC_P * 4;                                                   \
        const cudaError_t e = cudaFuncSetAttribute(decay_local_kernel<T, DT, ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_l);                   \
        if (e != cudaSuccess) return (int)e;                                                                                                              \
        for (p.h0 = 0; p.h0 < H; p.h0 += per_pass) {                                                                                                      \
            p.heads = H - p.h0 < per_pass ? H - p.h0 : per_pass;                                                                                          \
            /* a step of few chunks: the value columns in as many shares as the SMs have room for */                                                      \
            const int items = chunks * p.heads, room = items < sms ? sms / items : 1, tiles = (Dv_in + DC_COLS - 1) / DC_COLS;                             \
            const int per_share = (tiles + room - 1) / room, splits = (tiles + per_share - 1) / per_share;                 /* (no empty share) */          \
            rc = launch_kernel(decay_local_kernel<T, DT, ONE>, dim3(chunks, p.heads, splits), dim3(DC_THREADS), smem_l, stream, p, splits);                \
            if (rc) return rc;                                                                                                                            \
            const int64_t quads = (int64_t)p.heads * Dv * D / 4;                                                                                          \
            rc = launch_kernel(decay_combine_kernel, dim3((unsigned)((quads + 127) / 128), long_rows), dim3(128), 0, stream, p);                          \
            if (rc) return rc;                                                                                                                            \
            if (items * ((Dv_in + 127) / 128) > sms / 2) DC_OUTPUT(T, DT, ONE, 8) else DC_OUTPUT(T, DT, ONE, 4)                                            \
            if (rc) return rc;                                                                                                                            \
        }                                                                                                                                                 \
        return 0;                                                                                                                                         \
    }
    if (v_tag == MIE_F32) { if (D <= 64) DC_LAUNCH(float, 64, false) else DC_LAUNCH(float, 128, false) }
    if (v_tag == MIE_BF16 && v_act) { if (D <= 64) DC_LAUNCH(bf16, 64, false) else DC_LAUNCH(bf16, 128, false) }
    if (v_tag == MIE_BF16) { if (D <= 64) DC_LAUNCH(bf16, 64, true) else DC_LAUNCH(bf16, 128, true) }
#undef DC_LAUNCH
#undef DC_OUTPUT
    return MIE_ERR_BAD_ARG;
}
