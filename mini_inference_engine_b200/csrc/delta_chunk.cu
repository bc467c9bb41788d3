// The gated delta rule over long portions, in chunks of 64 tokens (delta_rule.cu walks token by token), with one decay per head or one per head and key channel.
//
// Within a chunk, with G_i the sum of the log decays up to token i, S the state in front of the chunk and
//   A_ij = beta_i exp(G_i - G_j) (k_i . k_j)  for j < i,      P_ij = exp(G_i - G_j) (q_i . k_j)  for j <= i,
// the recurrence S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q written out is
//   (I + A) U = diag(beta) (V - diag(e^G) K S),      O = diag(e^G) Q S + P U,      S <- e^{G_C} S + (diag(e^{G_C - G}) K)^T U,
// so a chunk is six small matrix products instead of 64 dependent steps.  Every exponent is a sum of log decays over a stretch of the
// chunk and never positive.  All of it is float32 on the CUDA cores (packed two to an instruction): the state is a 32-bit quantity, and
// the corrections that U holds cancel what earlier tokens wrote, which operands rounded for the tensor cores would not.
//
//   chunk_prep   a block per (chunk, key head): K K^T and Q K^T once, then for every head of the group the factors from its decays, the
//                inverse T of the unit triangular I + A (blocks of 16: each diagonal block by substitution, the rest by products),
//                and T diag(beta), P, e^G, e^{G_C - G} into scratch memory.
//   chunk_scan   a block per (row, head, 16 value columns) walks the row's chunks: its slice of the state stays in registers (and in shared
//                memory for the products that read it); keys and queries of the next chunk arrive by asynchronous copies while
//                this one is computed.
//
// With a decay per channel G_i is a vector: e^{G_i} multiplies k_i and q_i, e^{G_C - G_i} the k_i that the state takes, and the entries of A and P are
// sums over channels with a factor each.  channel_prep (a block per (chunk, head)) writes these keys and queries out, so the scan only reads other operands.  Between blocks of 16
// tokens the factor e^{G_i - G_j} is e^{G_i - G_r} e^{G_r - G_j} with r the last token in front of i's block: two products of a matrix, no exponent
// positive, whatever the decays; within a block it is the product of the tokens' own decays, carried from token to token.
//
// Rows with fewer than `min_len` new tokens are left to delta_rule.cu.  Chunks count from the start of a row's portion.
#include "common.cuh"

#define CH 64                  // tokens a chunk
#define CHP 68                 // their stride in shared memory: rows of 64 and four words more, so that neighbouring rows lie four banks apart
#define COLS 16                // value columns a block of the scan

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ float sum2(unsigned long long v) { const float2 f = unpack2(v); return f.x + f.y; }
template <bool B> struct Flag { static constexpr bool value = B; };
struct Quad { unsigned long long lo, hi; };                    // four consecutive floats as two pairs
__device__ __forceinline__ Quad quad(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return Quad{v.x, v.y};
}
// entries m .. m + 3 of which only those up to r count: the others, whatever they are (a later token's may not be finite), become zero
__device__ __forceinline__ Quad up_to(Quad b, int m, int r) {
    if (m + 1 > r) b.lo &= 0xffffffffull;
    if (m > r) b.lo = 0ull;
    if (m + 3 > r) b.hi &= 0xffffffffull;
    if (m + 2 > r) b.hi = 0ull;
    return b;
}
// 16 (or 4) bytes from global to shared memory; zeros where `on` is false (nothing is read then)
__device__ __forceinline__ void copy16(float* dst, const float* src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// 64 rows of up to DT entries (the rest zero) into rows of DT + 4; rows from `count` on are zero.
template <int DT>
__device__ __forceinline__ void copy_rows(float* dst, const float* src, int64_t stride, int D, int count) {
    for (int c = threadIdx.x; c < CH * (DT / 4); c += blockDim.x) {
        const int r = c / (DT / 4), d = (c - r * (DT / 4)) * 4;
        const bool on = r < count && d < D;
        copy16(dst + r * (DT + 4) + d, on ? src + r * stride + d : src, on);
    }
}

struct ChunkScratch {           // per (chunk, head): T diag(beta) [64, 64], P [64, 64], e^G [64], e^{G_C - G} [64]
    float* tb; float* p; float* eg; float* er;
    __device__ __forceinline__ ChunkScratch(float* base, int64_t item) {
        tb = base + item * (2 * CH * CH + 2 * CH);
        p = tb + CH * CH;
        eg = p + CH * CH;
        er = eg + CH;
    }
};

struct ChannelScratch {         // per (chunk, head): T diag(beta) [64, 64], P [64, 64], then rows of D: e^G k [64], e^G q [64], e^{G_C - G} k [64], e^{G_C} [1]
    float* tb; float* p; float* kt; float* qt; float* ke; float* ec;
    __device__ __forceinline__ ChannelScratch(float* base, int64_t item, int D) {
        tb = base + item * (2 * CH * CH + (3 * CH + 1) * D);
        p = tb + CH * CH;
        kt = p + CH * CH;
        qt = kt + CH * D;
        ke = qt + CH * D;
        ec = ke + CH * D;
    }
};

__device__ __forceinline__ int chunks_of(int n, int min_len) { return n >= min_len ? (n + CH - 1) / CH : 0; }

// T = (I + A)^-1 for A [64][CHP] with entries below the diagonal only, by the whole block (a barrier in front and behind); X: 3 x 256 floats.
__device__ __forceinline__ void unit_triangular_inverse(const float* A, float* T, float* X) {
    // diagonal blocks: a column of the inverse a thread, by substitution, in registers
    if (threadIdx.x < 64) {
        float t[16];
        const int db = (threadIdx.x >> 4) * 16, dc = threadIdx.x & 15;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float v = i == dc ? 1.f : 0.f;
#pragma unroll
            for (int m = 0; m < i; ++m) v = fmaf(-A[(db + i) * CHP + db + m], t[m], v);
            t[i] = v;
            T[(db + i) * CHP + db + dc] = v;
        }
    }
    __syncthreads();
    // the blocks below: T_ij = -T_ii (sum over j <= m < i of A_im T_mj), one diagonal of blocks after the other
    for (int w = 1; w < 4; ++w) {
        const int n = (4 - w) * 256;                       // entries of the blocks (i, i - w)
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int bi = w + (idx >> 8), bj = bi - w, r = (idx >> 4) & 15, c = idx & 15;
            float v = 0.f;
            for (int mb = bj * 16; mb < bi * 16; mb += 16) {
                float part = 0.f;
#pragma unroll
                for (int m = 0; m < 16; ++m) part = fmaf(A[(bi * 16 + r) * CHP + mb + m], T[(mb + m) * CHP + bj * 16 + c], part);
                v += part;
            }
            X[idx] = v;
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
            const int bi = w + (idx >> 8), bj = bi - w, r = (idx >> 4) & 15, c = idx & 15;
            float v = 0.f;
#pragma unroll
            for (int m = 0; m < 16; ++m)                       // (the inverse ends at its diagonal; a later token's sums, which may not be finite, are not read)
                v = fmaf(T[(bi * 16 + r) * CHP + bi * 16 + m], m <= r ? X[(idx & ~255) + m * 16 + c] : 0.f, v);
            T[(bi * 16 + r) * CHP + bj * 16 + c] = -v;
        }
        __syncthreads();
    }
}

template <int DT>
__global__ void __launch_bounds__(256, 2) delta_chunk_prep_kernel(const float* __restrict__ qn, const float* __restrict__ kn,
                                                               const float* __restrict__ beta, const float* __restrict__ log_decay,
                                                               const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                                                               int num_rows, int min_len, float* __restrict__ scratch, int H, int G, int D, int h0, int heads) {
    extern __shared__ __align__(16) float sm[];
    float* K = sm;                                             // [64][DT + 4]
    float* Q = K + CH * (DT + 4);
    float* KK = Q + CH * (DT + 4);                             // [64][68]: k_i . k_j
    float* QK = KK + CH * CHP;                                 // q_i . k_j
    float* X = QK + CH * CHP;                                  // products on the way to T [3][16][16]
    float* A = K;                                              // [64][68], and T: keys and queries are not read after the Gram matrices
    float* T = Q;
    __shared__ float lg[CH], be[CH];
    __shared__ int s_row, s_chunk;
    pdl_enter();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        int within, items;
        const int r = warp_find_row(row_q_len, num_rows, (int)blockIdx.x, [&](int n) { return chunks_of(n, min_len); }, within, items);
        if (lane == 0) { s_row = r; s_chunk = within; }
    }
    __syncthreads();
    if (s_row < 0) return;
    const int g = h0 / (H / G) + blockIdx.y, row = s_row;
    const int t0 = row_q_start[row] + s_chunk * CH, count = min(CH, row_q_len[row] - s_chunk * CH);
    copy_rows<DT>(K, kn + ((int64_t)t0 * G + g) * D, (int64_t)G * D, D, count);
    copy_rows<DT>(Q, qn + ((int64_t)t0 * G + g) * D, (int64_t)G * D, D, count);
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    {
        // four warps a Gram matrix, 32 x 32 entries a warp, 4 x 8 a lane (rows and columns interleaved over the lanes)
        const float* L = warp < 4 ? K : Q;
        float* out = warp < 4 ? KK : QK;
        const int rb = (warp & 1) * 32, cb = ((warp >> 1) & 1) * 32, r0 = rb + (lane >> 2), c0 = cb + (lane & 3);
        if (rb >= cb) {                                        // the block wholly above the diagonal is never read
            unsigned long long acc[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
#pragma unroll 2
            for (int d = 0; d < DT; d += 4) {
                Quad a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = quad(L + (r0 + 8 * i) * (DT + 4) + d);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const Quad b = quad(K + (c0 + 4 * j) * (DT + 4) + d);
#pragma unroll
                    for (int i = 0; i < 4; ++i) { fma2(acc[i][j], a[i].lo, b.lo); fma2(acc[i][j], a[i].hi, b.hi); }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) out[(r0 + 8 * i) * CHP + c0 + 4 * j] = sum2(acc[i][j]);
        }
    }
    for (int h = g * (H / G); h < (g + 1) * (H / G); ++h) {
        __syncthreads();                                       // the Gram matrices; and the head before is done with A, T, lg and be
        if (warp == 0) {
            // sums of the log decays: two tokens a lane (tokens beyond the row's end decay nothing and write nothing)
            const int i = 2 * lane;
            const int64_t at = (int64_t)(t0 + i) * H + h;
            const float a = i < count ? log_decay[at] : 0.f, b = i + 1 < count ? log_decay[at + H] : 0.f;
            float s = a + b;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const float up = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += up; }
            lg[i] = s - b;
            lg[i + 1] = s;
        } else if (warp == 1) {
#pragma unroll
            for (int k = 0; k < 2; ++k) { const int i = lane + 32 * k; be[i] = i < count ? beta[(int64_t)(t0 + i) * H + h] : 0.f; }
        }
        __syncthreads();
        const ChunkScratch out(scratch, (int64_t)blockIdx.x * heads + h - h0);
        if (threadIdx.x < CH) {
            out.eg[threadIdx.x] = expf(lg[threadIdx.x]);
            out.er[threadIdx.x] = expf(lg[CH - 1] - lg[threadIdx.x]);
        }
        for (int idx = threadIdx.x; idx < CH * CH; idx += blockDim.x) {
            const int i = idx >> 6, j = idx & 63;
            const float f = j <= i ? expf(lg[i] - lg[j]) : 0.f;
            out.p[idx] = j <= i ? f * QK[i * CHP + j] : 0.f;
            A[i * CHP + j] = j < i ? be[i] * f * KK[i * CHP + j] : 0.f;
        }
        __syncthreads();
        unit_triangular_inverse(A, T, X);
        for (int idx = threadIdx.x; idx < CH * CH; idx += blockDim.x) {
            const int i = idx >> 6, j = idx & 63;
            out.tb[idx] = j <= i ? T[i * CHP + j] * be[j] : 0.f;
        }
    }
}

// The sums over the lanes of v[0 .. 31], one a lane: lane l gets that of v[l].
__device__ __forceinline__ float transposed_sums(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

#define CP_THREADS 512

// 170 KB: one block of 16 warps on an SM.  1,500 tokens of 16 heads of 128: 136 us with a load of the decays in every step of the walk within a block, 75 us with
// a block's decays read ahead and all columns of a row summed over the lanes at once.
template <int DT>
__global__ void __launch_bounds__(CP_THREADS) delta_channel_prep_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ beta,
                                                                        const float* __restrict__ decay, const float* __restrict__ log_decay,
                                                                        const int* __restrict__ row_q_start, const int* __restrict__ row_q_len, int num_rows,
                                                                        int min_len, float* __restrict__ scratch, int H, int G, int D, int h0, int heads) {
    constexpr int DP = DT + 4;
    extern __shared__ __align__(16) float sm[];
    float* K = sm;                                             // [64][DP]; then e^(sum from the block's first token) k
    float* Q = K + CH * DP;                                    // ... q
    float* R = Q + CH * DP;                                    // log decays, then e^(sum from the next token to the block's last) k: no exponent is the difference of two larger ones
    float* KK = R + CH * DP;                                   // [64][CHP]: A before beta
    float* QK = KK + CH * CHP;                                 // P
    float* tot = QK + CH * CHP;                                // [4][DT]: the log decays of whole blocks
    float* Y = tot + 4 * DT;                                   // [4 quarters of the channels][KK, QK][64][16]: the blocks on the diagonal
    float* A = KK;
    float* T = K;                                              // (the keys and queries are not read after the products)
    float* X = Q;
    __shared__ float be[CH];
    __shared__ int s_row, s_chunk;
    pdl_enter();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        int within, items;
        const int r = warp_find_row(row_q_len, num_rows, (int)blockIdx.x, [&](int n) { return chunks_of(n, min_len); }, within, items);
        if (lane == 0) { s_row = r; s_chunk = within; }
    }
    __syncthreads();
    if (s_row < 0) return;
    const int h = h0 + blockIdx.y, g = h / (H / G);
    const int t0 = row_q_start[s_row] + s_chunk * CH, count = min(CH, row_q_len[s_row] - s_chunk * CH);
    copy_rows<DT>(K, kn + ((int64_t)t0 * G + g) * D, (int64_t)G * D, D, count);
    copy_rows<DT>(Q, qn + ((int64_t)t0 * G + g) * D, (int64_t)G * D, D, count);
    copy_rows<DT>(R, log_decay + ((int64_t)t0 * H + h) * D, (int64_t)H * D, D, count);       // (tokens beyond the row's end decay nothing and write nothing)
    copy_commit();
    if (threadIdx.x < CH) be[threadIdx.x] = threadIdx.x < count ? beta[(int64_t)(t0 + threadIdx.x) * H + h] : 0.f;
    // within a block of 16 tokens: a warp a block and a quarter of the channels; the factor of every column is carried from row to row
    constexpr int PER = DT / 128 > 0 ? DT / 128 : 1;           // (DT 64: half of the lanes have a channel)
    const int blk = warp >> 2, d = ((warp & 3) * 32 + lane) * PER;
    const bool on = d < DT && d < D;
    float w[16];
#pragma unroll
    for (int i = 1; i < 16; ++i) w[i] = on && 16 * blk + i < count ? decay[((int64_t)(t0 + 16 * blk + i) * H + h) * D + d] : 1.f;
    copy_wait<0>();
    __syncthreads();
    {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float k = on ? K[(16 * blk + i) * DP + d] : 0.f, q = on ? Q[(16 * blk + i) * DP + d] : 0.f;
            float v[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (j < i) f[j] *= w[i];
                if (j == i) f[j] = k;
                v[j] = j <= i ? k * f[j] : 0.f;
                v[16 + j] = j <= i ? q * f[j] : 0.f;
            }
            const float sum = transposed_sums(v, lane);        // lane j: k_i . k_j, lane 16 + j: q_i . k_j over this warp's channels
            Y[(((warp & 3) * 2 + (lane >> 4)) * CH + 16 * blk + i) * 16 + (lane & 15)] = sum;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * CH * CH; i += CP_THREADS) {
        const int which = i >> 12, r = (i >> 6) & 63, c = i & 63;
        const float* y = Y + (which * CH + r) * 16 + (c & 15);
        (which ? QK : KK)[r * CHP + c] = (r >> 4) == (c >> 4) ? (y[0] + y[2 * CH * 16]) + (y[4 * CH * 16] + y[6 * CH * 16]) : 0.f;
    }
    // sums of log decays; keys and queries with their factors, into scratch memory and, for the products between blocks, in place
    const ChannelScratch out(scratch, (int64_t)blockIdx.x * heads + blockIdx.y, D);
    for (int c = threadIdx.x; c < 4 * DT; c += CP_THREADS) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) s += R[((c / DT) * 16 + i) * DP + c % DT];
        tot[c] = s;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < 4 * DT; c += CP_THREADS) {
        const int b = c / DT, e = c % DT;
        if (e >= D) {
            for (int i = 16 * b; i < 16 * b + 16; ++i) R[i * DP + e] = 0.f;
            continue;
        }
        float before = 0.f, behind = 0.f, x[16], k[16];
        for (int m = 0; m < b; ++m) before += tot[m * DT + e];
        for (int m = b + 1; m < 4; ++m) behind += tot[m * DT + e];
#pragma unroll
        for (int i = 0; i < 16; ++i) { x[i] = R[(16 * b + i) * DP + e]; k[i] = K[(16 * b + i) * DP + e]; }
        float run = 0.f;
        const float all_behind = expf(behind), all_before = expf(before);
#pragma unroll
        for (int i = 15; i >= 0; --i) {
            const int at = 16 * b + i;
            const float back = expf(run);
            R[at * DP + e] = k[i] * back;
            out.ke[at * D + e] = k[i] * back * all_behind;
            run += x[i];
        }
        run = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int at = 16 * b + i;
            run += x[i];
            const float fwd = expf(run), q = Q[at * DP + e];
            K[at * DP + e] = k[i] * fwd;
            Q[at * DP + e] = q * fwd;
            out.kt[at * D + e] = k[i] * fwd * all_before;
            out.qt[at * D + e] = q * fwd * all_before;
            if (at == CH - 1) out.ec[e] = expf(before + run);
        }
    }
    __syncthreads();
    // between blocks: a warp a pair of blocks and half of the channels; the keys and the queries of block bi against the keys of block bj
    float part[4][4];
    const int pair = warp >> 1, bi = pair < 1 ? 1 : pair < 3 ? 2 : 3, bj = pair < 1 ? 0 : pair < 3 ? pair - 1 : pair - 3;
    const int r = lane >> 2, c = lane & 3;
    if (warp < 12) {
        unsigned long long acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        const int d0 = (warp & 1) * (DT / 2);
#pragma unroll 2
        for (int dd = d0; dd < d0 + DT / 2; dd += 4) {
            float4 m = make_float4(1.f, 1.f, 1.f, 1.f);        // the blocks between the two
            if (bi - bj > 1) {
                float4 s = *reinterpret_cast<const float4*>(tot + (bj + 1) * DT + dd);
                if (bi - bj > 2) {
                    const float4 t = *reinterpret_cast<const float4*>(tot + (bj + 2) * DT + dd);
                    s = make_float4(s.x + t.x, s.y + t.y, s.z + t.z, s.w + t.w);
                }
                m = make_float4(expf(s.x), expf(s.y), expf(s.z), expf(s.w));
            }
            Quad a[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 x = *reinterpret_cast<const float4*>((i < 2 ? K : Q) + (16 * bi + r + 8 * (i & 1)) * DP + dd);
                a[i].lo = pack2(x.x * m.x, x.y * m.y);
                a[i].hi = pack2(x.z * m.z, x.w * m.w);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const Quad y = quad(R + (16 * bj + c + 4 * j) * DP + dd);
#pragma unroll
                for (int i = 0; i < 4; ++i) { fma2(acc[i][j], a[i].lo, y.lo); fma2(acc[i][j], a[i].hi, y.hi); }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[i][j] = sum2(acc[i][j]);
    }
    for (int half = 0; half < 2; ++half) {
        if (warp < 12 && (warp & 1) == half) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float* to = (i < 2 ? KK : QK) + (16 * bi + r + 8 * (i & 1)) * CHP + 16 * bj + c + 4 * j;
                    *to = half ? *to + part[i][j] : part[i][j];
                }
        }
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < CH * CH; idx += CP_THREADS) {
        const int i = idx >> 6, j = idx & 63;
        out.p[idx] = QK[i * CHP + j];
        A[i * CHP + j] = j < i ? be[i] * KK[i * CHP + j] : 0.f;
    }
    __syncthreads();
    unit_triangular_inverse(A, T, X);
    for (int idx = threadIdx.x; idx < CH * CH; idx += CP_THREADS) {
        const int i = idx >> 6, j = idx & 63;
        out.tb[idx] = j <= i ? T[i * CHP + j] * be[j] : 0.f;
    }
}

// CHANNEL: a decay per channel -- the operands come with their factors from channel_prep, and the keys that the state takes replace the others in
// shared memory once the products with the state are done with those.
template <int DT, bool CHANNEL>
__global__ void __launch_bounds__(256) delta_chunk_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vn,
                                                               const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                                                               const int* __restrict__ state_slots, int min_len, const float* __restrict__ scratch,
                                                               float* __restrict__ state, float* __restrict__ out, int H, int G, int D, int Dv, int h0, int heads) {
    constexpr int DP = DT + 4;
    extern __shared__ __align__(16) float sm[];
    float* KQ = sm;                                            // two stages of K [64][DP] | Q [64][DP] | V [64][16] | e^G [64] | e^{G_C - G} [64]
    constexpr int STAGE = 2 * CH * DP + CH * COLS + 2 * CH;
    float* TB = KQ + 2 * STAGE;                                // [64][68]
    float* P = TB + CH * CHP;                                  // [64][68]
    float* S = P + CH * CHP;                                   // the state's columns [16][DP]
    float* R = S + COLS * DP;                                  // V - e^G K S, column by column [16][68]
    float* U = R + COLS * CHP;                                 // [16][68]
    float* UE = U + COLS * CHP;                                // U with e^{G_C - G} [16][68]
    __shared__ int s_first;
    pdl_enter();
    const int row = blockIdx.x, h = h0 + blockIdx.y, j0 = blockIdx.z * COLS;
    const int n = row_q_len[row], chunks = chunks_of(n, min_len);
    if (chunks == 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {                                           // where the row's chunks begin in the scratch memory
        int first = 0;
        for (int r = lane; r < row; r += 32) first += chunks_of(row_q_len[r], min_len);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
        if (lane == 0) s_first = first;
    }
    __syncthreads();
    const int t0 = row_q_start[row], g = h / (H / G);
    const int64_t first = s_first;
    float* sp = state + ((int64_t)state_slots[row] * H + h) * Dv * D;

    // the thread's part of the state, for warps 0 .. 3: entries d4 .. d4 + 3 of JT columns
    constexpr int JT = DT == 128 ? 4 : 2;
    const int d4 = (DT == 128 ? warp : warp & 1) * 32 + (lane & 7) * 4, jl = (lane >> 3) + (DT == 128 ? 0 : (warp >> 1) * 8);
    unsigned long long s_lo[JT], s_hi[JT];
    if (warp < 4) {
#pragma unroll
        for (int jj = 0; jj < JT; ++jj) {
            const int j = jl + 4 * jj;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 + j < Dv && d4 < D) v = *reinterpret_cast<const float4*>(sp + (int64_t)(j0 + j) * D + d4);
            *reinterpret_cast<float4*>(S + j * DP + d4) = v;
            s_lo[jj] = pack2(v.x, v.y);
            s_hi[jj] = pack2(v.z, v.w);
        }
    }
    auto issue_keys = [&](int c) {                             // every thread commits one group, also an empty one
        if (c < chunks) {
            float* st = KQ + (c & 1) * STAGE;
            const int64_t tf = t0 + c * CH;
            const int count = min(CH, n - c * CH);
            if constexpr (CHANNEL) {
                const ChannelScratch in(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y, D);
                copy_rows<DT>(st, in.kt, D, D, CH);
                copy_rows<DT>(st + CH * DP, in.qt, D, D, CH);
            } else {
                copy_rows<DT>(st, kn + (tf * G + g) * D, (int64_t)G * D, D, count);
                copy_rows<DT>(st + CH * DP, qn + (tf * G + g) * D, (int64_t)G * D, D, count);
            }
            float* v = st + 2 * CH * DP;
            for (int i = threadIdx.x; i < CH * COLS; i += 256) {
                const int t = i >> 4, j = i & 15;
                const bool on = t < count && j0 + j < Dv;
                copy4(v + i, on ? vn + ((tf + t) * H + h) * Dv + j0 + j : vn, on);
            }
            if constexpr (CHANNEL) {
                const float* ec = ChannelScratch(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y, D).ec;
                if (threadIdx.x < DT / 4) copy16(v + CH * COLS + threadIdx.x * 4, threadIdx.x * 4 < D ? ec + threadIdx.x * 4 : ec, threadIdx.x * 4 < D);
            } else if (threadIdx.x < 32) {
                const float* eg = ChunkScratch(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y).eg;      // e^G and e^{G_C - G} lie side by side
                copy16(v + CH * COLS + threadIdx.x * 4, eg + threadIdx.x * 4, true);
            }
        }
        copy_commit();
    };
    auto issue_squares = [&](int c) {
        const float* tb = CHANNEL ? ChannelScratch(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y, D).tb
                                  : ChunkScratch(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y).tb;
        for (int i = threadIdx.x; i < CH * CH / 4; i += 256) {
            const int r = i >> 4, m = (i & 15) * 4;
            copy16(TB + r * CHP + m, tb + i * 4, true);
            copy16(P + r * CHP + m, tb + CH * CH + i * 4, true);
        }
        copy_commit();
    };
    issue_keys(0);
    // rows and columns of a lane: in the products with S four rows and two columns (warps 0 .. 3 the keys, 4 .. 7 the queries, 16 rows
    // a warp), in U two rows and two columns (8 rows a warp); always interleaved over the lanes
    const int half = warp >> 2, r1 = (warp & 3) * 16 + (lane >> 3), c1 = lane & 7;
    // (warps w and w + 4 share a scheduler: short and long rows of the triangle are dealt to them in pairs)
    const int rw = half ? 7 - (warp & 3) : (warp & 3), r2 = rw * 8 + (lane >> 3);
    for (int c = 0; c < chunks; ++c) {
        copy_wait<0>();                                        // keys and queries of this chunk
        __syncthreads();                                       // ... of every thread; S of the chunk before; TB and P are free
        issue_squares(c);
        if constexpr (!CHANNEL) issue_keys(c + 1);
        float* st = KQ + (c & 1) * STAGE;
        const float* V = st + 2 * CH * DP;
        const float* eg = V + CH * COLS;
        const float* er = eg + CH;
        unsigned long long acc[4][2];
        float o[4][2];
        {
            const float* L = st + half * CH * DP;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
#pragma unroll 4
            for (int d = 0; d < DT; d += 4) {
                const Quad b0 = quad(S + c1 * DP + d), b1 = quad(S + (c1 + 8) * DP + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const Quad a = quad(L + (r1 + 4 * i) * DP + d);
                    fma2(acc[i][0], a.lo, b0.lo); fma2(acc[i][0], a.hi, b0.hi);
                    fma2(acc[i][1], a.lo, b1.lo); fma2(acc[i][1], a.hi, b1.hi);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = r1 + 4 * i;
                const float e = CHANNEL ? 1.f : eg[r];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    o[i][k] = e * sum2(acc[i][k]);
                    if (half == 0) R[(c1 + 8 * k) * CHP + r] = V[r * COLS + c1 + 8 * k] - o[i][k];
                }
            }
        }
        if constexpr (CHANNEL) {
            __syncthreads();                                   // the keys are done with: those that the state takes come in their place
            copy_rows<DT>(st, ChannelScratch(const_cast<float*>(scratch), (first + c) * heads + blockIdx.y, D).ke, D, D, CH);
            copy_commit();
            issue_keys(c + 1);
            copy_wait<2>();
        } else copy_wait<1>();                                 // TB and P of this chunk
        __syncthreads();
        {
            unsigned long long u[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
            const int end = rw * 8 + 8;                        // no row of the warp reads beyond its diagonal
            auto add = [&](int m, auto diagonal) {
                const Quad b0 = quad(R + c1 * CHP + m), b1 = quad(R + (c1 + 8) * CHP + m);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const Quad a = quad(TB + (r2 + 4 * i) * CHP + m);
                    const Quad x = diagonal.value ? up_to(b0, m, r2 + 4 * i) : b0, y = diagonal.value ? up_to(b1, m, r2 + 4 * i) : b1;
                    fma2(u[i][0], a.lo, x.lo); fma2(u[i][0], a.hi, x.hi);
                    fma2(u[i][1], a.lo, y.lo); fma2(u[i][1], a.hi, y.hi);
                }
            };
#pragma unroll 2
            for (int m = 0; m < end - 8; m += 4) add(m, Flag<false>{});
            add(end - 8, Flag<true>{});
            add(end - 4, Flag<true>{});
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = r2 + 4 * i;
                const float e = CHANNEL ? 1.f : er[r];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float v = sum2(u[i][k]);
                    U[(c1 + 8 * k) * CHP + r] = v;
                    if constexpr (!CHANNEL) UE[(c1 + 8 * k) * CHP + r] = e * v;
                }
            }
        }
        if constexpr (CHANNEL) copy_wait<1>();                 // the keys that the state takes
        __syncthreads();
        if (half == 0) {
            // the state: its columns times the chunk's whole decay, plus keys times U
            unsigned long long t_lo, t_hi;
            if constexpr (CHANNEL) { const Quad e = quad(eg + d4); t_lo = e.lo; t_hi = e.hi; }
            else t_lo = t_hi = pack2(eg[CH - 1], eg[CH - 1]);
            const float* taken = CHANNEL ? U : UE;
            unsigned long long n_lo[JT], n_hi[JT];
#pragma unroll
            for (int jj = 0; jj < JT; ++jj) { n_lo[jj] = n_hi[jj] = 0ull; fma2(n_lo[jj], s_lo[jj], t_lo); fma2(n_hi[jj], s_hi[jj], t_hi); }
#pragma unroll 2
            for (int i = 0; i < CH; i += 4) {
                float4 u[JT];
#pragma unroll
                for (int jj = 0; jj < JT; ++jj) u[jj] = *reinterpret_cast<const float4*>(taken + (jl + 4 * jj) * CHP + i);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const Quad key = quad(st + (i + k) * DP + d4);
#pragma unroll
                    for (int jj = 0; jj < JT; ++jj) {
                        const float x = k == 0 ? u[jj].x : k == 1 ? u[jj].y : k == 2 ? u[jj].z : u[jj].w;
                        const unsigned long long xx = pack2(x, x);
                        fma2(n_lo[jj], key.lo, xx);
                        fma2(n_hi[jj], key.hi, xx);
                    }
                }
            }
#pragma unroll
            for (int jj = 0; jj < JT; ++jj) {
                s_lo[jj] = n_lo[jj];
                s_hi[jj] = n_hi[jj];
                *reinterpret_cast<ulonglong2*>(S + (jl + 4 * jj) * DP + d4) = make_ulonglong2(n_lo[jj], n_hi[jj]);
            }
        } else {
            // the outputs: what the state gave the queries, plus P U
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
            const int end = (warp & 3) * 16 + 16;
            auto add = [&](int m, auto diagonal) {
                const Quad b0 = quad(U + c1 * CHP + m), b1 = quad(U + (c1 + 8) * CHP + m);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const Quad a = quad(P + (r1 + 4 * i) * CHP + m);
                    const Quad x = diagonal.value ? up_to(b0, m, r1 + 4 * i) : b0, y = diagonal.value ? up_to(b1, m, r1 + 4 * i) : b1;
                    fma2(acc[i][0], a.lo, x.lo); fma2(acc[i][0], a.hi, x.hi);
                    fma2(acc[i][1], a.lo, y.lo); fma2(acc[i][1], a.hi, y.hi);
                }
            };
#pragma unroll 2
            for (int m = 0; m < end - 16; m += 4) add(m, Flag<false>{});
#pragma unroll
            for (int m = 16; m > 0; m -= 4) add(end - m, Flag<true>{});
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = c * CH + r1 + 4 * i;
                if (t >= n) continue;
                float* dst = out + ((int64_t)(t0 + t) * H + h) * Dv + j0;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (j0 + c1 + 8 * k < Dv) dst[c1 + 8 * k] = o[i][k] + sum2(acc[i][k]);
            }
        }
    }
    if (warp < 4) {
#pragma unroll
        for (int jj = 0; jj < JT; ++jj) {
            const int j = jl + 4 * jj;
            if (j0 + j >= Dv || d4 >= D) continue;
            const float2 a = unpack2(s_lo[jj]), b = unpack2(s_hi[jj]);
            *reinterpret_cast<float4*>(sp + (int64_t)(j0 + j) * D + d4) = make_float4(a.x, a.y, b.x, b.y);
        }
    }
}

// The heads of `per_pass` key heads at a time, one pass behind the other on the same scratch memory.
template <int DT>
static int launch_chunks(const float* qn, const float* kn, const float* vn, const float* beta, const float* decay, const float* log_decay, const int* row_q_start,
                         const int* row_q_len, const int* state_slots, float* state, float* out, float* scratch, int max_chunks, int num_rows,
                         int min_len, int H, int G, int D, int Dv, int per_pass, cudaStream_t stream) {
    const size_t scan = (size_t)(2 * (2 * CH * (DT + 4) + CH * COLS + 2 * CH) + 2 * CH * CHP + COLS * (DT + 4) + 3 * COLS * CHP) * sizeof(float);
    // a decay per channel: one block on an SM; one per head: two
    const size_t prep = decay ? (size_t)(3 * CH * (DT + 4) + 2 * CH * CHP + 4 * DT + 8 * CH * 16) * sizeof(float)
                              : (size_t)(2 * CH * (DT + 4) + 2 * CH * CHP + 3 * 256) * sizeof(float);
    auto scan_kernel = decay ? delta_chunk_scan_kernel<DT, true> : delta_chunk_scan_kernel<DT, false>;
    cudaError_t e = decay ? cudaFuncSetAttribute(delta_channel_prep_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep)
                          : cudaFuncSetAttribute(delta_chunk_prep_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scan);
    if (e != cudaSuccess) return (int)e;
    for (int g0 = 0; g0 < G; g0 += per_pass) {
        const int groups = G - g0 < per_pass ? G - g0 : per_pass, h0 = g0 * (H / G), heads = groups * (H / G);
        int rc = decay ? launch_kernel(delta_channel_prep_kernel<DT>, dim3(max_chunks, heads), dim3(CP_THREADS), prep, stream, qn, kn, beta, decay, log_decay,
                                       row_q_start, row_q_len, num_rows, min_len, scratch, H, G, D, h0, heads)
                       : launch_kernel(delta_chunk_prep_kernel<DT>, dim3(max_chunks, groups), dim3(256), prep, stream, qn, kn, beta, log_decay, row_q_start,
                                       row_q_len, num_rows, min_len, scratch, H, G, D, h0, heads);
        if (rc) return rc;
        rc = launch_kernel(scan_kernel, dim3(num_rows, heads, (Dv + COLS - 1) / COLS), dim3(256), scan, stream, qn, kn, vn, row_q_start, row_q_len, state_slots,
                           min_len, (const float*)scratch, state, out, H, G, D, Dv, h0, heads);
        if (rc) return rc;
    }
    return 0;
}

// Floats of scratch memory for one (chunk, head); tokens a chunk.
extern "C" int mie_delta_chunk_floats(int per_channel, int D) { return 2 * CH * CH + (per_channel ? (3 * CH + 1) * D : 2 * CH); }
extern "C" int mie_delta_chunk_tokens(void) { return CH; }

// qn, kn: float32 [T, G, D]; vn, out: [T, H, Dv]; beta [T, H]; log_decay (not positive) [T, H] with `decay` null, or [T, H, D] with `decay` [T, H, D] its
// exponential; state [slots, H, Dv, D].  D a multiple of 4 up to 128, everything 16-byte aligned.  max_chunks: no fewer than the chunks of all rows with min_len tokens or more; the heads of
// `per_pass` key heads at a time: scratch holds max_chunks * per_pass * H / G times mie_delta_chunk_floats() floats.
extern "C" int mie_delta_chunks(const float* qn, const float* kn, const float* vn, const float* beta, const float* decay, const float* log_decay,
                                const int* row_q_start, const int* row_q_len, const int* state_slots, float* state, float* out, float* scratch,
                                int max_chunks, int num_rows, int min_len, int H, int G, int D, int Dv, int per_pass, cudaStream_t stream) {
    if (num_rows <= 0 || max_chunks <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || D % 4 || Dv <= 0 || min_len < 1 || per_pass < 1) return MIE_ERR_BAD_ARG;
    if (D > 128 || H > 65535) return MIE_ERR_TOO_LARGE;
    if (decay && ((reinterpret_cast<uintptr_t>(decay) | reinterpret_cast<uintptr_t>(log_decay)) & 15)) return MIE_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(qn) | reinterpret_cast<uintptr_t>(kn) | reinterpret_cast<uintptr_t>(state) | reinterpret_cast<uintptr_t>(scratch)) & 15)
        return MIE_ERR_BAD_ARG;
    if (D <= 64)
        return launch_chunks<64>(qn, kn, vn, beta, decay, log_decay, row_q_start, row_q_len, state_slots, state, out, scratch, max_chunks, num_rows, min_len, H, G, D, Dv, per_pass, stream);
    return launch_chunks<128>(qn, kn, vn, beta, decay, log_decay, row_q_start, row_q_len, state_slots, state, out, scratch, max_chunks, num_rows, min_len, H, G, D, Dv, per_pass, stream);
}
