// The recurrences of recurrent_block.cu (and retention) over long portions, 32 tokens at a time (fp32 in and out), for heads of 64 key channels; which
// steps take them is chunks_pay's choice, in the Python wrappers:
//
//     gated delta rule   S <- g_t S;   S <- S + k_t (b_t (v_t - S^T k_t))^T;   o_t = S^T q_t
//     one fixed decay    S <- g S + k_t v_t^T;   o_t = S^T q_t                        (lightning attention, retention; u_t = v_t)
//
// With S the state before a chunk of tokens 0 .. 31, P_j = g_0 .. g_j and R_ij = g_{i+1} .. g_j, the rule over the chunk is
//     u_j = b_j (v_j - P_j S^T k_j - sum_{i<j} R_ij (k_i . k_j) u_i)
//     o_j = P_j S^T q_j + sum_{i<=j} R_ij (k_i . q_j) u_i
//     S  <- P_31 S + sum_i R_i,31 k_i u_i^T
// and what waits for S is little: the triangle of the u_j is solved for both of its right-hand sides ahead, U from b_j v_j and W from
// b_j P_j k_j, so that u = U - W S.  Three kernels, of which only the second walks a request's chunks one after the other:
//     1  per (chunk, head)          W and U                          (fixed decay: Z = sum_i R_i,31 k_i v_i^T, all a chunk does to the state)
//     2  per (request, head, cols)  u = U - W S, the state before every chunk kept, S moved on
//                                   (fixed decay: S <- P_31 S + Z)
//     3  per (chunk, head)          the outputs, from the kept states
// The block scan they replace makes a chain of 900 instructions of every eight tokens with two to four warps an SM.  2,001 tokens in three portions, 32 heads:
// 216 us with its gram matrices, 140 us here (solve 29, walk 73, outputs 38).  Fixed decay, 1,500 tokens in two portions, 64 heads: 252 us token by
// token, 110 us here before the outputs went to the tensor cores.  Every R is a product of its decays (no quotients), so a decay of zero does no harm.  Scratch: W, U [chunks, N, 32, 64 | V] and the states
// [chunks, N, 64, V], chunks = T / 32 + S.
#include "common.cuh"
#include "mma_sync.cuh"

namespace {

constexpr int CH = 32, K = 64, kThreads = 128, LD = K + 4, VB = 64, kColsB = 16;

__device__ __forceinline__ void stage16(float* dst, const float* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void stages_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void stages_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Chunks {
    const float *q, *k, *v;
    int ld_q, ld_k, ld_v;
    const float* g;                   // DELTA: decays [T, N]; else [N]
    const float* beta;                // DELTA: [T, N]
    float *w, *u, *s;
    float* state;
    long long stride;
    const int32_t *q_start, *slots;
    float* out;
    int S, N, M, V;
};

// The first chunk of request s in the row of all requests' chunks (n tokens take at most n/32 + 1 of them).
__device__ __forceinline__ int first_chunk(const int32_t* __restrict__ q_start, int s) { return q_start[s] / CH + s; }

// The tokens of a chunk: the first one and how many (0: a chunk that its request does not have).
__device__ __forceinline__ int chunk_tokens(const Chunks& d, int chunk, int& t0) {
    int lo = 0, hi = d.S - 1;                                 // the last request whose first chunk is not behind this one
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (first_chunk(d.q_start, mid) <= chunk) lo = mid;
        else hi = mid - 1;
    }
    t0 = d.q_start[lo] + (chunk - first_chunk(d.q_start, lo)) * CH;
    return min(CH, d.q_start[lo + 1] - t0);
}

// 32 rows of 64 numbers (row t at src + t * ld), zeros from row n on, as rows of LD
template <int THREADS = kThreads>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int ld, int n) {
    for (int i = threadIdx.x; i < CH * K / 4; i += THREADS) {
        const int r = i / (K / 4), c = i % (K / 4) * 4;
        stage16(dst + r * LD + c, r < n ? src + (size_t)r * ld + c : src, r < n);
    }
}

// r[j][i] = g_{i+1} .. g_j for i <= j (zero above): thread j of the first 32 makes row j.
__device__ __forceinline__ void decay_triangle(float (*r)[CH + 1], const float* g) {
    if (threadIdx.x < CH) {
        const int j = threadIdx.x;
        float x = 1.f;
        for (int i = CH - 1; i >= 0; --i) {
            r[j][i] = i <= j ? x : 0.f;
            if (i <= j) x *= g[i];
        }
    }
}

// The products of chunks on the tensor cores (m16n8k16): an fp32 number as the sum of three bfloat16 ones (its rounding, the rounding of what that
// left, and of what that left: 2^-26 of it at most is missing), of the nine products of two such sums the six largest, each exact, fp32 sums.  The tensor
// core cuts what an addend has below a sum's last place, so the large terms have a sum of their own over few steps; the state itself is moved on by
// multiply-adds.  A number that is not finite, or that rounds to a bfloat16 infinity, makes NaN of the sums that it takes part in: a sum that is not finite
// is therefore made again by multiply-adds (made_again; in the walk, whose loop has neither a register nor a branch to spare, all of it: walk_again).
struct Terms { uint32_t h, m, l; };                           // of two neighbouring numbers each
__device__ __forceinline__ Terms split2(float x, float y) {
    Terms t;
    t.h = mma_sync::pack_bf16(x, y);
    x -= __uint_as_float(t.h << 16);
    y -= __uint_as_float(t.h & 0xffff0000u);
    t.m = mma_sync::pack_bf16(x, y);
    t.l = mma_sync::pack_bf16(x - __uint_as_float(t.m << 16), y - __uint_as_float(t.m & 0xffff0000u));
    return t;
}
// main += the large term, rest += the others, of A (rows g and g + 8, steps 2t and 2t + 8 on) times B (steps 2t and 2t + 8 on, column g)
__device__ __forceinline__ void mma_terms(float (&main)[4], float (&rest)[4], const Terms (&a)[4], const Terms (&b)[2]) {
    const uint32_t ah[4] = {a[0].h, a[1].h, a[2].h, a[3].h}, am[4] = {a[0].m, a[1].m, a[2].m, a[3].m}, al[4] = {a[0].l, a[1].l, a[2].l, a[3].l};
    mma_sync::mma_bf16(rest, al, b[0].h, b[1].h);
    mma_sync::mma_bf16(main, ah, b[0].h, b[1].h);
    mma_sync::mma_bf16(rest, ah, b[0].l, b[1].l);
    mma_sync::mma_bf16(rest, am, b[0].m, b[1].m);
    mma_sync::mma_bf16(rest, am, b[0].h, b[1].h);
    mma_sync::mma_bf16(rest, ah, b[0].m, b[1].m);
}
// (the walk's: two chains of the others, as little as possible waits for the sum before)
__device__ __forceinline__ void mma_terms(float (&main)[4], float (&rest)[2][4], const Terms (&a)[4], const Terms (&b)[2]) {
    const uint32_t ah[4] = {a[0].h, a[1].h, a[2].h, a[3].h}, am[4] = {a[0].m, a[1].m, a[2].m, a[3].m}, al[4] = {a[0].l, a[1].l, a[2].l, a[3].l};
    mma_sync::mma_bf16(rest[0], al, b[0].h, b[1].h);
    mma_sync::mma_bf16(rest[1], am, b[0].h, b[1].h);
    mma_sync::mma_bf16(main, ah, b[0].h, b[1].h);
    mma_sync::mma_bf16(rest[0], ah, b[0].l, b[1].l);
    mma_sync::mma_bf16(rest[1], ah, b[0].m, b[1].m);
    mma_sync::mma_bf16(rest[0], am, b[0].m, b[1].m);
}

// Whether a number among four is not finite, as one number that is then NaN, else zero.
__device__ __forceinline__ float odd4(const float (&x)[4]) { return fmaf(x[0], 0.f, x[1] * 0.f) + fmaf(x[2], 0.f, x[3] * 0.f); }
// A sum of the tensor cores, or if it is not finite the multiply-adds of a[i * lda] b[i * ldb], i < n, that it stands for.
__device__ __forceinline__ float made_again(float sum, const float* a, int lda, const float* b, int ldb, int n) {
    if (isfinite(sum)) return sum;
    sum = 0.f;
#pragma unroll 1
    for (int i = 0; i < n; ++i) sum = fmaf(a[i * lda], b[i * ldb], sum);
    return sum;
}

// A B^T, 16 x 16 over 64: rows gr (and 8 further on) of A and of B at rows of LD, two 16 x 8 tiles
__device__ __forceinline__ void square16(float (&main)[2][4], const float* a, const float* b, int gr, int tq) {
    float rest[2][4] = {};
    const float *a0 = a + gr * LD, *b0 = b + 2 * tq * LD;
    auto pair = [](const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return split2(v.x, v.y); };
    a += gr * LD + 2 * tq;
    b += gr * LD + 2 * tq;
#pragma unroll
    for (int kk = 0; kk < K; kk += 16) {
        const Terms at[4] = {pair(a + kk), pair(a + 8 * LD + kk), pair(a + kk + 8), pair(a + 8 * LD + kk + 8)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const Terms bt[2] = {pair(b + 8 * h * LD + kk), pair(b + 8 * h * LD + kk + 8)};
            mma_terms(main[h], rest[h], at, bt);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 4; ++e) main[h][e] += rest[h][e];
    if (odd4(main[0]) + odd4(main[1]) != 0.f) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) main[h][e] = made_again(main[h][e], a0 + (e >> 1) * 8 * LD, 1, b0 + (8 * h + (e & 1)) * LD, 1, K);
    }
}

// ------------------------------------------------------------------------------------------------ 1: before the walk
// DELTA: thread c solves the triangle for column c of [W | U].  The triangle itself, k k^T, is three 16 x 16 products on the tensor cores: as fp32 dot
// products its operands were two thirds of the shared-memory reads that bound the kernel (2,001 tokens, 32 heads: 38.8 us, 28.7 so).
__global__ void __launch_bounds__(kThreads)
chunk_solve_kernel(const Chunks d) {
    __shared__ __align__(16) float ks[CH * LD], A[CH][CH + 4];
    __shared__ float R[CH][CH + 1], gs[CH], bs[CH], P[CH];
    // (no early word to the scheduler: the walk's few CTAs would be placed between this kernel's many)
    forge::pdl_wait();
    int t0;
    const int chunk = blockIdx.x, head = blockIdx.y, n = chunk_tokens(d, chunk, t0), tid = threadIdx.x;
    if (n <= 0) return;
    stage_rows(ks, d.k + (size_t)t0 * d.ld_k + head / (d.N / d.M) * K, d.ld_k, n);
    stages_commit();
    if (tid < CH) {
        gs[tid] = tid < n ? d.g[(size_t)(t0 + tid) * d.N + head] : 1.0f;
        bs[tid] = tid < n ? d.beta[(size_t)(t0 + tid) * d.N + head] : 0.f;
    }
    __syncthreads();
    decay_triangle(R, gs);
    if (tid == CH) {
        float p = 1.f;
        for (int i = 0; i < CH; ++i) P[i] = p *= gs[i];
    }
    stages_wait<0>();
    __syncthreads();
    {
        // rows m0 .. m0 + 15, columns n0 .. n0 + 15 of k k^T under the diagonal, kept transposed: what row i does to the rows below
        const int warp = tid >> 5, gr = (tid & 31) >> 2, tq = tid & 3, m0 = (warp & 1) * 16, n0 = (warp >> 1) * 16;
        if (n0 <= m0) {
            float main[2][4] = {};
            square16(main, ks + m0 * LD, ks + n0 * LD, gr, tq);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = m0 + gr + (e >> 1) * 8, i = n0 + 8 * h + 2 * tq + (e & 1);
                    A[i][j] = bs[j] * R[j][i] * main[h][e];
                }
        }
    }
    __syncthreads();
    for (int c = tid; c < K + d.V; c += kThreads) {
        float x[CH];
        if (c < K) {
#pragma unroll
            for (int j = 0; j < CH; ++j) x[j] = bs[j] * P[j] * ks[j * LD + c];
        } else {
            const float* v = d.v + (size_t)t0 * d.ld_v + (size_t)head * d.V + c - K;
#pragma unroll
            for (int j = 0; j < CH; ++j) x[j] = j < n ? bs[j] * v[(size_t)j * d.ld_v] : 0.f;
        }
        // a finished x_i goes to all rows below at once: independent multiply-adds, where a row's own sum would be a chain
#pragma unroll
        for (int i = 0; i + 1 < CH; ++i) {
#pragma unroll
            for (int j = (i + 1) / 4 * 4; j < CH; j += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&A[i][j]);
                if (j > i) x[j] = fmaf(-a.x, x[i], x[j]);
                if (j + 1 > i) x[j + 1] = fmaf(-a.y, x[i], x[j + 1]);
                if (j + 2 > i) x[j + 2] = fmaf(-a.z, x[i], x[j + 2]);
                if (j + 3 > i) x[j + 3] = fmaf(-a.w, x[i], x[j + 3]);
            }
        }
        const size_t at = ((size_t)chunk * d.N + head) * CH;
        if (c < K) {
#pragma unroll
            for (int j = 0; j < CH; j += 4)                        // transposed, as the walk reads it: 32 tokens of a channel side by side
                *reinterpret_cast<float4*>(d.w + at * K + c * CH + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < CH; ++j) d.u[(at + j) * d.V + c - K] = x[j];
        }
    }
}

// Fixed decay: Z = sum_t g^(n-1-t) k_t v_t^T, 64 x 64 columns a CTA, a thread 8 x 4 of them.
__global__ void __launch_bounds__(kThreads)
chunk_update_kernel(const Chunks d) {
    __shared__ __align__(16) float ks[CH * LD], vs[CH * LD];
    forge::pdl_wait();
    int t0;
    const int chunk = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * VB, n = chunk_tokens(d, chunk, t0), tid = threadIdx.x;
    if (n <= 0) return;
    stage_rows(ks, d.k + (size_t)t0 * d.ld_k + head * K, d.ld_k, n);
    stage_rows(vs, d.v + (size_t)t0 * d.ld_v + (size_t)head * d.V + v0, d.ld_v, n);
    stages_commit();
    const float g = d.g[head];
    float acc[8][4];
#pragma unroll
    for (int a = 0; a < 8; ++a) acc[a][0] = acc[a][1] = acc[a][2] = acc[a][3] = 0.f;
    stages_wait<0>();
    __syncthreads();
    const int kr = tid / 16 * 4, c = tid % 16 * 4;            // rows kr .. kr+3 and 32 + kr ..
    float w = 1.f;
    for (int t = n - 1; t >= 0; --t, w *= g) {
        const float4 v = *reinterpret_cast<const float4*>(vs + t * LD + c);
        const float4 k0 = *reinterpret_cast<const float4*>(ks + t * LD + kr), k1 = *reinterpret_cast<const float4*>(ks + t * LD + 32 + kr);
        const float kk[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w}, vw[4] = {w * v.x, w * v.y, w * v.z, w * v.w};
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(kk[a], vw[b], acc[a][b]);
    }
    float* z = d.s + ((size_t)chunk * d.N + head) * K * d.V + v0 + c;
#pragma unroll
    for (int a = 0; a < 8; ++a)
        *reinterpret_cast<float4*>(z + (size_t)(kr + (a & 3) + (a >> 2) * 32) * d.V) = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
}

// ------------------------------------------------------------------------------------------------ 2: the walk
// DELTA: 16 columns of one head's S a CTA; the next chunk's W, K, U and decays are on their way while the present one is worked on.  A chunk is
// two small products, one after the other: u = U - W S (32 x 16 numbers over 64 channels, of which four warps take half and four the other half; those
// ask for the next chunk while the first finish u) and S <- P S + K^T u (64 x 16 over 32 tokens; a warp keeps its 16 x 8 numbers of S in registers).  As fp32 multiply-adds, 4 x 4 numbers a thread and the sums shared by the warps, shared memory was asked
// six times as often and a chunk had four meetings instead of three: three portions of 2,001 tokens in all, 32 heads, 104 us; 92 us so, and 74 us with the
// longest portion's CTAs first (what is left: the two products' splits and meetings, 32 times one after the other).
constexpr int kWalkThreads = 256, LDW = CH + 4, LDC = kColsB + 4;
constexpr int kStageB = K * LDW + CH * LD + CH * LDC + CH;    // floats of a chunk's W, K, U, decays
constexpr size_t kWalkSmem = sizeof(float) * (2 * kStageB + K * LDC + 2 * CH * LDC);

// The request that is the rank-th longest (of up to 32; of more they stay in their order): the kernel ends with the longest walk, whose CTAs come first
// and so each to an SM of its own.  Every lane gets it.
__device__ __forceinline__ int longest(const Chunks& d, int rank, int lane) {
    if (d.S > 32) return rank;
    const int n = lane < d.S ? d.q_start[lane + 1] - d.q_start[lane] : -1;
    int before = 0;
    for (int i = 0; i < d.S; ++i) {
        const int other = __shfl_sync(0xffffffffu, n, i);
        before += other > n || (other == n && i < lane);
    }
    return __ffs(__ballot_sync(0xffffffffu, lane < d.S && before == rank)) - 1;
}

// A CTA's whole walk once more, token by token with multiply-adds, where a sum of the tensor cores was not finite: from the inputs (u has taken U's place),
// the u of every token and the states before the chunks.  A thread has four rows of one column.  (A function of its own: its numbers would take registers
// from the loop that has none to spare.)
__device__ __noinline__ void walk_again(const Chunks& d, float* sm, int s, int head, int c0) {
    constexpr int kGroups = kWalkThreads / kColsB, kRows = K / kGroups;
    const int c = threadIdx.x % kColsB, rg = threadIdx.x / kColsB, t_lo = d.q_start[s], t_hi = d.q_start[s + 1];
    float* S_g = d.state + (size_t)d.slots[s] * d.stride + ((size_t)head * K + rg * kRows) * d.V + c0 + c;
    float S[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) S[i] = S_g[(size_t)i * d.V];
    for (int t = t_lo; t < t_hi; ++t) {
        const size_t at = (size_t)(first_chunk(d.q_start, s) + (t - t_lo) / CH) * d.N + head;
        const float* k = d.k + (size_t)t * d.ld_k + head / (d.N / d.M) * K + rg * kRows;
        const float g = d.g[(size_t)t * d.N + head];
        float part = 0.f;
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            if ((t - t_lo) % CH == 0) d.s[(at * K + rg * kRows + i) * d.V + c0 + c] = S[i];
            S[i] *= g;
            part = fmaf(S[i], k[i], part);
        }
        float* parts = sm + (t & 1) * kWalkThreads;           // (a meeting a token: the other half is still read by who is behind)
        parts[threadIdx.x] = part;
        __syncthreads();
        float sum = 0.f;
        for (int r = 0; r < kGroups; ++r) sum += parts[r * kColsB + c];
        const float u = d.beta[(size_t)t * d.N + head] * (d.v[(size_t)t * d.ld_v + (size_t)head * d.V + c0 + c] - sum);
#pragma unroll
        for (int i = 0; i < kRows; ++i) S[i] = fmaf(k[i], u, S[i]);
        if (rg == 0) d.u[(at * CH + (t - t_lo) % CH) * d.V + c0 + c] = u;
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) S_g[(size_t)i * d.V] = S[i];
}

__global__ void __launch_bounds__(kWalkThreads, 3)
chunk_walk_kernel(const __grid_constant__ Chunks d) {
    extern __shared__ __align__(16) float sm[];
    float* S = sm + 2 * kStageB;                              // [64][16 + 4]
    float* us = S + K * LDC;                                  // [32][16 + 4]: u_t times the decays behind it
    float* part = us + CH * LDC;                              // [32][16 + 4]: W S over the second half of the channels
    forge::pdl_launch_dependents();
    forge::pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, tq = lane & 3;
    const int cols = d.V / kColsB, head = blockIdx.x / cols % d.N, c0 = blockIdx.x % cols * kColsB, s = longest(d, blockIdx.x / (cols * d.N), lane);
    const int t_lo = d.q_start[s], t_hi = d.q_start[s + 1];
    if (t_lo >= t_hi) return;
    const int chunks = (t_hi - t_lo + CH - 1) / CH, at0 = first_chunk(d.q_start, s);
    const float* k = d.k + (size_t)head / (d.N / d.M) * K;
    constexpr int kFetch = kWalkThreads / 2;                  // threads that copy: the second half of the CTA
    auto fetch = [&](int i) {
        const int tid = (int)threadIdx.x - kFetch;
        if (i < chunks) {
            float* w = sm + (i & 1) * kStageB;
            const int t0 = t_lo + i * CH, n = min(CH, t_hi - t0);
            const size_t at = ((size_t)(at0 + i) * d.N + head) * CH;
#pragma unroll
            for (int h = 0; h < CH * K / 4; h += kFetch) {
                const int e = h + tid, r = e / (K / 4), c = e % (K / 4) * 4;
                stage16(w + e / (CH / 4) * LDW + e % (CH / 4) * 4, d.w + at * K + e * 4, true);                  // [channel][token]
                stage16(w + K * LDW + r * LD + c, k + (size_t)(r < n ? t0 + r : t0) * d.ld_k + c, r < n);        // [token][channel]
            }
            float* u = w + K * LDW + CH * LD;
            stage16(u + tid / 4 * LDC + tid % 4 * 4, d.u + (at + tid / 4) * d.V + c0 + tid % 4 * 4, true);
            if (tid < CH) {
                const int t = tid;
                float* dst = u + CH * LDC + t;
                if (t < n) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(d.g + (size_t)(t0 + t) * d.N + head) : "memory");
                else *dst = 1.0f;
            }
        }
        stages_commit();
    };
    static_assert(kFetch == CH * kColsB / 4, "a piece of U a thread");
    if (warp >= 4) fetch(0);
    // a warp's part of S: rows row0 + gr (and 8 further on), columns col0 + 2 tq and the next
    const int row0 = (warp >> 1) * 16 + gr, col0 = (warp & 1) * 8 + 2 * tq;
    float* S_g = d.state + (size_t)d.slots[s] * d.stride + (size_t)head * K * d.V + (size_t)row0 * d.V + c0 + col0;
    float2 own0 = *reinterpret_cast<const float2*>(S_g), own1 = *reinterpret_cast<const float2*>(S_g + 8 * d.V);
    *reinterpret_cast<float2*>(S + row0 * LDC + col0) = own0;
    *reinterpret_cast<float2*>(S + (row0 + 8) * LDC + col0) = own1;
    float odd = 0.f;                                          // NaN once a sum of a second product (and so of a first one) is not finite
    for (int i = 0; i < chunks; ++i) {
        stages_wait<0>();
        __syncthreads();                                      // chunk i is here, S stands, and nobody is at chunk i - 1 any more
        const float* w = sm + (i & 1) * kStageB;
        const float* ks = w + K * LDW;
        const float* U = ks + CH * LD;
        const int m0 = (warp & 1) * 16 + gr, n0 = (warp >> 1 & 1) * 8, c = n0 + 2 * tq;
        float main[4] = {0.f, 0.f, 0.f, 0.f}, rest[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < K / 2; kk += 16) {
            const int from = (warp >> 2) * (K / 2) + kk + 2 * tq;
            const float* a = w + from * LDW + m0;
            const float* b = S + from * LDC + n0 + gr;
            const Terms at[4] = {split2(a[0], a[LDW]), split2(a[8], a[LDW + 8]), split2(a[8 * LDW], a[9 * LDW]), split2(a[8 * LDW + 8], a[9 * LDW + 8])};
            const Terms bt[2] = {split2(b[0], b[LDC]), split2(b[8 * LDC], b[9 * LDC])};
            mma_terms(main, rest, at, bt);
        }
        // the decays behind token `lane`, and the chunk's (lane 0's)
        float x = U[CH * LDC + lane];                         // becomes g_lane .. g_31
#pragma unroll
        for (int o = 1; o < CH; o <<= 1) {
            const float y = __shfl_down_sync(0xffffffffu, x, o);
            if (lane + o < CH) x *= y;
        }
        const float p = __shfl_sync(0xffffffffu, x, 0), next = __shfl_down_sync(0xffffffffu, x, 1), behind = lane + 1 < CH ? next : 1.0f;
        if (warp >= 4) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(part + (m0 + 8 * h) * LDC + c) =
                    make_float2(main[2 * h] + (rest[0][2 * h] + rest[1][2 * h]), main[2 * h + 1] + (rest[0][2 * h + 1] + rest[1][2 * h + 1]));
        }
        __syncthreads();
        if (warp < 4) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = m0 + 8 * h;
                float2 u = *reinterpret_cast<const float2*>(U + t * LDC + c);
                const float2 half = *reinterpret_cast<const float2*>(part + t * LDC + c);
                u.x -= (main[2 * h] + (rest[0][2 * h] + rest[1][2 * h])) + half.x;
                u.y -= (main[2 * h + 1] + (rest[0][2 * h + 1] + rest[1][2 * h + 1])) + half.y;
                const float r = __shfl_sync(0xffffffffu, behind, t);
                *reinterpret_cast<float2*>(us + t * LDC + c) = make_float2(u.x * r, u.y * r);
                *reinterpret_cast<float2*>(d.u + (((size_t)(at0 + i) * d.N + head) * CH + t) * d.V + c0 + c) = u;
            }
        } else {
            fetch(i + 1);
        }
        float* kept = d.s + (((size_t)(at0 + i) * d.N + head) * K + row0) * d.V + c0 + col0;
        *reinterpret_cast<float2*>(kept) = own0;
        *reinterpret_cast<float2*>(kept + 8 * d.V) = own1;
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; ++e) main[e] = rest[0][e] = rest[1][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < CH; kk += 16) {
            const float* a = ks + (kk + 2 * tq) * LD + row0;
            const float* b = us + (kk + 2 * tq) * LDC + (warp & 1) * 8 + gr;
            const Terms at[4] = {split2(a[0], a[LD]), split2(a[8], a[LD + 8]), split2(a[8 * LD], a[9 * LD]), split2(a[8 * LD + 8], a[9 * LD + 8])};
            const Terms bt[2] = {split2(b[0], b[LDC]), split2(b[8 * LDC], b[9 * LDC])};
            mma_terms(main, rest, at, bt);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) main[e] += rest[0][e] + rest[1][e];
        odd += odd4(main);
        own0.x = fmaf(p, own0.x, main[0]); own0.y = fmaf(p, own0.y, main[1]);
        own1.x = fmaf(p, own1.x, main[2]); own1.y = fmaf(p, own1.y, main[3]);
        *reinterpret_cast<float2*>(S + row0 * LDC + col0) = own0;
        *reinterpret_cast<float2*>(S + (row0 + 8) * LDC + col0) = own1;
    }
    if (__syncthreads_or(odd != 0.f)) {
        walk_again(d, sm, s, head, c0);
        return;
    }
    *reinterpret_cast<float2*>(S_g) = own0;
    *reinterpret_cast<float2*>(S_g + 8 * d.V) = own1;
}

// Fixed decay: four neighbouring numbers of the state a thread; where Z of a chunk lay the state before it stays.
__global__ void __launch_bounds__(kThreads)
chunk_sum_kernel(const Chunks d) {
    forge::pdl_launch_dependents();
    forge::pdl_wait();
    const int s = blockIdx.x, head = blockIdx.y, e = (blockIdx.z * kThreads + threadIdx.x) * 4;
    const int t_lo = d.q_start[s], t_hi = d.q_start[s + 1], size = K * d.V;
    if (t_lo >= t_hi || e >= size) return;
    const int chunks = (t_hi - t_lo + CH - 1) / CH, last = t_hi - t_lo - (chunks - 1) * CH;
    const float g = d.g[head];
    float p = 1.f, p_last = 1.f;
    for (int i = 0; i < CH; ++i) {
        p *= g;
        if (i < last) p_last = p;
    }
    float* S_g = d.state + (size_t)d.slots[s] * d.stride + (size_t)head * size + e;
    float* z = d.s + ((size_t)first_chunk(d.q_start, s) * d.N + head) * size + e;
    const size_t step = (size_t)d.N * size;
    float4 x = *reinterpret_cast<const float4*>(S_g);
    constexpr int kAhead = 8;                                 // chunks whose Z is asked for before the first is used
    for (int i0 = 0; i0 < chunks; i0 += kAhead) {
        float4 y[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (i0 + i < chunks) y[i] = *reinterpret_cast<const float4*>(z + (size_t)(i0 + i) * step);
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (i0 + i < chunks) {
                *reinterpret_cast<float4*>(z + (size_t)(i0 + i) * step) = x;
                const float f = i0 + i + 1 < chunks ? p : p_last;
                x = make_float4(fmaf(f, x.x, y[i].x), fmaf(f, x.y, y[i].y), fmaf(f, x.z, y[i].z), fmaf(f, x.w, y[i].w));
            }
    }
    *reinterpret_cast<float4*>(S_g) = x;
}

// ------------------------------------------------------------------------------------------------ 3: the outputs
// A CTA has 64 of a head's value columns and makes three products on the tensor cores (terms as in the walk): q k^T (32 x 32, under the triangle of decays),
// q S (32 x 64 over 64 channels) and the triangle times u (over 32 tokens).  As fp32 multiply-adds, eight tokens x four columns a thread, shared memory was
// asked for 12 bytes a product: 2,001 tokens of 32 heads 44.5 us, 37.7 us so (q, k, u, S in and the outputs out: 10 us at full bandwidth; the rest is
// splits and a CTA's two waits).
constexpr int kOutThreads = 128, LDV = VB + 4, LDM = CH + 4;
constexpr size_t kOutSmem = sizeof(float) * (2 * CH * LD + K * LDV + CH * LDV + CH * LDM);

template <bool DELTA>
__global__ void __launch_bounds__(kOutThreads, 4)
chunk_output_kernel(const Chunks d) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float R[CH][CH + 1], gs[CH], P[CH];
    float* qs = sm;                                           // [32][64 + 4]
    float* ks = qs + CH * LD;                                 // [32][64 + 4]
    float* S = ks + CH * LD;                                  // [64][64 + 4]: the state before the chunk
    float* us = S + K * LDV;                                  // [32][64 + 4]
    float* Mx = us + CH * LDV;                                // [32][32 + 4]: the triangle
    forge::pdl_launch_dependents();
    forge::pdl_wait();
    int t0;
    const int chunk = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * VB, n = chunk_tokens(d, chunk, t0), tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, gr = lane >> 2, tq = lane & 3;
    if (n <= 0) return;
    const int hk = head / (d.N / d.M);
    stage_rows<kOutThreads>(qs, d.q + (size_t)t0 * d.ld_q + hk * K, d.ld_q, n);
    stage_rows<kOutThreads>(ks, d.k + (size_t)t0 * d.ld_k + hk * K, d.ld_k, n);
    stages_commit();
    const float* u = DELTA ? d.u + ((size_t)chunk * d.N + head) * CH * d.V + v0 : d.v + (size_t)t0 * d.ld_v + (size_t)head * d.V + v0;
    const int ld_u = DELTA ? d.V : d.ld_v;
    const float* kept = d.s + ((size_t)chunk * d.N + head) * K * d.V + v0;
    for (int i = tid; i < K * VB / 4; i += kOutThreads) stage16(S + i / (VB / 4) * LDV + i % (VB / 4) * 4, kept + (size_t)(i / (VB / 4)) * d.V + i % (VB / 4) * 4, true);
    for (int i = tid; i < CH * VB / 4; i += kOutThreads) {
        const int r = i / (VB / 4), c = i % (VB / 4) * 4;
        stage16(us + r * LDV + c, r < n ? u + (size_t)r * ld_u + c : u, r < n);
    }
    stages_commit();
    if (tid < CH) gs[tid] = tid >= n ? 1.0f : DELTA ? d.g[(size_t)(t0 + tid) * d.N + head] : d.g[head];
    __syncthreads();
    decay_triangle(R, gs);
    if (tid == CH) {
        float p = 1.f;
        for (int i = 0; i < CH; ++i) P[i] = p *= gs[i];
    }
    stages_wait<1>();
    __syncthreads();
    {
        // rows m0 .. m0 + 15 of the triangle, columns n0 .. n0 + 15 (above the diagonal: zeros, whatever the keys there)
        const int m0 = (warp & 1) * 16, n0 = (warp >> 1) * 16;
        float main[2][4] = {};
        if (n0 <= m0) square16(main, qs + m0 * LD, ks + n0 * LD, gr, tq);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int j = m0 + gr + (e >> 1) * 8, i = n0 + 8 * h + 2 * tq + (e & 1);
                Mx[j * LDM + i] = i <= j ? R[j][i] * main[h][e] : 0.f;
            }
    }
    stages_wait<0>();
    __syncthreads();
    // a warp's 16 columns of all tokens: 16 x 8 tiles [m][h]
    const int c0 = warp * 16;
    float main[2][2][4] = {}, rest[2][2][4] = {}, o[2][2][4];
#pragma unroll
    for (int kk = 0; kk < K; kk += 16) {
        Terms bt[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* b = S + (kk + 2 * tq) * LDV + c0 + 8 * h + gr;
            bt[h][0] = split2(b[0], b[LDV]);
            bt[h][1] = split2(b[8 * LDV], b[9 * LDV]);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const float* a = qs + (16 * m + gr) * LD + kk + 2 * tq;
            auto pair = [](const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return split2(v.x, v.y); };
            const Terms at[4] = {pair(a), pair(a + 8 * LD), pair(a + 8), pair(a + 8 * LD + 8)};
#pragma unroll
            for (int h = 0; h < 2; ++h) mma_terms(main[m][h], rest[m][h], at, bt[h]);
        }
    }
    float odd = 0.f;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[m][h][e] = main[m][h][e] + rest[m][h][e];
                main[m][h][e] = rest[m][h][e] = 0.f;
            }
            odd += odd4(o[m][h]);
        }
    if (odd != 0.f) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float& x = o[i >> 3][i >> 2 & 1][i & 3];
            x = made_again(x, qs + (16 * (i >> 3) + gr + (i >> 1 & 1) * 8) * LD, 1, S + c0 + 8 * (i >> 2 & 1) + 2 * tq + (i & 1), LDV, K);
        }
    }
    __syncwarp();                                             // (the lanes may have parted over a sum that was made again)
#pragma unroll
    for (int kk = 0; kk < CH; kk += 16) {
        Terms bt[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* b = us + (kk + 2 * tq) * LDV + c0 + 8 * h + gr;
            bt[h][0] = split2(b[0], b[LDV]);
            bt[h][1] = split2(b[8 * LDV], b[9 * LDV]);
        }
#pragma unroll
        for (int m = kk / 16; m < 2; ++m) {                               // (the first 16 tokens see none of the others)
            const float* a = Mx + (16 * m + gr) * LDM + kk + 2 * tq;
            auto pair = [](const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return split2(v.x, v.y); };
            const Terms at[4] = {pair(a), pair(a + 8 * LDM), pair(a + 8), pair(a + 8 * LDM + 8)};
#pragma unroll
            for (int h = 0; h < 2; ++h) mma_terms(main[m][h], rest[m][h], at, bt[h]);
        }
    }
    odd = 0.f;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int e = 0; e < 4; ++e) main[m][h][e] += rest[m][h][e];
            odd += odd4(main[m][h]);
        }
    if (odd != 0.f) {                                         // (a later token's number that is none has met the triangle's zeros: only up to the own token now)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int j = 16 * (i >> 3) + gr + (i >> 1 & 1) * 8;
            float& x = main[i >> 3][i >> 2 & 1][i & 3];
            x = made_again(x, Mx + j * LDM, 1, us + c0 + 8 * (i >> 2 & 1) + 2 * tq + (i & 1), LDV, j + 1);
        }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int j = 16 * m + gr + 8 * r;
            if (j >= n) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(d.out + (size_t)(t0 + j) * d.N * d.V + (size_t)head * d.V + v0 + c0 + 8 * h + 2 * tq) =
                    make_float2(__fmul_rn(o[m][h][2 * r], P[j]) + main[m][h][2 * r], __fmul_rn(o[m][h][2 * r + 1], P[j]) + main[m][h][2 * r + 1]);
        }
}

template <bool DELTA>
cudaError_t launch_output(const Chunks& d, unsigned chunks, cudaStream_t stream) {
    static forge::PerDeviceFlag flag;
    bool& done = flag.current();
    if (!done) {
        const cudaError_t e = cudaFuncSetAttribute(chunk_output_kernel<DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOutSmem);
        if (e != cudaSuccess) return e;
        done = true;
    }
    return forge::launch(chunk_output_kernel<DELTA>, dim3(chunks, d.N, d.V / VB), dim3(kOutThreads), kOutSmem, stream, 1, d);
}

bool aligned(const float* p, long long ld) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0; }

int check(const char* what, const Chunks& d, int T, int Kc) {
    if (T < 0 || d.S < 0 || d.N <= 0 || d.M <= 0 || d.N % d.M != 0 || d.V <= 0) return forge::fail(FORGE_ERR_ARG, "%s: bad sizes S=%d N=%d M=%d V=%d", what, d.S, d.N, d.M, d.V);
    if (Kc != K || d.V % VB != 0 || d.V > 65535 * kColsB || d.N > 65535) return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: heads of %d and %d channels", what, Kc, d.V);
    if (d.stride < (long long)d.N * K * d.V) return forge::fail(FORGE_ERR_ARG, "%s: state rows are too short", what);
    if (!aligned(d.q, d.ld_q) || !aligned(d.k, d.ld_k) || !aligned(d.v, d.ld_v) || !aligned(d.state, d.stride) || !aligned(d.out, 4) || !aligned(d.s, 4))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: rows that are not aligned to 16 bytes", what);
    return FORGE_OK;
}

}  // namespace

// 1 if the kernels take heads of these sizes (rows must be aligned to 16 bytes).
extern "C" int forge_chunk_scan_supports(int key_channels, int value_channels) { return key_channels == K && value_channels % VB == 0 ? 1 : 0; }

// The gated delta rule as forge_gated_delta_scan defines it; w, u, s fp32 scratch of C * N * 32 * 64, C * N * 32 * V and C * N * 64 * V
// numbers, C = T / 32 + S.
extern "C" int forge_gated_delta_chunks(const float* q, int ld_q, const float* k, int ld_k, const float* v, int ld_v, const float* g, const float* beta,
                                        float* w, float* u, float* s, float* state, long long state_stride, const int32_t* q_start, const int32_t* slots,
                                        float* out, int T, int S, int N, int M, int Kc, int V, cudaStream_t stream) {
    const Chunks d{q, k, v, ld_q, ld_k, ld_v, g, beta, w, u, s, state, state_stride, q_start, slots, out, S, N, M, V};
    const int rc = check("gated_delta_chunks", d, T, Kc);
    if (rc != FORGE_OK || S == 0 || T == 0) return rc;
    if (!aligned(w, 4) || !aligned(u, 4)) return forge::fail(FORGE_ERR_ARG, "gated_delta_chunks: scratch that is not aligned");
    static forge::PerDeviceFlag flag;
    bool& done = flag.current();
    if (!done) {
        const cudaError_t e = cudaFuncSetAttribute(chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWalkSmem);
        if (e != cudaSuccess) return forge::check_launch("gated_delta_chunks (shared memory)", e);
        done = true;
    }
    const unsigned chunks = T / CH + S;
    cudaError_t e = forge::launch(chunk_solve_kernel, dim3(chunks, N), dim3(kThreads), 0, stream, 1, d);
    if (e == cudaSuccess) e = forge::launch(chunk_walk_kernel, dim3((unsigned)S * N * (V / kColsB)), dim3(kWalkThreads), kWalkSmem, stream, 1, d);
    if (e == cudaSuccess) e = launch_output<true>(d, chunks, stream);
    return forge::check_launch("gated_delta_chunks", e);
}

// S <- decay[n] S + k v^T, out = S^T q per head over the step's tokens (q and k of every head); s as above.
extern "C" int forge_decay_chunks(const float* q, int ld_q, const float* k, int ld_k, const float* v, int ld_v, const float* decay, float* s, float* state,
                                  long long state_stride, const int32_t* q_start, const int32_t* slots, float* out, int T, int S, int N, int Kc, int V,
                                  cudaStream_t stream) {
    const Chunks d{q, k, v, ld_q, ld_k, ld_v, decay, nullptr, nullptr, nullptr, s, state, state_stride, q_start, slots, out, S, N, N, V};
    const int rc = check("decay_chunks", d, T, Kc);
    if (rc != FORGE_OK || S == 0 || T == 0) return rc;
    const unsigned chunks = T / CH + S;
    cudaError_t e = forge::launch(chunk_update_kernel, dim3(chunks, N, V / VB), dim3(kThreads), 0, stream, 1, d);
    if (e == cudaSuccess) e = forge::launch(chunk_sum_kernel, dim3(S, N, (K * V / 4 + kThreads - 1) / kThreads), dim3(kThreads), 0, stream, 1, d);
    if (e == cudaSuccess) e = launch_output<false>(d, chunks, stream);
    return forge::check_launch("decay_chunks", e);
}
