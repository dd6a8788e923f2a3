// C[M,N] (fp32) = A[M,K] . W[N,K]^T (+ bias[N]) (+ C), by fp32 FMA on the CUDA cores.
//
// This is the engine's true 32-bit matrix product: operands are widened to fp32 when they are read, every product and
// sum is an fp32 FMA, and no tensor-core mode (TF32/BF16) is involved.  It stands in for the reference's
// gemm_tiled_kernel / gemv_transB_kernel / cuBLAS SGEMM trio (src/operators/cuda/cuda_gemm.cu:7-55, cuda_gemv.cu:9-40,
// cuda_quant.cu:582-599).  Any M, N, K >= 1 is accepted (edges are zero-filled in shared memory).
//
// The order of an element's sum is fixed by K alone, so a token's row does not depend on the batch around it although two
// kernels share the work: chunks of 128 channels are FMA chains from zero in the channels' order, eight chunks in order make
// a section (1,024 channels), and the sections are added in order; then the bias, then the old C.  A section is what may be
// given to another CTA of a thread-block cluster (its sums meet through distributed shared memory).
#include <algorithm>
#include "common.cuh"

namespace {

typedef unsigned long long u64;
constexpr int kChunk = 128, kSection = 1024;
constexpr int kMaxCluster = 8;

// two fp32 FMAs (or sums) in one instruction, each rounded as fmaf (or +) rounds
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 pack2(float lo, float hi) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpack2(u64 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
// 16 or 4 bytes into shared memory without a stop in registers; ok == false: zeros
__device__ __forceinline__ void copy16(void* dst, const void* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(void* dst, const void* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the number at the same place of another CTA's shared memory
__device__ __forceinline__ float peer_load(const float* p, int rank) {
    uint32_t remote;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

// ------------------------------------------------------------------------------------------------ few rows of A
// Up to 32 rows of A: the product is as long as W takes to arrive.  A CTA has 32 rows of W and one section at a time, a warp
// one chunk of it: 32 rows x 128 channels come in stages of 32 channels (cp.async; 4 KB a warp are on their way while a stage is worked
// on, sixteen warps an SM up to 16 rows of A), lane n then walks row n's channels in order against all rows of A, which lie
// [channel][row] beside it so that one broadcast load brings four of them.  Sections go to the CTAs of a cluster in turn.
// Four layers of the TinyLlama shape and its head for two tokens (17 products, 0.97 GB of weights): 0.30 ms, 3.3 TB/s; as tiles of
// 64 x 64, which this replaces, 9.5 ms.
constexpr int kRowsW = 32, kKS = 32, kWStride = kKS + 4, kFewWarps = kSection / kChunk, kFewThreads = 32 * kFewWarps;

template <int MT> struct FewSmem {
    static constexpr int kStages = MT == 1 ? 3 : 2;                               // what fits two CTAs an SM (32 rows of A: one)
    static constexpr int kStage = kRowsW * kWStride + kKS * MT;                   // floats of a warp's stage
    static constexpr int kWarp = kStages * kStage;
    static constexpr int floats(int slots) { return kFewWarps * kWarp + slots * MT * kRowsW; }
    // row m of A at channel k: groups of four rows change places with the channel, so that a warp's 32 channels of one row do not all
    // meet in the same bank when they are written
    static __device__ __forceinline__ int x_at(int k, int m) { return MT < 8 ? k * MT + m : k * MT + ((((m >> 2) ^ ((k * MT / 32) & (MT / 4 - 1))) << 2) | (m & 3)); }
};

template <int MT, typename T>
__global__ void __launch_bounds__(kFewThreads, MT >= 32 ? 1 : 2)
gemm_simt_few_kernel(const T* __restrict__ A, const T* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K,
                     int accumulate, int cluster, int vec, int w_at_rest) {
    using L = FewSmem<MT>;
    extern __shared__ __align__(16) float sm[];
    float* slots = sm + kFewWarps * L::kWarp;                                     // [sections of this CTA][MT][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x / cluster, rank = blockIdx.x % cluster, n0 = tile * kRowsW;
    const int sections = (K + kSection - 1) / kSection;
    float* mine = sm + warp * L::kWarp;
    forge::pdl_launch_dependents();

    auto fetch_w = [&](int buf, int k0) {
        float* ws = mine + buf * L::kStage;
        if (sizeof(T) == 4 && vec) {
#pragma unroll
            for (int i = 0; i < kRowsW * kKS / 4 / 32; ++i) {
                const int r = i * 4 + (lane >> 3), c = (lane & 7) * 4;
                const bool ok = n0 + r < N && k0 + c < K;                         // (K is a multiple of 4)
                copy16(ws + r * kWStride + c, ok ? W + (size_t)(n0 + r) * K + k0 + c : W, ok);
            }
        } else {
            for (int r = 0; r < kRowsW; ++r) {
                const bool ok = n0 + r < N && k0 + lane < K;
                const T* src = ok ? W + (size_t)(n0 + r) * K + k0 + lane : W;
                if (sizeof(T) == 4) copy4(ws + r * kWStride + lane, src, ok);
                else ws[r * kWStride + lane] = ok ? forge::to_float(*src) : 0.f;
            }
        }
    };
    auto fetch_x = [&](int buf, int k0) {
        float* xs = mine + buf * L::kStage + kRowsW * kWStride;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const bool ok = m < M && k0 + lane < K;
            const T* src = ok ? A + (size_t)m * K + k0 + lane : A;
            if (sizeof(T) == 4) copy4(xs + L::x_at(lane, m), src, ok);
            else xs[L::x_at(lane, m)] = ok ? forge::to_float(*src) : 0.f;
        }
    };
    constexpr int kStages = L::kStages;
    bool waited = false;
    int slot = 0;
    for (int s = rank; s < sections; s += cluster, ++slot) {
        const int k0 = s * kSection + warp * kChunk;                              // this warp's chunk (may lie behind the end)
        const int n_stages = min(kChunk, max(0, K - k0) + kKS - 1) / kKS;
        constexpr int kPairs = (MT + 1) / 2;
        u64 acc2[kPairs];
        float acc1 = 0.f;
#pragma unroll
        for (int m = 0; m < kPairs; ++m) acc2[m] = 0;
        // weights at rest do not wait for the kernel before this one; the rows of A do, and a W that an earlier kernel may still be writing
        if (!waited && !w_at_rest) {
            forge::pdl_wait();
            waited = true;
        }
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i)
            if (i < n_stages) fetch_w(i, k0 + i * kKS);
        if (!waited) {
            forge::pdl_wait();
            waited = true;
        }
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i) {
            if (i < n_stages) fetch_x(i, k0 + i * kKS);
            copies_commit();
        }
        for (int st = 0; st < n_stages; ++st) {
            const int buf = st % kStages;
            copies_wait<kStages - 2>();
            __syncwarp();                                                         // the stage has landed for every lane, and the one before is done with
            if (st + kStages - 1 < n_stages) {
                const int to = (st + kStages - 1) % kStages;
                fetch_w(to, k0 + (st + kStages - 1) * kKS);
                fetch_x(to, k0 + (st + kStages - 1) * kKS);
            }
            copies_commit();
            const float* wr = mine + buf * L::kStage + lane * kWStride;
            const float* xs = mine + buf * L::kStage + kRowsW * kWStride;
#pragma unroll 1
            for (int c0 = 0; c0 < kKS; c0 += 8, wr += 8, xs += 8 * MT) {          // (rows of A change places with a period of at most eight channels)
#pragma unroll
                for (int c = 0; c < 8; c += 4) {
                    const float4 w4 = *reinterpret_cast<const float4*>(wr + c);
                    const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (MT == 1) {
                            acc1 = fmaf(xs[c + e], wv[e], acc1);
                        } else if (MT == 2) {
                            acc2[0] = fma2(*reinterpret_cast<const u64*>(xs + (c + e) * MT), pack2(wv[e], wv[e]), acc2[0]);
                        } else {
                            const u64 ww = pack2(wv[e], wv[e]);
#pragma unroll
                            for (int m = 0; m < MT; m += 4) {
                                const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(xs + L::x_at(c + e, m));
                                acc2[m / 2] = fma2(xv.x, ww, acc2[m / 2]);
                                acc2[(m / 2 + 1) % kPairs] = fma2(xv.y, ww, acc2[(m / 2 + 1) % kPairs]);
                            }
                        }
                    }
                }
            }
        }
        copies_wait<0>();
        __syncthreads();                                                          // every warp's stages are done with: the chunks' sums take their place
        float* part = sm + warp * (MT * kRowsW);
        if (MT == 1) {
            part[lane] = acc1;
        } else {
#pragma unroll
            for (int m = 0; m < MT; m += 2) {
                const float2 v = unpack2(acc2[m / 2]);
                part[m * kRowsW + lane] = v.x;
                part[(m + 1) * kRowsW + lane] = v.y;
            }
        }
        __syncthreads();
        const int chunks = min(kFewWarps, (K - s * kSection + kChunk - 1) / kChunk);
        for (int i = threadIdx.x; i < MT * kRowsW; i += kFewThreads) {
            float v = sm[i];
            for (int c = 1; c < chunks; ++c) v += sm[c * (MT * kRowsW) + i];
            slots[slot * (MT * kRowsW) + i] = v;
        }
        __syncthreads();
    }
    if (!waited) forge::pdl_wait();
    if (cluster > 1) cluster_sync();
    // the sections' sums, in order; each CTA of the cluster finishes its share of the tile
    for (int i = rank * kFewThreads + threadIdx.x; i < MT * kRowsW; i += cluster * kFewThreads) {
        const int m = i / kRowsW, n = n0 + i % kRowsW;
        if (m >= M || n >= N) continue;
        float v = 0.f;
        for (int s = 0; s < sections; ++s) {
            const float* p = slots + (s / cluster) * (MT * kRowsW) + i;
            const float part = cluster > 1 ? peer_load(p, s % cluster) : *p;
            v = s == 0 ? part : v + part;
        }
        if (bias) v += bias[n];
        float* c = C + (size_t)m * N + n;
        *c = accumulate ? (*c + v) : v;
    }
    if (cluster > 1) cluster_sync();                                              // nobody leaves while its sums are being read
}

// ------------------------------------------------------------------------------------------------ many rows of A
// More rows: tiles of BM x 64, a thread BM/16 x 4 elements (pairs of rows of A in one instruction), 16 channels a step through two
// buffers in shared memory (both operands lie [channel][row]), the next step's numbers held in registers meanwhile.  Bound by shared
// memory (three 16-byte loads a thread for 32 products).  Chunk sums are parked in shared memory.  Which tile height and how many CTAs share a
// tile's sections is chosen on the host (see run).
// The 16 products of a 333-token prompt through those layers (117 GFLOP): 4.0 ms, 29 TFLOP/s, of 74 that the FMA pipe has
// (an eighth of which 333 rows lose in tiles of 128).
constexpr int BN = 64, BK = 16, kTileThreads = 256;

template <int BM> struct TileSmem {
    static constexpr int kAStride = BM + 4, kWStride = BN + 4;
    static constexpr int kBuf = BK * (kAStride + kWStride);
    static constexpr int kSlot = BM * BN;                                         // floats of a parked section
    static constexpr int floats(int slots) { return 2 * kBuf + slots * kSlot; }
};

template <typename T> struct Four;
template <> struct Four<float> {
    static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
};
template <> struct Four<__nv_bfloat16> {
    static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
};

template <int BM, typename T>
__global__ void __launch_bounds__(kTileThreads, 2)
gemm_simt_tile_kernel(const T* __restrict__ A, const T* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K,
                      int accumulate, int cluster, int vec) {
    using L = TileSmem<BM>;
    constexpr int TM = BM / 16, TN = 4, AV = BM * BK / 4 / kTileThreads;          // a thread's rows and columns; its 4-channel pieces of A a step
    static_assert(AV >= 1 && BN * BK / 4 == kTileThreads, "one piece of W a thread and step");
    extern __shared__ __align__(16) float sm[];
    float* slots = sm + 2 * L::kBuf;
    forge::pdl_launch_dependents();
    forge::pdl_wait();
    const int tid = threadIdx.x, tile = blockIdx.x / cluster, rank = blockIdx.x % cluster;
    const int n_tiles = (N + BN - 1) / BN, m0 = (tile / n_tiles) * BM, n0 = (tile % n_tiles) * BN;
    const int sections = (K + kSection - 1) / kSection;
    // a warp's 32 threads are 4 x 8: rows ty*4 .. (and BM/2 further on), columns tx*4 ..
    const int warp = tid >> 5, lane = tid & 31, ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);

    float4 ra[AV], rw;
    auto read4 = [&](const T* base, int row, int rows, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= rows) return v;
        const T* p = base + (size_t)row * K + k;
        if (vec) {
            if (k < K) v = Four<T>::load(p);                                      // (K is a multiple of 4)
        } else {
            if (k < K) v.x = forge::to_float(p[0]);
            if (k + 1 < K) v.y = forge::to_float(p[1]);
            if (k + 2 < K) v.z = forge::to_float(p[2]);
            if (k + 3 < K) v.w = forge::to_float(p[3]);
        }
        return v;
    };
    auto read_step = [&](int k0) {
#pragma unroll
        for (int i = 0; i < AV; ++i) ra[i] = read4(A, m0 + (tid >> 2) + i * (kTileThreads / 4), M, k0 + (tid & 3) * 4);
        rw = read4(W, n0 + (tid >> 2), N, k0 + (tid & 3) * 4);
    };
    auto put_step = [&](int buf) {
        float* as = sm + buf * L::kBuf + (tid & 3) * 4 * L::kAStride + (tid >> 2);
        float* ws = sm + buf * L::kBuf + BK * L::kAStride + (tid & 3) * 4 * L::kWStride + (tid >> 2);
#pragma unroll
        for (int i = 0; i < AV; ++i) {
            float* a = as + i * (kTileThreads / 4);
            a[0] = ra[i].x; a[L::kAStride] = ra[i].y; a[2 * L::kAStride] = ra[i].z; a[3 * L::kAStride] = ra[i].w;
        }
        ws[0] = rw.x; ws[L::kWStride] = rw.y; ws[2 * L::kWStride] = rw.z; ws[3 * L::kWStride] = rw.w;
    };

    // element pair (j, i) of a thread lies at [(j * TM/2 + i)][thread] of a slot.  A CTA of a cluster keeps its sections apart; alone it
    // sums a section up in the second slot and adds it to the first.
    u64 acc[TN][TM / 2];
    int slot = 0;
    for (int s = rank; s < sections; s += cluster, ++slot) {
        const int k_lo = s * kSection, k_hi = min(K, k_lo + kSection), steps = (k_hi - k_lo + BK - 1) / BK;
        u64* park = reinterpret_cast<u64*>(slots + (size_t)min(slot, 1) * L::kSlot) + tid;
        read_step(k_lo);
        put_step(0);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
            for (int i = 0; i < TM / 2; ++i) acc[j][i] = 0;
        for (int st = 0; st < steps; ++st) {
            const int buf = st & 1;
            if (st + 1 < steps) read_step(k_lo + (st + 1) * BK);
            const float* as = sm + buf * L::kBuf + ty * 4;
            const float* ws = sm + buf * L::kBuf + BK * L::kAStride + tx * 4;
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                u64 a2[TM / 2];
#pragma unroll
                for (int i = 0; i < TM / 4; ++i) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(as + k * L::kAStride + i * (BM / 2));
                    a2[2 * i] = v.x;
                    a2[2 * i + 1] = v.y;
                }
                const float4 w4 = *reinterpret_cast<const float4*>(ws + k * L::kWStride);
                const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const u64 ww = pack2(wv[j], wv[j]);
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i) acc[j][i] = fma2(a2[i], ww, acc[j][i]);
                }
            }
            if ((st + 1) % (kChunk / BK) == 0 || st + 1 == steps) {               // a chunk is complete
                const bool first = st < kChunk / BK;
#pragma unroll
                for (int j = 0; j < TN; ++j)
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i) {
                        u64* p = park + (j * (TM / 2) + i) * kTileThreads;
                        *p = first ? acc[j][i] : add2(*p, acc[j][i]);
                        acc[j][i] = 0;
                    }
            }
            if (st + 1 < steps) put_step(buf ^ 1);
            __syncthreads();
        }
        if (cluster == 1 && slot > 0) {
            u64* total = reinterpret_cast<u64*>(slots) + tid;
#pragma unroll
            for (int e = 0; e < TN * (TM / 2); ++e) total[e * kTileThreads] = add2(total[e * kTileThreads], park[e * kTileThreads]);
        }
    }
    if (cluster > 1) cluster_sync();
    // pair e of the tile's elements per thread: every CTA of the cluster finishes its share of the pairs
    for (int e = rank; e < TN * (TM / 2); e += cluster) {
        const int j = e / (TM / 2), i = e % (TM / 2);
        const float* p = slots + ((size_t)e * kTileThreads + tid) * 2;
        float2 v;
        if (cluster == 1) {
            v = *reinterpret_cast<const float2*>(p);
        } else {
            for (int s = 0; s < sections; ++s) {
                const float* q = p + (size_t)(s / cluster) * L::kSlot;
                const float x = peer_load(q, s % cluster), y = peer_load(q + 1, s % cluster);
                v.x = s == 0 ? x : v.x + x;
                v.y = s == 0 ? y : v.y + y;
            }
        }
        const int n = n0 + tx * 4 + j, m = m0 + (i >> 1) * (BM / 2) + ty * 4 + (i & 1) * 2;
        if (n >= N) continue;
        const float b = bias ? bias[n] : 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (m + h >= M) continue;
            float x = h ? v.y : v.x;
            if (bias) x += b;
            float* c = C + (size_t)(m + h) * N + n;
            *c = accumulate ? (*c + x) : x;
        }
    }
    if (cluster > 1) cluster_sync();
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes, forge::PerDeviceFlag& flag) {
    bool& done = flag.current();
    if (done) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) done = true;
    return e;
}

// sections that one CTA of the few-rows kernel may keep, and the CTAs that share a tile's sections
constexpr int kFewMaxSlots = 64;

template <int MT, typename T>
int launch_few(const T* A, const T* W, const float* bias, float* C, int M, int N, int K, int accumulate, int vec, int w_at_rest, cudaStream_t stream) {
    static forge::PerDeviceFlag flag;
    const int sections = (K + kSection - 1) / kSection, rounds = (sections + kMaxCluster - 1) / kMaxCluster, cluster = (sections + rounds - 1) / rounds;
    const int slots = (sections + cluster - 1) / cluster;
    const size_t most = sizeof(float) * FewSmem<MT>::floats(MT >= 16 ? 8 : kFewMaxSlots);
    if (cudaError_t e = allow_smem(gemm_simt_few_kernel<MT, T>, most, flag)) return forge::check_launch("gemm_simt (shared memory)", e);
    return forge::check_launch("gemm_simt", forge::launch(gemm_simt_few_kernel<MT, T>, dim3((unsigned)((N + kRowsW - 1) / kRowsW) * cluster), dim3(kFewThreads),
                                                          sizeof(float) * FewSmem<MT>::floats(slots), stream, cluster, A, W, bias, C, M, N, K, accumulate, cluster, vec,
                                                          w_at_rest));
}

template <int BM, typename T>
int launch_tile(const T* A, const T* W, const float* bias, float* C, int M, int N, int K, int accumulate, int vec, int cluster, cudaStream_t stream) {
    static forge::PerDeviceFlag flag;
    const int sections = (K + kSection - 1) / kSection, slots = cluster > 1 ? (sections + cluster - 1) / cluster : std::min(sections, 2);
    if (cudaError_t e = allow_smem(gemm_simt_tile_kernel<BM, T>, sizeof(float) * TileSmem<BM>::floats(2), flag)) return forge::check_launch("gemm_simt (shared memory)", e);
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    if (tiles * cluster > 0x7fffffffLL) return forge::fail(FORGE_ERR_UNSUPPORTED, "gemm_simt: M=%d N=%d too large", M, N);
    return forge::check_launch("gemm_simt", forge::launch(gemm_simt_tile_kernel<BM, T>, dim3((unsigned)(tiles * cluster)), dim3(kTileThreads),
                                                          sizeof(float) * TileSmem<BM>::floats(slots), stream, cluster, A, W, bias, C, M, N, K, accumulate, cluster, vec));
}

template <typename T>
int run(const T* A, const T* W, const float* bias, float* C, int M, int N, int K, int accumulate, int w_at_rest, cudaStream_t stream) {
    const uintptr_t mask = 4 * sizeof(T) - 1;
    const int vec = K % 4 == 0 && ((uintptr_t)A & mask) == 0 && ((uintptr_t)W & mask) == 0 ? 1 : 0;
    const int sections = (K + kSection - 1) / kSection;
    // few rows: up to 32 (one walk over W serves them all), and sections that fit the CTA's slots
    // (16-bit operands come without cp.async, 32 rows of W by one or two warps where K is short: from nine rows of A on the tiles are faster there;
    // [101 x 73], 24 rows: 14.6 us, as tiles 6.9)
    const bool short_halves = sizeof(T) == 2 && M > 8 && K <= 2 * kChunk;
    if (M <= 32 && !short_halves && sections <= (M > 8 ? 8 : kFewMaxSlots) * kMaxCluster) {
#define FORGE_FEW(MT) if (M <= MT) return launch_few<MT, T>(A, W, bias, C, M, N, K, accumulate, vec, w_at_rest, stream);
        FORGE_FEW(1) FORGE_FEW(2) FORGE_FEW(4) FORGE_FEW(8) FORGE_FEW(16) FORGE_FEW(32)
#undef FORGE_FEW
    }
    // Tile height and CTAs per tile, by the time that their units take (a unit: a CTA's section of a tile, 40 us of 64 rows and 62 of 128 on an SM of its
    // own and hardly less for two side by side).  Up to a third of the SMs every CTA has one to itself; from there on some SMs get two while others get
    // none (a kernel's first CTAs go where the kernel ahead has left), as good as all at one CTA an SM; beyond two an SM they are dealt out as they
    // finish, with half a unit of tail.  Clusters of three, and of other odd sizes, leave SMs out.  Fitted to 64 sizes of 40 to 512 rows: 0.8 % over
    // the best choice on average, where the busiest SM's work alone (before) was 10 % over it: [2560 x 2048] at 333 rows 193 -> 124 us, [4096 x 4096] at 64
    // 136 -> 84, [4096 x 14336] at 100 917 -> 472.
    const double sms = forge::sm_count();
    int best_bm = 128, best_c = 1;
    double best = -1.0;
    for (int bm = 64; bm <= 128; bm *= 2)
        for (int c = 1; c <= kMaxCluster && c <= sections; ++c) {
            const int rounds = (sections + c - 1) / c;
            if (c > 1 && rounds > 2) continue;                                    // parked sections beyond two do not fit beside a second CTA
            const double ctas = (double)((M + bm - 1) / bm) * ((N + BN - 1) / BN) * c;
            const double share = ctas <= sms / 3 ? 1.0 : ctas <= 1.08 * sms ? 1.0 + (ctas - sms / 3) / (0.75 * sms) : ctas <= 2 * sms ? 2.0 : ctas / sms + 0.5;
            const double packing = c <= 2 || ctas <= 1.3 * sms ? 1.0 : c == 3 ? 1.4 : (c & (c - 1)) ? 1.15 : 1.03;
            const double cost = rounds * share * packing * (bm == 64 ? 40.0 : 62.0);
            if (best < 0 || cost < best) { best = cost; best_bm = bm; best_c = c; }
        }
    return best_bm == 64 ? launch_tile<64, T>(A, W, bias, C, M, N, K, accumulate, vec, best_c, stream)
                         : launch_tile<128, T>(A, W, bias, C, M, N, K, accumulate, vec, best_c, stream);
}

}  // namespace

// dtype: type of both A and W (FORGE_F32 or FORGE_BF16).  C is fp32.  accumulate != 0: C += A.W^T + bias.
// w_at_rest: no kernel that is still running when this one is launched writes W, which may then be read before the one ahead has finished.
extern "C" int forge_gemm_simt(const void* A, const void* W, const float* bias, float* C, int dtype,
                               int M, int N, int K, int accumulate, int w_at_rest, cudaStream_t stream) {
    if (M < 0 || N <= 0 || K <= 0) return forge::fail(FORGE_ERR_ARG, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return FORGE_OK;
    if (M > 64 * 65535) return forge::fail(FORGE_ERR_UNSUPPORTED, "gemm_simt: M=%d too large", M);
    FORGE_DISPATCH_DTYPE(dtype, TT, return run<TT>((const TT*)A, (const TT*)W, bias, C, M, N, K, accumulate, w_at_rest, stream));
}
