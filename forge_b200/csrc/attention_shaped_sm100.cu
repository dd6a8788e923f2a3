// Prompt portions of two attentions on the 5th-generation tensor cores: attention over latent rows (attention_latent.cu) and
// attention with shaped scores (attention_scored.cu: one or two maps a head, distance term, cap, window, chunk, sink).  Both are, per CTA,
// up to 128 rows of queries over tiles of 64 keys with a two-term softmax weight:
//
//   S = Q K^T      tcgen05.mma M=128 N=64 per 16 channels, Q (all its channels) and the key blocks in shared memory, S in TMEM (two buffers)
//   softmax        128 threads, one row each, 64 scores in registers, fp32; a weight becomes two bfloat16 numbers, its rounding and
//                  what the rounding left over (16 bits of mantissa, as in the mma.sync kernels), written to TMEM over the scores it came from
//   O += P V       tcgen05.mma M=128 N=VC with P from TMEM, once for the rest and once for the rounding, V MN-major as the cache has it
//
// A row is a (token, head) pair: a tile is 128 / heads tokens of one request (rows left over stay empty); the heads are all that read the
// same keys (every head of the latent attention, the group of one kv head otherwise).  A tile of keys is a set of blocks of 64 channels
// (64 keys x 128 bytes, 128-byte swizzle), one TMA box per page and block.  The blocks are of two kinds, each with a ring of its own: key
// blocks that only S reads, and value blocks that O reads (and, over latent rows, S too: a row's first C channels are key and value).
// Values wider than 256 channels are cut into chunks of 256, a CTA each (O is VC of the 512 TMEM columns); the CTAs of a latent row's
// two chunks both make the scores: 36 + 8 MMAs a tile each.  The queries of 576 channels (147 KB) would leave room for one tile of rows, so
// there the 256 channels that meet the value blocks lie in TMEM (128 columns beside S and O: the A operand may come from there), and two
// tiles fit.  With values of up to 128 channels two CTAs fit an SM.
//
// Warps 0-3 run one thread each (copies, P V, Q K^T), warps 4-7 are the rows; registers change hands with setmaxnreg.  Every wait is bounded.
#include "common.cuh"
#include "checks.cuh"
#include "sm100.cuh"

namespace {
using namespace sm100;

constexpr int BQ = 128, BKV = 64, kThreads = 256, kQkWarp = 2;
constexpr int kLaunchRegs = 128, kRegsFew = 64, kRegsMany = 192;
static_assert(kRegsFew + kRegsMany <= 2 * kLaunchRegs, "the two warpgroups cannot hold more registers than the CTA was given");
constexpr int kQBlock = BQ * 128, kBlock = BKV * 128;          // bytes of 64 channels of the queries / of a tile of keys
constexpr int kMaxStages = 3, kBarBytes = 512, kSmemLimit = 227 * 1024;
constexpr float kRefSlack = 8.0f;     // a row's reference exponent moves only when its maximum has grown by more than 2^8 (see attention_sm100.cu)
constexpr float kLog2e = 1.4426950408889634f;

struct ShapedParams {
    __nv_bfloat16* out;               // row t at out + t * out_ld, head h's values from h * E on (u == null)
    float* u;                         // fp32 [T, H, M, E], normalised (two maps)
    long long out_ld;
    const __nv_bfloat16* q;           // (q_tmem) [T, H, D]
    const int32_t *block_table, *tok_req, *positions, *tile_t0, *tile_n;
    const float *r1, *r2, *sink;
    int H, heads, inner, M, D, E, VC; // heads: of a CTA; inner: CTAs of one tile (groups x maps x chunks of values)
    int q_channels;                   // channels of a query row that enter S
    int key_blocks, value_blocks;     // blocks of 64 channels of the two kinds
    int latent;                       // the value blocks are key blocks too
    int q_tmem;                       // ... and the query channels that meet them are in TMEM, not in shared memory
    int stages, page_size, box_rows, max_pages, window, chunk, vec_out;
    float scale, softcap, out_scale;
    uint32_t tmem_cols;
    int* status;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// tanh(x) = 1 - 2 / (e^(2x) + 1), as the mma.sync kernel has it
__device__ __forceinline__ float tanh_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(ex2(x * 2.8853900817779268f) + 1.0f));
    return fmaf(-2.0f, r, 1.0f);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// D[tmem] (+)= A[tmem] . B[smem]^T: row r of A is lane r, 16 channels are eight columns of two bfloat16 numbers
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ int first_visible(int pos, int window, int chunk) {
    int lo = 0;
    if (window > 0) lo = max(lo, pos - window + 1);
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    return lo;
}

// score i of the row's 64 (i is a constant after unrolling)
#define SV(i) ((i) < 32 ? sv_lo[(i) & 31] : sv_hi[(i) & 31])

template <bool SHAPED>
__global__ void __launch_bounds__(kThreads, 2)
shaped_attention_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                              const __grid_constant__ CUtensorMap tmap_v, const ShapedParams p) {
    extern __shared__ uint8_t smem_raw[];
    const int tile = blockIdx.x / p.inner;
    const int t0 = p.tile_t0[tile], nq = p.tile_n[tile];
    if (!FORGE_TOKEN_OK(t0) || !FORGE_TOKEN_OK(t0 + nq - 1)) return;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int q_blocks = (p.q_channels + 63) / 64 - (p.q_tmem ? p.value_blocks : 0);
    uint8_t* q_s = smem;                                            // [q_blocks][128][64] bf16, K-major, swizzled
    uint8_t* k_s = q_s + q_blocks * kQBlock;                        // [stages][key_blocks][64 keys][64]
    uint8_t* v_s = k_s + p.stages * p.key_blocks * kBlock;          // [stages][value_blocks][64 keys][64]
    uint64_t* q_full = reinterpret_cast<uint64_t*>(v_s + p.stages * p.value_blocks * kBlock);
    uint64_t* tail = q_full + 1;                  // the copies of a tile whose last rows are cleared before anybody reads it
    uint64_t* k_full = tail + 1;                  // [kMaxStages]
    uint64_t* k_empty = k_full + kMaxStages;
    uint64_t* v_full = k_empty + kMaxStages;
    uint64_t* v_empty = v_full + kMaxStages;
    uint64_t* s_full = v_empty + kMaxStages;      // [2]
    uint64_t* p_ready = s_full + 2;               // [2]
    uint64_t* o_done = p_ready + 2;               // [2]
    uint64_t* q_ready = o_done + 2;               // the query channels in TMEM
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_ready + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int within = blockIdx.x % p.inner, chunks = p.E / p.VC;
    const int vc = within % chunks, mp = within / chunks % p.M, group = within / (chunks * p.M);
    const int box_tokens = BQ / p.heads, q_rows = box_tokens * p.heads;

    if (threadIdx.x == 0) {
        *abort = 0;
        mbar_init(q_full, 1);
        mbar_init(tail, 1);
        mbar_init(q_ready, 4);
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&p_ready[b], 4);
            mbar_init(&o_done[b], 1);
        }
        mbar_fence_init();
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
    }
    // the stages start as zeros: pages that are skipped (behind the window, beyond the request) leave their rows as they are, and those
    // rows must hold finite numbers (their weights are 0); so do the query rows that a tile of fewer than 128 leaves unwritten
    {
        uint4* z = reinterpret_cast<uint4*>(q_rows < BQ ? q_s : k_s);
        const int n = (int)(reinterpret_cast<uint8_t*>(q_full) - reinterpret_cast<uint8_t*>(z)) / 16;
        for (int i = threadIdx.x; i < n; i += kThreads) z[i] = make_uint4(0, 0, 0, 0);
    }
    fence_proxy_async();
    if (warp == 1) {
        tmem_alloc(tmem_slot, p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot, tmem_o = tmem_base + 2 * BKV;
    forge::pdl_launch_dependents();

    // (the step's tile lists, positions and tables were written before its first kernel started)
    const int req = p.tok_req[t0], pos0 = p.positions[t0], pos_last = pos0 + nq - 1;
    const int t_begin = first_visible(pos0, p.window, p.chunk) / BKV, t_end = pos_last / BKV + 1, n_iter = t_end - t_begin;
    const int seen_from = first_visible(pos0, p.window, p.chunk);
    forge::pdl_wait();

    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsFew));
    if (warp == 0) {
        // ------------------------------------------------------------------ copies
        const int32_t* table = p.block_table + (size_t)req * p.max_pages;
        const int ppt = p.page_size >= BKV ? 1 : BKV / p.page_size;       // boxes a tile and block
        const int k_col0 = p.latent ? 0 : mp * p.D, v_col0 = vc * p.VC, row0 = group * p.page_size;
        const int skip = p.latent ? vc * p.value_blocks : 1 << 20;        // key block i stands for channel block i, or i + value_blocks from here on
        if (lane == 0) {
            mbar_arrive_expect_tx(q_full, q_blocks * q_rows * 128);
            for (int b = 0; b < q_blocks; ++b)
                tma_load_3d(q_s + b * kQBlock, &tmap_q, q_full, k_col0 + (p.q_tmem && b >= skip ? b + p.value_blocks : b) * 64, group * p.heads, t0);
        }
        bool ok = true;
        int st = 0, ph = 0, tail_ph = 0;
        for (int it = 0; it < n_iter && ok; ++it) {
            const int j0 = (t_begin + it) * BKV;
            // one lane a box of rows: its page, or -1 where no token of the tile sees a key
            int page = -1;
            if (lane < ppt) {
                const int j = j0 + lane * p.box_rows;
                const int idx = j / p.page_size;
                if (j <= pos_last && j + p.box_rows > seen_from && idx < p.max_pages) page = table[idx];
                if (page >= 0 && !FORGE_PAGE_OK(page)) page = -1;
            }
            const int n_valid = __popc(__ballot_sync(0xffffffffu, page >= 0));
            const int off = p.page_size > BKV ? j0 % p.page_size : 0;
            const bool last = j0 + BKV - 1 > pos_last;                    // rows behind the last token: cleared below
            uint8_t* kd = k_s + st * p.key_blocks * kBlock;
            uint8_t* vd = v_s + st * p.value_blocks * kBlock;
            const uint32_t box_bytes = p.box_rows * 128;
            if (p.key_blocks > 0) {
                if (lane == 0) {
                    ok = mbar_wait<true>(&k_empty[st], ph ^ 1, abort, p.status, 1);
                    if (ok) mbar_arrive_expect_tx(&k_full[st], p.key_blocks * n_valid * box_bytes);
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                __syncwarp();
                if (page >= 0)
                    for (int b = 0; b < p.key_blocks; ++b)
                        tma_load_3d(kd + b * kBlock + lane * box_bytes, &tmap_k, &k_full[st], k_col0 + (b < skip ? b : b + p.value_blocks) * 64, row0 + off, page);
            }
            if (lane == 0) {
                ok = mbar_wait<true>(&v_empty[st], ph ^ 1, abort, p.status, 2);
                if (ok) mbar_arrive_expect_tx(last ? tail : &v_full[st], p.value_blocks * n_valid * box_bytes);
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            __syncwarp();
            if (page >= 0)
                for (int b = 0; b < p.value_blocks; ++b)
                    tma_load_3d(vd + b * kBlock + lane * box_bytes, &tmap_v, last ? tail : &v_full[st], v_col0 + b * 64, row0 + off, page);
            if (last) {
                // what lies in the cache behind the last token counts as zeros: a weight of 0 would not silence a NaN there
                if (lane == 0) ok = mbar_wait<true>(tail, tail_ph, abort, p.status, 3);
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) break;
                tail_ph ^= 1;
                const int from = pos_last + 1 - j0, pieces = (BKV - from) * 8;
                for (int b = 0; b < p.value_blocks; ++b)
                    for (int i = lane; i < pieces; i += 32) reinterpret_cast<uint4*>(vd + b * kBlock + from * 128)[i] = make_uint4(0, 0, 0, 0);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_full[st]);
            }
            if (++st == p.stages) { st = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ P V
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16_f32_bmn(BQ, p.VC);
            bool ok = true;
            int st = 0, ph = 0;
            for (int it = 0; it < n_iter && ok; ++it) {
                const int b = it & 1;
                if (!(ok = mbar_wait<true>(&v_full[st], ph, abort, p.status, 4))) break;
                if (!(ok = mbar_wait<true>(&p_ready[b], (it >> 1) & 1, abort, p.status, 5))) break;
                tc_fence_after_sync();
                const uint64_t vdesc = umma_desc_mn_sw128(smem_u32(v_s + st * p.value_blocks * kBlock), kBlock);
                const uint32_t pt = tmem_base + b * BKV;
#pragma unroll
                for (int k = 0; k < BKV / 16; ++k) {
                    const uint64_t vk = umma_desc_advance(vdesc, k * 2048);
                    umma_bf16_ta(tmem_o, pt + 32 + k * 8, vk, idesc, (it | k) != 0);
                    umma_bf16_ta(tmem_o, pt + k * 8, vk, idesc, 1);
                }
                umma_commit(&o_done[b]);
                umma_commit(&v_empty[st]);
                if (++st == p.stages) { st = 0; ph ^= 1; }
            }
        }
    } else if (warp == kQkWarp) {
        // ------------------------------------------------------------------ Q K^T
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16_f32(BQ, BKV);
            const int skip = p.latent ? vc * p.value_blocks : 1 << 20;
            bool ok = mbar_wait<true>(q_full, 0, abort, p.status, 6);
            int st = 0, ph = 0;
            for (int it = 0; it < n_iter && ok; ++it) {
                const int b = it & 1;
                // (the scores' buffer holds the weights of tile it - 2 until its P V is done)
                if (it >= 2 && !(ok = mbar_wait<true>(&o_done[b], ((it - 2) >> 1) & 1, abort, p.status, 7))) break;
                const uint64_t qdesc = umma_desc_k_sw128(smem_u32(q_s));
                uint32_t add = 0;
                // key block `blk` of a ring stage against the query's channel block in shared memory
                auto product = [&](const uint8_t* blocks, int blk, int q_block, int channel_block) {
                    const uint64_t a = umma_desc_advance(qdesc, q_block * kQBlock), w = umma_desc_k_sw128(smem_u32(blocks + blk * kBlock));
                    const int steps = min(4, (p.q_channels - channel_block * 64) / 16);
                    for (int k = 0; k < steps; ++k) {
                        umma_bf16(tmem_base + b * BKV, umma_desc_advance(a, k * 32), umma_desc_advance(w, k * 32), idesc, add);
                        add = 1;
                    }
                };
                if (p.key_blocks > 0) {
                    if (!(ok = mbar_wait<true>(&k_full[st], ph, abort, p.status, 8))) break;
                    tc_fence_after_sync();
                    for (int i = 0; i < p.key_blocks; ++i) {
                        const int channel_block = i < skip ? i : i + p.value_blocks;
                        product(k_s + st * p.key_blocks * kBlock, i, p.q_tmem ? i : channel_block, channel_block);
                    }
                    umma_commit(&k_empty[st]);
                }
                if (p.latent) {
                    if (it == 0 && p.q_tmem && !(ok = mbar_wait<true>(q_ready, 0, abort, p.status, 13))) break;
                    if (!(ok = mbar_wait<true>(&v_full[st], ph, abort, p.status, 9))) break;
                    tc_fence_after_sync();
                    for (int i = 0; i < p.value_blocks; ++i) {
                        const uint8_t* blocks = v_s + st * p.value_blocks * kBlock;
                        if (p.q_tmem) {
                            const uint64_t w = umma_desc_k_sw128(smem_u32(blocks + i * kBlock));
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                umma_bf16_ta(tmem_base + b * BKV, tmem_o + p.VC + i * 32 + k * 8, umma_desc_advance(w, k * 32), idesc, add);
                                add = 1;
                            }
                        } else {
                            product(blocks, i, skip + i, skip + i);
                        }
                    }
                }
                umma_commit(&s_full[b]);
                if (++st == p.stages) { st = 0; ph ^= 1; }
            }
        }
    }
    } else {
        // ------------------------------------------------------------------ the rows (warps 4..7)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMany));
        const int quarter = warp & 3, r = quarter * 32 + lane;
        const bool valid = r < nq * p.heads;
        const int tok = t0 + (valid ? r / p.heads : 0), head = group * p.heads + (valid ? r % p.heads : 0), pos = pos0 + tok - t0;
        const int see = first_visible(pos, p.window, p.chunk);
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16), t_out = t_lane + 2 * BKV;
        const float sl2 = p.scale * kLog2e;
        const float cap_in = p.softcap > 0.f ? p.scale / p.softcap : 0.f, cap_out = p.softcap * kLog2e;
        const float r1v = SHAPED && p.r1 ? p.r1[head] : 0.f, r2v = SHAPED && p.r1 ? p.r2[head] : 0.f;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        if (p.q_tmem) {                       // this row's channels vc * VC .. of the query, two to a column
            const __nv_bfloat16* src = p.q + ((size_t)tok * p.H + head) * p.D + vc * p.VC;
            for (int c = 0; c < p.VC; c += 64) {
                uint32_t w[32];
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const uint4 v = valid ? *reinterpret_cast<const uint4*>(src + c + 2 * i) : make_uint4(0, 0, 0, 0);
                    w[i] = v.x; w[i + 1] = v.y; w[i + 2] = v.z; w[i + 3] = v.w;
                }
                __syncwarp();
                tmem_st_32x32b_x32(t_out + p.VC + c / 2, w);
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_ready);
        }
        for (int it = 0; it < n_iter && ok; ++it) {
            const int j0 = (t_begin + it) * BKV, b = it & 1;
            if (!(ok = mbar_wait<true>(&s_full[b], (it >> 1) & 1, abort, p.status, 10))) break;
            tc_fence_after_sync();
            uint32_t sv_lo[32], sv_hi[32];
            tmem_ld_32x32b_x32(t_lane + b * BKV, sv_lo);
            tmem_ld_32x32b_x32(t_lane + b * BKV + 32, sv_hi);
            tmem_ld_wait();
            const bool need_mask = !valid || j0 + BKV - 1 > pos || j0 < see;
            if (SHAPED) {                     // in units of log2 e, shaped, from here on
#pragma unroll
                for (int i = 0; i < BKV; ++i) {
                    float s = __uint_as_float(SV(i));
                    s = p.softcap > 0.f ? cap_out * tanh_fast(s * cap_in) : s * sl2;
                    if (p.r1) s -= r1v * __log2f(fmaf(r2v, (float)max(pos - j0 - i, 0), 1.0f));
                    SV(i) = __float_as_uint(s);
                }
            }
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < BKV; ++i) {
                    const int j = j0 + i;
                    if (!(valid && j <= pos && j >= see)) SV(i) = __float_as_uint(-INFINITY);
                }
            }
            float a0 = -INFINITY, a1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < BKV; i += 4) {
                a0 = max3(a0, __uint_as_float(SV(i)), __uint_as_float(SV(i + 1)));
                a1 = max3(a1, __uint_as_float(SV(i + 2)), __uint_as_float(SV(i + 3)));
            }
            const float mult = SHAPED ? 1.0f : sl2;
            const float top = fmaxf(a0, a1) * mult;
            const float m_new = top > m + kRefSlack ? top : m;            // (-inf + slack is -inf: the first visible key sets it)
            const float alpha = m_new == m ? 1.0f : ex2(m - m_new);
            m = m_new;
            const float ref = m == -INFINITY ? 0.f : m;
            // O is rescaled only when some row of the warp moved its reference; P V of the tile before must be complete by then
            if (it > 0 && !__all_sync(0xffffffffu, alpha == 1.0f)) {
                if (!(ok = mbar_wait<true>(&o_done[b ^ 1], ((it - 1) >> 1) & 1, abort, p.status, 11))) break;
                tc_fence_after_sync();
                for (int c = 0; c < p.VC; c += 32) {
                    uint32_t ov[32];
                    tmem_ld_32x32b_x32(t_out + c, ov);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
                    tmem_st_32x32b_x32(t_out + c, ov);
                }
                tmem_st_wait();
            }
            __syncwarp();                     // (the lanes may have parted over the mask; what follows is warp-wide)
            // the weights, their sum, and P in two terms over the scores' columns: roundings in the first 32, the rest in the next
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
            for (int c = 0; c < BKV; c += 32) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 32; i += 4) {
                    const float p0 = ex2(fmaf(__uint_as_float(SV(c + i)), mult, -ref)), p1 = ex2(fmaf(__uint_as_float(SV(c + i + 1)), mult, -ref));
                    const float p2 = ex2(fmaf(__uint_as_float(SV(c + i + 2)), mult, -ref)), p3 = ex2(fmaf(__uint_as_float(SV(c + i + 3)), mult, -ref));
                    s0 += p0;
                    s1 += p1;
                    s2 += p2;
                    s3 += p3;
                    const uint32_t h01 = pack_bf16(p0, p1), h23 = pack_bf16(p2, p3);
                    hi[i / 2] = h01;
                    hi[i / 2 + 1] = h23;
                    lo[i / 2] = pack_bf16(p0 - __uint_as_float(h01 << 16), p1 - __uint_as_float(h01 & 0xffff0000u));
                    lo[i / 2 + 1] = pack_bf16(p2 - __uint_as_float(h23 << 16), p3 - __uint_as_float(h23 & 0xffff0000u));
                }
                tmem_st_32x32b_x16(t_lane + b * BKV + c / 2, hi);
                tmem_st_32x32b_x16(t_lane + b * BKV + 32 + c / 2, lo);
            }
            l = l * alpha + ((s0 + s1) + (s2 + s3));
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        if (ok) ok = mbar_wait<true>(&o_done[(n_iter - 1) & 1], ((n_iter - 1) >> 1) & 1, abort, p.status, 12);
        tc_fence_after_sync();
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            float inv = l > 0.f ? 1.0f / l : 0.f;
            if (p.sink != nullptr && l > 0.f) {          // the denominator also counts exp(sink of the head)
                const float sb = p.sink[head] * kLog2e, top = fmaxf(m, sb), x = ex2(m - top);
                inv = x / fmaf(l, x, ex2(sb - top));
            }
            inv *= p.out_scale;
            const int v0 = vc * p.VC;
            // every lane takes part in the TMEM loads (they are warp-wide instructions); only valid rows store
            for (int c = 0; c < p.VC; c += 32) {
                uint32_t ov[32];
                __syncwarp();
                tmem_ld_32x32b_x32(t_out + c, ov);
                tmem_ld_wait();
                if (!valid) {
                } else if (p.u != nullptr) {
                    float* dst = p.u + (((size_t)tok * p.H + head) * p.M + mp) * p.E + v0 + c;
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(ov[i]) * inv, __uint_as_float(ov[i + 1]) * inv,
                                                                          __uint_as_float(ov[i + 2]) * inv, __uint_as_float(ov[i + 3]) * inv);
                } else {
                    __nv_bfloat16* dst = p.out + (size_t)tok * p.out_ld + (size_t)head * p.E + v0 + c;
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) w[e] = pack_bf16(__uint_as_float(ov[i + 2 * e]) * inv, __uint_as_float(ov[i + 2 * e + 1]) * inv);
                        if (p.vec_out) {
                            *reinterpret_cast<uint4*>(dst + i) = make_uint4(w[0], w[1], w[2], w[3]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e) reinterpret_cast<uint32_t*>(dst + i)[e] = w[e];
                        }
                    }
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
}

// A bf16 tensor of three dimensions read in boxes of 64 x b1 x b2 with 128-byte swizzle; strides in elements.
bool map3(const void* ptr, unsigned long long d0, unsigned long long d1, unsigned long long d2, unsigned long long s1, unsigned long long s2, int b1, int b2,
          CUtensorMap* out, const char** err) {
    auto fn = encode_fn();
    if (!fn) { *err = "cuTensorMapEncodeTiled is not available from the driver"; return false; }
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {s1 * 2, s2 * 2};
    const cuuint32_t box[3] = {64u, (cuuint32_t)b1, (cuuint32_t)b2}, estr[3] = {1u, 1u, 1u};
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || strides[0] % 16 || strides[1] % 16) { *err = "TMA needs 16-byte aligned rows"; return false; }
    if (fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        *err = "cuTensorMapEncodeTiled failed";
        return false;
    }
    return true;
}

bool pages_fit(int page_size) { return page_size >= 8 && (page_size & (page_size - 1)) == 0 && page_size <= 65536; }

size_t smem_bytes(int q_blocks, int blocks, int stages) { return (size_t)q_blocks * kQBlock + (size_t)stages * blocks * kBlock + kBarBytes + 1024; }

// value columns of a CTA: all up to 256, else chunks of 256 (0: not taken)
int value_columns(int E) { return E % 64 ? 0 : E <= 256 ? E : E % 256 ? 0 : 256; }

template <bool SHAPED>
int launch(const char* what, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, ShapedParams p, int num_tiles, cudaStream_t stream) {
    int q_blocks = (p.q_channels + 63) / 64;
    const int blocks = p.key_blocks + p.value_blocks;
    // where the queries leave room for one tile of rows, those that meet the value blocks go to TMEM if it has the columns
    // (latent of 512 + 64 channels: one tile 268 us, two 110 for the portions of 512 and 1,024 tokens behind 700 and none)
    if (p.latent && smem_bytes(q_blocks, blocks, 2) > kSmemLimit && 2 * BKV + p.VC + p.value_blocks * 32 <= 512 && ((uintptr_t)p.q & 15) == 0 && p.D % 8 == 0) {
        p.q_tmem = 1;
        q_blocks -= p.value_blocks;
    }
    p.stages = kMaxStages;
    while (p.stages > 1 && smem_bytes(q_blocks, blocks, p.stages) > kSmemLimit) --p.stages;
    const size_t smem = smem_bytes(q_blocks, blocks, p.stages);
    if (smem > kSmemLimit) return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: queries of %d channels", what, p.q_channels);
    p.tmem_cols = 2 * BKV + p.VC + (p.q_tmem ? p.value_blocks * 32 : 0) <= 256 ? 256 : 512;
    p.box_rows = p.page_size < BKV ? p.page_size : BKV;
    static forge::PerDeviceFlag configured_on;
    bool& configured = configured_on.current();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(shaped_attention_sm100_kernel<SHAPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
        // the warpgroups trade registers inside what the CTA was given at launch: a build that gives less is refused
        cudaFuncAttributes attr;
        e = cudaFuncGetAttributes(&attr, shaped_attention_sm100_kernel<SHAPED>);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
        if (attr.numRegs * 2 < kRegsFew + kRegsMany)
            return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: built with %d registers per thread, needs %d", what, attr.numRegs, (kRegsFew + kRegsMany + 1) / 2);
        configured = true;
    }
    return forge::check_launch(what, forge::launch(shaped_attention_sm100_kernel<SHAPED>, dim3((unsigned)num_tiles * p.inner), dim3(kThreads), smem, stream, 1,
                                                   tq, tk, tv, p));
}

}  // namespace

// 1 if the kernel takes a latent of C channels with R rotated ones for H heads: up to 128 heads, C a multiple of 64 up to 256 or of 256,
// R a multiple of 16, queries that leave room for one tile of rows.
extern "C" int forge_latent_sm100_supports(int H, int C, int R, int page_size) {
    const int VC = value_columns(C), q_blocks = (C + R + 63) / 64;
    return (pages_fit(page_size) && H > 0 && H <= BQ && VC > 0 && R >= 0 && R % 16 == 0 && smem_bytes(q_blocks, q_blocks, 1) <= kSmemLimit) ? 1 : 0;
}

// 1 if it takes M maps of D channels and values of E: D a multiple of 64 up to 128, E of 64 up to 256 or of 256, up to 128 heads a kv head.
extern "C" int forge_scored_sm100_supports(int H, int G, int M, int D, int E, int page_size) {
    return (pages_fit(page_size) && H > 0 && G > 0 && H % G == 0 && H / G <= BQ && (M == 1 || M == 2) && (D == 64 || D == 128) && value_columns(E) > 0) ? 1 : 0;
}

// q bf16 [T, H, C+R]; cache: pages of page_size rows of C+R; out bf16 [T, H, C].  tile_t0 / tile_n: tiles of up to 128 / H tokens of one
// request, the first to run first.  window, sink as for forge_latent_attention_mma.  status: bit 1 is raised where a wait ran out.
extern "C" int forge_latent_attention_sm100(const void* q, const void* cache, const int32_t* block_table, const int32_t* tok_req,
                                            const int32_t* positions, const int32_t* tile_t0, const int32_t* tile_n, void* out, int* status, int T,
                                            int num_tiles, int num_pages, int H, int C, int R, int page_size, int max_pages, float scale, int window,
                                            const float* sink, cudaStream_t stream) {
    if (!forge_latent_sm100_supports(H, C, R, page_size)) return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: H=%d C=%d R=%d page=%d", H, C, R, page_size);
    if (T < 0 || num_tiles < 0 || num_pages <= 0 || max_pages <= 0 || !tile_t0 || !tile_n || !(scale > 0.f))
        return forge::fail(FORGE_ERR_ARG, "latent_attention_sm100: bad arguments");
    if (T == 0 || num_tiles == 0) return FORGE_OK;
    const int KD = C + R, VC = value_columns(C), chunks = C / VC;
    const char* err = nullptr;
    CUtensorMap tq, tk;
    if (!map3(q, KD, H, T, KD, (unsigned long long)H * KD, H, BQ / H, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: q: %s", err);
    if (!map3(cache, KD, page_size, num_pages, KD, (unsigned long long)page_size * KD, page_size < BKV ? page_size : BKV, 1, &tk, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: cache: %s", err);
    ShapedParams p{};
    p.out = (__nv_bfloat16*)out; p.out_ld = (long long)H * C;
    p.block_table = block_table; p.tok_req = tok_req; p.positions = positions; p.tile_t0 = tile_t0; p.tile_n = tile_n;
    p.sink = sink; p.q = (const __nv_bfloat16*)q;
    p.H = p.heads = H; p.inner = chunks; p.M = 1; p.D = KD; p.E = C; p.VC = VC;
    p.q_channels = KD; p.value_blocks = VC / 64; p.key_blocks = (KD + 63) / 64 - p.value_blocks; p.latent = 1;
    p.page_size = page_size; p.max_pages = max_pages; p.window = window;
    p.vec_out = ((uintptr_t)out & 15) == 0; p.scale = scale; p.out_scale = 1.0f; p.status = status;
    return launch<false>("latent_attention_sm100", tq, tk, tk, p, num_tiles, stream);
}

// q bf16 [T, H, M, D]; cache pages of page_stride numbers, [G, page_size, M*D] keys then [G, page_size, E] values; one map: out bf16, rows of
// out_ld, times out_scale; two: u fp32 [T, H, 2, E].  The rest as for forge_scored_attention_mma; tiles of up to 128 / (H/G) tokens.
extern "C" int forge_scored_attention_sm100(const void* q, const void* cache, const int32_t* block_table, const int32_t* tok_req,
                                            const int32_t* positions, const int32_t* tile_t0, const int32_t* tile_n, const float* r1, const float* r2,
                                            float* u, void* out, int* status, int T, int num_tiles, int num_pages, int H, int G, int M, int D, int E,
                                            int page_size, long long page_stride, int max_pages, float scale, float out_scale, long long out_ld, int window,
                                            int chunk, float softcap, const float* sink, cudaStream_t stream) {
    if (!forge_scored_sm100_supports(H, G, M, D, E, page_size))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: H=%d G=%d M=%d D=%d E=%d page=%d", H, G, M, D, E, page_size);
    if (T < 0 || num_tiles < 0 || num_pages <= 0 || max_pages <= 0 || !tile_t0 || !tile_n || !(scale > 0.f) || (r1 == nullptr) != (r2 == nullptr) ||
        (M == 2 && !u) || (M == 1 && !out) || (sink && M != 1) || window < 0 || chunk < 0 || softcap < 0.f ||
        (M == 1 && (out_ld < (long long)H * E || (out_ld & 1))) || page_stride < (long long)G * page_size * (M * D + E))
        return forge::fail(FORGE_ERR_ARG, "scored_attention_sm100: bad arguments");
    if (T == 0 || num_tiles == 0) return FORGE_OK;
    const int MD = M * D, Gq = H / G, VC = value_columns(E), rows = page_size < BKV ? page_size : BKV;
    const char* err = nullptr;
    CUtensorMap tq, tk, tv;
    if (!map3(q, MD, H, T, MD, (unsigned long long)H * MD, Gq, BQ / Gq, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: q: %s", err);
    if (!map3(cache, MD, (unsigned long long)G * page_size, num_pages, MD, page_stride, rows, 1, &tk, &err) ||
        !map3((const __nv_bfloat16*)cache + (size_t)G * page_size * MD, E, (unsigned long long)G * page_size, num_pages, E, page_stride, rows, 1, &tv, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: cache: %s", err);
    ShapedParams p{};
    p.out = (__nv_bfloat16*)out; p.out_ld = out_ld; p.u = M == 2 ? u : nullptr;
    p.block_table = block_table; p.tok_req = tok_req; p.positions = positions; p.tile_t0 = tile_t0; p.tile_n = tile_n;
    p.r1 = r1; p.r2 = r2; p.sink = sink;
    p.H = H; p.heads = Gq; p.inner = G * M * (E / VC); p.M = M; p.D = D; p.E = E; p.VC = VC;
    p.q_channels = D; p.key_blocks = D / 64; p.value_blocks = VC / 64; p.latent = 0;
    p.page_size = page_size; p.max_pages = max_pages; p.window = window; p.chunk = chunk; p.softcap = softcap;
    p.vec_out = ((uintptr_t)out & 15) == 0 && out_ld % 8 == 0; p.scale = scale; p.out_scale = M == 1 ? out_scale : 1.0f; p.status = status;
    return r1 != nullptr || softcap > 0.f ? launch<true>("scored_attention_sm100", tq, tk, tv, p, num_tiles, stream)
                                          : launch<false>("scored_attention_sm100", tq, tk, tv, p, num_tiles, stream);
}

extern "C" const char* forge_last_error() { return forge::error_buffer(); }

// (checks build) the bounds that this library's kernel tests page ids against
FORGE_DEFINE_CHECKS_ENTRY(attention_shaped_sm100)
