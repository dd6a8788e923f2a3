// Paged causal grouped-query attention for prompt portions on the 5th-generation tensor cores (head sizes 64 and
// 128; the library is built per head size, -DFORGE_ATT_HD).
//
// One CTA = one tile of up to 128 query rows of one (request, kv head); a row is a (token, head of the kv head's
// group) pair, row r <-> token r / G, head r % G, so a tile is 128 / G tokens (rounded down: with a group that
// does not divide 128 the last rows of the tile stay empty) and the G heads share every key/value tile.  Per tile
// of 64 keys (HD = head size):
//   S = Q K^T      tcgen05.mma M=128 N=64 K=HD, Q and K in shared memory (TMA, 128-byte swizzle), S in TMEM (two or three buffers)
//   softmax        256 threads, two a row with 32 of the tile's scores each in registers, online max/sum in fp32
//                  (exp2 domain, packed fp32 arithmetic), P as bf16 into TMEM over the scores it came from; the output
//                  accumulator in TMEM is rescaled only when a row's reference exponent has to move (a maximum that grew by more than 2^8)
//   O += P V       tcgen05.mma M=128 N=HD K=64, P from TMEM, V MN-major (keys are rows of 128 bytes), O in TMEM
// Warps 0 and 3 copy keys and values page by page through the request's block table (a ring of its own for either; the page is looked up a
// tile ahead), warp 1 multiplies P V, warp 2 Q K^T: the whole warp walks the loop and the elected lane issues, so that operands come from
// uniform registers.  Warps 4-11 are the softmax rows.  The first warpgroup hands most of its registers to the others (setmaxnreg).  Two such
// CTAs fit an SM.  Before (one thread a row, P through shared memory, products and copies issued from branches of one lane, heads of 128 with one CTA
// an SM) and now, in us: heads of 128, 32/8 of them, 1,500 tokens of three requests behind up to 1,000: 47.5, 29.4; 2,048 tokens 74, 48; heads of 64,
// 32/4: 1,021 tokens of eight requests 10.7, 8.4; 300 tokens of three behind up to 500 15.3, 11.6; 2,048 tokens 42.4, 42.3 (there the
// special-function unit is busy five sixths of the time: 64 weights of a tile and row at four a clock and scheduler).
// Tiles are listed longest first and the kv heads of a tile are neighbouring CTAs, so the
// long tiles of all heads start in the first wave.
// A step with fewer tiles than the GPU has places for CTAs (a short portion on a long context) may list a tile several
// times, each entry with a share of the tile's key tiles (``tile_cut``): such a CTA leaves its sums unnormalised in
// fp32 with the row's reference exponent and sum, and a second kernel adds a tile's shares up in the order of the
// shares.
//   s_j = (q . k_j) * scale for keys max(0, p - window + 1) <= j <= p of the row's position p;
//   o = sum_j softmax(s)_j v_j        (formulas of src/operators/cuda/cuda_flash_attn.cu:154-248)
// Needs G <= 128, 64 % page_size == 0 and page_size >= 8; everything else is served by attention_mma.cu.
#include "common.cuh"
#include "checks.cuh"
#include "sm100.cuh"

#ifndef FORGE_ATT_HD
#define FORGE_ATT_HD 64
#endif

namespace {

using namespace sm100;

constexpr int HD = FORGE_ATT_HD, BQ = 128, BKV = 64, UMMA_K = 16;
static_assert(HD == 64 || HD == 128, "head size 64 or 128");
constexpr int KB = HD / 64;                       // 64-wide blocks of the head: Q, K and V tiles are KB swizzled blocks
constexpr int kThreads = 384;                     // warps 0-3: keys, P V, Q K^T, values; warps 4-11: the softmax rows
constexpr int kQkWarp = 2, kValueWarp = 3, kRowWarps = 8, NK = BKV / 2;  // NK: a thread's keys of a tile
constexpr int kCtasPerSm = 2;
constexpr int kLaunchRegs = 65536 / (kThreads * kCtasPerSm) / 8 * 8;     // what the compiler gives every thread at launch
constexpr int kRegsFew = 48, kRegsMany = 96;       // registers per thread of the three warpgroups after they trade
// setmaxnreg only moves registers inside the CTA's allocation: asking for more than it holds waits for ever
static_assert(kRegsFew + 2 * kRegsMany <= 3 * kLaunchRegs, "the warpgroups cannot hold more registers than the CTA was given");
constexpr int kTileBytes = BQ * 128;              // one block of Q: 128 rows of 128 bytes
constexpr int kQBytes = KB * kTileBytes;
constexpr int kKVBlock = BKV * 128;               // one block of a K or V tile: 64 keys of 128 bytes
constexpr int kKVBytes = KB * kKVBlock;
constexpr int kStages = HD == 64 ? 4 : 2;         // ring slots for key tiles, and as many for value tiles: what two CTAs an SM leave
constexpr int kSmemBytes = kQBytes + 2 * kStages * kKVBytes + 1024 + 512;
static_assert(kSmemBytes <= 112 * 1024, "two CTAs an SM");
constexpr int kBufs = HD == 64 ? 3 : 2;           // tiles whose scores or weights are in TMEM at a time: what 256 columns leave beside O
constexpr int kTmemCols = 256, kTmemO = kBufs * BKV;                     // S of tile it: columns it % kBufs * 64 .. (P: the first 32 of them), then O
static_assert(kTmemO + HD <= kTmemCols, "scores and outputs");

struct AttnTcParams {
    __nv_bfloat16* out;           // [T, NH*HD]
    const int32_t* block_table;   // [S, max_pages]
    const int32_t* tile_req;      // [tiles]
    const int32_t* tile_row0;     // [tiles] first row (token * G + head) of the tile within its request
    const int32_t* tile_cut;      // [tiles][3] or null: this entry's share of the tile's keys (share, shares, first slot)
    float* part_o;                // [slots][NKV][128][HD] unnormalised sums of the entries that share a tile
    float* part_ml;               // [slots][NKV][128][2] reference exponent (exp2 domain) and sum of weights
    const int32_t* q_start;       // [S+1]
    const int32_t* ctx_before;    // [S]
    int NH, NKV, page_size, max_pages, window;
    float scale_log2;
    int* status;
};

// 2^x by the special-function unit (2 ulp); the weights are rounded to bfloat16 right after
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// two fp32 lanes per instruction (the packed fp32 pipe): d = a * b + c and d = a + b on register pairs
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// A row's reference exponent moves only when its maximum has grown by more than this (in the exp2 domain):
// until then the weights are at most 2^8, which fp32 sums and bfloat16 weights hold with the same relative
// precision, and the accumulator in TMEM needs no rescaling.  The final division by the row's sum, taken
// with the same references, makes the result independent of when the reference moved.
constexpr float kRefSlack = 8.0f;

// D[tmem] (+)= A[tmem] . B[smem]^T from the elected lane: row r of A is lane r, 16 keys are eight columns of two bfloat16 numbers
__device__ __forceinline__ void umma_ts_by(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__global__ void __launch_bounds__(kThreads, kCtasPerSm)
paged_attention_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                             const AttnTcParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ float meet[2][BQ];                                   // [half]: what a row's two threads tell each other
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_s = smem;                                            // [KB][128][64] bf16, K-major, swizzled
    uint8_t* k_s = smem + kQBytes;                                  // [kStages][KB][64 keys][64]
    uint8_t* v_s = k_s + kStages * kKVBytes;                        // [kStages][KB][64 keys][64]
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + kStages * kKVBytes);
    uint64_t* q_full = bars;
    uint64_t* k_full = bars + 1;                  // [kStages]
    uint64_t* k_empty = k_full + kStages;         // [kStages]
    uint64_t* v_full = k_empty + kStages;         // [kStages]
    uint64_t* v_empty = v_full + kStages;         // [kStages]
    uint64_t* s_full = v_empty + kStages;         // [kBufs]
    uint64_t* p_ready = s_full + kBufs;           // [kBufs]
    uint64_t* o_done = p_ready + kBufs;           // [kBufs]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + kBufs);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tiles come longest first, and CTAs are handed out in the order of blockIdx.x: the kv heads of one tile are
    // neighbours, so that the long tiles of every head start in the first wave
    const int tile = blockIdx.x / p.NKV, kvh = blockIdx.x % p.NKV;
    const int G = p.NH / p.NKV;

    if (threadIdx.x == 0) {
        *abort = 0;
        mbar_init(q_full, 1);
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int b = 0; b < kBufs; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&p_ready[b], kRowWarps);
            mbar_init(&o_done[b], 1);
        }
        mbar_fence_init();
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_kv);
    }
    fence_proxy_async();
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    forge::pdl_launch_dependents();

    // (the step's tile lists, request boundaries and block tables were written before its first kernel started: they
    // are read ahead of the dependency wait, which orders this kernel after the one that makes q and this step's keys)
    const int s_req = p.tile_req[tile], row0 = p.tile_row0[tile];
    const int qs0 = p.q_start[s_req], qlen = p.q_start[s_req + 1] - qs0, ctx = p.ctx_before[s_req];
    const int tile_rows = (BQ / G) * G;                             // rows of a full tile: whole tokens only
    const int rows_here = min(tile_rows, qlen * G - row0);
    const int pos_lo = ctx + row0 / G, pos_hi = ctx + (row0 + rows_here - 1) / G;
    const int kv_hi = pos_hi + 1;
    const int kv_lo = (p.window > 0 && pos_lo - p.window + 1 > 0) ? pos_lo - p.window + 1 : 0;
    // this entry's share of the tile's key tiles (all of them unless the step cut the tile's keys)
    int share = 0, shares = 1, slot = 0;
    if (p.tile_cut != nullptr) {
        share = p.tile_cut[3 * tile];
        shares = p.tile_cut[3 * tile + 1];
        slot = p.tile_cut[3 * tile + 2] + share;
    }
    const int t_first = kv_lo / BKV, n_all = (kv_hi + BKV - 1) / BKV - t_first;
    const int t_begin = t_first + (int)((long long)n_all * share / shares);
    const int t_end = t_first + (int)((long long)n_all * (share + 1) / shares);
    const int n_iter = t_end - t_begin;
    forge::pdl_wait();

    // the softmax rows keep their scores in registers; the other warpgroup gives its registers up for that
    const int rounds = __shfl_sync(0xffffffffu, n_iter, 0);
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsFew));
    if (warp == 0 || warp == kValueWarp) {
        // ------------------------------------------------------------------ copies: keys (and the queries), values
        const bool values = warp == kValueWarp;
        const int32_t* table = p.block_table + (size_t)s_req * p.max_pages;
        const int page_shift = 31 - __clz(p.page_size), ppt = BKV >> page_shift;       // (the page size divides 64); pages per key tile
        const uint32_t page_bytes = p.page_size * 128;
        if (!values && lane == 0) {
            mbar_arrive_expect_tx(q_full, KB * tile_rows * 128);
            for (int kb = 0; kb < KB; ++kb) tma_load_3d(q_s + kb * kTileBytes, &tmap_q, q_full, kb * 64, kvh * G, qs0 + row0 / G);
        }
        // one lane a page: its first row of the cache, or -1 where no row of the tile sees a key of it.  Asked for a tile ahead.
        auto page_of = [&](int it) {
            int page = -1;
            const int tp = (t_begin + it) * BKV + (lane << page_shift), idx = tp >> page_shift;
            if (lane < ppt && it < rounds && tp < kv_hi && tp + p.page_size > kv_lo && idx < p.max_pages) page = table[idx];
            return page;
        };
        uint64_t* full = values ? v_full : k_full;
        uint64_t* empty = values ? v_empty : k_empty;
        uint8_t* ring = values ? v_s : k_s;
        int st = 0, ph = 0, next_page = page_of(0);
        for (int it = 0; it < rounds; ++it) {
            int page = next_page;
            next_page = page_of(it + 1);
            if (page >= 0 && !FORGE_PAGE_OK(page)) page = -1;
            if (!warp_wait<true>(&empty[st], ph ^ 1, abort, p.status, values ? 9 : 1)) break;
            if (lane == 0) mbar_arrive_expect_tx(&full[st], kKVBytes);
            __syncwarp();
            // A page that brings nothing (beyond the request, released by the window, or none in the table) is copied all the same, from rows before the
            // cache's first: the copy fills zeros in.  What the slot held before may be no number, which a weight of 0 would not silence.
            if (lane < ppt) {
                const int row = ((page * 2 + (values ? 1 : 0)) * p.NKV + kvh) * p.page_size;
                uint8_t* dst = ring + st * kKVBytes + lane * page_bytes;
                if (ppt == 1) tma_load_3d(dst, &tmap_kv, &full[st], 0, row, 0);              // (a box of all blocks)
                else
                    for (int kb = 0; kb < KB; ++kb) tma_load_3d(dst + kb * kKVBlock, &tmap_kv, &full[st], 0, row, kb);
            }
            if (++st == kStages) { st = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ P V
        constexpr uint32_t idesc_pv = umma_idesc_bf16_f32_bmn(BQ, HD);
        const uint32_t leader = elect_one(), t_at = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t v_desc0 = umma_desc_mn_sw128(smem_u32(v_s), kKVBlock);
        int vst = 0, vph = 0;
        for (int it = 0; it < rounds; ++it) {
            const int b = it % kBufs, bp = it / kBufs & 1;
            if (!warp_wait<true>(&v_full[vst], vph, abort, p.status, 4)) break;
            if (!warp_wait<true>(&p_ready[b], bp, abort, p.status, 5)) break;
            tc_fence_after_sync();
            const uint64_t v_desc = umma_desc_advance(v_desc0, vst * kKVBytes);
#pragma unroll
            for (int k = 0; k < BKV / UMMA_K; ++k)
                umma_ts_by(leader, t_at + kTmemO, t_at + b * BKV + k * 8, umma_desc_advance(v_desc, k * 2048), idesc_pv, k > 0 ? 1 : (uint32_t)(it > 0));
            umma_commit_by(leader, &o_done[b]);
            umma_commit_by(leader, &v_empty[vst]);
            if (++vst == kStages) { vst = 0; vph ^= 1; }
        }
    } else if (warp == kQkWarp) {
        // ------------------------------------------------------------------ Q K^T
        constexpr uint32_t idesc_qk = umma_idesc_bf16_f32(BQ, BKV);
        const uint32_t leader = elect_one(), t_at = __shfl_sync(0xffffffffu, tmem_base, 0);
        const uint64_t q_desc = umma_desc_k_sw128(smem_u32(q_s)), k_desc0 = umma_desc_k_sw128(smem_u32(k_s));
        int kst = 0, kph = 0;
        if (warp_wait<true>(q_full, 0, abort, p.status, 2))
        for (int it = 0; it < rounds; ++it) {
            const int b = it % kBufs, bp = it / kBufs & 1;
            if (!warp_wait<true>(&k_full[kst], kph, abort, p.status, 3)) break;
            // (the scores' buffer holds the weights of tile it - kBufs until its P V is done)
            if (it >= kBufs && !warp_wait<true>(&o_done[b], bp ^ 1, abort, p.status, 10)) break;
            tc_fence_after_sync();
            const uint64_t k_desc = umma_desc_advance(k_desc0, kst * kKVBytes);
#pragma unroll
            for (int kb = 0; kb < KB; ++kb)
#pragma unroll
                for (int k = 0; k < 64 / UMMA_K; ++k)
                    umma_bf16_by(leader, t_at + b * BKV, umma_desc_advance(q_desc, kb * kTileBytes + k * 32), umma_desc_advance(k_desc, kb * kKVBlock + k * 32),
                                 idesc_qk, (kb | k) != 0);
            umma_commit_by(leader, &s_full[b]);
            umma_commit_by(leader, &k_empty[kst]);
            if (++kst == kStages) { kst = 0; kph ^= 1; }
        }
    }
    } else {
        // ------------------------------------------------------------------ softmax rows (warps 4..11)
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMany));
        const int half = (warp - 4) >> 2, quarter = warp & 3;    // the quarter of TMEM's lanes that this warp may touch
        const int r_local = quarter * 32 + lane;                 // row of the tile = TMEM lane
        const int r = row0 + r_local;
        const bool valid = r_local < rows_here;
        const int pos = ctx + r / G;
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t t_out = t_lane + kTmemO;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        // (a wait that ran out lets the loop go on without waiting: the two threads of a row have to meet in every round)
        for (int it = 0; it < n_iter; ++it) {
            const int j0 = (t_begin + it) * BKV + half * NK, b = it % kBufs, bp = it / kBufs & 1;
            const uint32_t t_s = t_lane + b * BKV;
            ok = ok && mbar_wait<true>(&s_full[b], bp, abort, p.status, 6);
            __syncwarp();
            tc_fence_after_sync();
            uint32_t sv[NK];
            tmem_ld_32x32b_x32(t_s + half * NK, sv);
            tmem_ld_wait();
            // rows whose keys of this tile are all visible skip the per-key tests (all tiles but the ones on the
            // diagonal or at the window's edge); masked scores become -inf here, once.  (A row that stands for no token may hold any number:
            // nobody reads what comes of it.)
            const bool need_mask = valid && (j0 + NK - 1 > pos || (p.window > 0 && j0 <= pos - p.window));
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < NK; ++i) {
                    const int j = j0 + i;
                    if (!(j <= pos && (p.window <= 0 || j > pos - p.window))) sv[i] = __float_as_uint(-INFINITY);
                }
            }
            // pass 1: the maximum of the raw scores (the scale is positive, so it commutes with the maximum),
            // in two independent chains of three-input maxima
            float a0 = -INFINITY, a1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < NK; i += 4) {
                a0 = max3(a0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
                a1 = max3(a1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
            }
            float mx_tile = fmaxf(a0, a1) * p.scale_log2;
            // Whether any of the two warps' rows has to move its reference; mostly none has, and the row's maximum is nobody's business.
            // (Both have read their scores by then: either's weights may overwrite the other's.)
            int moves;
            __syncwarp();
            tc_fence_before_sync();
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t"
                "setp.gt.f32 p, %1, %2;\n\t"
                "barrier.cta.red.or.pred.aligned q, %3, 64, p;\n\t"
                "selp.s32 %0, 1, 0, q;\n\t}"
                : "=r"(moves) : "f"(mx_tile), "f"(m + kRefSlack), "r"(1 + quarter) : "memory");
            tc_fence_after_sync();
            if (moves) {
                meet[half][r_local] = mx_tile;
                asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
                mx_tile = fmaxf(mx_tile, meet[half ^ 1][r_local]);
                asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
            }
            // m is the reference of the row's exponents; -inf + slack is -inf, so the first visible key sets it
            const float m_new = mx_tile > m + kRefSlack ? mx_tile : m;
            const float alpha = m_new == m ? 1.0f : ex2_approx(m - m_new);
            m = m_new;
            const float ref = m == -INFINITY ? 0.f : m;
            // the accumulator is rescaled only when some row of the warp moved its reference (the TMEM loads
            // and stores are warp-wide, so the decision is the warp's); P V of the previous tile must be
            // complete by then
            if (it > 0 && !__all_sync(0xffffffffu, alpha == 1.0f)) {
                ok = ok && mbar_wait<true>(&o_done[(it - 1) % kBufs], (it - 1) / kBufs & 1, abort, p.status, 7);
                __syncwarp();
                tc_fence_after_sync();
#pragma unroll 1
                for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 32) {
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
            // pass 2: weights (exp2 of -inf is 0), their sum, and P over the scores' columns
            const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), nref2 = pack_f32x2(-ref, -ref);
            uint64_t acc_a = pack_f32x2(0.f, 0.f), acc_b = acc_a;
            uint32_t packed[16];
#pragma unroll
            for (int i = 0; i < NK; i += 4) {
                float x0, x1, x2, x3;
                unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), scale2, nref2), x0, x1);
                unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3])), scale2, nref2), x2, x3);
                const float p0 = ex2_approx(x0), p1 = ex2_approx(x1), p2 = ex2_approx(x2), p3 = ex2_approx(x3);
                acc_a = add_f32x2(acc_a, pack_f32x2(p0, p1));
                acc_b = add_f32x2(acc_b, pack_f32x2(p2, p3));
                __nv_bfloat162 h0 = __floats2bfloat162_rn(p0, p1), h1 = __floats2bfloat162_rn(p2, p3);
                packed[i >> 1] = *reinterpret_cast<uint32_t*>(&h0);
                packed[(i >> 1) + 1] = *reinterpret_cast<uint32_t*>(&h1);
            }
            tmem_st_32x32b_x16(t_s + half * 16, packed);
            float s0, s1, s2, s3;
            unpack_f32x2(acc_a, s0, s1);
            unpack_f32x2(acc_b, s2, s3);
            l = l * alpha + ((s0 + s1) + (s2 + s3));
            // one arrival per warp: P is in TMEM for the tensor core to read (and O, if it was rescaled, too)
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        meet[half][r_local] = l;              // the row's sum of weights
        asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
        l = meet[0][r_local] + meet[1][r_local];
        if (ok && n_iter > 0) ok = mbar_wait<true>(&o_done[(n_iter - 1) % kBufs], (n_iter - 1) / kBufs & 1, abort, p.status, 8);
        tc_fence_after_sync();
        ok = __all_sync(0xffffffffu, ok);
        const bool have = ok && n_iter > 0;
        const size_t prow0 = ((size_t)slot * p.NKV + kvh) * BQ;
        // one share of the tile's keys: the sums as they are, with the reference they were taken against
        // (a share without a visible key, or one that gave up waiting, counts as nothing)
        if (shares > 1 && half == 0) {
            p.part_ml[(prow0 + r_local) * 2] = have ? m : -INFINITY;
            p.part_ml[(prow0 + r_local) * 2 + 1] = have ? l : 0.f;
        }
        if (have) {
            // 32 columns at a time go through 4 KB of shared memory of the warp's own (the queries and stages are done with), so that a store writes whole
            // rows' pieces of 128 (64) bytes.  Every lane takes part; only valid rows store.
            const float inv = shares > 1 ? 1.0f : l > 0.f ? 1.0f / l : 0.f;
            uint8_t* stage = smem + (warp - 4) * 4096;
            const long long own = shares > 1 ? (long long)(prow0 + r_local) * HD
                                : valid ? (long long)(qs0 + r / G) * p.NH * HD + (long long)(kvh * G + r % G) * HD : -1;
#pragma unroll 1
            for (int c = half * (HD / 2); c < (half + 1) * (HD / 2); c += 32) {
                uint32_t ov[32];
                __syncwarp();
                tmem_ld_32x32b_x32(t_out + c, ov);
                tmem_ld_wait();
                if (shares > 1) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<uint4*>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(ov[4 * j], ov[4 * j + 1], ov[4 * j + 2], ov[4 * j + 3]);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = i * 4 + (lane >> 3), j = lane & 7;
                        const long long at = __shfl_sync(0xffffffffu, own, row);
                        *reinterpret_cast<uint4*>(p.part_o + at + c + 4 * j) = *reinterpret_cast<const uint4*>(stage + row * 128 + ((j ^ (row & 7)) << 4));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(ov[8 * j + 2 * e]) * inv, __uint_as_float(ov[8 * j + 2 * e + 1]) * inv);
                            w[e] = *reinterpret_cast<uint32_t*>(&h);
                        }
                        *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ (lane >> 1 & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = i * 8 + (lane >> 2), j = lane & 3;
                        const long long at = __shfl_sync(0xffffffffu, own, row);
                        const uint4 v = *reinterpret_cast<const uint4*>(stage + row * 64 + ((j ^ (row >> 1 & 3)) << 4));
                        if (at >= 0) *reinterpret_cast<uint4*>(p.out + at + c + 8 * j) = v;
                    }
                }
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// Adds up the shares of the tiles whose keys were cut: a thread per (row, four neighbouring columns), 256 / (HD / 4)
// rows per CTA.  The shares are walked in their order, so the sum does not depend on timing.
//   M = max_z m_z;  o = sum_z 2^(m_z - M) o_z / sum_z 2^(m_z - M) l_z
constexpr int kMergeThreads = 256, kMaxShares = 32;
constexpr int kMergeRows = kMergeThreads / (HD / 4);             // rows per CTA
__global__ void __launch_bounds__(kMergeThreads)
attention_sm100_merge_kernel(const AttnTcParams p, const int32_t* __restrict__ merge_list) {
    forge::pdl_launch_dependents();
    forge::pdl_wait();
    const int mt = blockIdx.x / p.NKV, kvh = blockIdx.x % p.NKV;
    const int G = p.NH / p.NKV;
    const int s_req = merge_list[4 * mt], row0 = merge_list[4 * mt + 1], slot0 = merge_list[4 * mt + 2];
    const int shares = min(merge_list[4 * mt + 3], kMaxShares);
    const int qs0 = p.q_start[s_req], qlen = p.q_start[s_req + 1] - qs0;
    const int rows_here = min((BQ / G) * G, qlen * G - row0);
    const int r_local = blockIdx.y * kMergeRows + threadIdx.x / (HD / 4), c = (threadIdx.x % (HD / 4)) * 4;
    if (r_local >= rows_here) return;
    const size_t prow0 = ((size_t)slot0 * p.NKV + kvh) * BQ + r_local, pstep = (size_t)p.NKV * BQ;     // share z: prow0 + z * pstep
    float M = -INFINITY;
    for (int z = 0; z < shares; ++z) M = fmaxf(M, p.part_ml[(prow0 + z * pstep) * 2]);
    float L = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int z = 0; z < shares; ++z) {
        const size_t prow = prow0 + z * pstep;
        const float m_z = p.part_ml[prow * 2], l_z = p.part_ml[prow * 2 + 1];
        // a share without a visible key never wrote its sums
        const float w = m_z == -INFINITY ? 0.f : exp2f(m_z - M);
        const float4 v = w != 0.f ? *reinterpret_cast<const float4*>(p.part_o + prow * HD + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        L += w * l_z;
        acc.x += w * v.x; acc.y += w * v.y; acc.z += w * v.z; acc.w += w * v.w;
    }
    const float inv = L > 0.f ? 1.0f / L : 0.f;
    const int r = row0 + r_local;
    __nv_bfloat16* dst = p.out + (size_t)(qs0 + r / G) * p.NH * HD + (size_t)(kvh * G + r % G) * HD + c;
    __nv_bfloat162 h0 = __floats2bfloat162_rn(acc.x * inv, acc.y * inv), h1 = __floats2bfloat162_rn(acc.z * inv, acc.w * inv);
    *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<uint32_t*>(&h0), *reinterpret_cast<uint32_t*>(&h1));
}

}  // namespace

// q [T, NH*HD] bf16, kv cache [pages, 2, NKV, page_size, HD] bf16, out [T, NH*HD] bf16.  tile_req / tile_row0
// list tiles of (128 / G) * G query rows (rows = tokens * G); q_start / ctx_before as for forge_paged_attention_mma.
// tile_cut (or null) [num_tiles][3]: entry i works on share tile_cut[i][0] of tile_cut[i][1] equal shares of its tile's
// key tiles and, with more than one share, leaves its sums in slot tile_cut[i][2] + share of part_o [slots][NKV][128][HD]
// and part_ml [slots][NKV][128][2]; merge_list [num_merge][4] = (request, first row, first slot, shares) names the
// tiles to add up afterwards (at most 32 shares each).
extern "C" int forge_paged_attention_sm100(const void* q, const void* kv, void* out, const int32_t* block_table,
                                           const int32_t* tile_req, const int32_t* tile_row0, const int32_t* tile_cut,
                                           void* part_o, void* part_ml, const int32_t* merge_list, int num_merge,
                                           const int32_t* q_start,
                                           const int32_t* ctx_before, int* status, int num_tiles, int T, int num_pages,
                                           int NH, int NKV, int head_dim, int page_size, int max_pages, int window,
                                           float scale, cudaStream_t stream) {
    if (head_dim != HD) return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: this library was built for head_dim %d, got %d", HD, head_dim);
    if (NH <= 0 || NKV <= 0 || NH % NKV != 0 || NH / NKV > BQ)
        return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: %d query heads per kv head (at most 128)", NKV > 0 ? NH / NKV : 0);
    if (page_size < 8 || BKV % page_size != 0)
        return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: page size %d must be 8, 16, 32 or 64", page_size);
    if (!(scale > 0.f)) return forge::fail(FORGE_ERR_ARG, "paged_attention_sm100: scale %g must be positive", (double)scale);
    if (num_tiles < 0 || T <= 0 || num_pages <= 0 || max_pages <= 0)
        return forge::fail(FORGE_ERR_ARG, "paged_attention_sm100: bad sizes tiles=%d T=%d pages=%d", num_tiles, T, num_pages);
    if (num_merge < 0 || (num_merge > 0 && (!tile_cut || !part_o || !part_ml || !merge_list)))
        return forge::fail(FORGE_ERR_ARG, "paged_attention_sm100: %d tiles to add up need tile_cut, part_o, part_ml and merge_list", num_merge);
    if (num_tiles == 0) return FORGE_OK;
    const int G = NH / NKV;
    const char* err = nullptr;
    CUtensorMap tq, tkv;
    if (!bf16_q_map(q, T, NH, HD, BQ / G, G, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: q: %s", err);
    if (!bf16_kblock_map(kv, num_pages * 2 * NKV * page_size, HD, page_size, page_size == BKV ? KB : 1, &tkv, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: cache: %s", err);
    static forge::PerDeviceFlag configured_on;
    bool& configured = configured_on.current();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(paged_attention_sm100_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "paged_attention_sm100: %s", cudaGetErrorString(e));
        // the warpgroups trade registers inside what the CTA was given at launch; a build that gives less would wait
        // for registers that never come, so it is refused here
        cudaFuncAttributes attr;
        e = cudaFuncGetAttributes(&attr, paged_attention_sm100_kernel);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "paged_attention_sm100: %s", cudaGetErrorString(e));
        if (attr.numRegs * 3 < kRegsFew + 2 * kRegsMany)
            return forge::fail(FORGE_ERR_UNSUPPORTED, "paged_attention_sm100: built with %d registers per thread, needs %d",
                               attr.numRegs, (kRegsFew + 2 * kRegsMany + 2) / 3);
        configured = true;
    }
    AttnTcParams p{(__nv_bfloat16*)out, block_table, tile_req, tile_row0, tile_cut, (float*)part_o, (float*)part_ml,
                   q_start, ctx_before, NH, NKV, page_size, max_pages, window, scale * 1.4426950408889634f, status};
    int rc = forge::check_launch("paged_attention_sm100",
                                 forge::launch(paged_attention_sm100_kernel, dim3((unsigned)num_tiles * NKV), dim3(kThreads), kSmemBytes,
                                               stream, 1, tq, tkv, p));
    if (rc != FORGE_OK || num_merge == 0) return rc;
    return forge::check_launch("attention_sm100_merge",
                               forge::launch(attention_sm100_merge_kernel, dim3((unsigned)num_merge * NKV, BQ / kMergeRows), dim3(kMergeThreads), 0,
                                             stream, 1, p, merge_list));
}

extern "C" const char* forge_last_error() { return forge::error_buffer(); }

// (checks build) the bounds that this library's kernel tests page ids against
FORGE_DEFINE_CHECKS_ENTRY(attention_sm100)
