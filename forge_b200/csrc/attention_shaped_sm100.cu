// Prompt portions of two attentions on the 5th-generation tensor cores: attention over latent rows (attention_latent.cu) and
// attention with shaped scores (attention_scored.cu: one or two maps a head, distance term, cap, window, chunk, sink).  Both are, per CTA,
// up to 128 rows of queries over tiles of 64 keys with a two-term softmax weight:
//
//   S = Q K^T      tcgen05.mma M=128 N=64 per 16 channels, Q (all its channels) and the key blocks in shared memory, S in TMEM (two buffers)
//   softmax        256 threads, two a row with 32 of its scores each in registers, fp32; a weight becomes two bfloat16 numbers, its rounding and
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
// A third reading of the operands serves latent rows whose keys and values a product has spelled out for every head (forge_expanded_attention_sm100):
// they lie packed, request behind request, [rows, H, D + E], beside the rotated part [rows, R] that all heads share; a tile is 128 tokens of
// one head, the scores take D + R channels instead of C + R and the outputs E instead of C.
//
// Warps 0-3 copy keys, multiply P V, multiply Q K^T and copy values, warps 4-11 are the rows, two threads a row with 32 of a tile's keys each,
// which meet once a tile over the row's maximum; registers change hands with setmaxnreg where two CTAs share an SM.  Every wait is bounded.
#include "common.cuh"
#include "checks.cuh"
#include "scored_combine.cuh"
#include "sm100.cuh"

namespace {
using namespace sm100;

constexpr int BQ = 128, BKV = 64, kQkWarp = 2, kValueWarp = 3;
constexpr int kThreads = 384, kRowWarps = 8, NK = BKV / 2;      // four warps that run the copies and products, eight of rows; NK: a thread's keys of a tile
// two CTAs an SM: 65,536 / (2 x 384) registers a thread, dealt out anew between the three warpgroups
constexpr int kLaunchRegs = 80, kRegsFew = 48, kRegsMany = 96;
static_assert(kRegsFew + 2 * kRegsMany <= 3 * kLaunchRegs, "the warpgroups cannot hold more registers than the CTA was given");
constexpr int kQBlock = BQ * 128, kBlock = BKV * 128;          // bytes of 64 channels of the queries / of a tile of keys
constexpr int kMaxStages = 3, kBarBytes = 256, kSmemLimit = 227 * 1024 - 1024;      // (1 KB of it is the rows' meeting place)
constexpr int kSmemTwo = (228 * 1024 - 2 * 2048) / 2;          // of two CTAs an SM (1 KB of each is the system's, 1 KB the meeting place)
constexpr float kRefSlack = 8.0f;     // a row's reference exponent moves only when its maximum has grown by more than 2^8 (see attention_sm100.cu)
constexpr float kLog2e = 1.4426950408889634f;

struct ShapedParams {
    __nv_bfloat16* out;               // row t at out + t * out_ld, head h's values from h * E on (u == null)
    float* u;                         // fp32 [T, H, M, E], normalised (two maps)
    long long out_ld;
    const __nv_bfloat16* q;           // (q_tmem or packed) [T, H, q_channels]
    const int32_t* block_table;
    const int4* tiles;                // (first token, tokens, request, the first token's position)
    const float *r1, *r2, *sink;
    int H, heads, inner, M, D, E, VC; // heads: of a CTA; inner: CTAs of one tile (groups x maps x chunks of values)
    int q_channels;                   // channels of a query row that enter S
    int key_blocks, value_blocks;     // blocks of 64 channels of the two kinds
    int k_boxed, v_boxed;             // blocks that one copy of a tile of keys (values) brings: all, where a page holds a whole tile, else one
    int latent;                       // the value blocks are key blocks too
    const int32_t* row_start;         // (packed keys and values) a request's first row, else null
    const __nv_bfloat16 *kv, *kr;     // (packed) [rows, H, D + E] and [rows, q_channels - D]
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
// The products' descriptors as a low word that moves and a high word that does not: the one thread that issues them pays for every
// instruction between two of them (whole 64-bit descriptors worked out per product: 120 to 150 clocks each, where the tensor core needs 32).
// The whole warp walks the loop around them, with every operand the same in all lanes, and the instruction itself runs in the elected one
// (`leader`): operands that the compiler knows to be uniform come from uniform registers, while in a branch of one lane each has to be moved there
// first (160 clocks a product of the scores, 75 of the outputs).
// D[tmem] (+)= A[smem] . B[smem]^T
__device__ __forceinline__ void umma_ss(uint32_t leader, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
        "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
// D[tmem] (+)= A[tmem] . B[smem]^T: row r of A is lane r, 16 channels are eight columns of two bfloat16 numbers
__device__ __forceinline__ void umma_ts(uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// 4D tile load: c0 innermost (elements), then c1, c2, c3.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

__device__ __forceinline__ int first_visible(int pos, int window, int chunk) {
    int lo = 0;
    if (window > 0) lo = max(lo, pos - window + 1);
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    return lo;
}

typedef unsigned long long u64;
// two fp32 multiply-adds (or sums) in one instruction, each rounded as fmaf (or +) rounds
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
__device__ __forceinline__ u64 pair2(uint32_t lo, uint32_t hi) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
__device__ __forceinline__ float low2(u64 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high2(u64 v) { return __uint_as_float((uint32_t)(v >> 32)); }

// (Packed keys and values.)  A weight of 0 does not silence a number that is none: one among the values of a token reaches the tokens before it in its
// tile, up to 127 of them.  A row with such a result therefore looks whether a later token of its tile has such a value in these 32 columns, and if so adds
// its outputs up again over the keys that it sees, a thread on its own: time only where there is such a number.
__device__ __noinline__ void without_later_tokens(const ShapedParams& p, uint32_t columns, int head, int tok, int row0, int pos, int pos_last, float mult,
                                                  float ref, float inv) {
    const int R = p.q_channels - p.D, width = p.D + p.E;
    const size_t ld = (size_t)p.H * width;
    const __nv_bfloat16* q = p.q + ((size_t)tok * p.H + head) * p.q_channels;
    const __nv_bfloat16* kv = p.kv + row0 * ld + (size_t)head * width;
    const __nv_bfloat16* kr = p.kr + (size_t)row0 * R;
    auto low = [](uint32_t w) { return __uint_as_float(w << 16); };
    auto high = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
    auto dot = [&](const __nv_bfloat16* a, const __nv_bfloat16* b, int n, float sum) {
        for (int i = 0; i < n; i += 8) {
            const uint4 x = *reinterpret_cast<const uint4*>(a + i), y = *reinterpret_cast<const uint4*>(b + i);
            sum = fmaf(low(x.x), low(y.x), sum); sum = fmaf(high(x.x), high(y.x), sum); sum = fmaf(low(x.y), low(y.y), sum); sum = fmaf(high(x.y), high(y.y), sum);
            sum = fmaf(low(x.z), low(y.z), sum); sum = fmaf(high(x.z), high(y.z), sum); sum = fmaf(low(x.w), low(y.w), sum); sum = fmaf(high(x.w), high(y.w), sum);
        }
        return sum;
    };
    for (; columns != 0; columns &= columns - 1) {
        const int c = (__ffs(columns) - 1) * 32;
        bool none = false;
        for (int j = pos + 1; j <= pos_last && !none; ++j)
            for (int i = 0; i < 32; i += 2) {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(kv + j * ld + p.D + c + i);
                none |= !isfinite(low(w)) || !isfinite(high(w));
            }
        if (!none) continue;
        float acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
        for (int j = 0; j <= pos; ++j) {
            const float s = dot(q + p.D, kr + (size_t)j * R, R, dot(q, kv + j * ld, p.D, 0.f)), x = ex2(fmaf(s, mult, -ref));
            const uint32_t* v = reinterpret_cast<const uint32_t*>(kv + j * ld + p.D + c);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t w = v[i];
                acc[2 * i] = fmaf(x, low(w), acc[2 * i]);
                acc[2 * i + 1] = fmaf(x, high(w), acc[2 * i + 1]);
            }
        }
        uint32_t* dst = reinterpret_cast<uint32_t*>(p.out + (size_t)tok * p.out_ld + (size_t)head * p.E + c);
#pragma unroll
        for (int i = 0; i < 16; ++i) dst[i] = pack_bf16(acc[2 * i] * inv, acc[2 * i + 1] * inv);
    }
}

template <bool SHAPED, int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM)
shaped_attention_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                              const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ ShapedParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ float meet[2][BQ];                                   // [half]: what a row's two threads tell each other
    const int tile = blockIdx.x / p.inner;
    const int4 what = p.tiles[tile];
    const int t0 = what.x, nq = what.y;
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
        mbar_init(q_ready, kRowWarps);
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&p_ready[b], kRowWarps);
            mbar_init(&o_done[b], 1);
        }
        mbar_fence_init();
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
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

    // (the step's tiles and tables were written before its first kernel started)
    const int req = what.z, pos0 = what.w, pos_last = pos0 + nq - 1;
    const int t_begin = first_visible(pos0, p.window, p.chunk) / BKV, t_end = pos_last / BKV + 1, n_iter = t_end - t_begin;
    const int seen_from = first_visible(pos0, p.window, p.chunk);
    forge::pdl_wait();

    if (warp < 4) {
    if (PER_SM > 1) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsFew));
    if (warp == 0 || warp == kValueWarp) {
        // ------------------------------------------------------------------ copies: keys (and the queries), values
        // (a warp each, and nothing between two copies that could be worked out ahead: these warps get an instruction in every ten clocks or so
        // beside the rows, and a round of 150 instructions for both kinds was longer than the products and weights of a tile)
        const int32_t* table = p.block_table + (size_t)req * p.max_pages;
        const int ppt = p.page_size >= BKV ? 1 : BKV / p.page_size;       // boxes a tile and block
        const int page_shift = 31 - __clz(p.page_size), page_mask = p.page_size > BKV ? p.page_size - 1 : 0;     // (a power of two)
        const int k_col0 = p.latent ? 0 : mp * p.D;
        const int skip = p.latent ? vc * p.value_blocks : 1 << 20;        // key block i stands for channel block i, or i + value_blocks from here on
        const bool packed = p.row_start != nullptr;
        // key blocks that are the other chunk's value blocks (packed: the head's own blocks of keys): they come like them
        const int others = p.latent ? (chunks - 1) * p.value_blocks : packed ? p.D / 64 : 0;
        const int head_blocks = packed ? group * ((p.D + p.E) / 64) : 0, row0 = packed ? p.row_start[req] : group * p.page_size;
        const int rounds = __shfl_sync(0xffffffffu, n_iter, 0);
        // one lane a box of rows: its page, or -1 where no token of the tile sees a key.  Asked for a tile ahead: a trip to the table takes longer than
        // the products of a small tile.  A box without a page (behind the window, beyond the request, or none in the table) is copied all the same, from before
        // the cache's first page: the copy fills zeros in.  What the slot held before may be no number, which a weight of 0 would not silence
        auto page_of = [&](int it) {
            int page = -1;
            if (lane < ppt && it < rounds) {
                const int j = (t_begin + it) * BKV + lane * p.box_rows, idx = j >> page_shift;
                if (packed) page = 0;                                     // (rows behind the request's are another's, or fill: masked, and cleared below)
                else if (j <= pos_last && j + p.box_rows > seen_from && idx < p.max_pages) page = table[idx];
            }
            return page;
        };
        const uint32_t box_bytes = p.box_rows * 128;
        int st = 0, ph = 0, next_page = -1;
        if (warp == 0) {
            if (lane == 0) {
                mbar_arrive_expect_tx(q_full, q_blocks * q_rows * 128);
                for (int b = 0; b < q_blocks; ++b)
                    tma_load_3d(q_s + b * kQBlock, &tmap_q, q_full, k_col0 + (p.q_tmem && b >= skip ? b + p.value_blocks : b) * 64, group * p.heads, t0);
            }
            next_page = page_of(0);
            if (p.key_blocks > 0)
            for (int it = 0; it < rounds; ++it) {
                const int j0 = (t_begin + it) * BKV;
                int page = next_page;
                next_page = page_of(it + 1);
                if (page >= 0 && !packed && !FORGE_PAGE_OK(page)) page = -1;
                const int row = packed ? row0 + j0 : row0 + (j0 & page_mask);
                if (!warp_wait<true>(&k_empty[st], ph ^ 1, abort, p.status, 1)) break;
                if (lane == 0) mbar_arrive_expect_tx(&k_full[st], p.key_blocks * kBlock);
                __syncwarp();
                if (lane < ppt) {
                    uint8_t* dst = k_s + st * p.key_blocks * kBlock + lane * box_bytes;
                    for (int b = 0; b < others; b += p.v_boxed)
                        tma_load_4d(dst + b * kBlock, &tmap_v, &k_full[st], 0, row, head_blocks + (b < skip ? b : b + p.value_blocks), page);
                    for (int b = others; b < p.key_blocks; b += p.k_boxed) {
                        if (p.latent || packed) tma_load_4d(dst + b * kBlock, &tmap_k, &k_full[st], (p.latent ? p.E : 0) + (b - others) * 64, row, 0, page);
                        else tma_load_4d(dst + b * kBlock, &tmap_k, &k_full[st], 0, row, mp * p.key_blocks + b, page);
                    }
                }
                if (++st == p.stages) { st = 0; ph ^= 1; }
            }
        } else {
            const int block0 = head_blocks + (packed ? others : 0) + vc * p.value_blocks;
            int tail_ph = 0;
            next_page = page_of(0);
            for (int it = 0; it < rounds; ++it) {
                const int j0 = (t_begin + it) * BKV;
                int page = next_page;
                next_page = page_of(it + 1);
                if (page >= 0 && !packed && !FORGE_PAGE_OK(page)) page = -1;
                const int row = packed ? row0 + j0 : row0 + (j0 & page_mask);
                const bool last = j0 + BKV - 1 > pos_last;                // rows behind the last token: cleared below
                uint64_t* landed = last ? tail : &v_full[st];
                uint8_t* vd = v_s + st * p.value_blocks * kBlock;
                if (!warp_wait<true>(&v_empty[st], ph ^ 1, abort, p.status, 2)) break;
                if (lane == 0) mbar_arrive_expect_tx(landed, p.value_blocks * kBlock);
                __syncwarp();
                if (lane < ppt)
                    for (int b = 0; b < p.value_blocks; b += p.v_boxed)
                        tma_load_4d(vd + b * kBlock + lane * box_bytes, &tmap_v, landed, 0, row, block0 + b, page);
                if (last) {
                    // what lies in the cache behind the last token counts as zeros: a weight of 0 would not silence a NaN there
                    if (!warp_wait<true>(tail, tail_ph, abort, p.status, 3)) break;
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
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ P V
        const uint32_t leader = elect_one(), idesc = umma_idesc_bf16_f32_bmn(BQ, p.VC), v_step = p.value_blocks * kBlock >> 4;
        const uint64_t vdesc = umma_desc_mn_sw128(smem_u32(v_s), kBlock);
        const uint32_t v_lo0 = (uint32_t)vdesc, hi = (uint32_t)(vdesc >> 32), o_at = __shfl_sync(0xffffffffu, tmem_o, 0);
        const int rounds = __shfl_sync(0xffffffffu, n_iter, 0);
        int st = 0, ph = 0;
        for (int it = 0; it < rounds; ++it) {
            const int b = it & 1;
            if (!warp_wait<true>(&v_full[st], ph, abort, p.status, 4)) break;
            if (!warp_wait<true>(&p_ready[b], (it >> 1) & 1, abort, p.status, 5)) break;
            tc_fence_after_sync();
            const uint32_t v_lo = v_lo0 + st * v_step, pt = o_at - 2 * BKV + b * BKV;
#pragma unroll
            for (int k = 0; k < BKV / 16; ++k) {
                umma_ts(leader, o_at, pt + 32 + k * 8, v_lo + k * (2048 >> 4), hi, idesc, k > 0 ? 1 : (uint32_t)(it > 0));
                umma_ts(leader, o_at, pt + k * 8, v_lo + k * (2048 >> 4), hi, idesc, 1);
            }
            umma_commit_by(leader, &o_done[b]);
            umma_commit_by(leader, &v_empty[st]);
            if (++st == p.stages) { st = 0; ph ^= 1; }
        }
    } else if (warp == kQkWarp) {
        // ------------------------------------------------------------------ Q K^T
        const uint32_t leader = elect_one(), idesc = umma_idesc_bf16_f32(BQ, BKV);
        const int skip = p.latent ? vc * p.value_blocks : 1 << 20;
        const uint64_t qdesc = umma_desc_k_sw128(smem_u32(q_s));
        const uint32_t q_lo = (uint32_t)qdesc, hi = (uint32_t)(qdesc >> 32);
        const uint32_t k_lo0 = (uint32_t)umma_desc_k_sw128(smem_u32(k_s)), v_lo0 = (uint32_t)umma_desc_k_sw128(smem_u32(v_s));
        const uint32_t k_step = p.key_blocks * kBlock >> 4, v_step = p.value_blocks * kBlock >> 4;
        const int part_steps = p.q_channels % 64 / 16, part_block = part_steps ? p.q_channels / 64 : -1;
        const uint32_t s_at = __shfl_sync(0xffffffffu, tmem_base, 0);
        const int rounds = __shfl_sync(0xffffffffu, n_iter, 0);
        int st = 0, ph = 0;
        if (warp_wait<true>(q_full, 0, abort, p.status, 6))
        for (int it = 0; it < rounds; ++it) {
            const int b = it & 1;
            // (the scores' buffer holds the weights of tile it - 2 until its P V is done)
            if (it >= 2 && !warp_wait<true>(&o_done[b], ((it - 2) >> 1) & 1, abort, p.status, 7)) break;
            const uint32_t ds = s_at + b * BKV;
            uint32_t add = 0;
            // key block at w_lo against the query's channel block at a_lo
            auto product = [&](uint32_t a_lo, uint32_t w_lo, int channel_block) {
                if (channel_block != part_block) {
                    umma_ss(leader, ds, a_lo, w_lo, hi, idesc, add);
#pragma unroll
                    for (int k = 1; k < 4; ++k) umma_ss(leader, ds, a_lo + k * 2, w_lo + k * 2, hi, idesc, 1);
                } else {                                              // the last channels do not fill a block
                    for (int k = 0; k < part_steps; ++k) umma_ss(leader, ds, a_lo + k * 2, w_lo + k * 2, hi, idesc, add | (uint32_t)(k > 0));
                }
                add = 1;
            };
            if (p.key_blocks > 0) {
                if (!warp_wait<true>(&k_full[st], ph, abort, p.status, 8)) break;
                tc_fence_after_sync();
                const uint32_t w_lo = k_lo0 + st * k_step;
                for (int i = 0; i < p.key_blocks; ++i) {
                    const int channel_block = i < skip ? i : i + p.value_blocks;
                    product(q_lo + (p.q_tmem ? i : channel_block) * (kQBlock >> 4), w_lo + i * (kBlock >> 4), channel_block);
                }
                umma_commit_by(leader, &k_empty[st]);
            }
            if (p.latent) {
                if (it == 0 && p.q_tmem && !warp_wait<true>(q_ready, 0, abort, p.status, 13)) break;
                if (!warp_wait<true>(&v_full[st], ph, abort, p.status, 9)) break;
                tc_fence_after_sync();
                const uint32_t w_lo = v_lo0 + st * v_step;
                if (p.q_tmem) {
                    for (int i = 0; i < p.value_blocks; ++i) {
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_ts(leader, ds, s_at + 2 * BKV + p.VC + i * 32 + k * 8, w_lo + i * (kBlock >> 4) + k * 2, hi, idesc, k > 0 ? 1 : add);
                        add = 1;
                    }
                } else {
                    for (int i = 0; i < p.value_blocks; ++i) product(q_lo + (skip + i) * (kQBlock >> 4), w_lo + i * (kBlock >> 4), skip + i);
                }
            }
            umma_commit_by(leader, &s_full[b]);
            if (++st == p.stages) { st = 0; ph ^= 1; }
        }
    }
    } else {
        // ------------------------------------------------------------------ the rows (warps 4..11)
        if (PER_SM > 1) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMany));
        const int half = (warp - 4) >> 2;
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
            const int share = p.VC / 2;
            for (int c = half * share; c < (half + 1) * share; c += 64) {
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
        // (a wait that ran out lets the loop go on without waiting: the two threads of a row have to meet in every round)
        for (int it = 0; it < n_iter; ++it) {
            const int j0 = (t_begin + it) * BKV + half * NK, b = it & 1;
            const uint32_t t_s = t_lane + b * BKV;
            ok = ok && mbar_wait<true>(&s_full[b], (it >> 1) & 1, abort, p.status, 10);
            __syncwarp();
            tc_fence_after_sync();
            uint32_t sv[NK];
            tmem_ld_32x32b_x32(t_s + half * NK, sv);
            tmem_ld_wait();
            // (a row that stands for no token may hold any number: nobody reads what comes of it)
            const bool need_mask = valid && (j0 + NK - 1 > pos || j0 < see);
            if (SHAPED) {                     // in units of log2 e, shaped, from here on
#pragma unroll
                for (int i = 0; i < NK; ++i) {
                    float s = __uint_as_float(sv[i]);
                    s = p.softcap > 0.f ? cap_out * tanh_fast(s * cap_in) : s * sl2;
                    if (p.r1) s -= r1v * __log2f(fmaf(r2v, (float)max(pos - j0 - i, 0), 1.0f));
                    sv[i] = __float_as_uint(s);
                }
            }
            if (need_mask) {
#pragma unroll
                for (int i = 0; i < NK; ++i) {
                    const int j = j0 + i;
                    if (!(j <= pos && j >= see)) sv[i] = __float_as_uint(-INFINITY);
                }
            }
            float a0 = -INFINITY, a1 = -INFINITY;
#pragma unroll
            for (int i = 0; i < NK; i += 4) {
                a0 = max3(a0, __uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
                a1 = max3(a1, __uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3]));
            }
            const float mult = SHAPED ? 1.0f : sl2;
            float top = fmaxf(a0, a1) * mult;
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
                : "=r"(moves) : "f"(top), "f"(m + kRefSlack), "r"(1 + quarter) : "memory");
            tc_fence_after_sync();
            if (moves) {
                meet[half][r] = top;
                asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
                top = fmaxf(top, meet[half ^ 1][r]);
                asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
            }
            const float m_new = top > m + kRefSlack ? top : m;            // (-inf + slack is -inf: the first visible key sets it)
            const float alpha = m_new == m ? 1.0f : ex2(m - m_new);
            m = m_new;
            const float ref = m == -INFINITY ? 0.f : m;
            // O is rescaled only when some row of the warp moved its reference; P V of the tile before must be complete by then
            if (it > 0 && !__all_sync(0xffffffffu, alpha == 1.0f)) {
                ok = ok && mbar_wait<true>(&o_done[b ^ 1], ((it - 1) >> 1) & 1, abort, p.status, 11);
                __syncwarp();
                tc_fence_after_sync();
                const int share = p.VC / 2;
                for (int c = half * share; c < (half + 1) * share; c += 32) {
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
            u64 s01 = 0, s23 = 0;
            const u64 mult2 = pair2(__float_as_uint(mult), __float_as_uint(mult)), ref2 = pair2(__float_as_uint(-ref), __float_as_uint(-ref));
            const u64 minus2 = pair2(0xbf800000u, 0xbf800000u);
            {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < NK; i += 4) {
                    const u64 x01 = fma2(pair2(sv[i], sv[i + 1]), mult2, ref2), x23 = fma2(pair2(sv[i + 2], sv[i + 3]), mult2, ref2);
                    const float p0 = ex2(low2(x01)), p1 = ex2(high2(x01)), p2 = ex2(low2(x23)), p3 = ex2(high2(x23));
                    const u64 p01 = pair2(__float_as_uint(p0), __float_as_uint(p1)), p23 = pair2(__float_as_uint(p2), __float_as_uint(p3));
                    s01 = add2(s01, p01);
                    s23 = add2(s23, p23);
                    const uint32_t h01 = pack_bf16(p0, p1), h23 = pack_bf16(p2, p3);
                    hi[i / 2] = h01;
                    hi[i / 2 + 1] = h23;
                    const u64 l01 = fma2(pair2(h01 << 16, h01 & 0xffff0000u), minus2, p01), l23 = fma2(pair2(h23 << 16, h23 & 0xffff0000u), minus2, p23);
                    lo[i / 2] = pack_bf16(low2(l01), high2(l01));
                    lo[i / 2 + 1] = pack_bf16(low2(l23), high2(l23));
                }
                tmem_st_32x32b_x16(t_s + half * 16, hi);
                tmem_st_32x32b_x16(t_s + 32 + half * 16, lo);
            }
            l = l * alpha + ((low2(s01) + high2(s01)) + (low2(s23) + high2(s23)));
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[b]);
        }
        meet[half][r] = l;                    // the row's sum of weights
        asm volatile("barrier.cta.sync.aligned %0, 64;" ::"r"(1 + quarter) : "memory");
        l = meet[0][r] + meet[1][r];
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
            // 32 columns at a time go through 4 KB of shared memory of the warp's own (the queries and stages are done with), so that a store writes whole
            // rows' pieces of 128 (64) bytes: a row a thread, straight from the registers, took 2.9 to 4.3 us a CTA.  Every lane takes part; only valid
            // rows store.
            uint8_t* stage = smem + (warp - 4) * 4096;
            const long long own = !valid ? -1 : v0 + (p.u != nullptr ? (((long long)tok * p.H + head) * p.M + mp) * p.E : (long long)tok * p.out_ld + (long long)head * p.E);
            const int share = p.VC / 2;
            uint32_t odd = 0;                            // the 32 columns (a bit each) among whose results are numbers that are none
            for (int c = half * share; c < (half + 1) * share; c += 32) {
                uint32_t ov[32];
                __syncwarp();
                tmem_ld_32x32b_x32(t_out + c, ov);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * inv);
                if (!SHAPED && p.row_start != nullptr) {
                    float z = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; ++i) z = fmaf(__uint_as_float(ov[i]), 0.f, z);
                    if (z != 0.f) odd |= 1u << (c >> 5);
                }
                if (p.u != nullptr) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<uint4*>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(ov[4 * j], ov[4 * j + 1], ov[4 * j + 2], ov[4 * j + 3]);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int row = i * 4 + (lane >> 3), j = lane & 7;
                        const long long at = __shfl_sync(0xffffffffu, own, row);
                        const float4 v = *reinterpret_cast<const float4*>(stage + row * 128 + ((j ^ (row & 7)) << 4));
                        if (at >= 0) *reinterpret_cast<float4*>(p.u + at + c + 4 * j) = v;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) w[e] = pack_bf16(__uint_as_float(ov[8 * j + 2 * e]), __uint_as_float(ov[8 * j + 2 * e + 1]));
                        *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ (lane >> 1 & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = i * 8 + (lane >> 2), j = lane & 3;
                        const long long at = __shfl_sync(0xffffffffu, own, row);
                        const uint4 v = *reinterpret_cast<const uint4*>(stage + row * 64 + ((j ^ (row >> 1 & 3)) << 4));
                        if (at < 0) continue;
                        __nv_bfloat16* dst = p.out + at + c + 8 * j;
                        if (p.vec_out) {
                            *reinterpret_cast<uint4*>(dst) = v;
                        } else {
                            uint32_t* d = reinterpret_cast<uint32_t*>(dst);
                            d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
                        }
                    }
                }
            }
            if (!SHAPED && p.row_start != nullptr) {     // (a sum of weights that is none: a key or a query is, and the result what it has to be)
                __syncwarp();
                if (odd != 0 && valid && isfinite(l)) without_later_tokens(p, odd, head, tok, p.row_start[req], pos, pos_last, sl2, m == -INFINITY ? 0.f : m, inv);
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

// A bf16 tensor of three or four dimensions read in boxes of 64 x b1 x b2 (x b3) with 128-byte swizzle; strides in elements.
bool tensor_map(const void* ptr, int rank, const unsigned long long (&d)[4], const unsigned long long (&stride)[3], const int (&b)[4], CUtensorMap* out, const char** err) {
    auto fn = encode_fn();
    if (!fn) { *err = "cuTensorMapEncodeTiled is not available from the driver"; return false; }
    cuuint64_t dims[4], strides[3];
    cuuint32_t box[4], estr[4] = {1u, 1u, 1u, 1u};
    for (int i = 0; i < 4; ++i) { dims[i] = d[i]; box[i] = (cuuint32_t)b[i]; }
    for (int i = 0; i < 3; ++i) strides[i] = stride[i] * 2;
    bool aligned = (reinterpret_cast<uintptr_t>(ptr) & 15) == 0;
    for (int i = 0; i + 1 < rank; ++i) aligned = aligned && strides[i] % 16 == 0;
    if (!aligned) { *err = "TMA needs 16-byte aligned rows"; return false; }
    if (fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
        *err = "cuTensorMapEncodeTiled failed";
        return false;
    }
    return true;
}
// queries [T, heads, channels] in boxes of 64 channels of b1 heads of b2 tokens
bool query_map(const void* ptr, int channels, int heads, int T, int b1, int b2, CUtensorMap* out, const char** err) {
    return tensor_map(ptr, 3, {(unsigned long long)channels, (unsigned long long)heads, (unsigned long long)T, 1},
                      {(unsigned long long)channels, (unsigned long long)heads * channels, 0}, {64, b1, b2, 1}, out, err);
}
// rows of `channels` numbers, `pitch` apart, seen as blocks of 64: one box is `rows` rows of `blocks` neighbouring blocks of a page, and lands
// as `blocks` tiles one after the other.  An SM's copies complete about one per 0.3 us whatever their size, so a tile is one copy where a
// page holds it (latent of 512 + 64 channels: nine copies of 8 KB a tile took 5,300 clocks).
bool block_map(const void* ptr, int channels, int pitch, int rows, int pages, long long page_stride, int box_rows, int blocks, CUtensorMap* out, const char** err) {
    return tensor_map(ptr, 4, {64, (unsigned long long)rows, (unsigned long long)(channels / 64), (unsigned long long)pages},
                      {(unsigned long long)pitch, 64, (unsigned long long)page_stride}, {64, box_rows, blocks, 1}, out, err);
}

bool pages_fit(int page_size) { return page_size >= 8 && (page_size & (page_size - 1)) == 0 && page_size <= 65536; }

size_t smem_bytes(int q_blocks, int blocks, int stages) { return (size_t)q_blocks * kQBlock + (size_t)stages * blocks * kBlock + kBarBytes + 1024; }

// value columns of a CTA: all up to 256, else chunks of 256 (0: not taken)
int value_columns(int E) { return E % 64 ? 0 : E <= 256 ? E : E % 256 ? 0 : 256; }

template <bool SHAPED, int PER_SM>
int launch_one(const char* what, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const ShapedParams& p, size_t smem, int num_tiles,
               cudaStream_t stream) {
    auto* kernel = shaped_attention_sm100_kernel<SHAPED, PER_SM>;
    static forge::PerDeviceFlag configured_on;
    bool& configured = configured_on.current();
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
        // the warpgroups trade registers inside what the CTA was given at launch: a build that gives less is refused
        cudaFuncAttributes attr;
        e = cudaFuncGetAttributes(&attr, kernel);
        if (e != cudaSuccess) return forge::fail(FORGE_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
        if (PER_SM > 1 && attr.numRegs * 3 < kRegsFew + 2 * kRegsMany)
            return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: built with %d registers per thread, needs %d", what, attr.numRegs, (kRegsFew + 2 * kRegsMany + 2) / 3);
        configured = true;
    }
    return forge::check_launch(what, forge::launch(kernel, dim3((unsigned)num_tiles * p.inner), dim3(kThreads), smem, stream, 1, tq, tk, tv, p));
}

template <bool SHAPED>
int launch(const char* what, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, ShapedParams p, int num_tiles, cudaStream_t stream) {
    int q_blocks = (p.q_channels + 63) / 64;
    const int blocks = p.key_blocks + p.value_blocks;
    // where the queries leave room for one tile of rows, those that meet the value blocks go to TMEM if it has the columns
    if (p.latent && smem_bytes(q_blocks, blocks, 2) > kSmemLimit && 2 * BKV + p.VC + p.value_blocks * 32 <= 512 && ((uintptr_t)p.q & 15) == 0 && p.D % 8 == 0) {
        p.q_tmem = 1;
        q_blocks -= p.value_blocks;
    }
    p.stages = kMaxStages;
    while (p.stages > 1 && smem_bytes(q_blocks, blocks, p.stages) > kSmemLimit) --p.stages;
    // Two CTAs an SM with fewer stages beat one with more where there are CTAs for both (one map, heads of 128 and values of 128, 2,048 tokens: 80.9 ->
    // 58.9 us; 128 + 64 channels packed, which leaves one stage each, 1,536 tokens: 52.7 -> 39.5); where every CTA has an SM of its own the stages win
    // (100 tokens behind 1,000: 24.8 us against 31.1).
    if ((long long)num_tiles * p.inner > forge::sm_count() && 2 * BKV + p.VC <= 256 && smem_bytes(q_blocks, blocks, 1) <= kSmemTwo)
        while (smem_bytes(q_blocks, blocks, p.stages) > kSmemTwo) --p.stages;
    const size_t smem = smem_bytes(q_blocks, blocks, p.stages);
    if (smem > kSmemLimit) return forge::fail(FORGE_ERR_UNSUPPORTED, "%s: queries of %d channels", what, p.q_channels);
    p.tmem_cols = 2 * BKV + p.VC + (p.q_tmem ? p.value_blocks * 32 : 0) <= 256 ? 256 : 512;
    p.box_rows = p.page_size < BKV ? p.page_size : BKV;
    // one CTA an SM, by its tensor memory or its shared memory, or two
    const bool alone = p.tmem_cols > 256 || smem > kSmemTwo;
    return alone ? launch_one<SHAPED, 1>(what, tq, tk, tv, p, smem, num_tiles, stream) : launch_one<SHAPED, 2>(what, tq, tk, tv, p, smem, num_tiles, stream);
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

// q bf16 [T, H, C+R]; cache: pages of page_size rows of C+R; out bf16 [T, H, C].  tiles int32 [num_tiles, 4]: up to 128 / H tokens of one
// request each (first token, tokens, request, the first token's position), the first to run first.  window, sink as for forge_latent_attention_mma.  status: bit 1 is raised where a wait ran out.
extern "C" int forge_latent_attention_sm100(const void* q, const void* cache, const int32_t* block_table, const int32_t* tiles, void* out, int* status, int T,
                                            int num_tiles, int num_pages, int H, int C, int R, int page_size, int max_pages, float scale, int window,
                                            const float* sink, cudaStream_t stream) {
    if (!forge_latent_sm100_supports(H, C, R, page_size)) return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: H=%d C=%d R=%d page=%d", H, C, R, page_size);
    if (T < 0 || num_tiles < 0 || num_pages <= 0 || max_pages <= 0 || !tiles || ((uintptr_t)tiles & 15) || !(scale > 0.f))
        return forge::fail(FORGE_ERR_ARG, "latent_attention_sm100: bad arguments");
    if (T == 0 || num_tiles == 0) return FORGE_OK;
    const int KD = C + R, VC = value_columns(C), chunks = C / VC;
    const char* err = nullptr;
    CUtensorMap tq, tk, tv;
    const int rows = page_size < BKV ? page_size : BKV, v_boxed = rows == BKV ? VC / 64 : 1;
    if (!query_map(q, KD, H, T, H, BQ / H, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: q: %s", err);
    const unsigned long long pages = (unsigned long long)num_pages, page = (unsigned long long)page_size * KD;
    if (!block_map(cache, C, KD, page_size, num_pages, (long long)page, rows, v_boxed, &tv, &err) ||
        !tensor_map(cache, 4, {(unsigned long long)KD, (unsigned long long)page_size, 1, pages}, {(unsigned long long)KD, page, page}, {64, rows, 1, 1}, &tk, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "latent_attention_sm100: cache: %s", err);
    ShapedParams p{};
    p.out = (__nv_bfloat16*)out; p.out_ld = (long long)H * C;
    p.block_table = block_table; p.tiles = reinterpret_cast<const int4*>(tiles);
    p.sink = sink; p.q = (const __nv_bfloat16*)q;
    p.H = p.heads = H; p.inner = chunks; p.M = 1; p.D = KD; p.E = C; p.VC = VC;
    p.q_channels = KD; p.value_blocks = VC / 64; p.key_blocks = (KD + 63) / 64 - p.value_blocks; p.latent = 1;
    p.k_boxed = 1; p.v_boxed = v_boxed;
    p.page_size = page_size; p.max_pages = max_pages; p.window = window;
    p.vec_out = ((uintptr_t)out & 15) == 0; p.scale = scale; p.out_scale = 1.0f; p.status = status;
    return launch<false>("latent_attention_sm100", tq, tk, tv, p, num_tiles, stream);
}

// 1 if the kernel takes keys and values of H heads spelled out: D unrotated channels and E values a head (multiples of 64, D up to 256, E up
// to 256), R rotated ones (a multiple of 16).
extern "C" int forge_expanded_sm100_supports(int H, int D, int R, int E) {
    const int q_blocks = (D + R + 63) / 64;
    return (H > 0 && D > 0 && D % 64 == 0 && D <= 256 && R > 0 && R % 16 == 0 && R <= 128 && E > 0 && E % 64 == 0 && E <= 256 &&
            smem_bytes(q_blocks, q_blocks + E / 64, 1) <= kSmemLimit) ? 1 : 0;
}

// q bf16 [T, H, D+R]; kv bf16 [rows, H, D+E]: keys and values of every request of the step, position by position, request s from row row_start[s]
// on; kr bf16 [rows, R]; out bf16, rows of out_ld, head h's E values from h * E on.  Tiles of up to 128 tokens; the rest as above.
extern "C" int forge_expanded_attention_sm100(const void* q, const void* kv, const void* kr, const int32_t* row_start, const int32_t* tiles, void* out, int* status, int T,
                                              int num_tiles, int rows, int H, int D, int R, int E, float scale, const float* sink, long long out_ld,
                                              cudaStream_t stream) {
    if (!forge_expanded_sm100_supports(H, D, R, E)) return forge::fail(FORGE_ERR_UNSUPPORTED, "expanded_attention_sm100: H=%d D=%d R=%d E=%d", H, D, R, E);
    if (T < 0 || num_tiles < 0 || rows <= 0 || !row_start || !tiles || ((uintptr_t)tiles & 15) || !(scale > 0.f) || out_ld < (long long)H * E || (out_ld & 1) ||
        ((uintptr_t)out & 3))
        return forge::fail(FORGE_ERR_ARG, "expanded_attention_sm100: bad arguments");
    if (T == 0 || num_tiles == 0) return FORGE_OK;
    const int width = H * (D + E), boxed = D == E ? E / 64 : 1;
    const char* err = nullptr;
    CUtensorMap tq, tk, tv;
    if (!query_map(q, D + R, H, T, 1, BQ, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "expanded_attention_sm100: q: %s", err);
    const unsigned long long n = (unsigned long long)rows;
    if (!block_map(kv, width, width, rows, 1, (long long)n * width, BKV, boxed, &tv, &err) ||
        !tensor_map(kr, 4, {(unsigned long long)R, n, 1, 1}, {(unsigned long long)R, n * R, n * R}, {64, BKV, 1, 1}, &tk, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "expanded_attention_sm100: keys and values: %s", err);
    ShapedParams p{};
    p.out = (__nv_bfloat16*)out; p.out_ld = out_ld;
    p.tiles = reinterpret_cast<const int4*>(tiles); p.row_start = row_start;
    p.sink = sink;
    p.H = H; p.heads = 1; p.inner = H; p.M = 1; p.D = D; p.E = E; p.VC = E;
    p.q_channels = D + R; p.key_blocks = (D + R + 63) / 64; p.value_blocks = E / 64; p.latent = 0;
    p.q = (const __nv_bfloat16*)q; p.kv = (const __nv_bfloat16*)kv; p.kr = (const __nv_bfloat16*)kr;
    p.k_boxed = 1; p.v_boxed = boxed;
    p.page_size = BKV; p.max_pages = 1;
    p.vec_out = ((uintptr_t)out & 15) == 0 && out_ld % 8 == 0; p.scale = scale; p.out_scale = 1.0f; p.status = status;
    return launch<false>("expanded_attention_sm100", tq, tk, tv, p, num_tiles, stream);
}

// q bf16 [T, H, M, D]; cache pages of page_stride numbers, [G, page_size, M*D] keys then [G, page_size, E] values; one map: out bf16, rows of
// out_ld, times out_scale; two: the maps' outputs go through u fp32 [T, H, 2, E], and a second kernel makes (a_1 - lambda a_2) / its root mean square
// * post * out_scale of them.  The rest as for forge_scored_attention_mma; tiles of up to 128 / (H/G) tokens.
extern "C" int forge_scored_attention_sm100(const void* q, const void* cache, const int32_t* block_table, const int32_t* tiles, const float* r1, const float* r2,
                                            float* u, void* out, int* status, int T, int num_tiles, int num_pages, int H, int G, int M, int D, int E,
                                            int page_size, long long page_stride, int max_pages, float scale, float lambda, float post, float eps, float out_scale,
                                            long long out_ld, int window, int chunk, float softcap, const float* sink, cudaStream_t stream) {
    if (!forge_scored_sm100_supports(H, G, M, D, E, page_size))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: H=%d G=%d M=%d D=%d E=%d page=%d", H, G, M, D, E, page_size);
    if (T < 0 || num_tiles < 0 || num_pages <= 0 || max_pages <= 0 || !tiles || ((uintptr_t)tiles & 15) || !(scale > 0.f) || (r1 == nullptr) != (r2 == nullptr) ||
        (M == 2 && !u) || !out || (sink && M != 1) || window < 0 || chunk < 0 || softcap < 0.f ||
        out_ld < (long long)H * E || (out_ld & 1) || page_stride < (long long)G * page_size * (M * D + E))
        return forge::fail(FORGE_ERR_ARG, "scored_attention_sm100: bad arguments");
    if (T == 0 || num_tiles == 0) return FORGE_OK;
    const int MD = M * D, Gq = H / G, VC = value_columns(E), rows = page_size < BKV ? page_size : BKV;
    const char* err = nullptr;
    CUtensorMap tq, tk, tv;
    if (!query_map(q, MD, H, T, Gq, BQ / Gq, &tq, &err)) return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: q: %s", err);
    const int k_boxed = rows == BKV ? D / 64 : 1, v_boxed = rows == BKV ? VC / 64 : 1;
    if (!block_map(cache, MD, MD, G * page_size, num_pages, page_stride, rows, k_boxed, &tk, &err) ||
        !block_map((const __nv_bfloat16*)cache + (size_t)G * page_size * MD, E, E, G * page_size, num_pages, page_stride, rows, v_boxed, &tv, &err))
        return forge::fail(FORGE_ERR_UNSUPPORTED, "scored_attention_sm100: cache: %s", err);
    ShapedParams p{};
    p.out = (__nv_bfloat16*)out; p.out_ld = out_ld; p.u = M == 2 ? u : nullptr;
    p.block_table = block_table; p.tiles = reinterpret_cast<const int4*>(tiles);
    p.r1 = r1; p.r2 = r2; p.sink = sink;
    p.H = H; p.heads = Gq; p.inner = G * M * (E / VC); p.M = M; p.D = D; p.E = E; p.VC = VC;
    p.q_channels = D; p.key_blocks = D / 64; p.value_blocks = VC / 64; p.latent = 0;
    p.k_boxed = k_boxed; p.v_boxed = v_boxed;
    p.page_size = page_size; p.max_pages = max_pages; p.window = window; p.chunk = chunk; p.softcap = softcap;
    p.vec_out = ((uintptr_t)out & 15) == 0 && out_ld % 8 == 0; p.scale = scale; p.out_scale = M == 1 ? out_scale : 1.0f; p.status = status;
    const int rc = r1 != nullptr || softcap > 0.f ? launch<true>("scored_attention_sm100", tq, tk, tv, p, num_tiles, stream)
                                                  : launch<false>("scored_attention_sm100", tq, tk, tv, p, num_tiles, stream);
    if (rc != FORGE_OK || M == 1) return rc;
    return forge::check_launch("scored_combine", launch_combine(u, nullptr, 1, (__nv_bfloat16*)out, T, H, 2, E, lambda, post * out_scale, eps, out_ld, nullptr, stream));
}

extern "C" const char* forge_last_error() { return forge::error_buffer(); }

// (checks build) the bounds that this library's kernel tests page ids against
FORGE_DEFINE_CHECKS_ENTRY(attention_shaped_sm100)
