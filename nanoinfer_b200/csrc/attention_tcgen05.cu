// Paged causal attention for prompt portions on the 5th-generation tensor cores (tcgen05 + TMEM), for
// bfloat16 and head sizes 64 and 128.
//
// A CTA owns a tile of up to 128 rows, where a row is one (token, query head of the kv group): the keys and
// values of a kv head are read once for all the query heads that share it. For every block of 128 keys:
//         S = Q . K^T         (tcgen05.mma, accumulator S in tensor memory)
//         P = exp2(S*scale - max), row sums       (a thread per row: no exchange between threads)
//         O += P . V          (tcgen05.mma, P from tensor memory, V as the MN-major operand; O stays in tensor memory
//                              over all blocks)
// TWO CTAs share an SM (256 columns of tensor memory, half of the shared memory and of the registers each): while one
// waits for its scores, its keys, its first block or its next tile, the other's softmax has the exponential unit, which
// bounds the kernel (16 a clock and SM: 1,024 cycles for a tile's block; the two products take 512 at heads of 64, 1,024 at
// heads of 128). Heads of 64: scores, probabilities and output have columns of their own, so the scores of block j+1 are
// multiplied as soon as those of block j are in registers. Heads of 128: the probabilities overwrite the scores they come
// from, and keys and values have one stage each, whose next copies run under the softmax. Against one CTA an SM with two
// threads a row, probabilities through shared memory and blocks of 64 keys at heads of 128 (us a launch, that one
// first): 2,048 tokens of 14 query and 2 key heads of 64, 27 and 29; 601 + 461 + 320 tokens of them, 13.7 and 11.8; 4,096 tokens
// behind 4,096, 207 and 150; 2,048 behind 14,336, 12 and 2 heads of 128, 596 and 217; 2 x 4,096, 28 and 4 heads of 128, 806 and 235.
// The running maximum that the exponents refer to is only replaced when the row's maximum grew by more than
// 2^8; only then is the row of O rescaled (read from tensor memory, multiplied, written back). At the end O is
// read once and divided by the sum.
// Q, K and V tiles arrive by TMA (cp.async.bulk.tensor, 128-byte swizzle): Q through a 3-D map over
// (head dim, heads of the group, tokens), K and V through a 3-D map over the page pool, one box per
// page of the block table; a page the request does not hold is fetched from an out-of-range coordinate
// and arrives as zeros. Roles: warp 0 = TMA producer, warp 1 = MMA issuer and TMEM owner, warps 2..5 =
// softmax and output. Every wait is bounded; a wait that runs out records an error word, the CTA stops,
// drains its copies, frees its TMEM and returns.
//
// A second instance of the kernel (FLEX) takes the options that other designs put on the scores: a soft cap
// c tanh(s / c) (monotone, so the row's maximum is still the cap of the largest raw score; applied to every score in
// 32-bit with the fast exponential and division before the exponent of the softmax), a chunked mask (a position sees its
// own block of `chunk` positions, counted from the request's start), a sink per head (exp(sink) once more in the
// denominator, added where the row is divided by its sum), kept first tokens (the first `keep_first` positions are seen however far
// back they are: their key blocks come ahead of the window's), and a gate per (token, head) (a factor sigmoid(gate) where the row is
// divided by its sum). The instance without options is compiled without any of it.
//
// Formula as in attention_generic.cu (cpp/src/ops.cpp:206-270); the reference's prefill attention is a
// SIMT kernel with 32-key shared-memory slabs (cpp/src/cuda/cuda_backend.cu:489-575).
#include "tcgen05.cuh"
#include <type_traits>

using namespace nibp;
using namespace nibt;

namespace {

constexpr int ROWS = 128;        // rows of a tile (UMMA M): TMEM lanes
constexpr int THREADS = 192;     // TMA warp, MMA warp, four softmax warps (a thread per row)
constexpr int KEYS = 128;        // keys per block (UMMA N of S, K of P.V)
constexpr float LOG2E = 1.4426950408889634f;

__device__ int g_attn_error = 0;

// The hand-overs between the roles of this kernel are short and on the critical path of every block of keys: poll
// without sleeping for a long while (the limit still holds).
__device__ __forceinline__ bool mbar_spin(unsigned long long* bar, unsigned parity) {
#pragma unroll 1      // (unrolled, each of the kernel's thirty waits would be several copies of this loop: instruction cache)
    for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (i > (1u << 16)) __nanosleep(100);
    }
    return false;
}
__device__ __forceinline__ bool warp_spin(unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_spin(bar, parity)); }
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
// Two floats side by side: one instruction of the fused multiply-add unit works on both.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 two(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void split(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 2^x of two numbers in the multiply-add unit, for x < 127: x = n + f with n the nearest whole number (the low bits of
// x + 1.5 * 2^23), 2^f on [-1/2, 1/2] by a polynomial of degree 5 (Remez exchange for the relative error: 7.5e-8, 2.1e-7 as
// evaluated here; ex2.approx allows itself 2.4e-7), n added to the exponent. What the polynomial does not cover is what
// ex2.approx.ftz gives: 0 below -126 (-inf, too) and NaN for NaN (a score that overflowed has to show in its row).
__device__ __forceinline__ float or_limit(float x, float p) {
    float limit;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(limit) : "f"(x));
    return x >= -126.f ? p : limit;
}
__device__ __forceinline__ void exp2_fma(f32x2 x, float& p0, float& p1) {
    const f32x2 magic = two(12582912.f, 12582912.f);
    const f32x2 n = add2(x, magic);
    const f32x2 f = fma2(add2(n, two(-12582912.f, -12582912.f)), two(-1.f, -1.f), x);
    f32x2 p = fma2(two(1.3276472454890609e-3f, 1.3276472454890609e-3f), f, two(9.675540961325169e-3f, 9.675540961325169e-3f));
    p = fma2(p, f, two(5.550713092088699e-2f, 5.550713092088699e-2f));
    p = fma2(p, f, two(0.24022120237350464f, 0.24022120237350464f));
    p = fma2(p, f, two(0.6931469440460205f, 0.6931469440460205f));
    p = fma2(p, f, two(1.0000001192092896f, 1.0000001192092896f));
    float x0, x1, n0, n1;
    split(x, x0, x1);
    split(n, n0, n1);
    split(p, p0, p1);
    p0 = or_limit(x0, __int_as_float(__float_as_int(p0) + (__float_as_int(n0) << 23)));
    p1 = or_limit(x1, __int_as_float(__float_as_int(p1) + (__float_as_int(n1) << 23)));
}
template <int HD> struct Cfg {
    static constexpr int SUB = HD / 64;                       // sub-tiles of 64 elements (128 bytes) along the head dim
    static constexpr int SUBTILE = 128 * 128;                 // bytes of a [128 rows x 64 elements] sub-tile
    static constexpr int Q_BYTES = SUB * SUBTILE;             // the tile of queries
    static constexpr int KV_BYTES = KEYS * HD * 2;            // one block of keys (or values)
    static constexpr int STAGES = HD == 64 ? 2 : 1;
    static constexpr int OFF_Q = 0, OFF_K = Q_BYTES, OFF_V = OFF_K + STAGES * KV_BYTES, OFF_BAR = OFF_V + STAGES * KV_BYTES;
    static constexpr int SMEM = OFF_BAR + 256 + 1024;
    static constexpr bool P_OWN = HD == 64;                   // the probabilities have columns of their own
    static constexpr int COL_S = 0, COL_P = P_OWN ? KEYS : 0, COL_O = P_OWN ? KEYS + KEYS / 2 : KEYS;
    static constexpr int TMEM_COLS = 256;
    static_assert(COL_O + HD <= TMEM_COLS, "two CTAs share an SM's tensor memory");
    static_assert(prompt_fits_tmem(SMEM, TMEM_COLS), "CTAs that share an SM must not wait for one another's tensor memory");
};

// The running maximum of a row is replaced by a larger one only when it grew by more than this (in log2 units):
// the output accumulator in tensor memory then has to be rescaled, which costs a read and a write of the row.
// Meanwhile probabilities are at most 2^8, harmless in bfloat16 and in the 32-bit sums.
constexpr float RESCALE_ABOVE = 8.0f;

// Of 16 pairs of exponentials, how many go to the multiply-add unit: at heads of 128, 2,048 tokens behind 14,336 (12 query and 2
// key heads), 0 / 3 / 6 of them took 243 / 223 / 270 us, at heads of 64, 4,096 behind 4,096, 150 / 150 / 166.
template <int HD> constexpr int EMULATED = HD == 128 ? 3 : 0;

// grid: row tiles x requests x kv heads, the kv head fastest: the tiles that see the most keys start first
template <int HD, bool FLEX>
__global__ void __launch_bounds__(THREADS, 2)
attention_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                            const int* __restrict__ q_start, const int* __restrict__ ctx_lens,
                            const int* __restrict__ block_table, int bt_stride, int page_size, int num_pages, int n_req,
                            int heads, int kv_heads, float scale, int window, unsigned long long* trace, int trace_cap,
                            float softcap, int chunk, const float* __restrict__ sinks, float out_scale, int keep_first,
                            const float* __restrict__ gate, int ld_gate) {
    using C = Cfg<HD>;
    constexpr int STAGES = C::STAGES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(smem + C::OFF_BAR);
    unsigned long long* q_full = bars;            // 1
    unsigned long long* k_full = bars + 1;        // [STAGES]
    unsigned long long* k_empty = bars + 3;
    unsigned long long* v_full = bars + 5;
    unsigned long long* v_empty = bars + 7;
    // Phase j of each of these belongs to block j. A wait for a phase is one for its parity, so it must not come while the phase two
    // before it is still open. Every phase is seen by its waiter before the next can complete, except those of o_done where the
    // probabilities lie on the scores: it is waited for only when a row is rescaled and at the end. There the scores of block j are
    // multiplied and told behind P.V of block j - 1 by the same thread, and a softmax warp that waits for o_done has seen s_full(j):
    // P.V of block j - 1 is done then, and o_done at most about to be told of it, never a phase behind that.
    unsigned long long* s_full = bars + 9;        // the scores are in tensor memory
    unsigned long long* s_empty = bars + 10;      // P_OWN: ... and in registers (an arrival per softmax warp)
    unsigned long long* p_full = bars + 11;       // [2] the probabilities of a half of the keys are in tensor memory (an arrival per softmax warp)
    unsigned long long* o_done = bars + 13;       // P.V has been added
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 14);
    __shared__ volatile int s_failed;

    pdl_launch_dependents();
    if (threadIdx.x == 0) nib_trace_mark(trace, trace_cap, NIB_TK_ATTN_PREFILL, 0, 0);
    const int n_rep = heads / kv_heads;
    const int tpt = ROWS / n_rep;                         // tokens per tile
    const int rows_tile = tpt * n_rep;
    const int kvh = blockIdx.x % kv_heads, req = (blockIdx.x / kv_heads) % n_req, tile = blockIdx.x / (kv_heads * n_req);
    const int n_tiles = gridDim.x / (kv_heads * n_req);
    const int row_begin = q_start[req], q_len = q_start[req + 1] - row_begin;
    // tiles late in the portion see the most keys: they start first
    const int tok0 = (n_tiles - 1 - tile) * tpt;          // first token of this tile within the request's portion
    if (tok0 >= q_len) return;
    const int n_tok = min(tpt, q_len - tok0);
    const int ctx = ctx_lens[req];
    const int pos0 = ctx - q_len + tok0;                  // position of the tile's first token
    const int hi_cta = pos0 + n_tok - 1;
    int lo_cta = window > 0 ? max(0, pos0 - window + 1) : 0;
    if (FLEX && chunk > 0) lo_cta = max(lo_cta, (pos0 / chunk) * chunk);      // (the first visible key never decreases with the position)
    const int b_begin = lo_cta / KEYS;
    const int n_kept = FLEX ? min((keep_first + KEYS - 1) / KEYS, b_begin) : 0;      // key blocks with kept tokens before the window's first
    const int n_blk = n_kept + hi_cta / KEYS - b_begin + 1;
    auto block_at = [&](int j) { return FLEX && j < n_kept ? j : b_begin + j - n_kept; };
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int* bt = block_table + (size_t)req * bt_stride;

    if (threadIdx.x == 0) {
        s_failed = 0;
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        mbar_init(q_full, 1);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
            mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
        }
        mbar_init(s_full, 1);
        mbar_init(s_empty, 4);
        mbar_init(&p_full[0], 4);
        mbar_init(&p_full[1], 4);
        mbar_init(o_done, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // The producer's look-ups: a lane's block-table entry of block j, or -1 where there is no page to fetch. The entry of block
    // j+1 is asked for while block j is being sent for and is looked at only a block later (the first before the wait for the
    // kernel before this one: no kernel writes the table): the look-up's latency (more than half a microsecond) must not stand
    // between two blocks' copies.
    const int pages_per_block = KEYS / page_size;
    const int oob = num_pages * kv_heads;             // a coordinate outside the pool: the box arrives as zeros
    auto entry_of = [&](int j) -> int {
        const int key = block_at(j) * KEYS + lane * page_size;
        if (lane >= pages_per_block || key > hi_cta || (key + page_size <= lo_cta && !(FLEX && key < keep_first))) return -1;
        return __ldg(bt + key / page_size);
    };
    const int entry_first = warp == 0 ? entry_of(0) : -1;
    const unsigned tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_wait();
    if (threadIdx.x == 0) nib_trace_mark(trace, trace_cap, NIB_TK_ATTN_PREFILL, 0, 1);

    if (warp == 0) {
        // ---------------- producer: one thread fetches Q, arms the barriers and fetches the pages of every block of keys;
        // lane i looks page i up, one block ahead, so that the look-up of a page never stands between two copies
        if (elect_one()) {
            mbar_expect_tx(q_full, (unsigned)(rows_tile * 128 * C::SUB));
#pragma unroll
            for (int s = 0; s < C::SUB; ++s)
                tma_load_3d(smem + C::OFF_Q + s * C::SUBTILE, &map_q, q_full, s * 64, kvh * n_rep, row_begin + tok0);
        }
        __syncwarp();
        int entry_next = entry_first;
        int issued = 0;
        bool ok = true;
        for (int j = 0; j < n_blk && ok; ++j) {
            const int st = j % STAGES;
            const int entry = entry_next;
            if (j + 1 < n_blk) entry_next = entry_of(j + 1);
            const int z = (entry >= 0 && entry < num_pages) ? entry * kv_heads + kvh : oob;      // third coordinate of the page
            // keys first (the scores are wanted before the values), values when their stage is free
            const unsigned par = ((j / STAGES) & 1) ^ 1;
#pragma unroll
            for (int kv = 0; kv < 2; ++kv) {
                unsigned long long* full = kv ? &v_full[st] : &k_full[st];
                ok = __all_sync(0xffffffffu, mbar_spin(kv ? &v_empty[st] : &k_empty[st], par));
                if (!ok) break;
                if (elect_one()) mbar_expect_tx(full, C::KV_BYTES);
                __syncwarp();
                unsigned char* to = smem + (kv ? C::OFF_V : C::OFF_K) + st * C::KV_BYTES;
                for (int i = 0; i < pages_per_block; ++i) {
                    const int zi = __shfl_sync(0xffffffffu, z, i);
                    if (elect_one()) {
#pragma unroll
                        for (int s = 0; s < C::SUB; ++s)
                            tma_load_3d(to + s * (KEYS * 128) + i * page_size * 128, kv ? &map_v : &map_k, full, s * 64, 0, zi);
                    }
                    __syncwarp();
                }
                issued = 2 * j + kv + 1;
            }
        }
        if (!ok && lane == 0 && !s_failed) { atomicCAS(&g_attn_error, 0, (1 << 16) | (int)(blockIdx.x & 0xffff)); s_failed = 1; }
        if (s_failed && lane == 0) {
            // copies already issued still target this CTA's shared memory: wait for them, bounded
            mbar_wait(q_full, 0);
            for (int j = max(0, issued / 2 - STAGES); j < (issued + 1) / 2; ++j) {
                mbar_wait(&k_full[j % STAGES], (j / STAGES) & 1);
                if (2 * j + 1 < issued) mbar_wait(&v_full[j % STAGES], (j / STAGES) & 1);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer. Products run in the order of issue, so where the probabilities lie on the scores
        // the next scores are issued behind the P.V that reads them.
        constexpr unsigned idesc_s = instr_desc(ROWS, KEYS, false);
        constexpr unsigned idesc_o = instr_desc(ROWS, HD, true);
        const unsigned q_addr = smem_u32(smem + C::OFF_Q);
        auto issue_qk = [&](int j) -> bool {
            if (!warp_spin(&k_full[j % STAGES], (j / STAGES) & 1)) return false;
            if (C::P_OWN && j > 0 && !warp_spin(s_empty, (j - 1) & 1)) return false;
            tc_fence_after();
            const unsigned k_addr = smem_u32(smem + C::OFF_K + (j % STAGES) * C::KV_BYTES);
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < HD / 16; ++kk) {
                    const unsigned long long adv = (unsigned long long)(((kk & 3) * 32) >> 4);
                    tc_mma(tmem_base + C::COL_S, desc_kmajor(q_addr + (kk >> 2) * C::SUBTILE) + adv,
                           desc_kmajor(k_addr + (kk >> 2) * (KEYS * 128)) + adv, idesc_s, kk > 0);
                }
                tc_commit(s_full);
                tc_commit(&k_empty[j % STAGES]);
            }
            __syncwarp();
            return true;
        };
        auto issue_pv = [&](int j) -> bool {
            if (!warp_spin(&v_full[j % STAGES], (j / STAGES) & 1)) return false;
            const unsigned v_addr = smem_u32(smem + C::OFF_V + (j % STAGES) * C::KV_BYTES);
#pragma unroll
            for (int half = 0; half < 2; ++half) {          // of the keys, as their probabilities come
                if (!warp_spin(&p_full[half], j & 1)) return false;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int kk = half * (KEYS / 32); kk < (half + 1) * (KEYS / 32); ++kk) {
                        // P: 16 keys are 8 columns; V: 16 keys = 2048 bytes further down, the second 64 elements of the head
                        // dim KEYS*128 bytes further on
                        const unsigned long long b = desc_mnmajor(v_addr + kk * 16 * 128, KEYS * 128);
                        tc_mma_ts(tmem_base + C::COL_O, tmem_base + C::COL_P + kk * 8, b, idesc_o, j > 0 || kk > 0);
                    }
                    if (half == 1) {
                        tc_commit(o_done);
                        tc_commit(&v_empty[j % STAGES]);
                    }
                }
                __syncwarp();
            }
            return true;
        };
        bool ok = warp_spin(q_full, 0) && issue_qk(0);
        for (int j = 0; j < n_blk && ok; ++j) {
            if (C::P_OWN && j + 1 < n_blk) ok = issue_qk(j + 1);
            ok = ok && issue_pv(j);
            if (!C::P_OWN && j + 1 < n_blk) ok = ok && issue_qk(j + 1);
        }
        if (!ok && lane == 0 && !s_failed) { atomicCAS(&g_attn_error, 0, (3 << 16) | (int)(blockIdx.x & 0xffff)); s_failed = 1; }
    } else if (warp >= 2) {
        // ---------------- softmax and output: a thread owns a row, in the warp that may read its TMEM lane
        // (32*(warp%4)...). Rows past the tile's last (the tile holds a whole number of tokens) see what the last row
        // sees; nothing of them is stored.
        const int quad = warp & 3, row = quad * 32 + lane;
        const unsigned lane_addr = tmem_base + ((unsigned)(quad * 32) << 16);
        const unsigned o_addr = lane_addr + C::COL_O;
        const bool live = row < n_tok * n_rep;
        const int ti = min(row / n_rep, n_tok - 1), head = kvh * n_rep + (row % n_rep);
        const int hi = pos0 + ti;
        int lo = window > 0 ? max(0, hi - window + 1) : 0;
        if (FLEX && chunk > 0) lo = max(lo, (hi / chunk) * chunk);
        const bool capped = FLEX && softcap > 0.f;
        // capped scores are turned into base-2 units where they are read, so the factor on them afterwards is one
        const float scale2 = capped ? 1.0f : scale * LOG2E;
        const float cap_in = capped ? 2.0f * scale / softcap : 0.f, cap_out = softcap * LOG2E;
        float m_cur = -INFINITY, l_run = 0.f;       // the maximum that the exponents refer to, and the row's sum
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < n_blk; ++j) {
            ok = warp_spin(s_full, j & 1);
            if (!ok) break;
            tc_fence_after();
            const int key0 = block_at(j) * KEYS;
            // the same branch for the whole warp: a warp that took both would do the work twice
            const bool all_visible = __all_sync(0xffffffffu, key0 >= lo && key0 + KEYS - 1 <= hi);
            // the row's scores of the block: all loads are issued, then waited for once (a load from tensor memory
            // takes hundreds of cycles)
            unsigned raw[KEYS / 32][32];
#pragma unroll
            for (int c = 0; c < KEYS / 32; ++c) tmem_ld32_async(lane_addr + C::COL_S + c * 32, raw[c]);
            tmem_wait_ld();
            if (C::P_OWN) {         // the next scores may take their place
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_empty);
            }
            if (capped) {
                // c tanh(x / c) = c (1 - 2 / (1 + e^(2x/c))), off by a few 1e-7 in absolute terms
#pragma unroll
                for (int c = 0; c < KEYS / 32; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        raw[c][i] = __float_as_uint(cap_out * (1.0f - __fdividef(2.0f, 1.0f + __expf(cap_in * __uint_as_float(raw[c][i])))));
            }
            if (!all_visible) {
#pragma unroll
                for (int c = 0; c < KEYS / 32; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = key0 + c * 32 + i;
                        if (!((key >= lo || (FLEX && key < keep_first)) && key <= hi)) raw[c][i] = 0xff800000u;      // -inf: its probability will be 0
                    }
            }
            // four maxima side by side, so that no instruction waits for the one before it
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < KEYS / 32; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2)
                    mx4[(i >> 1) & 3] = max3(mx4[(i >> 1) & 3], __uint_as_float(raw[c][i]), __uint_as_float(raw[c][i + 1]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale2;      // scale2 > 0
            float corr = 1.f;
            bool grow = false;
            if (m_cur == -INFINITY) {
                m_cur = mx;                                 // nothing summed yet: sum and output row are zero
            } else if (mx > m_cur + RESCALE_ABOVE) {
                corr = ex2(m_cur - mx);
                l_run *= corr;
                m_cur = mx;
                grow = true;
            }
            const float m_use = (m_cur == -INFINITY) ? 0.f : m_cur;
            const bool rescale = j > 0 && __any_sync(0xffffffffu, grow);
            if (j > 0 && (C::P_OWN || rescale)) {
                // P.V of the block before has been added: it has read its probabilities, and the output row is at rest
                ok = warp_spin(o_done, (j - 1) & 1);
                if (!ok) break;
                tc_fence_after();
            }
            if (rescale) {      // rare: the output row is rescaled in tensor memory
#pragma unroll 1
                for (int c = 0; c < HD; c += 16) {
                    unsigned ov[16];
                    tmem_ld16_async(o_addr + c, ov);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * corr);
                    tmem_st16(o_addr + c, ov);
                }
            }
            // the probabilities into tensor memory (two keys a column), their sum (four partial sums). Of 16 pairs the
            // exponential unit takes 16 - EMULATED, the multiply-add unit the others (not where scores are masked: 2^-inf).
            const f32x2 scale_2 = two(scale2, scale2), less_m = two(-m_use, -m_use);
            f32x2 sum2[2] = {two(0.f, 0.f), two(0.f, 0.f)};
            auto tell = [&](int half) {
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[half]);
            };
            auto probabilities = [&](auto emulated) {
                constexpr int EMU = decltype(emulated)::value;
#pragma unroll
                for (int c = 0; c < KEYS / 32; ++c) {
                    unsigned pk[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const f32x2 x = fma2(two(__uint_as_float(raw[c][2 * i]), __uint_as_float(raw[c][2 * i + 1])), scale_2, less_m);
                        float p0, p1;
                        if ((i * EMU) / 16 != ((i + 1) * EMU) / 16) {
                            exp2_fma(x, p0, p1);
                        } else {
                            split(x, p0, p1);
                            p0 = ex2(p0);                                   // ex2(-inf) = 0
                            p1 = ex2(p1);
                        }
                        sum2[i & 1] = add2(sum2[i & 1], two(p0, p1));
                        pk[i] = pack2(p0, p1);
                    }
                    // a half of the keys is complete: its P.V may start. The first half is told once the next keys'
                    // exponentials are under way, so that nothing waits for its stores.
                    if (c == KEYS / 64) tell(0);
                    tmem_st16(lane_addr + C::COL_P + c * 16, pk);
                    if (c == KEYS / 32 - 1) tell(1);
                }
            };
            if (all_visible)
                probabilities(std::integral_constant<int, EMULATED<HD>>());
            else
                probabilities(std::integral_constant<int, 0>());
            float s0, s1, s2, s3;
            split(sum2[0], s0, s1);
            split(sum2[1], s2, s3);
            l_run += (s0 + s1) + (s2 + s3);
        }
        if (ok) ok = warp_spin(o_done, (n_blk - 1) & 1);
        if (!ok) {
            if (lane == 0 && !s_failed) { atomicCAS(&g_attn_error, 0, (4 << 16) | (int)(blockIdx.x & 0xffff)); s_failed = 1; }
        } else {
            tc_fence_after();
            unsigned ov[HD / 32][32];
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) tmem_ld32_async(o_addr + c * 32, ov[c]);
            tmem_wait_ld();
            if (live) {
                if (FLEX && sinks != nullptr && m_cur != -INFINITY) l_run += ex2(__ldg(sinks + head) * LOG2E - m_cur);   // the sink: no key, no value
                float inv = l_run > 0.f ? out_scale / l_run : 0.f;
                if (FLEX && gate != nullptr) inv *= 1.0f / (1.0f + expf(-gate[(size_t)(row_begin + tok0 + ti) * ld_gate + head]));
                __nv_bfloat16* orow = out + ((size_t)(row_begin + tok0 + ti) * heads + head) * HD;
#pragma unroll
                for (int c = 0; c < HD / 32; ++c)
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint4 w;
                        w.x = pack2(__uint_as_float(ov[c][d]) * inv, __uint_as_float(ov[c][d + 1]) * inv);
                        w.y = pack2(__uint_as_float(ov[c][d + 2]) * inv, __uint_as_float(ov[c][d + 3]) * inv);
                        w.z = pack2(__uint_as_float(ov[c][d + 4]) * inv, __uint_as_float(ov[c][d + 5]) * inv);
                        w.w = pack2(__uint_as_float(ov[c][d + 6]) * inv, __uint_as_float(ov[c][d + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + c * 32 + d) = w;
                    }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) nib_trace_mark(trace, trace_cap, NIB_TK_ATTN_PREFILL, 0, 2);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ---------------------------------------------------------------------------------- host side
// 3-D map over bfloat16 data: dims (d0 innermost), strides in elements for d1 and d2, box (64, b1, b2).
int make_map3(CUtensorMap* map, const void* ptr, long long d0, long long d1, long long d2, long long s1, long long s2,
              int b1, int b2) {
    NibEncodeTiledFn enc = nib_tensor_map_encoder();
    NIB_REQUIRE(enc != nullptr, "attention (tcgen05): cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
    cuuint64_t strides[2] = {(cuuint64_t)s1 * 2, (cuuint64_t)s2 * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)b1, (cuuint32_t)b2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    NIB_REQUIRE(r == CUDA_SUCCESS, "attention (tcgen05): cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

template <int HD, bool FLEX>
int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, void* out, const int* q_start,
           const int* ctx_lens, const int* block_table, int bt_stride, int page_size, int num_pages, int n_req,
           int max_q_len, int heads, int kv_heads, float scale, int window, float softcap, int chunk, const float* sinks,
           float out_scale, int keep_first, const float* gate, int ld_gate, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        NIB_CUDA(cudaFuncSetAttribute(attention_prefill_tc_kernel<HD, FLEX>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<HD>::SMEM));
        configured = true;
    }
    const int tpt = ROWS / (heads / kv_heads);
    const long long blocks = (long long)ceil_div(max_q_len, tpt) * n_req * kv_heads;
    NIB_REQUIRE(blocks <= 0x7fffffffLL, "attention (tcgen05): too many tiles for one launch");
    NIB_CUDA(launch_pdl(attention_prefill_tc_kernel<HD, FLEX>, dim3((unsigned)blocks), dim3(THREADS), (size_t)Cfg<HD>::SMEM, stream, mq, mk, mv,
                        (__nv_bfloat16*)out, q_start, ctx_lens, block_table, bt_stride, page_size, num_pages, n_req, heads,
                        kv_heads, scale, window, nib_trace_buffer(), nib_trace_capacity(), softcap, chunk, sinks, out_scale, keep_first, gate, ld_gate));
    return 0;
}

}  // namespace

// 1 if the tcgen05 kernel takes this shape: head size 64 or 128, at most 128 query heads per kv head,
// pages of 8..128 tokens that divide 128, 16-byte aligned rows.
NIB_API int nib_attention_prefill_tc_supported(int heads, int kv_heads, int head_dim, int page_size, int q_stride) {
    if (kv_heads <= 0 || heads % kv_heads || heads / kv_heads > ROWS) return 0;
    if (head_dim != 64 && head_dim != 128) return 0;
    if (page_size < 8 || page_size > KEYS || KEYS % page_size) return 0;
    if (q_stride % 8) return 0;
    return nib_tensor_map_encoder() != nullptr;
}

// The error word of the kernel's bounded waits (0 = none); synchronises with the device and clears it.
NIB_API int nib_attention_tc_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_attn_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_attn_error, &zero, sizeof(int));
    return v;
}

// Same arguments as nib_attention_prefill_mma plus the number of rows of qkv (m_tokens, for the map's extent), and the
// options: softcap (0 = none), chunk (0 = none), sinks [heads] (null = none), a factor on the output (32-bit, before it is rounded),
// keep_first (0 = none), gate [tokens, heads] with rows of ld_gate floats (null = none).
NIB_API int nib_attention_prefill_tc(const void* qkv, int q_stride, void* out, const int* q_start, const int* ctx_lens,
                                     const int* block_table, int bt_stride, int page_size, const void* k_pages,
                                     const void* v_pages, int num_pages, int n_req, int max_q_len, int m_tokens,
                                     int heads, int kv_heads, int head_dim, float scale, int window, float softcap, int chunk,
                                     const float* sinks, float out_scale, int keep_first, const float* gate, int ld_gate,
                                     cudaStream_t stream) {
    NIB_REQUIRE(nib_attention_prefill_tc_supported(heads, kv_heads, head_dim, page_size, q_stride),
                "attention (tcgen05): head_dim %d, %d/%d heads, page size %d are not supported", head_dim, heads, kv_heads, page_size);
    NIB_REQUIRE(n_req >= 0 && max_q_len > 0 && num_pages > 0 && window >= 0 && m_tokens > 0 && chunk >= 0 && softcap >= 0.f && scale > 0.f && keep_first >= 0,
                "attention (tcgen05): bad sizes");
    NIB_REQUIRE((((uintptr_t)qkv | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) & 15) == 0, "attention (tcgen05): bases must be 16-byte aligned");
    if (n_req == 0) return 0;
    const int n_rep = heads / kv_heads, tpt = ROWS / n_rep;
    CUtensorMap mq, mk, mv;
    // queries: (head dim, heads, tokens); a box is 64 x n_rep heads x tpt tokens
    if (make_map3(&mq, qkv, head_dim, heads, m_tokens, head_dim, q_stride, n_rep, tpt)) return 1;
    // pool: (head dim, slot in page, page * kv_heads + kv head); a box is one page of one kv head
    const long long planes = (long long)num_pages * kv_heads;
    if (make_map3(&mk, k_pages, head_dim, page_size, planes, head_dim, (long long)page_size * head_dim, page_size, 1)) return 1;
    if (make_map3(&mv, v_pages, head_dim, page_size, planes, head_dim, (long long)page_size * head_dim, page_size, 1)) return 1;
#define NIB_TC_ATTN(HD, FLEX) launch<HD, FLEX>(mq, mk, mv, out, q_start, ctx_lens, block_table, bt_stride, page_size, num_pages, n_req, max_q_len, \
                                               heads, kv_heads, scale, window, softcap, chunk, sinks, out_scale, keep_first, gate, ld_gate, stream)
    const bool flex = softcap > 0.f || chunk > 0 || sinks != nullptr || (keep_first > 0 && window > 0) || gate != nullptr;
    if (head_dim == 64) return flex ? NIB_TC_ATTN(64, true) : NIB_TC_ATTN(64, false);
    return flex ? NIB_TC_ATTN(128, true) : NIB_TC_ATTN(128, false);
#undef NIB_TC_ATTN
}
