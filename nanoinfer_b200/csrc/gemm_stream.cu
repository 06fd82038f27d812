// Matrix product for a decode step of up to 16 tokens (whose activations are at most 64 KB) over wide weights: out[tokens, N] =
// A[tokens, K] . W[N, K]^T, bfloat16 operands, 32-bit sums. What bounds it is reading the weights once and the chain from the kernel before it to its own result.
//
// One CTA an SM, every SM the same number of output features (RB = ceil(N / SMs), in several chunks where that is more than 64):
// no last wave. (With 16 features a CTA the 4,864 features of the 0.5B widths are 304 CTAs, two an SM and eight over, and those eight
// start when the first 296 are done.) One warp sends for the weights by tensor-map copies, BEFORE the wait for the kernel before this
// one (they are nobody's output): all of them at once where they fit, else through a ring of stages. The copies cost no registers and
// no issue slots of whatever runs meanwhile, and the kernels before this one (attention, output projection) let the next one in at their
// first instruction, so the weights of the products that follow are on their way while a chain of small kernels waits for itself.
//
// Behind the wait a CTA reads all activations into shared memory, warp w the w-th eighth of every token, and where a norm stands
// before the product it computes that itself: bfloat16(x * gain) as the operand, the sum of x^2 beside it, and 1 / sqrt(mean(x^2)
// + eps) as a factor on the sums.
//
// Weights lie as [block of 64 k][RB rows][128 bytes] (gated: gate rows, then up rows), swizzled by their address, so eight rows of one
// block are read by ldmatrix without bank conflicts whatever RB is. KG groups of warps take the blocks in turn (KG = 8, or 4 with two
// halves of the row tiles: gated, the gate rows and the up rows). Their sums meet in shared memory and are added up in a fixed order by
// the warp that owns the token: a row's result depends on neither the batch nor the run, unless CTAs share K (`splits`), whose sums
// meet in memory.
//
// Measured (us a step, replayed graphs, before: the small-M product behind a norm kernel of its own / with this): 0.5B widths, one
// request at 777 tokens 565 / 498, 4 at 1,000 618 / 530, 8 at 4,096 675 / 640, 16 at 1,000 814 / 699 (a norm of its own: see the dispatch);
// 1.5B, 1 at 1,000 1,060 / 1,005, 8 at 4,096 1,291 / 1,243; four layers of the 7B, 4 at 800 607 / 574. Alone, over and over with
// weights from memory: 4,864 x 896 5.0 us (3.5 TB/s; the small-M product 5.2), 8,960 x 1,536 10.3 (5.4; 12.0), 18,944 x 3,584 41.4
// (6.6; tcgen05 48.3). The down projection of one token, 896 x 4,864, 3.6 (tcgen05 4.2; the step 498 / 474).
// Tried and slower: weights and activations through one ring (a line of the activations a stage); the norm's values left by the output
// projection's epilogue (its sums of squares are one more trip to memory); the output and the q/k/v projections in this kernel (1.6 to 2
// MB: the small-M product's registers hold them); a dry pass of the consuming code before the wait, to have its instructions cached (the
// step 498 / 526).
#include "attention_common.cuh"
#include "tcgen05.cuh"
#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>

using namespace nibp;
using nibt::elect_one;
using nibt::uniform_warp;
using std::max;
using std::min;

extern "C" int nib_sm_count();

namespace {

constexpr int WARPS = 8;                    // consumer warps; one more sends
constexpr int THREADS = (WARPS + 1) * 32;
constexpr int STREAM_TOKENS = 16;
constexpr int MAX_RB = 64;
constexpr int PITCH = 20;                   // floats between two tokens of a tile of sums: no bank conflicts
// Shared memory of a CTA that holds all its weights at once, at most: less than what an SM has, so that a CTA of the kernel before it
// or behind it fits beside it. Larger ones run through a ring, in all there is.
constexpr int WHOLE_GATED = 140 * 1024, WHOLE_SUM = 100 * 1024, RING_SMEM = 208 * 1024;

__device__ int g_stream_error = 0;          // 0, or (code << 16 | blockIdx.x) of the first wait that ran out

struct StreamArgs {
    const void* A; const float* bias; void* out; int tokens, N, K, lda, ldo;        // A: bfloat16, or with a norm the stream (floats)
    int rb, kb, splits, split_blocks, stages, w_region, w_stage, a_pitch, a_bytes, part_at, bars_at;      // (from w_region on in bytes)
    const float* gain; float eps;
    NibGlu glu;
};

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, 256;\n" ::: "memory"); }
__device__ __forceinline__ void copy16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
// NT: token tiles of 8. TW: row tiles of 16 per warp. KG: warps that share the blocks (8, or 4 with two halves of the row tiles).
template <int NT, int TW, int KG, int EPI, bool NORM>
__global__ void __launch_bounds__(THREADS)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_w, const StreamArgs p, unsigned long long* trace, int trace_cap) {
    constexpr bool TWO = epi_dual(EPI);
    constexpr int HALVES = WARPS / KG, TT = TW * HALVES, TOK = NT * 8;               // row tiles of a chunk
    static_assert(TWO ? KG == 4 : EPI == EPI_ADD && !NORM, "gated, half of the warps on the gate rows and half on the up rows, or a sum");
    static_assert(!NORM || NT == 1, "from 9 tokens on the norm is a kernel of its own");
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* a_s = smem + (size_t)p.stages * p.w_stage;               // [tokens][a_pitch]
    // [KG][TT][NT * 8][PITCH] sums: where the weights were, if there is one chunk only
    float* part = reinterpret_cast<float*>(smem + p.part_at);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem + p.bars_at);
    unsigned long long* empty = full + p.stages;
    __shared__ float s_sq[TOK][WARPS];          // NORM: sums of x^2 of the eighths of a token
    __shared__ volatile int s_failed;

    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int split = (int)blockIdx.x % p.splits, first = (int)blockIdx.x / p.splits, step = (int)gridDim.x / p.splits;
    const int k0 = split * p.split_blocks, k_blocks = min(p.split_blocks, (p.K >> 6) - k0);       // this CTA's blocks of 64 k
    const int all_chunks = (p.N + p.rb - 1) / p.rb;
    const int my_chunks = (all_chunks - first + step - 1) / step;
    if (tid == 0) {
        nib_trace_mark(trace, trace_cap, NIB_TK_GEMM_STREAM, EPI, 0);
        s_failed = 0;
        prefetch_tensormap(&map_w);
        for (int s = 0; s < p.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], HALVES); }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == WARPS) {
        // ---------------- the sending warp: weights only, which no kernel writes
        const unsigned bytes = (TWO ? 2u : 1u) * (unsigned)(p.kb * p.rb * 128);
        const int items = my_chunks * ((k_blocks + p.kb - 1) / p.kb);
        int issued = 0, st = 0, kk = 0, f0 = first * p.rb;
        for (int it = 0; it < items; ++it) {
            if (it >= p.stages && !__all_sync(0xffffffffu, mbar_wait(&empty[st], ((it / p.stages) - 1) & 1))) {
                if (lane == 0 && !s_failed) { atomicCAS(&g_stream_error, 0, (2 << 16) | (int)(blockIdx.x & 0xffff)); s_failed = 1; }
                break;
            }
            unsigned char* to = smem + (size_t)st * p.w_stage;
            if (elect_one()) {
                mbar_expect_tx(&full[st], bytes);
                tma_load_3d(to, &map_w, &full[st], 0, f0, k0 + kk);
                if (TWO) tma_load_3d(to + p.w_region, &map_w, &full[st], 0, p.N + f0, k0 + kk);
            }
            __syncwarp();
            issued = it + 1;
            if (++st == p.stages) st = 0;
            kk += p.kb;
            if (kk >= k_blocks) {
                kk = 0;
                f0 += step * p.rb;
            }
        }
        // the last copies have this CTA's shared memory for a target: this warp stays until they are there (bounded)
        for (int it = max(0, issued - p.stages); it < issued; ++it) mbar_wait(&full[it % p.stages], (it / p.stages) & 1);
        return;
    }

    // ---------------- the consuming warps. What does not depend on earlier kernels comes before the wait.
    const int kg = warp % KG, half = warp / KG, g = lane >> 2, t = lane & 3;
    // warp w reads the w-th eighth of every token's k (of this CTA's stretch) ...
    const int seg = k_blocks * 8;           // elements of an eighth
    constexpr int GQ = 4;                   // float4 of the gain kept in registers; longer eighths read theirs again
    float4 gn[NORM ? GQ : 1];
    if (NORM) {
#pragma unroll
        for (int q = 0; q < GQ; ++q)
            gn[q] = (lane + 32 * q) * 4 < seg ? __ldg(reinterpret_cast<const float4*>(p.gain + warp * seg) + lane + 32 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // ... and finishes the tokens w and w + 8, a lane the rows lane and lane + 32 of a chunk
    float bias[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int f = first * p.rb + lane + 32 * j;
        bias[j] = !TWO && p.bias != nullptr && split == 0 && lane + 32 * j < p.rb && f < p.N ? __ldg(p.bias + f) : 0.f;
    }
    // ldmatrix addresses: this lane's token and 16-byte column (A: two steps of a token tile, or a step of two); its row and column
    // (W), where step s is 32 s further on before the swizzle and so one exclusive or away. Rows past the chunk's last one are
    // whatever lies there: their sums go nowhere.
    const int b_row = min(NT == 1 ? (lane & 7) : (lane & 7) + ((lane >> 4) << 3), p.tokens - 1);
    const unsigned b_at = smem_u32(a_s) + (unsigned)(b_row * p.a_pitch) + (NT == 1 ? (unsigned)(lane >> 3) * 16u : (unsigned)((lane >> 3) & 1) * 16u);
    const int w_row = (TWO ? 0 : half * TW * 16) + (lane & 15);
    const unsigned w_half = lane >> 4;
    const unsigned w_base = smem_u32(smem) + (TWO ? (unsigned)(half * p.w_region) : 0u);

    const char* a_from = static_cast<const char*>(p.A) + (NORM ? (size_t)(warp * seg + lane * 4) * 4 : (size_t)(k0 * 64 + warp * seg + lane * 8) * 2);
    const size_t a_stride = (size_t)p.lda * (NORM ? 4 : 2);
    const unsigned a_to = smem_u32(a_s) + (unsigned)(warp * seg * 2 + lane * (NORM ? 8 : 16));

    pdl_wait();
    if (tid == 0) nib_trace_mark(trace, trace_cap, NIB_TK_GEMM_STREAM, EPI, 1);
    float x_old[NT][2];
    const auto read_sums = [&](int f0, int nf) {        // what a sum is added to
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (n * 8 + warp < p.tokens && lane + 32 * j < nf) x_old[n][j] = __ldcg((const float*)p.out + (size_t)(n * 8 + warp) * p.ldo + f0 + lane + 32 * j);
    };
    if (NORM) {
        float sq[TOK];
#pragma unroll
        for (int i = 0; i < TOK; ++i) sq[i] = 0.f;
        for (int q = 0; q * 128 < seg; ++q) {
            const bool there = (lane + 32 * q) * 4 < seg;
            float4 x[TOK];
#pragma unroll
            for (int i = 0; i < TOK; ++i)
                x[i] = there && i < p.tokens ? __ldcg(reinterpret_cast<const float4*>(a_from + (size_t)i * a_stride + (size_t)q * 512)) : make_float4(0.f, 0.f, 0.f, 0.f);
            float4 w = gn[0];
            if (q > 0) w = q == 1 ? gn[NORM ? 1 : 0] : q == 2 ? gn[NORM ? 2 : 0] : q == 3 ? gn[NORM ? 3 : 0]
                                 : there ? __ldg(reinterpret_cast<const float4*>(p.gain + warp * seg) + lane + 32 * q) : w;
#pragma unroll
            for (int i = 0; i < TOK; ++i) {
                if (there && i < p.tokens)
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(a_to + (unsigned)(i * p.a_pitch + q * 256)), "r"(pack_bf16(x[i].x * w.x, x[i].y * w.y)),
                                 "r"(pack_bf16(x[i].z * w.z, x[i].w * w.w)) : "memory");
                sq[i] = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, fmaf(x[i].z, x[i].z, fmaf(x[i].w, x[i].w, sq[i]))));
            }
        }
#pragma unroll
        for (int i = 0; i < TOK; ++i) {
            if (i < p.tokens) {
                const float s = warp_sum(sq[i]);
                if (lane == 0) s_sq[i][warp] = s;
            }
        }
    } else {
        const char* src = a_from;
        for (int e = lane; e * 8 < seg; e += 32, src += 512) {
            const unsigned to = a_to + (unsigned)(e - lane) * 16u;
#pragma unroll
            for (int i = 0; i < TOK; ++i)
                if (i < p.tokens) copy16(to + (unsigned)(i * p.a_pitch), src + (size_t)i * a_stride);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (EPI == EPI_ADD && p.splits == 1) read_sums(first * p.rb, min(p.rb, p.N - first * p.rb));
    }
    // Block i of a CTA's work (its chunks' blocks behind one another) is the warps' of group i mod KG. Either one stage holds all of
    // them (one barrier, waited for under the activations' way), or every block is a stage of a ring of a multiple of KG stages: a
    // stage that is used again is used by the same warps, who so see every phase of its barrier.
    const bool whole = p.stages == 1;
    bool dead = whole && !__all_sync(0xffffffffu, mbar_wait(&full[0], 0));
    if (!NORM) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    consumers_sync();

    float scale[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        scale[n] = 1.f;
        if (NORM && n * 8 + warp < p.tokens) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) s += s_sq[n * 8 + warp][w];
            scale[n] = 1.0f / sqrtf(s / (float)p.K + p.eps);
        }
    }
    int st = kg, turn = 0, at = kg;        // this group's next stage, that stage's turn, and the block's place behind the chunk's first
    for (int c = 0; c < my_chunks; ++c) {
        const int chunk = first + c * step, f0 = chunk * p.rb, nf = min(p.rb, p.N - f0);
        float acc[2][TW][NT][4];        // of even and odd steps: the instructions on one set of sums are a chain
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < TW; ++i)
#pragma unroll
                for (int n = 0; n < NT; ++n) acc[h][i][n][0] = acc[h][i][n][1] = acc[h][i][n][2] = acc[h][i][n][3] = 0.f;
        for (; at < k_blocks; at += KG) {
            if (!whole && !dead) dead = !__all_sync(0xffffffffu, mbar_wait(&full[st], turn & 1));
            if (!dead) {
                const unsigned x_at = b_at + (unsigned)at * 128u;
                const unsigned r = (unsigned)((whole ? at * p.rb : 0) + w_row);
                const unsigned w_at = w_base + (whole ? 0u : (unsigned)st * (unsigned)p.w_stage) + r * 128u + ((w_half ^ (r & 7u)) << 4);
                unsigned bf[4][2 * NT], wf[4][TW][4];
#pragma unroll
                for (int s = 0; s < 4; s += 2 / NT) {
                    unsigned f[4];
                    ldmatrix_x4_addr(f, x_at + 32u * s);
                    bf[s][0] = f[0]; bf[s][1] = f[1];
                    if constexpr (NT == 1) { bf[s + 1][0] = f[2]; bf[s + 1][1] = f[3]; }
                    else { bf[s][2] = f[2]; bf[s][3] = f[3]; }
                }
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int i = 0; i < TW; ++i) ldmatrix_x4_addr(wf[s][i], (w_at ^ (32u * s)) + 2048u * i);
#pragma unroll
                for (int s = 0; s < 4; ++s)
#pragma unroll
                    for (int i = 0; i < TW; ++i)
#pragma unroll
                        for (int n = 0; n < NT; ++n) mma_bf16(acc[s & 1][i][n], wf[s][i], bf[s][2 * n], bf[s][2 * n + 1]);
                if (!whole) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[st]);
                }
            }
            if (!whole) {
                st += KG;
                if (st >= p.stages) { st -= p.stages; ++turn; }
            }
        }
        at -= k_blocks;
        if (c > 0) {
#pragma unroll
            for (int j = 0; j < 2; ++j) bias[j] = !TWO && p.bias != nullptr && split == 0 && lane + 32 * j < nf ? __ldg(p.bias + f0 + lane + 32 * j) : 0.f;
            if (EPI == EPI_ADD && p.splits == 1) read_sums(f0, nf);
        }
        consumers_sync();            // every warp is done with the weights, and the sums of the chunk before have been read
#pragma unroll
        for (int i = 0; i < TW; ++i)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float* to = part + ((kg * TT + half * TW + i) * TOK + n * 8 + 2 * t) * PITCH + g;
                to[0] = acc[0][i][n][0] + acc[1][i][n][0];
                to[PITCH] = acc[0][i][n][1] + acc[1][i][n][1];
                to[8] = acc[0][i][n][2] + acc[1][i][n][2];
                to[PITCH + 8] = acc[0][i][n][3] + acc[1][i][n][3];
            }
        if (dead && lane == 0 && !s_failed) { atomicCAS(&g_stream_error, 0, (1 << 16) | (int)(blockIdx.x & 0xffff)); s_failed = 1; }
        consumers_sync();
        if (s_failed) continue;
        // ---- this warp's tokens, a lane a row
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int tok = n * 8 + warp;
            if (tok >= p.tokens) continue;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int r = lane + 32 * j;
                if (r >= nf) continue;
                const int f = f0 + r;
                float v = 0.f, u = 0.f;
#pragma unroll
                for (int k = 0; k < KG; ++k) {
                    const float* from = part + ((k * TT + (r >> 4)) * TOK + tok) * PITCH + (r & 15);
                    v += from[0];
                    if (TWO) u += from[TW * TOK * PITCH];
                }
                v = v * scale[n] + bias[j];
                u *= scale[n];
                const size_t o = (size_t)tok * p.ldo + f;
                if (EPI == EPI_SWIGLU) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(__fdividef(v, 1.0f + __expf(-v)) * u);
                else if (EPI == EPI_GLU) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(nib_glu_fast(p.glu, v, u));
                else if (EPI == EPI_GEGLU) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(nib_geglu_fast(v, u));
                else if (p.splits > 1) atomicAdd((float*)p.out + o, v);
                else ((float*)p.out)[o] = x_old[n][j] + v;
            }
        }
    }
    if (tid == 0) nib_trace_mark(trace, trace_cap, NIB_TK_GEMM_STREAM, EPI, 2);
}

// ---------------------------------------------------------------------------------- host side
// Map of a row-major bfloat16 matrix [rows, k] (k a multiple of 64) as (64 of k, row, block of 64 k); box: `box_rows` rows of
// `box_blocks` blocks, a block's rows behind one another.
int make_block_map(CUtensorMap* map, const void* ptr, long long rows, long long k, int box_rows, int box_blocks) {
    NibEncodeTiledFn enc = nib_tensor_map_encoder();
    NIB_REQUIRE(enc != nullptr, "gemm (streamed): cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(k / 64)};
    cuuint64_t strides[2] = {(cuuint64_t)k * 2, 128};
    cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, (cuuint32_t)box_blocks};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    NIB_REQUIRE(r == CUDA_SUCCESS, "gemm (streamed): cuTensorMapEncodeTiled failed with code %d (rows=%lld k=%lld)", (int)r, rows, k);
    return 0;
}

// The maps of weights, which live as long as the model: what a map holds is its key and nothing else. (Made anew, and the attribute set, on
// every call, a step that is not replayed took the host 2,384 us instead of 2,354 for 12 tokens of the 24 layers of the 0.5B widths.)
struct BlockMapKey {
    const void* p; long long rows, k; int box_rows, box_blocks;
    bool operator==(const BlockMapKey& o) const { return p == o.p && rows == o.rows && k == o.k && box_rows == o.box_rows && box_blocks == o.box_blocks; }
};
struct BlockMapKeyHash {
    size_t operator()(const BlockMapKey& x) const {
        return std::hash<const void*>()(x.p) ^ (std::hash<long long>()(x.rows) * 31) ^ (std::hash<long long>()(x.k) * 131) ^ (size_t)(x.box_rows * 977 + x.box_blocks);
    }
};
std::unordered_map<BlockMapKey, CUtensorMap, BlockMapKeyHash> g_block_maps;
std::mutex g_block_map_mutex;

int block_map(CUtensorMap* map, const void* ptr, long long rows, long long k, int box_rows, int box_blocks) {
    std::lock_guard<std::mutex> lock(g_block_map_mutex);
    const BlockMapKey key{ptr, rows, k, box_rows, box_blocks};
    const auto it = g_block_maps.find(key);
    if (it != g_block_maps.end()) {
        *map = it->second;
        return 0;
    }
    if (make_block_map(map, ptr, rows, k, box_rows, box_blocks)) return 1;
    if (g_block_maps.size() >= 4096) g_block_maps.clear();
    g_block_maps.emplace(key, *map);
    return 0;
}

int up1024(int n) { return (n + 1023) & ~1023; }

struct Plan { int splits, split_blocks, rb, chunks, tw, kg; };

// Rows of a chunk: every SM the same number of chunks of the same size, at most 64 rows.
Plan plan_of(int N, int k_blocks, bool two, int splits, int sms) {
    Plan p;
    p.split_blocks = ceil_div(k_blocks, splits);
    p.splits = ceil_div(k_blocks, p.split_blocks);
    const int share = sms / p.splits;             // CTAs along N
    const int turns = ceil_div(N, (long long)share * MAX_RB);
    p.rb = ceil_div(N, (long long)share * turns);
    p.chunks = ceil_div(N, p.rb);
    const int tiles = ceil_div(p.rb, 16);
    p.kg = !two && tiles == 1 ? 8 : 4;
    p.tw = two || tiles == 1 ? tiles : ceil_div(tiles, 2);
    return p;
}

template <int NT, int TW, int KG, int EPI, bool NORM>
int launch(const void* W, StreamArgs p, int grid, int chunks, cudaStream_t stream) {
    constexpr int TT = TW * (WARPS / KG);
    constexpr int PART = KG * TT * NT * 8 * PITCH * 4;
    constexpr bool TWO = epi_dual(EPI);
    const int turns = ceil_div(chunks, grid / p.splits), room = (TWO ? WHOLE_GATED : WHOLE_SUM) - 1024 - 4352 - p.a_bytes;
    const auto set = [&](int kb) {      // blocks of a stage
        p.kb = kb;
        p.w_region = up1024(kb * p.rb * 128);
        p.w_stage = (TWO ? 2 : 1) * p.w_region;
    };
    // All weights at once and one wait if there is room; else a ring of blocks, a multiple of KG.
    set(p.split_blocks);
    p.stages = 1;
    if (turns > 1 || p.w_stage > room || p.kb > 256) {
        set(1);
        const int ring_room = RING_SMEM - 1024 - 4352 - p.a_bytes;
        p.stages = max(1, min((ring_room - (turns > 1 ? PART : 0)) / (p.w_stage + 16), ceil_div((long long)turns * p.split_blocks, KG) * KG) / KG) * KG;
    }
    const int ring = p.stages * p.w_stage;
    p.part_at = turns > 1 ? ring + p.a_bytes : 0;
    p.bars_at = ring + p.a_bytes + (turns > 1 ? PART : 0);
    if (turns == 1 && PART > p.bars_at) p.bars_at = PART;
    const size_t smem = (size_t)p.bars_at + 16 * p.stages + 1024 + 4096;        // (up to 31 rows past the last one are read as well)
    CUtensorMap mw;
    if (block_map(&mw, W, epi_dual(EPI) ? 2LL * p.N : p.N, p.K, p.rb, p.kb)) return 1;
    // (the most that any call takes: the attribute is the kernel's)
    static std::atomic<unsigned long long> configured{0};       // a bit a device
    int dev = 0;
    NIB_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        NIB_CUDA(cudaFuncSetAttribute(gemm_stream_kernel<NT, TW, KG, EPI, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_SMEM + 8 * 1024));
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    NIB_REQUIRE(smem <= RING_SMEM + 8 * 1024, "gemm (streamed): %zu bytes of shared memory", smem);
    NIB_CUDA(launch_pdl(gemm_stream_kernel<NT, TW, KG, EPI, NORM>, dim3(grid), dim3(THREADS), smem, stream, mw, p, nib_trace_buffer(), nib_trace_capacity()));
    return 0;
}

template <int NT, int EPI, bool NORM>
int launch_plan(const Plan& plan, const void* W, const StreamArgs& p, int grid, cudaStream_t stream) {
    if constexpr (epi_dual(EPI)) {
        switch (plan.tw) {
            case 1: return launch<NT, 1, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
            case 2: return launch<NT, 2, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
            case 3: return launch<NT, 3, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
            default: return launch<NT, 4, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
        }
    } else {
        if (plan.kg == 8) return launch<NT, 1, 8, EPI, NORM>(W, p, grid, plan.chunks, stream);
        if (plan.tw == 1) return launch<NT, 1, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
        return launch<NT, 2, 4, EPI, NORM>(W, p, grid, plan.chunks, stream);
    }
}

template <int EPI>
int launch_epi(const Plan& plan, const void* W, const StreamArgs& p, int grid, cudaStream_t stream) {
    if constexpr (epi_dual(EPI)) {
        if (p.gain != nullptr) return launch_plan<1, EPI, true>(plan, W, p, grid, stream);
    }
    return p.tokens <= 8 ? launch_plan<1, EPI, false>(plan, W, p, grid, stream) : launch_plan<2, EPI, false>(plan, W, p, grid, stream);
}

}  // namespace

// 1 if the kernel takes these operands: up to 16 tokens, K a multiple of 64, 16-byte aligned rows, and activations that fit. elem_bytes:
// 2 for a bfloat16 A operand, 4 for the 32-bit stream of the form with a norm.
NIB_API int nib_gemm_stream_supported(const void* A, const void* W, int tokens, int K, int lda, int elem_bytes, int splits) {
    if (tokens <= 0 || tokens > STREAM_TOKENS || K <= 0 || K % 64 || lda < K || (lda * elem_bytes) % 16 || splits < 1) return 0;
    if (((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return 0;
    if ((long long)tokens * ceil_div(K / 64, splits) * 128 > 64 * 1024) return 0;
    return nib_tensor_map_encoder() != nullptr;
}

// The error word of the kernel's bounded waits (0 = none); synchronises with the device and clears it.
NIB_API int nib_gemm_stream_error() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_stream_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_stream_error, &zero, sizeof(int));
    return v;
}

// Operands as nib_gemm_smallm, the gated epilogues (with a norm of up to 8 tokens before them if ``gain`` is there) and EPI_ADD. ``splits``: CTAs that share
// K (EPI_ADD only: their sums meet in memory, in any order).
NIB_API int nib_gemm_stream(const void* A, const void* W, const float* bias, void* out, int tokens, int N, int K, int lda, int ldo, int epi,
                            int splits, const float* gain, float eps, const NibGlu* glu, cudaStream_t stream) {
    NIB_REQUIRE(N > 0 && ldo >= N, "gemm (streamed): bad sizes tokens=%d N=%d K=%d", tokens, N, K);
    NIB_REQUIRE(nib_gemm_stream_supported(A, W, tokens, K, lda, gain ? 4 : 2, splits), "gemm (streamed): needs 1..16 tokens, K %% 64 == 0 and 16-byte aligned rows (tokens=%d K=%d)", tokens, K);
    NIB_REQUIRE(!epi_dual(epi) || bias == nullptr, "gemm (streamed): the gated epilogues take no bias");
    NIB_REQUIRE(epi != EPI_GLU || glu != nullptr, "gemm (streamed): the gated epilogue needs its constants");
    NIB_REQUIRE(splits == 1 || epi == EPI_ADD, "gemm (streamed): only sums are split along K");
    NIB_REQUIRE(gain == nullptr || (((uintptr_t)gain & 15) == 0 && epi_dual(epi) && tokens <= 8),
                "gemm (streamed): no norm before this epilogue or %d tokens, or a gain that is not 16-byte aligned", tokens);
    const int sms = nib_sm_count();
    NIB_REQUIRE(sms > 0 && splits <= sms, "gemm (streamed): no device, or too many splits");
    const Plan plan = plan_of(N, K / 64, epi_dual(epi), splits, sms);
    StreamArgs p{};
    p.A = A; p.bias = bias; p.out = out; p.tokens = tokens; p.N = N; p.K = K; p.lda = lda; p.ldo = ldo;
    p.rb = plan.rb; p.splits = plan.splits; p.split_blocks = plan.split_blocks;
    p.a_pitch = plan.split_blocks * 128 + 16;
    p.a_bytes = (tokens * p.a_pitch + 15) & ~15;
    p.gain = gain; p.eps = eps;
    if (glu != nullptr) p.glu = *glu;
    const int grid = min(plan.chunks, sms / plan.splits) * plan.splits;
    switch (epi) {
        case EPI_ADD: return launch_epi<EPI_ADD>(plan, W, p, grid, stream);
        case EPI_SWIGLU: return launch_epi<EPI_SWIGLU>(plan, W, p, grid, stream);
        case EPI_GLU: return launch_epi<EPI_GLU>(plan, W, p, grid, stream);
        case EPI_GEGLU: return launch_epi<EPI_GEGLU>(plan, W, p, grid, stream);
        default: nib_set_error("gemm (streamed): unknown epilogue %d", epi); return 1;
    }
}
