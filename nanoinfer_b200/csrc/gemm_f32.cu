// The matrix products of the true 32-bit path: C[M,N] = A[M,K] . W[N,K]^T (+ bias) in floats on the CUDA cores, any M, N,
// K, no reduced-precision matrix mode.
//
// ONE ORDER OF SUMMATION for every M, so that a row's result does not depend on how many rows the call has (the reference
// guarantees the same: cpp/src/cuda/cuda_gemm.cu:37-45): k is cut into chunks of 256 at absolute multiples of 256; a chunk
// is one chain of fused multiply-adds in ascending k that starts at 0; the chunks' sums are added up in ascending order.
// Against one chain over all of K that is also the smaller error, and it is what lets threads, warps and CTAs share K. Two
// kernels give these same sums bit for bit:
//
// * gemm_f32_rows_kernel, up to 16 tokens: bound by reading W once. A CTA owns 8 or 16 rows of W and a stretch of K that
//   fits its shared memory whole, so everything it will ever read is in flight before anything is waited for (asynchronous
//   16-byte copies, sent before the wait for the kernel before it); then a thread per (row, chunk) walks its chain, eight
//   rows side by side in a warp (rows lie one 16-byte unit off a multiple of eight apart: no bank conflicts; the tokens'
//   values are broadcast). A long K is shared by the CTAs of a cluster, whose chunk sums the first one adds up in order.
// * gemm_f32_tile_kernel, more tokens: bound by the multiply-adds. Tiles of 64 x 64, 4 x 4 outputs a thread, the next 16 k
//   fetched into registers under this block's arithmetic. Few tiles: the chunks are shared by the CTAs of a cluster.
//
// Measured on B200 at the 0.5B widths (us; before: a thread per output and one chain over all of K): one token, gate/up 189 -> 10.0
// (35 MB: 5.2 at the copy bandwidth), down 445 -> 4.4 (with the output projection), the head's 545 MB 111 (82); 128 tokens,
// gate/up 91, the sums into the residual stream 42. With chunks of 128 the one-token kernels are faster (8.2 and 92: half the chain
// a thread walks), but a product of K <= 256 keeps the bits of one ascending chain with 256.
//
// Epilogues: STORE and F32 (out = sum + bias), ADD (out += sum + bias: the residual sum), and the gated ones on W rows n and
// n + N: SWIGLU silu(gate) * up with silu(g) = g / (1 + exp(-g)) (cpp/src/ops.cpp:86-93), GLU (with limits and constants),
// GEGLU (gelu(gate) * up).
#include "pipeline.cuh"

using namespace nibp;

namespace {

constexpr int CHUNK = 256;

__device__ __forceinline__ void copy16(unsigned dst, const float* src, int bytes) {      // bytes < 16: the rest is zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy4(unsigned dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int EPI>
__device__ __forceinline__ void finish(float* out, size_t o, float v, float u, const NibGlu& glu) {
    if (EPI == EPI_ADD)
        out[o] += v;
    else if (EPI == EPI_GLU)
        out[o] = nib_glu_exact(glu, v, u);
    else if (EPI == EPI_GEGLU)
        out[o] = nib_geglu_exact(v, u);
    else if (EPI == EPI_SWIGLU)
        out[o] = v / (1.0f + expf(-v)) * u;
    else
        out[o] = v;
}

// `count` rows of `len` floats each (the last `len - valid` of a row zeros), row r from src + r * stride, to dst + r * pitch.
// Rows from `rows` on are zeros. All of a CTA's 128 threads take part.
__device__ __forceinline__ void send_rows(float* dst, int pitch, const float* src, size_t stride, int rows, int count, int len, int valid, bool wide) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < count; r += 4) {
        const float* row = src + (r < rows ? r * stride : 0);
        const int have = r < rows ? valid : 0;
        const unsigned to = smem_u32(dst + (size_t)r * pitch);
        if (wide)
            for (int k = 4 * lane; k < len; k += 128) copy16(to + 4 * k, have > k ? row + k : src, have > k ? 16 : 0);
        else
            for (int k = lane; k < len; k += 32) copy4(to + 4 * k, have > k ? row + k : src, have > k ? 4 : 0);
    }
}

// ------------------------------------------------------------------------------------------------ few tokens
constexpr int ROWS_THREADS = 128;

// Rows of W a CTA holds: 8 * RB (gated: gate rows n0.. and up rows N + n0..); MT tokens at a time, TT of them per thread.
template <int EPI, int RB, int MT>
__global__ void __launch_bounds__(ROWS_THREADS)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out,
                     int M, int N, int K, int lda, int ldo, int chunks_per_cta, int wide, const NibGlu glu) {
    constexpr bool DUAL = epi_dual(EPI);
    constexpr int TT = MT < 4 ? MT : 4;
    constexpr int FEATURES = DUAL ? 8 : 8 * RB;         // outputs of a CTA per token
    extern __shared__ __align__(16) float smem[];
    const int ranks = (int)cluster_size(), rank = (int)cluster_rank();
    const int n0 = (blockIdx.x / ranks) * FEATURES;
    const int all_chunks = (K + CHUNK - 1) / CHUNK;
    const int c_lo = rank * chunks_per_cta, nch = min(chunks_per_cta, all_chunks - c_lo);      // nch >= 1: see the launch
    const int k_lo = c_lo * CHUNK, len = nch * CHUNK;
    const int pitch = chunks_per_cta * CHUNK + 4;
    float* w_s = smem;                                   // [8 RB][pitch]
    float* a_s = w_s + 8 * RB * pitch;                   // [MT][pitch]
    float* part = a_s + MT * pitch;                      // [MT][chunks_per_cta][8 RB]
    const int tid = threadIdx.x;

    pdl_launch_dependents();
    const int valid = min(len, K - k_lo);
    send_rows(w_s, pitch, W + (size_t)n0 * K + k_lo, (size_t)K, min(FEATURES, N - n0), FEATURES, len, valid, wide);
    if (DUAL) send_rows(w_s + 8 * pitch, pitch, W + (size_t)(N + n0) * K + k_lo, (size_t)K, min(8, N - n0), 8, len, valid, wide);
    pdl_wait();
    for (int m0 = 0; m0 < M; m0 += MT) {
        send_rows(a_s, pitch, A + (size_t)m0 * lda + k_lo, (size_t)lda, min(MT, M - m0), MT, len, valid, wide);
        copies_done();
        __syncthreads();
        for (int t = tid; t < 8 * nch * (MT / TT); t += ROWS_THREADS) {
            const int r = t & 7, c = (t >> 3) % nch, g = (t >> 3) / nch * TT;
            const float4* wp = reinterpret_cast<const float4*>(w_s + r * pitch + c * CHUNK);
            const float4* ap = reinterpret_cast<const float4*>(a_s + g * pitch + c * CHUNK);
            float acc[RB][TT];
#pragma unroll
            for (int j = 0; j < RB; ++j)
#pragma unroll
                for (int i = 0; i < TT; ++i) acc[j][i] = 0.f;
#pragma unroll 4
            for (int q = 0; q < CHUNK / 4; ++q) {
                float4 w[RB];
#pragma unroll
                for (int j = 0; j < RB; ++j) w[j] = wp[j * 2 * pitch + q];      // 8 rows further: 8 * pitch floats
#pragma unroll
                for (int i = 0; i < TT; ++i) {
                    const float4 a = ap[i * (pitch / 4) + q];
#pragma unroll
                    for (int j = 0; j < RB; ++j)
                        acc[j][i] = fmaf(a.w, w[j].w, fmaf(a.z, w[j].z, fmaf(a.y, w[j].y, fmaf(a.x, w[j].x, acc[j][i]))));
                }
            }
#pragma unroll
            for (int j = 0; j < RB; ++j)
#pragma unroll
                for (int i = 0; i < TT; ++i) part[((g + i) * chunks_per_cta + c) * (8 * RB) + 8 * j + r] = acc[j][i];
        }
        if (ranks > 1)
            cluster_sync();
        else
            __syncthreads();
        if (rank == 0) {
            for (int t = tid; t < FEATURES * MT; t += ROWS_THREADS) {
                const int f = t % FEATURES, i = t / FEATURES;
                if (m0 + i >= M || n0 + f >= N) continue;
                float v = 0.f, u = 0.f;
                for (int s = 0; s < ranks; ++s) {
                    const int n = min(chunks_per_cta, all_chunks - s * chunks_per_cta);
                    const float* p = part + i * chunks_per_cta * (8 * RB) + f;
                    if (s == 0) {
                        for (int c = 0; c < n; ++c) {
                            v += p[c * (8 * RB)];
                            if (DUAL) u += p[c * (8 * RB) + 8];
                        }
                    } else {
                        const unsigned peer = peer_smem(p, s);
#pragma unroll 4
                        for (int c = 0; c < n; ++c) {
                            v += ld_peer_f32(peer + 4 * c * (8 * RB));
                            if (DUAL) u += ld_peer_f32(peer + 4 * (c * (8 * RB) + 8));
                        }
                    }
                }
                if (!DUAL && bias != nullptr) v += bias[n0 + f];
                finish<EPI>(out, (size_t)(m0 + i) * ldo + n0 + f, v, u, glu);
            }
        }
        if (ranks > 1)
            cluster_sync();      // the other CTAs' sums have been read: they may be overwritten, or their CTA may end
        else
            __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------ more tokens
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, TILE_THREADS = 256, TILE_PITCH = 68;

// A thread's share of a 64 x 16 block of a row-major matrix: four k of one row, zeros outside.
__device__ __forceinline__ float4 fetch_block(const float* src, size_t stride, int rows, int k, int K, bool wide) {
    const int r = threadIdx.x >> 2, kk = k + 4 * (threadIdx.x & 3);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows && kk < K) {
        const float* p = src + (size_t)r * stride + kk;
        if (wide) {
            v = *reinterpret_cast<const float4*>(p);
        } else {
            v.x = p[0];
            if (kk + 1 < K) v.y = p[1];
            if (kk + 2 < K) v.z = p[2];
            if (kk + 3 < K) v.w = p[3];
        }
    }
    return v;
}
__device__ __forceinline__ void put_block(float (*dst)[TILE_PITCH], const float4& v) {
    const int r = threadIdx.x >> 2, kk = 4 * (threadIdx.x & 3);
    dst[kk][r] = v.x;
    dst[kk + 1][r] = v.y;
    dst[kk + 2][r] = v.z;
    dst[kk + 3][r] = v.w;
}

template <int EPI, bool SPLIT>
__global__ void __launch_bounds__(TILE_THREADS, 2)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out,
                     int M, int N, int K, int lda, int ldo, int chunks_per_cta, int wide, const NibGlu glu) {
    constexpr bool DUAL = epi_dual(EPI);
    constexpr int ACCS = DUAL ? 2 : 1;
    __shared__ __align__(16) float As[2][BK][TILE_PITCH];
    __shared__ __align__(16) float Ws[2][BK][TILE_PITCH];
    __shared__ __align__(16) float Us[DUAL ? 2 : 1][DUAL ? BK : 1][TILE_PITCH];
    extern __shared__ __align__(16) float part[];        // SPLIT: [chunks_per_cta][ACCS][BM][BN], this CTA's chunk sums

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int ranks = SPLIT ? (int)cluster_size() : 1, rank = SPLIT ? (int)cluster_rank() : 0;
    const int n0 = (blockIdx.x / ranks) * BN, m0 = blockIdx.y * BM;
    const int all_chunks = (K + CHUNK - 1) / CHUNK;
    const int c_lo = SPLIT ? rank * chunks_per_cta : 0, c_hi = SPLIT ? min(c_lo + chunks_per_cta, all_chunks) : all_chunks;
    const int k_hi = min(K, c_hi * CHUNK);
    const int a_rows = min(BM, M - m0), w_rows = min(BN, N - n0);
    const float* a_src = A + (size_t)m0 * lda;
    const float* w_src = W + (size_t)n0 * K;
    const float* u_src = W + (size_t)(N + n0) * K;

    float acc[ACCS][TM][TN], tot[SPLIT ? 1 : ACCS][SPLIT ? 1 : TM][SPLIT ? 1 : TN];
#pragma unroll
    for (int h = 0; h < ACCS; ++h)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                acc[h][i][j] = 0.f;
                if (!SPLIT) tot[SPLIT ? 0 : h][SPLIT ? 0 : i][SPLIT ? 0 : j] = 0.f;
            }

    pdl_launch_dependents();
    int k = c_lo * CHUNK;
    float4 fw = fetch_block(w_src, K, w_rows, k, k_hi, wide), fu;
    if (DUAL) fu = fetch_block(u_src, K, w_rows, k, k_hi, wide);
    pdl_wait();
    float4 fa = fetch_block(a_src, lda, a_rows, k, k_hi, wide);
    int buf = 0;
    for (int c = c_lo; c < c_hi; ++c) {
#pragma unroll 1
        for (int b = 0; b < CHUNK / BK; ++b) {
            put_block(As[buf], fa);
            put_block(Ws[buf], fw);
            if (DUAL) put_block(Us[DUAL ? buf : 0], fu);
            __syncthreads();
            k += BK;
            if (k < k_hi) {
                fa = fetch_block(a_src, lda, a_rows, k, k_hi, wide);
                fw = fetch_block(w_src, K, w_rows, k, k_hi, wide);
                if (DUAL) fu = fetch_block(u_src, K, w_rows, k, k_hi, wide);
            }
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[TM], w[TN], u[TN];
                *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * TM]);
                *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(&Ws[buf][kk][tx * TN]);
                if (DUAL) *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(&Us[DUAL ? buf : 0][DUAL ? kk : 0][tx * TN]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        acc[0][i][j] = fmaf(a[i], w[j], acc[0][i][j]);
                        if (DUAL) acc[ACCS - 1][i][j] = fmaf(a[i], u[j], acc[ACCS - 1][i][j]);
                    }
            }
            buf ^= 1;
            if (k >= k_hi) break;       // the rest of the chunk is zeros, which change no sum
        }
#pragma unroll
        for (int h = 0; h < ACCS; ++h)
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                if (SPLIT) {
                    *reinterpret_cast<float4*>(part + (((size_t)(c - c_lo) * ACCS + h) * BM + ty * TM + i) * BN + tx * TN) =
                        make_float4(acc[h][i][0], acc[h][i][1], acc[h][i][2], acc[h][i][3]);
                } else {
#pragma unroll
                    for (int j = 0; j < TN; ++j) tot[SPLIT ? 0 : h][SPLIT ? 0 : i][SPLIT ? 0 : j] += acc[h][i][j];
                }
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[h][i][j] = 0.f;
            }
    }
    if (SPLIT) {
        cluster_sync();
        for (int t = rank * TILE_THREADS + tid; t < BM * BN / 4; t += ranks * TILE_THREADS) {
            const int i = t / (BN / 4), j = 4 * (t % (BN / 4));
            if (m0 + i >= M || n0 + j >= N) continue;
            float v[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s < ranks; ++s) {
                const int n = min(chunks_per_cta, all_chunks - s * chunks_per_cta);
                const unsigned peer = peer_smem(part + i * BN + j, s);
#pragma unroll 4
                for (int c = 0; c < n; ++c) {
                    const float4 p = ld_peer_f32x4(peer + 4u * (unsigned)(c * ACCS * BM * BN));
                    v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
                    if (DUAL) {
                        const float4 q = ld_peer_f32x4(peer + 4u * (unsigned)((c * ACCS + 1) * BM * BN));
                        u[0] += q.x; u[1] += q.y; u[2] += q.z; u[3] += q.w;
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n0 + j + e < N) {
                    if (!DUAL && bias != nullptr) v[e] += bias[n0 + j + e];
                    finish<EPI>(out, (size_t)(m0 + i) * ldo + n0 + j + e, v[e], u[e], glu);
                }
        }
        cluster_sync();      // a CTA's shared memory stays until everyone has read it
    } else {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + ty * TM + i;
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int n = n0 + tx * TN + j;
                if (n >= N) continue;
                float v = tot[0][SPLIT ? 0 : i][SPLIT ? 0 : j];
                if (!DUAL && bias != nullptr) v += bias[n];
                finish<EPI>(out, (size_t)m * ldo + n, v, DUAL ? tot[SPLIT ? 0 : ACCS - 1][SPLIT ? 0 : i][SPLIT ? 0 : j] : 0.f, glu);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------ launches
struct Args {
    const float *A, *W, *bias;
    float* out;
    int M, N, K, lda, ldo, wide;
    NibGlu glu;
    cudaStream_t stream;
};

// `most`: what the kernel's largest launch takes. The attribute belongs to the kernel, not to a launch: set to a call's own size it
// would be lowered under a larger launch that another thread has just allowed.
template <typename Kernel>
int launch_cluster(Kernel kernel, dim3 grid, int threads, size_t smem, size_t most, int ranks, const Args& a, int chunks_per_cta) {
    if (smem > 16 * 1024) NIB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));   // (beside up to 26 KB of static)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = a.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nib_pdl_enabled() ? 2 : 1;
    NIB_CUDA(cudaLaunchKernelEx(&cfg, kernel, a.A, a.W, a.bias, a.out, a.M, a.N, a.K, a.lda, a.ldo, chunks_per_cta, a.wide, a.glu));
    NIB_LAUNCH_CHECK();
    return 0;
}

constexpr int ROWS_MAX_TOKENS = 16;
constexpr int ROWS_CHUNKS = 5;            // of a CTA while that needs no more than eight CTAs for K
constexpr size_t ROWS_SMEM = 200 * 1024, TILE_SMEM = 160 * 1024;

template <int EPI, int RB>
size_t rows_smem(int mt, int cpc) { return sizeof(float) * ((size_t)(8 * RB + mt) * (cpc * CHUNK + 4) + (size_t)mt * cpc * 8 * RB); }

template <int EPI, int RB>
int launch_rows(const Args& a, int cpc, int ranks) {
    constexpr int FEATURES = epi_dual(EPI) ? 8 : 8 * RB;
    const dim3 grid(ceil_div(a.N, FEATURES) * ranks);
    if (a.M == 1) return launch_cluster(gemm_f32_rows_kernel<EPI, RB, 1>, grid, ROWS_THREADS, rows_smem<EPI, RB>(1, cpc), ROWS_SMEM, ranks, a, cpc);
    if (a.M == 2) return launch_cluster(gemm_f32_rows_kernel<EPI, RB, 2>, grid, ROWS_THREADS, rows_smem<EPI, RB>(2, cpc), ROWS_SMEM, ranks, a, cpc);
    if (a.M <= 4) return launch_cluster(gemm_f32_rows_kernel<EPI, RB, 4>, grid, ROWS_THREADS, rows_smem<EPI, RB>(4, cpc), ROWS_SMEM, ranks, a, cpc);
    return launch_cluster(gemm_f32_rows_kernel<EPI, RB, 8>, grid, ROWS_THREADS, rows_smem<EPI, RB>(8, cpc), ROWS_SMEM, ranks, a, cpc);
}

template <int EPI>
int launch_f32(const Args& a) {
    constexpr bool DUAL = epi_dual(EPI);
    const int chunks = ceil_div(a.K, CHUNK);
    // Not where a chunk is mostly the zeros that fill it up, which a thread of the rows kernel walks like the rest and the tile kernel
    // leaves out: 20,000 rows of 64 k, 16 tokens, 25 us by rows and 10.9 by tiles (a thread per output: 13.9), 4 tokens 12.6 and 10.6; 24
    // rows of 16 k, one token, 3.7 and 2.5. Of 128 k: 896 rows, 16 tokens, 9.1 and 6.9, 8 tokens 5.6 and 6.6.
    const int short_k = a.M > 8 ? 128 : a.M > 2 ? 64 : 32;
    if (a.M <= ROWS_MAX_TOKENS && a.K > short_k) {
        int ranks = min(8, ceil_div(chunks, ROWS_CHUNKS));
        const int cpc = ceil_div(chunks, ranks);
        ranks = ceil_div(chunks, cpc);          // every CTA of a cluster has a chunk
        const int mt = a.M == 1 ? 1 : a.M == 2 ? 2 : a.M <= 4 ? 4 : 8;
        const bool two = DUAL || a.N >= 16 * 2 * 148;       // sixteen rows a CTA once that still gives every SM two CTAs
        if (two && rows_smem<EPI, 2>(mt, cpc) <= ROWS_SMEM) return launch_rows<EPI, 2>(a, cpc, ranks);
        if constexpr (!DUAL) {
            if (rows_smem<EPI, 1>(mt, cpc) <= ROWS_SMEM) return launch_rows<EPI, 1>(a, cpc, ranks);
        }
    }
    const int tiles = ceil_div(a.N, BN) * ceil_div(a.M, BM);
    // CTAs that share the chunks of a tile: as many as keep all CTAs on the GPU at once, two an SM; with more tiles than SMs none,
    // unless their last turn would leave most SMs idle and there are four chunks to share. us by a CTA a tile and by four, 64 tokens:
    // 152 tiles of 896 k, 65 and 57, gated 104 and 86; of 4,864, 340 and 245, gated 545 and 450; 184 tiles of 2,048, 144 and 119; but 152 of
    // 300 k 25 and (by two) 39, of 520 (by three) 40 and 43, 190 tiles of 1,536 108 and 106, gated 176 and 173, 196 gated 176 and 184. (By
    // eight: 152 gated tiles of 4,864 609, 184 721.)
    int ranks = 2 * 148 / tiles;
    if (tiles > 148 && 8 * tiles < 5 * 2 * 148 && chunks >= 4) ranks = 4;
    ranks = max(1, min(min(8, chunks), ranks));
    const int cpc = ceil_div(chunks, ranks);
    ranks = ceil_div(chunks, cpc);
    const size_t smem = sizeof(float) * (size_t)cpc * (DUAL ? 2 : 1) * BM * BN;
    const dim3 grid(ceil_div(a.N, BN) * (smem <= TILE_SMEM ? ranks : 1), ceil_div(a.M, BM));
    if (ranks > 1 && smem <= TILE_SMEM) return launch_cluster(gemm_f32_tile_kernel<EPI, true>, grid, TILE_THREADS, smem, TILE_SMEM, ranks, a, cpc);
    return launch_cluster(gemm_f32_tile_kernel<EPI, false>, grid, TILE_THREADS, (size_t)0, (size_t)0, 1, a, chunks);
}

}  // namespace

// A [M, K] with row stride lda; W [N, K] (gated: [2N, K], gate rows then up rows); out [M, N] floats with row stride ldo.
// epi: 0 store, 1 add, 2 store float, 3 swiglu, 5 the gated form with the constants glu, 6 geglu.
NIB_API int nib_gemm_f32(const float* A, const float* W, const float* bias, float* out, int M, int N, int K, int lda, int ldo, int epi,
                         const NibGlu* glu, cudaStream_t stream) {
    NIB_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldo >= N, "gemm: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
    NIB_REQUIRE(!epi_dual(epi) || bias == nullptr, "gemm: the gated epilogues take no bias");
    NIB_REQUIRE(epi != EPI_GLU || glu != nullptr, "gemm: the gated epilogue needs its constants");
    if (M == 0) return 0;
    NIB_REQUIRE(ceil_div(M, BM) <= 65535, "gemm: M=%d is too large for one launch", M);
    const int wide = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
    const Args a = {A, W, bias, out, M, N, K, lda, ldo, wide, glu != nullptr ? *glu : NibGlu{}, stream};
    switch (epi) {
        case EPI_STORE:
        case EPI_F32: return launch_f32<EPI_F32>(a);
        case EPI_ADD: return launch_f32<EPI_ADD>(a);
        case EPI_SWIGLU: return launch_f32<EPI_SWIGLU>(a);
        case EPI_GLU: return launch_f32<EPI_GLU>(a);
        case EPI_GEGLU: return launch_f32<EPI_GEGLU>(a);
        default: nib_set_error("gemm: unknown epilogue %d", epi); return 1;
    }
}
