// The general attention kernel over the paged cache: any mix of prompt portions and decoded tokens, any head size up to
// 256, any page size, grouped kv heads, optional window. All arithmetic is 32-bit whatever the storage type. It is the
// attention of the true 32-bit path and the fallback of the bfloat16 path.
//
// A query at position p sees the keys at positions lo..p of its own request (lo = 0, or
// p - window + 1 with a window), read from the cache through the request's block table; the keys
// of this step were written there before. Keys are taken in blocks of 32 that start at absolute multiples of 32, four
// blocks to a segment with a running max and sum of its own (online softmax); the segments are merged in ascending order.
// So the result for a position does not depend on how the request was cut into steps, on what else is in the batch, nor on
// how many warps share the segments.
//
// A CTA takes one token and up to eight query heads that read the same keys: a key is fetched once for all of them (a warp
// per head fetched it for each, a row per lane with scattered 4-byte loads, and had only heads * tokens warps: bound by the
// latency of a chain of dependent blocks, one warp an SM when a single token decodes). Its warps take segments in turn; a
// warp copies a block's keys to shared memory with coalesced loads, a lane then owns a key for the scores and channels
// lane, lane + 32, ... of the output for the values.
//
// Formula: cpp/src/ops.cpp:206-270 (score = dot * scale, scale after the dot; max-subtracted exp;
// sum of p_j v_j / sum p_j); kv head = head / (heads / kv_heads): cpp/src/paged.cpp:171. Warp-level
// online softmax in the reference: cpp/src/cuda/cuda_backend.cu:113-178, 419-487.
#include "common.cuh"

constexpr int GEN_MAX_D = 256;
constexpr int GEN_MAX_WARPS = 8;
constexpr int GEN_SEGMENT = 128;         // keys of a segment
constexpr size_t GEN_SMEM = 200 * 1024;

// Floats of a CTA's shared memory: queries [d][R], running output [R][d], running (max, sum) twice, and per warp keys
// [32][pitch], weights [32][R], the segment's output [R][d] and its (max, sum).
__host__ __device__ constexpr int gen_pitch(int d) { return d | 1; }
__host__ __device__ constexpr int gen_warp_floats(int R, int d) { return (32 * gen_pitch(d) + 3) / 4 * 4 + 32 * R + R * d + 2 * R; }
__host__ __device__ constexpr int gen_cta_floats(int R, int d) { return 2 * R * d + 4 * R; }

// R floats from shared memory (16-byte aligned where R is a multiple of four).
template <int R>
__device__ __forceinline__ void gen_load(float (&v)[R], const float* p) {
    if constexpr (R % 4 == 0) {
#pragma unroll
        for (int i = 0; i < R; i += 4) {
            const float4 f = *reinterpret_cast<const float4*>(p + i);
            v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = p[i];
    }
}

template <typename T, int R, int DI>
__global__ void __launch_bounds__(GEN_MAX_WARPS * 32)
attention_generic_kernel(const T* __restrict__ qkv, int q_stride, T* __restrict__ out,
                         const int* __restrict__ positions, const int* __restrict__ req_index,
                         const int* __restrict__ block_table, int bt_stride, int page_size,
                         const T* __restrict__ k_pages, const T* __restrict__ v_pages, int num_pages,
                         int heads, int kv_heads, int head_dim, float scale, int window) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int group = heads / kv_heads, sets = (group + R - 1) / R;
    const int set = blockIdx.x % sets, kvh = (blockIdx.x / sets) % kv_heads, token = blockIdx.x / (sets * kv_heads);
    const int h0 = kvh * group + set * R, n_heads = min(R, group - set * R);
    const int pitch = gen_pitch(head_dim);
    float* q_s = smem;                                  // [head_dim][R]
    float* tot = q_s + R * head_dim;                    // [R][head_dim]
    float* ml = tot + R * head_dim;                     // two copies of [R][2]
    float* base = ml + 4 * R;
    float* k_s = base + (size_t)warp * gen_warp_floats(R, head_dim);
    float* p_s = k_s + (32 * pitch + 3) / 4 * 4;        // [32][R]
    pdl_launch_dependents();
    pdl_wait();
    const int pos = positions[token];
    const int* bt = block_table + (size_t)req_index[token] * bt_stride;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;

    const T* q = qkv + (size_t)token * q_stride + (size_t)h0 * head_dim;
    for (int e = threadIdx.x; e < R * head_dim; e += blockDim.x) {
        const int r = e / head_dim, d = e % head_dim;
        q_s[d * R + r] = r < n_heads ? Elem<T>::load(q + e) : 0.f;
        tot[e] = 0.f;
    }
    if (threadIdx.x < R) {
        ml[2 * threadIdx.x] = -INFINITY;
        ml[2 * threadIdx.x + 1] = 0.f;
    }
    __syncthreads();

    int round = 0;
    for (int seg0 = lo / GEN_SEGMENT; seg0 * GEN_SEGMENT <= pos; seg0 += warps, ++round) {
        float m_run[R], l_run[R], acc[R][DI];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m_run[r] = -INFINITY;
            l_run[r] = 0.f;
#pragma unroll
            for (int i = 0; i < DI; ++i) acc[r][i] = 0.f;
        }
        const int k_end = (seg0 + warp + 1) * GEN_SEGMENT;
        for (int kb = max((seg0 + warp) * GEN_SEGMENT, lo / 32 * 32); kb <= pos && kb < k_end; kb += 32) {
            const int j = kb + lane;
            int row = -1;       // this lane's key: its row in the pages
            if (j >= lo && j <= pos) {
                const int page = bt[j / page_size];
                if (page >= 0 && page < num_pages) row = (page * kv_heads + kvh) * page_size + j % page_size;
            }
            __syncwarp();
#pragma unroll 1
            for (int j0 = 0; j0 < 32; j0 += 8) {
                float v[8][DI];
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    const int rj = __shfl_sync(0xffffffffu, row, j0 + jj);
                    const T* kr = k_pages + (long long)max(rj, 0) * head_dim;
#pragma unroll
                    for (int i = 0; i < DI; ++i) v[jj][i] = rj >= 0 && lane + 32 * i < head_dim ? Elem<T>::load(kr + lane + 32 * i) : 0.f;
                }
#pragma unroll
                for (int jj = 0; jj < 8; ++jj)
#pragma unroll
                    for (int i = 0; i < DI; ++i)
                        if (lane + 32 * i < head_dim) k_s[(j0 + jj) * pitch + lane + 32 * i] = v[jj][i];
            }
            __syncwarp();
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 8
            for (int d = 0; d < head_dim; ++d) {
                const float kd = k_s[lane * pitch + d];
                float qd[R];
                gen_load<R>(qd, q_s + d * R);
#pragma unroll
                for (int r = 0; r < R; ++r) s[r] = fmaf(qd[r], kd, s[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                s[r] = row >= 0 ? s[r] * scale : -INFINITY;
                const float m_new = fmaxf(m_run[r], warp_max(s[r]));
                const float p = s[r] == -INFINITY ? 0.f : expf(s[r] - m_new);
                const float corr = m_run[r] == -INFINITY ? 0.f : expf(m_run[r] - m_new);
                l_run[r] = l_run[r] * corr + warp_sum(p);
#pragma unroll
                for (int i = 0; i < DI; ++i) acc[r][i] *= corr;
                m_run[r] = m_new;
                p_s[lane * R + r] = p;
            }
            __syncwarp();
#pragma unroll 1
            for (int j0 = 0; j0 < 32; j0 += 8) {
                float v[8][DI];
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    const int rj = __shfl_sync(0xffffffffu, row, j0 + jj);
                    const T* vr = v_pages + (long long)max(rj, 0) * head_dim;
#pragma unroll
                    for (int i = 0; i < DI; ++i) v[jj][i] = rj >= 0 && lane + 32 * i < head_dim ? Elem<T>::load(vr + lane + 32 * i) : 0.f;
                }
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    float p[R];
                    gen_load<R>(p, p_s + (j0 + jj) * R);
#pragma unroll
                    for (int r = 0; r < R; ++r)
#pragma unroll
                        for (int i = 0; i < DI; ++i) acc[r][i] = p[r] == 0.f ? acc[r][i] : fmaf(p[r], v[jj][i], acc[r][i]);
                }
            }
        }
        // this round's segments, merged in ascending order
        float* o_s = p_s + 32 * R;                      // [R][head_dim]
        float* s_ml = o_s + R * head_dim;               // [R][2]
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int i = 0; i < DI; ++i)
                if (lane + 32 * i < head_dim) o_s[r * head_dim + lane + 32 * i] = acc[r][i];
            if (lane == 0) {
                s_ml[2 * r] = m_run[r];
                s_ml[2 * r + 1] = l_run[r];
            }
        }
        __syncthreads();
        const float* ml_in = ml + (round & 1) * 2 * R;
        float* ml_out = ml + ((round + 1) & 1) * 2 * R;
        const int live = min(warps, pos / GEN_SEGMENT - seg0 + 1);
        const float* o_0 = base + (o_s - k_s);
        for (int e = threadIdx.x; e < R * head_dim; e += blockDim.x) {
            const int r = e / head_dim;
            float m = ml_in[2 * r], l = ml_in[2 * r + 1], o = tot[e];
            for (int w = 0; w < live; ++w) {
                const float* other = o_0 + (size_t)w * gen_warp_floats(R, head_dim);
                const float mw = other[R * head_dim + 2 * r], lw = other[R * head_dim + 2 * r + 1];
                if (mw == -INFINITY) continue;          // no key of the segment is seen
                const float m_new = fmaxf(m, mw);
                const float a = m == -INFINITY ? 0.f : expf(m - m_new), b = expf(mw - m_new);
                o = o * a + other[e] * b;
                l = l * a + lw * b;
                m = m_new;
            }
            tot[e] = o;
            if (e % head_dim == 0) {
                ml_out[2 * r] = m;
                ml_out[2 * r + 1] = l;
            }
        }
        __syncthreads();
    }
    T* o = out + (size_t)token * heads * head_dim + (size_t)h0 * head_dim;
    for (int e = threadIdx.x; e < n_heads * head_dim; e += blockDim.x) {
        const float l = ml[(round & 1) * 2 * R + 2 * (e / head_dim) + 1];
        Elem<T>::store(o + e, l > 0.f ? tot[e] * (1.0f / l) : 0.f);
    }
}

// qkv: rows of q_stride elements whose first heads*head_dim are the (rotated) queries.
// out: [m_tokens, heads*head_dim]. Pages: [num_pages, kv_heads, page_size, head_dim]. max_keys: no token sees more keys than
// that (how many warps share a token's keys is chosen by it; results do not depend on it).
template <typename T, int R, int DI>
static int launch_generic(const void* qkv, int q_stride, void* out, const int* positions, const int* req_index, const int* block_table,
                          int bt_stride, int page_size, const void* k_pages, const void* v_pages, int num_pages, int m_tokens, int heads,
                          int kv_heads, int head_dim, float scale, int window, int max_keys, cudaStream_t stream) {
    const long long blocks = (long long)m_tokens * kv_heads * ceil_div(heads / kv_heads, R);
    NIB_REQUIRE(blocks <= 0x7fffffffLL, "attention: too many tokens for one launch");
    // one warp per segment, as many as eight; of a prompt's many tokens each gets fewer: their CTAs fill the GPU anyway
    int warps = max(1, min(blocks >= 8 * 148 ? 2 : GEN_MAX_WARPS, ceil_div(max_keys, GEN_SEGMENT)));
    const size_t cta = sizeof(float) * gen_cta_floats(R, head_dim), per_warp = sizeof(float) * gen_warp_floats(R, head_dim);
    while (warps > 1 && cta + warps * per_warp > GEN_SMEM) --warps;
    const size_t smem = cta + warps * per_warp;
    if (smem > 48 * 1024) NIB_CUDA(cudaFuncSetAttribute(attention_generic_kernel<T, R, DI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    NIB_CUDA(launch_pdl(attention_generic_kernel<T, R, DI>, dim3((unsigned)blocks), dim3(32 * warps), smem, stream, (const T*)qkv, q_stride,
                        (T*)out, positions, req_index, block_table, bt_stride, page_size, (const T*)k_pages, (const T*)v_pages, num_pages,
                        heads, kv_heads, head_dim, scale, window));
    NIB_LAUNCH_CHECK();
    return 0;
}

template <typename T, int R>
static int launch_generic_d(const void* qkv, int q_stride, void* out, const int* positions, const int* req_index, const int* block_table,
                            int bt_stride, int page_size, const void* k_pages, const void* v_pages, int num_pages, int m_tokens, int heads,
                            int kv_heads, int head_dim, float scale, int window, int max_keys, cudaStream_t stream) {
    auto* run = head_dim <= 64 ? launch_generic<T, R, 2> : head_dim <= 128 ? launch_generic<T, R, 4> : launch_generic<T, R, 8>;
    return run(qkv, q_stride, out, positions, req_index, block_table, bt_stride, page_size, k_pages, v_pages, num_pages, m_tokens, heads,
               kv_heads, head_dim, scale, window, max_keys, stream);
}

NIB_API int nib_attention_generic(const void* qkv, int q_stride, void* out, const int* positions,
                                  const int* req_index, const int* block_table, int bt_stride, int page_size,
                                  const void* k_pages, const void* v_pages, int num_pages, int m_tokens,
                                  int heads, int kv_heads, int head_dim, float scale, int window, int dtype, int max_keys,
                                  cudaStream_t stream) {
    NIB_REQUIRE(m_tokens >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0, "attention: bad head counts %d / %d", heads, kv_heads);
    NIB_REQUIRE(head_dim > 0 && head_dim <= GEN_MAX_D, "attention: head_dim %d is outside 1..%d", head_dim, GEN_MAX_D);
    NIB_REQUIRE(page_size > 0 && num_pages > 0 && window >= 0, "attention: bad page_size/num_pages/window");
    NIB_REQUIRE((long long)num_pages * kv_heads * page_size <= 0x7fffffffLL, "attention: more rows of keys than a 32-bit index counts");
    NIB_REQUIRE(dtype == NIB_F32 || dtype == NIB_BF16, "attention: unknown dtype %d", dtype);
    if (m_tokens == 0) return 0;
    const int group = heads / kv_heads;
    const bool f32 = dtype == NIB_F32;
    auto* run = group == 1 ? (f32 ? launch_generic_d<float, 1> : launch_generic_d<__nv_bfloat16, 1>)
        : group <= 2 ? (f32 ? launch_generic_d<float, 2> : launch_generic_d<__nv_bfloat16, 2>)
        : group <= 4 ? (f32 ? launch_generic_d<float, 4> : launch_generic_d<__nv_bfloat16, 4>)
                     : (f32 ? launch_generic_d<float, 8> : launch_generic_d<__nv_bfloat16, 8>);
    return run(qkv, q_stride, out, positions, req_index, block_table, bt_stride, page_size, k_pages, v_pages, num_pages, m_tokens, heads,
               kv_heads, head_dim, scale, window, max_keys, stream);
}
