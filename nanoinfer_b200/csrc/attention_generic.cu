// The general attention kernel over the paged cache: any mix of prompt portions and decoded tokens, any head size up to
// 256, any page size, grouped kv heads, optional window. All arithmetic is 32-bit whatever the storage type. It is the
// attention of the true 32-bit path and the fallback of the bfloat16 path.
//
// A query at position p sees the keys at positions lo..p of its own request (lo = 0, or
// p - window + 1 with a window), read from the cache through the request's block table; the keys
// of this step were written there before. Keys are taken in blocks of 32 that start at absolute multiples of 32; every
// block has a maximum, a sum and an output of its own, and they are merged in ascending order. So the result for a position
// does not depend on how the request was cut into steps, on what else is in the batch, nor on how many warps share the
// blocks.
//
// A CTA takes one token and up to eight query heads that read the same keys: a key is fetched once for all of them. Its
// warps take blocks in turn; a warp sends for all keys and values of its block at once (a block costs one trip to memory:
// that latency is what bounds a token with a short context), then a lane owns a key for the scores and channels lane,
// lane + 32, ... of the output for the values.
//
// Formula: cpp/src/ops.cpp:206-270 (score = dot * scale, scale after the dot; max-subtracted exp;
// sum of p_j v_j / sum p_j); kv head = head / (heads / kv_heads): cpp/src/paged.cpp:171. Warp-level
// online softmax in the reference: cpp/src/cuda/cuda_backend.cu:113-178, 419-487.
#include "common.cuh"

constexpr int GEN_MAX_D = 256;
constexpr int GEN_MAX_WARPS = 8;
constexpr int GEN_BLOCK = 32;            // keys of a block: a lane each
constexpr size_t GEN_SMEM = 200 * 1024;

// Floats of a CTA's shared memory: queries [R][pitch], running output [R][pitch], running (max, sum) twice; per warp keys
// and values [32][pitch], weights [32][R], the block's (max, sum). Rows are padded with zeros to a multiple of four and lie
// an odd number of 16-byte units apart: eight lanes that read a row each meet no bank conflict. A block's output takes
// the place of its keys.
__host__ __device__ constexpr int gen_pitch(int d) { return ((d + 3) / 4 | 1) * 4; }
__host__ __device__ constexpr int gen_warp_floats(int R, int d) { return 2 * GEN_BLOCK * gen_pitch(d) + GEN_BLOCK * R + (2 * R + 3) / 4 * 4; }
__host__ __device__ constexpr int gen_cta_floats(int R, int d) { return 2 * R * gen_pitch(d) + 4 * R; }

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

// The block's rows of keys or values into shared memory as floats, by one warp: row jj is row `row` of lane jj in the pages
// (below 0: zeros). 32-bit rows that start on 16 bytes go as asynchronous copies, as many rows at a time as the warp's lanes
// cover: nothing waits for them here. (What lies behind a row is read, but what comes of it is not.)
template <typename T>
__device__ __forceinline__ void gen_send_rows(float* dst, const T* pages, long long row, int d, int pitch, bool wide, int lane) {
    if (sizeof(T) == 4 && wide) {
        const int units = d >> 2, per_row = units <= 8 ? 8 : units <= 16 ? 16 : 32, u0 = lane & (per_row - 1);
#pragma unroll 4
        for (int r = lane / per_row; r < GEN_BLOCK; r += 32 / per_row) {
            const long long rj = __shfl_sync(0xffffffffu, row, r);
            const T* src = pages + max(rj, 0ll) * d;
            const unsigned to = (unsigned)__cvta_generic_to_shared(dst + r * pitch);
            for (int u = u0; u < units; u += per_row)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to + 16 * u), "l"(src + 4 * u), "r"(rj >= 0 ? 16 : 0) : "memory");
        }
    } else {
        for (int r = 0; r < GEN_BLOCK; ++r) {
            const long long rj = __shfl_sync(0xffffffffu, row, r);
            const T* src = pages + max(rj, 0ll) * d;
            for (int i = lane; i < pitch; i += 32) dst[r * pitch + i] = rj >= 0 && i < d ? Elem<T>::load(src + i) : 0.f;
        }
    }
}

template <typename T, int R, int DI>
__global__ void __launch_bounds__(GEN_MAX_WARPS * 32)
attention_generic_kernel(const T* __restrict__ qkv, int q_stride, T* __restrict__ out,
                         const int* __restrict__ positions, const int* __restrict__ req_index,
                         const int* __restrict__ block_table, int bt_stride, int page_size,
                         const T* __restrict__ k_pages, const T* __restrict__ v_pages, int num_pages,
                         int heads, int kv_heads, int head_dim, float scale, int window, int wide) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int group = heads / kv_heads, sets = (group + R - 1) / R;
    const int set = blockIdx.x % sets, kvh = (blockIdx.x / sets) % kv_heads, token = blockIdx.x / (sets * kv_heads);
    const int h0 = kvh * group + set * R, n_heads = min(R, group - set * R);
    const int pitch = gen_pitch(head_dim);
    float* q_s = smem;                                  // [R][pitch]
    float* tot = q_s + R * pitch;                       // [R][pitch]
    float* ml = tot + R * pitch;                        // two copies of [R][2]
    float* base = ml + 4 * R;
    float* k_s = base + (size_t)warp * gen_warp_floats(R, head_dim);      // [32][pitch]; then the block's output [R][pitch]
    float* v_s = k_s + GEN_BLOCK * pitch;               // [32][pitch]
    float* p_s = v_s + GEN_BLOCK * pitch;               // [32][R]
    float* b_ml = p_s + GEN_BLOCK * R;                  // [R][2]
    pdl_launch_dependents();
    pdl_wait();
    const int pos = positions[token];
    const int* bt = block_table + (size_t)req_index[token] * bt_stride;
    const int lo = window > 0 ? max(0, pos - window + 1) : 0;

    const T* q = qkv + (size_t)token * q_stride + (size_t)h0 * head_dim;
    for (int e = threadIdx.x; e < R * pitch; e += blockDim.x) {
        const int r = e / pitch, d = e % pitch;
        q_s[e] = r < n_heads && d < head_dim ? Elem<T>::load(q + r * head_dim + d) : 0.f;
        tot[e] = 0.f;
    }
    if (threadIdx.x < R) {
        ml[2 * threadIdx.x] = -INFINITY;
        ml[2 * threadIdx.x + 1] = 0.f;
    }
    __syncthreads();

    const int b_last = pos / GEN_BLOCK;
    int round = 0;
    for (int b0 = lo / GEN_BLOCK; b0 <= b_last; b0 += warps, ++round) {
        if (b0 + warp <= b_last) {
            const int j = (b0 + warp) * GEN_BLOCK + lane;
            long long row = -1;       // this lane's key: its row in the pages
            if (j >= lo && j <= pos) {
                const int page = bt[j / page_size];
                if (page >= 0 && page < num_pages) row = ((long long)page * kv_heads + kvh) * page_size + j % page_size;
            }
            gen_send_rows(k_s, k_pages, row, head_dim, pitch, wide, lane);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            gen_send_rows(v_s, v_pages, row, head_dim, pitch, wide, lane);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncwarp();
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 4
            for (int d = 0; d < head_dim; d += 4) {
                const float4 kd = *reinterpret_cast<const float4*>(k_s + lane * pitch + d);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 qd = *reinterpret_cast<const float4*>(q_s + r * pitch + d);
                    s[r] = fmaf(qd.w, kd.w, fmaf(qd.z, kd.z, fmaf(qd.y, kd.y, fmaf(qd.x, kd.x, s[r]))));
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                s[r] = row >= 0 ? s[r] * scale : -INFINITY;
                const float m = warp_max(s[r]);
                const float p = s[r] == -INFINITY ? 0.f : expf(s[r] - m);
                const float l = warp_sum(p);
                p_s[lane * R + r] = p;
                if (lane == 0) {
                    b_ml[2 * r] = m;
                    b_ml[2 * r + 1] = l;
                }
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            float acc[R][DI];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < DI; ++i) acc[r][i] = 0.f;
#pragma unroll 4
            for (int jj = 0; jj < GEN_BLOCK; ++jj) {
                float p[R], v[DI];
                gen_load<R>(p, p_s + jj * R);
#pragma unroll
                for (int i = 0; i < DI; ++i) v[i] = lane + 32 * i < pitch ? v_s[jj * pitch + lane + 32 * i] : 0.f;
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int i = 0; i < DI; ++i) acc[r][i] = p[r] == 0.f ? acc[r][i] : fmaf(p[r], v[i], acc[r][i]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < DI; ++i)
                    if (lane + 32 * i < pitch) k_s[r * pitch + lane + 32 * i] = acc[r][i];
        }
        __syncthreads();
        // this round's blocks, merged in ascending order
        const float* ml_in = ml + (round & 1) * 2 * R;
        float* ml_out = ml + ((round + 1) & 1) * 2 * R;
        const int live = min(warps, b_last - b0 + 1);
        for (int e = threadIdx.x; e < R * pitch; e += blockDim.x) {
            const int r = e / pitch;
            float m = ml_in[2 * r], l = ml_in[2 * r + 1], o = tot[e];
            for (int w = 0; w < live; ++w) {
                const float* other = base + (size_t)w * gen_warp_floats(R, head_dim);
                const float* other_ml = other + 2 * GEN_BLOCK * pitch + GEN_BLOCK * R;
                const float mw = other_ml[2 * r], lw = other_ml[2 * r + 1];
                if (mw == -INFINITY && lw == 0.f) continue;          // no key of the block is seen (or only scores of -inf); a sum of NaN goes on
                const float m_new = fmaxf(m, mw);
                const float a = m == -INFINITY ? 0.f : expf(m - m_new), b = expf(mw - m_new);
                o = o * a + other[e] * b;
                l = l * a + lw * b;
                m = m_new;
            }
            tot[e] = o;
            if (e % pitch == 0) {
                ml_out[2 * r] = m;
                ml_out[2 * r + 1] = l;
            }
        }
        __syncthreads();
    }
    T* o = out + (size_t)token * heads * head_dim + (size_t)h0 * head_dim;
    for (int e = threadIdx.x; e < n_heads * head_dim; e += blockDim.x) {
        const int r = e / head_dim, d = e % head_dim;
        const float l = ml[(round & 1) * 2 * R + 2 * r + 1];
        Elem<T>::store(o + e, tot[r * pitch + d] * (l > 0.f ? 1.0f / l : 0.f));       // a row with an undefined score stays NaN
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
    // a warp per block of keys, as many as eight; of a prompt's many tokens each gets fewer: their CTAs fill the GPU anyway
    int warps = max(1, min(blocks >= 8 * 148 ? 4 : GEN_MAX_WARPS, ceil_div(max_keys, GEN_BLOCK)));
    const size_t cta = sizeof(float) * gen_cta_floats(R, head_dim), per_warp = sizeof(float) * gen_warp_floats(R, head_dim);
    while (warps > 1 && cta + warps * per_warp > GEN_SMEM) --warps;
    const size_t smem = cta + warps * per_warp;
    const int wide = head_dim % 4 == 0 && ((uintptr_t)k_pages | (uintptr_t)v_pages) % 16 == 0;
    // the most that any call takes: the attribute is the kernel's, and a call's own size would lower it under another thread's launch
    if (smem > 48 * 1024) NIB_CUDA(cudaFuncSetAttribute(attention_generic_kernel<T, R, DI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM));
    NIB_CUDA(launch_pdl(attention_generic_kernel<T, R, DI>, dim3((unsigned)blocks), dim3(32 * warps), smem, stream, (const T*)qkv, q_stride,
                        (T*)out, positions, req_index, block_table, bt_stride, page_size, (const T*)k_pages, (const T*)v_pages, num_pages,
                        heads, kv_heads, head_dim, scale, window, wide));
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
    NIB_REQUIRE(dtype == NIB_F32 || dtype == NIB_BF16, "attention: unknown dtype %d", dtype);
    if (m_tokens == 0) return 0;
    // As many heads a CTA as still leaves a CTA for every SM: few tokens take fewer (a warp's arithmetic on a block of keys is
    // what bounds them: 17 us for one token of 14 heads and 140 keys with eight heads a CTA), many share the keys they fetch.
    const long long units = (long long)m_tokens * kv_heads;
    int group = heads / kv_heads, share = 1;
    while (share < 8 && share < group && units * ceil_div(group, share) > 148) share *= 2;
    const bool f32 = dtype == NIB_F32;
    group = share;
    auto* run = group == 1 ? (f32 ? launch_generic_d<float, 1> : launch_generic_d<__nv_bfloat16, 1>)
        : group <= 2 ? (f32 ? launch_generic_d<float, 2> : launch_generic_d<__nv_bfloat16, 2>)
        : group <= 4 ? (f32 ? launch_generic_d<float, 4> : launch_generic_d<__nv_bfloat16, 4>)
                     : (f32 ? launch_generic_d<float, 8> : launch_generic_d<__nv_bfloat16, 8>);
    return run(qkv, q_stride, out, positions, req_index, block_table, bt_stride, page_size, k_pages, v_pages, num_pages, m_tokens, heads,
               kv_heads, head_dim, scale, window, max_keys, stream);
}
