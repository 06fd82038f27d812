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
// warps take blocks in turn; a warp sends for all keys and values of its block at once, as they are stored (a block costs one
// trip to memory: that latency is what bounds a token with a short context, and how many blocks an SM has under way a prompt),
// then a lane owns a key for the scores and channels of the output for the values. (Sending for the next block's keys under
// the sums of this one's values was slower: one token of 777 keys, 14 heads of 64, 32-bit, 27.5 us instead of 23.7.)
//
// us, with a warp per (token, head) that reads keys from global memory / with rows of 32-bit numbers that bfloat16 was copied into
// element by element / this: bfloat16, 8 heads of 72, a prompt of 1,024 tokens, 757 / 3,896 / 300; 64 tokens of 500 keys,
// 218 / 299 / 25; 16 tokens, 8 and 2 heads of 100, 14.6 / 44.8 / 8.1; 32-bit, 8 heads of 72, 1,024 tokens, 873 / 1,039 / 620; one token of
// 777 keys, 14 and 2 heads of 64, 323 / 22.3 / 19.9. Rows of an odd number of elements go as 32-bit words: 8 heads of 33 and 16 tokens,
// 9.1 / 26 / 8.2. With an odd width and one query head a kv head the copies' instructions are what a long prompt waits for (a
// fourth of the bytes each): 8 heads of 129 and 1,024 tokens, bfloat16, 1,134 / - / 1,725 (one token of 777 keys, 458 / - / 65; 64 of 500
// keys, 348 / - / 184; eight heads on two kv heads, 1,142 / - / 614), 32-bit 1,052 / - / 3,587 (458 / - / 85; 345 / - / 212).
//
// Formula: cpp/src/ops.cpp:206-270 (score = dot * scale, scale after the dot; max-subtracted exp;
// sum of p_j v_j / sum p_j); kv head = head / (heads / kv_heads): cpp/src/paged.cpp:171. Warp-level
// online softmax in the reference: cpp/src/cuda/cuda_backend.cu:113-178, 419-487.
#include "common.cuh"

constexpr int GEN_MAX_D = 256;
constexpr int GEN_MAX_WARPS = 8;
constexpr int GEN_BLOCK = 32;            // keys of a block: a lane each
constexpr size_t GEN_SMEM = 200 * 1024;

// A CTA's shared memory: queries [R][pitch] floats, running output [R][pitch], running (max, sum) twice; per warp keys and values
// [32][row] in the storage type, weights [32][R], the block's (max, sum). Rows are padded with zeros to whole 16-byte units of the
// storage type and lie an odd number of them apart: eight lanes that read a row each meet no bank conflict. A block's output,
// [R][pitch] floats, takes the place of its keys (R <= 8, and a row has at least as many bytes as a pitch has floats).
// (`unit`, see gen_send_rows(): 0 takes room for one element more.)
template <typename T> __host__ __device__ constexpr int gen_row(int d, int unit) { return (int)(((d + (unit == 0)) * sizeof(T) + 15) / 16 | 1) * 16; }      // bytes
template <typename T> __host__ __device__ constexpr int gen_filled(int d) { return (int)((d * sizeof(T) + 15) / 16 * (16 / sizeof(T))); }  // elements
template <typename T> __host__ __device__ constexpr int gen_pitch(int d) { return (gen_filled<T>(d) / 4 | 1) * 4; }              // floats
template <typename T> __host__ __device__ constexpr int gen_warp_bytes(int R, int d, int unit) {
    return 2 * GEN_BLOCK * gen_row<T>(d, unit) + 4 * (GEN_BLOCK * R + (2 * R + 3) / 4 * 4);
}
template <typename T> __host__ __device__ constexpr int gen_cta_bytes(int R, int d) { return 4 * (2 * R * gen_pitch<T>(d) + 4 * R); }

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

// The block's rows of keys or values into shared memory, by one warp: row jj is row `row` of lane jj in the pages (below 0:
// zeros). Asynchronous copies of U bytes, 32 consecutive ones of the block at a time: nothing waits for them here.
template <typename T, int U>
__device__ __forceinline__ void gen_send_units(unsigned char* dst, int pitch, const T* pages, long long row, int d, int lane) {
    const int units = gen_filled<T>(d) * (int)sizeof(T) / U, have = U == 16 ? units : d * (int)sizeof(T) / U;
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    const int step_r = 32 / units, step_u = 32 - step_r * units;
    int r = lane / units, u = lane - r * units;
#pragma unroll 4
    for (int k = 0; k < units; ++k) {
        const long long rj = __shfl_sync(0xffffffffu, row, r);
        const char* src = reinterpret_cast<const char*>(pages + max(rj, 0ll) * d);
        const bool there = rj >= 0 && u < have;
        if (U == 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to + r * pitch + U * u), "l"(src + U * u), "r"(there ? U : 0) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n"
                         ::"r"(to + r * pitch + U * u), "l"(there ? src + U * u : src), "n"(U), "r"(there ? U : 0) : "memory");
        r += step_r;
        u += step_u;
        if (u >= units) {
            u -= units;
            ++r;
        }
    }
}
// Rows of bfloat16 that begin at any element (an odd width, say): the 32-bit words that a row lies in, its first element in the upper
// half of the first one if the row begins in the middle of a word (the lower half is the row's before it; no word is read that holds
// nothing of the row). gen_align_rows() moves such a row down by an element. A lane reads and writes its own words only and gets the upper half
// of a word from the lane above.
__device__ __forceinline__ void gen_send_words(unsigned char* dst, int pitch, const __nv_bfloat16* pages, long long row, int d, int lane) {
    const int words = max(gen_filled<__nv_bfloat16>(d), d + 2) / 2, step_r = 32 / words, step_u = 32 - step_r * words;
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    int r = lane / words, u = lane - r * words;
#pragma unroll 4
    for (int k = 0; k < words; ++k) {
        const long long rj = __shfl_sync(0xffffffffu, row, r);
        const uintptr_t begin = reinterpret_cast<uintptr_t>(pages + max(rj, 0ll) * d), first = begin & ~(uintptr_t)3;
        const int bytes = rj >= 0 ? max(0, min(4, (int)(begin - first) + 2 * d - 4 * u)) : 0;       // 2: the word's upper half is not the row's
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n"
                     ::"r"(to + r * pitch + 4 * u), "l"(first + (bytes > 0 ? 4 * u : 0)), "r"(bytes) : "memory");
        r += step_r;
        u += step_u;
        if (u >= words) {
            u -= words;
            ++r;
        }
    }
}
__device__ __forceinline__ void gen_align_rows(unsigned char* dst, int pitch, const __nv_bfloat16* pages, long long row, int d, int lane) {
    const int words = max(gen_filled<__nv_bfloat16>(d), d + 2) / 2;
    unsigned odd = __ballot_sync(0xffffffffu, row >= 0 && (reinterpret_cast<uintptr_t>(pages + max(row, 0ll) * d) & 2) != 0);
    constexpr int TURNS = (GEN_MAX_D + 2 + 63) / 64;        // of 32 words
    for (; odd != 0; odd &= odd - 1) {
        unsigned* w = reinterpret_cast<unsigned*>(dst + (__ffs(odd) - 1) * pitch);
        unsigned v[TURNS + 1];
#pragma unroll
        for (int i = 0; i <= TURNS; ++i) v[i] = lane + 32 * i < words ? w[lane + 32 * i] : 0u;
#pragma unroll
        for (int i = 0; i < TURNS; ++i) {
            if (32 * i >= words) break;
            const unsigned next = __shfl_sync(0xffffffffu, lane == 0 ? v[i + 1] : v[i], lane + 1);      // (lane 31's: lane 0's next word)
            if (lane + 32 * i < words) w[lane + 32 * i] = v[i] >> 16 | next << 16;
        }
    }
    __syncwarp();
}
// `unit`: the largest of 16, 8 and 4 bytes that the rows are made of; 0 where there is none.
template <typename T>
__device__ __forceinline__ void gen_send_rows(unsigned char* dst, int pitch, const T* pages, long long row, int d, int unit, int lane) {
    if (unit == 16) {
        gen_send_units<T, 16>(dst, pitch, pages, row, d, lane);
    } else if (unit == 8) {
        gen_send_units<T, 8>(dst, pitch, pages, row, d, lane);
    } else if (sizeof(T) == 4 || unit == 4) {
        gen_send_units<T, 4>(dst, pitch, pages, row, d, lane);
    } else {
        if constexpr (sizeof(T) == 2) gen_send_words(dst, pitch, pages, row, d, lane);
    }
}

// Two bfloat16 of a 32-bit word.
__device__ __forceinline__ float gen_low(unsigned w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float gen_high(unsigned w) { return __uint_as_float(w & 0xffff0000u); }

// s[r] += q[r] . k over the 16 bytes of a key at `k`, in ascending order of the elements; queries `pitch` floats apart.
template <typename T, int R>
__device__ __forceinline__ void gen_dot(float (&s)[R], const float* q, int pitch, const unsigned char* k) {
    float kd[16 / sizeof(T)];
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(kd) = *reinterpret_cast<const float4*>(k);
    } else {
        const uint4 w = *reinterpret_cast<const uint4*>(k);
        kd[0] = gen_low(w.x); kd[1] = gen_high(w.x); kd[2] = gen_low(w.y); kd[3] = gen_high(w.y);
        kd[4] = gen_low(w.z); kd[5] = gen_high(w.z); kd[6] = gen_low(w.w); kd[7] = gen_high(w.w);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < (int)(16 / sizeof(T)); i += 4) {
            const float4 qd = *reinterpret_cast<const float4*>(q + r * pitch + i);
            s[r] = fmaf(qd.w, kd[i + 3], fmaf(qd.z, kd[i + 2], fmaf(qd.y, kd[i + 1], fmaf(qd.x, kd[i], s[r]))));
        }
}
// The output channel that a lane's i-th sum is of: 32 apart, or pairs 64 apart where a word holds two values.
template <typename T> __device__ __forceinline__ int gen_channel(int i, int lane) {
    return sizeof(T) == 4 ? lane + 32 * i : 2 * lane + 64 * (i >> 1) + (i & 1);
}
template <typename T, int DI>
__device__ __forceinline__ void gen_values(float (&v)[DI], const unsigned char* row, int filled, int lane) {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < DI; ++i) v[i] = lane + 32 * i < filled ? reinterpret_cast<const float*>(row)[lane + 32 * i] : 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < DI; i += 2) {
            const unsigned w = 2 * lane + 32 * i < filled ? reinterpret_cast<const unsigned*>(row)[lane + 16 * i] : 0u;
            v[i] = gen_low(w);
            v[i + 1] = gen_high(w);
        }
    }
}

template <typename T, int R, int DI>
__global__ void __launch_bounds__(GEN_MAX_WARPS * 32, R <= 2 ? 4 : 2)
attention_generic_kernel(const T* __restrict__ qkv, int q_stride, T* __restrict__ out,
                         const int* __restrict__ positions, const int* __restrict__ req_index,
                         const int* __restrict__ block_table, int bt_stride, int page_size,
                         const T* __restrict__ k_pages, const T* __restrict__ v_pages, int num_pages,
                         int heads, int kv_heads, int head_dim, float scale, int window, int unit) {
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int group = heads / kv_heads, sets = (group + R - 1) / R;
    const int set = blockIdx.x % sets, kvh = (blockIdx.x / sets) % kv_heads, token = blockIdx.x / (sets * kv_heads);
    const int h0 = kvh * group + set * R, n_heads = min(R, group - set * R);
    const int pitch = gen_pitch<T>(head_dim), key_row = gen_row<T>(head_dim, unit), filled = gen_filled<T>(head_dim);
    const int warp_floats = gen_warp_bytes<T>(R, head_dim, unit) / 4;
    float* q_s = smem;                                  // [R][pitch]
    float* tot = q_s + R * pitch;                       // [R][pitch]
    float* ml = tot + R * pitch;                        // two copies of [R][2]
    float* base = ml + 4 * R;                           // per warp: keys (then the block's output), values, weights, (max, sum)
    float* o_s = base + (size_t)warp * warp_floats;     // [R][pitch]
    unsigned char* k_s = reinterpret_cast<unsigned char*>(o_s);      // [32][key_row]
    unsigned char* v_s = k_s + GEN_BLOCK * key_row;
    float* p_s = reinterpret_cast<float*>(v_s + GEN_BLOCK * key_row);      // [32][R]
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
            gen_send_rows(k_s, key_row, k_pages, row, head_dim, unit, lane);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            gen_send_rows(v_s, key_row, v_pages, row, head_dim, unit, lane);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncwarp();
            if constexpr (sizeof(T) == 2)
                if (unit == 0) gen_align_rows(k_s, key_row, k_pages, row, head_dim, lane);
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 4
            for (int d = 0; d < filled; d += 16 / sizeof(T)) gen_dot<T, R>(s, q_s + d, pitch, k_s + lane * key_row + d * sizeof(T));
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
            if constexpr (sizeof(T) == 2)
                if (unit == 0) gen_align_rows(v_s, key_row, v_pages, row, head_dim, lane);
            float acc[R][DI];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < DI; ++i) acc[r][i] = 0.f;
#pragma unroll 4
            for (int jj = 0; jj < GEN_BLOCK; ++jj) {
                float p[R], v[DI];
                gen_load<R>(p, p_s + jj * R);
                gen_values<T, DI>(v, v_s + jj * key_row, filled, lane);
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int i = 0; i < DI; ++i) acc[r][i] = p[r] == 0.f ? acc[r][i] : fmaf(p[r], v[i], acc[r][i]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int i = 0; i < DI; ++i)
                    if (gen_channel<T>(i, lane) < pitch) o_s[r * pitch + gen_channel<T>(i, lane)] = acc[r][i];
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
                const float* other = base + (size_t)w * warp_floats;
                const float* other_ml = other + GEN_BLOCK * key_row / 2 + GEN_BLOCK * R;
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
    const uintptr_t bytes = (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)(head_dim * sizeof(T));      // what rows begin at and are long
    const int unit = bytes % 16 == 0 ? 16 : bytes % 8 == 0 ? 8 : bytes % 4 == 0 ? 4 : 0;
    const size_t cta = gen_cta_bytes<T>(R, head_dim), per_warp = gen_warp_bytes<T>(R, head_dim, unit);
    while (warps > 1 && cta + warps * per_warp > GEN_SMEM) --warps;
    const size_t smem = cta + warps * per_warp;
    // the most that any call takes: the attribute is the kernel's, and a call's own size would lower it under another thread's launch
    if (smem > 48 * 1024) NIB_CUDA(cudaFuncSetAttribute(attention_generic_kernel<T, R, DI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM));
    NIB_CUDA(launch_pdl(attention_generic_kernel<T, R, DI>, dim3((unsigned)blocks), dim3(32 * warps), smem, stream, (const T*)qkv, q_stride,
                        (T*)out, positions, req_index, block_table, bt_stride, page_size, (const T*)k_pages, (const T*)v_pages, num_pages,
                        heads, kv_heads, head_dim, scale, window, unit));
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
