// Choosing the next token on the device from 32-bit logits [rows, vocab].
//
// Pipeline, in the reference's order (nanoinfer/sampling.py:126-151, cpp/src/sampling.cpp:90-108):
// repetition penalty on the raw logits -> greedy (first index of the maximum) when temperature is 0
// -> logits / temperature -> top-k (ties at the k-th value stay) -> top-p (a token is dropped iff the
// probability of those before it, in descending order, exceeds p; the first stays) -> softmax ->
// draw. The draw is an inverse CDF in vocabulary order with a uniform number made from (seed, number of
// tokens generated), here up to 64 rows and by the host beyond, the same one: a request's tokens do not depend on
// the batch it was sampled in. The reference samples on the host (cpp/python/ni/scheduler.py:89-147).
#include "pipeline.cuh"

// ---------------------------------------------------------------------------------- penalty
// seen: flat list of distinct token ids per row, seen_start[row]..seen_start[row+1]. pending (may be null): one more id
// per row that is still on the device (the token of a step whose result the host has not read yet); it is penalised
// too unless the row's list holds it already, so no logit is penalised twice.
__global__ void penalty_kernel(float* __restrict__ logits, int vocab, const int* __restrict__ seen,
                               const int* __restrict__ seen_start, const float* __restrict__ penalty,
                               const int* __restrict__ pending) {
    __shared__ int listed;
    const int row = blockIdx.x;
    const float p = penalty[row];
    if (p == 1.0f) return;
    const int extra = pending ? pending[row] : -1;
    if (threadIdx.x == 0) listed = 0;
    __syncthreads();
    float* l = logits + (size_t)row * vocab;
    for (int i = seen_start[row] + threadIdx.x; i < seen_start[row + 1]; i += blockDim.x) {
        const int id = seen[i];
        if (id < 0 || id >= vocab) continue;
        if (id == extra) listed = 1;
        const float s = l[id];
        l[id] = s > 0.f ? s / p : s * p;
    }
    __syncthreads();
    if (threadIdx.x == 0 && extra >= 0 && extra < vocab && !listed) {
        const float s = l[extra];
        l[extra] = s > 0.f ? s / p : s * p;
    }
}

NIB_API int nib_repetition_penalty(float* logits, int rows, int vocab, const int* seen, const int* seen_start,
                                   const float* penalty, const int* pending, cudaStream_t stream) {
    NIB_REQUIRE(rows >= 0 && vocab > 0, "penalty: bad sizes");
    if (rows == 0) return 0;
    penalty_kernel<<<rows, 256, 0, stream>>>(logits, vocab, seen, seen_start, penalty, pending);
    NIB_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------------- argmax
constexpr int SAMP_THREADS = 1024;

__device__ __forceinline__ void argmax_combine(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}

// First index of the maximum of each row. NaN entries never win.
__global__ void __launch_bounds__(SAMP_THREADS)
argmax_kernel(const float* __restrict__ logits, int vocab, int* __restrict__ out) {
    __shared__ float sv[SAMP_THREADS / 32];
    __shared__ int si[SAMP_THREADS / 32];
    const float* l = logits + (size_t)blockIdx.x * vocab;
    float v = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = threadIdx.x; i < vocab; i += SAMP_THREADS) argmax_combine(v, idx, l[i], i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        argmax_combine(v, idx, ov, oi);
    }
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = v; si[threadIdx.x >> 5] = idx; }
    __syncthreads();
    if (threadIdx.x < 32) {
        v = sv[threadIdx.x];
        idx = si[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            argmax_combine(v, idx, ov, oi);
        }
        if (threadIdx.x == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
    }
}

NIB_API int nib_argmax(const float* logits, int rows, int vocab, int* out, cudaStream_t stream) {
    NIB_REQUIRE(rows >= 0 && vocab > 0, "argmax: bad sizes");
    if (rows == 0) return 0;
    argmax_kernel<<<rows, SAMP_THREADS, 0, stream>>>(logits, vocab, out);
    NIB_LAUNCH_CHECK();
    return 0;
}

// The same with every row cut into `chunks` pieces that different CTAs scan: a few rows of a large
// vocabulary otherwise keep a few SMs busy and the rest idle. A piece's best (value, index) is packed
// into 64 bits (order-preserving bits of the value above the complement of the index), so the maximum
// of the packed words is the largest value at its first index, in whatever order they are compared. The
// CTA that finishes a row's last piece (a counter per row, left at zero) writes the result.
__device__ __forceinline__ unsigned long long argmax_pack(float x, int i) {
    if (x != x) return 0ull;                                   // NaN never wins
    const unsigned b = __float_as_uint(x);
    const unsigned key = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return ((unsigned long long)key << 32) | (unsigned long long)(0xffffffffu - (unsigned)i);
}

__global__ void __launch_bounds__(256)
argmax_chunk_kernel(const float* __restrict__ logits, int vocab, int chunk, int chunks, unsigned long long* __restrict__ part,
                    int* __restrict__ counters, int* __restrict__ out, unsigned long long* trace, int trace_cap) {
    __shared__ unsigned long long s_best[8];
    __shared__ int s_last;
    if (threadIdx.x == 0) nib_trace_mark(trace, trace_cap, NIB_TK_ARGMAX, 0, 1);
    const int row = blockIdx.y, cid = blockIdx.x;
    const float* l = logits + (size_t)row * vocab;
    const int begin = cid * chunk, end = min(vocab, begin + chunk);
    unsigned long long best = 0ull;
    for (int i = begin + threadIdx.x; i < end; i += 256) best = max(best, argmax_pack(l[i], i));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) best = max(best, s_best[w]);
        part[(size_t)row * chunks + cid] = best;
        __threadfence();
        s_last = (atomicAdd(&counters[row], 1) == chunks - 1) ? 1 : 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    best = 0ull;
    for (int c = threadIdx.x; c < chunks; c += 256) best = max(best, __ldcg(part + (size_t)row * chunks + c));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) best = max(best, s_best[w]);
        out[row] = best == 0ull ? 0 : (int)(0xffffffffu - (unsigned)(best & 0xffffffffull));
        counters[row] = 0;                                      // ready for the next launch
    }
}

// scratch: rows * chunks 64-bit words; counters: rows ints that are zero between launches.
NIB_API int nib_argmax_chunked(const float* logits, int rows, int vocab, int* out, int chunks, unsigned long long* scratch,
                               int* counters, cudaStream_t stream) {
    NIB_REQUIRE(rows >= 0 && vocab > 0 && chunks >= 1 && chunks <= 65535 && rows <= 65535, "argmax: bad sizes");
    NIB_REQUIRE(scratch != nullptr && counters != nullptr, "argmax (chunked): scratch and counters are needed");
    if (rows == 0) return 0;
    const int chunk = ceil_div(vocab, chunks);
    argmax_chunk_kernel<<<dim3(chunks, rows), 256, 0, stream>>>(logits, vocab, chunk, chunks, scratch, counters, out, nib_trace_buffer(), nib_trace_capacity());
    NIB_LAUNCH_CHECK();
    return 0;
}

// ---------------------------------------------------------------------------------- sampling
// Order-preserving map from float to unsigned: larger float <-> larger key.
__device__ __forceinline__ unsigned key_of(float x) {
    const unsigned b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float float_of_key(unsigned k) {
    const unsigned b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(b);
}

// Scaled probabilities are histogrammed as 64-bit fixed point so that sums do not depend on the
// order in which threads add (integer addition is associative): sampling stays reproducible.
constexpr float FIX_ONE = 1099511627776.0f;  // 2^40

// A mass into the three histograms of 14-bit chunks. 64-bit adds to shared memory are loops of compare-and-swap, and
// the first radix pass (the key's top 8 bits: sign and exponent of the scaled logit) puts almost every element of a
// row into a handful of bins: a thousand threads queueing there with such loops made a pure top-p row cost two
// milliseconds. A row's masses sum to 2^40, so every chunk's sum over up to 2^17 elements stays below 2^32. Lanes that add
// to one bin queue too, so there are copies of every histogram, a lane uses its own and each lies a bank further on. `at`: the
// bin's place in the first of the three histograms, which lie `apart` places from one another.
constexpr int BINS = 257;       // bins of a copy, with the bank in between
__device__ __forceinline__ void mass_add(unsigned* at, int apart, unsigned long long q) {
    const unsigned a = (unsigned)(q & 0x3fffull), b = (unsigned)((q >> 14) & 0x3fffull), c = (unsigned)(q >> 28);
    if (a) atomicAdd(at, a);
    if (b) atomicAdd(at + apart, b);
    if (c) atomicAdd(at + 2 * apart, c);
}

// ---- the sampling kernel: a cluster of CS CTAs per row. One SM working through a row of 152K logits a dozen times was
// the whole cost (0.1 to 2 ms for eight rows); with the row cut into CS slices every pass is CS times shorter, and what
// the CTAs have to tell each other (maxima, sums, histograms, the radix digit chosen) goes through distributed shared
// memory between cluster barriers. Everything that decides a token is either an integer sum (histograms of counts
// and of fixed-point masses: any order gives the same) or a float sum in a fixed order (threads, warps, lanes and CTAs
// in ascending order), so a row's token depends on the row alone.
constexpr int ST = 256;      // chunks of a CTA's slice: what is summed in order is summed by so many threads
constexpr int CS = 8;        // CTAs of the cluster that shares a row
constexpr size_t SAMPLE_SMEM = 200 * 1024;      // dynamic shared memory of a CTA at most
// Threads of a CTA (NT) and copies of its histograms: 512 and 4 while all rows are at work at once, which is a matter of latency;
// 256 and 1 for more rows, where what counts is the work of all of them together and how many an SM holds (see the launch).
template <int NT> constexpr int COPIES = NT == 512 ? 4 : 1;

__device__ __forceinline__ unsigned ld_peer_u32(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_peer_u64(unsigned addr) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];\n" : "=l"(v) : "r"(addr) : "memory");
    return v;
}

// The scaled logits l[i] / temperature of a CTA's slice of a row, as the kernel's passes read them: from shared memory, where
// the first pass has left them (a dozen passes over global memory, two loads in flight a thread, took half of the kernel's
// time), or, for a vocabulary whose slice does not fit, from global memory each time. Element i of the slice; ``vec``: the
// row starts on 16 bytes.
template <bool KEPT, int NT>
struct Slice {
    const float* p;         // KEPT: shared memory, scaled; else the slice's first logit
    int n;
    float inv_t;
    bool vec;
    __device__ __forceinline__ float at(int i) const { return KEPT ? p[i] : p[i] * inv_t; }
    __device__ __forceinline__ float4 at4(int i4) const {
        float4 v = reinterpret_cast<const float4*>(p)[i4];
        if (!KEPT) { v.x *= inv_t; v.y *= inv_t; v.z *= inv_t; v.w *= inv_t; }
        return v;
    }
    // f(x) for the groups of four tid, tid + T, tid + 2 T, ... in ascending order; from global memory two of them are in flight (a
    // thread with one load in flight waits out the whole latency of the memory system for every group)
    template <int T, typename F>
    __device__ __forceinline__ int fours(F&& f) const {
        const int n4 = n >> 2;
        int i = threadIdx.x;
        for (; i + T < n4; i += 2 * T) {
            const float4 a = at4(i), b = at4(i + T);
            f(a.x); f(a.y); f(a.z); f(a.w);
            f(b.x); f(b.y); f(b.z); f(b.w);
        }
        if (i < n4) {
            const float4 a = at4(i);
            f(a.x); f(a.y); f(a.z); f(a.w);
        }
        return 4 * n4;
    }
    // f(x) for every element, in no particular order, by all threads of the CTA
    template <typename F>
    __device__ __forceinline__ void each(F&& f) const {
        const int done = KEPT || vec ? fours<NT>(f) : 0;
        for (int i = done + threadIdx.x; i < n; i += NT) f(at(i));
    }
    // the same by threads 0..ST-1, each its elements in ascending order: groups of four ST groups apart where the row starts
    // on 16 bytes, elements ST apart otherwise
    template <typename F>
    __device__ __forceinline__ void each_in_order(F&& f) const {
        if (threadIdx.x >= ST) return;
        const int done = vec ? fours<ST>(f) : 0;
        for (int i = done + threadIdx.x; i < n; i += ST) f(at(i));
    }
    // f(i, x) for i = begin .. end - 1 in ascending order (a thread's chunk; begin is a multiple of 4), until f returns false; from
    // global memory all of a group of 16 elements are sent for before the first is used
    template <typename F>
    __device__ __forceinline__ void chunk(int begin, int end, F&& f) const {
        int i = begin;
        if (!KEPT && vec) {
            for (; i + 16 <= end; i += 16) {
                float4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = at4((i >> 2) + j);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (!f(i + 4 * j, v[j].x)) return;
                    if (!f(i + 4 * j + 1, v[j].y)) return;
                    if (!f(i + 4 * j + 2, v[j].z)) return;
                    if (!f(i + 4 * j + 3, v[j].w)) return;
                }
            }
        }
        if (KEPT) {
            for (; i + 4 <= end; i += 4) {
                const float4 v = at4(i >> 2);
                if (!f(i, v.x)) return;
                if (!f(i + 1, v.y)) return;
                if (!f(i + 2, v.z)) return;
                if (!f(i + 3, v.w)) return;
            }
        }
        for (; i < end; ++i)
            if (!f(i, at(i))) return;
    }
};

// The unnormalised probability of a scaled logit d = x - max <= 0, the same function wherever the kernel needs it. The
// fast exponential (2 ulp) is plenty for a draw.
__device__ __forceinline__ float weight(float d) { return __expf(d); }

// What a row is sampled with, as the host passes it by value: up to this many rows need no copy to the device ahead of the launch. The
// uniform number is made here: 24 bits of the splitmix64 finaliser of (seed, counter).
struct NibSampleRow { float temperature; int top_k; float top_p; int first; unsigned long long seed, counter; };      // first: draw at 0
constexpr int ROWS_BY_VALUE = 64;
struct SampleRows { NibSampleRow row[ROWS_BY_VALUE]; };

__device__ __forceinline__ float uniform_of(unsigned long long seed, unsigned long long counter) {
    unsigned long long x = seed * 0x9E3779B97F4A7C15ull + (counter + 1ull) * 0xD1B54A32D192ED03ull;
    x ^= x >> 30;
    x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27;
    x *= 0x94D049BB133111EBull;
    x ^= x >> 31;
    return (float)(unsigned)(x >> 40) * (1.0f / 16777216.0f);
}

// temperature > 0 for every row given to this kernel. grid: CS CTAs (one cluster) per row. Dynamic shared memory: the
// histograms' copies and, KEPT, the slice.
template <bool KEPT, int NT>
__global__ void __launch_bounds__(NT, NT == 512 ? 2 : 5)
sample_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ uniform,
              int* __restrict__ out, const __grid_constant__ SampleRows by_value) {
    using namespace nibp;
    extern __shared__ __align__(16) float dyn[];
    constexpr int HIST = COPIES<NT> * BINS;
    unsigned* copies = reinterpret_cast<unsigned*>(dyn);      // [4][HIST]: counts, then masses as three histograms
    float* kept = dyn + 4 * HIST;                   // of 14-bit chunks: mass = m1 + m2 * 2^14 + m3 * 2^28
    __shared__ float scratch[NT / 32];
    __shared__ unsigned pub[2][4][256];             // this CTA's histograms of a radix pass, for the cluster; the passes take turns
    __shared__ unsigned tot_hist[256];              // the cluster's sums
    __shared__ unsigned long long tot_mass[256];
    __shared__ unsigned dec_prefix, dec_remaining;  // what a radix pass decided (512 threads: every CTA for itself, alike; 256: CTA 0)
    __shared__ unsigned long long dec_above;
    __shared__ float x_max, x_z, x_total;           // what this CTA tells the others
    __shared__ int x_ties;
    __shared__ float chunk_sum[ST];
    __shared__ int tie_count[ST];
    __shared__ float lane_total[32];
    __shared__ int s_pick;
    __shared__ unsigned s_count, x_count;           // elements that this CTA has gathered
    __shared__ unsigned s_low, s_high;              // keys chosen among the gathered ones

    const int row = blockIdx.x / CS;
    const unsigned rank = cluster_rank();
    const float* l = logits + (size_t)row * vocab;
    const bool given = temperature == nullptr;      // the rows' parameters come by value
    const float inv_t = 1.0f / (given ? by_value.row[row].temperature : temperature[row]);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // a thread's chunk of the row (vocabulary order: rank, then thread), a multiple of 4 long so that chunks start on 16 bytes;
    // begin and end count from the slice's first element
    const int per = ((vocab + CS * ST - 1) / (CS * ST) + 3) & ~3;
    const int s_begin = min(vocab, (int)rank * ST * per), s_n = min(vocab, s_begin + ST * per) - s_begin;
    const int begin = tid < ST ? min(s_n, tid * per) : 0, end = tid < ST ? min(s_n, begin + per) : 0;
    const bool vec = (reinterpret_cast<uintptr_t>(l) & 15) == 0;
    const Slice<KEPT, NT> slice{KEPT ? kept : l + s_begin, s_n, inv_t, vec};

    auto cta_reduce = [&](float v, bool is_max, int warps) -> float {      // over the CTA's first warps, in a fixed order
        v = is_max ? warp_max(v) : warp_sum(v);
        if (lane == 0) scratch[warp] = v;
        __syncthreads();
        float r = scratch[0];
        for (int i = 1; i < warps; ++i) r = is_max ? fmaxf(r, scratch[i]) : r + scratch[i];
        __syncthreads();
        return r;
    };

    // ---- the row's maximum; KEPT: what is read for it stays
    float mx = -INFINITY;
    if (KEPT) {
        const float* src = l + s_begin;
        int done = 0;
        if (vec) {
            const int n4 = s_n >> 2;
#pragma unroll 8
            for (int i = tid; i < n4; i += NT) {
                float4 v = reinterpret_cast<const float4*>(src)[i];
                v.x *= inv_t; v.y *= inv_t; v.z *= inv_t; v.w *= inv_t;
                reinterpret_cast<float4*>(kept)[i] = v;
                mx = fmaxf(fmaxf(fmaxf(mx, v.x), fmaxf(v.y, v.z)), v.w);
            }
            done = 4 * n4;
        }
#pragma unroll 8
        for (int i = done + tid; i < s_n; i += NT) {
            const float x = src[i] * inv_t;
            kept[i] = x;
            mx = fmaxf(mx, x);
        }
    } else {
        slice.each([&](float x) { mx = fmaxf(mx, x); });
    }
    mx = cta_reduce(mx, true, NT / 32);
    if (tid == 0) x_max = mx;
    cluster_sync();
    for (unsigned r = 0; r < CS; ++r) mx = fmaxf(mx, ld_peer_f32(peer_smem(&x_max, r)));

    // One radix pass over the slice: histogram (and masses), told to the cluster, which sums them up and chooses the digit
    // (``choose``, warp 0). With 512 threads every CTA does so for itself: one barrier of the cluster a pass instead of two. With 256
    // CTA 0 does it for all, an eighth of the reads of peers' memory. A pass tells its results in the buffer of the pass before
    // the last one: whoever is past the last pass's barrier has read that.
    int pass = 0;
    const unsigned copy = (lane & (COPIES<NT> - 1)) * BINS;
    auto radix_pass = [&](bool with_mass, auto&& add, auto&& choose) {
        unsigned (*mine)[256] = pub[pass++ & 1];
        const int used = with_mass ? 4 : 1;
        for (int i = tid; i < used * HIST; i += NT) copies[i] = 0u;
        __syncthreads();
        slice.each(add);
        __syncthreads();
        for (int i = tid; i < used * 256; i += NT) {
            const int h = i >> 8, b = i & 255;
            unsigned sum = 0u;
#pragma unroll
            for (int c = 0; c < COPIES<NT>; ++c) sum += copies[h * HIST + c * BINS + b];
            mine[h][b] = sum;
        }
        cluster_sync();
        if (NT == 512 || rank == 0) {
            const int b = tid & 255;
            if (NT == 256 || tid < 256) {
                unsigned v[CS], n = 0u;
#pragma unroll
                for (unsigned r = 0; r < CS; ++r) v[r] = ld_peer_u32(peer_smem(&mine[0][b], r));
#pragma unroll
                for (unsigned r = 0; r < CS; ++r) n += v[r];
                tot_hist[b] = n;
            }
            if (with_mass && (NT == 256 || tid >= 256)) {
                unsigned v[3][CS];
                unsigned long long m = 0ull;
#pragma unroll
                for (unsigned r = 0; r < CS; ++r)
#pragma unroll
                    for (int h = 0; h < 3; ++h) v[h][r] = ld_peer_u32(peer_smem(&mine[1 + h][b], r));
#pragma unroll
                for (unsigned r = 0; r < CS; ++r) m += (unsigned long long)v[0][r] + ((unsigned long long)v[1][r] << 14) + ((unsigned long long)v[2][r] << 28);
                tot_mass[b] = m;
            }
            __syncthreads();
            if (tid < 32) choose();          // warp 0: lane j looks at the bins 8j..8j+7
        }
        if (NT == 512)
            __syncthreads();
        else
            cluster_sync();
    };
    // The elements that `wanted` says yes to, of the whole row, as keys into every CTA's shared memory (in the histograms' place, in no
    // order): few enough are left after the first pass of a select, and each then finds its own rank among them, without a pass and a
    // barrier of the cluster for every further digit. A pass in the buffers' turn. Returns how many there are. (8 rows of 151,936, us
    // without / with lists and the first pass by distance: top-p 0.9 at temperature 0.7 48.5 / 39.8, top-k 50 with top-p 0.95 48.9 / 34.0,
    // top-k 40 27.2 / 23.5; with bins of an eighth instead of a sixteenth the first of them overflows the list: 57.4.)
    constexpr int LIST = NT == 512 ? 1024 : 0;
    static_assert(LIST <= 4 * 256 && 3 * LIST <= 4 * HIST, "a CTA's list lies in a buffer of pub, the cluster's and its masses where the histograms are");
    unsigned* keys = copies;                                                                // [LIST], filled up with zeros to whole fours
    unsigned long long* masses = reinterpret_cast<unsigned long long*>(copies + LIST);      // [LIST]
    auto gather = [&](auto&& wanted) {
        unsigned* mine = &pub[pass++ & 1][0][0];
        if (tid == 0) s_count = 0u;
        __syncthreads();
        slice.each([&](float x) {
            if (wanted(x, key_of(x))) {
                const unsigned at = atomicAdd(&s_count, 1u);
                if ((int)at < LIST) mine[at] = key_of(x);
            }
        });
        __syncthreads();
        if (tid == 0) x_count = s_count;
        cluster_sync();
        unsigned n[CS], before = 0u;
#pragma unroll
        for (unsigned r = 0; r < CS; ++r) n[r] = ld_peer_u32(peer_smem(&x_count, r));
#pragma unroll
        for (unsigned r = 0; r < CS; ++r) {
            for (unsigned i = tid; i < n[r] && (int)(before + i) < LIST; i += NT) keys[before + i] = ld_peer_u32(peer_smem(mine + i, r));
            before += n[r];
        }
        const int listed = min((int)before, LIST);
        if (tid < ((4 - listed) & 3)) keys[listed + tid] = 0u;
        __syncthreads();
        return listed;
    };
    static_assert(NT == 512 || NT == 256, "the first 256 threads sum the counts, the last 256 the masses");
    const unsigned decider = NT == 512 ? rank : 0u;

    // ---- top-k: key of the k-th largest scaled logit (0 keeps everything)
    unsigned kth_key = 0u;
    const int k = given ? by_value.row[row].top_k : top_k[row];
    int survivors = vocab;      // elements whose key is at least kth_key
    if (k > 0 && k < vocab) {
        unsigned prefix = 0u, remaining = (unsigned)k;
        for (int shift = 24; shift >= 0; shift -= 8) {
            const unsigned mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
            radix_pass(false,
                       [&](float x) {
                           const unsigned key = key_of(x);
                           if ((key & mask) == prefix) atomicAdd(&copies[copy + ((key >> shift) & 255u)], 1u);
                       },
                       [&]() {
                           // the highest bin b >= 1 with (elements in bins >= b) >= remaining, else bin 0; what is still to
                           // find inside it: remaining - (elements in the bins above b)
                           unsigned mine = 0u;
                           for (int i = 0; i < 8; ++i) mine += tot_hist[lane * 8 + i];
                           unsigned above = mine;                       // inclusive sum over this lane and the lanes above
#pragma unroll
                           for (int o = 1; o < 32; o <<= 1) {
                               const unsigned v = __shfl_down_sync(0xffffffffu, above, o);
                               if (lane + o < 32) above += v;
                           }
                           above -= mine;                               // elements in the bins above this lane's
                           int found = -1;
                           unsigned rem_found = 0u, run = above;
                           for (int i = 7; i >= 0; --i) {
                               const int b = lane * 8 + i;
                               if (found < 0 && b > 0 && run + tot_hist[b] >= remaining) { found = b; rem_found = remaining - run; }
                               run += tot_hist[b];
                           }
                           const unsigned has = __ballot_sync(0xffffffffu, found >= 0);
                           const int top = has ? 31 - __clz(has) : 0;   // the highest lane that found one holds the highest bin
                           const int b = __shfl_sync(0xffffffffu, found, top);
                           const unsigned r = __shfl_sync(0xffffffffu, rem_found, top);
                           const unsigned all = __shfl_sync(0xffffffffu, above + mine, 0);       // every element that matched
                           if (lane == 0) {
                               dec_prefix = prefix | ((unsigned)(has ? b : 0) << shift);
                               dec_remaining = has ? r : remaining - (all - tot_hist[0]);
                           }
                       });
            prefix = ld_peer_u32(peer_smem(&dec_prefix, decider));
            remaining = ld_peer_u32(peer_smem(&dec_remaining, decider));
            if constexpr (NT == 512) {
                const unsigned inside = tot_hist[(prefix >> shift) & 255u];
                if (shift == 0) {
                    survivors = (int)((unsigned)k - remaining + inside);
                } else if (inside <= LIST) {
                    const int listed = gather([&](float, unsigned key) { return (key & (0xffffffffu << shift)) == prefix; });
                    for (int i = tid; i < listed; i += NT) {
                        const unsigned key = keys[i];
                        unsigned above = 0u, same = 0u;
#pragma unroll 4
                        for (int j = 0; j < listed; j += 4) {
                            const uint4 o = *reinterpret_cast<const uint4*>(keys + j);      // (the zeros behind the last one: neither, unless the key is 0, an element's last of all)
                            above += (o.x > key) + (o.y > key) + (o.z > key) + (o.w > key);
                            same += (o.x == key) + (o.y == key) + (o.z == key) + (o.w == key);
                        }
                        if (above < remaining && remaining <= above + same) {       // the key of that rank; equal ones all say so
                            dec_prefix = key;
                            dec_remaining = (unsigned)k - remaining + above + same;
                        }
                    }
                    __syncthreads();
                    prefix = dec_prefix;
                    survivors = (int)dec_remaining;
                    __syncthreads();
                    break;
                }
            }
        }
        kth_key = prefix;
    }

    // ---- normaliser over what top-k kept: threads, warps, CTAs in ascending order
    float z = 0.f;
    slice.each_in_order([&](float x) {
        if (key_of(x) >= kth_key) z += weight(x - mx);
    });
    z = cta_reduce(z, false, ST / 32);
    if (tid == 0) x_z = z;
    cluster_sync();
    z = 0.f;
    for (unsigned r = 0; r < CS; ++r) z += ld_peer_f32(peer_smem(&x_z, r));
    const float fix_over_z = FIX_ONE / z;

    // ---- top-p: smallest key whose "probability of strictly larger keys" is <= p
    unsigned p_key = kth_key;
    long long ties_kept = -1;  // -1: every element equal to p_key stays
    const float tp = given ? by_value.row[row].top_p : top_p[row];
    if (tp < 1.0f) {
        const unsigned long long limit = (unsigned long long)((double)tp * (double)FIX_ONE);
        unsigned prefix = 0u;
        unsigned long long above0 = 0ull;
        // (nothing for an undefined value: the histograms hold 42 bits of a mass, and a NaN's 2^63 is none of them)
        const auto mass_of = [&](float x) {
            const float m = weight(x - mx) * fix_over_z;
            return m > 0.f ? (unsigned long long)m : 0ull;
        };
        const auto choose = [&]() {
            // the lowest non-empty bin whose "mass above" (the bins above it, and what earlier passes left
            // above) is still within the limit; the very first (largest) element always stays, so if even
            // the highest non-empty bin is past the limit, that one
            unsigned long long mine = 0ull;
            for (int i = 0; i < 8; ++i) mine += tot_mass[lane * 8 + i];
            unsigned long long above = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long v = __shfl_down_sync(0xffffffffu, above, o);
                if (lane + o < 32) above += v;
            }
            above = above - mine + above0;               // mass above this lane's bins
            int low = -1, high = -1;
            unsigned long long low_above = 0ull, high_above = 0ull, run = above;
            for (int i = 7; i >= 0; --i) {
                const int b = lane * 8 + i;
                if (tot_hist[b] != 0u) {
                    if (high < 0) { high = b; high_above = run; }
                    if (run <= limit) { low = b; low_above = run; }
                }
                run += tot_mass[b];
            }
            const unsigned within = __ballot_sync(0xffffffffu, low >= 0), any = __ballot_sync(0xffffffffu, high >= 0);
            int chosen = 0;
            unsigned long long chosen_above = above0;
            if (within) {                                // the lowest lane with one holds the lowest such bin
                const int src = __ffs(within) - 1;
                chosen = __shfl_sync(0xffffffffu, low, src);
                chosen_above = __shfl_sync(0xffffffffu, low_above, src);
            } else if (any) {
                const int src = 31 - __clz(any);
                chosen = __shfl_sync(0xffffffffu, high, src);
                chosen_above = __shfl_sync(0xffffffffu, high_above, src);
            }
            if (lane == 0) {
                dec_prefix = (unsigned)chosen;
                dec_above = chosen_above;
            }
        };
        const auto count_mass = [&](float x, unsigned bin) {
            unsigned* at = copies + copy + bin;
            mass_add(at + HIST, HIST, mass_of(x));
            atomicAdd(at, 1u);
        };
        // Among the keys of a list: the lowest whose mass above is within the limit (else the highest, as a pass would have it).
        const auto choose_listed = [&](int listed) {
            for (int i = tid; i < ((listed + 3) & ~3); i += NT) masses[i] = i < listed ? mass_of(float_of_key(keys[i])) : 0ull;
            if (tid == 0) {
                s_low = 0xffffffffu;
                s_high = 0u;
            }
            __syncthreads();
            unsigned long long above[LIST > 0 ? (LIST + NT - 1) / NT : 1];
#pragma unroll
            for (int t = 0; t < (LIST + NT - 1) / NT; ++t) {
                const int i = tid + t * NT;
                above[t] = above0;
                if (i >= listed) continue;
                const unsigned key = keys[i];
#pragma unroll 2
                for (int j = 0; j < listed; j += 4) {
                    const uint4 o = *reinterpret_cast<const uint4*>(keys + j);
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(masses + j), b = *reinterpret_cast<const ulonglong2*>(masses + j + 2);
                    above[t] += (o.x > key ? a.x : 0ull) + (o.y > key ? a.y : 0ull) + (o.z > key ? b.x : 0ull) + (o.w > key ? b.y : 0ull);
                }
                if (above[t] <= limit) atomicMin(&s_low, key);
                atomicMax(&s_high, key);
            }
            __syncthreads();
            // (0xffffffff is the key of a NaN only, and then every key's mass is nothing and the lowest is taken)
            const unsigned key = s_low != 0xffffffffu ? s_low : s_high;
#pragma unroll
            for (int t = 0; t < (LIST + NT - 1) / NT; ++t)
                if (tid + t * NT < listed && keys[tid + t * NT] == key) dec_above = above[t];
            __syncthreads();
            prefix = key;
            above0 = dec_above;
            __syncthreads();
        };
        if (NT == 512 && survivors <= LIST) {
            choose_listed(gather([&](float, unsigned key) { return key >= kth_key; }));
        } else {
            // The first pass goes by the distance from the maximum, in sixteenths, which spreads a row over the bins (by the key's first eight
            // bits, sign and exponent, almost all of it falls into a handful, where the adds queue: 20 of a nucleus row's 48 us); what
            // it chooses is a stretch of keys like any other digit's.
            const auto bin_of = [&](float x) { return 255u - (unsigned)min(255, (int)((mx - x) * 16.0f)); };
            // (With 256 threads, whose rows have no lists, it would be one more pass: 64 rows 184 us instead of 178.)
            unsigned bin = 0u;
            bool found = false;
            if constexpr (NT == 512) {
                radix_pass(true, [&](float x) { if (key_of(x) >= kth_key) count_mass(x, bin_of(x)); }, choose);
                bin = dec_prefix;
                above0 = dec_above;
                if (tot_hist[bin] <= LIST) {
                    choose_listed(gather([&](float x, unsigned key) { return key >= kth_key && bin_of(x) == bin; }));
                    found = true;
                }
            }
            for (int shift = 24; shift >= 0 && !found; shift -= 8) {
                const unsigned mask = shift == 24 ? 0u : (0xffffffffu << (shift + 8));
                radix_pass(true,
                           [&](float x) {
                               const unsigned key = key_of(x);
                               if (key >= kth_key && (key & mask) == prefix && (NT != 512 || bin_of(x) == bin)) count_mass(x, (key >> shift) & 255u);
                           },
                           choose);
                const unsigned digit = ld_peer_u32(peer_smem(&dec_prefix, decider));
                prefix |= digit << shift;
                above0 = ld_peer_u64(peer_smem(&dec_above, decider));
                if constexpr (NT == 512) {
                    if (shift > 0 && tot_hist[digit] <= LIST) {
                        const unsigned low = 0xffffffffu << shift, want = prefix;
                        choose_listed(gather([&](float x, unsigned key) { return key >= kth_key && (key & low) == want && bin_of(x) == bin; }));
                        found = true;
                    }
                }
            }
        }
        p_key = prefix;
        if (p_key < kth_key) p_key = kth_key;
        // ties at p_key: the r-th of them (in vocabulary order) stays iff above + r*q <= limit
        const float xv = float_of_key(p_key);
        const unsigned long long q = (unsigned long long)(weight(xv - mx) * fix_over_z);
        if (q > 0ull && above0 <= limit) ties_kept = (long long)((limit - above0) / q) + 1;
        else ties_kept = 1;
    }

    // ---- inverse CDF in vocabulary order over what is kept
    // rank of the ties before this thread's chunk: the CTAs before this one, then the threads before it (lane j of warp
    // 0 takes the chunks 8j..8j+7; integers, so any order gives the same)
    long long tie_rank = 0;
    if (ties_kept >= 0) {
        int my_ties = 0;
        slice.chunk(begin, end, [&](int, float x) { my_ties += key_of(x) == p_key; return true; });
        if (tid < ST) tie_count[tid] = my_ties;
        __syncthreads();
        if (tid < 32) {
            constexpr int G = ST / 32;
            int mine = 0;
            for (int t = 0; t < G; ++t) mine += tie_count[tid * G + t];
            int before = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, before, o);
                if (tid >= o) before += v;
            }
            if (tid == 31) x_ties = before;
            int run = before - mine;
            for (int t = 0; t < G; ++t) { const int c = tie_count[tid * G + t]; tie_count[tid * G + t] = run; run += c; }
        }
        __syncthreads();
        cluster_sync();
        tie_rank = tie_count[tid & (ST - 1)];
        for (unsigned r = 0; r < rank; ++r) tie_rank += (int)ld_peer_u32(peer_smem(&x_ties, r));
    }
    float csum = 0.f;
    {
        long long tr = tie_rank;
        slice.chunk(begin, end, [&](int, float x) {
            const unsigned key = key_of(x);
            bool keep = key >= p_key;
            if (keep && ties_kept >= 0 && key == p_key) keep = (tr++) < ties_kept;
            if (keep) csum += weight(x - mx);
            return true;
        });
    }
    if (tid < ST) chunk_sum[tid] = csum;
    __syncthreads();
    // The sums in a fixed order, in three levels: lane j of warp 0 adds the sums of the CTA's chunks 8j..8j+7 in order and
    // the 32 lane totals in order; the CTAs' totals are added in rank order. The CTA whose chunks hold the drawn point
    // of the row's mass finds the lane, the lane its chunk, the chunk's thread the element.
    constexpr int G = ST / 32;
    if (tid < 32) {
        float mine = 0.f;
        for (int t = 0; t < G; ++t) mine += chunk_sum[tid * G + t];
        lane_total[tid] = mine;
        __syncwarp();
        if (tid == 0) {
            float total = 0.f;
            for (int j = 0; j < 32; ++j) total += lane_total[j];
            x_total = total;
        }
    }
    __syncthreads();
    cluster_sync();
    float cta_total[CS], total = 0.f;
    for (unsigned r = 0; r < CS; ++r) { cta_total[r] = ld_peer_f32(peer_smem(&x_total, r)); total += cta_total[r]; }
    const float target = (!given ? uniform[row] : by_value.row[row].first ? 0.f : uniform_of(by_value.row[row].seed, by_value.row[row].counter)) * total;
    // which CTA: the first whose totals reach past the target; if rounding runs past the end, the last with mass
    int cta_pick = -1, last_cta = CS - 1;
    float cta_before = 0.f;
    {
        float run = 0.f;
        for (int r = 0; r < CS; ++r) {
            if (cta_total[r] > 0.f) last_cta = r;
            if (cta_pick < 0 && run + cta_total[r] > target && cta_total[r] > 0.f) { cta_pick = r; cta_before = run; }
            if (cta_pick < 0) run += cta_total[r];
        }
        if (cta_pick < 0) {
            cta_pick = last_cta;
            cta_before = 0.f;
            for (int r = 0; r < cta_pick; ++r) cta_before += cta_total[r];
        }
    }
    if ((int)rank == cta_pick) {
        if (tid < 32) {
            float run = cta_before;
            int lane_pick = -1, last_lane = 31;
            for (int j = 0; j < 32; ++j) {
                if (lane_total[j] > 0.f) last_lane = j;
                if (lane_pick < 0 && run + lane_total[j] > target && lane_total[j] > 0.f) lane_pick = j;
                if (lane_pick < 0) run += lane_total[j];
            }
            if (lane_pick < 0) {
                lane_pick = last_lane;
                run = cta_before;
                for (int j = 0; j < lane_pick; ++j) run += lane_total[j];
            }
            if (tid == lane_pick) {
                int pick = tid * G + G - 1;
                float before = run;
                bool found = false;
                for (int t = 0; t < G; ++t) {
                    const float c = chunk_sum[tid * G + t];
                    if (c > 0.f) pick = tid * G + t;
                    if (before + c > target && c > 0.f) { pick = tid * G + t; found = true; break; }
                    before += c;
                }
                if (!found) {
                    before = run;
                    for (int t = tid * G; t < pick; ++t) before += chunk_sum[t];
                }
                s_pick = pick;
                scratch[0] = before;
            }
        }
        __syncthreads();
        if (tid == s_pick) {
            float run = scratch[0];
            long long tr = tie_rank;
            int chosen = -1, last_kept = -1;
            slice.chunk(begin, end, [&](int i, float x) {
                const unsigned key = key_of(x);
                bool keep = key >= p_key;
                if (keep && ties_kept >= 0 && key == p_key) keep = (tr++) < ties_kept;
                if (!keep) return true;
                last_kept = i;
                run += weight(x - mx);
                if (run > target) { chosen = i; return false; }
                return true;
            });
            out[row] = chosen >= 0 ? s_begin + chosen : (last_kept >= 0 ? s_begin + last_kept : 0);
        }
    }
    cluster_sync();         // nobody leaves while a peer may still read its shared memory
}

static int launch_sample(const float* logits, int rows, int vocab, const float* temperature, const int* top_k, const float* top_p,
                         const float* uniform, int* out, const SampleRows& by_value, cudaStream_t stream) {
    NIB_REQUIRE(rows >= 0 && vocab > 0, "sample: bad sizes");
    if (rows == 0) return 0;
    NIB_REQUIRE((long long)vocab <= (1LL << 17) * 8, "sample: a row of %d logits is more than the fixed-point histograms hold", vocab);
    const int per = (ceil_div(vocab, CS * ST) + 3) & ~3;
    // Up to 32 rows all CTAs are at work at once, two an SM, and a row's time is what counts: 512 threads, and the slice kept in
    // shared memory if two of them fit an SM's (else for the 12 rows that one an SM holds). More rows: as many CTAs an SM as there can
    // be (five), and the slice kept only where it is small. Measured, us with 512 / 256 threads, at a vocabulary of 151,936: top-p 0.9, 1 row
    // 38 / 68, 12 rows 46 / 75, 16 51 / 86, 32 58 / 90; top-k 40, 32 rows 35 / 52; neither, 30 / 33. From 34 rows on 512 threads are two turns: 34
    // rows, top-p 80 / 104, top-k 52 / 55, neither 41 / 33; 64 rows 110 / 131, 65 / 67, 54 / 41; at 32,000, 34 rows 39 / 37, 31 / 22, 21 / 14, 64 rows 49 /
    // 44, 37 / 25, 25 / 15 (one kernel takes all rows of a call, whatever each asks for).
    const size_t slice = sizeof(float) * (size_t)ST * per;
    const auto room = [&](int copies) { return sizeof(unsigned) * 4 * copies * BINS + slice; };
    const bool wide = rows <= 32;
    const bool kept = wide ? room(COPIES<512>) <= (rows <= 12 ? SAMPLE_SMEM : 98 * 1024) : room(COPIES<256>) <= 30 * 1024;
    const size_t smem = room(wide ? COPIES<512> : COPIES<256>) - (kept ? 0 : slice);
    auto* kernel = wide ? (kept ? sample_kernel<true, 512> : sample_kernel<false, 512>) : (kept ? sample_kernel<true, 256> : sample_kernel<false, 256>);
    // the most that any call takes: the attribute is the kernel's, and a call's own size would lower it under another thread's launch
    if (kept && wide) NIB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SAMPLE_SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * CS);
    cfg.blockDim = dim3(wide ? 512 : 256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    NIB_CUDA(cudaLaunchKernelEx(&cfg, kernel, logits, vocab, temperature, top_k, top_p, uniform, out, by_value));
    NIB_LAUNCH_CHECK();
    return 0;
}

NIB_API int nib_sample(const float* logits, int rows, int vocab, const float* temperature, const int* top_k,
                       const float* top_p, const float* uniform, int* out, cudaStream_t stream) {
    NIB_REQUIRE(rows == 0 || (temperature && top_k && top_p && uniform), "sample: parameters are needed");
    static const SampleRows none{};
    return launch_sample(logits, rows, vocab, temperature, top_k, top_p, uniform, out, none, stream);
}

NIB_API int nib_sample_rows_most() { return ROWS_BY_VALUE; }

// The same for up to nib_sample_rows_most() rows whose parameters lie in host memory (read before this returns) and whose uniform
// numbers are made on the device. ``out`` may be page-locked host memory: each row's token is one store.
NIB_API int nib_sample_rows(const float* logits, int rows, int vocab, const NibSampleRow* params, int* out, cudaStream_t stream) {
    NIB_REQUIRE(rows >= 0 && rows <= ROWS_BY_VALUE && (rows == 0 || params != nullptr), "sample: up to %d rows by value", ROWS_BY_VALUE);
    SampleRows by_value;
    memset(&by_value, 0, sizeof(by_value));
    if (rows > 0) memcpy(by_value.row, params, sizeof(NibSampleRow) * (size_t)rows);
    return launch_sample(logits, rows, vocab, nullptr, nullptr, nullptr, nullptr, out, by_value, stream);
}
