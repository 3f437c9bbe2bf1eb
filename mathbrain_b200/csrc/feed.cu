// Chunk feeding: slot lists, chunk-start states and the advance of per-document slot state.
//
// A document's chunk tokens and its list of seen tokens become bitmaps over the vocabulary in shared memory (V / 8 bytes
// each, 6 KB at 50257), whose set bits in order are the sorted distinct tokens: no sort, one CTA per document.  Built from
// batched tensor operations (sorts, searches, scatters) the same step took 1.5 ms for 56 chunks of 512 tokens, most of it
// forty launches and three reads back to the host; here it is three kernels of 5 to 15 us and one read (the widest list).
#include "common.cuh"

namespace mbema {
namespace feed {

static constexpr int THREADS = 1024;
static constexpr int SEG_WORDS = 12288;            // vocabulary segment held at a time: 393216 tokens, 2 x 48 KB

// block-wide exclusive scan of one value per thread; *total receives the sum
__device__ __forceinline__ int block_scan(int v, int* wsum, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += u; }
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    if (warp == 0) {
        int w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += u; }
        wsum[lane] = w;
    }
    __syncthreads();
    const int before = (warp ? wsum[warp - 1] : 0) + s - v;
    *total = wsum[31];
    __syncthreads();
    return before;
}

// put(rank, token) for every set bit of `word(i)`, i < words, in order; returns the number of set bits
template <class Word, class Put>
__device__ __forceinline__ int for_bits(int words, int first_token, int* wsum, Word word, Put put) {
    const int per = (words + THREADS - 1) / THREADS, lo = threadIdx.x * per, hi = min(lo + per, words);
    int n = 0, total;
    for (int i = lo; i < hi; ++i) n += __popc(word(i));
    int at = block_scan(n, wsum, &total);
    for (int i = lo; i < hi; ++i)
        for (unsigned w = word(i); w; w &= w - 1) put(at++, first_token + i * 32 + __ffs(w) - 1);
    return total;
}

// lists[b]: the chunk's distinct tokens in order, then those seen before and not in the chunk; counts[b], counts[B] = the most
__global__ void __launch_bounds__(THREADS)
k_feed_lists(const int64_t* __restrict__ x, const int32_t* __restrict__ fill, const int64_t* __restrict__ seen,
             const int64_t* __restrict__ n_seen, int32_t* __restrict__ lists, int32_t* __restrict__ counts, int T, int V, int cap, int L) {
    extern __shared__ unsigned bits[];
    __shared__ int wsum[32];
    const int b = blockIdx.x, tid = threadIdx.x;
    const int F = min(max(fill[b], 0), T), S = (int)min((int64_t)cap, n_seen[b]);
    const int seg_words = min(SEG_WORDS, (V + 31) / 32);
    unsigned* cur = bits;
    unsigned* old = bits + seg_words;
    int n = 0;
    for (int pass = 0; pass < 2; ++pass)
        for (int v0 = 0; v0 < V; v0 += seg_words * 32) {
            const int words = min(seg_words, (V - v0 + 31) / 32);
            if (pass == 0 || V > seg_words * 32) {       // one segment: the bitmaps of the first pass serve the second
                __syncthreads();
                for (int i = tid; i < words; i += THREADS) cur[i] = old[i] = 0u;
                __syncthreads();
                const int top = min(V - v0, words * 32);
                for (int t = tid; t < F; t += THREADS) {
                    const int64_t v = x[(size_t)b * T + t] - v0;
                    if (v >= 0 && v < top) atomicOr(&cur[v >> 5], 1u << (v & 31));
                }
                for (int i = tid; i < S; i += THREADS) {
                    const int64_t v = seen[(size_t)b * cap + i] - v0;
                    if (v >= 0 && v < top) atomicOr(&old[v >> 5], 1u << (v & 31));
                }
                __syncthreads();
            }
            int32_t* out = lists + (size_t)b * L + n;
            auto put = [&](int r, int tok) { out[r] = tok; };
            n += pass == 0 ? for_bits(words, v0, wsum, [&](int i) { return cur[i]; }, put)
                           : for_bits(words, v0, wsum, [&](int i) { return old[i] & ~cur[i]; }, put);
        }
    if (tid == 0) {
        counts[b] = n;
        atomicMax(&counts[gridDim.x], n);
    }
}

// a warp per list entry: the token (0 behind the list), its mask, its state decayed to the chunk's first step
__global__ void __launch_bounds__(256)
k_feed_batch(const int32_t* __restrict__ lists, const int32_t* __restrict__ counts, const float* __restrict__ state,
             const int32_t* __restrict__ last_t, const int32_t* __restrict__ t0, const float* __restrict__ rhos, int64_t* __restrict__ unique,
             unsigned char* __restrict__ mask, float* __restrict__ c_base, int B, int K, int V, int N, int L) {
    const int lane = threadIdx.x & 31;
    const int64_t R = (int64_t)B * K, stride = (int64_t)gridDim.x * 8;
    for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < R; r += stride) {
        const int b = (int)(r / K), k = (int)(r - (int64_t)b * K);
        const bool in = k < counts[b];
        const int v = in ? lists[(size_t)b * L + k] : 0;
        const int lt = in ? last_t[(size_t)b * V + v] : -1;
        if (lane == 0) {
            unique[r] = v;
            mask[r] = in ? 1 : 0;
        }
        const float dt = (float)(t0[b] - lt);
        for (int n = lane; n < N; n += 32)
            c_base[r * N + n] = lt >= 0 ? state[((size_t)b * V + v) * N + n] * exp2f(dt * log2f(rhos[n])) : 0.f;
    }
}

// Moves a document past its chunk.  `check`: nothing is changed, status[0] becomes the longest list that would result.
__global__ void __launch_bounds__(THREADS)
k_feed_advance(const int64_t* __restrict__ x, const int32_t* __restrict__ fill, const float* __restrict__ C_seq, float* __restrict__ state,
               int32_t* last_t, int64_t* __restrict__ seen, int64_t* __restrict__ n_seen, int32_t* __restrict__ t0, int32_t* __restrict__ status,
               int T, int V, int N, int cap, int check) {
    extern __shared__ unsigned bits[];
    __shared__ int wsum[32];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int F = min(max(fill[b], 0), T), start = t0[b];
    const int64_t n0 = n_seen[b];
    const int seg_words = min(SEG_WORDS, (V + 31) / 32);
    int32_t* lt = last_t + (size_t)b * V;
    int n = 0;
    for (int v0 = 0; v0 < V; v0 += seg_words * 32) {       // tokens seen for the first time join the list, in token order
        const int words = min(seg_words, (V - v0 + 31) / 32), top = min(V - v0, words * 32);
        __syncthreads();
        for (int i = tid; i < words; i += THREADS) bits[i] = 0u;
        __syncthreads();
        for (int t = tid; t < F; t += THREADS) {
            const int64_t v = x[(size_t)b * T + t] - v0;
            if (v >= 0 && v < top && lt[v0 + v] < 0) atomicOr(&bits[v >> 5], 1u << (v & 31));
        }
        __syncthreads();
        n += for_bits(words, v0, wsum, [&](int i) { return bits[i]; }, [&](int r, int tok) {
            const int64_t at = n0 + n + r;
            if (!check && at < cap) seen[(size_t)b * cap + at] = tok;
        });
    }
    if (check) {
        if (tid == 0) atomicMax(status, (int)(n0 + n));
        return;
    }
    for (int t = tid; t < F; t += THREADS) {
        const int64_t v = x[(size_t)b * T + t];
        if (v >= 0 && v < V) atomicMax(&lt[v], start + t);
    }
    __syncthreads();
    // a token's last occurrence leaves its state
    for (int t = tid >> 5; t < F; t += THREADS / 32) {
        const int64_t v = x[(size_t)b * T + t];
        if (v < 0 || v >= V || __ldcg(&lt[v]) != start + t) continue;
        const float* src = C_seq + ((size_t)b * T + t) * N;
        float* dst = state + ((size_t)b * V + v) * N;
        for (int c = lane; c < N; c += 32) dst[c] = src[c] + 1.0f;
    }
    if (tid == 0) {
        n_seen[b] = n0 + n;
        t0[b] = start + F;
    }
}

static int bitmap_bytes(int64_t V) {
    const int64_t w = (V + 31) / 32;
    return (int)(w < SEG_WORDS ? w : SEG_WORDS) * 4;
}

}  // namespace feed
}  // namespace mbema

using namespace mbema;

static int feed_check(int64_t B, int64_t T, int64_t V, int64_t cap) {
    if (B < 0 || T < 1 || V < 1 || cap < 1) return MBEMA_ERR_SHAPE;
    if (T > (1 << 30) || V > (1 << 30) || cap > (1 << 30) || B > (1 << 30)) return MBEMA_ERR_UNSUPPORTED;
    return MBEMA_OK;
}

extern "C" int mbema_feed_lists(const int64_t* x, const int32_t* fill, const int64_t* seen, const int64_t* n_seen, int32_t* lists,
                                int32_t* counts, int64_t B, int64_t T, int64_t V, int64_t cap, void* stream) {
    int rc = feed_check(B, T, V, cap);
    if (rc) return rc;
    if (!counts) return MBEMA_ERR_NULL;
    cudaStream_t st = (cudaStream_t)stream;
    MBEMA_CUDA_TRY(cudaMemsetAsync(counts + B, 0, sizeof(int32_t), st));
    if (B == 0) return MBEMA_OK;
    if (!x || !fill || !seen || !n_seen || !lists) return MBEMA_ERR_NULL;
    const int smem = 2 * feed::bitmap_bytes(V);
    MBEMA_CUDA_TRY(cudaFuncSetAttribute(feed::k_feed_lists, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * feed::SEG_WORDS * 4));
    feed::k_feed_lists<<<(unsigned)B, feed::THREADS, smem, st>>>(x, fill, seen, n_seen, lists, counts, (int)T, (int)V, (int)cap, (int)(T + cap));
    return check_launch();
}

extern "C" int mbema_feed_batch(const int32_t* lists, const int32_t* counts, const float* state, const int32_t* last_t, const int32_t* t0,
                                const float* rhos, int64_t* unique, uint8_t* pad_mask, float* c_base, int64_t B, int64_t K, int64_t T,
                                int64_t V, int64_t N, int64_t cap, void* stream) {
    int rc = feed_check(B, T, V, cap);
    if (rc) return rc;
    if (K < 0 || N < 1) return MBEMA_ERR_SHAPE;
    if (B == 0 || K == 0) return MBEMA_OK;
    if (!lists || !counts || !state || !last_t || !t0 || !rhos || !unique || !pad_mask || !c_base) return MBEMA_ERR_NULL;
    const int64_t want = (B * K + 7) / 8, most = 148 * 8;      // eight CTAs of eight warps per SM
    feed::k_feed_batch<<<(unsigned)(want < most ? want : most), 256, 0, (cudaStream_t)stream>>>(
        lists, counts, state, last_t, t0, rhos, unique, pad_mask, c_base, (int)B, (int)K, (int)V, (int)N, (int)(T + cap));
    return check_launch();
}

extern "C" int mbema_feed_advance(const int64_t* x, const int32_t* fill, const float* C_seq, float* state, int32_t* last_t, int64_t* seen,
                                  int64_t* n_seen, int32_t* t0, int32_t* status, int64_t B, int64_t T, int64_t V, int64_t N, int64_t cap,
                                  int check, void* stream) {
    int rc = feed_check(B, T, V, cap);
    if (rc) return rc;
    if (N < 1) return MBEMA_ERR_SHAPE;
    if (B == 0) return MBEMA_OK;
    if (!x || !fill || (!check && !C_seq) || !state || !last_t || !seen || !n_seen || !t0 || (check && !status)) return MBEMA_ERR_NULL;
    MBEMA_CUDA_TRY(cudaFuncSetAttribute(feed::k_feed_advance, cudaFuncAttributeMaxDynamicSharedMemorySize, feed::SEG_WORDS * 4));
    feed::k_feed_advance<<<(unsigned)B, feed::THREADS, feed::bitmap_bytes(V), (cudaStream_t)stream>>>(
        x, fill, C_seq, state, last_t, seen, n_seen, t0, status, (int)T, (int)V, (int)N, (int)cap, check);
    return check_launch();
}
