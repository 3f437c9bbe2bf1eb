// Row-wise softmax cross-entropy over a chunk of logits, forward and backward in one launch, in place:
//   loss[r] = logsumexp(logits[r, :V]) - logits[r, target[r]],   logits[r, :] <- (softmax(logits[r, :V]) - onehot) * scale
// The chunked tied lm_head (mathbrain/model.py:185-186 computes [B*T, V] logits at once; train.py:320-323 applies the
// masked cross-entropy) runs a library GEMM per chunk of VALID rows, this kernel on the chunk, and two more GEMMs
// (dh = dlogits E, dE += dlogits^T h), so the full logits never exist and masked positions cost nothing.
// HBM-bound: one read and one write of the chunk (the later reads of a row come from L2: a bf16 row is 100 KB).
// Rows have a padded leading dimension (a multiple of 8 elements) so that every row starts 16-byte aligned; the
// padding columns [V, ld) are written as zeros.
#include "common.cuh"

namespace mbema {

constexpr int CE_THREADS = 256;

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// (m, s) <- merge with (m2, s2): maxima in log2 units, sums relative to them
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
    const float mn = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * ex2_approx(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * ex2_approx(m2 - mn));
    m = mn;
}

template <int DT, int VEC>
__device__ __forceinline__ void ce_load(const void* p, size_t i, float* v) {
    const float4 a = ld4_dyn_f32(p, DT, i);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    if (VEC == 8) {
        const float4 b = ld4_dyn_f32(p, DT, i + 4);
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}

// One CTA per row, two sweeps: an online (maximum, sum of exp) per thread over its share of the row, merged across the
// CTA; then the gradient, written over the logits.  The first sweep reads DRAM, the second finds the row (100 KB in
// bf16) in L2; the grid is sized so that the rows in flight fit there.  Full vectors take a path without per-element
// bounds tests, the one-hot term is subtracted afterwards by one thread, exponentials are ex2 of pre-scaled arguments.
template <int DT>
__global__ void __launch_bounds__(CE_THREADS)
k_ce_rows(void* __restrict__ logits, const int64_t* __restrict__ targets, float scale, float* __restrict__ loss_rows,
          int64_t R, int64_t V64, int64_t ld64) {
    constexpr int VEC = (DT == MBEMA_F32) ? 4 : 8;
    constexpr float L2E = 1.4426950408889634f;
    __shared__ float red_m[CE_THREADS / 32], red_s[CE_THREADS / 32];
    __shared__ float bc[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int V = (int)V64, ld = (int)ld64, Vfull = V / VEC * VEC;
    for (int64_t r = blockIdx.x; r < R; r += gridDim.x) {
        const size_t base = (size_t)r * ld;
        float m = -INFINITY, s = 0.f;          // in units of log2: m = max(x) * log2(e), s = sum 2^(x log2e - m)
        for (int c = tid * VEC; c < V; c += CE_THREADS * VEC) {
            float v[VEC];
            ce_load<DT, VEC>(logits, base + c, v);
            if (c >= Vfull) {
#pragma unroll
                for (int i = 0; i < VEC; ++i) if (c + i >= V) v[i] = -INFINITY;
            }
            float mx = v[0];
#pragma unroll
            for (int i = 1; i < VEC; ++i) mx = fmaxf(mx, v[i]);
            mx = fmaxf(m, mx * L2E);
            float acc = s * ex2_approx(m - mx);        // m = -inf at the start: 0 * 2^(-inf) = 0
#pragma unroll
            for (int i = 0; i < VEC; ++i) acc += ex2_approx(fmaf(v[i], L2E, -mx));
            m = mx; s = acc;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
            ce_merge(m, s, m2, s2);
        }
        if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
        __syncthreads();
        if (tid == 0) {
            float mm = red_m[0], ss = red_s[0];
            for (int i = 1; i < CE_THREADS / 32; ++i) ce_merge(mm, ss, red_m[i], red_s[i]);
            bc[0] = mm; bc[1] = ss;
            const int64_t t = targets[r];
            const float xt = (t >= 0 && t < V) ? ld_dyn_f32(logits, DT, base + t) : 0.f;
            loss_rows[r] = (t >= 0 && t < V) ? (logf(ss) + mm * (1.0f / L2E) - xt) : 0.f;
        }
        __syncthreads();
        const int64_t t = targets[r];
        const bool has_t = t >= 0 && t < V;
        const float mm = bc[0], inv = has_t ? scale / bc[1] : 0.f;       // a row without a target gets a zero gradient
        for (int c = tid * VEC; c < ld; c += CE_THREADS * VEC) {
            float v[VEC];
            ce_load<DT, VEC>(logits, base + c, v);
#pragma unroll
            for (int i = 0; i < VEC; ++i) v[i] = ex2_approx(fmaf(v[i], L2E, -mm)) * inv;
            if (c >= Vfull) {
#pragma unroll
                for (int i = 0; i < VEC; ++i) if (c + i >= V) v[i] = 0.f;
            }
            if (has_t && (int)t >= c && (int)t < c + VEC) {      // the one-hot term (one thread per row takes this branch)
#pragma unroll
                for (int i = 0; i < VEC; ++i) if (c + i == (int)t) v[i] -= scale;
            }
            st4_dyn(logits, DT, base + c, make_float4(v[0], v[1], v[2], v[3]));
            if (VEC == 8) st4_dyn(logits, DT, base + c + 4, make_float4(v[4], v[5], v[6], v[7]));
        }
        __syncthreads();
    }
}

// The same for bf16 rows of which two fit an SM's shared memory: a thread's share of the row is copied there (it reads back only
// what it copied itself, so no barrier stands between), the row is read from memory once, and of the CTAs on an SM one loads
// while another computes.  At 15200 rows of 50257 (3.06 GB read and written): k_ce_rows 785 us (the second sweep's reads
// compete with the writes), this 670 us; 16384 rows of 32000: 481 and 454 us, of 16384: 262 and 280 us (too little of a row a
// thread between the barriers), so shorter rows than CE_SH_MIN_LD stay with k_ce_rows.
constexpr int CE_SH_THREADS = 512;
constexpr int CE_SH_MIN_LD = 24 * 1024, CE_SH_MAX_LD = 56 * 1024;          // 112 KB a row
__global__ void __launch_bounds__(CE_SH_THREADS, 2)
k_ce_rows_shared(__nv_bfloat16* __restrict__ logits, const int64_t* __restrict__ targets, float scale, float* __restrict__ loss_rows,
                 int64_t R, int V, int ld) {
    extern __shared__ __align__(16) unsigned char row_sh[];
    constexpr float L2E = 1.4426950408889634f;
    constexpr int WARPS = CE_SH_THREADS / 32, STEP = CE_SH_THREADS * 8;
    __shared__ float red_m[2][WARPS], red_s[2][WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, Vfull = V / 8 * 8;
    const uint32_t sh = (uint32_t)__cvta_generic_to_shared(row_sh);
    auto unpack = [](const uint4& q, float (&v)[8]) {
        const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
    };
    int buf = 0;
    for (int64_t r = blockIdx.x; r < R; r += gridDim.x, buf ^= 1) {
        __nv_bfloat16* row = logits + (size_t)r * ld;
        for (int c = tid * 8; c < ld; c += STEP)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sh + c * 2), "l"(row + c) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        const int64_t t = targets[r];
        const bool has_t = t >= 0 && t < V;
        const float xt = has_t && tid == 0 ? __bfloat162float(row[t]) : 0.f;
        float m = -INFINITY, s = 0.f;          // in units of log2: m = max(x) * log2(e), s = sum 2^(x log2e - m)
        for (int c = tid * 8; c < V; c += STEP) {
            float v[8];
            unpack(*reinterpret_cast<const uint4*>(row_sh + c * 2), v);
            if (c >= Vfull) {
#pragma unroll
                for (int i = 0; i < 8; ++i) if (c + i >= V) v[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) m = fmaxf(m, v[i]);
        }
        m *= L2E;
        for (int c = tid * 8; c < V; c += STEP) {
            float v[8];
            unpack(*reinterpret_cast<const uint4*>(row_sh + c * 2), v);
            if (c >= Vfull) {
#pragma unroll
                for (int i = 0; i < 8; ++i) if (c + i >= V) v[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) s += ex2_approx(fmaf(v[i], L2E, -m));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
            ce_merge(m, s, m2, s2);
        }
        if (lane == 0) { red_m[buf][warp] = m; red_s[buf][warp] = s; }
        __syncthreads();          // (two buffers: a warp may be a row ahead of the readers of the last)
        m = red_m[buf][lane % WARPS];
        s = red_s[buf][lane % WARPS];
#pragma unroll
        for (int o = WARPS / 2; o > 0; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
            ce_merge(m, s, m2, s2);
        }
        const float mm = __shfl_sync(0xffffffffu, m, 0), ss = __shfl_sync(0xffffffffu, s, 0);
        if (tid == 0) loss_rows[r] = has_t ? (logf(ss) + mm * (1.0f / L2E) - xt) : 0.f;
        const float inv = has_t ? scale / ss : 0.f;       // a row without a target gets a zero gradient
        for (int c = tid * 8; c < ld; c += STEP) {
            float v[8];
            unpack(*reinterpret_cast<const uint4*>(row_sh + c * 2), v);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = ex2_approx(fmaf(v[i], L2E, -mm)) * inv;
            if (c >= Vfull) {
#pragma unroll
                for (int i = 0; i < 8; ++i) if (c + i >= V) v[i] = 0.f;
            }
            if (has_t && (int)t >= c && (int)t < c + 8) {      // the one-hot term (one thread per row takes this branch)
#pragma unroll
                for (int i = 0; i < 8; ++i) if (c + i == (int)t) v[i] -= scale;
            }
            uint4 o;
            uint32_t* w = &o.x;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&p);
            }
            *reinterpret_cast<uint4*>(row + c) = o;
        }
    }
}

// dst (+)= src, fp32 and bf16, eight elements a thread: bytes only (a 50264 x 512 chunk: 257 MB, 36 us; as a mixed-type tensor
// addition 86 us, as conversion and addition 125 us)
__global__ void __launch_bounds__(256) k_accumulate_bf16(float* __restrict__ dst, const uint4* __restrict__ src, int64_t n8, int add) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n8) return;
    const uint4 q = __ldcs(src + i);
    float4* d = reinterpret_cast<float4*>(dst) + 2 * i;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (add) { a = d[0]; b = d[1]; }
    auto lo = [](uint32_t u) { return __uint_as_float(u << 16); };
    auto hi = [](uint32_t u) { return __uint_as_float(u & 0xffff0000u); };
    d[0] = make_float4(a.x + lo(q.x), a.y + hi(q.x), a.z + lo(q.y), a.w + hi(q.y));
    d[1] = make_float4(b.x + lo(q.z), b.y + hi(q.z), b.z + lo(q.w), b.w + hi(q.w));
}

}  // namespace mbema

using namespace mbema;

extern "C" int mbema_ce_rows(void* logits, int dtype, const int64_t* targets, float scale, float* loss_rows, int64_t R,
                             int64_t V, int64_t ld, void* stream) {
    if (R < 0 || V <= 0 || ld < V || ld % 8 != 0) return MBEMA_ERR_SHAPE;
    if (R == 0) return MBEMA_OK;
    if (!logits || !targets || !loss_rows) return MBEMA_ERR_NULL;
    if (dtype != MBEMA_F32 && dtype != MBEMA_BF16) return MBEMA_ERR_DTYPE;
    if ((uintptr_t)logits & 15) return MBEMA_ERR_ALIGN;
    int dev = 0, sms = 148;
    MBEMA_CUDA_TRY(cudaGetDevice(&dev));
    MBEMA_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int64_t cap = (int64_t)sms * 4;        // rows in flight: 592 x 100 KB stay below the L2 capacity
    const int grid = (int)(R < cap ? R : cap);
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == MBEMA_BF16 && ld >= CE_SH_MIN_LD && ld <= CE_SH_MAX_LD) {
        const int row_bytes = (int)ld * 2;
        const int64_t most = (int64_t)sms * 2;
        MBEMA_CUDA_TRY(cudaFuncSetAttribute(k_ce_rows_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * CE_SH_MAX_LD));
        k_ce_rows_shared<<<(unsigned)(R < most ? R : most), CE_SH_THREADS, row_bytes, st>>>((__nv_bfloat16*)logits, targets, scale, loss_rows, R, (int)V, (int)ld);
        return check_launch();
    }
    if (dtype == MBEMA_F32) k_ce_rows<MBEMA_F32><<<grid, CE_THREADS, 0, st>>>(logits, targets, scale, loss_rows, R, V, ld);
    else k_ce_rows<MBEMA_BF16><<<grid, CE_THREADS, 0, st>>>(logits, targets, scale, loss_rows, R, V, ld);
    return check_launch();
}

extern "C" int mbema_accumulate_bf16(float* dst, const void* src, int64_t n, int add, void* stream) {
    if (n < 0 || n % 8 != 0) return MBEMA_ERR_SHAPE;
    if (n == 0) return MBEMA_OK;
    if (!dst || !src) return MBEMA_ERR_NULL;
    if (((uintptr_t)dst | (uintptr_t)src) & 15) return MBEMA_ERR_ALIGN;
    const int64_t blocks = (n / 8 + 255) / 256;
    if (blocks > 0x7fffffff) return MBEMA_ERR_UNSUPPORTED;
    k_accumulate_bf16<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(dst, (const uint4*)src, n / 8, add);
    return check_launch();
}
