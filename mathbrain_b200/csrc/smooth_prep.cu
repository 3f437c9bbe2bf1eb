// What the smooth attention kernels read: node-scaled W_pe images, the Gram matrix of W_pe, and per (sample, tile) the
// items (slots, and occurrences inside the tile) with their states as ready-made operand tiles.
#include "smooth.cuh"
#include "sm100_ptx.cuh"

namespace mbema {
namespace smooth {

using namespace ptx;

// swizzled byte offset of 16-byte chunk `c8` (0..7) of row `r` in an operand tile of 128-byte rows
__device__ __forceinline__ int sw_chunk(int r, int c8) { return r * 128 + ((c8 ^ (r & 7)) << 4); }

// ---------------------------------------------------------------------------------------------------------------
// blocks [0, SEG_IMAGES * H * NCH): the W' image of (segment, head, column chunk): row i * 16 + dd holds
// W[n, head * 64 + chunk * 16 + dd] rho_n^(node i of the segment), fp16, 64 x (the states carry 1/64) and, for SiLU,
// 1/2 x (SiLU(x) = h + h tanh h, h = x / 2).  The remaining N N / 8 blocks: a warp per entry of the Gram matrix (a warp for
// eight of them, one after the other: 11 us; one each: 6.6 us).
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_weights(FlashArgs a, Ws w) {
    const int N = a.N, D = a.H * HD, NK = N >> 6, tid = threadIdx.x;
    const int n_img = SEG_IMAGES * a.H * NCH;
    if ((int)blockIdx.x >= n_img) {
        const int pair = ((int)blockIdx.x - n_img) * 8 + (tid >> 5), n = pair / N, m = pair % N, lane = tid & 31;
        float s = 0.f;
#pragma unroll 4
        for (int d = lane; d < D; d += 32) s = fmaf(a.W[(size_t)n * D + d], a.W[(size_t)m * D + d], s);
        s = warp_sum(s);
        if (lane == 0) w.gram[n * N + m] = s / (float)D;
        return;
    }
    const int c = blockIdx.x % NCH, h = (blockIdx.x / NCH) % a.H, img = blockIdx.x / (NCH * a.H);
    const int level = 31 - __clz(img + 1), seg = img + 1 - (1 << level);
    const float len = (float)(TM >> level);
    unsigned char* out = w.w_img + (size_t)blockIdx.x * NK * WPIECE;
    const float scale = (a.silu ? 0.5f : 1.0f) * STATE_F16_UNSCALE;
    // a thread: column dd, eight channels of one node -> one 16-byte chunk of a row
    for (int i = tid; i < (N / 8) * 64; i += blockDim.x) {
        const int dd = i & 15, node = (i >> 4) & 3, c8 = i >> 6;
        const float theta = node == 0 ? 0.9238795325f : node == 1 ? 0.3826834324f : node == 2 ? -0.3826834324f : -0.9238795325f;
        const float tau = (float)seg * len + 0.5f * (len - 1.0f) + 0.5f * len * theta;
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int n = c8 * 8 + e;
            v[e] = a.W[(size_t)n * D + h * HD + c * 16 + dd] * scale * exp2f(tau * log2f(a.rhos[n]));
        }
        *reinterpret_cast<uint4*>(out + (c8 >> 3) * WPIECE + sw_chunk(node * 16 + dd, c8 & 7)) =
            make_uint4(pack_f16x2(v[0], v[1]), pack_f16x2(v[2], v[3]), pack_f16x2(v[4], v[5]), pack_f16x2(v[6], v[7]));
    }
}

// ---------------------------------------------------------------------------------------------------------------
// one CTA per (tile, sample): the item list.  A slot is an item from the tile start to its first occurrence; every
// occurrence is one from the next step to the next occurrence.  Slots in list order, then occurrences in step order; the
// hot slots and their occurrences the same way in blocks after them.
// ---------------------------------------------------------------------------------------------------------------
static constexpr int IL_THREADS = 1024;

struct ListSmem {
    int tok[TM], head[TM], next[TM], occ[TM], slot_of[TM], hkey[256], hval[256], wsum[2][32], hot[HOT], n_hot, dup, total[2];
    unsigned long long best[32];
};

__global__ void __launch_bounds__(IL_THREADS) k_items_list(FlashArgs a, Items it) {
    extern __shared__ float metric[];          // [K]: size of the slot's state in this tile; negative: not a hot candidate
    __shared__ ListSmem s;
    const int tile = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = a.N, CH = N / 8, t0 = tile * TM, bt = b * a.nT + tile;
    const int Lb = a.seq_lens ? min(max(a.seq_lens[b], 0), a.T) : a.T;
    if (t0 >= Lb) {
        if (tid == 0) { it.count[bt] = make_int4(0, 0, 0, 0); it.hot[bt * (HOT + 1)] = 0; }
        return;
    }
    int2* meta = it.meta + (size_t)bt * it.IB * IBLK;
    int* src = it.src + (size_t)bt * it.IB * IBLK;
    if (tid == 0) { s.n_hot = 0; s.dup = 0; s.total[0] = s.total[1] = 0; }
    if (tid < 256) s.hkey[tid] = -1;
    if (tid < TM) {
        s.tok[tid] = (t0 + tid < Lb) ? (int)(a.x[(size_t)b * a.T + t0 + tid] & 0x7fffffffLL) : -1;
        s.slot_of[tid] = -1;
    }
    __syncthreads();
    if (tid < TM) {            // equal tokens inside the tile: their first step, their number, the next one after this
        const int me = s.tok[tid];
        int hd = tid, nx = TM - 1, n = 0;
        for (int j = TM - 1; j >= 0; --j) {
            const bool same = s.tok[j] == me;
            n += same;
            if (same && j < hd) hd = j;
            if (same && j > tid) nx = j;
        }
        s.head[tid] = hd;
        s.next[tid] = nx;
        s.occ[tid] = n;
        if (me >= 0 && hd == tid) {
            int p = (me * 0x9E3779B1u) >> 24;
            while (atomicCAS(&s.hkey[p], -1, me) != -1) p = (p + 1) & 255;
            s.hval[p] = tid;
        }
    }
    __syncthreads();
    // sizes: |state at the tile start| + sqrt(N) per occurrence in the tile
    const __half* snap = reinterpret_cast<const __half*>(a.tile_state + (size_t)a.B * a.nT * a.K * N) + (size_t)bt * a.K * N;
#pragma unroll 2
    for (int i0 = 0; i0 < a.K * CH; i0 += IL_THREADS) {
        const int i = i0 + tid, k = i / CH, c8 = i % CH;
        const bool in = k < a.K;
        const uint4 v = in ? __ldg(reinterpret_cast<const uint4*>(snap + (size_t)k * N) + c8) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float q = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_f16x2(u[e]);
            q = fmaf(f.x, f.x, fmaf(f.y, f.y, q));
        }
        for (int o = CH / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (c8 == 0 && in) {
            const long long kv = a.unique[(size_t)b * a.K + k];
            float m = -1.f;
            if (kv >= 0) {
                m = sqrtf(q) * STATE_F16_UNSCALE;
                const int key = (int)(kv & 0x7fffffffLL);
                int p = (key * 0x9E3779B1u) >> 24;
                while (s.hkey[p] != -1) {
                    if (s.hkey[p] == key) {
                        const int f = s.hval[p];
                        m += (float)s.occ[f] * sqrtf((float)N);
                        if (atomicExch(&s.slot_of[f], k) >= 0) s.dup = 1;     // a token listed twice: every-step kernels
                        break;
                    }
                    p = (p + 1) & 255;
                }
            }
            metric[k] = m;
        }
    }
    __syncthreads();
    // the HOT largest, ties by list order
    for (int r = 0; r < HOT; ++r) {
        unsigned long long best = 0ull;
        for (int k = tid; k < a.K; k += IL_THREADS)
            if (metric[k] >= 0.f) best = max(best, ((unsigned long long)__float_as_uint(metric[k]) << 32) | (unsigned)(0x7fffffff - k));
        for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (lane == 0) s.best[warp] = best;
        __syncthreads();
        if (warp == 0) {
            best = s.best[lane];
            for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && best != 0ull) {
                const int k = 0x7fffffff - (int)(best & 0xffffffffull);
                metric[k] = -2.f;                              // hot
                s.hot[s.n_hot++] = k;
            }
        }
        __syncthreads();
    }
    if (tid <= HOT) it.hot[bt * (HOT + 1) + tid] = tid == 0 ? s.n_hot : (tid - 1 < s.n_hot ? s.hot[tid - 1] : 0);
    // ordered compaction, cold items first
    auto put = [&](bool ok, int cls, int k, int lohi, int from, int base) -> int {     // returns the number of items of class `cls`
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) s.wsum[0][warp] = __popc(m);
        __syncthreads();
        if (warp == 0) {
            int v = s.wsum[0][lane];
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
            s.wsum[1][lane] = v;
        }
        __syncthreads();
        if (ok) {
            const int pos = base + s.total[cls] + (warp ? s.wsum[1][warp - 1] : 0) + __popc(m & ((1u << lane) - 1u));
            meta[pos] = make_int2(k, lohi);
            src[pos] = from;
        }
        const int n = s.wsum[1][31];
        __syncthreads();
        if (tid == 0) s.total[cls] += n;
        __syncthreads();
        return s.total[cls];
    };
    auto first_of = [&](int k) -> int {       // first step of slot k's token in the tile, or the last row
        const int key = (int)(a.unique[(size_t)b * a.K + k] & 0x7fffffffLL);
        int p = (key * 0x9E3779B1u) >> 24;
        while (s.hkey[p] != -1) {
            if (s.hkey[p] == key) return s.hval[p];
            p = (p + 1) & 255;
        }
        return TM - 1;
    };
    for (int k0 = 0; k0 < a.K; k0 += IL_THREADS) {
        const int k = k0 + tid;
        const bool ok = k < a.K && metric[k] >= 0.f;
        put(ok, 0, k, ok ? first_of(k) << 8 : 0, k, 0);
    }
    const int own = tid < TM - 1 && s.tok[tid] >= 0 ? s.slot_of[s.head[tid]] : -1;
    const bool occ = own >= 0, is_hot = occ && metric[own] < 0.f;
    const int n_cold = put(occ && !is_hot, 0, own, occ ? (tid + 1) | (s.next[tid] << 8) : 0, -1 - tid, 0);
    const int base = (n_cold + IBLK - 1) / IBLK * IBLK;
    put(tid < s.n_hot, 1, tid < s.n_hot ? s.hot[tid] : 0, tid < s.n_hot ? first_of(s.hot[tid]) << 8 : 0, tid < s.n_hot ? s.hot[tid] : 0, base);
    const int n_hot = put(is_hot, 1, own, occ ? (tid + 1) | (s.next[tid] << 8) : 0, -1 - tid, base);
    const int n_all = base + n_hot, n_blk = (n_all + IBLK - 1) / IBLK;
    // padding: no valid step, state zero; it names a listed slot, since E rows of unlisted ones may hold anything
    for (int i = n_cold + tid; i < base; i += IL_THREADS) { meta[i] = make_int2(meta[0].x, 1); src[i] = 0x7fffffff; }
    for (int i = n_all + tid; i < n_blk * IBLK; i += IL_THREADS) { meta[i] = make_int2(s.hot[0], 1); src[i] = 0x7fffffff; }
    if (tid == 0) it.count[bt] = make_int4(s.dup ? -1 - n_cold : n_cold, base / IBLK, n_all, n_blk);
}

// ---------------------------------------------------------------------------------------------------------------
// one CTA per (block of items, tile, sample): operand tile, validity masks, |lambda . state|^2
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_items_fill(FlashArgs a, Items it) {
    __shared__ float rho_sh[128], lam_sh[128];
    __shared__ int lohi_sh[IBLK], src_sh[IBLK];
    const int blk = blockIdx.x, bt = blockIdx.z * a.nT + blockIdx.y, tid = threadIdx.x;
    if (blk >= it.count[bt].w) return;
    const int N = a.N, NK = N >> 6, CH = N / 8, b = blockIdx.z, t0 = blockIdx.y * TM;
    const size_t i0 = ((size_t)bt * it.IB + blk) * IBLK;
    if (tid < N) {
        const float r = a.rhos[tid];
        rho_sh[tid] = log2f(r);
        lam_sh[tid] = fabsf(logf(r)) * STATE_F16_UNSCALE;
    }
    if (tid < IBLK) { lohi_sh[tid] = it.meta[i0 + tid].y; src_sh[tid] = it.src[i0 + tid]; }
    __syncthreads();
    const __half* snap = reinterpret_cast<const __half*>(a.tile_state + (size_t)a.B * a.nT * a.K * N) + (size_t)bt * a.K * N;
    const float* toks = a.tok_state + ((size_t)b * a.T + t0) * N;
    unsigned char* img = it.a_img + ((size_t)bt * it.IB + blk) * NK * ATOM;
#pragma unroll 4
    for (int i = tid; i < IBLK * CH; i += 256) {
        const int r = i / CH, c8 = i % CH, from = src_sh[r];
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (from >= 0 && from != 0x7fffffff) {
            v = __ldg(reinterpret_cast<const uint4*>(snap + (size_t)from * N) + c8);
        } else if (from < 0) {
            const int s = -1 - from;
            const float4* p = reinterpret_cast<const float4*>(toks + (size_t)s * N + c8 * 8);
            const float4 p0 = __ldg(p), p1 = __ldg(p + 1);
            const float st[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = (st[e] + 1.0f) * STATE_F16_SCALE * exp2f(-(float)s * rho_sh[c8 * 8 + e]);
            v = make_uint4(pack_f16x2_sat(o[0], o[1]), pack_f16x2_sat(o[2], o[3]), pack_f16x2_sat(o[4], o[5]), pack_f16x2_sat(o[6], o[7]));
        }
        *reinterpret_cast<uint4*>(img + (c8 >> 3) * ATOM + sw_chunk(r, c8 & 7)) = v;
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float q = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_f16x2(u[e]);
            const float x = f.x * lam_sh[c8 * 8 + 2 * e], y = f.y * lam_sh[c8 * 8 + 2 * e + 1];
            q = fmaf(x, x, fmaf(y, y, q));
        }
        for (int o = CH / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (c8 == 0) it.q[i0 + r] = q;
    }
    const int row = tid & (TM - 1), half = tid >> 7;
    unsigned m0 = 0u, m1 = 0u;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
        const int p = lohi_sh[half * 64 + i], q = lohi_sh[half * 64 + 32 + i];
        m0 |= (row >= (p & 255) && row <= (p >> 8)) ? (1u << i) : 0u;
        m1 |= (row >= (q & 255) && row <= (q >> 8)) ? (1u << i) : 0u;
    }
    reinterpret_cast<uint2*>(it.mask + i0 + row)[half] = make_uint2(m0, m1);
}

// ---------------------------------------------------------------------------------------------------------------
// one CTA per (tile, sample): the levels.  v' G v <= |v|^2 times the largest absolute row sum of G (its largest eigenvalue is
// no larger); items whose bound could matter are looked at closely, the others are not.  (The trace bounds it too, but
// twenty times looser: with it a thousand items a tile were looked at, 84 us for 224 tiles.)
// ---------------------------------------------------------------------------------------------------------------
static constexpr int MAX_CHECKED = 1024;
static constexpr int LV_THREADS = 1024, LV_ITEMS = 4;      // a warp looks at four items at once: one read of the Gram matrix for all

__global__ void __launch_bounds__(LV_THREADS) k_levels(FlashArgs a, Items it, Ws w) {
    __shared__ int chk[MAX_CHECKED], n_chk;
    __shared__ unsigned swing_sh[2], decay_sh;          // [0] items before the hot ones, [1] hot items
    __shared__ unsigned row_sh;
    __shared__ float lam_sh[128];
    const int bt = blockIdx.y * a.nT + blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = a.N, NK = N >> 6;
    const int4 cnt = it.count[bt];
    if (cnt.w == 0) {
        if (tid == 0) w.level[bt] = w.level_bwd[bt] = 0;
        return;
    }
    if (tid == 0) { n_chk = 0; row_sh = 0u; swing_sh[0] = swing_sh[1] = decay_sh = 0u; }
    __syncthreads();
    if (tid < N) {
        const float lam = fabsf(logf(a.rhos[tid]));               // rho = 0: infinite, every step
        lam_sh[tid] = lam;
        atomicMax(&decay_sh, __float_as_uint(lam == lam ? lam : INFINITY));
    }
    for (int n = warp; n < N; n += LV_THREADS / 32) {
        float t = 0.f;
        for (int m = lane; m < N; m += 32) t += fabsf(w.gram[n * N + m]);
        t = warp_sum(t);
        if (lane == 0) atomicMax(&row_sh, __float_as_uint(t));
    }
    __syncthreads();
    const float row_sum = __uint_as_float(row_sh);
    const float look = (MAX_SWING / 64.0f) * (MAX_SWING / 64.0f) / fmaxf(row_sum, 1e-30f);
    const float* q = it.q + (size_t)bt * it.IB * IBLK;
    for (int i = tid; i < cnt.w * IBLK; i += LV_THREADS)
        if (!(q[i] <= look)) {
            const int at = atomicAdd(&n_chk, 1);
            if (at < MAX_CHECKED) chk[at] = i;
            else atomicMax(&swing_sh[i >= cnt.y * IBLK], __float_as_uint(q[i] * row_sum));       // list full: the bound itself
        }
    __syncthreads();
    const unsigned char* img = it.a_img + (size_t)bt * it.IB * NK * ATOM;
    const int n_look = min(n_chk, MAX_CHECKED);
    for (int j0 = warp * LV_ITEMS; j0 < n_look; j0 += LV_THREADS / 32 * LV_ITEMS) {      // a lane per channel
        float vl[LV_ITEMS][4], y[LV_ITEMS][4];
#pragma unroll
        for (int g = 0; g < LV_ITEMS; ++g) {
            const int item = chk[min(j0 + g, n_look - 1)], r = item & (IBLK - 1);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int n = lane + 32 * e;
                vl[g][e] = y[g][e] = 0.f;
                if (n < N)
                    vl[g][e] = __half2float(*reinterpret_cast<const __half*>(img + (size_t)(item / IBLK) * NK * ATOM + (n >> 6) * ATOM +
                                                                             sw_chunk(r, (n >> 3) & 7) + (n & 7) * 2)) * (STATE_F16_UNSCALE * lam_sh[n]);
            }
        }
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
            if (32 * e2 >= N) break;
#pragma unroll 4
            for (int l = 0; l < 32; ++l) {
                const float* g = w.gram + (size_t)(32 * e2 + l) * N;
                float gr[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) gr[e] = 32 * e < N ? __ldg(g + lane + 32 * e) : 0.f;
#pragma unroll
                for (int i = 0; i < LV_ITEMS; ++i) {
                    const float vm = __shfl_sync(0xffffffffu, vl[i][e2], l);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (32 * e < N) y[i][e] = fmaf(vm, gr[e], y[i][e]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < LV_ITEMS; ++i) {
            const float v = warp_sum(vl[i][0] * y[i][0] + vl[i][1] * y[i][1] + vl[i][2] * y[i][2] + vl[i][3] * y[i][3]);
            const int item = chk[min(j0 + i, n_look - 1)];
            if (lane == 0) atomicMax(&swing_sh[item >= cnt.y * IBLK], __float_as_uint(v >= 0.f ? v : (v < 0.f ? 0.f : INFINITY)));
        }
    }
    __syncthreads();
    if (tid == 0) {
        const float decay = 64.0f * __uint_as_float(decay_sh);
        auto pick = [&](float max_decay, float q2) {
            const float swing = 64.0f * sqrtf(q2);
            int level = 0;
            while (level < LEVEL_EXACT && !(decay <= max_decay * (float)(1 << level) && swing <= MAX_SWING * (float)(1 << level))) ++level;
            return cnt.x < 0 ? LEVEL_EXACT : level;
        };
        const float cold = __uint_as_float(swing_sh[0]), hot = __uint_as_float(swing_sh[1]);
        w.level[bt] = pick(MAX_DECAY, fmaxf(cold, hot));
        w.level_bwd[bt] = pick(MAX_DECAY_BWD, cold);
    }
}

int build_items(const FlashArgs& a, const Items& it, cudaStream_t st) {
    const size_t smem = (size_t)a.K * sizeof(float);
    k_items_list<<<dim3(a.nT, a.B), IL_THREADS, smem, st>>>(a, it);
    k_items_fill<<<dim3(it.IB, a.nT, a.B), 256, 0, st>>>(a, it);
    return check_launch();
}

int prepare(const FlashArgs& a, const Items& it, const Ws& w, cudaStream_t st) {
    k_weights<<<SEG_IMAGES * a.H * NCH + a.N * a.N / 8, 256, 0, st>>>(a, w);
    k_levels<<<dim3(a.nT, a.B), LV_THREADS, 0, st>>>(a, it, w);
    return check_launch();
}

}  // namespace smooth
}  // namespace mbema
