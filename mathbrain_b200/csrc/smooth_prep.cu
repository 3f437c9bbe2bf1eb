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
// 1/2 x (SiLU(x) = h + h tanh h, h = x / 2).  The remaining N blocks: one row of the Gram matrix each.
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_weights(FlashArgs a, Ws w) {
    const int N = a.N, D = a.H * HD, NK = N >> 6, tid = threadIdx.x;
    const int n_img = SEG_IMAGES * a.H * NCH;
    if ((int)blockIdx.x >= n_img) {
        const int n = blockIdx.x - n_img, lane = tid & 31;
        for (int m = tid >> 5; m < N; m += 8) {
            float s = 0.f;
            for (int d = lane; d < D; d += 32) s = fmaf(a.W[(size_t)n * D + d], a.W[(size_t)m * D + d], s);
            s = warp_sum(s);
            if (lane == 0) w.gram[n * N + m] = s / (float)D;
        }
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
// one CTA per (tile, sample): items, their operand tiles, validity masks and the tile's level
// ---------------------------------------------------------------------------------------------------------------
static constexpr int IT_THREADS = 256;
static constexpr int MAX_CHECKED = 1024;

__global__ void __launch_bounds__(IT_THREADS) k_items(FlashArgs a, Ws w) {
    __shared__ int tok[TM], head[TM], next[TM], slot_of[TM];
    __shared__ int hkey[256], hval[256];
    __shared__ int wsum[8], n_items_sh, exact_sh, n_chk;
    __shared__ unsigned swing_sh, decay_sh;
    __shared__ int chk[MAX_CHECKED];
    __shared__ float rho_sh[128], lam_sh[128];
    __shared__ int lohi_sh[IBLK];
    const int tile = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = a.N, NK = N >> 6, CH = N / 8, t0 = tile * TM;
    const int bt = b * a.nT + tile;
    const int Lb = a.seq_lens ? min(max(a.seq_lens[b], 0), a.T) : a.T;
    if (t0 >= Lb) {
        if (tid == 0) { w.n_items[bt] = 0; w.level[bt] = w.level_bwd[bt] = 0; }
        return;
    }
    int2* meta = w.meta + (size_t)bt * w.IB * IBLK;
    if (tid == 0) { n_items_sh = 0; exact_sh = 0; n_chk = 0; swing_sh = 0u; decay_sh = 0u; }
    hkey[tid] = -1;
    if (tid < TM) {
        tok[tid] = (t0 + tid < Lb) ? (int)(a.x[(size_t)b * a.T + t0 + tid] & 0x7fffffffLL) : -1;
        slot_of[tid] = -1;
    }
    __syncthreads();
    if (tid < N) {
        const float r = a.rhos[tid];
        const float lam = fabsf(logf(r));                     // rho = 0: infinite, exact path
        rho_sh[tid] = log2f(r);
        lam_sh[tid] = lam;
        atomicMax(&decay_sh, __float_as_uint(lam == lam ? lam : INFINITY));
    }
    if (tid < TM) {            // chains of equal tokens inside the tile: their first step, and the next one after this
        const int me = tok[tid];
        int hd = tid, nx = TM - 1;
        for (int j = TM - 1; j >= 0; --j) {
            const bool same = tok[j] == me;
            if (same && j < hd) hd = j;
            if (same && j > tid) nx = j;
        }
        head[tid] = hd;
        next[tid] = nx;
        if (me >= 0 && hd == tid) {
            int p = (me * 0x9E3779B1u) >> 24;
            while (atomicCAS(&hkey[p], -1, me) != -1) p = (p + 1) & 255;
            hval[p] = tid;
        }
    }
    __syncthreads();
    // slots in list order
    const int n_valid = a.kcount[b];
    for (int k0 = 0; k0 < a.K && n_items_sh < n_valid; k0 += IT_THREADS) {
        const int k = k0 + tid;
        const long long kv = (k < a.K) ? a.unique[(size_t)b * a.K + k] : -1;
        const bool ok = kv >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int pos = n_items_sh + __popc(m & ((1u << lane) - 1u)), total = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) { if (i < warp) pos += wsum[i]; total += wsum[i]; }
        if (ok) {
            const int key = (int)(kv & 0x7fffffffLL);
            int p = (key * 0x9E3779B1u) >> 24, first = -1;
            while (hkey[p] != -1) {
                if (hkey[p] == key) { first = hval[p]; break; }
                p = (p + 1) & 255;
            }
            if (first >= 0 && atomicExch(&slot_of[first], k) >= 0) exact_sh = 1;     // a token listed twice
            meta[pos] = make_int2(k, (first >= 0 ? first : TM - 1) << 8);
        }
        __syncthreads();
        if (tid == 0) n_items_sh += total;
        __syncthreads();
    }
    const int n_slots = n_items_sh;
    {   // occurrences that have steps after them in the tile
        const bool ok = tid < TM - 1 && tok[tid & (TM - 1)] >= 0 && slot_of[head[tid & (TM - 1)]] >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int pos = n_slots + __popc(m & ((1u << lane) - 1u)), total = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) { if (i < warp) pos += wsum[i]; total += wsum[i]; }
        if (ok) meta[pos] = make_int2(-1 - tid, (tid + 1) | (next[tid] << 8));
        __syncthreads();
        if (tid == 0) n_items_sh += total;
        __syncthreads();
    }
    const int n_items = n_items_sh, n_blk = (n_items + IBLK - 1) / IBLK;
    // operand tiles; the items' lambda . M is bounded on the way, and those that could matter are listed for a closer look
    float trace = 0.f;
    for (int n = 0; n < N; ++n) trace += w.gram[n * N + n];
    const float look = (MAX_SWING / 64.0f) * (MAX_SWING / 64.0f) / fmaxf(trace, 1e-30f);     // |v|^2 tr(G) >= v' G v
    const __half* snap = reinterpret_cast<const __half*>(a.tile_state + (size_t)a.B * a.nT * a.K * N) + (size_t)bt * a.K * N;
    const float* toks = a.tok_state + ((size_t)b * a.T + t0) * N;
    unsigned char* img = w.a_img + (size_t)bt * w.IB * NK * ATOM;
    for (int i = tid; i < n_blk * IBLK * CH; i += IT_THREADS) {
        const int item = i / CH, c8 = i % CH, r = item & (IBLK - 1);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (item < n_items) {
            const int src = meta[item].x;
            if (src >= 0) {
                v = __ldg(reinterpret_cast<const uint4*>(snap + (size_t)src * N) + c8);
            } else {
                const int s = -1 - src;
                const float4* p = reinterpret_cast<const float4*>(toks + (size_t)s * N + c8 * 8);
                const float4 p0 = __ldg(p), p1 = __ldg(p + 1);
                const float st[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
                float o[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) o[e] = (st[e] + 1.0f) * STATE_F16_SCALE * exp2f(-(float)s * rho_sh[c8 * 8 + e]);
                v = make_uint4(pack_f16x2_sat(o[0], o[1]), pack_f16x2_sat(o[2], o[3]), pack_f16x2_sat(o[4], o[5]), pack_f16x2_sat(o[6], o[7]));
            }
        }
        *reinterpret_cast<uint4*>(img + (size_t)(item / IBLK) * NK * ATOM + (c8 >> 3) * ATOM + sw_chunk(r, c8 & 7)) = v;
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        float q = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_f16x2(u[e]);
            const float x = f.x * lam_sh[c8 * 8 + 2 * e], y = f.y * lam_sh[c8 * 8 + 2 * e + 1];
            q = fmaf(x, x, fmaf(y, y, q));
        }
        for (int o = CH / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        q *= STATE_F16_UNSCALE * STATE_F16_UNSCALE;
        if (c8 == 0 && !(q <= look)) {
            const int at = atomicAdd(&n_chk, 1);
            if (at < MAX_CHECKED) chk[at] = item;
            else atomicMax(&swing_sh, __float_as_uint(q * trace));       // list full: the bound itself
        }
    }
    __syncthreads();
    // v' G v of the listed items: a warp each, a lane per channel
    for (int j = warp; j < min(n_chk, MAX_CHECKED); j += IT_THREADS / 32) {
        const int item = chk[j], r = item & (IBLK - 1);
        float vl[4], y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = lane + 32 * e;
            vl[e] = y[e] = 0.f;
            if (n < N)
                vl[e] = __half2float(*reinterpret_cast<const __half*>(img + (size_t)(item / IBLK) * NK * ATOM + (n >> 6) * ATOM +
                                                                      sw_chunk(r, (n >> 3) & 7) + (n & 7) * 2)) * (STATE_F16_UNSCALE * lam_sh[n]);
        }
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
            if (32 * e2 >= N) break;
            for (int l = 0; l < 32; ++l) {
                const float vm = __shfl_sync(0xffffffffu, vl[e2], l);
                const float* g = w.gram + (size_t)(32 * e2 + l) * N;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (32 * e < N) y[e] = fmaf(vm, __ldg(g + lane + 32 * e), y[e]);
            }
        }
        const float q = warp_sum(vl[0] * y[0] + vl[1] * y[1] + vl[2] * y[2] + vl[3] * y[3]);
        if (lane == 0) atomicMax(&swing_sh, __float_as_uint(q >= 0.f ? q : (q < 0.f ? 0.f : INFINITY)));
    }
    // what the kernels read of an item: its row of the E tables and its steps
    __syncthreads();
    for (int i = tid; i < n_blk * IBLK; i += IT_THREADS) {
        int2 o = make_int2(0, 1);                          // padding: first step after the last
        if (i < n_items) {
            const int2 mt = meta[i];
            const int k = mt.x >= 0 ? mt.x : slot_of[head[-1 - mt.x]];
            o = make_int2(a.erow ? a.erow[(size_t)b * a.K + k] : b * a.K + k, mt.y);
        } else if (a.erow == nullptr) {
            o.x = b * a.K;
        }
        meta[i] = o;
    }
    __syncthreads();
    uint4* mask = w.mask + (size_t)bt * w.IB * IBLK;
    for (int blk = 0; blk < n_blk; ++blk) {
        if (tid < IBLK) lohi_sh[tid] = meta[blk * IBLK + tid].y;
        __syncthreads();
        const int row = tid & (TM - 1), half = tid >> 7;
        unsigned m0 = 0u, m1 = 0u;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
            const int p = lohi_sh[half * 64 + i], q = lohi_sh[half * 64 + 32 + i];
            m0 |= (row >= (p & 255) && row <= (p >> 8)) ? (1u << i) : 0u;
            m1 |= (row >= (q & 255) && row <= (q >> 8)) ? (1u << i) : 0u;
        }
        reinterpret_cast<uint2*>(mask + blk * IBLK + row)[half] = make_uint2(m0, m1);
        __syncthreads();
    }
    if (tid == 0) {
        w.n_items[bt] = n_items;
        const float swing = 64.0f * sqrtf(__uint_as_float(swing_sh)), decay = 64.0f * __uint_as_float(decay_sh);
        auto pick = [&](float max_decay) {
            int level = 0;
            while (level < LEVEL_EXACT && !(decay <= max_decay * (float)(1 << level) && swing <= MAX_SWING * (float)(1 << level))) ++level;
            return exact_sh ? LEVEL_EXACT : level;
        };
        w.level[bt] = pick(MAX_DECAY);
        w.level_bwd[bt] = pick(MAX_DECAY_BWD);
    }
}

int prepare(const FlashArgs& a, const Ws& w, cudaStream_t st) {
    k_weights<<<SEG_IMAGES * a.H * NCH + a.N, 256, 0, st>>>(a, w);
    k_items<<<dim3(a.nT, a.B), IT_THREADS, 0, st>>>(a, w);
    return check_launch();
}

}  // namespace smooth
}  // namespace mbema
