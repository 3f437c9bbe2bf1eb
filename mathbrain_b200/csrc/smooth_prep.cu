// What the smooth attention kernels read: node-scaled W_pe images, the segments a tile is cut into, and per (sample, tile) the
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
// 1/2 x (SiLU(x) = h + h tanh h, h = x / 2).  The remaining D * N / 2048 blocks, a thread per column and eight channels: the probe
// images (rows of N fp16, 64 x as well) that k_levels reads, and the columns' squared norms.
// ---------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_weights(FlashArgs a, Ws w) {
    const int N = a.N, D = a.H * HD, NK = N >> 6, tid = threadIdx.x;
    const int n_img = SEG_IMAGES * a.H * NCH;
    if ((int)blockIdx.x >= n_img) {
        __shared__ float part[256];
        const int cols = 2048 / N, dd = tid % cols, c8 = tid / cols, d = ((int)blockIdx.x - n_img) * cols + dd;      // D is a multiple of 64
        float f[3][8], sq = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int n = c8 * 8 + e;
            const float l2 = log2f(a.rhos[n]), lam = fabsf(l2) * 0.6931471806f, v = a.W[(size_t)n * D + d];
            sq = fmaf(v, v, sq);
            f[0][e] = v * STATE_F16_UNSCALE * exp2f(63.5f * l2);
            f[1][e] = v * STATE_F16_UNSCALE * 64.0f * lam;
            f[2][e] = f[1][e] * exp2f(127.0f * l2);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint4*>(w.probe + ((size_t)p * D + d) * N + c8 * 8) =
                make_uint4(pack_f16x2(f[p][0], f[p][1]), pack_f16x2(f[p][2], f[p][3]), pack_f16x2(f[p][4], f[p][5]), pack_f16x2(f[p][6], f[p][7]));
        part[tid] = sq;
        __syncthreads();
        if (c8 == 0) {
            for (int i = 1; i < N / 8; ++i) sq += part[i * cols + dd];
            w.wnorm[d] = sq;
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
// one CTA per (block of items, tile, sample): operand tile, validity masks, |lambda . state|^2 (or the share of |state|^2)
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
        float q = 0.f, m2 = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = unpack_f16x2(u[e]);
            m2 = fmaf(f.x, f.x, fmaf(f.y, f.y, m2));
            const float x = f.x * lam_sh[c8 * 8 + 2 * e], y = f.y * lam_sh[c8 * 8 + 2 * e + 1];
            q = fmaf(x, x, fmaf(y, y, q));
        }
        for (int o = CH / 2; o > 0; o >>= 1) {
            q += __shfl_xor_sync(0xffffffffu, q, o);
            m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        }
        constexpr float WT = (STATE_F16_UNSCALE / STATE_WEIGHT) * (STATE_F16_UNSCALE / STATE_WEIGHT);
        if (c8 == 0) it.q[i0 + r] = m2 * WT > q ? m2 * WT : q;        // (NaN stays)
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
// one CTA per (tile, sample): the levels (see smooth.cuh).  Items whose change over half a tile is below SMALL_SWING by Cauchy-Schwarz are
// passed over.  The others (some eighty of the 46M training chunks' 2500) go through warp-level products with every column, for the
// pre-activation at mid-tile and its change over half a tile at the tile's start and end: too few items and columns for a tensor-memory
// pipeline to pay.  A warp keeps half a head's columns and walks the items, so that the images are read once.  Items that one segment does not
// resolve, rare ones, go through another pass for two, and so on.  Bound by the issue of some 25
// instructions a value: 62 us for 224 tiles of N = 64 and 8 heads, 35 us for 64; a root mean square over all columns, which one large column
// escapes, took 31 and 17.
// ---------------------------------------------------------------------------------------------------------------
static constexpr int LV_THREADS = 512, LV_WINDOW = 4096, LV_HEADS = LV_THREADS / 64;      // heads at a time: half a head a warp

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// a lane's share of eight staged rows or columns: contiguous channels, since the contraction may take them in any order
template <int NK> struct Frag {
    uint32_t v[8 * NK];
    __device__ __forceinline__ void load(const __half* p) {
#pragma unroll
        for (int i = 0; i < 2 * NK; ++i) *reinterpret_cast<uint4*>(v + 4 * i) = *(reinterpret_cast<const uint4*>(p) + i);
    }
};
template <int NK>
__device__ __forceinline__ void product(float (&c)[4], const Frag<NK>& lo, const Frag<NK>& hi, const Frag<NK>& col) {
    c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
    for (int k = 0; k < 4 * NK; ++k) {
        const uint32_t a[4] = {lo.v[2 * k], hi.v[2 * k], lo.v[2 * k + 1], hi.v[2 * k + 1]};
        mma_16816(c, a, col.v[2 * k], col.v[2 * k + 1]);
    }
}
// interpolation error of SiLU, root mean square over a segment, for a change of d over half of it
__device__ __forceinline__ float cubic_error(float d) {
    const float d2 = d * d;
    return __fdividef(1.8e-3f * d2 * d2, fmaf(0.033f * d, d2, 1.0f));
}
__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// over a head's columns: squared interpolation error, gate, a quarter for every column with SiLU' >= 1/2
struct Sums { float err, gate, slope; };
template <bool SILU>
__device__ __forceinline__ void add_column(Sums& s, float x, float d, float shrink) {
    const float gate = SILU ? x * fmaf(0.5f, tanh_approx(0.5f * x), 0.5f) : fabsf(x);
    const float er = SILU && fabsf(x) <= d + 3.5f ? cubic_error(d * shrink) : 0.f;
    s.err = fmaf(er, er, s.err);
    s.gate = fmaf(gate, gate, s.gate);
    s.slope += !SILU || x >= 0.f ? 0.25f : 0.f;
}

template <bool SILU, int NK>
__global__ void __launch_bounds__(LV_THREADS) k_levels(FlashArgs a, Items it, Ws w) {
    constexpr int N = NK * 64, LD = N + 8, SH = 16 * NK;          // halves a staged row, a lane's share of it
    constexpr int CHUNK = 64, MT = CHUNK / 16;                    // items at a time
    __shared__ __align__(16) __half rows[CHUNK * LD];
    __shared__ Sums sums[2 * LV_HEADS][CHUNK];
    __shared__ unsigned short chk[LV_WINDOW];             // items to look at, from the start of the window
    __shared__ unsigned char open[2][CHUNK];              // rows that the level before did not resolve
    __shared__ int n_chk, n_open[2];
    __shared__ unsigned fail[2][CHUNK / 32], decay_sh, wmax_sh;      // rows whose gate, slope is not resolved at this level
    __shared__ int need[2];                  // levels of the forward (all items) and of the backward (cold ones)
    const int bt = blockIdx.y * a.nT + blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, jq = lane & 3;
    const int D = a.H * HD;
    const int4 cnt = it.count[bt];
    if (cnt.w == 0) {
        if (tid == 0) w.level[bt] = w.level_bwd[bt] = 0;
        return;
    }
    if (tid == 0) decay_sh = wmax_sh = 0u;
    __syncthreads();
    if (tid < N) {
        const float lam = fabsf(logf(a.rhos[tid]));               // rho = 0: infinite, every step
        atomicMax(&decay_sh, __float_as_uint(lam == lam ? lam : INFINITY));
    }
    float m = 0.f;
    for (int d = tid; d < D; d += LV_THREADS) { const float v = w.wnorm[d]; m = v <= m ? m : (v == v ? v : INFINITY); }
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    if (lane == 0) atomicMax(&wmax_sh, __float_as_uint(m));
    __syncthreads();
    const float decay = 64.0f * __uint_as_float(decay_sh), wmax = __uint_as_float(wmax_sh);
    if (tid == 0) {
        auto resolves = [&](float max_decay) {
            int level = 0;
            while (level < LEVEL_EXACT && !(decay <= max_decay * (float)(1 << level))) ++level;
            return cnt.x < 0 ? LEVEL_EXACT : level;          // a token listed twice: every step in any case
        };
        need[0] = resolves(MAX_DECAY);
        need[1] = resolves(MAX_DECAY_BWD);
    }
    const float look = (SMALL_SWING / 64.0f) * (SMALL_SWING / 64.0f) / fmaxf(wmax, 1e-30f);
    const float* q = it.q + (size_t)bt * it.IB * IBLK;
    const unsigned char* img = it.a_img + (size_t)bt * it.IB * NK * ATOM;
    const int total = cnt.w * IBLK, n_cold = cnt.y * IBLK;
    for (int i0 = 0; i0 < total; i0 += LV_WINDOW) {
        __syncthreads();
        if (tid == 0) n_chk = 0;
        __syncthreads();
        for (int i = i0 + tid; i < min(i0 + LV_WINDOW, total); i += LV_THREADS)
            if (!(q[i] < look)) chk[atomicAdd(&n_chk, 1)] = (unsigned short)(i - i0);
        __syncthreads();
        const int n_look = n_chk;
        for (int j0 = 0; j0 < n_look; j0 += CHUNK) {
            const int n = min(CHUNK, n_look - j0);
            if (need[0] >= LEVEL_EXACT && need[1] >= LEVEL_EXACT) break;          // uniform: written before the last barrier only
            for (int i = tid; i < CHUNK * (N / 8); i += LV_THREADS) {
                const int j = i / (N / 8), c8 = i % (N / 8), item = i0 + chk[j0 + min(j, n - 1)];
                *reinterpret_cast<uint4*>(rows + j * LD + c8 * 8) =
                    *reinterpret_cast<const uint4*>(img + ((size_t)(item / IBLK) * NK + (c8 >> 3)) * ATOM + sw_chunk(item & (IBLK - 1), c8 & 7));
            }
            if (tid < CHUNK) open[0][tid] = (unsigned char)min(tid, n - 1);
            if (tid == 0) n_open[0] = n;
            // of row `tid`: gate, slope (cold items only) not resolved yet at the level; a level that the tile needs anyway is not looked at
            const bool cold = tid < n && i0 + chk[j0 + tid] < n_cold;
            bool open_g = true, open_s = cold;
            const int first = min(need[0], need[1]);
            for (int level = first; level < LEVEL_EXACT; ++level) {
                const unsigned char* list = open[(level - first) & 1];
                int* m_open = &n_open[(level - first) & 1];
                if (tid < CHUNK / 32) fail[0][tid] = fail[1][tid] = 0u;
                if (tid == 0) n_open[(level - first + 1) & 1] = 0;
                __syncthreads();
                const int m_rows = *m_open, mts = (m_rows + 15) / 16;
                if (m_rows == 0) break;
                const float shrink = 1.0f / (float)(1 << level);
                for (int h0 = 0; h0 < a.H; h0 += LV_HEADS) {
                    const int heads = min(LV_HEADS, a.H - h0);
                    if (warp < 2 * heads) {
                        Sums acc[MT][2];
#pragma unroll
                        for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = Sums{0.f, 0.f, 0.f};
                        const __half* col = w.probe + ((size_t)h0 * HD + warp * 32 + g) * N + jq * SH;
                        Frag<NK> B[3];
#pragma unroll
                        for (int p = 0; p < 3; ++p) B[p].load(col + (size_t)p * D * N);
#pragma unroll 1
                        for (int nt = 0; nt < 4; ++nt) {
                            // the next columns are on their way while these are worked on
                            const __half* next = col + (size_t)min(nt + 1, 3) * 8 * N;
#pragma unroll
                            for (int p = 0; p < 3; ++p) asm volatile("prefetch.global.L1 [%0];" ::"l"(next + (size_t)p * D * N));
#pragma unroll
                            for (int m = 0; m < MT; m += 2) {          // two at a time: their chains run side by side
                                if (m >= mts) break;
                                float c[2][3][4];
#pragma unroll
                                for (int k = 0; k < 2; ++k) {
                                    Frag<NK> lo, hi;
                                    lo.load(rows + list[min((m + k) * 16 + g, m_rows - 1)] * LD + jq * SH);
                                    hi.load(rows + list[min((m + k) * 16 + 8 + g, m_rows - 1)] * LD + jq * SH);
#pragma unroll
                                    for (int p = 0; p < 3; ++p) product<NK>(c[k][p], lo, hi, B[p]);
                                }
#pragma unroll
                                for (int e = 0; e < 4; ++e)
#pragma unroll
                                    for (int k = 0; k < 2; ++k)
                                        add_column<SILU>(acc[m + k][e >> 1], c[k][0][e], fmaxf(fabsf(c[k][1][e]), fabsf(c[k][2][e])), shrink);
                            }
#pragma unroll
                            for (int p = 0; p < 3; ++p) B[p].load(next + (size_t)p * D * N);
                        }
#pragma unroll
                        for (int m = 0; m < MT; ++m)
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const Sums t{quad_sum(acc[m][s].err), quad_sum(acc[m][s].gate), quad_sum(acc[m][s].slope)};
                                if (jq == 0) sums[warp][m * 16 + 8 * s + g] = t;
                            }
                    }
                    __syncthreads();
                    for (int i = tid; i < m_rows * heads; i += LV_THREADS) {
                        const int j = i % m_rows, h = i / m_rows, r = list[j];
                        const Sums u = sums[2 * h][j], v = sums[2 * h + 1][j];
                        const float es = u.err + v.err, gs = u.gate + v.gate;
                        if (!(gs < MAX_GATE * MAX_GATE && es <= TOL_GATE * TOL_GATE * gs)) atomicOr(&fail[0][r >> 5], 1u << (r & 31));
                        if (!(gs < MAX_GATE * MAX_GATE && es <= TOL_SLOPE * TOL_SLOPE * (u.slope + v.slope))) atomicOr(&fail[1][r >> 5], 1u << (r & 31));
                    }
                    __syncthreads();
                }
                if (tid < n) {
                    open_g = open_g && ((fail[0][tid >> 5] >> (tid & 31)) & 1u);
                    open_s = open_s && ((fail[1][tid >> 5] >> (tid & 31)) & 1u);
                    if (open_g) atomicMax(&need[0], level + 1);
                    if (cold && (open_g || open_s)) atomicMax(&need[1], level + 1);
                    if (open_g || open_s) open[(level - first + 1) & 1][atomicAdd(&n_open[(level - first + 1) & 1], 1)] = (unsigned char)tid;
                }
                __syncthreads();
            }
            __syncthreads();
        }
    }
    __syncthreads();
    if (tid == 0) {
        w.level[bt] = need[0];
        w.level_bwd[bt] = need[1];
    }
}

int build_items(const FlashArgs& a, const Items& it, cudaStream_t st) {
    const size_t smem = (size_t)a.K * sizeof(float);
    k_items_list<<<dim3(a.nT, a.B), IL_THREADS, smem, st>>>(a, it);
    k_items_fill<<<dim3(it.IB, a.nT, a.B), 256, 0, st>>>(a, it);
    return check_launch();
}

int prepare(const FlashArgs& a, const Items& it, const Ws& w, cudaStream_t st) {
    k_weights<<<SEG_IMAGES * a.H * NCH + a.H * HD * a.N / 2048, 256, 0, st>>>(a, w);
    const dim3 grid(a.nT, a.B);
    if (a.silu) {
        if (a.N == 64) k_levels<true, 1><<<grid, LV_THREADS, 0, st>>>(a, it, w);
        else k_levels<true, 2><<<grid, LV_THREADS, 0, st>>>(a, it, w);
    } else {
        if (a.N == 64) k_levels<false, 1><<<grid, LV_THREADS, 0, st>>>(a, it, w);
        else k_levels<false, 2><<<grid, LV_THREADS, 0, st>>>(a, it, w);
    }
    return check_launch();
}

}  // namespace smooth
}  // namespace mbema
