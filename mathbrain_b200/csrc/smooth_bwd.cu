// Flash-EMA attention backward over smooth slot states (see smooth.cuh): one CTA per (tile, head, sample).
//
// Per block of 128 items, with K_c = E_k c_j and V_c = E_v c_j per chunk of 16 columns (x 4 coefficients) as in the forward:
//   first pass     S^T  [items x steps] += K_c . Q'_c^T,   dP^T += V_c . dO'_c^T
//   softmax        P^T = exp(S - LSE), dS^T = P (dP - D): tensor memory, dS^T also in shared memory
//   second pass    dK_c = dS^T . Q'_c,   dV_c = P^T . dO'_c,   dQ'_c = dS . K_c (K_c built again),
//                  dE_k, dE_v, and the gate's node gradients dpre from them; dW += A^T . (sum_i dpre_i, sum_i theta_i dpre_i)
// W_pe's gradient takes the node powers rho^tau_i as a0 + a1 theta_i (two products instead of four): the part left out is
// (lambda * half tile)^2 / 4 <= 5e-4 of the fastest channel (MAX_DECAY_BWD), a rounding of the fp16 operand.
// Its products take two chunks at once (64 columns): products of 32 cost the tensor pipe as much, 2.40 ms a layer at B=56, T=512,
// N=64 against 2.34.
//
// Two gate warpgroups (a thread per item, half of a chunk's columns each), two step warpgroups (softmax: a thread per item and half
// the steps; then a thread per step for dQ), a loader lane and two issuing lanes.  Registers and tensor memory hold all
// that shared memory (224 KB: Q' 64, dO' 64, states 16, dS 32, W' 16, two operand tiles 32) has no room for; for 128
// channels dO' is streamed through two stages from a copy in the workspace instead.
// The 16-bit gradients are scaled by powers of two, so that none leaves the fp16 range whatever the values: P by 2^kappa from
// the share of the listed slots in the softmax, dO by a factor per row from the
// row's largest value (rows of very different size stand in a tile: well predicted tokens beside others), dS per block from the largest P |dP - D| of
// its items (|dP - D| has no bound of its own: it is of the size of dO times the values), the moments per block from a bound on
// the sums in them; dW, summed in tensor memory, leaves it when its unit changes.
#include "smooth.cuh"
#include "smooth_dev.cuh"

namespace mbema {
namespace smooth {

using namespace ptx;

namespace bwd {

static constexpr int GATE_WARPS = 8, SM_WARPS = 8;
static constexpr int W_LOAD = 16, W_GATE = 17, W_ATT = 18;       // warp 19 only fills the warpgroup
static constexpr int THREADS = 20 * 32;      // launched with 96 registers a thread: 61440 = 512 * 104 + 128 * 64
static constexpr uint32_t T_S = 0, T_DP = 128, T_DQ = 256, T_PRE = 320, T_DW = 384;
static constexpr float LN2 = 0.6931471806f;

struct Bars {
    uint64_t a_full, w_full[2], w_free[2], do_full[2], do_free[2];
    uint64_t pre1_full[2], pre2_full[2], pre_empty[2], kv_full[2], kv_free[2], sdp_full, s_read, pds_full;
    uint64_t dkv_full[2], dkv_empty, kg_full[2], kg_free[2], dq_full[2], dq_empty, dpre_full[2], dp_free, blk_done, drain;
    uint32_t tmem_base;
    int abort_flag, drain_flag, emin, bad;      // emin: exponent of the row factor of the largest |dO|; bad: a row of dO is not finite
    unsigned spin_limit, pmax, qmax;
    // of the block worked on, per warp: largest P |dP - D| of an item (a bound on it), |dP - D|, P; largest |E / 4|
    alignas(16) float red_b[SM_WARPS], red_x[SM_WARPS], red_p[SM_WARPS], red_e[GATE_WARPS];
    float fs, fm;                              // its factors of dS and of the moments
    float fw, fw_old;                          // their product, the unit of the dW sums: it stays while the blocks fit; the one before
    int dw_fresh;                              // the block's dW products start the sums anew
};

template <int NK> struct L {
    static constexpr int NDO = NK == 1 ? NCH : 2;
    static constexpr int Q = 0, DO = Q + NCH * ATOM, A = DO + NDO * ATOM, DS = A + NK * ATOM, W = DS + 2 * ATOM, B0 = W + 2 * WPIECE,
                         B1 = B0 + ATOM, LSE = B1 + ATOM, DL = LSE + TM * 4, GF = DL + TM * 4, RX = GF + TM * 2, BAR = RX + TM, SMEM = BAR + 640 + 1024;
    static_assert(sizeof(Bars) <= 640 && BAR % 16 == 0 && SMEM <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ f32x2 unpack_h2(uint32_t v) {
    const float2 f = unpack_f16x2(v);
    return pack2(f.x, f.y);
}
__device__ __forceinline__ void red_v4(float* p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

__device__ __forceinline__ uint32_t max_f16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ float larger_half(uint32_t v) {
    const float2 f = unpack_f16x2(v);
    return fmaxf(f.x, f.y);
}
__device__ __forceinline__ float warp_max(float v) {      // v >= 0
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ float max8(const float* p) {
    const float4 u = *reinterpret_cast<const float4*>(p), v = *reinterpret_cast<const float4*>(p + 4);
    return fmaxf(fmaxf(fmaxf(u.x, u.y), fmaxf(u.z, u.w)), fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
}
// 2^14 <= v * scale < 2^15, a power of two between 2^-lo and 2^hi
__device__ __forceinline__ float scale_to_f16(float v, int lo, int hi) {
    const int e = 14 - ((int)(__float_as_uint(v) >> 23) - 127);
    return __uint_as_float((uint32_t)(127 + max(-lo, min(hi, e))) << 23);
}
__device__ __forceinline__ float inverse(float power_of_two) { return __uint_as_float((254u << 23) - __float_as_uint(power_of_two)); }
// factor of dS beside those of P and dO: neither P |dP - D| nor |dP - D| leaves the fp16 range
__device__ __forceinline__ float ds_scale(const Bars* bars) { return scale_to_f16(fmaxf(max8(bars->red_b), max8(bars->red_x)), 60, 16); }

template <bool SILU, int NK, bool EF32>
__global__ void __launch_bounds__(THREADS, 1) k_smooth_bwd(FlashArgs a, Items it, Ws w, int* status) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    using M = L<NK>;
    Bars* bars = reinterpret_cast<Bars*>(sm + M::BAR);
    float* lse_sh = reinterpret_cast<float*>(sm + M::LSE);     // log2(e) LSE - kappa; +inf for rows that do not count
    float* dl_sh = reinterpret_cast<float*>(sm + M::DL);       // row factor times D
    __half* gf_sh = reinterpret_cast<__half*>(sm + M::GF);     // smallest row factor over the row's
    unsigned char* rx_sh = sm + M::RX;                         // its exponent, negated; 255: dO is not finite
    volatile int* abort_flag = &bars->abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x, h = blockIdx.y, b = a.order ? a.order[blockIdx.z] : (int)blockIdx.z;
    const int bt = b * a.nT + tile, t0 = tile * TM, D = a.H * HD, N = NK * 64;
    const int Lb = a.seq_lens ? min(max(a.seq_lens[b], 0), a.T) : a.T;
    const int level = w.level_bwd[bt];
    if (level == LEVEL_EXACT) return;
    const size_t row0 = ((size_t)b * a.H + h) * a.T + t0;
    // this head's half of the tile's dW_pe partial [N][128]
    float* part = a.dW_part + (((size_t)b * (a.H / 2) + (h >> 1)) * a.nT + tile) * N * 128 + (h & 1) * HD;
    if (t0 >= Lb) {          // a tile beyond the valid length
        for (int i = tid; i < min(TM, a.T - t0) * (HD / 4); i += THREADS)
            *reinterpret_cast<float4*>(a.dQ + (row0 + i / (HD / 4)) * HD + (i % (HD / 4)) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = tid; i < N * (HD / 4); i += THREADS)
            *reinterpret_cast<float4*>(part + (i / (HD / 4)) * 128 + (i % (HD / 4)) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        return;
    }
    if (tid == 0) {
        mbar_init(&bars->a_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->w_full[i], 1); mbar_init(&bars->w_free[i], 1);
            mbar_init(&bars->do_full[i], 1); mbar_init(&bars->do_free[i], 1);
            mbar_init(&bars->pre1_full[i], 1); mbar_init(&bars->pre2_full[i], 1); mbar_init(&bars->pre_empty[i], GATE_WARPS);
            mbar_init(&bars->kv_full[i], GATE_WARPS); mbar_init(&bars->kv_free[i], 1);
            mbar_init(&bars->dkv_full[i], 1); mbar_init(&bars->kg_full[i], GATE_WARPS); mbar_init(&bars->kg_free[i], 1);
            mbar_init(&bars->dq_full[i], 1); mbar_init(&bars->dpre_full[i], GATE_WARPS);
        }
        mbar_init(&bars->sdp_full, 1); mbar_init(&bars->s_read, SM_WARPS); mbar_init(&bars->pds_full, SM_WARPS);
        mbar_init(&bars->dkv_empty, GATE_WARPS); mbar_init(&bars->dq_empty, 4);
        mbar_init(&bars->dp_free, 1); mbar_init(&bars->blk_done, 1); mbar_init(&bars->drain, 2);
        bars->abort_flag = *reinterpret_cast<volatile int*>(status);
        bars->drain_flag = 0;
        bars->spin_limit = a.test_withhold ? 64u : MBEMA_SPIN_LIMIT;
        bars->emin = INT_MAX;
        bars->bad = 0;
        bars->pmax = 0u;
        bars->fw = 0.f;
        bars->qmax = 0u;
        fence_barrier_init();
    }
    if (warp == W_GATE) {
        tmem_alloc(&bars->tmem_base, 512);
        tmem_relinquish();
    }
    __syncthreads();
    // Q' and dO' tiles (thread: step t, chunk c), D = dO . O, the scales
    const float rest = a.v_total - (float)a.kcount[b];
    float kappa = 15.f;
    int emin;
    {
        const int t = tid & (TM - 1), c = (tid >> 7) & 3;
        const bool ok = t0 + t < Lb;
        float beta[NJ], v[16];
        basis(t, level, beta);
        float* scr = reinterpret_cast<float*>(sm + M::B0);                    // [4][128] partial sums of dO . O
        unsigned* scm = reinterpret_cast<unsigned*>(sm + M::B0) + NCH * TM;    // [4][128] largest |dO| (as bits: NaN above infinity)
        if (tid < TM * NCH) {
            float dot = 0.f, qm = 0.f;
            unsigned mx = 0u;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 q = ok ? ld4_dyn_f32(a.Q, a.q_dt, (row0 + t) * HD + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
                qm = fmaxf(qm, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))));
            }
            qm = warp_max(qm);
            if (lane == 0) atomicMax(&bars->qmax, __float_as_uint(qm));
            store_basis_rows(sm + M::Q + c * ATOM, t, v, beta, 0.125f * 1.4426950409f);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 g = ok ? ld4_dyn_f32(a.dO, a.do_dt, (row0 + t) * HD + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 o = ok ? *reinterpret_cast<const float4*>(a.O + (row0 + t) * HD + c * 16 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[i] = g.x; v[i + 1] = g.y; v[i + 2] = g.z; v[i + 3] = g.w;
                dot += g.x * o.x + g.y * o.y + g.z * o.z + g.w * o.w;
#pragma unroll
                for (int e = 0; e < 4; ++e) mx = max(mx, __float_as_uint(fabsf(v[i + e])));
            }
            scr[c * TM + t] = dot;
            scm[c * TM + t] = mx;
            if (c == 0) {
                float share = 1.f;
                if (!a.listed_only && rest > 0.f) share = ok ? 1.f - rest * __expf(-a.LSE[row0 + t]) : 0.f;
                for (int o = 16; o > 0; o >>= 1) share = fmaxf(share, __shfl_xor_sync(0xffffffffu, share, o));
                if (lane == 0) atomicMax(&bars->pmax, __float_as_uint(fmaxf(share, 0.f)));
            }
        }
        __syncthreads();
        kappa = 15.f + floorf(-log2f(fminf(fmaxf(__uint_as_float(bars->pmax), 1.0f / 512.0f), 1.0f)));
        int er = INT_MAX;          // exponent of the row's factor: largest |dO| of the row in [2^13, 2^14)
        bool bad = false;
        if (tid < TM * NCH) {
            const unsigned m = max(max(scm[t], scm[TM + t]), max(scm[2 * TM + t], scm[3 * TM + t]));
            const float dl = scr[t] + scr[TM + t] + scr[2 * TM + t] + scr[3 * TM + t];
            if (m != 0u) er = max(-114, min(80, 13 + 127 - (int)(m >> 23)));
            const float rs = m != 0u ? exp2f((float)er) : 1.f;
            bad = m >= 0x7f800000u || !(fabsf(dl * rs) < INFINITY);
            // a row that is not finite is left out of the products; everything it reaches becomes NaN at the end
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = bad ? 0.f : v[i] * rs;
            if (NK == 1) {
                store_basis_rows(sm + M::DO + c * ATOM, t, v, beta, 1.0f);
            } else {
                unsigned char* img = w.do_img + ((size_t)bt * a.H + h) * NCH * ATOM;
                store_basis_rows(img + c * ATOM, t, v, beta, 1.0f);
            }
            if (c == 0) {
                lse_sh[t] = ok ? a.LSE[row0 + t] * 1.4426950409f - kappa : INFINITY;
                dl_sh[t] = bad ? 0.f : dl * rs;
                const int e = __reduce_min_sync(0xffffffffu, bad ? INT_MAX : er);
                const bool any = __any_sync(0xffffffffu, bad);
                if (lane == 0) {
                    atomicMin(&bars->emin, e);
                    if (any) bars->bad = 1;
                }
            }
        }
        __syncthreads();
        emin = bars->emin == INT_MAX ? 0 : bars->emin;
        if (tid < TM) {
            const int k = bad || er == INT_MAX ? 0 : er - emin;
            gf_sh[t] = __float2half_rn(exp2f((float)-k));
            rx_sh[t] = bad ? 255 : k;
        }
    }
    for (int i = tid; i < N * (HD / 4); i += THREADS)
        *reinterpret_cast<float4*>(part + (i / (HD / 4)) * 128 + (i % (HD / 4)) * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    asm volatile("fence.proxy.async;" ::: "memory");      // the operand tiles, in shared memory and (NK = 2) in the workspace
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = bars->tmem_base;
    const int n_items = it.count[bt].x, n_blk = it.count[bt].y;          // the hot slots are the every-step kernel's
    const int n_it = bars->abort_flag ? 0 : n_blk << level;
    const unsigned* lim = &bars->spin_limit;
    const float unit = exp2f(kappa + (float)emin);      // factor of P dO; dS, dK, dc and dpre carry it times the block's factor (dS ln 2 more)

    if (warp < GATE_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        // ======================================================== gate: item r, columns 8 wg .. 8 wg + 7 of every chunk
        const int wg = warp >> 2, r = tid & 127, x7 = r & 7;
        const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int2* meta = it.meta + (size_t)bt * it.IB * IBLK + r;
        const float ov = 0.25f / unit * (bars->bad ? NAN : 1.0f);
        // the dW sums in tensor memory, in the unit `fw`: lane n, chunks 2 wg and 2 wg + 1
        auto flush = [&](int seg, float fw) {
            tc_fence_after_sync();
            if (r < N) {         // whole warps
                const float len = (float)(TM >> level), l2 = log2f(a.rhos[r]);
                const float mid = (float)seg * len + 0.5f * (len - 1.0f), ha = 0.5f * len * 0.9238795325f, hb = 0.5f * len * 0.3826834324f;
                const float pa = exp2f(l2 * (mid + ha)), pb = exp2f(l2 * (mid + hb)), pc = exp2f(l2 * (mid - hb)), pd = exp2f(l2 * (mid - ha));
                const float sc = 4.0f * STATE_F16_UNSCALE * ov * inverse(fw);
                const float r0 = 0.25f * (pa + pb + pc + pd) * sc, r1 = 0.5f * (0.9238795325f * (pa - pd) + 0.3826834324f * (pb - pc)) * sc;
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    float d0[8], d1[8];
                    const uint32_t td = t_lane + T_DW + wg * 64 + (q >> 1) * 32 + (q & 1) * 8;
                    tmem_ld_32x32b_x8(td, d0);
                    tmem_ld_32x32b_x8(td + 16, d1);
                    tmem_wait_ld();
                    float* o = part + (size_t)r * 128 + (2 * wg + (q >> 1)) * 16 + (q & 1) * 8;
#pragma unroll
                    for (int dd = 0; dd < 8; dd += 4) {
                        const float4 v = make_float4(r0 * d0[dd] + r1 * d1[dd], r0 * d0[dd + 1] + r1 * d1[dd + 1], r0 * d0[dd + 2] + r1 * d1[dd + 2],
                                                     r0 * d0[dd + 3] + r1 * d1[dd + 3]);
                        red_v4(o + dd, v.x, v.y, v.z, v.w);
                    }
                }
            }
            tc_fence_before_sync();
        };
        size_t eo = 0;          // this item's E columns of chunk 0
        ERow<EF32> ek, ev;
        if (n_it > 0) {
            eo = e_row(a, b, __ldg(&meta[0].x)) * D + h * HD + wg * 8;
            ek = load_e<EF32>(a.Ek, eo);
            ev = load_e<EF32>(a.Ev, eo);
        }
        bool alive = true;
        for (int i = 0; i < n_it && alive; ++i) {
            const int blk = i % n_blk;
            uint32_t em = 0u;        // largest |E / 4|
            // ---------------------------------------------------- first pass: K_c and V_c
#pragma unroll 1
            for (int c = 0; c < NCH; ++c) {
                // the E columns of the next chunk fly while this one is worked on
                const size_t off = eo + ((c + 1) & (NCH - 1)) * 16;
                const ERow<EF32> nk = load_e<EF32>(a.Ek, off), nv = load_e<EF32>(a.Ev, off);
                const int st = c & 1;
                if (!(alive = warp_wait(&bars->pre1_full[st], (uint32_t)((2 * i + (c >> 1)) & 1), abort_flag, 1, lim))) break;
                tc_fence_after_sync();
                uint32_t cf[NJ][4], none[1][4];
                {
                    float x[NJ][8];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) tmem_ld_32x32b_x8(t_lane + (st ? T_DQ : T_PRE) + j * 16 + wg * 8, x[j]);
                    tmem_wait_ld();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0 && !(a.test_withhold && i == 0 && c == 0)) mbar_arrive(&bars->pre_empty[st]);
                    gate_coefficients<SILU, false>(x, cf, none);
                }
                // where the operand tiles go: free once the products that read them last have completed
                if (c == 0) { if (i >= 1) alive = warp_wait(&bars->blk_done, (uint32_t)((i - 1) & 1), abort_flag, 2, lim); }
                else if (c >= 2) alive = warp_wait(&bars->kv_free[st], (uint32_t)(i & 1), abort_flag, 3, lim);
                if (!alive) break;
                unsigned char* kd = sm + (st ? M::DS : M::B0) + r * 128;
#pragma unroll
                for (int t = 0; t < 2; ++t) {      // K to the first tile, V to the one behind it
                    uint32_t e4[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        e4[p] = e_pair<EF32>(t == 0 ? ek : ev, p);
                        em = max_f16x2(em, e4[p] & 0x7fff7fffu);
                    }
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
                        st_shared_v4(kd + t * ATOM + (((2 * j + wg) ^ x7) << 4), mul_f16x2(cf[j][0], e4[0]), mul_f16x2(cf[j][1], e4[1]), mul_f16x2(cf[j][2], e4[2]), mul_f16x2(cf[j][3], e4[3]));
                }
                if (c == NCH - 1) {
                    const float m = warp_max(larger_half(em));
                    if (lane == 0) bars->red_e[warp] = m;
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->kv_full[st]);
                ek = nk;
                ev = nv;
            }
            if (!alive) break;
            // ---------------------------------------------------- second pass: K_c again; dE rows, node gradients
            size_t eo_next = eo;
#pragma unroll 1
            for (int c = 0; c < NCH; ++c) {
                if (c == NCH - 1 && i + 1 < n_it) eo_next = e_row(a, b, __ldg(&meta[(size_t)((i + 1) % n_blk) * IBLK].x)) * D + h * HD + wg * 8;
                const size_t off = eo_next + ((c + 1) & (NCH - 1)) * 16;
                const ERow<EF32> nk = load_e<EF32>(a.Ek, off), nv = load_e<EF32>(a.Ev, off);
                const int st = c & 1, use = 2 * i + (c >> 1);
                if (!(alive = warp_wait(&bars->pre2_full[st], (uint32_t)(use & 1), abort_flag, 1, lim))) break;
                tc_fence_after_sync();
                uint32_t cf[NJ][4], sp[NJ][4];
                {
                    float x[NJ][8];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) tmem_ld_32x32b_x8(t_lane + T_PRE + j * 16 + wg * 8, x[j]);
                    tmem_wait_ld();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars->pre_empty[0]);
                    gate_coefficients<SILU, true>(x, cf, sp);
                }
                if (c == 0) alive = warp_wait(&bars->sdp_full, (uint32_t)(i & 1), abort_flag, 4, lim);
                else alive = warp_wait(&bars->kg_free[(c - 1) & 1], (uint32_t)((2 * i + ((c - 1) >> 1)) & 1), abort_flag, 5, lim);
                if (!alive) break;
                {
                    uint32_t e4[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) e4[p] = e_pair<EF32>(ek, p);
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
                        st_shared_v4(sm + M::B0 + r * 128 + (((2 * j + wg) ^ x7) << 4), mul_f16x2(cf[j][0], e4[0]), mul_f16x2(cf[j][1], e4[1]), mul_f16x2(cf[j][2], e4[2]), mul_f16x2(cf[j][3], e4[3]));
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->kg_full[st]);
                if (c == 0) {      // the block's factors, from the step warps
                    if (!(alive = warp_wait(&bars->pds_full, (uint32_t)(i & 1), abort_flag, 8, lim))) break;
                    if (i > 0 && bars->dw_fresh) flush((i - 1) / n_blk, bars->fw_old);       // (blk_done has been waited for)
                }
                if (!(alive = warp_wait(&bars->dkv_full[st], (uint32_t)(use & 1), abort_flag, 6, lim))) break;
                tc_fence_after_sync();
                float* gk = a.dEk + eo + c * 16;
                float* gv = a.dEv + eo + c * 16;
                const bool live = blk * IBLK + r < n_items;
                const float fs = bars->fs, fm = bars->fm, oe = ov * inverse(fs);
                uint32_t m0[4], m1[4];
#pragma unroll
                for (int q = 0; q < 2; ++q) {      // four columns at a time
                    float dk[NJ][4], dv[NJ][4];
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        tmem_ld_x4(t_lane + T_DP + j * 16 + wg * 8 + q * 4, dk[j]);
                        tmem_ld_x4(t_lane + T_DP + 64 + j * 16 + wg * 8 + q * 4, dv[j]);
                    }
                    tmem_wait_ld();
                    if (q == 1) {          // all columns are in registers
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->dkv_empty);
                    }
                    float ok[4], ovv[4];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const int pp = 2 * q + p;
                        const f32x2 e = unpack_h2(e_pair<EF32>(ek, pp)), f0 = unpack_h2(e_pair<EF32>(ev, pp));
                        const f32x2 f = mul2(f0, pack2(fs, fs));
                        f32x2 dc[NJ], sk = 0ull, sv = 0ull;
#pragma unroll
                        for (int j = 0; j < NJ; ++j) {
                            const f32x2 k2 = pack2(dk[j][2 * p], dk[j][2 * p + 1]), v2 = pack2(dv[j][2 * p], dv[j][2 * p + 1]);
                            const f32x2 cj = unpack_h2(cf[j][pp]);
                            sk = j == 0 ? mul2(cj, k2) : fma2(cj, k2, sk);
                            sv = j == 0 ? mul2(cj, v2) : fma2(cj, v2, sv);
                            dc[j] = fma2(f, v2, mul2(e, k2));
                        }
                        const f32x2 m = pack2(-1.f, -1.f), ka = pack2(TAN_PI_8, TAN_PI_8), kn = pack2(-TAN_PI_8, -TAN_PI_8);
                        const f32x2 u0 = add2(dc[0], dc[2]), u1 = fma2(dc[2], m, dc[0]), v0 = fma2(dc[3], kn, dc[1]), v1 = fma2(dc[1], ka, dc[3]);
                        f32x2 d0 = add2(u0, v0), d3 = fma2(v0, m, u0), d1 = add2(u1, v1), d2 = fma2(v1, m, u1);
                        if (SILU) {
                            d0 = mul2(d0, unpack_h2(sp[0][pp])); d1 = mul2(d1, unpack_h2(sp[1][pp]));
                            d2 = mul2(d2, unpack_h2(sp[2][pp])); d3 = mul2(d3, unpack_h2(sp[3][pp]));
                        }
                        // moments over the nodes
                        const float fa = fm * 0.9238795325f, fb = fm * 0.3826834324f;
                        const f32x2 c8 = pack2(fm, fm), ta = pack2(fa, fa), tb = pack2(fb, fb);
                        const f32x2 s = mul2(add2(add2(d0, d3), add2(d1, d2)), c8);
                        const f32x2 x = fma2(fma2(d2, m, d1), tb, mul2(fma2(d3, m, d0), ta));
                        float lo, hi;
                        unpack2(s, lo, hi); m0[pp] = pack_f16x2_sat(lo, hi);
                        unpack2(x, lo, hi); m1[pp] = pack_f16x2_sat(lo, hi);
                        unpack2(sk, ok[2 * p], ok[2 * p + 1]);
                        unpack2(sv, ovv[2 * p], ovv[2 * p + 1]);
                    }
                    if (live) {
                        red_v4(gk + q * 4, ok[0] * oe, ok[1] * oe, ok[2] * oe, ok[3] * oe);
                        red_v4(gv + q * 4, ovv[0] * ov, ovv[1] * ov, ovv[2] * ov, ovv[3] * ov);
                    }
                }
                // the tile of the moments takes two chunks: free once the dW product of the first two has read it
                if (c == 2 && !(alive = warp_wait(&bars->dp_free, (uint32_t)(i & 1), abort_flag, 7, lim))) break;
                unsigned char* zd = sm + M::B1 + r * 128;
                st_shared_v4(zd + (((4 * st + wg) ^ x7) << 4), m0[0], m0[1], m0[2], m0[3]);
                st_shared_v4(zd + (((4 * st + 2 + wg) ^ x7) << 4), m1[0], m1[1], m1[2], m1[3]);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->dpre_full[st]);
                ek = nk;
                ev = nv;
            }
            eo = eo_next;
        }
        if (n_it > 0 && alive && warp_wait(&bars->blk_done, (uint32_t)((n_it - 1) & 1), abort_flag, 8, lim)) flush((n_it - 1) / n_blk, bars->fw);
    } else if (warp < GATE_WARPS + SM_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        // ======================================================== softmax (item r, steps 64 half ..), then dQ (step r)
        const int half = (warp >> 2) & 1, r = tid & 127, x7 = r & 7;
        const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const int2* meta = it.meta + (size_t)bt * it.IB * IBLK + r;
        float acc[2][16];
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[0][e] = acc[1][e] = 0.f;
        int range = n_it > 0 ? __ldg(&meta[0].y) : 0;
        bool alive = true;
        const int len = TM >> level;
        for (int i = 0; i < n_it; ++i) {
            const int seg = i / n_blk;
            const int lo = max(range & 255, seg * len), hi = min(range >> 8, seg * len + len - 1);
            if (i + 1 < n_it) range = __ldg(&meta[(size_t)((i + 1) % n_blk) * IBLK].y);
            if (!(alive = warp_wait(&bars->sdp_full, (uint32_t)(i & 1), abort_flag, 9, lim))) break;
            tc_fence_after_sync();
            uint32_t p2[32];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int tb = half * 64 + k * 16;
                float s[16];
                tmem_ld_32x32b_x16(t_lane + T_S + tb, s);
                tmem_wait_ld();
                const bool full = __all_sync(0xffffffffu, lo <= tb && hi >= tb + 15);
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 ls = *reinterpret_cast<const float4*>(lse_sh + tb + e);
                    s[e] -= ls.x; s[e + 1] -= ls.y; s[e + 2] -= ls.z; s[e + 3] -= ls.w;
                }
                if (!full) {
                    const int l0 = max(lo - tb, 0), h0 = min(hi - tb, 15);
                    const unsigned mask = l0 > h0 ? 0u : ((0xffffffffu >> (31 - h0)) & (0xffffffffu << l0));
#pragma unroll
                    for (int e = 0; e < 16; ++e) s[e] = (mask >> e) & 1u ? s[e] : -INFINITY;
                }
#pragma unroll
                for (int e = 0; e < 16; e += 2) p2[k * 8 + e / 2] = pack_f16x2_sat(ex2_approx(s[e]), ex2_approx(s[e + 1]));
            }
            // this item's part in the choice of the block's factor of dS
            uint32_t pm2 = 0u;
            float xm = 0.f;
#pragma unroll
            for (int k = 0; k < 32; ++k) pm2 = max_f16x2(pm2, p2[k]);
#pragma unroll 1
            for (int tb = half * 64; tb < half * 64 + 64; tb += 16) {
                float dp[16];
                tmem_ld_32x32b_x16(t_lane + T_DP + tb, dp);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 dl = *reinterpret_cast<const float4*>(dl_sh + tb + e);
                    xm = fmaxf(fmaxf(fmaxf(xm, fabsf(dp[e] - dl.x)), fmaxf(fabsf(dp[e + 1] - dl.y), fabsf(dp[e + 2] - dl.z))), fabsf(dp[e + 3] - dl.w));
                }
            }
            const float pm = larger_half(pm2);
            if (pm == 0.f) xm = 0.f;
            const float wb = warp_max(pm * xm), wx = warp_max(xm), wp = warp_max(pm);
            if (lane == 0) { bars->red_b[warp - GATE_WARPS] = wb; bars->red_x[warp - GATE_WARPS] = wx; bars->red_p[warp - GATE_WARPS] = wp; }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_read);
            if (!(alive = warp_wait(&bars->s_read, (uint32_t)(i & 1), abort_flag, 10, lim))) break;
            tc_fence_after_sync();
            const float fs = ds_scale(bars), cs = LN2 * fs;
            // the scores have been read by both halves: P^T takes their first 64 columns, dS^T the other 64, both over the smallest row
            // factor (they are summed over the steps); dS^T for dQ keeps the rows' own
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int tb = half * 64 + k * 16;
                float dp[16];
                uint32_t g2[8], d2[8];
                tmem_ld_32x32b_x16(t_lane + T_DP + tb, dp);
                *reinterpret_cast<uint4*>(g2) = *reinterpret_cast<const uint4*>(gf_sh + tb);
                *reinterpret_cast<uint4*>(g2 + 4) = *reinterpret_cast<const uint4*>(gf_sh + tb + 8);
#pragma unroll
                for (int e = 0; e < 8; ++e) d2[e] = mul_f16x2(p2[k * 8 + e], g2[e]);
                tmem_st_x8(t_lane + T_S + half * 32 + k * 8, d2);
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 dl = *reinterpret_cast<const float4*>(dl_sh + tb + e);
                    d2[e / 2] = mul_f16x2(p2[k * 8 + e / 2], pack_f16x2_sat((dp[e] - dl.x) * cs, (dp[e + 1] - dl.y) * cs));
                    d2[e / 2 + 1] = mul_f16x2(p2[k * 8 + e / 2 + 1], pack_f16x2_sat((dp[e + 2] - dl.z) * cs, (dp[e + 3] - dl.w) * cs));
                }
                unsigned char* ds = sm + M::DS + half * ATOM + r * 128;
                st_shared_v4(ds + (((2 * k) ^ x7) << 4), d2[0], d2[1], d2[2], d2[3]);
                st_shared_v4(ds + (((2 * k + 1) ^ x7) << 4), d2[4], d2[5], d2[6], d2[7]);
#pragma unroll
                for (int e = 0; e < 8; ++e) d2[e] = mul_f16x2(d2[e], g2[e]);
                tmem_st_x8(t_lane + T_S + 64 + half * 32 + k * 8, d2);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            fence_proxy_async_smem();
            if (warp == GATE_WARPS) {      // the factors for the gate warps (red_e is theirs)
                if (!(alive = warp_wait(&bars->kv_full[1], 1u, abort_flag, 3, lim))) break;
                // what the moments are at most: 128 steps, basis of at most 1.85, four coefficients into each of four nodes, a
                // derivative below 1.1; dS, P, dO (below 2^14) and q (log2(e) / 8) at their largest
                constexpr float SUM = 128.0f * 1.85f * 16.0f * 1.1f;
                const float qm = 0.125f * 1.4426950409f * __uint_as_float(bars->qmax);
                const float top = SUM * fs * max8(bars->red_e) * (qm * max8(bars->red_b) + 16384.0f * max8(bars->red_p));
                if (lane == 0) {
                    // The unit of the dW sums stays while the blocks fit (64 times smaller than the first one needs: rarely more than one
                    // a segment); with a smaller one, or a new segment, what has been summed leaves tensor memory.
                    const float fits = fs * scale_to_f16(top, 50, 30), fw = bars->fw;
                    const bool fresh = i % n_blk == 0 || fw > fits;
                    bars->dw_fresh = fresh;
                    bars->fw_old = fw;
                    if (fresh) bars->fw = fits * 0.015625f;
                    bars->fs = fs;
                    bars->fm = bars->fw * inverse(fs);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->pds_full);
            int rr = r;
            asm volatile("" : "+r"(rr));          // formed here in every block, not kept in registers
            float beta[NJ];
            basis(rr, level, beta);
            const float inv = inverse(fs);
#pragma unroll
            for (int e = 0; e < NJ; ++e) beta[e] *= inv;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                if (!(alive = warp_wait(&bars->dq_full[half], (uint32_t)((2 * i + cc) & 1), abort_flag, 11, lim))) break;
                tc_fence_after_sync();
                float v[2][16];        // a coefficient's columns at a time, the next ones in flight
                tmem_ld_32x32b_x16(t_lane + T_DQ, v[0]);
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    tmem_wait_ld();
                    if (j + 1 < NJ) {
                        tmem_ld_32x32b_x16(t_lane + T_DQ + (j + 1) * 16, v[(j + 1) & 1]);
                    } else {
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->dq_empty);
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[cc][e] = fmaf(beta[j], v[j & 1][e], acc[cc][e]);
                }
            }
            if (!alive) break;
        }
        if (alive && t0 + r < a.T) {
            const int k = rx_sh[r];
            const float sc = k == 255 ? NAN : t0 + r < Lb ? 0.125f / LN2 * exp2f(-kappa - (float)(emin + k)) : 0.f;
#pragma unroll
            for (int cc = 0; cc < 2; ++cc)
#pragma unroll
                for (int e = 0; e < 16; e += 4)
                    *reinterpret_cast<float4*>(a.dQ + (row0 + r) * HD + (half + 2 * cc) * 16 + e) =
                        make_float4(acc[cc][e] * sc, acc[cc][e + 1] * sc, acc[cc][e + 2] * sc, acc[cc][e + 3] * sc);
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == W_LOAD && lane == 0) {
            // ==================================================== loader: A per block; W' (and dO') chunks for both passes
            const unsigned char* img = it.a_img + (size_t)bt * it.IB * NK * ATOM;
            const unsigned char* dimg = NK == 1 ? nullptr : w.do_img + ((size_t)bt * a.H + h) * NCH * ATOM;
            int np = 0, nd = 0;
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                const int seg = i / n_blk, blk = i - seg * n_blk;
                const unsigned char* wi = w.w_img + (size_t)((((1 << level) - 1 + seg) * a.H + h) * NCH) * NK * WPIECE;
                if (i >= 1 && !(alive = mbar_wait(&bars->blk_done, (uint32_t)((i - 1) & 1), abort_flag, 12, lim))) break;
                mbar_expect_tx(&bars->a_full, NK * ATOM);
                bulk_load(sm + M::A, img + (size_t)blk * NK * ATOM, NK * ATOM, &bars->a_full);
                for (int p = 0; p < 2 * NCH * NK && alive; ++p, ++np) {
                    const int sw = np & 1, uw = np >> 1;
                    if (NK == 2 && p % NK == 0) {
                        const int sd = nd & 1, ud = nd >> 1;
                        if (ud >= 1 && !(alive = mbar_wait(&bars->do_free[sd], (uint32_t)((ud - 1) & 1), abort_flag, 13, lim))) break;
                        mbar_expect_tx(&bars->do_full[sd], ATOM);
                        bulk_load(sm + M::DO + sd * ATOM, dimg + (size_t)((p / NK) % NCH) * ATOM, ATOM, &bars->do_full[sd]);
                        ++nd;
                    }
                    if (uw >= 1 && !(alive = mbar_wait(&bars->w_free[sw], (uint32_t)((uw - 1) & 1), abort_flag, 14, lim))) break;
                    mbar_expect_tx(&bars->w_full[sw], WPIECE);
                    bulk_load(sm + M::W + sw * WPIECE, wi + (size_t)(p % (NCH * NK)) * WPIECE, WPIECE, &bars->w_full[sw]);
                }
                mbar_wait<100>(&bars->a_full, (uint32_t)(i & 1), &bars->drain_flag, 15);
            }
            // no copy of this CTA is in flight when it ends
            for (int s = 0; s < 2; ++s) {
                if (np > s) mbar_wait<100>(&bars->w_full[s], (uint32_t)(((np - 1 - s) >> 1) & 1), &bars->drain_flag, 15);
                if (nd > s) mbar_wait<100>(&bars->do_full[s], (uint32_t)(((nd - 1 - s) >> 1) & 1), &bars->drain_flag, 15);
            }
        } else if (warp == W_GATE && lane == 0) {
            // ==================================================== gate products of both passes
            const uint32_t idesc = umma_idesc_16(IBLK, 64, 0, 0, 0, 0);
            int np = 0, n0 = 0, n1 = 0;            // pieces; uses of the accumulators at T_PRE and T_DQ
            bool alive = true;
            for (int i = 0; i < n_it && alive; ++i) {
                if (!(alive = mbar_wait(&bars->a_full, (uint32_t)(i & 1), abort_flag, 16, lim))) break;
                for (int p8 = 0; p8 < 2 * NCH && alive; ++p8) {
                    const int c = p8 & 3;
                    const bool second = p8 >= NCH;
                    const bool slot1 = !second && (c & 1);
                    if (slot1) {
                        // the first use in a block also waits for the last dQ' of the block before to be read
                        if (c == 1 && i >= 1 && !(alive = mbar_wait(&bars->dq_empty, 1u, abort_flag, 17, lim))) break;
                        if (n1 >= 1 && !(alive = mbar_wait(&bars->pre_empty[1], (uint32_t)((n1 - 1) & 1), abort_flag, 18, lim))) break;
                        ++n1;
                    } else {
                        if (n0 >= 1 && !(alive = mbar_wait(&bars->pre_empty[0], (uint32_t)((n0 - 1) & 1), abort_flag, 19, lim))) break;
                        ++n0;
                    }
                    for (int p = 0; p < NK; ++p, ++np) {
                        if (!(alive = mbar_wait(&bars->w_full[np & 1], (uint32_t)((np >> 1) & 1), abort_flag, 20, lim))) break;
                        tc_fence_after_sync();
                        const uint32_t ab = smem_u32(sm + M::A + p * ATOM), wb = smem_u32(sm + M::W + (np & 1) * WPIECE);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16_ss(tmem + (slot1 ? T_DQ : T_PRE), umma_desc_k_sw128(ab + k * 32), umma_desc_k_sw128(wb + k * 32), idesc, (p | k) != 0);
                        umma_commit(&bars->w_free[np & 1]);
                    }
                    if (alive) umma_commit(second ? &bars->pre2_full[c & 1] : &bars->pre1_full[c & 1]);
                }
            }
            umma_commit(&bars->drain);
        } else if (warp == W_ATT && lane == 0) {
            // ==================================================== all other products
            const uint32_t id_s = umma_idesc_16(IBLK, TM, 0, 0, 0, 0), id_kv = umma_idesc_16(IBLK, 64, 0, 1, 0, 0),
                           id_q = umma_idesc_16(TM, 64, 1, 1, 0, 0), id_w = umma_idesc_16(128, 64, 1, 1, 0, 0);
            const uint32_t qb = smem_u32(sm + M::Q), db = smem_u32(sm + M::DO), b0 = smem_u32(sm + M::B0), b1 = smem_u32(sm + M::B1),
                           ds = smem_u32(sm + M::DS), ab = smem_u32(sm + M::A);
            int nd = 0;
            bool alive = true;
            // dO' chunk c: resident, or the next stage of the ring
            auto do_tile = [&](int c) -> uint32_t {
                if (NK == 1) return db + c * ATOM;
                alive = mbar_wait(&bars->do_full[nd & 1], (uint32_t)((nd >> 1) & 1), abort_flag, 21, lim);
                tc_fence_after_sync();
                return db + (nd & 1) * ATOM;
            };
            auto do_release = [&]() { if (NK == 2) { umma_commit(&bars->do_free[nd & 1]); ++nd; } };
            auto dw = [&](int i, int pair) {          // chunks 2 pair and 2 pair + 1
                for (int st = 0; st < 2; ++st)
                    if (!(alive = mbar_wait(&bars->dpre_full[st], (uint32_t)((2 * i + pair) & 1), abort_flag, 22, lim))) return;
                tc_fence_after_sync();
                const bool fresh = *reinterpret_cast<volatile int*>(&bars->dw_fresh) != 0;
                // M = 128 channels; with 64 the second half reads the tile behind the states and is not used
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    umma_bf16_ss(tmem + T_DW + pair * 64, umma_desc_mn_sw128(ab + k * 2048, ATOM, 1024), umma_desc_mn_sw128(b1 + k * 2048, ATOM, 1024), id_w, k != 0 || !fresh);
                if (pair == 0) umma_commit(&bars->dp_free);
            };
            for (int i = 0; i < n_it && alive; ++i) {
                if (i >= 1 && !(alive = mbar_wait(&bars->dkv_empty, 1u, abort_flag, 24, lim))) break;      // chunk 3 of the block before
                for (int c = 0; c < NCH; ++c) {
                    if (!(alive = mbar_wait(&bars->kv_full[c & 1], (uint32_t)((2 * i + (c >> 1)) & 1), abort_flag, 25, lim))) break;
                    const uint32_t dt = do_tile(c);
                    if (!alive) break;
                    tc_fence_after_sync();
                    const uint32_t kt = (c & 1) ? ds : b0, vt = (c & 1) ? ds + ATOM : b1;
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_ss(tmem + T_S, umma_desc_k_sw128(kt + k * 32), umma_desc_k_sw128(qb + c * ATOM + k * 32), id_s, (c | k) != 0);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_bf16_ss(tmem + T_DP, umma_desc_k_sw128(vt + k * 32), umma_desc_k_sw128(dt + k * 32), id_s, (c | k) != 0);
                    do_release();
                    if (c < 2) umma_commit(&bars->kv_free[c]);
                }
                if (!alive) break;
                umma_commit(&bars->sdp_full);
                if (!(alive = mbar_wait(&bars->pds_full, (uint32_t)(i & 1), abort_flag, 26, lim))) break;
                tc_fence_after_sync();
                for (int c = 0; c < NCH; ++c) {
                    if (c >= 1 && !(alive = mbar_wait(&bars->dkv_empty, (uint32_t)((c - 1) & 1), abort_flag, 27, lim))) break;
                    const uint32_t dt = do_tile(c);
                    if (!alive) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_16_ts(tmem + T_DP, tmem + T_S + 64 + k * 8, umma_desc_mn_sw128(qb + c * ATOM + k * 2048, ATOM, 1024), id_kv, k != 0);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_16_ts(tmem + T_DP + 64, tmem + T_S + k * 8, umma_desc_mn_sw128(dt + k * 2048, ATOM, 1024), id_kv, k != 0);
                    do_release();
                    umma_commit(&bars->dkv_full[c & 1]);
                    if (c == 2) dw(i, 0);
                    if (!alive) break;
                    if (!(alive = mbar_wait(&bars->kg_full[c & 1], (uint32_t)((2 * i + (c >> 1)) & 1), abort_flag, 28, lim))) break;
                    if (4 * i + c >= 1 && c >= 1 && !(alive = mbar_wait(&bars->dq_empty, (uint32_t)((c - 1) & 1), abort_flag, 29, lim))) break;
                    tc_fence_after_sync();
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        umma_bf16_ss(tmem + T_DQ, umma_desc_mn_sw128(ds + k * 2048, ATOM, 1024), umma_desc_mn_sw128(b0 + k * 2048, ATOM, 1024), id_q, k != 0);
                    umma_commit(&bars->dq_full[c & 1]);
                    umma_commit(&bars->kg_free[c & 1]);
                }
                if (alive) dw(i, 1);
                if (alive) umma_commit(&bars->blk_done);
            }
            umma_commit(&bars->drain);
        }
    }
    // ---------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (warp == W_GATE) {
        mbar_wait<100>(&bars->drain, 0u, &bars->drain_flag, 30);
        tc_fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
    if (tid == 0 && (bars->abort_flag | bars->drain_flag)) atomicOr(status, bars->abort_flag | bars->drain_flag);
}

}  // namespace bwd

int backward(const FlashArgs& a, const Items& it, const Ws& w, int* status, cudaStream_t st) {
    const dim3 grid(a.nT, a.H, a.B);
#define MBEMA_SMOOTH(S_, NK_, E_)                                                                                                     \
    do {                                                                                                                               \
        MBEMA_CUDA_TRY(cudaFuncSetAttribute(bwd::k_smooth_bwd<S_, NK_, E_>, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd::L<NK_>::SMEM)); \
        bwd::k_smooth_bwd<S_, NK_, E_><<<grid, bwd::THREADS, bwd::L<NK_>::SMEM, st>>>(a, it, w, status);                                    \
    } while (0)
#define MBEMA_SMOOTH_E(S_, NK_) do { if (a.e_dt == MBEMA_F32) MBEMA_SMOOTH(S_, NK_, true); else MBEMA_SMOOTH(S_, NK_, false); } while (0)
    if (a.N == 64) { if (a.silu) MBEMA_SMOOTH_E(true, 1); else MBEMA_SMOOTH_E(false, 1); }
    else { if (a.silu) MBEMA_SMOOTH_E(true, 2); else MBEMA_SMOOTH_E(false, 2); }
#undef MBEMA_SMOOTH_E
#undef MBEMA_SMOOTH
    return check_launch();
}

}  // namespace smooth
}  // namespace mbema
